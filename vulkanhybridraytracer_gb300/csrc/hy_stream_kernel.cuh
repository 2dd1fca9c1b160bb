// The tile-stream shadow kernel (the default shadow schedule), instantiated in
// hy_stream_raw.cu (raw per-light images), hy_stream_accum.cu (folded into the
// history) and hy_stream_two.cu (two-level structures), so the variants
// compile in parallel.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "hy_device.cuh"
#include "hy_pass.h"
#include "hy_shade.cuh"
#include "hy_stream.cuh"

namespace hy {

// ---------------------------------------------------------------------------------
// Shadow rays, light-major over a tile: a warp takes an 8x4 tile (or, near the end of
// the launch, some of a tile's lights) and, light by light, traces all 32 x n_rays
// samples of its pixels, item q being sample q % n_rays of pixel q / n_rays; idle lanes
// take the items in order, a round of node visits at a time (stream_round).  Lane i sets
// up light l for pixel i (its G-buffer texel, the skip tests of
// shadowRaygen.rgen:43-63) and publishes position, distance, sampleDisk's frame
// (tangent, bitangent, position + L: the same for every sample of the
// pixel-light) and the RNG state of its first sample in shared memory; every
// lane then traces items without waiting for the others' rays, counting unoccluded
// samples per pixel with shared-memory atomics; once the warp's items for light l are
// all traced, lane i folds pixel i's count into its factor.  A lane waits only at
// the end of a light (for the slowest sum of spp rays) instead of after every
// pixel-light (for the slowest single ray), and the samples in flight stay within a few
// adjacent pixels of one light.  Seeds as in k_shadow_group (LCG jump-ahead),
// so the rays equal those of k_shadow.
// ---------------------------------------------------------------------------------
// ONE: one ray per pixel and light (stream_tile_one).
template <bool TWO>
struct OneRayBlockT {
    WalkAreaT<TWO> warp[4];
};
template <bool COUNT, bool ACCUM, int MINB, bool TWO = false, bool SHORT = false, bool ONE = false>
__global__ void __launch_bounds__(128, MINB) k_shadow_stream(const SceneDev S, const PassParams P) {
    __shared__ std::conditional_t<ONE, OneRayBlockT<TWO>, StreamSlotsT<4, TWO>> sm;
    __shared__ uint2 s_stack[SHORT ? kShortStack * 128 : 1];
    __shared__ float s_world[TWO ? 6 * 128 : 1];  // two-level: WorldRaySlot words
    LaneStats ls;
    const uint32_t lane = threadIdx.x & 31;
    uint2 stk[kStackMax];
    ShadowLane s;
    Trav t;
    std::conditional_t<TWO, WorldRaySlot, RayPre> r{};
    if constexpr (TWO) {
        r.p = s_world + threadIdx.x;
        if constexpr (ONE) r.ray = &sm.warp[threadIdx.x >> 5].ray[lane];
        else r.ray = &sm.scratch[threadIdx.x >> 5].walk.ray[lane];
    }
    uint32_t chunk_cur = 0, chunk_end = 0, nn = 0, nt = 0;
    const bool reference = P.rng_mode == HY_RNG_REFERENCE;
    for (;;) {
        if (chunk_cur == chunk_end) {
            uint32_t t0 = 0;
            if (lane == 0) t0 = atomicAdd(P.queue, P.chunk);
            t0 = __shfl_sync(0xffffffffu, t0, 0);
            if (t0 >= P.units) break;
            chunk_cur = t0;
            chunk_end = min(t0 + P.chunk, P.units);
        }
        // a unit: a whole tile, or (the last ones) one part of a tile's lights
        const uint32_t unit = chunk_cur++;
        uint32_t tile = unit, l0 = 0, l1 = P.num_lights;
        if (unit >= P.whole_tiles) {
            const uint32_t u = unit - P.whole_tiles, part = u % P.parts;
            tile = P.whole_tiles + u / P.parts;
            l0 = part * P.part_lights;
            l1 = min(l0 + P.part_lights, P.num_lights);
        }
        auto walk = [&](auto stack) {
            if constexpr (ONE)
                stream_tile_one<COUNT, TWO, ACCUM ? 1 : 0>(S, P, tile, l0, l1, reference, ACCUM,
                                                           sm.warp[threadIdx.x >> 5], stack, t, r, s, ls, nn, nt);
            else
                stream_tile<COUNT, TWO, ACCUM ? 1 : 0>(S, P, tile, l0, l1, reference, ACCUM, sm, stack, t, r, s, ls, nn, nt);
        };
        if constexpr (SHORT) walk(SplitStack{s_stack + threadIdx.x, stk});
        else walk((uint2*)stk);
    }
    if (COUNT) { ls.nodes += nn; ls.tris += nt; }
    flush_stats(ls, P.stats);
}

// one-level kernels: the register cap as resident 128-thread blocks per SM
// (5-8), or 8 with the first stack entries in shared memory; the caller's choice, 8
// without (one ray per light, 4K with 64 lights, shadow kernel at 5 / 6 / 7 / 8 / 8 with
// shared entries: 98.3 / 90.3 / 88.1 / 89.7 / 90.2 ms; 1700x900 with 4: 1.13 / 1.06 /
// 1.04 / 1.06 / 1.09 ms)
template <bool ACCUM, bool ONE>
static void* stream_kernel_flat(bool count, int minb, bool short_stack) {
    if (short_stack)
        return count ? (void*)k_shadow_stream<true, ACCUM, 8, false, true, ONE>
                     : (void*)k_shadow_stream<false, ACCUM, 8, false, true, ONE>;
    if (minb >= 8)
        return count ? (void*)k_shadow_stream<true, ACCUM, 8, false, false, ONE>
                     : (void*)k_shadow_stream<false, ACCUM, 8, false, false, ONE>;
    if (minb == 7)
        return count ? (void*)k_shadow_stream<true, ACCUM, 7, false, false, ONE>
                     : (void*)k_shadow_stream<false, ACCUM, 7, false, false, ONE>;
    if (minb >= 6)
        return count ? (void*)k_shadow_stream<true, ACCUM, 6, false, false, ONE>
                     : (void*)k_shadow_stream<false, ACCUM, 6, false, false, ONE>;
    return count ? (void*)k_shadow_stream<true, ACCUM, 5, false, false, ONE>
                 : (void*)k_shadow_stream<false, ACCUM, 5, false, false, ONE>;
}

}  // namespace hy
