// Tile streams: the warp-cooperative shadow-ray schedule shared by the hybrid
// pass (hy_pass.cu) and the path-traced mode (hy_pt.cu).  Per light, each lane
// publishes one pixel's shadow-ray inputs (position, distance, sampleDisk's
// frame, the RNG state of the pixel-light's first sample) in shared memory;
// the warp then traces the 32 x n_rays samples as items q (sample q % n_rays of
// pixel q / n_rays), taken in order by whichever lanes are free, each lane
// walking its rays with several node visits per scheduling round and without
// waiting for the others' rays to end; the triangles a round reaches are tested
// by the whole warp together; unoccluded samples are counted per pixel with
// shared-memory atomics.
#pragma once
#include <cuda_runtime.h>

#include "hy_device.cuh"
#include "hy_pass.h"
#include "hy_shade.cuh"

namespace hy {

// Per-warp shared state of the tile streams, per pixel of the warp's tile and
// the current light: position and distance to the light; the disk frame of
// sampleDisk (position + L, tangent, bitangent); the RNG state of the
// pixel-light's first sample (w of PL, as bits); a not-traced mark (w of T,
// 0xffffffff); the unoccluded count (w of B, as bits).
// Items of a light are traced in the order of their disk samples, sorted in
// chunks of SORT items per warp and light.
// The size matters beyond occupancy: shared memory and L1 share each SM's
// 256 KB, and the driver carves shared memory in steps (..., 100, 132, 164,
// 196 KB).  The sort's scratch and the walk's are used in turn and overlap, so
// at 4 warps per block and 8 blocks per SM this layout (15.3 KB, + 1 KB the
// driver keeps per block) takes the 132 KB step and leaves the kernel 124 KB of
// L1 for the nodes, triangles and traversal stacks it re-reads; the two-level
// kernel (instance ids per pair, 3 KB of world rays) takes the 164 KB step.
constexpr uint32_t kSortItems = 512, kSortBuckets = 64;
constexpr uint32_t kPairs = 64;  // (ray, triangle) pairs a warp collects between two test phases

// A warp's walk: each lane's ray (direction, tmax) and the (ray, triangle) pairs
// waiting for their test.
template <bool TWO>
struct WalkAreaT {
    float4 ray[32];
    uint32_t rec[kPairs];             // triangle record
    uint32_t inst[TWO ? kPairs : 1];  // two-level: its instance
    uint8_t owner[kPairs];            // the lane whose ray it is
    uint32_t npairs;                  // pairs collected (may count past kPairs: those wait on their lanes)
};

template <int NW, bool TWO = false, uint32_t SORT = kSortItems>  // warps per block, items sorted together
struct StreamSlotsT {
    static constexpr uint32_t kSort = SORT;
    float4 pos[NW * 32];
    float4 PL[NW * 32];
    float4 T[NW * 32];
    float4 B[NW * 32];
    uint16_t order[NW][SORT];  // per warp: the traced items of the light ordered by their disk sample
    union Scratch {
        // the sort: the sample's cell per item, the cell counts / cursors
        struct {
            uint8_t key[SORT];
            uint32_t bucket[kSortBuckets];
        } sort;
        WalkAreaT<TWO> walk;
    };
    alignas(16) Scratch scratch[NW];
};
using StreamSlots = StreamSlotsT<4>;

constexpr uint32_t kNotTraced = 0xffffffffu;

// lane's slot for the current light; first_state: the RNG state of sample 0
// the current light's unoccluded-sample count of slot i
template <class Slots>
__device__ __forceinline__ uint32_t* unocc_count(Slots& sm, uint32_t i) {
    return reinterpret_cast<uint32_t*>(&sm.B[i].w);
}

template <class Slots>
__device__ __forceinline__ void stream_publish(Slots& sm, bool traced, f3 position, f3 L, float dist,
                                               uint32_t first_state) {
    const uint32_t i = threadIdx.x;
    if (traced) {
        const DiskFrame d = disk_frame(position, L);
        sm.pos[i] = make_float4(position.x, position.y, position.z, dist);
        sm.PL[i] = make_float4(d.PL.x, d.PL.y, d.PL.z, __uint_as_float(first_state));
        sm.T[i] = make_float4(d.T.x, d.T.y, d.T.z, 0.f);
        sm.B[i] = make_float4(d.B.x, d.B.y, d.B.z, 0.f);  // w: the unoccluded count, 0
    } else {
        sm.T[i].w = __uint_as_float(kNotTraced);
        sm.B[i].w = 0.f;
    }
}

// The triangles of the leaf slots a lane's last node visit hit, put into the
// warp's pair list; what does not fit stays in t.pend_bits.
template <bool TWO, class Area>
__device__ __forceinline__ void pairs_push(Area& w, Trav& t) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t at = atomicAdd(&w.npairs, (uint32_t)__popc(t.pend_bits));
    while (t.pend_bits && at < kPairs) {
        const uint32_t b = __ffs(t.pend_bits) - 1;
        t.pend_bits &= t.pend_bits - 1u;
        w.rec[at] = t.pend_base + b;
        w.owner[at] = (uint8_t)lane;
        if (TWO) w.inst[at] = t.inst;
        at++;
    }
}

// Tests the warp's pairs, one per lane: the lane takes the ray of the pair's
// owner (origin by shuffle, direction and tmax from the owner's slot; two-level:
// moved into the pair's instance) and sets it up for the test as the owner would
// have.  Returns the mask of owners with a hit.  All lanes call it, np uniform.
template <bool TWO, class Area, class RW>
__device__ __forceinline__ uint32_t pairs_test(const SceneDev& S, const Area& w, uint32_t np, const RW& r, float tmin,
                                               uint32_t* status) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t hits = 0;
    for (uint32_t b = 0; b < np; b += 32) {
        const uint32_t i = b + lane;
        const bool valid = i < np;
        const uint32_t owner = valid ? (uint32_t)w.owner[i] : lane;
        f3 o;
        if constexpr (TWO) {
            const int d = (int)owner - (int)lane;
            o = mk(r.p[d], r.p[d + 128], r.p[d + 256]);
        } else {
            o = mk(__shfl_sync(0xffffffffu, r.o.x, owner), __shfl_sync(0xffffffffu, r.o.y, owner),
                   __shfl_sync(0xffffffffu, r.o.z, owner));
        }
        if (valid) {
            const uint32_t rec = w.rec[i];
            if (rec >= S.num_tris) { atomicOr(status, HY_STATUS_BAD_INDEX); continue; }
            const float4 ray = w.ray[owner];
            f3 dir = mk(ray.x, ray.y, ray.z);
            if constexpr (TWO) {
                const float4* I = S.inst + (size_t)w.inst[i] * 4;
                const float4 r0 = __ldg(I), r1 = __ldg(I + 1), r2 = __ldg(I + 2);
                o = xform_point(r0, r1, r2, o);
                dir = xform_dir(r0, r1, r2, dir);
            }
            const float4* tp = S.tris + (size_t)rec * 3;
            float tt, b1, b2;
            if (tri_test(ray_pre(o, dir), __ldg(tp), __ldg(tp + 1), __ldg(tp + 2), tmin, ray.w, tt, b1, b2))
                hits |= 1u << owner;
        }
    }
    return __reduce_or_sync(0xffffffffu, hits);
}

// One round of a warp's walks: up to P.inner node visits per lane, then the
// triangles those visits reached, tested together.  All lanes call it; a lane with a
// ray (live) gets whether the ray is done and whether it is occluded.
//
// A lane does not test its triangles where it finds them: it puts (ray, triangle)
// pairs into the warp's list and walks on, and at the end of the round the warp's
// lanes take one pair each.  On the 1080p frame a node visit of the warp reaches
// 2.5 triangles, on 2.5 lanes: tested at once they took as many warp instructions
// as a third of the whole kernel; collected over a round they fill the lanes
// (4.85 -> 4.27 G warp instructions on the 960x540 frame, 15.5 -> 20.2 lanes each;
// 1080p shadow kernel 20.1 -> 17.9 ms, 1277x719 two-level 16.3 -> 13.0 ms).
// A lane whose ray has already found its occluder walks on until the round ends,
// where it would have waited for the round anyway.  The outcome of a ray does not
// change: any-hit walks visit the same nodes whatever was hit before, so the
// triangles tested are those of the plain walk up to its first hit and a few
// more of a ray that is known to be occluded by then.  A limit that runs out
// (node visits, stack) is reported only if none of the ray's waiting pairs hit.
// COUNT: the plain walk, each visit's triangles tested at once, so the counts are
// those of each ray's walk up to its first hit.
struct RoundResult { bool over, occluded; };
template <bool COUNT, bool TWO, class Area, class Stack, class RW>
__device__ __forceinline__ RoundResult stream_round(const SceneDev& S, const PassParams& P, Area& w, bool live,
                                                    Stack stk, Trav& t, RW& r, uint32_t& nn, uint32_t& nt) {
    const uint32_t lane = threadIdx.x & 31;
    RoundResult res{false, false};
    uint32_t limits = 0;
    if (live) {
        for (uint32_t it = 0, ni = max(P.inner, 1u); it < ni; it++) {
            if constexpr (COUNT) {
                if (trav_step<true, true, TWO>(S, r, 0.001f, t, stk, nn, nt, P.status)) {
                    res.over = true;
                    res.occluded = t.h.id != HY_NO_HIT;
                    break;
                }
            } else {
                if (trav_node<true, false, TWO>(S, r, 0.001f, t, stk, nn, DeferredStatus{limits})) {
                    res.over = true;
                    break;
                }
                if (t.pend_bits) {
                    pairs_push<TWO>(w, t);
                    if (t.pend_bits) break;  // the list is full: the rest after the test below
                }
            }
        }
    }
    if constexpr (!COUNT) {
        for (;;) {
            __syncwarp();
            const uint32_t np = min(w.npairs, kPairs);
            if (np == 0) break;
            const uint32_t hits = pairs_test<TWO>(S, w, np, r, 0.001f, P.status);
            if (lane == 0) w.npairs = 0;
            if ((hits >> lane) & 1u) { res.occluded = true; t.pend_bits = 0; }
            __syncwarp();
            if (__ballot_sync(0xffffffffu, live && t.pend_bits != 0) == 0) break;
            if (live && t.pend_bits) pairs_push<TWO>(w, t);
        }
    }
    if (limits && !res.occluded) atomicOr(P.status, limits);
    res.over = res.over || res.occluded;
    return res;
}

// ---- closest-hit walks of a warp, their triangles tested together ------------------
// (k_trace_closest.  For the G-buffer's primary rays, whose plain walks agree already,
// the later shrinking interval cost more than the tests: 1080p, the call 458 -> 543 us.)
// As stream_round, for closest-hit rays: pairs are collected over a round, each
// tested by one lane against its owner's interval as it was when the round began;
// hits meet in the owner's 64-bit key (distance, id; the lower id on equal
// distances), and the pair whose key is left hands its distance and barycentrics
// over.  The closest hit does not depend on the order of visits or on how early the
// interval shrinks, so it is the plain walk's, bit for bit (rays for which the box test's
// slack does not hold are not walked here: k_trace_closest); a ray may make a few more
// node visits.  A ray that runs into a limit is walked anew by itself (plain), so
// that the limit holds for the plain walk's visits.
template <bool TWO>
struct ClosestAreaT : WalkAreaT<TWO> {  // ray[].w: tmin
    unsigned long long key[32];         // per owner: (order-preserving distance bits, id)
    float4 best[32];                    // its distance and barycentrics
};

// distances as unsigned keys in order (-0 and +0 one key)
__device__ __forceinline__ uint32_t distance_key(float t) {
    const uint32_t b = __float_as_uint(__fadd_rn(t, 0.f));
    return b & 0x80000000u ? ~b : b | 0x80000000u;
}

template <bool TWO, class RW>
__device__ __forceinline__ void closest_start(ClosestAreaT<TWO>& w, Trav& t, RW& r, f3 o, f3 d, float tmin, float tmax) {
    const uint32_t lane = threadIdx.x & 31;
    w.ray[lane] = make_float4(d.x, d.y, d.z, tmin);
    w.key[lane] = ~0ull;
    trav_init(t, world_set(r, o, d), tmax);
}

// One round; live lanes get whether their walk is over (t.h then holds the hit).
// The interval shrinks only at the end of a round, the tests fill their lanes only
// over several visits: 2M incoherent queries over 1.5M triangles at 1 / 2 / 3 / 4 / 6
// visits 525 / 457 / 425 / 415 / 438 us (a thread per ray, tests at once: 904 us).
constexpr uint32_t kClosestVisits = 4;
template <bool TWO, class Stack, class RW>
__device__ __forceinline__ bool closest_round(const SceneDev& S, ClosestAreaT<TWO>& w, bool live, float tmin,
                                              Stack stk, Trav& t, RW& r, uint32_t& limits, uint32_t* status) {
    const uint32_t lane = threadIdx.x & 31;
    bool over = false;
    if (live) {
        uint32_t none = 0;
#pragma unroll 1
        for (uint32_t it = 0; it < kClosestVisits; it++) {
            if (trav_node<false, false, TWO>(S, r, tmin, t, stk, none, DeferredStatus{limits})) {
                over = true;
                break;
            }
            if (t.pend_bits) {
                pairs_push<TWO>(w, t);
                if (t.pend_bits) break;
            }
        }
    }
    for (;;) {
        __syncwarp();
        const uint32_t np = min(w.npairs, kPairs);
        if (np == 0) break;
        for (uint32_t b = 0; b < np; b += 32) {
            const uint32_t i = b + lane;
            const uint32_t owner = i < np ? (uint32_t)w.owner[i] : lane;
            const float tmax = __shfl_sync(0xffffffffu, t.tmax, owner);
            f3 o;
            if constexpr (TWO) {
                const int d = (int)owner - (int)lane;
                o = mk(r.p[d], r.p[d + 128], r.p[d + 256]);
            } else {
                o = mk(__shfl_sync(0xffffffffu, r.o.x, owner), __shfl_sync(0xffffffffu, r.o.y, owner),
                       __shfl_sync(0xffffffffu, r.o.z, owner));
            }
            unsigned long long key = ~0ull;
            float tt = 0.f, b1 = 0.f, b2 = 0.f;
            if (i < np) {
                const uint32_t rec = w.rec[i];
                if (rec < S.num_tris) {
                    const float4 ray = w.ray[owner];
                    f3 dir = mk(ray.x, ray.y, ray.z);
                    uint32_t id0 = 0;
                    if constexpr (TWO) {
                        const float4* I = S.inst + (size_t)w.inst[i] * 4;
                        const float4 r0 = __ldg(I), r1 = __ldg(I + 1), r2 = __ldg(I + 2);
                        id0 = __float_as_uint(__ldg(I + 3).y);
                        o = xform_point(r0, r1, r2, o);
                        dir = xform_dir(r0, r1, r2, dir);
                    }
                    const float4* tp = S.tris + (size_t)rec * 3;
                    const float4 v0 = __ldg(tp);
                    if (tri_test(ray_pre(o, dir), v0, __ldg(tp + 1), __ldg(tp + 2), ray.w, tmax, tt, b1, b2)) {
                        key = ((unsigned long long)distance_key(tt) << 32) | (id0 + __float_as_uint(v0.w));
                        atomicMin(&w.key[owner], key);
                    }
                } else {
                    atomicOr(status, HY_STATUS_BAD_INDEX);
                }
            }
            __syncwarp();
            if (key != ~0ull && w.key[owner] == key) w.best[owner] = make_float4(tt, b1, b2, 0.f);
            __syncwarp();
        }
        if (lane == 0) w.npairs = 0;
        const unsigned long long key = w.key[lane];
        if (live && key != ~0ull) {
            const float4 h = w.best[lane];
            t.h = Hit{h.x, (uint32_t)key, h.y, h.z};
            t.tmax = h.x;
        }
        __syncwarp();
        if (__ballot_sync(0xffffffffu, live && t.pend_bits != 0) == 0) break;
        if (live && t.pend_bits) pairs_push<TWO>(w, t);
    }
    return over;
}

// The warp's items of one light (every lane calls it, after all lanes have
// published): sample k of a pixel starts from its first state advanced 2k LCG
// steps (sampleDisk's two draws per sample), its ray from position +
// offset * dir to distance + 1.  On return unocc_count holds each pixel's
// unoccluded samples.
template <bool COUNT, bool TWO, class Stack, class Slots, class RW>
__device__ __forceinline__ void stream_light(const SceneDev& S, const PassParams& P, Slots& sm, uint32_t nrays,
                                             float radius, float offset, Stack stk, Trav& t, RW& r,
                                             LaneStats& ls, uint32_t& nn, uint32_t& nt) {
    const uint32_t lane = threadIdx.x & 31, wb = threadIdx.x & ~31u, warp = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t all = 32u * nrays;
    __syncwarp();
    // the light's items in chunks of Slots::kSort (one chunk unless spp > 16)
    for (uint32_t c0 = 0; c0 < all; c0 += Slots::kSort) {
        const uint32_t cn = min(Slots::kSort, all - c0);
        uint32_t total = cn;
        // ---- the order of the chunk's items: a counting sort of the traced items by
        //      the cell of their disk sample on an 8x8 grid over the disk (cells in
        //      Morton order), so that the lanes' rays at any moment are nearly
        //      parallel rays from the tile's nearby pixels and walk the same nodes
        //      (1080p: 31.96 -> 29.90 ms per shadow launch).  The rays themselves do
        //      not change: only which lane traces which ray, and when ----
        const bool sorted = nrays > 1;
        if (sorted) {
            uint32_t* bk = sm.scratch[warp].sort.bucket;
            uint8_t* keys = sm.scratch[warp].sort.key;
            bk[lane] = 0;
            bk[lane + 32] = 0;
            __syncwarp();
            for (uint32_t j = lane; j < cn; j += 32) {
                uint32_t key = 0xffu;
                const uint32_t q = c0 + j, pi = q / nrays, k = q - pi * nrays;
                if (__float_as_uint(sm.T[wb + pi].w) != kNotTraced) {
                    uint32_t st = lcg_jump_even(__float_as_uint(sm.PL[wb + pi].w), k);
                    const float r1 = rnd(st), r2 = rnd(st);
                    // the disk point in units of the radius (approximate: it only orders the items)
                    float sn, cs;
                    __sincosf(6.2831853f * r2, &sn, &cs);
                    const float rr = r1 > 0.f ? r1 * rsqrtf(r1) : 0.f;
                    const uint32_t ix = min(7u, (uint32_t)fmaxf((rr * cs + 1.0f) * 4.0f, 0.0f));
                    const uint32_t iy = min(7u, (uint32_t)fmaxf((rr * sn + 1.0f) * 4.0f, 0.0f));
                    key = (ix & 1u) | ((iy & 1u) << 1) | ((ix & 2u) << 1) | ((iy & 2u) << 2) | ((ix & 4u) << 2) |
                          ((iy & 4u) << 3);
                    atomicAdd(&bk[key], 1u);
                }
                keys[j] = (uint8_t)key;
            }
            __syncwarp();
            // exclusive scan of the 64 counts, two per lane
            const uint32_t cnt0 = bk[2 * lane], cnt1 = bk[2 * lane + 1], c = cnt0 + cnt1;
            uint32_t incl = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= (uint32_t)d) incl += y;
            }
            total = __shfl_sync(0xffffffffu, incl, 31);  // the chunk's traced items
            __syncwarp();
            bk[2 * lane] = incl - c;
            bk[2 * lane + 1] = incl - c + cnt0;
            __syncwarp();
            for (uint32_t j = lane; j < cn; j += 32) {
                const uint32_t key = keys[j];
                if (key != 0xffu) sm.order[warp][atomicAdd(&bk[key], 1u)] = (uint16_t)j;
            }
        }
        __syncwarp();  // the sort's scratch becomes the walk's
        if (lane == 0) sm.scratch[warp].walk.npairs = 0;
        __syncwarp();
        bool live = false;
        uint32_t cur = 0, head = 0;  // head: the first unclaimed item (the same on every lane)
        for (;;) {
            // ---- idle lanes take the next items, in order ----
            const uint32_t idle = __ballot_sync(0xffffffffu, !live);
            if (head < total) {
                const uint32_t at = head + (uint32_t)__popc(idle & lt_mask);
                head += (uint32_t)__popc(idle);
                if (!live && at < total) {
                    const uint32_t q = c0 + (sorted ? (uint32_t)sm.order[warp][at] : at);
                    const uint32_t pi = q / nrays, k = q - pi * nrays;
                    const float4 tp = sm.T[wb + pi];
                    if (__float_as_uint(tp.w) != kNotTraced) {
                        const float4 pp = sm.pos[wb + pi], pl = sm.PL[wb + pi], bp = sm.B[wb + pi];
                        const f3 pos = mk(pp.x, pp.y, pp.z);
                        const DiskFrame d{mk(tp.x, tp.y, tp.z), mk(bp.x, bp.y, bp.z), mk(pl.x, pl.y, pl.z)};
                        uint32_t st = lcg_jump_even(__float_as_uint(pl.w), k);
                        const f3 dir = sampleDisk(radius, pos, d, st);
                        const float tmax = __fadd_rn(pp.w, 1.0f);
                        sm.scratch[warp].walk.ray[lane] = make_float4(dir.x, dir.y, dir.z, tmax);
                        trav_init(t, world_set(r, add_rn(pos, scale_rn(dir, offset)), dir), tmax);
                        cur = pi;
                        live = true;
                        ls.shadow++;
                    }
                }
            } else if (idle == 0xffffffffu) {
                break;
            }
            const RoundResult res = stream_round<COUNT, TWO>(S, P, sm.scratch[warp].walk, live, stk, t, r, nn, nt);
            if (live && res.over) {
                live = false;
                if (!res.occluded) atomicAdd(unocc_count(sm, wb + cur), 1u);
            }
        }
        __syncwarp();
    }
}

__device__ __forceinline__ float roundtrip(uint32_t fmt, float v) {
    return fmt == HY_ACCUM_U8 ? __fdiv_rn((float)quant8(v), 255.0f) : v;
}

// A lane's pixel in the shadow kernels (set-up, current light, sample state).
struct ShadowLane {
    f3 position, N, L;
    float dist, radius;
    uint32_t pix, seed, light, k, nrays;
    float sf;
    int smode;
    bool in_blur, setup;
};

template <bool ACCUM>
__device__ __forceinline__ void shadow_finalize(const PassParams& P, const ShadowLane& s, size_t plane, float v) {
    const size_t li = (size_t)s.light * plane + s.pix;
    if (!ACCUM) {
        accum_store(P.accum_fmt, P.shadow, li, v);
    } else if (s.in_blur) {
        const float center = roundtrip(P.accum_fmt, v);
        const float old = accum_load(P.accum_fmt, P.hist, li);
        const float a = __fdiv_rn(1.0f, __fadd_rn((float)P.accum_frame, 1.0f));
        accum_store(P.accum_fmt, P.hist, li, __fadd_rn(__fmul_rn(old, __fsub_rn(1.0f, a)), __fmul_rn(center, a)));
    }
}

// a lane's pixel: its G-buffer texel and the RNG state of its first sample
__device__ __forceinline__ void stream_pixel(const SceneDev& S, const PassParams& P, uint32_t x, uint32_t y,
                                             ShadowLane& s) {
    s.pix = y * P.W + x;
    const float4 g0 = fetch_texel(P.plane[0], P.fmt[0], s.pix);
    const float4 g1 = fetch_texel(P.plane[1], P.fmt[1], s.pix);
    s.position = mk(g0.x, g0.y, g0.z);
    s.N = normalize_rn(mk(__fsub_rn(__fmul_rn(g1.x, 2.0f), 1.0f), __fsub_rn(__fmul_rn(g1.y, 2.0f), 1.0f),
                          __fsub_rn(__fmul_rn(g1.z, 2.0f), 1.0f)));
    const int mi = mat_index(g0.w, S.num_mats);
    s.smode = mi >= 0 ? (int)S.mats[mi].smr[0] : 0;
    s.seed = tea(s.pix, P.frame_u);
    s.in_blur = x < P.blur_w && y < P.blur_h;
}

// whether a light's shadow rays are traced for the pixel (shadowRaygen.rgen:43-63)
__device__ __forceinline__ bool light_traced(const HyLight& lt, const ShadowLane& s) {
    const LightGeo lg = light_geo(lt, s.position, s.N);
    return s.smode != 4 && lg.NdotL > 0.f && lg.dist < lg.maxd;
}

// ---------------------------------------------------------------------------------
// Lights light0 .. light1 - 1 of one 8x4 tile of a view, light by light.  ACC: 0 raw shadow images, 1 the
// running mean into the history, 2 either (accum) at run time.  reference:
// REFERENCE RNG (one ray per pixel-light from the pixel's seed, by value).
template <bool COUNT, bool TWO, int ACC, class Stack, class Slots, class RW>
__device__ __forceinline__ void stream_tile(const SceneDev& S, const PassParams& P, uint32_t tile, uint32_t light0,
                                            uint32_t light1, bool reference, bool accum, Slots& sm, Stack stk, Trav& t, RW& r,
                                            ShadowLane& s, LaneStats& ls, uint32_t& nn, uint32_t& nt) {
    const uint32_t lane = threadIdx.x & 31, wb = threadIdx.x & ~31u;
    const size_t plane = (size_t)P.W * P.H;
    const uint32_t spp = P.spp, nrays = reference ? 1u : spp;
    const uint32_t x = (tile % P.tiles_x) * 8 + (lane & 7), y = (tile / P.tiles_x) * 4 + (lane >> 3);
    const bool present = x < P.W && y < P.H;
    auto finalize = [&](float v) {
        if (ACC == 0 || (ACC == 2 && !accum)) shadow_finalize<false>(P, s, plane, v);
        else shadow_finalize<true>(P, s, plane, v);
    };
    uint32_t seed0 = 0, rays_before = 0;
    if (present) {
        stream_pixel(S, P, x, y, s);
        seed0 = s.seed;
#pragma unroll 1
        for (uint32_t l = 0; l < light0; l++) rays_before += light_traced(S.lights[l], s) ? spp : 0u;
    }
    for (uint32_t l = light0; l < light1; l++) {
        // ---- light l for this lane's pixel ----
        bool traced = false;
        s.light = l;
        if (present) {
            const LightGeo lg = light_geo(S.lights[l], s.position, s.N);
            float v = -1.f;
            if (s.smode == 4) v = 1.0f;
            else if (!(lg.NdotL > 0.f)) v = 0.0f;
            else if (!(lg.dist < lg.maxd)) v = 1.0f;
            if (v >= 0.f) finalize(v);
            else traced = true;
            stream_publish(sm, traced, s.position, lg.L, lg.dist,
                           !traced || reference ? seed0 : lcg_jump(seed0, 2u * rays_before));
        } else {
            stream_publish(sm, false, s.position, s.position, 0.f, 0u);
        }
        if (__ballot_sync(0xffffffffu, traced) != 0) {
            // shadowRaygen.rgen:78: origin position + 0.1 dir, tmax distance + 1
            stream_light<COUNT, TWO>(S, P, sm, nrays, S.lights[l].radius, 1e-1f, stk, t, r, ls, nn, nt);
            if (traced) {
                const uint32_t unocc = *unocc_count(sm, wb + lane);
                finalize(reference ? (float)unocc : __fdiv_rn((float)unocc, (float)spp));
            }
        }
        if (traced) rays_before += spp;
        __syncwarp();  // the slots are rewritten by the next light's set-up
    }
}

// The same tile with one ray per pixel and light (REFERENCE RNG, or one sample).
// A light then gives the warp 32 rays at most, and taking the lights one by one
// every lane would wait for each light's longest ray (17.8 of 32 lanes walking on
// the 4K frame with 64 lights).  Here a lane walks its own pixel's rays, light
// after light, without waiting for the others.  The ray's set-up (light geometry,
// disk sample) costs two node visits, so it runs on many lanes at a time: when
// kSetupLanes lanes have nothing to walk, every lane whose slot is free prepares
// its pixel's next traced light, the walking lanes ahead of time.  Lanes stay
// within kLightDrift lights of the last one, so that their rays go the same way.
// Each pixel's lights keep their order, so the RNG states are the sequential loop's.
constexpr uint32_t kSetupLanes = 16, kLightDrift = 8;
template <bool COUNT, bool TWO, int ACC, class Area, class Stack, class RW>
__device__ __forceinline__ void stream_tile_one(const SceneDev& S, const PassParams& P, uint32_t tile,
                                                uint32_t light0, uint32_t light1, bool reference, bool accum, Area& w,
                                                Stack stk, Trav& t, RW& r, ShadowLane& s, LaneStats& ls, uint32_t& nn,
                                                uint32_t& nt) {
    const uint32_t lane = threadIdx.x & 31;
    const size_t plane = (size_t)P.W * P.H;
    const uint32_t x = (tile % P.tiles_x) * 8 + (lane & 7), y = (tile / P.tiles_x) * 4 + (lane >> 3);
    auto finalize = [&](uint32_t l, float v) {
        s.light = l;
        if (ACC == 0 || (ACC == 2 && !accum)) shadow_finalize<false>(P, s, plane, v);
        else shadow_finalize<true>(P, s, plane, v);
    };
    uint32_t next = light1;  // the pixel's next light to set up
    if (x < P.W && y < P.H) {
        stream_pixel(S, P, x, y, s);
        next = light0;
#pragma unroll 1
        for (uint32_t l = 0; l < light0 && !reference; l++)
            if (light_traced(S.lights[l], s)) s.seed = lcg_jump_even(s.seed, 1);
    }
    bool live = false, ready = false;       // walking a ray; a prepared one waits
    uint32_t light = 0, ready_light = 0;    // their lights
    f3 ready_dir = mk(0.f, 0.f, 0.f);       // the prepared ray
    float ready_tmax = 0.f;
    __syncwarp();
    if (lane == 0) w.npairs = 0;
    __syncwarp();
    for (;;) {
        const uint32_t starved = __ballot_sync(0xffffffffu, !live && !ready && next < light1);
        if (starved && ((uint32_t)__popc(starved) >= kSetupLanes || __ballot_sync(0xffffffffu, live || ready) == 0)) {
            const uint32_t last = __reduce_min_sync(0xffffffffu, live ? light : (ready ? ready_light : next));
            while (!ready && next < light1 && next - last <= kLightDrift) {
                const uint32_t l = next++;
                const HyLight& lt = S.lights[l];
                const LightGeo lg = light_geo(lt, s.position, s.N);
                float v = -1.f;
                if (s.smode == 4) v = 1.0f;
                else if (!(lg.NdotL > 0.f)) v = 0.0f;
                else if (!(lg.dist < lg.maxd)) v = 1.0f;
                if (v >= 0.f) {
                    finalize(l, v);
                    continue;
                }
                uint32_t seed = s.seed;
                ready_dir = sampleDisk(lt.radius, s.position, lg.L, seed);
                ready_tmax = __fadd_rn(lg.dist, 1.0f);
                if (!reference) s.seed = seed;  // REFERENCE: sampleDisk takes the pixel's seed by value
                ready = true;
                ready_light = l;
                ls.shadow++;
            }
        }
        if (!live && ready) {
            w.ray[lane] = make_float4(ready_dir.x, ready_dir.y, ready_dir.z, ready_tmax);
            // shadowRaygen.rgen:78: origin position + 0.1 dir, tmax distance + 1
            trav_init(t, world_set(r, add_rn(s.position, scale_rn(ready_dir, 1e-1f)), ready_dir), ready_tmax);
            light = ready_light;
            live = true;
            ready = false;
        }
        if (__ballot_sync(0xffffffffu, live) == 0) {
            if (__ballot_sync(0xffffffffu, next < light1) == 0) break;
            continue;
        }
        const RoundResult res = stream_round<COUNT, TWO>(S, P, w, live, stk, t, r, nn, nt);
        if (live && res.over) {
            live = false;
            finalize(light, res.occluded ? 0.0f : 1.0f);
        }
    }
}

// the view of a batch tile: s_begin holds each view's first tile (ascending)
__device__ __forceinline__ uint32_t view_of_tile(const uint32_t* s_begin, uint32_t nviews, uint32_t tile) {
    uint32_t lo = 0, hi = nviews;  // s_begin[lo] <= tile < s_begin[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (s_begin[mid] <= tile) lo = mid;
        else hi = mid;
    }
    return lo;
}

// the same from the views' own first tiles in the batch's table (global memory,
// L1-cached): the tile-stream batch kernel keeps its shared memory for the slots
__device__ __forceinline__ uint32_t view_of_tile(const PassParams* views, uint32_t nviews, uint32_t tile) {
    uint32_t lo = 0, hi = nviews;  // views[lo].tile_begin <= tile < views[hi].tile_begin
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&views[mid].tile_begin) <= tile) lo = mid;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void finalize_rt(const PassParams& P, bool accum, const ShadowLane& s, size_t plane,
                                            float v) {
    if (accum) shadow_finalize<true>(P, s, plane, v);
    else shadow_finalize<false>(P, s, plane, v);
}

}  // namespace hy
