// Tile-stream shadow kernels over two-level structures (hy_stream_kernel.cuh):
// 8 resident blocks (64 registers; the 4K instanced frame 290 ms against 309 at
// 5 blocks and 296 at 6).
#include "hy_stream_kernel.cuh"

namespace hy {
template <bool ACCUM, bool ONE>
static void* two_kernel(bool count) {
    return count ? (void*)k_shadow_stream<true, ACCUM, 8, true, false, ONE>
                 : (void*)k_shadow_stream<false, ACCUM, 8, true, false, ONE>;
}
void* stream_kernel_two(bool accum, bool count, bool one) {
    if (accum) return one ? two_kernel<true, true>(count) : two_kernel<true, false>(count);
    return one ? two_kernel<false, true>(count) : two_kernel<false, false>(count);
}
}  // namespace hy
