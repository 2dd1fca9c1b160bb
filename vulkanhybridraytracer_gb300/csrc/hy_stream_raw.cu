// Tile-stream shadow kernels writing raw per-light images (hy_stream_kernel.cuh).
#include "hy_stream_kernel.cuh"

namespace hy {
void* stream_kernel_raw(bool count, int minb, bool short_stack, bool one) {
    return one ? stream_kernel_flat<false, true>(count, minb, short_stack)
               : stream_kernel_flat<false, false>(count, minb, short_stack);
}
}  // namespace hy
