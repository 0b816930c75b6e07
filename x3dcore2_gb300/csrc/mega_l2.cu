// Megakernel instantiations for the eight-wide tree (layout 2).
#include "mega_pool.cuh"

namespace e8g {

void launch_mega_l2(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum, float *path_rgb,
                    unsigned long long *work, unsigned long long *counters, int grid, bool plain, cudaStream_t st) {
    launch_layout<2>(S, A, fh, accum, path_rgb, work, counters, grid, plain, st);
}

void launch_mega_pool_l2(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum, float *path_rgb,
                         unsigned long long *work, float4 *pool, int num_sms, cudaStream_t st) {
    launch_pool<2>(S, A, fh, accum, path_rgb, work, pool, num_sms, st);
}

} // namespace e8g
