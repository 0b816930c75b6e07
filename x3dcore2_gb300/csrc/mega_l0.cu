// Megakernel instantiations for SAH child pairs (layout 0).
#include "mega_pool.cuh"

namespace e8g {

void launch_mega_l0(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum, float *path_rgb,
                    unsigned long long *work, unsigned long long *counters, int grid, bool plain, cudaStream_t st) {
    launch_layout<0>(S, A, fh, accum, path_rgb, work, counters, grid, plain, st);
}

int megakernel_blocks_per_sm() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_mega<RngPhilox, false, 0>, kBlock, 0);
    return n > 0 ? n : 1;
}

void launch_mega_pool_l0(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum, float *path_rgb,
                         unsigned long long *work, float4 *pool, int num_sms, cudaStream_t st) {
    launch_pool<0>(S, A, fh, accum, path_rgb, work, pool, num_sms, st);
}

size_t mega_pool_bytes(RenderArgs const &A, int num_sms) {
    return static_cast<size_t>(num_sms) * kPoolBlocks * pool_slots(A, num_sms) * kPoolArrays * sizeof(float4);
}

} // namespace e8g
