// Megakernel dispatch and the many-scene megakernel (e8g_batch_render); the per-layout
// integrator kernels are instantiated in mega_l0.cu (SAH pairs), mega_l1.cu (reference tree)
// and mega_l2.cu (eight-wide).
#include "mega.cuh"

namespace e8g {

// rng_kinds: bit E8G_RNG_MINSTD / bit E8G_RNG_PHILOX set when some scene of the batch uses it.
void launch_megakernel_batch(BatchDev const &B, FirstHit const *fh_all, float4 *accum_all, unsigned long long *work,
                             uint32_t rng_kinds, int grid, cudaStream_t st) {
    if (rng_kinds == (1u << E8G_RNG_PHILOX))
        k_mega_batch<RngPhilox><<<grid, kBlock, 0, st>>>(B, fh_all, accum_all, work);
    else if (rng_kinds == (1u << E8G_RNG_MINSTD))
        k_mega_batch<RngMinstd><<<grid, kBlock, 0, st>>>(B, fh_all, accum_all, work);
    else
        k_mega_batch<RngAny><<<grid, kBlock, 0, st>>>(B, fh_all, accum_all, work);
}

int megakernel_batch_blocks_per_sm(uint32_t rng_kinds) {
    int n = 0;
    if (rng_kinds == (1u << E8G_RNG_PHILOX))
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_mega_batch<RngPhilox>, kBlock, 0);
    else if (rng_kinds == (1u << E8G_RNG_MINSTD))
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_mega_batch<RngMinstd>, kBlock, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_mega_batch<RngAny>, kBlock, 0);
    return n > 0 ? n : 1;
}


void launch_megakernel(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum, float *path_rgb,
                       unsigned long long *work, unsigned long long *counters, int grid, cudaStream_t st, bool plain) {
    if (S.layout == 1)
        launch_mega_l1(S, A, fh, accum, path_rgb, work, counters, grid, plain, st);
    else if (S.layout == 2)
        launch_mega_l2(S, A, fh, accum, path_rgb, work, counters, grid, plain, st);
    else if (S.layout == 3)
        launch_mega_l3(S, A, fh, accum, path_rgb, work, counters, grid, plain, st);
    else
        launch_mega_l0(S, A, fh, accum, path_rgb, work, counters, grid, plain, st);
}

// The estimators with a random walk on their default streams, on the two fast trees, from 2^19 paths
// on (four per lane of the pools); below that the pools hardly refill and k_mega is as fast or faster.
// Where the two break even depends on how long paths are. One-sample frames of 541,000 / 1.07M / 2.07M paths, k_mega
// against pools, ms, on the pairs: a 50,000-triangle soup in a closed room MIS 1.51 / 2.53 / 4.55 against
// 1.22 / 1.81 / 2.81, lt1 1.34 / 2.31 / 4.13 against 1.09 / 1.49 / 2.31; the 1.3M-triangle icosphere, an open
// scene whose paths have one or two rays, MIS 0.67 / 1.06 / 1.90 against 0.81 / 1.13 / 1.71, lt1 0.59 / 0.97 /
// 1.79 against 0.66 / 0.98 / 1.44. On the eight-wide tree the pools win in both (541,000 paths: 1.76 against
// 1.10, 0.70 against 0.60). The unidirectional estimator has no shadow rays to fill lanes with and starts
// later on the pairs (541,000 / 1.07M / 1.44M paths: soup 0.81 / 1.42 / 1.87 against 0.81 / 1.12 / 1.33, icosphere
// 0.39 / 0.56 / 0.75 against 0.51 / 0.67 / 0.79).
bool mega_pool_takes(DevScene const &S, RenderArgs const &A) {
    const uint64_t least = S.layout == 0 && A.mode == E8G_MODE_REF_UNI ? 5u << 18 : 1u << 19;
    return (S.layout == 0 || S.layout == 2) && A.total_paths >= least &&
           ((A.mode == E8G_MODE_MIS && A.rng == E8G_RNG_PHILOX) ||
            ((A.mode == E8G_MODE_REF_LT1 || A.mode == E8G_MODE_REF_UNI) && A.rng == E8G_RNG_MINSTD));
}

void launch_mega_pool(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float4 *accum, float *path_rgb,
                      unsigned long long *work, void *pool, int num_sms, cudaStream_t st) {
    if (S.layout == 0)
        launch_mega_pool_l0(S, A, fh, accum, path_rgb, work, static_cast<float4 *>(pool), num_sms, st);
    else
        launch_mega_pool_l2(S, A, fh, accum, path_rgb, work, static_cast<float4 *>(pool), num_sms, st);
}

} // namespace e8g
