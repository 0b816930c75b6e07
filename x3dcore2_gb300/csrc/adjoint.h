// Path-replay adjoint (adjoint.cu).
#pragma once

#include "device.cuh"

namespace e8g {

// Accumulates dLoss/d(albedo) (3 per material) and dLoss/d(roughness) into device arrays given
// dLoss/d(image) (3 floats per pixel); path_rgb (optional) receives each path's radiance.
cudaError_t launch_adjoint(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float const *dl_dimage,
                           float inv_spp, unsigned long long *work, float *d_albedo, float *d_rough, float *path_rgb,
                           int num_sms, cudaStream_t st);

// The same over block-local path pools (large renders on the fast trees): its blocks, slots and
// device bytes (slots 0: not for this scene and render), and the launch with that many bytes.
struct AdjointPool {
    int grid = 0;
    uint32_t slots = 0;
    size_t bytes = 0;
};
AdjointPool adjoint_pool(DevScene const &S, RenderArgs const &A, int num_sms);
cudaError_t launch_adjoint_pool(DevScene const &S, RenderArgs const &A, FirstHit const *fh, float const *dl_dimage,
                                float inv_spp, unsigned long long *work, float *d_albedo, float *d_rough,
                                AdjointPool const &p, void *pool, cudaStream_t st);

} // namespace e8g
