"""Paths are numbered tile by tile, a tile's samples in a row: whatever the size of the image and the
number of samples, every sample of every pixel is traced once."""
import numpy as np
import pytest

from x3dcore2_gb300 import abi
from x3dcore2_gb300 import scene as S
from x3dcore2_gb300.core import default_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", [abi.INTEGRATOR_MEGAKERNEL, abi.INTEGRATOR_WAVEFRONT])
@pytest.mark.parametrize("w,h,spp", [(2, 2, 1), (9, 5, 7), (8, 4, 33), (257, 131, 17)])
def test_image_is_the_mean_of_its_paths(ctx, w, h, spp, integrator):
    ctx.upload(S.cornell(w, h))
    p = default_params(abi.MODE_MIS, w, h, spp, seed=3, max_depth=5, rr_start=3)
    p.integrator = integrator
    img = ctx.render(p)[..., :3]
    px = np.tile(np.arange(w * h, dtype=np.uint32), spp)
    smp = np.repeat(np.arange(spp, dtype=np.uint32), w * h)
    paths = ctx.render_paths(p, px, smp).reshape(spp, h, w, 3)
    mean = paths.mean(axis=0, dtype=np.float64)
    # float sums of spp terms in any order: spp rounding errors of the running sum
    assert np.all(np.abs(img - mean) <= spp * 2.0**-23 * np.abs(paths).mean(axis=0, dtype=np.float64) + 1e-12)
