"""The wavefront's bounces after the last path was taken visit a list of the occupied slots: renders
that fit the slots exactly, overflow them by a few paths, hold one tile, or run without lists (memory
limit) are the megakernel's image; so is the split bidirectional form the one-thread form's."""
import numpy as np
import pytest

from x3dcore2_gb300 import abi
from x3dcore2_gb300 import scene as S
from x3dcore2_gb300.core import default_params

pytestmark = pytest.mark.gpu

# width, height, samples, slots, bounces per graph: 8x4-pixel tiles pad each sample to whole warps
SIZES = [(32, 32, 1, 1024, 1), (37, 29, 1, 1024, 3), (2, 2, 1, 1024, 2), (64, 64, 3, 1024, 5), (64, 64, 3, 16384, 2),
         # lists are kept from 155,649 slots on (1,024 for each of 152 SMs)
         (500, 400, 1, 1 << 18, 2), (500, 400, 2, 160000, 3), (512, 304, 1, 155648, 1), (512, 304, 2, 155649, 1)]


def _close(a, b):
    ok = np.all(np.abs(a - b) <= np.maximum(1e-4 * np.abs(b), 1e-6), axis=-1)
    return ok.mean()


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE])
@pytest.mark.parametrize("shade", [0, 6])
@pytest.mark.parametrize("w,h,spp,slots,bounces", SIZES)
def test_wavefront_with_lists_equals_megakernel(ctx, w, h, spp, slots, bounces, shade, layout):
    ctx.upload(S.displaced_icosphere(level=3, seed=5, num_materials=8, width=w, height=h), layout=layout)
    p = default_params(abi.MODE_MIS, w, h, spp, seed=11, max_depth=8, rr_start=3)
    ref = ctx.render(p)
    p.integrator = abi.INTEGRATOR_WAVEFRONT
    assert ctx.lib.e8g_wavefront_set(ctx.h, slots, bounces, 8) == 0
    assert ctx.lib.e8g_wavefront_set_shade(ctx.h, shade) == 0
    try:
        img = ctx.render(p)
        ctx.set_memory_limit(ctx.memory_used() + (64 << 20))
        plain = ctx.render(p)
    finally:
        ctx.set_memory_limit(0)
        ctx.lib.e8g_wavefront_set(ctx.h, 1 << 21, 4, 16)
        ctx.lib.e8g_wavefront_set_shade(ctx.h, 0)
    assert _close(img, ref) >= 0.999
    assert _close(plain, ref) >= 0.999


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE])
@pytest.mark.parametrize("w,h,spp", [(2, 2, 1), (37, 29, 1), (64, 64, 3), (512, 304, 1), (500, 400, 2)])
def test_split_bdpt_with_lists_equals_the_one_thread_form(ctx, w, h, spp, layout):
    ctx.upload(S.cornell(w, h), layout=layout)
    p = default_params(abi.MODE_BDPT_POWER, w, h, spp, seed=6, bdpt_max_len=8)
    ref = ctx.render(p)
    p.integrator = abi.INTEGRATOR_WAVEFRONT
    img = ctx.render(p)
    assert _close(img, ref) >= 0.999
