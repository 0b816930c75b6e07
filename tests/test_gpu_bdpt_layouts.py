"""The bidirectional kernels compiled per tree, on a scene that is half sky: per-path radiance
against the oracle fed the same streams, and nothing from paths whose camera ray leaves the scene
(their light subpaths are not walked)."""
import numpy as np
import pytest

import oracle_bind as ob
from test_gpu_paths import match_fraction
from x3dcore2_gb300 import abi
from x3dcore2_gb300 import scene as S
from x3dcore2_gb300.core import default_params

pytestmark = pytest.mark.gpu
W, H = 64, 36


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE, abi.BVH_REFERENCE])
@pytest.mark.parametrize("mode,integ,max_len", [(abi.MODE_REF_BDPT, abi.INTEGRATOR_MEGAKERNEL, 8),
                                                (abi.MODE_REF_BDPT, abi.INTEGRATOR_MEGAKERNEL, 1),
                                                (abi.MODE_BDPT_POWER, abi.INTEGRATOR_MEGAKERNEL, 6),
                                                (abi.MODE_BDPT_POWER, abi.INTEGRATOR_WAVEFRONT, 6)])
def test_paths_and_sky(ctx, mode, integ, max_len, layout):
    sc = S.displaced_icosphere(level=3, seed=2, num_materials=16, width=W, height=H)
    ctx.upload(sc, layout=layout)
    osc = ob.OracleScene(sc)
    n = 3001
    px = np.random.default_rng(max_len).integers(0, W * H, n).astype(np.uint32)
    smp = np.arange(n, dtype=np.uint32)
    p = default_params(mode, W, H, 1, seed=9, bdpt_max_len=max_len)
    p.integrator = integ
    got = ctx.render_paths(p, px, smp)
    pol = ob.OPolicy(0, 2, 0.5, max_len)
    if p.rng == abi.RNG_MINSTD:
        seeds = np.array([ob.oracle().o_path_seed(9, int(a), int(b)) for a, b in zip(px, smp)], np.uint32)
        ref = osc.render_paths(mode, W, H, px, seeds, policy=pol)
    else:
        ref = osc.render_paths(mode, W, H, px, smp, policy=pol, rng=abi.RNG_PHILOX, seed=9)
    assert match_fraction(got, ref) >= 0.995
    sky = osc.trace_closest(osc.camera_rays(W, H))["mesh"][px] < 0
    assert 0.1 < sky.mean() < 0.9
    assert np.all(got[sky] == 0)
