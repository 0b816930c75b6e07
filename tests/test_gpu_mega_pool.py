"""The pooled megakernel against the one-thread-per-path kernel: the same paths from the same
streams, so images and per-path lists agree up to the order of a pixel's sum."""
import numpy as np
import pytest

from x3dcore2_gb300 import abi
from x3dcore2_gb300 import scene as S
from x3dcore2_gb300.core import default_params

pytestmark = pytest.mark.gpu

# contributions are not negative and a pixel adds at most 16 samples of about 10: 160 roundings of 2^-24
RTOL = 1e-5


def plain(p):
    q = abi.RenderParams.from_buffer_copy(p)
    q.integrator = abi.INTEGRATOR_PLAIN
    return q


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE])
@pytest.mark.parametrize("mode,depth", [(abi.MODE_MIS, 6), (abi.MODE_REF_LT1, 0), (abi.MODE_REF_UNI, 0)])
@pytest.mark.parametrize("kind,w,h,spp", [("soup", 331, 211, 8), ("ico", 1023, 517, 1), ("cornell", 257, 255, 16)])
def test_image_is_the_plain_kernels(ctx, kind, w, h, spp, mode, depth, layout):
    """Odd sizes, from the fewest paths the pools take (2^19) to several fills of every slot; a tree
    of a few nodes (no ray outlives its phase) and deep ones."""
    sc = {"soup": lambda: S.soup(20_000, seed=3, width=w, height=h), "cornell": lambda: S.cornell(w, h),
          "ico": lambda: S.displaced_icosphere(level=6, seed=2, num_materials=64, width=w, height=h)}[kind]()
    ctx.upload(sc, layout=layout)
    p = default_params(mode, w, h, spp, seed=11, max_depth=depth, rr_start=3)
    got, want = ctx.render(p), ctx.render(plain(p))
    assert want[..., :3].sum() > 0
    np.testing.assert_allclose(got, want, rtol=RTOL, atol=1e-12)


@pytest.mark.parametrize("mode", [abi.MODE_MIS, abi.MODE_REF_LT1])
def test_path_list_and_firefly_images(ctx, mode):
    """Per-path output: a list with repeats and paths that end at once, and the clamp's sample images."""
    w, h = 300, 250
    sc = S.displaced_icosphere(level=5, seed=2, num_materials=16, width=w, height=h)
    ctx.upload(sc)
    p = default_params(mode, w, h, 8, seed=5, max_depth=6, rr_start=3)
    r = np.random.default_rng(1)
    px = r.integers(0, w * h, 600_001).astype(np.uint32)
    smp = r.integers(0, 8, len(px)).astype(np.uint32)
    np.testing.assert_allclose(ctx.render_paths(p, px, smp), ctx.render_paths(plain(p), px, smp), rtol=RTOL, atol=1e-12)
    p.firefly = 1
    np.testing.assert_allclose(ctx.render(p), ctx.render(plain(p)), rtol=RTOL, atol=1e-12)


def test_memory_limit_keeps_the_kernel_without_pools(lib):
    from x3dcore2_gb300.core import Context
    w, h = 1023, 517
    sc = S.displaced_icosphere(level=5, seed=2, num_materials=16, width=w, height=h)
    p = default_params(abi.MODE_MIS, w, h, 1, seed=5, max_depth=6, rr_start=3)
    with Context(0) as c:
        c.upload(sc)
        want = c.render(p)
        pooled = c.memory_used()
    with Context(0) as c:
        c.set_memory_limit(1 << 30)
        c.upload(sc)
        np.testing.assert_allclose(c.render(p), want, rtol=RTOL, atol=1e-12)
        assert c.memory_used() < pooled


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE])
@pytest.mark.parametrize("kind,depth,rr", [("cornell", 6, 3), ("cornell", 20, 20), ("ico", 9, 9)])
def test_backward_is_the_one_path_per_lane_kernels(lib, kind, depth, rr, layout):
    """Gradients of the pooled backward against those of the kernel a context with a memory limit
    keeps: paths within the scatter list, far beyond it (a second walk), and one vertex beyond.
    The image gradient is positive, so albedo terms do not cancel: a block sums at most about 10,000
    of them per material, in any order, within 10,000 x 2^-24 of their sum."""
    from x3dcore2_gb300.core import Context
    w, h = 257, 255
    sc = (S.cornell(w, h) if kind == "cornell"
          else S.displaced_icosphere(level=5, seed=2, num_materials=16, width=w, height=h))
    p = default_params(abi.MODE_MIS, w, h, 8, seed=5, max_depth=depth, rr_start=rr)
    dl = np.random.default_rng(2).uniform(0.5, 1.0, (h, w, 3)).astype(np.float32)
    got = []
    for limit in (0, 4 << 30):
        with Context(0) as c:
            c.set_memory_limit(limit)
            c.upload(sc, layout=layout)
            c.forward(p)
            got.append(c.backward(dl))
    (da, dr), (wa, wr) = got
    assert np.abs(wa).sum() > 0
    np.testing.assert_allclose(da, wa, rtol=1e-3, atol=1e-6 * np.abs(wa).max())
    assert np.linalg.norm(dr - wr) <= 1e-3 * max(np.linalg.norm(wr), 1e-12)
