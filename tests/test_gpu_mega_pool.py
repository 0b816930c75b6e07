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


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE])
@pytest.mark.parametrize("mode,depth", [(abi.MODE_MIS, 6), (abi.MODE_REF_LT1, 0), (abi.MODE_REF_UNI, 0)])
@pytest.mark.parametrize("kind", ["cornell", "soup"])
def test_image_adds_a_path_once(ctx, kind, mode, depth, layout):
    """A pixel of two samples is the sum of its two paths' radiances rounded once, bit for bit, however many
    contributions each has (halving is exact)."""
    w, h = 1027, 1023
    sc = S.cornell(w, h) if kind == "cornell" else S.soup(20_000, seed=3, width=w, height=h)
    ctx.upload(sc, layout=layout)
    p = default_params(mode, w, h, 2, seed=11, max_depth=depth, rr_start=3)
    px = np.tile(np.arange(w * h, dtype=np.uint32), 2)
    paths = ctx.render_paths(plain(p), px, np.repeat(np.arange(2, dtype=np.uint32), w * h))
    want = paths.astype(np.float64).reshape(2, h, w, 3).sum(axis=0).astype(np.float32) * np.float32(0.5)
    assert want.sum() > 0
    assert np.array_equal(ctx.render(p)[..., :3], want)


@pytest.mark.parametrize("mode,depth", [(abi.MODE_MIS, 6), (abi.MODE_REF_LT1, 0), (abi.MODE_REF_UNI, 0)])
@pytest.mark.parametrize("kind", ["cornell", "soup"])
def test_a_path_is_the_same_in_a_short_and_a_long_list(ctx, kind, mode, depth):
    """Long lists run over the pools, short ones a path per lane: the same bits for every path, those that start
    on a light (here one that reflects) among them."""
    w, h = 1024, 512
    sc = S.cornell(w, h) if kind == "cornell" else S.soup(20_000, seed=3, width=w, height=h)
    for light in sc.lights[:sc.num_lights]:
        sc.mesh_mat[light.mesh] = sc.mesh_mat[0]
    ctx.upload(sc)
    p = default_params(mode, w, h, 4, seed=11, max_depth=depth, rr_start=3)
    px, smp = np.tile(np.arange(w * h, dtype=np.uint32), 4), np.repeat(np.arange(4, dtype=np.uint32), w * h)
    long = ctx.render_paths(p, px, smp)
    for k in range(3):
        at = slice(k * 300_007, (k + 1) * 300_007)
        short = ctx.render_paths(p, px[at], smp[at])
        assert short.sum() > 0
        assert np.array_equal(long[at].view(np.uint32), short.view(np.uint32))


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE])
@pytest.mark.parametrize("mode,depth", [(abi.MODE_MIS, 6), (abi.MODE_REF_LT1, 0)])
@pytest.mark.parametrize("spp,slots", [(1, 128), (16, 640), (32, 1024)])
def test_smaller_and_larger_pools(lib, spp, slots, mode, depth, layout):
    """Renders for the fewest slots a block, for 640 and for all 1,024 (128 bytes each, seven blocks an SM), at an
    odd size: a pixel is a sum of at most 32 equal terms in any order."""
    import torch

    from x3dcore2_gb300.core import Context
    w, h = 1023, 577
    p = default_params(mode, w, h, spp, seed=11, max_depth=depth, rr_start=3)
    with Context(0) as c:
        c.set_memory_limit(64 << 30)
        c.upload(S.soup(20_000, seed=3, width=w, height=h), layout=layout)
        c.render(p)
        lanes = c.memory_used()
        c.set_memory_limit(0)
        got = c.render(p)
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert sms != 152 or c.memory_used() - lanes == sms * 7 * slots * 128
        np.testing.assert_allclose(got, c.render(plain(p)), rtol=RTOL, atol=1e-12)
        p.firefly = 1  # sample images of single paths, which are the same bits, and the same clamp
        np.testing.assert_allclose(c.render(p), c.render(plain(p)), rtol=RTOL, atol=1e-12)


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE])
def test_backward_with_its_most_slots(lib, layout):
    """512 slots a block (twice a small render's) against the one-path-per-lane kernel; tolerance as above."""
    from x3dcore2_gb300.core import Context
    grew = []
    for w, h, spp in ((257, 255, 16), (513, 511, 32)):
        p = default_params(abi.MODE_MIS, w, h, spp, seed=5, max_depth=6, rr_start=3)
        dl = np.random.default_rng(2).uniform(0.5, 1.0, (h, w, 3)).astype(np.float32)
        with Context(0) as c:
            c.set_memory_limit(64 << 30)
            c.upload(S.displaced_icosphere(level=5, seed=2, num_materials=16, width=w, height=h), layout=layout)
            c.forward(p)
            wa, wr = c.backward(dl)
            lanes = c.memory_used()
            c.set_memory_limit(0)
            c.forward(p)
            da, dr = c.backward(dl)
            grew.append(c.memory_used() - lanes)
        assert np.abs(wa).sum() > 0
        np.testing.assert_allclose(da, wa, rtol=1e-3, atol=1e-6 * np.abs(wa).max())
        assert np.linalg.norm(dr - wr) <= 1e-3 * max(np.linalg.norm(wr), 1e-12)
    assert grew[1] == 2 * grew[0] > 0


@pytest.mark.parametrize("what", ["render", "wavefront", "backward"])
def test_a_limit_set_later_takes_back_the_pools_room(lib, what):
    """What fits a limit does not depend on when it was set: path pools and slot lists of an earlier call give
    way to the buffers of a later one."""
    from x3dcore2_gb300.core import Context
    w, h = 1027, 1023
    sc = S.displaced_icosphere(level=5, seed=2, num_materials=16, width=w, height=h)
    p = default_params(abi.MODE_MIS, w, h, 2, seed=5, max_depth=6, rr_start=3)
    if what == "wavefront":
        p.integrator = abi.INTEGRATOR_WAVEFRONT
    dl = np.ones((h, w, 3), np.float32)
    r = np.random.default_rng(1)
    rays = np.concatenate([r.uniform(-2, 2, (1_500_000, 3)), r.normal(0, 1, (1_500_000, 3))], axis=1).astype(np.float32)

    def call(c):
        if what != "backward":
            return c.render(p)
        c.forward(p)
        return c.backward(dl)[0]

    with Context(0) as c:
        c.set_memory_limit(64 << 30)
        c.upload(sc)
        want = call(c)
        hits = c.trace_closest(rays)
        need = c.memory_used()
    with Context(0) as c:
        c.upload(sc)
        call(c)
        more = c.memory_used()
        c.set_memory_limit(need)
        got = c.trace_closest(rays)
        assert np.array_equal(got["t"], hits["t"]) and more + 44 * len(rays) > need >= c.memory_used()
        np.testing.assert_allclose(call(c), want, rtol=1e-3, atol=1e-6 * np.abs(want).max())
