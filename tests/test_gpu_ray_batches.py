"""Ray batches at the edges of the trace kernels' warp chunks, and trees at the edges of their
stacks: a single leaf, and chains deeper than the part of the stack kept in shared memory."""
import numpy as np
import pytest

import oracle_bind as ob
from test_gpu_trace import compare_hits, random_rays
from x3dcore2_gb300 import abi
from x3dcore2_gb300 import scene as S

pytestmark = pytest.mark.gpu
LAYOUTS = [abi.BVH_SAH, abi.BVH_WIDE]


def check(ctx, sc, layout, rays):
    ctx.upload(sc, layout=layout)
    osc = ob.OracleScene(sc)
    o = osc.trace_closest(rays)
    compare_hits(ctx.trace_closest(rays), o["mesh"], o["tri"], o["t"])
    tmin = np.full(len(rays), 1e-4, np.float32)
    tmax = np.random.default_rng(len(rays)).uniform(1e-3, 2.5, len(rays)).astype(np.float32)
    assert np.mean(ctx.trace_any(rays, tmin, tmax) == osc.trace_any(rays, tmin, tmax)) >= 0.9999


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("n", [1, 31, 33, 4097, 155_649, 400_003])
def test_batch_sizes(ctx, layout, n):
    """One ray, part of a warp, one ray per lane, and chunks of 64 and 96 rays per warp with a ragged last one."""
    check(ctx, S.soup(3000, seed=7, width=64, height=64), layout, random_rays(max(n, 64), -1.0, 1.0, seed=n)[-n:])


def mesh_scene(tris):
    """Triangles (T, 3, 3) as one mesh, with a small light above them."""
    def mesh(t):
        t = np.asarray(t, np.float32)
        n = np.cross(t[:, 1] - t[:, 0], t[:, 2] - t[:, 0])
        n /= np.linalg.norm(n, axis=1, keepdims=True)
        return S.Mesh(t.reshape(-1, 3), np.repeat(n, 3, axis=0), np.arange(3 * len(t)).reshape(-1, 3))
    m = S.material(abi.MAT_OREN_NAYAR, albedo=(0.5, 0.5, 0.5))
    light = abi.Light()
    light.mesh = 1
    light.radiance[:] = [1.0, 1.0, 1.0]
    lamp = mesh([[[0.0, 0.0, 5.0], [0.0, 0.1, 5.0], [0.1, 0.0, 5.0]]])
    cam = S.soup(10, seed=1, width=32, height=32).camera
    return S.from_meshes([mesh(tris), lamp], [0, 0], [m], [light], cam)


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("count", [1, 6])
def test_tree_of_few_triangles(ctx, layout, count):
    r = np.random.default_rng(count)
    check(ctx, mesh_scene(r.uniform(-1, 1, (count, 3, 3))), layout, random_rays(2000, -1.0, 1.0, seed=count))


@pytest.mark.parametrize("layout", LAYOUTS)
def test_stack_beyond_its_shared_part(ctx, layout):
    """Sheets whose spacing doubles along x: the tree is a chain, and a ray along it that hits none
    of the nearer sheets keeps a far child per level."""
    tris = []
    for k in range(20):
        x = 2.0 ** (k - 18)
        for j in range(12):
            y = -1.0 + j / 6.0
            tris.append([[x, y, -1.0], [x, y + 0.16, -1.0], [x, y, 1.0]])
    r = np.random.default_rng(3)
    n = 4000
    o = np.stack([np.full(n, -1.0), r.uniform(-1, 1, n), r.uniform(-1, 1, n)], axis=1)
    d = np.stack([np.ones(n), r.normal(0, 0.05, n), r.normal(0, 0.05, n)], axis=1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    back = np.stack([o[:, 0] + 4.0, o[:, 1], o[:, 2]], axis=1)
    rays = np.concatenate([ob.rays_array(o.astype(np.float32), d.astype(np.float32)),
                           ob.rays_array(back.astype(np.float32), -d.astype(np.float32))])
    sc = mesh_scene(tris)
    check(ctx, sc, layout, rays)
    if layout == abi.BVH_SAH:
        assert ctx.bvh_stats()["max_depth"] > 9


@pytest.mark.parametrize("layout", [abi.BVH_SAH, abi.BVH_WIDE, abi.BVH_REFERENCE, abi.BVH_LINEAR])
@pytest.mark.parametrize("n", [1, 33, 5000])
def test_hit_records_equal_hit_arrays(ctx, layout, n):
    """e8g_trace_closest's records and e8g_trace_closest_arrays (which Context.trace_closest uses) are
    the same hits, misses among them; the arrays are contiguous."""
    ctx.upload(S.displaced_icosphere(level=3, seed=2, num_materials=16, width=64, height=36), layout=layout)
    rays = random_rays(max(n, 64), -2.0, 2.0, seed=n)[-n:]
    g = ctx.trace_closest(rays)
    raw = np.zeros((n, 5), np.float32)
    ctx._check(ctx.lib.e8g_trace_closest(ctx.h, rays.ctypes.data, n, raw.ctypes.data), "e8g_trace_closest")
    assert all(g[k].flags["C_CONTIGUOUS"] and g[k].flags["WRITEABLE"] for k in g)
    assert np.array_equal(g["t"], raw[:, 0]) and np.array_equal(g["b"], raw[:, 3:])
    assert np.array_equal(g["mesh"], raw[:, 1].view(np.int32)) and np.array_equal(g["tri"], raw[:, 2].view(np.int32))
    assert n == 1 or (g["mesh"] < 0).any()


@pytest.mark.parametrize("n", [11_915, 11_916, 15_887, 15_888])
def test_batches_around_the_pinned_limit(ctx, n):
    """512 KiB hold the rays and hits of 11,915 closest-hit queries and of 15,887 any-hit ones: beyond
    that the batch goes through device memory. Both give what the first rays alone give."""
    ctx.upload(S.soup(500, seed=3, width=64, height=64), layout=abi.BVH_SAH)
    rays = random_rays(n, -1.0, 1.0, seed=5)
    tmin, tmax = np.full(n, 1e-4, np.float32), np.linspace(0.01, 2.0, n, dtype=np.float32)
    hit, occ = ctx.trace_closest(rays), ctx.trace_any(rays, tmin, tmax)
    for lo, hi in ((0, 4000), (n - 4000, n)):
        part = ctx.trace_closest(rays[lo:hi])
        assert all(np.array_equal(hit[k][lo:hi], part[k]) for k in part)
        assert np.array_equal(occ[lo:hi], ctx.trace_any(rays[lo:hi], tmin[lo:hi], tmax[lo:hi]))


def edge_rays(sc, n, seed):
    """Rays of which half are aimed at vertices and at points of edges, where two triangles lie at the
    same distance, and some along an axis."""
    r = np.random.default_rng(seed)
    tri = sc.world_triangles().astype(np.float64)
    t = tri[r.integers(0, len(tri), n)]
    w = r.uniform(0, 1, (n, 1))
    aim = np.where(r.random((n, 1)) < 0.3, t[:, 0], t[:, 0] * w + t[:, 1] * (1 - w))
    aim = np.where(r.random((n, 1)) < 0.5, aim, r.uniform(-1, 1, (n, 3)))
    o = r.uniform(-1, 1, (n, 3))
    d = aim - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    d[: n // 16] = np.eye(3)[r.integers(0, 3, n // 16)]
    return np.concatenate([o, d], axis=1).astype(np.float32)


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("scene", ["soup", "ico", "cornell", "doubled", "one"])
def test_warp_per_ray_equals_lane_per_ray(ctx, layout, scene):
    """Small batches give each ray a warp, large ones a lane: the same rays have the same hits in both,
    bit for bit, also where two triangles lie at one distance."""
    r = np.random.default_rng(1)
    sc = {"soup": lambda: S.soup(3000, seed=2, width=64, height=64),
          "ico": lambda: S.displaced_icosphere(level=4, seed=3, num_materials=8, width=64, height=64),
          "cornell": lambda: S.cornell(64, 64),
          "doubled": lambda: mesh_scene(np.repeat(r.uniform(-1, 1, (40, 3, 3)), 9, axis=0)),
          "one": lambda: mesh_scene(r.uniform(-1, 1, (1, 3, 3)))}[scene]()
    ctx.upload(sc, layout=layout)
    n, copies = 3001, 30  # more than four rays for every warp the GPU holds in one call of all copies
    rays = edge_rays(sc, n, seed=4)
    tmin = r.choice(np.array([1e-4, 0.0, -1.0, 0.5], np.float32), n)
    tmax = r.choice(np.array([0.25, 1.0, 1e-5, np.inf], np.float32), n)
    many = ctx.trace_closest(np.tile(rays, (copies, 1)))
    occ = ctx.trace_any(np.tile(rays, (copies, 1)), np.tile(tmin, copies), np.tile(tmax, copies))
    for lo, hi in ((0, n), (0, 1), (5, 38)):
        few = ctx.trace_closest(rays[lo:hi])
        for k in few:
            assert np.array_equal(few[k].view(np.uint32), np.ascontiguousarray(many[k][lo:hi]).view(np.uint32)), k
        assert np.array_equal(ctx.trace_any(rays[lo:hi], tmin[lo:hi], tmax[lo:hi]), occ[lo:hi])


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("far", [3e8, 4e8, 1e12, 1e18])
def test_axis_parallel_rays_far_from_the_origin(ctx, layout, far):
    """Sheets across the z axis around x = far, and rays along it whose other components are zero or tiny:
    the planes' distances leave the float range there. The linear layout, which tests every triangle,
    says what is hit; closest hits and shadow rays, a warp and a lane per ray."""
    r = np.random.default_rng(7)
    side = far * 1e-3
    tris = []
    for z in range(1, 9):
        for i in range(6):
            for j in range(6):
                x0, x1 = far + side * (i / 3 - 1), far + side * ((i + 1) / 3 - 1)
                y0, y1 = side * (j / 3 - 1), side * ((j + 1) / 3 - 1)
                tris += [[[x0, y0, z], [x1, y0, z], [x1, y1, z]], [[x0, y0, z], [x1, y1, z], [x0, y1, z]]]
    sc = mesh_scene(tris)
    n, copies = 3000, 30
    o = np.stack([far + side * r.uniform(-0.9, 0.9, n), side * r.uniform(-0.9, 0.9, n), r.integers(0, 9, n) + 0.5], axis=1)
    tiny = np.array([0.0, -0.0, 1e-35, -1e-31, 1e-29])
    d = np.stack([r.choice(tiny, n), r.choice(tiny, n), r.choice([-1.0, 1.0], n)], axis=1)
    rays = np.concatenate([o, d], axis=1).astype(np.float32)
    tmin = np.full(n, 1e-4, np.float32)
    tmax = r.choice(np.array([0.25, 2.0, 1000.0, np.inf], np.float32), n)
    ctx.upload(sc, layout=abi.BVH_LINEAR)
    want, occ = ctx.trace_closest(rays), ctx.trace_any(rays, tmin, tmax)
    assert (want["mesh"] == 0).mean() > 0.8 and 0.2 < occ.mean() < 0.9
    ctx.upload(sc, layout=layout)
    for k in (1, copies):
        got = ctx.trace_closest(np.tile(rays, (k, 1)))
        assert np.array_equal(got["mesh"], np.tile(want["mesh"], k)) and np.array_equal(got["t"], np.tile(want["t"], k))
        assert np.array_equal(ctx.trace_any(np.tile(rays, (k, 1)), np.tile(tmin, k), np.tile(tmax, k)), np.tile(occ, k))
