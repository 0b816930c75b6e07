"""The work the path-tracing core is measured on: ray queries, whole renders of every integrator a
user picks (the default megakernel, the reference's own estimators, the wavefront, the split
bidirectional form, the many-scene batch), the differentiable render and scene edits, each through
the calls a program makes (`Context`, `render_batch`, `autograd.render`).

A case is a dict: "kind" says which call, the rest are its sizes and options. Scenes are the
generators' (Cornell room, displaced icosphere, triangle soup), seeded; a state's seed picks the
scene's noise and materials, the rays and the sample streams.
"""
import math

import numpy as np
import torch

from x3dcore2_gb300 import abi, autograd, scene
from x3dcore2_gb300.core import Context, default_params, pipeline_config, render_batch

MODES = {"mis": abi.MODE_MIS, "lt1": abi.MODE_REF_LT1, "uni": abi.MODE_REF_UNI,
         "bdpt": abi.MODE_REF_BDPT, "bdpt_power": abi.MODE_BDPT_POWER}
LAYOUTS = {"sah": abi.BVH_SAH, "wide": abi.BVH_WIDE}
INTEGRATORS = {"megakernel": abi.INTEGRATOR_MEGAKERNEL, "wavefront": abi.INTEGRATOR_WAVEFRONT}


def listed():
    return [
        # Picking and visibility queries from host code: a few rays against a small scene, where
        # the call itself is what costs.
        {"name": "rays_few", "kind": "rays", "scene": "soup", "tris": 1000, "n": 1500, "layout": "sah"},
        # Visibility, ambient occlusion or light baking: a million rays of no order against a
        # large mesh.
        {"name": "rays_many", "kind": "rays", "scene": "ico", "level": 7, "n": 1000003, "layout": "sah"},
        # A thumbnail or material preview: the Cornell room at 256 x 256, 16 samples, depth 5, the
        # default tree and integrator, the image on the host.
        {"name": "cornell_mis", "kind": "render", "scene": "cornell", "w": 256, "h": 256, "spp": 16, "mode": "mis",
         "layout": "sah", "integrator": "megakernel", "depth": 5, "rr": 3, "out": "host"},
        # A frame with every default left alone: 1080p of the 1.3 M-triangle scene.
        {"name": "frame_default", "kind": "render", "scene": "ico", "level": 8, "w": 1920, "h": 1080, "spp": 16,
         "mode": "mis", "layout": "sah", "integrator": "megakernel", "depth": 8, "rr": 3, "out": "host"},
        # The same for users of the reference's estimator and streams (unidirectional_lt1).
        {"name": "frame_lt1", "kind": "render", "scene": "ico", "level": 7, "w": 1280, "h": 720, "spp": 16,
         "mode": "lt1", "layout": "sah", "integrator": "megakernel", "depth": 0, "rr": 2, "out": "host"},
        # The production frame: 64 samples, eight-wide tree, wavefront, the image stays on the device.
        {"name": "frame_wavefront", "kind": "render", "scene": "ico", "level": 8, "w": 1920, "h": 1080, "spp": 64,
         "mode": "mis", "layout": "wide", "integrator": "wavefront", "depth": 8, "rr": 3, "out": "dev"},
        # The bidirectional frame with power-heuristic weights (subpaths of at most 6 vertices).
        {"name": "frame_bdpt", "kind": "render", "scene": "ico", "level": 8, "w": 1280, "h": 720, "spp": 32,
         "mode": "bdpt_power", "layout": "wide", "integrator": "wavefront", "depth": 0, "rr": 2, "len": 6,
         "out": "dev"},
        # The reference's bidirectional tracer (bidirectional_mis) at an odd preview size.
        {"name": "preview_bdpt_ref", "kind": "render", "scene": "ico", "level": 6, "w": 641, "h": 361, "spp": 8,
         "mode": "bdpt", "layout": "sah", "integrator": "megakernel", "depth": 0, "rr": 2, "len": 8, "out": "host"},
        # Dataset generation: many small scenes, each at its own size, in one call.
        {"name": "batch_scenes", "kind": "batch", "n": 16, "tris_lo": 1000, "tris_hi": 50000, "spp": 16,
         "integrator": "wavefront"},
        # Fitting materials: one forward and backward of the differentiable render (256 materials).
        {"name": "fit_materials", "kind": "adjoint", "level": 7, "materials": 256, "w": 512, "h": 512, "spp": 32,
         "depth": 6, "layout": "sah"},
        # An editor: one object of the 1.3 M-triangle scene moves, the tree is refitted, and a
        # one-sample frame is shown.
        {"name": "edit_frame", "kind": "edit", "level": 8, "w": 1920, "h": 1080, "spp": 1, "layout": "sah"},
        # Deforming geometry: the tree is rebuilt on the device, then a picking batch is traced.
        {"name": "rebuild", "kind": "rebuild", "level": 8, "n": 65536, "layout": "wide"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rays", "default", "default", "lt1", "wavefront", "bdpt_power", "bdpt", "batch", "adjoint",
                       "edit", "rebuild"])
    if kind == "rays":
        c = {"kind": "rays", "n": _log(rng, 1000, 1000000), "layout": rng.choice(["sah", "wide"])}
        if rng.random() < 0.5:
            return {**c, "scene": "soup", "tris": _log(rng, 1000, 200000)}
        return {**c, "scene": "ico", "level": rng.randint(4, 7)}
    if kind == "batch":
        hi = _log(rng, 5000, 50000)
        return {"kind": "batch", "n": rng.randint(2, 16), "tris_lo": 1000, "tris_hi": hi,
                "spp": rng.choice([4, 16]), "integrator": rng.choice(["wavefront", "megakernel"])}
    if kind == "adjoint":
        s = _log(rng, 100, 512)
        return {"kind": "adjoint", "level": rng.randint(5, 7), "materials": _log(rng, 8, 256), "w": s,
                "h": _log(rng, 100, 512), "spp": rng.randint(4, 32), "depth": rng.randint(4, 8),
                "layout": rng.choice(["sah", "wide"])}
    if kind == "edit":
        w = _log(rng, 200, 1920)
        return {"kind": "edit", "level": rng.randint(5, 8), "w": w, "h": max(2, w * 9 // 16), "spp": 1,
                "layout": rng.choice(["sah", "wide"])}
    if kind == "rebuild":
        return {"kind": "rebuild", "level": rng.randint(5, 8), "n": _log(rng, 1000, 65536),
                "layout": rng.choice(["sah", "wide"])}
    w = _log(rng, 100, 1920)
    c = {"kind": "render", "w": w, "h": max(2, w * rng.randint(9, 16) // 16), "out": rng.choice(["host", "dev"])}
    where = rng.choice(["cornell", "soup", "ico"])
    if where == "cornell":
        c |= {"scene": "cornell"}
    elif where == "soup":
        c |= {"scene": "soup", "tris": _log(rng, 1000, 200000)}
    else:
        c |= {"scene": "ico", "level": rng.randint(5, 8)}
    # closed rooms and bidirectional paths trace several times the rays of the open scene
    most = 132e6 if kind == "wavefront" else 29e6
    most /= {"cornell": 8, "soup": 12, "ico": 1}[where] * (4 if kind == "bdpt" else 1)
    c["spp"] = _log(rng, 1, max(1.0, min(64.0, most / (c["w"] * c["h"]))))
    if kind == "wavefront":
        return c | {"mode": "mis", "layout": "wide", "integrator": "wavefront", "depth": rng.randint(4, 10), "rr": 3}
    if kind == "bdpt_power":
        return c | {"mode": "bdpt_power", "layout": "wide", "integrator": "wavefront", "depth": 0, "rr": 2,
                    "len": rng.randint(3, 8)}
    if kind == "bdpt":
        return c | {"mode": "bdpt", "layout": "sah", "integrator": "megakernel", "depth": 0, "rr": 2, "len": 8}
    if kind == "lt1":
        return c | {"mode": rng.choice(["lt1", "uni"]), "layout": "sah", "integrator": "megakernel", "depth": 0,
                    "rr": 2}
    return c | {"mode": "mis", "layout": rng.choice(["sah", "wide"]), "integrator": "megakernel",
                "depth": rng.randint(4, 10), "rr": 3}


def _scene(case, seed, w, h):
    if case.get("scene") == "cornell":
        return scene.cornell(w, h)
    if case.get("scene") == "soup":
        return scene.soup(num_tris=case["tris"], seed=1 + seed % 100000, width=w, height=h)
    return scene.displaced_icosphere(level=case["level"], seed=1 + seed % 100000,
                                     num_materials=case.get("materials", 512), width=w, height=h)


def _num_tris(case):
    return {"cornell": 36, "soup": case.get("tris", 0)}.get(case.get("scene"), 20 * 4 ** case.get("level", 0) + 10)


def _rays(case, seed, box):
    """Rays of no order through the scene's box, and the bounds of the shadow query on them."""
    r = np.random.default_rng(seed)
    lo, hi = box
    n = case["n"]
    o = r.uniform(lo, hi, (n, 3))
    d = r.uniform(lo, hi, (n, 3)) - o
    d /= np.maximum(np.linalg.norm(d, axis=1, keepdims=True), 1e-12)
    rays = np.concatenate([o, d], axis=1).astype(np.float32)
    return rays, np.full(n, 1e-4, np.float32), r.uniform(0.1, 2.0, n).astype(np.float32)


def _box(case):
    return (-0.95, 0.95) if case.get("scene") == "soup" else (-2.0, 2.0)


def _params(case, seed):
    p = default_params(MODES[case["mode"]], case["w"], case["h"], case["spp"], seed=1 + seed,
                       max_depth=case["depth"], rr_start=case["rr"])
    p.integrator = INTEGRATORS[case["integrator"]]
    if case.get("len"):
        p.bdpt_max_len = case["len"]
    return p


def _batch(case, seed):
    r = np.random.default_rng(seed)
    scenes, params = [], []
    for k in range(case["n"]):
        tris = int(round(math.exp(r.uniform(math.log(case["tris_lo"]), math.log(case["tris_hi"])))))
        side = (256, 128, 200)[k % 3]
        scenes.append(scene.soup(num_tris=tris, seed=1 + (seed * 64 + k) % 1000000, width=side, height=side))
        p = default_params(abi.MODE_MIS, side, side, case["spp"], seed=1 + seed + k, max_depth=int(r.integers(4, 11)),
                           rr_start=3)
        p.integrator = INTEGRATORS[case["integrator"]]
        params.append(p)
    return scenes, params


def _turn(seed):
    a = 0.05 + 0.3 * np.random.default_rng(seed).random()
    c, s = math.cos(a), math.sin(a)
    return np.array([[c, 0, s, 0], [0, 1, 0, 0], [-s, 0, c, 0], [0, 0, 0, 1]], np.float32)


def prepare(case, seed):
    ctx = Context(0)
    kind = case["kind"]
    st = {"kind": kind, "ctx": ctx}
    if kind == "batch":
        st["scenes"], st["params"] = _batch(case, seed)
        return st
    w, h = case.get("w", 256), case.get("h", 256)
    sc = _scene(case, seed, w, h)
    ctx.upload(sc, layout=LAYOUTS[case["layout"]],
               builder=abi.BUILDER_DEVICE if kind == "rebuild" else abi.BUILDER_HOST)
    if kind in ("rays", "rebuild"):
        st["rays"], st["tmin"], st["tmax"] = _rays(case, seed, _box(case))
    if kind in ("edit", "rebuild"):
        st["mesh"], st["matrix"] = int(np.argmax(np.diff(sc.toff))), _turn(seed)
    if kind == "edit":
        st["cfg"] = pipeline_config(path_space={"sah": "static_bvh", "wide": "wide_bvh"}[case["layout"]],
                                    samples_per_frame=case["spp"], seed=1 + seed, auto_exposure=True)
        st["size"] = (w, h)
    if kind == "render":
        st["params"] = _params(case, seed)
        if case["out"] == "dev":
            st["image"] = torch.zeros((h, w, 4), dtype=torch.float32, device="cuda")
        if case["integrator"] == "wavefront" and case["mode"] == "mis" and w * h * case["spp"] > 1 << 24:
            # long renders: the configuration the autotuner picks for them, as a program keeps it
            abi.check(ctx.lib.e8g_wavefront_set(ctx.h, 1 << 23, 2, 8), ctx.h)
            abi.check(ctx.lib.e8g_wavefront_set_shade(ctx.h, 6), ctx.h)
    if kind == "adjoint":
        st["params"] = default_params(abi.MODE_MIS, w, h, case["spp"], seed=1 + seed, max_depth=case["depth"],
                                      rr_start=3)
        mats = sc.material_list()
        st["albedo"] = torch.tensor([list(m.albedo) for m in mats], dtype=torch.float32, requires_grad=True)
        st["rough"] = torch.tensor([m.roughness for m in mats], dtype=torch.float32, requires_grad=True)
        st["base"] = mats
        st["dl"] = torch.from_numpy(np.random.default_rng(seed).normal(0.0, 1.0, (h, w, 3)).astype(np.float32))
    return st


def run(st):
    ctx, kind = st["ctx"], st["kind"]
    if kind == "rays":
        return {"hit": ctx.trace_closest(st["rays"]), "occluded": ctx.trace_any(st["rays"], st["tmin"], st["tmax"])}
    if kind == "render":
        if "image" not in st:
            return ctx.render(st["params"])
        ctx.render_dev(st["params"], st["image"].data_ptr())
        return st["image"]
    if kind == "batch":
        return render_batch(ctx, st["scenes"], st["params"])[0]
    if kind == "adjoint":
        st["albedo"].grad = st["rough"].grad = None
        img = autograd.render(ctx, st["params"], st["albedo"], st["rough"], st["base"])
        img.backward(st["dl"])
        return {"image": img.detach(), "albedo": st["albedo"].grad, "roughness": st["rough"].grad}
    ctx.transform_mesh(st["mesh"], st["matrix"])
    if kind == "edit":
        px, rgba = ctx.pipeline_frame(st["cfg"], *st["size"], want_rgba=True)
        return {"pixels": px, "image": rgba}
    stats = ctx.commit(abi.COMMIT_REBUILD)
    return {"hit": ctx.trace_closest(st["rays"]), "nodes": stats["num_nodes"], "leaves": stats["num_leaves"]}


def work(case):
    """Bytes: the scene's nodes, triangles and vertices once, inputs and outputs once. Operations:
    rays times a descent of a binary tree (two box tests of 20 operations a level) and one
    triangle test (45)."""
    kind = case["kind"]
    nt = (case["tris_lo"] + case["tris_hi"]) // 2 * case["n"] if kind == "batch" else _num_tris(case)
    tree = nt * (64 + 48)
    per_ray = 40 * max(1.0, math.log2(max(2, nt))) + 45
    if kind == "rays":
        return {"bytes": tree + case["n"] * (2 * 24 + 8 + 20 + 1), "flops": 2 * case["n"] * per_ray}
    if kind == "rebuild":
        return {"bytes": nt * (16 + 3 * 32) + tree + case["n"] * 44, "flops": case["n"] * per_ray}
    if kind == "batch":
        px = case["n"] * 200 * 200
        return {"bytes": tree + nt * 112 + px * 16, "flops": px * case["spp"] * 8 * per_ray}
    px = case["w"] * case["h"]
    rays = px * case["spp"] * (1.5 if case.get("scene", "ico") == "ico" else 6)
    if kind == "render" and case["mode"].startswith("bdpt"):
        rays *= 4
    if kind == "adjoint":
        return {"bytes": tree + nt * 112 + px * 28, "flops": 2 * rays * per_ray}
    if kind == "edit":
        return {"bytes": 2 * tree + nt * 2 * 96 + px * 20, "flops": rays * per_ray}
    return {"bytes": tree + nt * 112 + px * 16, "flops": rays * per_ray}


def exact(case, seed):
    """Ray queries on small scenes: every triangle against every ray in 64 bits. A render's value
    is an integral over random paths and has none that is quick to compute."""
    if case["kind"] != "rays" or case["n"] * _num_tris(case) > 4e9:
        return None
    sc = _scene(case, seed, 256, 256)
    rays, tmin, tmax = _rays(case, seed, _box(case))
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tri = torch.from_numpy(sc.world_triangles().astype(np.float64)).to(dev)
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.cross(e1, e2, dim=1)
    out_t, out_b = [], []
    step = max(1, int(2e7 // len(tri)))
    for k in range(0, len(rays), step):
        r = torch.from_numpy(rays[k:k + step].astype(np.float64)).to(dev)
        o, d = r[:, None, :3], r[:, None, 3:]
        s = o - a
        det = -(d * n).sum(-1)
        q = torch.cross(s, d.expand_as(s), dim=-1)
        t = (s * n).sum(-1) / det
        b1, b2 = (q * e2).sum(-1) / det, -(q * e1).sum(-1) / det
        ok = (det != 0) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1) & (t >= 1e-4) & (t <= 1000.0)
        t = torch.where(ok, t, torch.inf)
        best, at = t.min(dim=1)
        hit = torch.isfinite(best)
        out_t.append(torch.where(hit, best, 0.0))
        b = torch.stack([b1.gather(1, at[:, None])[:, 0], b2.gather(1, at[:, None])[:, 0]], dim=1)
        out_b.append(torch.where(hit[:, None], b, 0.0))
    hit = {"t": torch.cat(out_t).cpu().numpy(), "mesh": None, "tri": None, "b": torch.cat(out_b).cpu().numpy()}
    return {"hit": hit, "occluded": None}
