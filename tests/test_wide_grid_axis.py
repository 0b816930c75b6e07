"""The eight-wide grid of a node's axis in single precision equals the double-precision form bit for bit:
boxes of all sizes and places, empty ones, extents at and beside 251 times a power of two, origins at and
beside multiples of the step, and values near the ends of the float range."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "x3dcore2_gb300", "csrc")


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    path = tmp_path_factory.mktemp("grid") / "grid.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", "-o", str(path), f"-I{CSRC}",
                    os.path.join(ROOT, "tests", "cpp", "wide_grid_axis.cpp")], check=True)
    return C.CDLL(str(path))


def cases(kind, n, r):
    scale = np.ldexp(1.0, r.integers(-20, 20, n))
    lo = r.uniform(-1, 1, n) * scale
    hi = lo + r.uniform(0, 1, n) * scale * np.ldexp(1.0, r.integers(-22, 1, n))
    step = np.abs(scale) * 2.0**-18
    if kind == "powers":  # extents of 251 steps, and a few ulps beside them
        e = r.integers(-18, 10, n)
        lo = np.where(r.random(n) < 0.3, 0.0, lo)
        hi = lo.astype(np.float32) + (251 * np.ldexp(1.0, e)).astype(np.float32)
        hi = hi.astype(np.float32).view(np.int32) + np.where(hi > 0, r.integers(-40, 41, n), 0).astype(np.int32)
        hi = hi.astype(np.int32).view(np.float32)
    elif kind == "grid":  # origins on multiples of powers of two
        e = r.integers(-12, 12, n)
        lo = r.integers(-300, 300, n) * np.ldexp(1.0, e)
        hi = lo + r.integers(0, 600, n) * np.ldexp(1.0, e)
    elif kind == "flat":
        hi = lo
    elif kind == "extreme":
        scale = np.ldexp(1.0, r.integers(-149, 127, n))
        lo = r.uniform(-1, 1, n) * scale
        hi = lo + r.uniform(0, 1, n) * np.ldexp(1.0, r.integers(-149, 127, n))
        step = np.maximum(np.abs(scale) * 2.0**-18 * np.ldexp(1.0, r.integers(0, 30, n)), 2.0**-100)
    lo, hi = lo.astype(np.float32), hi.astype(np.float32)
    return lo, np.maximum(lo, hi), np.maximum(step, 2.0**-100)


@pytest.mark.parametrize("kind", ["random", "powers", "grid", "flat", "extreme"])
def test_single_precision_grid_equals_double(lib, kind):
    r = np.random.default_rng(len(kind))
    n = 400000
    lo, hi, step = cases(kind, n, r)
    out = []
    for single in (0, 1):
        e, org, inv = np.zeros(n, np.uint32), np.zeros(n, np.float32), np.zeros(n, np.float32)
        f = np.ctypeslib.as_ctypes
        lib.grid_axes(f(lo), f(hi), f(step), C.c_int(n), C.c_int(single), f(e), f(org), f(inv))
        out.append((e, org.view(np.uint32), inv.view(np.uint32)))
    for a, b in zip(*out):
        bad = np.flatnonzero(a != b)
        assert len(bad) == 0, (lo[bad[:3]], hi[bad[:3]], step[bad[:3]], a[bad[:3]], b[bad[:3]])
