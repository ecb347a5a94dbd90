"""The march by half a warp, two pairs per warp, on the CPU (tests/
fmst_half_host.cpp runs the warp's lanes in lockstep): its heap operations
against the reference's heap, at every depth a grid may reach, and its grids
against the one-lane march over the forms that a call may have."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "fmst_half_host.cpp")
HDR = os.path.join(ROOT, "jdsurfg_b200", "csrc", "swdk_fmst_march.cuh")
OUT = os.path.join(ROOT, "tests", "_build", "libfm_half.so")


def _lib():
    if not os.path.exists(OUT) or max(os.path.getmtime(SRC), os.path.getmtime(HDR)) > os.path.getmtime(OUT):
        os.makedirs(os.path.dirname(OUT), exist_ok=True)
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-strict-aliasing", "-shared", "-fPIC",
                        "-I" + os.path.dirname(HDR), SRC, "-o", OUT], check=True)
    return C.CDLL(OUT)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


# heap sizes on both sides of 16 levels (65 535 / 65 536 entries), the two
# halves different, one stopping early; keys below, inside and above the heap's, ties, infinity
@pytest.mark.parametrize("n", [(0, 3), (1, 14), (15, 16), (300, 1), (65534, 9), (65535, 65534), (140000, 65536)])
def test_heap_operations_at_every_depth(n):
    rng = np.random.default_rng(sum(n))
    keys = [np.sort(rng.integers(10, 1000, k)).astype(np.float32) for k in n]  # sorted: a heap, with ties
    for a in keys:
        a[len(a) - len(a) // 50:] = np.inf
    nan = np.nan
    ops = np.array([5, 4, 3, nan, 2000, 500, nan, nan, 1, 7, 7, nan, 0.5, np.inf, 700, nan, 10, nan, 0.25, 0.125],
                   np.float32)
    for cap in (max(n) + len(ops), max(n) + 2):  # the second: the heap gets full
        ns = np.array(n, np.int32)
        bad = _lib().fm_half_heap(_p(ns), _p(keys[0]), _p(keys[1]), _p(ops), len(ops), 13, cap)
        assert bad == 0


def _grid(nx, ny):
    return nx, ny, 40.0, 100.0, 0.3, 0.25


def _sources(grid, n, seed):
    """n sources: on a node, near sides and corners, inside."""
    nx, ny, lat0, lon0, dx, dz = grid
    lat, lon = (lat0 - (nx - 2) * dx, lat0 - dx), (lon0 + dz, lon0 + (ny - 2) * dz)
    e = 0.01
    rng = np.random.default_rng(seed)
    pts = [(lat[0] + e, lon[0] + e), (lat[1] - e, lon[1] - e), (lat[1] - dx / 8, lon[0] + dz / 8),
           (lat[0] + e, lon[1] - e)]
    while len(pts) < n:
        pts.append((rng.uniform(*lat), rng.uniform(*lon)))
    d2r = np.float32(np.pi / 180)
    x = np.array([(np.float32(90.0) - np.float32(a)) * d2r for a, _ in pts[:n]], np.float32)
    z = np.array([np.float32(b) * d2r for _, b in pts[:n]], np.float32)
    return x, z


def _map(grid, kind, seed):
    nx, ny = grid[:2]
    v = np.full((ny, nx), 3.0)
    rng = np.random.default_rng(seed)
    if kind == "rough":
        v *= rng.uniform(0.4, 2.5, v.shape)
    elif kind == "nan":
        v[ny // 2, nx // 2] = np.nan
    elif kind == "inf":
        v[ny // 2, nx // 2] = np.inf
    elif kind == "zero":
        v[:] = 0.0
    elif kind == "sign":
        v[ny // 2, nx // 2] = -30.0
    return np.ascontiguousarray(v)


# grids of one to six cells a side (the smallest lie within the refined box
# and never off their sides' stencils), a lone last pair, maps out of range
@pytest.mark.parametrize("nx,ny,npairs,kind", [
    (4, 4, 1, "flat"), (4, 4, 3, "rough"), (4, 4, 2, "nan"), (4, 9, 2, "inf"), (9, 4, 3, "rough"), (5, 6, 5, "rough"),
    (5, 6, 3, "zero"), (6, 6, 2, "sign"), (6, 5, 2, "nan"), (9, 7, 3, "flat")])
def test_half_warp_march_equals_one_lane(nx, ny, npairs, kind):
    grid = _grid(nx, ny)
    x, z = _sources(grid, npairs, nx)
    if npairs == 5:
        x[1] = np.float32(1.5)  # outside the grid: this half has no pair to march
    v, out = _map(grid, kind, ny), np.zeros(2, np.int32)
    nx_, ny_, *deg = grid
    bad = _lib().fm_half_pairs(nx_, ny_, *[C.c_float(d) for d in deg], npairs, _p(x), _p(z), _p(v), 0, 0, _p(out))
    assert bad == 0 and out[0] == 0


CAPS = ((2, 30, 300, 70000), (2, 30, 64, 300))  # 70 000: the deep heap's march
# bands that outgrow the heap in one half, in both or in none; shared-memory heaps
@pytest.mark.parametrize("shared", [0, 1])
def test_a_half_that_overflows_beside_one_that_does_not(shared):
    grid = _grid(9, 8)
    x, z = _sources(grid, 3, 5)
    v = _map(grid, "rough", 3)
    seen = set()
    nx, ny, *deg = grid
    for cap in CAPS[shared]:
        out = np.zeros(2, np.int32)
        bad = _lib().fm_half_pairs(nx, ny, *[C.c_float(d) for d in deg], 3, _p(x), _p(z), _p(v), cap, shared, _p(out))
        assert bad == 0, cap
        seen.add(int(out[0]))
    assert {0, 1} <= seen
