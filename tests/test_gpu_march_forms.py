"""The march by half a warp on the device against the march by one lane per
pair, over the forms a call may have (tests/test_fmst_half_host.py compares
the same code on the CPU)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D2R = np.float32(np.pi / 180)


def _pairs(grid, npairs, nrcv, seed):
    nx, ny, lat0, lon0, dx, dz = grid
    rng = np.random.default_rng(seed)
    lat = lambda n: rng.uniform(lat0 - (nx - 2) * dx + 0.01, lat0 - dx - 0.01, n)
    lon = lambda n: rng.uniform(lon0 + dz + 0.01, lon0 + (ny - 2) * dz - 0.01, n)
    col = lambda a: ((np.float32(90.0) - a.astype(np.float32)) * D2R).astype(np.float32)
    rad = lambda a: (a.astype(np.float32) * D2R).astype(np.float32)
    return dict(slot=np.zeros(npairs, np.int32), srcx=col(lat(npairs)), srcz=rad(lon(npairs)),
                group=np.zeros(npairs, np.int32), rcv_ptr=np.arange(npairs + 1, dtype=np.int64) * nrcv,
                rcx=col(lat(npairs * nrcv)), rcz=rad(lon(npairs * nrcv)))


def _run(grid, pairs, v, **opt):
    import torch
    from jdsurfg_b200.fmst import FMST
    f = FMST(*grid)
    f.set_options(**opt)
    m = torch.from_numpy(np.ascontiguousarray(v.reshape(1, -1))).cuda()
    r = f.pairs(pairs, m, m, want_fdm=True)
    out = [r[k].cpu().numpy() for k in ("ttime", "status", "fdm")], f.last_info()
    f.close()
    return out


def _same(a, b):
    return all(np.array_equal(x, y, equal_nan=x.dtype.kind == "f") for x, y in zip(a, b))


def _rough(grid, seed):
    return np.random.default_rng(seed).uniform(1.5, 4.5, (grid[1], grid[0]))


# pairs whose band outgrows the first pass's heap are marched again with the
# grid's full heap: 71 065 entries here, the sift-up of 17 levels
@pytest.mark.parametrize("npairs", [1, 3])
def test_full_heap_of_more_than_65535_entries(npairs):
    grid = (50, 50, 40.0, 100.0, 0.2, 0.2)
    pairs, v = _pairs(grid, npairs, 7, npairs), _rough(grid, 1)
    ref, _ = _run(grid, pairs, v, lanes_per_warp=1, lanes_per_pair=1, smem_heap=0)
    got, info = _run(grid, pairs, v, smem_heap=64)
    assert info["overflow_pairs"] == npairs and (ref[1] == 0).all()
    assert _same(ref, got)


# odd numbers of pairs leave a warp's second half without one; the smallest grids lie within the refined box
@pytest.mark.parametrize("nx,ny", [(4, 4), (5, 6), (6, 4), (21, 6)])
@pytest.mark.parametrize("npairs", [1, 2, 3])
def test_small_grids_and_lone_pairs(nx, ny, npairs):
    grid = (nx, ny, 40.0, 100.0, 0.3, 0.25)
    pairs, v = _pairs(grid, npairs, 5, nx + ny), _rough(grid, ny)
    ref, _ = _run(grid, pairs, v, lanes_per_warp=1, lanes_per_pair=1)
    for heap in (-1, 0, 40):
        got, _ = _run(grid, pairs, v, smem_heap=heap)
        assert _same(ref, got), heap


# shared-memory heaps up to all of a block's 200 KB (25 598 entries, one pair a
# warp); the largest two of a warp (12 798); the next sizes are refused
@pytest.mark.parametrize("lanes,per,heap", [(4, 4, 25598), (8, 8, 25598), (4, 4, 12800), (8, 4, 12798), (8, 8, 12798),
                                            (1, 1, 25598)])
def test_largest_shared_heaps(lanes, per, heap):
    from jdsurfg_b200.engine import SwdkError
    grid = (33, 36, 40.0, 100.0, 0.2, 0.2)  # a full heap of 31 933 entries
    pairs, v = _pairs(grid, 5, 5, 9), _rough(grid, 2)
    ref, _ = _run(grid, pairs, v, lanes_per_warp=1, lanes_per_pair=1, smem_heap=0)
    got, info = _run(grid, pairs, v, lanes_per_warp=lanes, lanes_per_pair=per, smem_heap=heap)
    assert info["overflow_pairs"] == 0 and _same(ref, got)
    with pytest.raises(SwdkError, match="set_options"):
        _run(grid, pairs, v, lanes_per_warp=lanes, lanes_per_pair=per,
             smem_heap=25600 if lanes == per else 12800)
