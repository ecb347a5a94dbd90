"""The eigenfunction passes where their launch changes shape: group slots around
the slots of one round (a third of 32, 64, 96 or 128 threads), one to several
rounds, and more columns than the resident blocks take at once."""
import numpy as np
import pytest

import oracle_lib as O
from jdsurfg_b200 import Engine, synth
from test_gpu_parity import TOL_C, TOL_K, _kernel_relerr

pytestmark = pytest.mark.gpu


def _case(ncol, nz, nt, waves, nmode=1, water=0.3, seed=1):
    depth = np.arange(nz, dtype=np.float32) * 2.0
    return synth.make_case(ncol, 1, depth, 2.5, 4.6, 0.08, np.geomspace(3.0, 40.0, nt), waves, nmode, seed,
                           lvz_frac=0.2, water_frac=water)


@pytest.mark.parametrize("nt,waves,nmode", [(1, ("Rg",), 1), (10, ("Lg",), 1), (11, ("Rg",), 1), (21, ("Rg", "Lg"), 1),
                                            (22, ("Rg",), 1), (32, ("Lg",), 1), (33, ("Rg",), 1), (42, ("Rg",), 1),
                                            (43, ("Lg", "Rc"), 1), (17, ("Rg", "Lg"), 2), (86, ("Rg",), 1)])
def test_group_kernels_match_oracle(nt, waves, nmode):
    case = _case(4, 7 + nt % 3, nt, waves, nmode, seed=nt)
    r = Engine(refine=1).run_case(case)
    ref = O.get_1d_kernel(case, refine=1)
    np.testing.assert_array_equal(r["status"], ref["status"])
    assert np.abs(r["vc"] - ref["vc"]).max() <= TOL_C
    assert np.abs(r["vout"] - ref["vout"]).max() <= TOL_C
    assert _kernel_relerr(r["kernel"], ref["kernel"]) <= TOL_K


@pytest.mark.parametrize("path", ["kernel", "map"])
@pytest.mark.parametrize("waves", [("Rc", "Rg"), ("Lc", "Lg")])
def test_columns_beyond_the_resident_blocks(waves, path):
    """A column's outputs are the same bits alone and among 6500 (two to four
    columns per block), invalid columns between them."""
    case = _case(6500, 6, 5, waves, seed=3)
    case["vs"][2, 5::97] = np.nan
    eng = Engine(refine=1)
    a = eng.run_case(case, path=path)
    cols = np.array([0, 1, 5, 6, 1775, 1776, 1777, 2960, 3552, 5920, 6499])
    b = eng.run_case(synth.subset_columns(case, cols), path=path)
    for k in a:
        if isinstance(a[k], np.ndarray):
            assert np.array_equal(a[k][..., cols], b[k]), k
