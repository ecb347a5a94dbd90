"""The eigenfunction passes where their launch changes shape: more columns than
the resident blocks take at once."""
import numpy as np
import pytest

from jdsurfg_b200 import Engine, synth

pytestmark = pytest.mark.gpu


def _case(ncol, nz, nt, waves, nmode=1, water=0.3, seed=1):
    depth = np.arange(nz, dtype=np.float32) * 2.0
    return synth.make_case(ncol, 1, depth, 2.5, 4.6, 0.08, np.geomspace(3.0, 40.0, nt), waves, nmode, seed,
                           lvz_frac=0.2, water_frac=water)


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
