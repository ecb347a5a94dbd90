"""The root search with several lanes per chain (calls with few chains, and
the deferred retries) against the one-lane search, which a caller's own block
count (block_roots) selects."""
import numpy as np
import pytest

from jdsurfg_b200 import synth

pytestmark = pytest.mark.gpu

PERIODS = np.geomspace(1.5, 40.0, 7)


def _case(ncol, nz, waves, nmode, water, seed):
    depth = synth.depth_grid(min(nz, 21), 1.0, nz, 2.5) if nz > 21 else np.arange(nz, dtype=np.float32) * 2.0
    return synth.make_case(ncol, 1, depth, 2.5, 4.6, 0.08, PERIODS, waves, nmode, seed, lvz_frac=0.2,
                           water_frac=0.3 if water else 0.0)


def _roots(case, learned, **kw):
    import torch
    from jdsurfg_b200 import Engine, learn
    eng = Engine(**kw)
    nets = learn.load_proposals(eng) if learned else None
    eng.setup(case)
    t = lambda a: None if a is None else torch.from_numpy(a).cuda()
    eng.roots_device(case["nx"], case["ny"], case["nz"], t(case["vs"]), t(case["vp"]), t(case["rho"]))
    torch.cuda.synchronize()
    out = eng.last_roots(case["nx"] * case["ny"])
    del nets
    eng.close()
    return out


# chains on both sides of every line of the launch rule (4500, 16000; scans 18000, 26000) and
# the smallest ones; layer counts that leave every remainder of a group's lanes
@pytest.mark.parametrize("ncol,nz,waves,nmode,water,learned", [
    (1, 2, ("Rc",), 1, False, False), (1, 80, ("Rc", "Lc"), 2, True, False), (3, 5, ("Lg",), 1, True, True),
    (4500, 9, ("Rc",), 1, False, True), (4501, 9, ("Rc",), 1, True, True), (751, 12, ("Rc", "Lc"), 2, True, True),
    (3000, 7, ("Rc", "Lc"), 1, False, True), (18000, 6, ("Rc",), 1, True, False), (16000, 4, ("Lc",), 1, False, True),
    (18001, 4, ("Rc",), 1, False, False), (13001, 5, ("Lc", "Rc"), 1, False, False)])
def test_group_search_equals_one_lane(ncol, nz, waves, nmode, water, learned):
    case = _case(ncol, nz, waves, nmode, water, seed=ncol + nz)
    c1, s1 = _roots(case, learned, block_roots=592)
    cg, sg = _roots(case, learned)
    assert np.array_equal(s1, sg) and np.array_equal(c1, cg)
    # the evaluations are the same bits, so the unrounded roots are too
    u1, _ = _roots(case, learned, block_roots=592, sngl=False)
    ug, _ = _roots(case, learned, sngl=False)
    assert np.array_equal(u1, ug)


@pytest.mark.parametrize("waves", [("Rc",), ("Lc",)])
def test_group_search_reference_refinement(waves):
    case = _case(300, 11, waves, 2, True, seed=5)
    c1, s1 = _roots(case, False, block_roots=592, refine="reference")
    cg, sg = _roots(case, False, refine="reference")
    assert np.array_equal(s1, sg) and np.array_equal(c1, cg)


# layered models: 32 lanes per model up to 18 000 of them, 4 up to 26 000, then one
@pytest.mark.parametrize("iwave,mode,igr,nlayer", [(2, 1, 0, 5), (1, 2, 0, 4), (2, 2, 1, 7)])
def test_layered_models_are_the_same_in_any_batch(iwave, mode, igr, nlayer):
    from jdsurfg_b200 import Engine
    n = 26001
    rng = np.random.default_rng(nlayer)
    vs = (np.linspace(2.4, 4.6, nlayer) * (1.0 + 0.05 * rng.standard_normal((n, nlayer)))).astype(np.float32)
    vs[::7, 0] = 0.0  # a fluid layer on top
    vp = np.where(vs > 0, 1.76 * vs, 1.5).astype(np.float32)
    rho = np.where(vs > 0, 0.32 * vp + 0.77, 1.03).astype(np.float32)
    thk = np.full((n, nlayer), 3.0, np.float32)
    thk[:, -1] = 0.0
    t = np.array([3.0, 8.0, 20.0])
    eng = Engine()
    cg, ierr = eng.surfdisp96_batch(thk, vp, vs, rho, 1, iwave, mode, igr, t)
    for a, b in ((0, 1), (1, 130), (130, 18130), (0, 18001)):
        c, e = eng.surfdisp96_batch(thk[a:b], vp[a:b], vs[a:b], rho[a:b], 1, iwave, mode, igr, t)
        assert np.array_equal(e, ierr[a:b]) and np.array_equal(c, cg[a:b])
    eng.close()
