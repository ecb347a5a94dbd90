"""Unrounded roots (sngl=False) do not depend on how many lanes search a
chain: layered models in batches on every side of the launch rule's lines and
grid chains at its last one.  The group kernel evaluates several trial
velocities with a lane each or one with all its lanes, so both have to be the
one-lane kernel's function."""
import numpy as np
import pytest

from jdsurfg_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refine", ["tight", "reference"])
@pytest.mark.parametrize("iwave,mode,igr,nlayer", [(1, 1, 0, 6), (1, 2, 1, 37), (2, 1, 0, 37), (2, 2, 0, 5),
                                                   (2, 1, 1, 2)])
def test_layered_models_unrounded(iwave, mode, igr, nlayer, refine):
    from jdsurfg_b200 import Engine
    n = 26001
    rng = np.random.default_rng(nlayer)
    vs = (np.linspace(2.4, 4.6, nlayer) * (1.0 + 0.05 * rng.standard_normal((n, nlayer)))).astype(np.float32)
    if nlayer > 2:
        vs[::7, 0] = 0.0  # a fluid layer on top
    vp = np.where(vs > 0, 1.76 * vs, 1.5).astype(np.float32)
    rho = np.where(vs > 0, 0.32 * vp + 0.77, 1.03).astype(np.float32)
    thk = rng.uniform(1.0, 4.0, (n, nlayer)).astype(np.float32)
    thk[:, -1] = 0.0
    t = np.array([2.0, 5.0, 11.0, 30.0])
    eng = Engine(sngl=False, refine=refine)
    cg, ierr = eng.surfdisp96_batch(thk, vp, vs, rho, 1, iwave, mode, igr, t)
    for a, b in ((0, 1), (1, 130), (0, 3000), (9, 18009), (0, 18001), (1, 26001)):
        c, e = eng.surfdisp96_batch(thk[a:b], vp[a:b], vs[a:b], rho[a:b], 1, iwave, mode, igr, t)
        assert np.array_equal(e, ierr[a:b]) and np.array_equal(c, cg[a:b], equal_nan=True), (a, b)
    eng.close()


# 32 lanes (6000 chains), 4 (9000), and 32 where the launch rule finds the
# columns under water (6000); 592 blocks: one lane
@pytest.mark.parametrize("ncol,waves,learned", [(3000, ("Lc", "Rc"), False), (4500, ("Rc", "Lc"), True),
                                                (6000, ("Lc",), True)])
def test_grid_chains_unrounded(ncol, waves, learned):
    import torch
    from torch.profiler import ProfilerActivity, profile
    from jdsurfg_b200 import Engine, learn
    case = synth.make_case(ncol, 1, np.arange(6, dtype=np.float32) * 3.0, 2.5, 4.6, 0.08,
                           np.array([2.0, 6.0, 15.0, 40.0]), waves, 1, ncol, lvz_frac=0.2, water_frac=0.3)
    out = []
    for kw, kernel in ((dict(), "k_roots_coop"), (dict(block_roots=592), "k_roots_queue")):
        eng = Engine(sngl=False, **kw)
        nets = learn.load_proposals(eng) if learned else None
        eng.setup(case)
        dev = [None if case[k] is None else torch.from_numpy(case[k]).cuda() for k in ("vs", "vp", "rho")]
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
            eng.roots_device(ncol, 1, case["nz"], *dev)
            torch.cuda.synchronize()
        ran = {k for e in prof.events() for k in ("k_roots_coop", "k_roots_queue") if k in e.name}
        assert ran == {kernel}
        out.append(eng.last_roots(ncol))
        del nets
        eng.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
