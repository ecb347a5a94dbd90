"""A captured call keeps the scratch it was captured with: host-memory calls,
calls on a larger grid and the other path's calls on the same context, made
between the capture and a replay, must not move it."""
import numpy as np
import pytest

from jdsurfg_b200 import Engine, learn, synth

pytestmark = pytest.mark.gpu


def _case(ncol, seed):
    depth = synth.depth_grid(21, 1.0, 24, 2.5)
    return synth.make_case(ncol, 1, depth, 2.5, 4.6, 0.08, np.geomspace(3.0, 40.0, 11), ("Rc", "Rg", "Lc", "Lg"), 1,
                           seed, lvz_frac=0.2, water_frac=0.2)


def _dev(case):
    import torch
    return [None if case[k] is None else torch.from_numpy(case[k]).cuda() for k in ("vs", "vp", "rho")]


def _outputs(eng, case, path):
    import torch
    k, n = eng.kmax, case["nx"] * case["ny"]
    vc = torch.zeros((k, n), dtype=torch.float64, device="cuda")
    st = torch.zeros((k, n), dtype=torch.int32, device="cuda")
    ker = torch.zeros((k, case["nz"], n), dtype=torch.float64, device="cuda") if path == "kernel" else None
    return vc, torch.zeros_like(vc), ker, st


def _host(eng, case, path):
    f = eng.get_1d_kernel if path == "kernel" else eng.get_2d_map
    return f(case["vs"], case["vp"], case["rho"], nx=case["nx"])


# 3000 columns: several chunks of a host call's outputs, so its second stream's store is used
@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("ncol", [70, 3000])
@pytest.mark.parametrize("path", ["kernel", "map"])
def test_replay_after_other_calls(path, ncol, learned):
    import torch
    a, larger = _case(ncol, 3), _case(2 * ncol + 5, 4)
    other = "map" if path == "kernel" else "kernel"
    eng = Engine(device=0)
    nets = learn.load_proposals(eng) if learned else None
    eng.setup(a)
    vs, vp, rho = _dev(a)
    vc, vout, ker, st = out = _outputs(eng, a, path)
    eng.graph_capture(path, a["nx"], a["ny"], a["nz"], vs, vp, rho, vc, vout, ker, st)
    ref = [None if t is None else t.cpu().numpy() for t in out]  # the eager call of the capture
    calls = [lambda: _host(eng, a, path), lambda: _host(eng, a, other), lambda: _host(eng, larger, path),
             lambda: eng.roots_device(larger["nx"], 1, larger["nz"], *_dev(larger))]
    for call in calls:
        call()
        # whoever gets memory that was freed would have it overwritten by the replay
        fill = [torch.full((1 << 26,), 7, dtype=torch.uint8, device="cuda") for _ in range(8)]
        for t in out:
            if t is not None:
                t.zero_()
        torch.cuda.synchronize()
        eng.graph_launch(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        for t, r in zip(out, ref):
            assert t is None or np.array_equal(t.cpu().numpy(), r)
        assert all(bool((f == 7).all()) for f in fill)
        del fill
    h = _host(eng, a, path)
    assert np.array_equal(h["vc"], ref[0]) and np.array_equal(h["vout"], ref[1])
    assert path == "map" or np.array_equal(h["kernel"], ref[2])
    del nets
    eng.close()


@pytest.mark.parametrize("path", ["kernel", "map"])
def test_branches_batch_replay_after_host_calls(path):
    from jdsurfg_b200.batch import UnevenBatch
    cases = [_case(n, n) for n in (40, 900, 2600)]
    b = UnevenBatch(cases, path=path, mode="branches")
    b.capture()
    b.launch()
    ref = [b.outputs(i) for i in range(len(cases))]
    for i, c in enumerate(cases):
        eng = b.engines[i]
        for p in ("kernel", "map"):
            _host(eng, c, p)
            _host(eng, _case(3 * c["nx"], 5), p)
    b.launch()
    for i, r in enumerate(ref):
        got = b.outputs(i)
        for k in r:
            assert np.array_equal(got[k], r[k]), (i, k)
    b.close()
