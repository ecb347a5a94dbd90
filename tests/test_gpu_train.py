"""The training step's kernels at batch sizes around their tiles: rows of a
GEMM tile (64, 128), of a weight-gradient slice and its pipeline's stages."""
import numpy as np
import pytest

from test_gpu_mlp import _np_mlp_loss_grads

pytestmark = pytest.mark.gpu


# BF16 operands (half an ulp 2^-9) through five layers and back: about 1 % of a
# layer's gradient; 5 % as the bound, as for the one batch size tested beside it
@pytest.mark.parametrize("M", [5, 31, 32, 33, 63, 64, 65, 127, 128, 129, 1000, 4097])
def test_gradients_match_fp64_at_tile_edges(M):
    import torch
    from jdsurfg_b200.mlp import MLP, layout
    net = MLP(seed=7)
    wb = torch.from_numpy(net.params()).bfloat16().double().numpy()
    rng = np.random.default_rng(M)
    x = np.zeros((M, 320), np.float32)
    x[:, :258] = rng.standard_normal((M, 258)).astype(np.float32) * 0.5
    y = rng.standard_normal(M).astype(np.float32) * 0.3
    xb = torch.from_numpy(x).cuda().bfloat16()
    loss = net.train_step(xb, torch.from_numpy(y).cuda(), 0.0)
    g = net.grads().astype(np.float64)
    lref, gref = _np_mlp_loss_grads(wb, xb.double().cpu().numpy(), y.astype(np.float64))
    assert abs(loss - lref) < 1e-2 * max(1.0, abs(lref))
    for wo, n, k, bo in layout():  # weights and biases of a layer together: a bias alone may nearly cancel
        a, b = (np.concatenate([v[wo:wo + n * k], v[bo:bo + n]]) for v in (g, gref))
        assert np.linalg.norm(a - b) < 0.05 * np.linalg.norm(b)
