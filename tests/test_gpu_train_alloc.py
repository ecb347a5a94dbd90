"""A network's first step, and one on a larger batch, pay for two device
allocations (activations, a training step's buffers), however many parts they
have: one allocation per part made a first step slower than all its kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _allocations(f):
    import torch
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        f()
        torch.cuda.synchronize()
    return sum(e.name == "cudaMalloc" for e in prof.events())


def test_first_steps_make_two_allocations():
    import torch
    from jdsurfg_b200.mlp import MLP
    x = torch.randn(4096, 320, device="cuda").bfloat16()
    y = torch.randn(4096, device="cuda")
    MLP(seed=1).train_step(x[:128], y[:128], 1e-3)  # the kernels are loaded
    assert _allocations(lambda: MLP(seed=2)) > 0    # the profiler sees this library's allocations
    net = MLP(seed=3)
    assert _allocations(lambda: net.train_step(x[:1000], y[:1000], 1e-3)) == 2
    assert _allocations(lambda: net.train_step(x[:64], y[:64], 1e-3)) == 0
    assert _allocations(lambda: net.train_step(x, y, 1e-3)) == 2
    net = MLP(seed=4)
    assert _allocations(lambda: net.forward(x)) == 1
    assert _allocations(lambda: net.train_step(x, y, 0.0)) == 1


# the parts of an allocation lie apart: the same gradients on a network whose
# buffers are a larger batch's (the transposes are laid out by the batch at hand)
@pytest.mark.parametrize("M", [1, 129, 1000])
def test_buffers_of_a_larger_batch(M):
    import torch
    from jdsurfg_b200.mlp import MLP
    x = torch.randn(4097, 320, device="cuda").bfloat16()
    y = torch.randn(4097, device="cuda")
    new, used = MLP(seed=5), MLP(seed=5)
    used.train_step(x, y, 0.0)
    used.forward(x)
    assert new.train_step(x[:M], y[:M], 0.0) == used.train_step(x[:M], y[:M], 0.0)
    assert np.array_equal(new.grads(), used.grads())
    assert torch.equal(new.forward(x[:M]), used.forward(x[:M]))
