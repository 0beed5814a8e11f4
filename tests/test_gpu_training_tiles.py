"""The training kernels' splits: one tile of 128 points, as many as the parts of the batch that the
weight gradients are split into and one more, one more than the SMs (a block's second turn). The
gradient of a batch is the mean of its halves' gradients: dout scales by a power of two, which no
BF16 rounding sees, so only the order of the FP32 sums differs (2^-24 relative per addition of at
most a few hundred partial sums: 1e-5 of the gradient's norm)."""
import numpy as np
import pytest

from oracle import surrogate_oracle as O
from tests.test_gpu_surrogate import _inputs, _params

pytestmark = pytest.mark.gpu


def network(batch):
    from pacuda_b200 import surrogate as S

    net = S.Network(12, max_batch=batch, seed=3)
    p = _params(3)
    net.set_params(p)
    return net, p


def gradients(net, x, y):
    import torch

    g, loss = net.gradients(torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda"))
    assert net.error() == 0
    return g.cpu().numpy(), float(loss.cpu()[0])


@pytest.mark.parametrize("tiles", [1, 2, 10, 11, 12, 20, 21, 22, 42])
def test_gradients_match_the_oracle(tiles):
    net, p = network(128 * 42)
    x = _inputs(128 * tiles, 4)
    y = np.random.default_rng(5).normal(size=len(x)).astype(np.float32)
    g, loss = gradients(net, x, y)
    want, want_loss = O.gradients(p, x, y)
    assert loss == pytest.approx(want_loss, rel=1e-2)
    for a, b in zip(O.unpack(g), O.unpack(want)):  # as tests/test_gpu_surrogate.py compares them
        a, b = a.astype(np.float64).ravel(), b.astype(np.float64).ravel()
        assert np.linalg.norm(a - b) < 3e-2 * np.linalg.norm(b) + 1e-30
        assert a @ b > 0.999 * np.linalg.norm(a) * np.linalg.norm(b)


@pytest.mark.parametrize("tiles", [2, 22, 42, 150, 298])
def test_a_batch_is_the_mean_of_its_halves(tiles):
    net, _ = network(128 * tiles)
    x = _inputs(128 * tiles, 7)
    y = np.random.default_rng(8).normal(size=len(x)).astype(np.float32)
    half = len(x) // 2
    g, loss = gradients(net, x, y)
    parts = [gradients(net, x[k * half:(k + 1) * half], y[k * half:(k + 1) * half]) for k in range(2)]
    assert loss == pytest.approx(parts[0][1] + parts[1][1], rel=1e-5)
    mean = (parts[0][0].astype(np.float64) + parts[1][0]) / 2
    for a, b in zip(O.unpack(g), O.unpack(mean)):
        assert np.linalg.norm(a - b) < 1e-5 * np.linalg.norm(b)


def test_a_step_equals_gradients_then_apply():
    import torch

    batch = 128 * 23
    x, y = torch.tensor(_inputs(batch, 9), device="cuda"), torch.randn(batch, device="cuda")
    a, b = network(batch)[0], network(batch)[0]
    for step in range(3):
        a.train_step(x, y, 1e-3)
        grad, _ = b.gradients(x, y)
        shifted = torch.empty(grad.numel() + 1, device="cuda")[1:]  # a gradient at an unaligned address
        shifted.copy_(grad)
        b.apply_gradients(shifted, 1e-3)
    assert a.error() == 0 and b.error() == 0
    assert np.array_equal(a.params().view(np.uint32), b.params().view(np.uint32))
    assert torch.equal(a.forward(x), b.forward(x))
