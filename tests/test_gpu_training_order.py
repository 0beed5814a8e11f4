"""Training calls back to back on one stream, each kernel placed before the one ahead of it ends: inputs
that the stream's other kernels write just before a step and overwrite just after it, losses cleared
between steps, gradients applied by separate calls, inference between steps, the same calls captured
in a graph, and a second network on a second stream. Every parameter and loss has the bits that it
has when the device is waited for after each call."""
import numpy as np
import pytest

from tests.test_gpu_surrogate import _inputs, _params

pytestmark = pytest.mark.gpu


def steps(net, xs, ys, settle, separate):
    import torch

    x, y = torch.empty_like(xs[0]), torch.empty_like(ys[0])
    loss = torch.zeros(1, device="cuda")
    seen = []
    for k in range(len(xs)):
        x.copy_(xs[k])
        y.copy_(ys[k])
        if separate and k % 2:
            g, l = net.gradients(x, y)
            settle()
            net.apply_gradients(g, 1e-3)
            seen.append(l.clone())
        else:
            net.train_step(x, y, 1e-3, loss)
        settle()
        seen.append(loss.clone())
        if k % 3 == 1:
            loss.zero_()
        x.fill_(float("nan"))  # (must not reach the step before)
        y.fill_(float("nan"))
        if k % 3 == 2:
            seen.append(net.forward(xs[k]).sum().view(1))
        settle()
    return torch.cat(seen)


def data(tiles, count):
    import torch

    xs = [torch.tensor(_inputs(128 * tiles, 20 + k), device="cuda") for k in range(count)]
    rng = np.random.default_rng(9)
    return xs, [torch.tensor(rng.normal(size=128 * tiles).astype(np.float32), device="cuda") for _ in xs]


def network(tiles):
    from pacuda_b200 import surrogate as S

    net = S.Network(12, max_batch=128 * tiles, seed=3)
    net.set_params(_params(3))
    return net


@pytest.mark.parametrize("separate", [False, True])
@pytest.mark.parametrize("tiles", [1, 128, 160])
def test_back_to_back_steps(tiles, separate):
    import torch

    xs, ys = data(tiles, 7)
    got = []
    for settle in (torch.cuda.synchronize, lambda: None):
        net = network(tiles)
        seen = steps(net, xs, ys, settle, separate)
        torch.cuda.synchronize()
        assert net.error() == 0
        got.append((seen.cpu().numpy(), np.array(net.params())))
    assert np.array_equal(got[0][0], got[1][0]) and np.isfinite(got[0][0]).all()
    assert np.array_equal(got[0][1], got[1][1])


def test_two_streams():
    import torch

    xs, ys = data(64, 6)
    alone = network(64)
    want = steps(alone, xs, ys, torch.cuda.synchronize, False).cpu().numpy()
    nets, streams, seen = [network(64), network(64)], [torch.cuda.Stream(), torch.cuda.Stream()], []
    torch.cuda.synchronize()
    for net, s in zip(nets, streams):
        with torch.cuda.stream(s):
            seen.append(steps(net, xs, ys, lambda: None, False))
    torch.cuda.synchronize()
    for net, o in zip(nets, seen):
        assert net.error() == 0
        assert np.array_equal(o.cpu().numpy(), want)
        assert np.array_equal(np.array(net.params()), np.array(alone.params()))


def test_captured_step():
    import torch

    xs, ys = data(32, 5)
    want = network(32)
    x, y, loss = xs[0].clone(), ys[0].clone(), torch.zeros(1, device="cuda")
    net = network(32)
    net.gradients(x, y)  # (the kernels' attributes are set by a first call)
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        grad, _ = net.gradients(x, y)
    for a, b in zip(xs, ys):
        x.copy_(a)
        y.copy_(b)
        g.replay()
        got = grad.clone()
        ref, _ = want.gradients(a, b)
        assert torch.equal(got, ref)
    torch.cuda.synchronize()
    assert net.error() == 0
