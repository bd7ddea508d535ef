"""The network's fused passes (one launch each for the forward pass, the chain
of input gradients and the weight gradients) against the float64 oracle at the
edges of their tiles: widths around 16, 64, 256 and the widest that is fused,
one layer, a width beyond it (per-layer GEMMs), row counts around the 8-, 16-
and 32-row tiles and a second wave of them; tolerances as in test_gpu_mlp.py."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_mlp import mlp_ref

pytestmark = pytest.mark.gpu

NETS = [[3, 4], [6, 128, 128, 1], [5, 33, 300, 17], [7, 1024, 20], [65, 16, 257], [6, 1100, 5]]


def _net(pkg, widths, seed=3):
    rng = np.random.default_rng(seed)
    p = mlp_ref.init_params(widths, seed=seed)
    pos = 0
    for k, n in zip(widths[:-1], widths[1:]):
        p[pos + n * k:pos + n * k + n] = rng.normal(0, 0.1, n)
        pos += n * k + n
    net = pkg.gpu.Network(widths)
    net.set_params(p)
    return net, p


@pytest.mark.parametrize("widths", NETS)
@pytest.mark.parametrize("n", [1, 8, 9, 1217, 2500])
def test_forward_device_matches_oracle(pkg, widths, n):
    torch = pytest.importorskip("torch")
    net, p = _net(pkg, widths)
    x = np.random.default_rng(n).uniform(-1, 1, (n, widths[0])).astype(np.float32)
    y_ref, _ = mlp_ref.forward(p, widths, x[-200:])
    xd = torch.from_numpy(x).cuda()
    yd = torch.full((n + 1, widths[-1]), 7.0, device="cuda")  # one row that must stay
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    net.forward_device(xd.data_ptr(), n, yd.data_ptr(), stream.cuda_stream)
    torch.cuda.synchronize()
    y = yd.cpu().numpy()
    assert np.all(y[n] == 7.0)
    assert rel_l2(y[:n][-200:], y_ref) <= 1e-5
    np.testing.assert_array_equal(net.forward(x), y[:n])


def test_forward_device_with_overlapping_arrays(pkg):
    torch = pytest.importorskip("torch")
    widths, n = [8, 64, 8], 700
    net, p = _net(pkg, widths)
    x = np.random.default_rng(0).uniform(-1, 1, (n, 8)).astype(np.float32)
    want = net.forward(x)
    for shift in (0, 1):  # in place, and one row further on
        buf = torch.zeros((n + 1, 8), device="cuda")
        buf[:n] = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        net.forward_device(buf.data_ptr(), n, buf[shift:].data_ptr(), None)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(buf[shift:shift + n].cpu().numpy(), want)


def test_non_finite_rows_stay_apart(pkg):
    widths, n = [6, 40, 24, 5], 64
    net, p = _net(pkg, widths)
    x = np.random.default_rng(1).uniform(-1, 1, (n, 6)).astype(np.float32)
    want = net.forward(x)
    x[3, 2], x[10, 0], x[20, 1] = np.inf, -np.inf, np.nan
    y = net.forward(x)
    ok = np.setdiff1d(np.arange(n), [3, 10, 20])
    np.testing.assert_array_equal(y[ok], want[ok])
    assert np.all(np.isnan(y[20])) and not np.any(np.isfinite(y[[3, 10]]).all(axis=1))


@pytest.mark.parametrize("widths", NETS)
@pytest.mark.parametrize("n", [1, 16, 33, 1300])
def test_gradient_matches_oracle(pkg, widths, n):
    net, p = _net(pkg, widths)
    rng = np.random.default_rng(n + 1)
    x = rng.uniform(-1, 1, (n, widths[0])).astype(np.float32)
    t = rng.normal(size=(n, widths[-1])).astype(np.float32)
    g, loss = net.gradient(x, t)
    loss_ref, g_ref = mlp_ref.loss_and_grad(p, widths, x, t)
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    pos = 0
    for k, m in zip(widths[:-1], widths[1:]):
        for size in (m * k, m):
            assert rel_l2(g[pos:pos + size], g_ref[pos:pos + size]) <= 1e-4, (k, m, size)
            pos += size


@pytest.mark.parametrize("widths", [[6, 32, 300, 9], [6, 1100, 5]])
def test_training_step_is_adamw_of_the_gradient(pkg, widths):
    net, p = _net(pkg, widths)
    n, lr, wd = 24, 1e-3, 0.1
    rng = np.random.default_rng(2)
    x = rng.uniform(-1, 1, (n, widths[0])).astype(np.float32)
    t = rng.normal(size=(n, widths[-1])).astype(np.float32)
    g, loss = net.gradient(x, t)
    net.set_data(x, t)
    losses = net.train(1, n, lr, lr, seed=5, weight_decay=wd)  # one batch of all rows, in another order
    assert abs(losses[0] - loss) <= 1e-6 * loss
    q = net.get_params()
    # first step: m / c1 = g, v / c2 = g^2
    want = p - lr * (g / (np.abs(g) + 1e-8) + wd * p)
    sure = np.abs(g) > 1e-3 * np.abs(g).max()  # where the order of the rows cannot turn the sign
    assert np.max(np.abs(q - want)[sure]) <= 1e-3 * lr
    # the weights that the passes read follow the masters
    y_ref, _ = mlp_ref.forward(q, widths, x)
    assert rel_l2(net.forward(x), y_ref) <= 1e-5
