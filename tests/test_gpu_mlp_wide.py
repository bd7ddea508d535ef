"""Networks with two adjacent wide layers, around the widths whose activations
still fit beside the fused passes' weight stream: those that fit forward and
backward, forward only, or not at all give the oracle's outputs and gradients;
tolerances as in test_gpu_mlp.py."""
import numpy as np
import pytest

from conftest import rel_l2
from test_gpu_mlp import mlp_ref
from test_gpu_mlp_fused import _net

pytestmark = pytest.mark.gpu

# the widest sum that fits, one beyond it; forward only; neither
NETS = [[6, 704, 704, 5], [6, 704, 705, 5], [6, 512, 1024], [6, 512, 512, 1024], [6, 768, 768], [6, 1024, 512, 9],
        [6, 1024, 1024, 5]]


@pytest.mark.parametrize("widths", NETS)
@pytest.mark.parametrize("n", [9, 300])
def test_wide_networks_match_oracle(pkg, widths, n):
    torch = pytest.importorskip("torch")
    net, p = _net(pkg, widths)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, (n, widths[0])).astype(np.float32)
    t = rng.normal(size=(n, widths[-1])).astype(np.float32)
    y_ref, _ = mlp_ref.forward(p, widths, x)
    y = net.forward(x)
    assert rel_l2(y, y_ref) <= 1e-5
    xd, yd = torch.from_numpy(x).cuda(), torch.empty((n, widths[-1]), device="cuda")
    torch.cuda.synchronize()
    net.forward_device(xd.data_ptr(), n, yd.data_ptr(), None)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(yd.cpu().numpy(), y)
    g, loss = net.gradient(x, t)
    loss_ref, g_ref = mlp_ref.loss_and_grad(p, widths, x, t)
    assert abs(loss - loss_ref) <= 1e-5 * abs(loss_ref)
    assert rel_l2(g, g_ref) <= 1e-4
    # a training step, and the forward pass of the weights after it
    net.set_data(x, t)
    losses = net.train(1, n, 1e-3, 1e-3, seed=5)
    assert abs(losses[0] - loss) <= 1e-6 * loss
    y_ref, _ = mlp_ref.forward(net.get_params(), widths, x)
    assert rel_l2(net.forward(x), y_ref) <= 1e-5
