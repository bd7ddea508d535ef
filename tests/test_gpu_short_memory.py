"""Calls whose buffers do not fit (more than the device has) fail, and the next
ones that fit give what they gave before."""
import ctypes as C

import numpy as np
import pytest

from conftest import smooth_state
from test_gpu_bernstein import _sized
from test_gpu_parity import _phys, _sources_observers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,variant", [("fp64", 80), ("fp64", 64), ("fp32", 64), ("fp64", -1)])
def test_run_after_one_whose_results_do_not_fit(pkg, prec, variant):
    mesh = _sized(pkg, 2, 2, 5)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64 if prec == "fp64" else pkg.gpu.DG_FP32, **_phys(2))
    S.tune(variant)
    u = smooth_state(mesh, seed=3)
    _, od, ow = _sources_observers(mesh, [], [(0.5, 0.3, 0.0, 2.0)])
    S.set_observers(od, ow)

    def run():
        S.set_state(u)
        S.snapshot()
        S.step = 0
        res, obs = S.run(20, 1e-4)
        return res, obs, S.get_state()

    want = run()
    for n in (1 << 38, 1 << 36):  # 11 and 2 TB of residuals
        assert pkg.gpu.lib().dg_run(S.h, C.c_int64(n), C.c_double(1e-4), None, None) == 2  # DG_ERR_CUDA
        for a, b in zip(run(), want):
            np.testing.assert_array_equal(a, b)
    S.close()


@pytest.mark.parametrize("tc", [False, True])
def test_network_calls_after_one_whose_rows_do_not_fit(pkg, tc):
    net = pkg.gpu.Network([6, 40, 24, 5])
    rng = np.random.default_rng(0)
    net.set_params(rng.normal(0, 0.3, net.n_params).astype(np.float32))
    net.set_tensor_cores(tc)
    x = rng.uniform(-1, 1, (64, 6)).astype(np.float32)
    t = rng.normal(size=(64, 5)).astype(np.float32)
    y, (g, loss) = net.forward(x), net.gradient(x, t)
    L, n = pkg.gpu._mlp_lib(), C.c_int64(1 << 38)  # 6 TB of inputs: refused before any array is read
    f = lambda a: a.ctypes.data_as(C.POINTER(C.c_float))  # noqa: E731
    assert L.dg_mlp_forward(net.h, f(x), n, f(y.copy())) == 2
    np.testing.assert_array_equal(net.forward(x), y)
    assert L.dg_mlp_gradient(net.h, f(x), f(t), n, f(g.copy()), None) == 2
    again, loss2 = net.gradient(x, t)
    assert loss2 == loss
    np.testing.assert_array_equal(again, g)
    net.set_data(x, t)
    assert L.dg_mlp_set_data(net.h, f(x), f(t), n) == 2
    with pytest.raises(pkg.gpu.SolverError, match="DG_ERR_ARG"):  # no training rows any more
        net.train(1, 16, 1e-3, 1e-3)
    net.set_data(x, t)
    assert np.isfinite(net.train(1, 16, 1e-3, 1e-3)).all()
