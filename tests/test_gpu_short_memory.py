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
