"""Host arrays that the conversion kernels must not reach themselves, though
their first and last value lie in page-locked memory."""
import numpy as np
import pytest

from conftest import smooth_state
from test_gpu_bernstein import _sized
from test_gpu_parity import _phys

pytestmark = pytest.mark.gpu


def _solver(pkg, dim=2, p=2, counts=5):
    mesh = _sized(pkg, dim, p, counts)
    return pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **_phys(dim)), smooth_state(mesh, seed=4)


@pytest.mark.parametrize("off", [1, 4])
@pytest.mark.parametrize("variant", [64, -1])
def test_page_locked_array_off_the_values_alignment(pkg, off, variant):
    S, u = _solver(pkg)
    S.tune(variant)
    raw = pkg.gpu.pinned_empty((u.nbytes + 8,), np.uint8)
    odd = np.ndarray(u.shape, dtype=np.float64, buffer=raw.data, offset=off)
    odd[:] = u
    assert odd.ctypes.data % 8 == off and not odd.flags.aligned
    S.set_state(u)
    want = S.get_state()
    k = S.rhs(u, 1e-4)
    S.set_state(np.zeros_like(u))
    S.set_state(odd)
    assert np.array_equal(S.get_state(), want) and np.array_equal(S.rhs(odd, 1e-4), k)
    odd[:] = 0.0
    S.get_state(out=odd)
    assert np.array_equal(odd, want)
    S.close()
