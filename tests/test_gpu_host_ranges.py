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


def test_two_registrations_with_pageable_memory_between(pkg):
    """Such an array is refused, as a copy refuses it; one registration of all of it is taken."""
    torch = pytest.importorskip("torch")
    rt, page = torch.cuda.cudart(), 65536
    S, u = _solver(pkg, counts=30)
    S.set_state(u)
    want = S.get_state()
    k = S.rhs(u, 1e-4)
    raw = np.empty(u.nbytes + 2 * page, np.uint8)
    start = -raw.ctypes.data % page
    arr = raw[start:start + u.nbytes].view(np.float64).reshape(u.shape)
    arr[:] = u
    ptr, last = arr.ctypes.data, (u.nbytes - 1) // page * page
    assert last >= 4 * page
    for p, n in ((ptr, page), (ptr + last, u.nbytes - last)):
        assert int(rt.cudaHostRegister(p, n, 0)) == 0
    try:
        with pytest.raises(pkg.gpu.SolverError, match="DG_ERR_CUDA"):
            S.set_state(arr)
        with pytest.raises(pkg.gpu.SolverError, match="DG_ERR_CUDA"):
            S.rhs(arr, 1e-4)
        with pytest.raises(pkg.gpu.SolverError, match="DG_ERR_CUDA"):
            S.get_state(out=arr)
    finally:
        for p in (ptr, ptr + last):
            assert int(rt.cudaHostUnregister(p)) == 0
    assert np.array_equal(arr, u) and np.array_equal(S.get_state(), want)
    assert int(rt.cudaHostRegister(raw.ctypes.data, raw.nbytes, 0)) == 0
    try:
        S.set_state(np.zeros_like(u))
        S.set_state(arr)
        assert np.array_equal(S.rhs(arr, 1e-4), k)
        S.get_state(out=arr)
        assert np.array_equal(arr, want)
    finally:
        assert int(rt.cudaHostUnregister(raw.ctypes.data)) == 0
    S.close()
