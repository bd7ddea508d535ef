"""dg_set_state, dg_get_state and dg_rhs on page-locked host arrays (read and
written by the kernels themselves) and on pageable ones: the same bits, for
whole arrays and for parts of a larger one; and the batch's states, whose large
planes are copied by several threads."""
import numpy as np
import pytest

from conftest import smooth_state
from test_gpu_bernstein import _sized
from test_gpu_parity import _phys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,p,counts,prec,variant", [(2, 1, 1, "fp64", None), (2, 4, 7, "fp32", None),
                                                       (3, 3, (3, 3, 2), "fp32", None), (3, 2, (3, 3, 3), "fp64", None),
                                                       (3, 2, (3, 3, 3), "fp64", -1)])
def test_page_locked_and_pageable_arrays_agree(pkg, dim, p, counts, prec, variant):
    g = pkg.gpu
    mesh = _sized(pkg, dim, p, counts)
    S = g.Solver(mesh, precision=g.DG_FP64 if prec == "fp64" else g.DG_FP32, **_phys(dim))
    if variant is not None:
        S.tune(variant)
    u = smooth_state(mesh, seed=4)
    n = S.ndof
    room = g.pinned_empty((4 * n + 3,))
    inner = room[3:].reshape(4, n)  # an interior part, not 16-byte aligned
    room[:] = -7.0
    inner[:] = u
    S.set_state(u)
    want = S.get_state()
    k = S.rhs(u, 1e-4)
    assert np.array_equal(S.rhs(inner, 1e-4), k)
    S.set_state(np.zeros_like(u))
    S.set_state(inner)
    assert np.array_equal(S.get_state(), want)
    out = g.pinned_empty((4, n))
    assert np.array_equal(S.get_state(out=out), want)
    S.get_state(out=inner)
    assert np.array_equal(inner, want) and np.all(room[:3] == -7.0)
    S.close()


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_batch_states_return(pkg, prec):
    meshes = [_sized(pkg, 2, p, n) for p, n in ((4, 5), (4, 60), (1, 3))]  # planes of 750, 108,000 and 54 values
    B = pkg.gpu.Batch([dict(mesh=m, v0=(0.0, 0.0, 0.0), dt=1e-6) for m in meshes], rho0=1.2, c0=340.0,
                      precision=pkg.gpu.DG_FP64 if prec == "fp64" else pkg.gpu.DG_FP32)
    states = [smooth_state(m, seed=k) for k, m in enumerate(meshes)]
    for k, u in enumerate(states):
        B.set_state(k, u)
    for k, u in enumerate(states):
        # to the rounding of the state and of the change of basis
        assert np.max(np.abs(B.get_state(k) - u)) <= (4e-14 if prec == "fp64" else 2e-6) * np.max(np.abs(u))
    B.close()
