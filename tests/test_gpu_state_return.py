"""What dg_get_state returns after dg_set_state: to the roundings that the header
names, and as set or rounded to FP32 by the kernels on nodal values.

The bound: a coefficient is off by its rounding to the context's precision, half
a spacing of at most m times the largest value, and by the FP64 rounding of the
sums of up to 35 terms each way; the basis functions at a node are non-negative
and sum to one."""
import numpy as np
import pytest

from test_gpu_bernstein import _sized
from test_gpu_parity import _phys

pytestmark = pytest.mark.gpu

M = {1: 1.0, 2: 3.0, 3: 10.0, 4: 35.0}  # largest row sum of the inverse basis matrix in 3-D


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("dim", [2, 3])
def test_state_comes_back_to_rounding(pkg, dim, p, prec):
    mesh = _sized(pkg, dim, p, 5 if dim == 2 else (3, 2, 2))
    g = pkg.gpu
    S = g.Solver(mesh, precision=g.DG_FP64 if prec == "fp64" else g.DG_FP32, **_phys(dim))
    E, npe = mesh["elem_nodes"].shape
    u = np.zeros((4, E, npe))
    u[:dim + 1] = np.random.default_rng(p).normal(size=(dim + 1, E, npe))
    u = u.reshape(4, -1)
    S.set_state(u)
    err = np.abs(S.get_state() - u).reshape(4, E, npe).max(axis=2)
    top = np.abs(u).reshape(4, E, npe).max(axis=2)
    half = 2.0 ** -53 if prec == "fp64" else 2.0 ** -24
    assert np.all(err <= M[p] * (half + 70 * 2.0 ** -53) * top)
    S.tune(-1)
    S.set_state(u)
    assert np.array_equal(S.get_state(), u if prec == "fp64" else u.astype(np.float32).astype(np.float64))
    S.close()
