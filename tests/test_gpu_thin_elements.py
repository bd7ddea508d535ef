"""FP64 right-hand sides on elements a million times thinner than wide: what
varies along the layer keeps FP64's precision beside the metric across it.

With v_x = x, nothing else and no mean flow, an element without boundary faces has
dp/dt = -rho0 c0^2 (the field is continuous). Its terms are products of metric
entries along x (at most 6 for these boxes) and coefficients of at most 1, lifted
with weights of some 100 at order 4: 1e-13 leaves a factor of ten. One unit of
2^-57 at the scale of the metric across the layer is 2e-11."""
import numpy as np
import pytest

from test_gpu_bernstein import _sized, _variants

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,p", [(2, 1), (2, 4), (3, 1), (3, 2), (3, 3), (3, 4)])
def test_divergence_along_a_thin_layer(pkg, dim, p):
    mesh = _sized(pkg, dim, p, 6 if dim == 2 else (3, 3, 3))
    xyz = mesh["xyz"] = mesh["xyz"] * np.array([0.2, 0.2, 1.0] if dim == 2 else [1.0, 1.0, 1.0])
    xyz[:, dim - 1] *= 2.0 ** -20
    en = mesh["elem_nodes"]
    corners = xyz[en[:, :dim + 1]]
    inner = np.ones(len(en), bool)
    for d in range(dim):
        for side in (xyz[:, d].min(), xyz[:, d].max()):
            inner &= (corners[:, :, d] == side).sum(1) < dim
    assert inner.sum() >= 6
    rho0, c0, dt = 1.2, 100.0, 1.0
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, v0=(0.0, 0.0, 0.0), rho0=rho0, c0=c0)
    u = np.zeros((4, en.size))
    u[1] = xyz[en.reshape(-1), 0]
    for v in _variants(S):
        S.tune(v)
        k = S.rhs(u, dt)[0].reshape(en.shape)[inner]
        assert np.max(np.abs(k / (-dt * rho0 * c0 * c0) - 1.0)) <= 1e-13, v
    S.close()
