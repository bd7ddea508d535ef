"""The Runge-Kutta sum of an FP32 step keeps its own 24 bits: where a step
changes the state by about the spacing of its FP32 numbers, every coefficient
ends on the FP32 number nearest to the exact result.

The state is given by random Bernstein coefficients that are FP32 numbers in
[1.2, 1.8], whose spacing is 2^-23: their nodal values, formed in FP64, lead back
to them exactly. One step in FP64 gives the exact result (to 1e-9 of a spacing).
The FP32 right-hand side is off by some 1e-5 of the largest change at most, which
is below 500 spacings: 0.5 spacings and 1 % of one are allowed."""
import math

import numpy as np
import pytest

from test_gpu_bernstein import _sized, _variants

pytestmark = pytest.mark.gpu

ULP = 2.0 ** -23


def _basis(pkg, dim, p):
    """V[i][j] = Bernstein polynomial j at node i, both in the mesh's node order."""
    lat = pkg.meshgen._simplex_lattice_order(dim, p)
    f = math.factorial
    return np.array([[f(p) * math.prod((x / p) ** int(a) / f(int(a)) for x, a in zip(pt, al)) for al in lat]
                     for pt in lat])


@pytest.mark.parametrize("dim,p,counts", [(2, 1, 9), (2, 4, 5), (3, 1, (3, 3, 3)), (3, 3, (3, 3, 2)), (3, 4, (3, 3, 2))])
def test_a_step_of_about_one_spacing_is_rounded_once(pkg, dim, p, counts):
    mesh = _sized(pkg, dim, p, counts)
    V = _basis(pkg, dim, p)
    npe, nv = len(V), dim + 1
    ph = dict(v0=(0.1, 0.05, 0.0), rho0=1.0, c0=1.0)
    rng = np.random.default_rng(dim * 10 + p)
    c0 = np.zeros((4, mesh["elem_nodes"].shape[0], npe))
    c0[:nv] = rng.uniform(1.2, 1.8, (nv,) + c0.shape[1:]).astype(np.float32)
    coef = lambda u: np.linalg.solve(V, u.reshape(-1, npe).T).T.reshape(c0.shape)  # noqa: E731
    u0 = (c0 @ V.T).reshape(4, -1)
    D = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **ph)
    dt = 0.9 * ULP / np.median(np.abs(coef(D.rhs(u0, 1.0))[:nv]))
    D.set_state(u0)
    D.snapshot()
    D.run(1, dt)
    want = coef(D.get_state())
    D.close()
    assert np.max(np.abs(want - c0)) < 500 * ULP
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP32, **ph)
    for v in _variants(S):
        S.tune(v)
        S.set_state(u0)
        S.snapshot()
        assert np.max(np.abs(coef(S.get_state()) - c0)) <= 1e-3 * ULP
        S.run(1, dt)
        err = np.max(np.abs(coef(S.get_state()) - want)[:nv]) / ULP
        assert err <= 0.51, (v, err)
    S.close()
