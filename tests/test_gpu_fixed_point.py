"""FP64 stage kernels' fixed-point sums (3-D: gradients, lift and elevation) on
states far from one: scaled by powers of two, single variables, one value far
above the rest, zeros and infinities. Against the CPU oracle at the project's
tolerance for a right-hand side, 5e-11 relative L2; a scaled state's result is
the scaled result to the last bit, since every scale is a power of two."""
import numpy as np
import pytest

from conftest import rel_l2, smooth_state
from test_gpu_bernstein import _sized
from test_gpu_parity import _phys

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,p,counts", [(3, 1, (3, 3, 2)), (3, 2, (3, 2, 2)), (3, 3, (2, 2, 3)), (3, 4, (2, 2, 2)),
                                          (2, 3, 6)])
def test_states_far_from_one(pkg, oracle, dim, p, counts):
    mesh, ph = _sized(pkg, dim, p, counts), _phys(dim)
    u, dt = smooth_state(mesh, seed=9), 1e-4
    P = oracle.Problem(mesh, dt=dt, **ph)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **ph)
    k = S.rhs(u, dt)
    nv = dim + 1
    for e in (-600, -40, 300, 600):
        assert np.array_equal(S.rhs(np.ldexp(u, e), dt)[:nv], np.ldexp(k[:nv], e)), e
    for keep in range(nv):
        w = np.zeros_like(u)
        w[keep] = u[keep]
        assert rel_l2(S.rhs(w, dt)[:nv], P.stage(w)[:nv]) <= 5e-11, keep
    w = u.copy()
    w[0, 3] *= 1e12
    assert rel_l2(S.rhs(w, dt)[:nv], P.stage(w)[:nv]) <= 5e-11
    # elements that it does not reach keep every bit
    same = np.all(P.stage(w) == P.stage(u), axis=0)
    assert np.array_equal(S.rhs(w, dt)[:, same], k[:, same])
    assert not np.any(S.rhs(np.zeros_like(u), dt))
    w = u.copy()
    w[0, 3] = np.inf
    assert not np.all(np.isfinite(S.rhs(w, dt)))
    S.close()
