"""FP64 right-hand sides where whole tiles, some lanes or no lane of a face lie
on the boundary: walls and absorbing boundaries, without flow, with inflow and
with outflow (in 3-D the absorbing matrix of an outflow through a face with an
oblique tangent frame has no five-term form), against the CPU oracle.
Tolerance: the project's for a single FP64 right-hand side, 5e-11 relative L2."""
import numpy as np
import pytest

from conftest import rel_l2, smooth_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,p,counts", [(2, 1, 1), (2, 3, 8), (2, 4, 5), (3, 1, (1, 1, 1)), (3, 2, (4, 4, 3)),
                                          (3, 3, (3, 3, 3)), (3, 4, (2, 2, 2))])
@pytest.mark.parametrize("kind", ["Reflecting", "Absorbing", "mixed"])
@pytest.mark.parametrize("v0", [(0.0, 0.0, 0.0), (31.0, -17.0, 12.0), (-40.0, 25.0, -33.0)])
def test_rhs_matches_oracle(pkg, oracle, dim, p, counts, kind, v0):
    mg = pkg.meshgen
    sides = ["xmin", "xmax", "ymin", "ymax", "zmin", "zmax"]
    if dim == 2:
        m = mg.square(n=counts, order=p, seed=5, side_names=sides[:4])
        v0 = (v0[0], v0[1], 0.0)
    else:
        m = mg.box(counts=counts, order=p, seed=6)
    bcs = {s: kind if kind != "mixed" else ("Absorbing", "Reflecting")[i % 2] for i, s in enumerate(sides[:2 * dim])}
    mesh = dict(dim=dim, order=p, xyz=m["xyz"], elem_nodes=m["elem_nodes"], groups=mg.solver_groups(m, bcs))
    ph = dict(v0=v0, rho0=1.2, c0=340.0)
    u, dt = smooth_state(mesh, seed=dim + p), 1e-5
    ref = oracle.Problem(mesh, dt=dt, **ph).stage(u)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **ph)
    k = S.rhs(u, dt)
    S.close()
    assert rel_l2(k[:dim + 1], ref[:dim + 1]) <= 5e-11
