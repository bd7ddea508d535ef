"""A batch used more than once: a state set for one instance after a run, and
a run longer than the ones before it."""
import numpy as np
import pytest

from conftest import rel_l2, smooth_state
from test_gpu_bernstein import _sized
from test_gpu_parity import _sources_observers

pytestmark = pytest.mark.gpu

ORDERS = (2, 3, 2, 4, 2)


def _batch(pkg, prec, dt=1e-4):
    """Instances 0, 2 and 4 share an element type; their sizes end inside tiles of 32 elements."""
    meshes = [_sized(pkg, 2, p, 3 + k) for k, p in enumerate(ORDERS)]
    B = pkg.gpu.Batch([dict(mesh=m, v0=(3.0 * k, -2.0, 0.0), dt=dt / (1 + k)) for k, m in enumerate(meshes)],
                      rho0=1.2, c0=100.0, precision=pkg.gpu.DG_FP64 if prec == "fp64" else pkg.gpu.DG_FP32)
    return B, meshes


@pytest.mark.parametrize("prec,fused", [("fp64", False), ("fp32", False), ("fp32", True)])
def test_a_longer_run_after_a_shorter_one(pkg, prec, fused):
    """Beyond 1024 steps the result buffers of the runs before are too small."""
    dt, parts = 1e-6, (11, 1100, 9)
    n = sum(parts)
    # 1120 steps of rounding, as a random walk of the states' spacing, with room
    tol = 1e-13 if prec == "fp64" else 2e-5
    B, meshes = _batch(pkg, prec, dt)
    if fused:
        B.set_fused(True)
    obs = [(0.5, 0.5, 0.0, 2.0), (-2.0, 1.0, 0.0, 1.5)]
    src = [[-3.0, -3.0, 0.0, 1.2]]
    sets = [_sources_observers(m, src, obs) for m in meshes]
    vals = np.sin(0.01 * np.arange(n))[:, None]
    for k, m in enumerate(meshes):
        B.set_state(k, smooth_state(m, seed=k))
        B.set_sources(k, sets[k][0], vals)
        B.set_observers(k, sets[k][1], sets[k][2])
    runs = [B.run(s) for s in parts]
    for k, m in enumerate(meshes):
        S = pkg.gpu.Solver(m, v0=(3.0 * k, -2.0, 0.0), rho0=1.2, c0=100.0,
                           precision=pkg.gpu.DG_FP64 if prec == "fp64" else pkg.gpu.DG_FP32)
        S.set_state(smooth_state(m, seed=k))
        S.snapshot()
        S.set_sources(sets[k][0])
        S.set_source_values(vals)
        S.set_observers(sets[k][1], sets[k][2])
        want = np.concatenate([S.run(s, dt / (1 + k))[1] for s in parts])
        assert rel_l2(np.concatenate([r[k] for r in runs]), want) <= tol, k
        assert rel_l2(B.get_state(k), S.get_state()) <= tol, k
        S.close()
    B.close()


@pytest.mark.parametrize("variant", ["", "-1"])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("which", [(2,), (0, 4), (0, 2, 4)])
def test_state_of_some_instances_after_a_run(pkg, monkeypatch, which, prec, variant):
    if variant:
        monkeypatch.setenv("DGFEM_STAGE_VARIANT", variant)
    B, meshes = _batch(pkg, prec)
    A, _ = _batch(pkg, prec)
    for k, m in enumerate(meshes):
        u = smooth_state(m, seed=k)
        A.set_state(k, u)
        B.set_state(k, u)
    A.run(5)
    B.run(5)
    want = [A.get_state(k) for k in range(A.n)]
    for k in which:
        B.set_state(k, smooth_state(meshes[k], seed=10 + k))
    got = [B.get_state(k) for k in range(B.n)]
    tol = 4e-14 if prec == "fp64" else 2e-6  # of a change of basis, as in test_gpu_host_arrays.py
    for k in range(B.n):
        if k in which:
            u = smooth_state(meshes[k], seed=10 + k)
            assert np.max(np.abs(got[k] - u)) <= tol * np.max(np.abs(u)), k
        else:
            np.testing.assert_array_equal(got[k], want[k])
    A.close()
    B.close()
