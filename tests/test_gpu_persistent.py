"""Many RK4 steps in one launch, on FP64 meshes whose tiles all fit on the GPU
at once: runs across launches of 64 steps with sources and observers in the same
elements against the oracle, meshes from one tile up to the resident limit
against one launch per stage, the selection rule, and bounded waits.

Tolerances are the ones the project holds every stage kernel to
(test_gpu_parity.py): states after a run 1e-12 relative L2, observer samples
ten times that, residuals 1e-10."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

from conftest import rel_l2, smooth_state
from test_gpu_bernstein import _sized
from test_gpu_parity import _phys, _sources_observers

pytestmark = pytest.mark.gpu

BB, PERSIST = 64, 80
DT = 1e-4


def _solver(pkg, mesh, ph):
    return pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **ph)


@pytest.mark.parametrize("dim,p,counts", [(2, 1, 5), (2, 2, 4), (2, 3, 9), (2, 4, 5), (3, 1, (3, 3, 3)), (3, 2, (1, 1, 1)),
                                          (3, 3, (3, 3, 3)), (3, 4, (2, 2, 3))])
def test_runs_across_launches_match_oracle(pkg, oracle, dim, p, counts):
    mesh = _sized(pkg, dim, p, counts)
    ph = _phys(dim)
    nsteps = 70
    z = 0.1 if dim == 3 else 0.0
    srcs = [[0.1, -0.2, z, 0.45, 1.0, 50.0, 0.3, 1.0], [0.3, -0.1, z, 0.5, 0.7, 80.0, 0.0, 66.5 * DT]]
    # the first observer reads elements that hold source nodes, the second most tiles
    obs = [(0.2, -0.1, z, 0.4), (-0.4, -0.5, z, 1.1)]
    P = oracle.Problem(mesh, t_start=0.0, t_end=(nsteps - 0.5) * DT, dt=DT, t_rate=1.0, method=0,
                       sources=[dict(kind=oracle.SRC_SINE, params=s) for s in srcs], observers=obs,
                       ics=[(0.2, 0.1, 0.0, 0.3, 1.0)], **ph)
    ref = P.run()
    assert ref["steps"] == nsteps
    sdofs, odofs, ows = _sources_observers(mesh, srcs, obs)
    times, _ = pkg.host.schedule(0.0, (nsteps - 0.5) * DT, DT, 1.0)
    vals = np.stack([np.where(times < s[7], s[4] * np.sin(2 * np.pi * s[5] * times + s[6]), np.nan) for s in srcs], 1)
    S = _solver(pkg, mesh, ph)
    # the default here, but for the one element that it is not built for
    assert (S.info()["kernel_variant"] >= PERSIST) == ((dim, p) != (3, 4))
    u0 = P.initial_state()
    S.set_state(u0)
    S.snapshot()
    S.set_sources(sdofs)
    S.set_source_values(vals)
    S.set_observers(odofs, ows)
    S.step = 0
    parts = [S.run(n, DT) for n in (1, 2, nsteps - 3)]
    res, tr = np.concatenate([r for r, _ in parts]), np.concatenate([t for _, t in parts])
    nv, tol = dim + 1, 1e-12
    assert rel_l2(S.get_state()[:nv], ref["state"][:nv]) <= tol
    assert rel_l2(res[:, :4], ref["residuals"][:, :4]) <= 1e-10
    want = ref["obs"][:, :, [1, 2, 3, 4]]
    ok = np.isfinite(want)
    assert np.array_equal(np.isfinite(tr), ok)
    assert rel_l2(tr[ok], want[ok]) <= tol * 10
    S.close()


@pytest.mark.parametrize("dim,p", [(2, 1), (2, 4), (3, 2), (3, 3)])
def test_from_one_tile_to_the_resident_limit(pkg, dim, p):
    S = _solver(pkg, _sized(pkg, dim, p, 4 if dim == 2 else (4, 2, 2)), _phys(dim))
    tiles = S.kernel_info(PERSIST)[3]  # resident blocks per SM
    S.close()
    assert tiles > 0
    import torch
    limit = tiles * torch.cuda.get_device_properties(0).multi_processor_count

    def counts(n):  # about n elements
        if dim == 2:
            return int(round((n / 2) ** 0.5))
        k = max(1, int(round((n / 6) ** (1 / 3))))
        return (k, k, max(1, int(n // (6 * k * k))))

    below, above = counts(limit * 32 * 0.97), counts(limit * 32 * 1.25)
    for c, fits in ((4 if dim == 2 else (4, 2, 2), True), (below, True), (above, False)):
        mesh = _sized(pkg, dim, p, c)
        ph = _phys(dim)
        S = _solver(pkg, mesh, ph)
        assert (S.info()["n_elems"] + 31) // 32 <= limit if fits else S.info()["n_elems"] > 32 * limit
        v = S.info()["kernel_variant"]
        assert (v >= PERSIST) == fits and (S.kernel_info(PERSIST)[0] > 0) == fits
        if not fits:
            with pytest.raises(pkg.gpu.SolverError):
                S.tune(PERSIST)
            S.close()
            continue
        u0 = smooth_state(mesh, seed=2)
        out = []
        for variant in (v, BB):
            S.tune(variant)
            S.set_state(u0)
            S.snapshot()
            S.step = 0
            res, _ = S.run(67, 1e-5)
            out.append((S.get_state(), res))
        S.close()
        nv, tol = dim + 1, 1e-12
        assert rel_l2(out[0][0][:nv], out[1][0][:nv]) <= tol
        assert rel_l2(out[0][1], out[1][1]) <= 1e-10


@pytest.mark.parametrize("dim,p,counts", [(2, 3, 9), (3, 2, (3, 3, 3)), (2, 1, 1)])
def test_wait_that_gives_up_and_non_finite_state(pkg, dim, p, counts):
    mesh = _sized(pkg, dim, p, counts)
    S = _solver(pkg, mesh, _phys(dim))
    S.tune(PERSIST)
    u0 = smooth_state(mesh, seed=3)
    S.set_state(u0)
    S.snapshot()
    want = S.run(5, DT)[0]
    u = S.get_state()
    S.set_wait_limit(0)
    S.set_state(u0)
    with pytest.raises(pkg.gpu.SolverError, match="DG_ERR_TIMEOUT"):
        S.run(5, DT)
    S.set_wait_limit(1 << 20)
    bad = u0.copy()
    bad[0, 1] = np.nan
    S.set_state(bad)
    with pytest.raises(pkg.gpu.SolverError, match="DG_ERR_NONFINITE"):
        S.run(5, DT)
    S.set_state(u0)
    assert np.array_equal(S.run(5, DT)[0], want) and np.array_equal(S.get_state(), u)
    S.close()


def test_two_contexts_in_two_threads(pkg):
    """Launches that each need most of the GPU, from two threads at once."""
    ph, tiles = _phys(2), 900
    mesh = _sized(pkg, 2, 1, int((tiles * 16) ** 0.5))
    u0 = smooth_state(mesh, seed=1)
    ctx = [_solver(pkg, mesh, ph) for _ in range(2)]
    assert all(S.info()["kernel_variant"] >= PERSIST for S in ctx)

    def run(S):
        S.set_state(u0)
        S.snapshot()
        for _ in range(5):
            S.run(100, 1e-6)
        return S.get_state()

    want = run(ctx[0])
    with ThreadPoolExecutor(2) as pool:
        for u in pool.map(run, ctx):
            assert np.array_equal(u, want)
    for S in ctx:
        S.close()
