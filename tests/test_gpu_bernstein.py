"""Bernstein-basis stage kernels (the default on straight-sided triangles and
tetrahedra): parity with the CPU oracle at every order and precision on meshes
around the 32-element tiles, with sources that cover parts of elements,
observers, Euler steps, element means and changes between the state layouts.

Tolerances are the ones the project holds every stage kernel to
(test_gpu_parity.py): a single right-hand side 5e-11 (FP64) / 5e-4 (FP32)
relative L2, states and observer samples after a run 1e-12 / 1e-5 (samples
ten times that)."""
import numpy as np
import pytest

from conftest import rel_l2, smooth_state
from test_gpu_parity import _mesh, _phys, _sources_observers

pytestmark = pytest.mark.gpu

BB = 64  # first Bernstein-basis variant


def _variants(S):
    return [v for v in range(BB, BB + 16) if S.kernel_info(v)[0] > 0]


def _sized(pkg, dim, p, counts):
    mg = pkg.meshgen
    if dim == 2:
        m = mg.square(n=counts, order=p, seed=3, side_names=["xmin", "xmax", "ymin", "ymax"])
    else:
        m = mg.box(counts=counts, order=p, seed=4)
    bcs = {"xmin": "Reflecting", "xmax": "Absorbing", "ymin": "Absorbing", "ymax": "Reflecting", "zmin": "Absorbing",
           "zmax": "Reflecting"}
    return dict(dim=dim, order=p, xyz=m["xyz"], elem_nodes=m["elem_nodes"], groups=mg.solver_groups(m, bcs))


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
# 2, 32 (one full tile), 50; 6, 96 (three full tiles), 162 elements
@pytest.mark.parametrize("dim,counts", [(2, 1), (2, 4), (2, 5), (3, (1, 1, 1)), (3, (4, 2, 2)), (3, (3, 3, 3))])
def test_rhs_matches_oracle_around_tile_sizes(pkg, oracle, dim, counts, p, prec):
    mesh = _sized(pkg, dim, p, counts)
    ph = _phys(dim)
    u = smooth_state(mesh, seed=7 * dim + p)
    dt = 1e-4
    ref = oracle.Problem(mesh, dt=dt, **ph).stage(u)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64 if prec == "fp64" else pkg.gpu.DG_FP32, **ph)
    assert S.info()["kernel_variant"] >= BB
    variants = _variants(S)
    assert variants
    for v in variants:
        S.tune(v)
        k = S.rhs(u, dt)
        assert rel_l2(k[:dim + 1], ref[:dim + 1]) <= (5e-11 if prec == "fp64" else 5e-4), v
        if dim == 2:
            assert np.all(k[3] == 0.0)
    S.close()


@pytest.mark.parametrize("dim,p,prec", [(2, 1, "fp64"), (2, 4, "fp64"), (3, 3, "fp64"), (2, 2, "fp32"), (2, 4, "fp32"),
                                        (3, 1, "fp32"), (3, 4, "fp32")])
@pytest.mark.parametrize("method", ["Runge-Kutta", "Euler1"])
def test_run_with_partial_sources_matches_oracle(pkg, oracle, dim, p, prec, method):
    mesh = _mesh(pkg, dim, p)
    ph = _phys(dim)
    dt, nsteps = 1e-4, 12
    # overlapping sources whose radii cut elements, the second inactive from step 6 on
    srcs = [[0.1, -0.2, 0.1 if dim == 3 else 0.0, 0.45, 1.0, 50.0, 0.3, 1.0],
            [0.3, -0.1, 0.0, 0.5, 0.7, 80.0, 0.0, 5.5 * dt]]
    obs = [(0.5, 0.3, 0.2 if dim == 3 else 0.0, 0.4), (-0.4, -0.5, 0.0, 1.1)]
    euler = method == "Euler1"
    P = oracle.Problem(mesh, t_start=0.0, t_end=(nsteps - 0.5) * dt, dt=dt, t_rate=1.0, method=1 if euler else 0,
                       sources=[dict(kind=oracle.SRC_SINE, params=s) for s in srcs], observers=obs,
                       ics=[(0.2, 0.1, 0.0, 0.3, 1.0)], **ph)
    ref = P.run()
    assert ref["steps"] == nsteps
    u0 = P.initial_state()
    sdofs, odofs, ows = _sources_observers(mesh, srcs, obs)
    times, _ = pkg.host.schedule(0.0, (nsteps - 0.5) * dt, dt, 1.0)
    vals = np.stack([np.where(times < s[7], s[4] * np.sin(2 * np.pi * s[5] * times + s[6]), np.nan) for s in srcs], 1)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64 if prec == "fp64" else pkg.gpu.DG_FP32, **ph)
    tol = 1e-12 if prec == "fp64" else 1e-5
    nv, npe = dim + 1, mesh["elem_nodes"].shape[1]
    for v in _variants(S):
        S.tune(v)
        S.set_state(u0)
        S.snapshot()
        S.set_sources(sdofs)
        S.set_source_values(vals)
        S.set_observers(odofs, ows)
        S.step = 0
        res, tr = S.run(nsteps, dt, euler=euler)
        u = S.get_state()
        assert rel_l2(u[:nv], ref["state"][:nv]) <= tol, v
        assert rel_l2(res[:, :4], ref["residuals"][:, :4]) <= (1e-10 if prec == "fp64" else 1e-3), v
        ob_ref = ref["obs"][:, :, [1, 2, 3, 4]]  # p, vx, vy, vz
        ok = np.isfinite(ob_ref)
        assert np.array_equal(np.isfinite(tr), ok)
        assert rel_l2(tr[ok], ob_ref[ok]) <= tol * 10, v
        # element means: those of the nodal values
        pm, rm, vm = S.cell_means()
        m = u.reshape(4, -1, npe).mean(axis=2)
        assert rel_l2(pm, m[0]) <= tol and rel_l2(rm, m[0] / ph["c0"] ** 2) <= tol and rel_l2(vm, m[1:].T) <= tol
        # the hard overwrite: source nodes hold the injected values, the other
        # nodes of their elements are left alone (one step of almost no length)
        S.set_state(u0)
        S.step = 0
        S.run(1, 1e-30)
        want = u0[0].copy()
        for k, d in enumerate(sdofs):
            want[d] = vals[0, k]
        assert np.max(np.abs(S.get_state()[0] - want)) <= tol * np.max(np.abs(want))
    S.close()


@pytest.mark.parametrize("dim,p", [(2, 3), (3, 2)])
def test_state_and_snapshot_follow_a_change_of_kernel(pkg, dim, p):
    """dg_tune between kernels of different state layouts keeps state,
    snapshot, sources and observers."""
    mesh = _mesh(pkg, dim, p)
    ph = _phys(dim)
    u0 = smooth_state(mesh, seed=5)
    obs = [(0.5, 0.3, 0.2 if dim == 3 else 0.0, 0.4)]
    sdofs, odofs, ows = _sources_observers(mesh, [[0.1, -0.2, 0.0, 0.45]], obs)
    dt = 1e-4
    vals = np.sin(1.0 + np.arange(9))[:, None]

    def run(plan):
        S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **ph)
        S.tune(plan[0])
        S.set_state(u0)
        S.snapshot()
        S.set_sources(sdofs)
        S.set_source_values(vals)
        S.set_observers(odofs, ows)
        out = []
        for v in plan:
            S.tune(v)
            out.append(S.run(3, dt))
        u = S.get_state()
        S.close()
        return u, np.concatenate([r for r, _ in out]), np.concatenate([o for _, o in out])

    ref = run([-1, -1, -1])
    got = run([BB, -1, BB])
    for a, b, tol in zip(got, ref, (1e-12, 1e-10, 1e-11)):
        assert rel_l2(a, b) <= tol


@pytest.mark.parametrize("dim,p,prec", [(2, 1, "fp64"), (2, 3, "fp32"), (3, 2, "fp64"), (3, 3, "fp32")])
@pytest.mark.parametrize("chunks", [[21], [1, 7, 8, 5], [3] * 7])
def test_sources_apart_from_observers_in_any_split_of_a_run(pkg, oracle, dim, p, prec, chunks):
    """Where no observer reads a source's element, a step's end also places
    the next step's sources; runs of one to 21 steps (around the 8 steps of
    the longer step graph) follow the oracle, step index and source rows
    included."""
    mesh = _sized(pkg, dim, p, 6 if dim == 2 else (3, 3, 3))
    ph = _phys(dim)
    half = 5.0 if dim == 2 else 1.0
    dt, nsteps = (2e-4 if dim == 2 else 1e-4), sum(chunks)
    src = [-0.7 * half, -0.6 * half, -0.5 * half if dim == 3 else 0.0, 0.25 * half, 1.0, 60.0, 0.3, 1.0]
    obs = [(0.6 * half, 0.6 * half, 0.6 * half if dim == 3 else 0.0, 0.3 * half)]
    P = oracle.Problem(mesh, t_start=0.0, t_end=(nsteps - 0.5) * dt, dt=dt, t_rate=1.0,
                       sources=[dict(kind=oracle.SRC_SINE, params=src)], observers=obs,
                       ics=[(0.5 * half, 0.5 * half, 0.0, 0.1 * half, 1.0)], **ph)
    ref = P.run()
    sdofs, odofs, ows = _sources_observers(mesh, [src], obs)
    npe = mesh["elem_nodes"].shape[1]
    assert len(sdofs[0]) and len(odofs[0]) and not set(sdofs[0] // npe) & set(odofs[0] // npe)
    times, _ = pkg.host.schedule(0.0, (nsteps - 0.5) * dt, dt, 1.0)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64 if prec == "fp64" else pkg.gpu.DG_FP32, **ph)
    S.set_state(P.initial_state())
    S.snapshot()
    S.set_sources(sdofs)
    S.set_source_values((src[4] * np.sin(2 * np.pi * src[5] * times + src[6]))[:, None])
    S.set_observers(odofs, ows)
    out = [S.run(n, dt) for n in chunks]
    assert S.step == nsteps
    tol = 1e-12 if prec == "fp64" else 1e-5
    res, tr = np.concatenate([r for r, _ in out]), np.concatenate([o for _, o in out])
    assert rel_l2(S.get_state()[:dim + 1], ref["state"][:dim + 1]) <= tol
    assert rel_l2(res[:, :4], ref["residuals"][:, :4]) <= (1e-10 if prec == "fp64" else 1e-3)
    assert rel_l2(tr, ref["obs"][:, :, [1, 2, 3, 4]]) <= tol * 10
    S.close()


@pytest.mark.parametrize("dim,p", [(2, 4), (3, 2)])
def test_fp32_residual_of_a_large_finite_state_is_finite(pkg, dim, p):
    """FP32 squares overflow from 1.8e19 on; a state beyond that is reported
    as non-finite only when it is."""
    mesh = _mesh(pkg, dim, p)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP32, **_phys(dim))
    u = smooth_state(mesh, seed=3)
    for scale in (1.0, 1e25):
        S.set_state(np.zeros_like(u))
        S.snapshot()
        S.set_state(u * scale)
        res, _ = S.run(1, 1e-30)
        m = (u * scale) ** 2
        want = np.array([m[0].mean(), m[0].mean() / _phys(dim)["c0"] ** 4] + [m[q].mean() for q in (1, 2, 3)])
        assert np.max(np.abs(res[0] - want)[want > 0] / want[want > 0]) <= 1e-5
    u[0, 5] = np.inf
    S.set_state(u)
    with pytest.raises(pkg.gpu.SolverError, match="DG_ERR_NONFINITE"):
        S.run(1, 1e-30)
    S.close()


@pytest.mark.parametrize("dim,p", [(2, 1), (2, 4), (3, 2), (3, 4)])
def test_fp64_fixed_point_follows_the_scale_of_the_state(pkg, oracle, dim, p):
    """The FP64 kernels lift in integers at the scale of each element's data:
    a state times a power of two gives the right-hand side times it, bit for
    bit, over the exponent range; elements at rest beside loud ones and
    variables of very different size keep the single right-hand side's bound."""
    mesh = _mesh(pkg, dim, p)
    ph = _phys(dim)
    S = pkg.gpu.Solver(mesh, precision=pkg.gpu.DG_FP64, **ph)
    u = smooth_state(mesh, seed=21)
    k = S.rhs(u, 0.5)
    for e in (-600, -52, 1, 300, 900):
        np.testing.assert_array_equal(S.rhs(np.ldexp(u, e), 0.5), np.ldexp(k, e))
    assert np.all(S.rhs(np.zeros_like(u), 0.5) == 0.0)
    npe = mesh["elem_nodes"].shape[1]
    quiet = u.copy()
    quiet[:, :u.shape[1] // npe // 2 * npe] = 0.0
    uneven = u * np.array([1e6, 1.0, 1e-6, 1e-3])[:, None]
    for v in (quiet, uneven):
        if dim == 2:
            v[3] = 0.0
        ref = oracle.Problem(mesh, dt=1e-4, **ph).stage(v)
        assert rel_l2(S.rhs(v, 1e-4)[:dim + 1], ref[:dim + 1]) <= 5e-11
    bad = u.copy()
    bad[0, 0], bad[1, npe * 7] = np.nan, np.inf
    r = S.rhs(bad, 1e-4).reshape(4, -1, npe)
    assert not np.isfinite(r[0, 0]).any() and not np.isfinite(r[1, 7]).all()
    S.close()
