"""The work that users of this framework have it do, as cases that can be timed.

A solver case is one output interval of a run, as the dgalerkin driver and a
program on the C ABI have it: the residual snapshot, a number of RK4 steps
with sources and observers, and the whole state read back. The meshes are the
project's seeded jittered ones (meshgen), the sizes those of its
configurations and tests and the range around them. FP64 is the driver's
default; a context made for FP32 computes FP32 numbers which the ABI hands
over as doubles, so they are returned as the FP32 numbers that they are.
"""
import functools
import importlib
import math

import numpy as np
import torch

RHO0, C0, CFL = 1.225, 340.0, 0.5
SURROGATE = "6,256,256,256,256,512"  # the spectral surrogate's layers
ERROR_NET = "6,128,128,1"            # its error network's
SIDES = ("xmin", "xmax", "ymin", "ymax", "zmin", "zmax")


def _pkg():
    return importlib.import_module("dgfem-acoustic_gb300")


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _solver(name, order, counts, precision, steps, walls, mach, what="run"):
    c = dict(kind=what, dim=len(counts), order=order, nx=counts[0], ny=counts[1], nz=counts[2] if len(counts) > 2 else 0,
             precision=precision, steps=steps, walls=walls, mach=mach)
    return dict(c, name=name) if name else c


def _net(name, what, widths, rows):
    c = dict(kind=what, widths=widths, rows=rows)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the driver's default run of a small linear-element mesh with walls (the hilltop example's
        # size): a step is a handful of short kernels
        _solver("hilltop_p1_fp64", 1, (60, 60), "fp64", 100, "mixed", 0.1),
        # the 2-D study at its real size: 4050 triangles of order 3, FP64
        _solver("square_p3_fp64", 3, (45, 45), "fp64", 100, "open", 0.1),
        # a 2-D run of order 4 in FP32 on an odd grid
        _solver("square_p4_fp32", 4, (101, 97), "fp32", 50, "mixed", 0.2),
        # a large 2-D domain of order 2, whose state is larger than the caches
        _solver("plane_p2_fp32", 2, (640, 480), "fp32", 50, "open", 0.3),
        # the 3-D cube: 196,608 tetrahedra of order 3, FP32
        _solver("cube_p3_fp32", 3, (32, 32, 32), "fp32", 50, "mixed", 0.0),
        # the same cube at a size a reference-precision (default) run uses
        _solver("cube_p3_fp64", 3, (17, 16, 15), "fp64", 20, "mixed", 0.1),
        # the 3-D study at scale: order 4, FP32, an eighth of the 2M-tetrahedron box
        _solver("box_p4_fp32", 4, (56, 28, 27), "fp32", 60, "open", 0.1),
        # a small 3-D FP64 run with ragged counts
        _solver("box_p2_fp64", 2, (13, 11, 9), "fp64", 50, "open", 0.1),
        # a parameter study: uneven 2-D instances of orders 2-4 advanced together
        dict(kind="ensemble", instances=48, emin=1000, emax=50000, steps=200, name="ensemble_fp32"),
        # one right-hand side for a caller that has its own time integrator (host arrays in and out)
        _solver("rhs_p3_fp64", 3, (12, 11, 13), "fp64", 1, "mixed", 0.1, "rhs"),
        # the surrogate answering one study's queries, and the gradient of one training batch
        _net("surrogate_forward", "forward", SURROGATE, 2000),
        _net("surrogate_gradient", "gradient", SURROGATE, 256),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["run"] * 7 + ["rhs", "ensemble", "forward", "forward", "gradient"])
    if kind == "forward":
        return _net(None, kind, rng.choice([SURROGATE, SURROGATE, ERROR_NET]), int(_log(rng, 1, 20000)))
    if kind == "gradient":
        return _net(None, kind, rng.choice([SURROGATE, SURROGATE, ERROR_NET]), int(_log(rng, 16, 2048)))
    if kind == "ensemble":
        return dict(kind=kind, instances=int(_log(rng, 2, 48)), emin=500, emax=int(_log(rng, 2000, 50000)),
                    steps=rng.choice([50, 100, 150]))
    dim, order, prec = rng.choice([2, 2, 3, 3]), rng.randint(1, 4), rng.choice(["fp32", "fp64"])
    npe = math.comb(order + dim, dim)
    nodes = _log(rng, 2000, 4e6 if prec == "fp32" else 6e5)
    cells = max(nodes / npe / (2 if dim == 2 else 6), 4)
    stretch = rng.uniform(0.7, 1.4)
    side = cells ** (1.0 / dim)
    counts = [max(2, round(side * stretch)), max(2, round(side / stretch))]
    if dim == 3:
        counts.append(max(2, round(side)))
    steps = 1 if kind == "rhs" else rng.choice([10, 25, 50])
    return _solver(None, order, tuple(counts), prec, steps, rng.choice(["open", "mixed"]),
                   rng.choice([0.0, 0.1, 0.2, 0.3]), kind)


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=3)
def _mesh(dim, order, nx, ny, nz, walls):
    """The mesh a user loads (the same for every seed): its arrays, its time step without flow, its
    monopole's and observers' node sets."""
    mg = _pkg().meshgen
    if dim == 2:
        # an nx x ny grid over [-5,5]^2: the project's square generator makes equal counts, the box of
        # cells is stretched to the same area per cell
        m = _rectangle(nx, ny, order)
        size, radius, half = 0.3, 0.4, 5.0
    else:
        m = mg.box(counts=(nx, ny, nz), order=order, jitter=0.2, seed=2, side_names=list(SIDES))
        size, radius, half = 0.15, 0.15, 1.0
    bc = {s: "Absorbing" for s in SIDES}
    if walls == "mixed":
        bc["xmin"] = bc["xmax"] = "Reflecting"
    mesh = dict(dim=dim, order=order, xyz=m["xyz"], elem_nodes=m["elem_nodes"], groups=mg.solver_groups(m, bc))
    x = torch.from_numpy(mesh["xyz"][mesh["elem_nodes"].reshape(-1)]).cuda()
    sets, weights = [], []
    for p in [(0.0, 0.0, 0.0, size)] + [(a * half, b * half, 0.1 * half if dim == 3 else 0.0, radius)
                                        for a, b in ((0.5, 0.45), (-0.5, 0.4), (-0.45, -0.5), (0.55, -0.4))]:
        d = (x - torch.tensor(p[:3], dtype=torch.float64, device="cuda")).norm(dim=1)
        r = max(p[3], 1.0001 * float(d.min()))  # at least the nearest node on a coarse mesh
        i = torch.nonzero(d < r)[:, 0]
        sets.append(i.cpu().numpy())
        weights.append((1.0 / (d[i] ** 2 + 1e-12)).cpu().numpy())
    return mesh, mg.min_altitude(mesh), sets, weights


def _rectangle(nx, ny, order):
    """[-5,5] x [-5,5] cut into nx x ny jittered rectangles of two triangles (meshgen's construction)."""
    mg = _pkg().meshgen
    rng = np.random.default_rng(1)
    hx, hy = 10.0 / nx, 10.0 / ny
    i, j = [a.reshape(-1) for a in np.meshgrid(np.arange(nx + 1), np.arange(ny + 1), indexing="xy")]
    ci = np.stack([i, j], 1).astype(np.int64)
    xyz = np.zeros((len(ci), 3))
    xyz[:, 0], xyz[:, 1] = -5.0 + hx * i, -5.0 + hy * j
    inner = (i > 0) & (i < nx) & (j > 0) & (j < ny)
    xyz[inner, :2] += rng.uniform(-0.2, 0.2, (inner.sum(), 2)) * (hx, hy)
    ii, jj = [a.reshape(-1) for a in np.meshgrid(np.arange(nx), np.arange(ny), indexing="xy")]
    v = lambda a, b: b * (nx + 1) + a  # noqa: E731
    a, b, c, d = v(ii, jj), v(ii + 1, jj), v(ii + 1, jj + 1), v(ii, jj + 1)
    elems = np.stack([np.stack([a, b, c], 1), np.stack([a, c, d], 1)], 1).reshape(-1, 3)
    return mg._build(2, ci, xyz, elems, order, [(k + 1, SIDES[k], ax, val) for k, (ax, val) in
                                                 enumerate([(0, 0), (0, nx), (1, 0), (1, ny)])])


def _flow(case):
    v = case["mach"] * C0
    return (v, 0.0, 0.0) if case["dim"] == 2 else (0.8 * v, 0.6 * v, 0.0)


def _acoustic_state(x, dim, seed):
    """[4][nodes] FP64 on the GPU: superposed plane waves of a few tenths of a pascal with their
    velocities v = k p / (rho0 c0), some of them resolved by a handful of elements only."""
    g = torch.Generator().manual_seed(int(seed) * 7919 + 13)
    half = 5.0 if dim == 2 else 1.0
    u = torch.zeros((4, x.shape[0]), dtype=torch.float64, device=x.device)
    for _ in range(4):
        k = torch.randn(3, generator=g, dtype=torch.float64)
        if dim == 2:
            k[2] = 0.0
        k = (k / k.norm()).to(x.device)
        num = float(2.0 + 8.0 * torch.rand((), generator=g, dtype=torch.float64)) / half
        amp = float(0.1 + 0.3 * torch.rand((), generator=g, dtype=torch.float64))
        ph = float(2 * math.pi * torch.rand((), generator=g, dtype=torch.float64))
        p = amp * torch.sin(num * (x @ k) + ph)
        u[0] += p
        u[1:] += k[:, None] * (p / (RHO0 * C0))
    return u


def _signal(case, seed, dt):
    """Monopole values of the steps of one pass."""
    f = 50.0 + 10.0 * (seed % 17)
    return 0.1 * np.sin(2 * np.pi * f * np.arange(case["steps"]) * dt + 0.1 * (seed % 11))[:, None]


def _nodes(mesh):
    return torch.from_numpy(mesh["xyz"][mesh["elem_nodes"].reshape(-1)]).cuda()


def _time_step(h, order, mach):
    return CFL * h / (C0 * (1.0 + mach) * (2 * order + 1))


@functools.lru_cache(maxsize=2)
def _instances(n, emin, emax):
    """The study's instances (the ensemble module's distributions, elements log-uniform in [emin, emax])."""
    ens = _pkg().ensemble
    rng = np.random.default_rng(4)
    out = []
    for _ in range(n):
        grid = int(np.ceil(np.sqrt(np.exp(rng.uniform(np.log(emin), np.log(emax))) / 2)))
        p = int(rng.integers(2, 5))
        mesh = ens.square_mesh(grid, p, int(rng.integers(1 << 30)))
        sx, sy = rng.uniform(-4, 4, 2)
        out.append(ens.instance(mesh, p, sx, sy, rng.uniform(20, 400), rng.uniform(0, 0.3), rng.uniform(0, 2 * np.pi)))
    return out


def _ensemble_state(inst, k, seed):
    return _acoustic_state(_nodes(inst["mesh"]), 2, seed * 101 + k)


def _network(case, seed):
    w = [int(v) for v in case["widths"].split(",")]
    g = torch.Generator().manual_seed(int(seed) * 31 + 7)
    parts = []
    for k, n in zip(w[:-1], w[1:]):
        parts += [torch.randn(n * k, generator=g) * math.sqrt(2.0 / k), 0.05 * torch.randn(n, generator=g)]
    # features are uniform in [-1, 1] (surrogate.features), targets log-spectra after standardising
    x = torch.rand((case["rows"], w[0]), generator=g) * 2 - 1
    t = torch.randn((case["rows"], w[-1]), generator=g)
    return w, torch.cat(parts), x, t


def prepare(case, seed):
    gpu = _pkg().gpu
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        w, params, x, t = _network(case, seed)
        net = gpu.Network(w)
        net.set_params(params.numpy())
        if kind == "gradient":
            return dict(kind=kind, net=net, x=x.numpy(), t=t.numpy())
        x = x.cuda()
        return dict(kind=kind, net=net, x=x, y=torch.empty((len(x), w[-1]), device="cuda"))
    if kind == "ensemble":
        insts = _instances(case["instances"], case["emin"], case["emax"])
        B = _pkg().ensemble.make_batch(insts, gpu.DG_FP32, case["steps"])
        for k, i in enumerate(insts):
            B.set_state(k, _ensemble_state(i, k, seed).cpu().numpy())
        return dict(kind=kind, B=B, steps=case["steps"])
    mesh, h, sets, weights = _mesh(case["dim"], case["order"], case["nx"], case["ny"], case["nz"], case["walls"])
    dt = _time_step(h, case["order"], case["mach"])
    S = gpu.Solver(mesh, v0=_flow(case), rho0=RHO0, c0=C0,
                   precision=gpu.DG_FP32 if case["precision"] == "fp32" else gpu.DG_FP64)
    u = gpu.pinned_empty((4, S.ndof))
    u[:] = _acoustic_state(_nodes(mesh), case["dim"], seed).cpu().numpy()
    if kind == "run":
        S.set_state(u)
        S.set_sources(sets[:1])
        S.set_source_values(_signal(case, seed, dt))
        S.set_observers(sets[1:], weights[1:])
    return dict(kind=kind, S=S, u=u, dt=dt, steps=case["steps"], fp32=case["precision"] == "fp32")


def run(state):
    kind = state["kind"]
    if kind == "forward":
        state["net"].forward_device(state["x"].data_ptr(), len(state["x"]), state["y"].data_ptr(),
                                    torch.cuda.current_stream().cuda_stream)
        return state["y"]
    if kind == "gradient":
        grad, loss = state["net"].gradient(state["x"], state["t"])
        return dict(grad=grad, loss=loss)
    if kind == "ensemble":
        B = state["B"]
        obs = B.run(state["steps"])
        u = torch.from_numpy(np.concatenate([B.get_state(k).reshape(-1) for k in range(B.n)])).float()
        return dict(obs=np.concatenate([o.reshape(-1) for o in obs]).astype(np.float32), u=u)
    S = state["S"]
    if kind == "rhs":
        k = S.rhs(state["u"], state["dt"])
        out = dict(p=k[0], v=k[1:])
        return {n: torch.from_numpy(a).float() for n, a in out.items()} if state["fp32"] else out
    S.step = 0
    S.snapshot()
    res, obs = S.run(state["steps"], state["dt"])
    u = S.get_state(out=state["u"])
    if state["fp32"]:
        u = torch.from_numpy(u).to("cuda", non_blocking=True).float()
        res, obs = res.astype(np.float32), obs.astype(np.float32)
    return dict(p=u[0], v=u[1:], residuals=res, obs=obs)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _dg_work(dim, order, elements, steps, word, stages=4):
    """Each stage depends on every neighbour's last one, so each reads its input and writes its results
    once: 18 state words per unknown and RK4 step (input, state, accumulator, snapshot), and the
    element's geometry. Operations: the fluxes of the nodes and of the face nodes and the update."""
    npe, nfp = math.comb(order + dim, dim), math.comb(order + dim - 1, dim - 1)
    nv, nf = dim + 1, dim + 1
    geo = (dim * dim + nf * (dim + 1)) * word + 2 * nf * 4
    words = 18 if stages == 4 else 2
    return dict(bytes=steps * elements * (words * npe * nv * word + stages * geo),
                flops=steps * stages * elements * nv * (npe * (4 * dim + 6) + nf * nfp * 10))


def work(case):
    kind = case["kind"]
    if kind in ("forward", "gradient"):
        w, n = [int(v) for v in case["widths"].split(",")], case["rows"]
        weights = sum(a * b for a, b in zip(w[:-1], w[1:]))
        if kind == "forward":
            return dict(bytes=4 * n * (w[0] + w[-1]) + 2 * weights + 4 * sum(w[1:]), flops=2 * n * weights)
        return dict(bytes=4 * n * (w[0] + w[-1]) + 6 * weights + 8 * sum(w[1:]), flops=6 * n * weights)
    if kind == "ensemble":
        t = [_dg_work(2, i["p"], len(i["mesh"]["elem_nodes"]), case["steps"], 4)
             for i in _instances(case["instances"], case["emin"], case["emax"])]
        return {k: sum(d[k] for d in t) for k in ("bytes", "flops")}
    e = 2 * case["nx"] * case["ny"] if case["dim"] == 2 else 6 * case["nx"] * case["ny"] * case["nz"]
    return _dg_work(case["dim"], case["order"], e, case["steps"], 4 if case["precision"] == "fp32" else 8,
                    1 if kind == "rhs" else 4)


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------

# local faces (element corners in order) and the leading face quadrature points that define the tangent
# frame of an absorbing face in 3-D (the reference's recipe)
FACES = {2: [(0, 1), (1, 2), (2, 0)], 3: [(0, 2, 1), (0, 1, 3), (0, 3, 2), (3, 1, 2)]}


def _head(order):
    if order == 3:
        a, b = 0.053145049844817, 0.310352451033784
        c = 1.0 - a - b
        return [(a, b, c), (b, c, a), (c, a, b)]
    a = {1: 1.0 / 6.0, 2: 0.445948490915965, 4: 0.050547228317031}[order]
    c = 1.0 - 2.0 * a
    return [(a, c, a), (c, a, a), (a, a, c)] if order == 4 else [(c, a, a), (a, c, a), (a, a, c)]


def _exponents(dim, p):
    if dim == 1:
        return [(i,) for i in range(p + 1)]
    return [(i,) + r for i in range(p + 1) for r in _exponents(dim - 1, p - i)]


def _simplex(dim, p, lattice):
    """Mass matrix over a simplex of measure 1 and the derivative matrices of the Lagrange basis on the
    lattice points (integer reference coordinates, p times)."""
    ex = _exponents(dim, p)
    pts = np.asarray(lattice, dtype=np.float64) / p
    V = np.array([[np.prod([x ** k for x, k in zip(pt, e)]) for e in ex] for pt in pts])
    fact = math.factorial
    M = np.array([[fact(dim) * np.prod([fact(a + b) for a, b in zip(e, f)], dtype=object)
                   / fact(sum(e) + sum(f) + dim) for f in ex] for e in ex], dtype=np.float64)
    Vi = np.linalg.inv(V)
    D = []
    for r in range(dim):
        dV = np.array([[e[r] * np.prod([x ** (k - (d == r)) if k - (d == r) >= 0 else 0.0
                                        for d, (x, k) in enumerate(zip(pt, e))]) for e in ex] for pt in pts])
        D.append(dV @ Vi)
    return Vi.T @ M @ Vi, D


class _DG:
    """The semi-discrete linearised Euler equations on a straight-sided mesh, FP64, dense operators."""

    def __init__(self, dim, order, xyz, en, groups, v0):
        dev, f8 = "cuda", torch.float64
        self.dim = dim
        E, npe = en.shape
        X = torch.from_numpy(xyz).to(dev)
        en = torch.from_numpy(en).to(dev)
        P = X[en[:, :dim + 1]][:, :, :dim]
        J = (P[:, 1:] - P[:, :1]).transpose(1, 2)  # dx/dxi
        self.G = torch.linalg.inv(J)               # dxi/dx
        lat0 = torch.linalg.solve(J[0], (X[en[0]][:, :dim] - P[0, 0]).T).T
        lat = np.rint(lat0.cpu().numpy() * order).astype(int)
        M, D = _simplex(dim, order, lat)
        Mi = np.linalg.inv(M)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.Dt = [t(Mi @ d.T @ M) for d in D]
        self.v0 = v0[:, :dim].to(dev) if v0.dim() == 2 else v0[:dim].to(dev).expand(E, dim)
        bary = np.concatenate([order - lat.sum(1, keepdims=True), lat], 1)
        grad = torch.cat([-self.G.sum(1, keepdim=True), self.G], 1)  # grad lambda_k
        gmask = torch.zeros(len(X), dtype=torch.int64, device=dev)
        for k, (_, nodes) in enumerate(groups):
            gmask[torch.from_numpy(np.asarray(nodes)).to(dev)] |= 1 << k
        # faces: node lists, corners for matching
        fnodes, keys, nv = [], [], len(X)
        self.lift, self.n, self.sj = [], [], []
        for f, fc in enumerate(FACES[dim]):
            opp = [k for k in range(dim + 1) if k not in fc][0]
            loc = [i for i in range(npe) if bary[i, opp] == 0]
            fl = np.stack([bary[loc][:, fc[k]] for k in range(1, dim)], 1)
            Mf, _ = _simplex(dim - 1, order, fl)
            E_f = np.zeros((npe, len(loc)))
            E_f[loc, np.arange(len(loc))] = 1.0
            self.lift.append(t(Mi @ E_f @ Mf))
            g = grad[:, opp]
            nrm = g.norm(dim=1)
            self.n.append(-g / nrm[:, None])
            self.sj.append(dim * nrm)  # |face| / |element|
            fnodes.append(torch.tensor(loc, device=dev))
            c = en[:, list(fc)].sort(dim=1).values
            key = c[:, 0]
            for k in range(1, dim):
                key = key * nv + c[:, k]
            keys.append(key)
        self.fnodes = fnodes
        nf = dim + 1
        key = torch.stack(keys, 1).reshape(-1)  # (element, face)
        order_k = torch.argsort(key, stable=True)
        ks = key[order_k]
        same = ks[1:] == ks[:-1]
        partner = torch.full_like(key, -1)
        a, b = order_k[:-1][same], order_k[1:][same]
        partner[a], partner[b] = b, a
        partner = partner.reshape(E, nf)
        allf = torch.stack([en[:, fn] for fn in fnodes], 1)           # [E][nf][nfp] mesh nodes
        slots = torch.stack([torch.arange(E, device=dev)[:, None] * npe + fn for fn in fnodes], 1)
        srt = torch.argsort(allf, dim=2)
        sorted_slots = torch.gather(slots, 2, srt).reshape(E * nf, -1)
        rank = torch.argsort(srt, dim=2)
        self.nbr, self.bnd = [], []
        for f, fc in enumerate(FACES[dim]):
            pf = partner[:, f]
            self.nbr.append(torch.where((pf >= 0)[:, None], torch.gather(sorted_slots[pf.clamp(min=0)], 1, rank[:, f]),
                                        slots[:, f]))
            be = torch.nonzero(pf < 0)[:, 0]
            m = gmask[en[be, fc[0]]]
            bc = torch.zeros(len(be), dtype=torch.int64, device=dev)
            for k, (code, _) in enumerate(groups):
                bc = torch.where((m >> k) & 1 == 1, torch.full_like(bc, code), bc)
            self.bnd.append((be, self._boundary(f, be, bc, P, fc, order)))
        self.E, self.npe = E, npe

    def _boundary(self, f, be, bc, P, fc, order):
        d, n, v0 = self.dim, self.n[f][be], self.v0[be]
        vn = (v0 * n).sum(1)
        eye = torch.eye(d, dtype=torch.float64, device=n.device)
        nn = n[:, :, None] * n[:, None, :]
        W = torch.zeros((len(be), d + 1, d + 1), dtype=torch.float64, device=n.device)  # wall
        W[:, 0, 0] = vn
        W[:, 1:, 0] = n / RHO0
        W[:, 1:, 1:] = vn[:, None, None] * (eye - nn)
        if d == 2:
            tt = eye - nn
        else:
            x0, x1, x2 = (P[be, k] for k in fc)
            q = [h[0] * x0 + h[1] * x1 + h[2] * x2 for h in _head(order)]
            a, b = q[1] - q[0], q[2] - q[0]
            h = a.norm(dim=1)
            i = (a * b).sum(1) / h
            j = ((b * b).sum(1) - i * i).clamp(min=0).sqrt()
            s = -(i.abs()[:, None] * a - h[:, None] * b) / (h * j)[:, None]
            tv, sv = a / h[:, None], s / s.norm(dim=1, keepdim=True)
            tt = tv[:, :, None] * tv[:, None, :] + sv[:, :, None] * sv[:, None, :]
        cv = C0 + vn
        lam = torch.where(vn < 0, 0.0, -1.0).to(torch.float64)
        A = torch.zeros_like(W)  # non-reflecting
        A[:, 0, 0] = 0.25 * cv
        A[:, 0, 1:] = 0.25 * C0 * RHO0 * cv[:, None] * n
        A[:, 1:, 0] = 0.25 * n * (cv / (RHO0 * C0))[:, None]
        A[:, 1:, 1:] = 0.25 * (cv[:, None, None] * nn - (vn * lam)[:, None, None] * tt)
        return torch.where((bc == 1)[:, None, None], W, A)

    def rhs(self, u):
        """L(u) of u [d+1][E][npe]."""
        d, rc2 = self.dim, RHO0 * C0 * C0
        out = torch.zeros_like(u)
        for r in range(d):
            g = self.G[:, r, :]
            gv0 = (g * self.v0).sum(1)[:, None]
            F = torch.empty_like(u)
            F[0] = gv0 * u[0] + rc2 * sum(g[:, k, None] * u[1 + k] for k in range(d))
            for k in range(d):
                F[1 + k] = gv0 * u[1 + k] + g[:, k, None] / RHO0 * u[0]
            out += F @ self.Dt[r].T
        flat = u.reshape(d + 1, -1)
        for f in range(d + 1):
            um, up = u[:, :, self.fnodes[f]], flat[:, self.nbr[f]]
            n, a, j = self.n[f], 0.5 * (um + up), 0.5 * C0 * (um - up)
            vn0 = (n * self.v0).sum(1)[:, None]
            h = vn0 * a + j
            h[0] += rc2 * sum(n[:, k, None] * a[1 + k] for k in range(d))
            for k in range(d):
                h[1 + k] += n[:, k, None] / RHO0 * a[0]
            be, B = self.bnd[f]
            h[:, be] = torch.einsum("eij,jen->ien", B, um[:, be])
            out -= (self.sj[f][:, None] * h) @ self.lift[f].T
        return out


def _march(dg, u, dt, steps, inject, observe):
    """RK4 steps of u [d+1][E][npe]; inject(u, step) overwrites the sources, observe(u, step) samples."""
    for s in range(steps):
        inject(u, s)
        k1 = dt * dg.rhs(u)
        k2 = dt * dg.rhs(u + 0.5 * k1)
        k3 = dt * dg.rhs(u + 0.5 * k2)
        k4 = dt * dg.rhs(u + k3)
        u = u + (k1 + 2 * k2 + 2 * k3 + k4) / 6
        observe(u, s)
    return u


def _idw(u, sets, weights):
    """[observers][4] weighted means."""
    flat = u.reshape(u.shape[0], -1)
    rows = []
    for i, w in zip(sets, weights):
        r = torch.zeros(4, dtype=torch.float64, device=u.device)
        r[:u.shape[0]] = (flat[:, i] * w).sum(1) / w.sum()
        rows.append(r)
    return torch.stack(rows)


def _exact_run(case, seed):
    mesh, h, sets, weights = _mesh(case["dim"], case["order"], case["nx"], case["ny"], case["nz"], case["walls"])
    d = case["dim"]
    dt = _time_step(h, case["order"], case["mach"])
    dg = _DG(d, case["order"], mesh["xyz"], mesh["elem_nodes"], mesh["groups"],
             torch.tensor(_flow(case), dtype=torch.float64))
    u = _acoustic_state(_nodes(mesh), d, seed)[:d + 1].reshape(d + 1, dg.E, dg.npe)
    pad = lambda a: torch.cat([a.reshape(d + 1, -1), torch.zeros((3 - d, a[0].numel()), dtype=a.dtype, device=a.device)])  # noqa: E731
    if case["kind"] == "rhs":
        k = pad(dt * dg.rhs(u))
        return dict(p=k[0], v=k[1:])
    dev = u.device
    sets = [torch.from_numpy(s).to(dev) for s in sets]
    weights = [torch.from_numpy(w).to(dev) for w in weights]
    val = _signal(case, seed, dt)[:, 0]
    snap, res, obs = u.clone(), [], []

    def inject(a, s):
        a[0].view(-1)[sets[0]] = float(val[s])

    def observe(a, s):
        r = torch.zeros(5, dtype=torch.float64, device=dev)
        m = ((snap - a) ** 2).reshape(d + 1, -1).mean(1)
        r[0], r[1], r[2:2 + d] = m[0], m[0] / C0 ** 4, m[1:]
        res.append(r)
        obs.append(_idw(a, sets[1:], weights[1:]))

    u = pad(_march(dg, u, dt, case["steps"], inject, observe))
    return dict(p=u[0], v=u[1:], residuals=torch.stack(res), obs=torch.stack(obs))


def _exact_ensemble(case, seed):
    """The instances of one order as one mesh of their elements, each with its own flow and time step."""
    insts = _instances(case["instances"], case["emin"], case["emax"])
    ens, steps = _pkg().ensemble, case["steps"]
    states, traces = [None] * len(insts), [None] * len(insts)
    for p in sorted({i["p"] for i in insts}):
        mine = [k for k, i in enumerate(insts) if i["p"] == p]
        xyz, en, nodes, v0, dts, u, ssets, svals, osets, ows = [], [], [], [], [], [], [], [], [], []
        noff = eoff = 0
        for k in mine:
            i = insts[k]
            m = i["mesh"]
            xyz.append(m["xyz"])
            en.append(m["elem_nodes"] + noff)
            nodes.append(np.asarray(m["groups"][0][1]) + noff)
            ne, npe = m["elem_nodes"].shape
            v0.append(torch.tensor(i["v0"], dtype=torch.float64).expand(ne, 3))
            dts.append(torch.full((ne, 1), i["dt"], dtype=torch.float64))
            u.append(_ensemble_state(i, k, seed)[:3].reshape(3, ne, npe))
            sd, od, ow = ens.node_sets(m, i["src"], i["obs"])
            ssets.append(torch.from_numpy(sd[0] + eoff * npe).cuda())
            svals.append(i["src"][4] * np.sin(2 * np.pi * i["src"][5] * np.arange(steps + 1) * i["dt"] + i["src"][6]))
            osets += [torch.from_numpy(o + eoff * npe).cuda() for o in od]
            ows += [torch.from_numpy(w).cuda() for w in ow]
            noff += len(m["xyz"])
            eoff += ne
        dg = _DG(2, p, np.concatenate(xyz), np.concatenate(en), [(0, np.concatenate(nodes))], torch.cat(v0))
        obs = []

        # one index list, one value per step and node, one weight matrix for all instances
        src = torch.cat(ssets)
        vals = torch.from_numpy(np.stack(svals, 1)).cuda()
        which = torch.cat([torch.full((len(s),), n, device="cuda") for n, s in enumerate(ssets)])
        oi, ow = torch.cat(osets), torch.cat(ows)
        oo = torch.cat([torch.full((len(o),), n, device="cuda") for n, o in enumerate(osets)])
        wsum = torch.zeros(len(osets), dtype=torch.float64, device="cuda").index_add_(0, oo, ow)

        def inject(a, s):
            a[0].view(-1)[src] = vals[s][which]

        def observe(a, s):
            r = torch.zeros((len(osets), 4), dtype=torch.float64, device="cuda")
            r[:, :3].index_add_(0, oo, (a.reshape(3, -1)[:, oi] * ow).T)
            obs.append(r / wsum[:, None])

        out = _march(dg, torch.cat(u, 1), torch.cat(dts).cuda(), steps, inject, observe)
        obs = torch.stack(obs)  # [steps][observers][4]
        e = o = 0
        for k in mine:
            ne, no = len(insts[k]["mesh"]["elem_nodes"]), len(insts[k]["obs"])
            s = out[:, e:e + ne].reshape(3, -1)
            states[k] = torch.cat([s, torch.zeros_like(s[:1])]).reshape(-1)
            traces[k] = obs[:, o:o + no].reshape(-1)
            e, o = e + ne, o + no
    return dict(obs=torch.cat(traces), u=torch.cat(states))


def _exact_network(case, seed):
    w, params, x, t = _network(case, seed)
    params = params.cuda().double().requires_grad_()
    x, t = x.cuda().double(), t.cuda().double()
    layers, pos = [], 0
    for k, n in zip(w[:-1], w[1:]):
        W = params[pos:pos + n * k].reshape(n, k)
        # the weights enter rounded to BF16, the gradient is taken at the rounded values
        W = W + (W.detach().float().bfloat16().double() - W.detach())
        layers.append((W, params[pos + n * k:pos + n * k + n]))
        pos += n * k + n
    a = x
    for li, (W, b) in enumerate(layers):
        a = a @ W.T + b
        if li < len(layers) - 1:
            a = 0.5 * a * (1 + torch.erf(a / math.sqrt(2.0)))
    if case["kind"] == "forward":
        return a.detach()
    loss = ((a - t) ** 2).mean()
    loss.backward()
    return dict(grad=params.grad, loss=float(loss))


def exact(case, seed):
    if case["kind"] in ("forward", "gradient"):
        return _exact_network(case, seed)
    if case["kind"] == "ensemble":
        return _exact_ensemble(case, seed)
    return _exact_run(case, seed)
