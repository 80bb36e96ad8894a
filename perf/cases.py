"""Measured workloads of the package: what its users run, over the range of
sizes they run it at.

Kinds of case
  step      the RK4 free-surface step (four Laplace solves), driven as a host
            program drives it between outputs: put E and P, advance `steps`
            steps, read E, P and W back
  solve     the drop-in Laplace solve on host arrays (iterative_solution)
  residual  rhs - A(eta) phi and its norm on the caller's device arrays
  batch     several independent simulations advanced together from one host
            thread (the serving loop's call)

Inputs are synthetic and seeded. Every simulation keeps its handle (grid,
multigrid hierarchy, workspace) between passes, as a time loop does.
"""
import ctypes
import importlib
import math
import random

import numpy as np
import torch

ow = importlib.import_module("oceanwave3d-fortran90_b200")
G = 9.81
DEV = "cuda"


# ------------------------------------------------------------------ cases
def listed():
    return [
        # one nonlinear wavelength, periodic: the smallest grid in use, all latency
        dict(name="flume_periodic_65x9", kind="step", basin="periodic", Nx=65, Ny=1, Nz=9,
             precision="fp64", krylov="fgmres", steps=10),
        # 2-D wave flume with a generation zone and a sponge
        dict(name="flume_zones_513x9", kind="step", basin="zones", Nx=513, Ny=1, Nz=9,
             precision="fp64", krylov="fgmres", steps=4),
        # 2-D flume over a slope, in the reference's solver form (left GMRES); not a power of two
        dict(name="flume_slope_385x9", kind="step", basin="slope", Nx=385, Ny=1, Nz=9,
             precision="fp64", krylov="lgmres", steps=4),
        # small 3-D basin of a ragged size
        dict(name="sea_97x49x9", kind="step", basin="sea", Nx=97, Ny=49, Nz=9,
             precision="fp64", krylov="fgmres", steps=2),
        # the shoal experiment: sloping bottom, generation zone and sponge
        dict(name="shoal_257x33x9", kind="step", basin="shoal", Nx=257, Ny=33, Nz=9,
             precision="fp64", krylov="fgmres", steps=1),
        # a finer shoal in mixed precision
        dict(name="shoal_513x65x9_mixed", kind="step", basin="shoal", Nx=513, Ny=65, Nz=9,
             precision="mixed", krylov="fgmres", steps=1),
        # the irregular sea the benchmark runs, in both precisions
        dict(name="sea_1025x257x17_mixed", kind="step", basin="sea", Nx=1025, Ny=257, Nz=17,
             precision="mixed", krylov="fgmres", steps=1),
        dict(name="sea_1025x257x17_fp64", kind="step", basin="sea", Nx=1025, Ny=257, Nz=17,
             precision="fp64", krylov="fgmres", steps=1),
        # the largest instance
        dict(name="sea_2049x513x9_mixed", kind="step", basin="sea", Nx=2049, Ny=513, Nz=9,
             precision="mixed", krylov="fgmres", steps=1),
        # the drop-in solve called by a host program, reference solver form
        dict(name="solve_257x65x13", kind="solve", basin="bumps", Nx=257, Ny=65, Nz=13,
             precision="fp64", krylov="lgmres"),
        # the operator on a host program's own device arrays
        dict(name="residual_1025x257x17", kind="residual", basin="bumps", Nx=1025, Ny=257, Nz=17,
             precision="fp64", krylov="fgmres"),
        # the serving loop's mix of small and middling simulations
        dict(name="batch_6_mixed", kind="batch", mix=3, count=6, steps=2),
    ]


def _coarsens(nx, ny, nz):
    """Whether the reference's coarsening rule (standard strategy) can halve this grid all the way."""
    levels = int(math.floor(math.log2(max(nx, ny, nz) - 1) + 0.5))
    for _ in range(levels - 1):
        if ny == 1:
            xc, yc, zc = 1, 0, int(nx == nz)
        elif nx == ny == nz:
            xc = yc = zc = 1
        else:
            xc, yc, zc = int(nx > nz), int(ny > nz), int(nx < nz and ny < nz)
        if (xc and nx % 2 == 0) or (yc and ny % 2 == 0) or (zc and (nz - 1) // 2 % 2 == 1):
            return False
        nx, ny, nz = [(n - 1) // 2 + 1 if c else n for n, c in ((nx, xc), (ny, yc), (nz, zc))]
        if min(nx, nz) < 2 or (ny > 1 and ny < 2):
            return False
    return (nx + 2) * (ny + 2 if ny > 1 else 1) * (nz + 1) <= 1500


def draw(rng):
    """A case of the same kinds; sizes over the log of the range, ragged ones (3, 5, 7 times a power of two) among them."""
    while True:
        kind = rng.choice(["step", "step", "step", "step", "step", "solve", "residual", "batch"])
        if kind == "batch":
            return dict(kind="batch", mix=rng.randrange(10, 100000), count=rng.randrange(2, 7), steps=rng.randrange(1, 4))
        precision = rng.choice(["fp64", "fp64", "mixed"])
        krylov = rng.choice(["fgmres", "fgmres", "lgmres"]) if precision == "fp64" else "fgmres"
        nz = rng.choice([9, 9, 13, 17])
        nx = rng.choice([1, 1, 3, 5, 7]) * 2 ** rng.randrange(5, 11) + 1
        flume = rng.random() < 0.35 and kind != "residual"
        ny = 1 if flume else rng.choice([1, 1, 3, 5]) * 2 ** rng.randrange(3, 9) + 1
        if not 33 <= nx <= 2049 or ny > nx or nx * ny * nz > 4_500_000:
            continue
        if flume:
            basin = rng.choice(["zones", "slope", "slope", "periodic"]) if kind == "step" else "bumps"
            if basin in ("zones", "periodic") and nx not in (65, 129, 257, 513, 1025):
                continue
            if basin == "periodic" and nx > 257:
                continue
        else:
            if ny < 9 or not _coarsens(nx, ny, nz):
                continue
            basin = rng.choice(["sea", "shoal", "bumps"]) if kind == "step" else "bumps"
        c = dict(kind=kind, basin=basin, Nx=nx, Ny=ny, Nz=nz, precision=precision, krylov=krylov)
        if kind == "step":
            c["steps"] = rng.randrange(1, 5) if nx * ny * nz < 200_000 else 1
        return c


# ----------------------------------------------------------------- inputs
def _sea(x, y, h, Hs, Tp, seed, nfreq=48, ndir=9):
    """Linear directional JONSWAP sea (eta, surface potential) on the grid, from the seed's phases."""
    rng = np.random.default_rng(seed)
    fp = 1.0 / Tp
    f = np.linspace(0.5 * fp, 3.0 * fp, nfreq)
    S = ow.workloads.jonswap(f, Hs, Tp)
    om = 2 * np.pi * f
    k = ow.workloads.dispersion_k(om, h)
    if len(y) == 1:
        th, D = np.zeros(1), np.ones(1)
    else:
        th = np.linspace(-np.pi / 2, np.pi / 2, ndir + 2)[1:-1]
        D = np.cos(th) ** 2
        D = D / D.sum()
    amp = np.sqrt(2 * S[:, None] * (f[1] - f[0]) * D[None, :])
    ph = rng.uniform(0, 2 * np.pi, size=amp.shape)
    X = torch.tensor(x, device=DEV)[None, :]
    Y = torch.tensor(y, device=DEV)[:, None]
    eta = torch.zeros((len(y), len(x)), dtype=torch.float64, device=DEV)
    phis = torch.zeros_like(eta)
    for a in range(nfreq):
        for b in range(len(th)):
            arg = k[a] * (math.cos(th[b]) * X + math.sin(th[b]) * Y) + ph[a, b]
            eta += amp[a, b] * torch.cos(arg)
            phis += amp[a, b] * G / om[a] * torch.sin(arg)
    return eta.cpu().numpy().ravel(), phis.cpu().numpy().ravel()


def _options(case):
    return dict(precision=ow.capi.PREC_MIXED if case["precision"] == "mixed" else ow.capi.PREC_FP64,
                krylov=ow.capi.KRYLOV_LGMRES if case["krylov"] == "lgmres" else ow.capi.KRYLOV_FGMRES,
                reltol=1e-8, abstol=1e-6)


def _basin(case, seed):
    """Parameters, geometry, initial E and P and the relaxation targets {zone: (mode, nt, dt, eta, phis)} of a case."""
    nx, ny, nz, kw = case["Nx"], case["Ny"], case["Nz"], _options(case)
    rng = np.random.default_rng(seed)
    targets = {}
    if case["basin"] == "periodic":
        p, geo, E, P, _ = ow.workloads.periodic_wave_2d(Nx=nx, Nz=nz, steepness=float(rng.uniform(0.4, 0.5)), **kw)
        # the wave at another phase: a cyclic shift over the distinct points
        s = int(rng.integers(0, nx - 1))
        idx = 1 + (np.arange(E.size) - 1 + s) % (nx - 1)
        E, P = E[idx], P[idx]
    elif case["basin"] == "zones":
        # 8 waves; generation over the first, sponge over the last three
        p, geo, E, P, targets = ow.workloads.stream_function_2d(n_waves=8, ppw=(nx - 1) // 8, Nz=nz, steps=20,
                                                               steepness=float(rng.uniform(0.3, 0.5)), **kw)
    elif case["basin"] == "slope":
        # smooth rise from 1 m to 0.6 m, a random sea in it; multigrid grids as the halving allows
        grids = 1
        n = nx
        while (n - 1) % 2 == 0 and n > 13:
            n, grids = (n - 1) // 2 + 1, grids + 1
        p = ow.default_params(Nx=nx, Ny=1, Nz=nz, Lx=0.1 * (nx - 1), Ly=1.0, Lz=1.0, GridZ=1, MGmaxgrids=grids, **kw)
        x, y = ow.workloads.grid_xy(p)
        a, xm = 3.0 / p.Lx, 0.5 * p.Lx
        t = np.tanh(a * (x - xm))
        geo = dict(h=0.8 - 0.2 * t, hx=-0.2 * a * (1 - t ** 2), hxx=0.4 * a * a * t * (1 - t ** 2))
        p.dt = 0.5 * 0.1 / math.sqrt(G)
        E, P = _sea(x, y, 0.8, 0.02, 1.5, seed)
    elif case["basin"] == "shoal":
        zones = [dict(x1=0.0, x2=3.0, y1=0.0, y2=6.0, ftype=-10, param=3.5, wavegen=1),
                 dict(x1=30.0, x2=35.0, y1=0.0, y2=6.0, ftype=9, param=3.5)]
        p, geo = ow.workloads.shoal(Nx=nx, Ny=ny, Nz=nz, relaxONOFF=1, relaxNo=2, relaxTransientTime=1.0, zones=zones, **kw)
        x, y = ow.workloads.grid_xy(p)
        E, P = _sea(x, y, 0.45, 0.01, 1.2, seed)
        targets = {0: None}
    else:
        dx = 0.05 if case["basin"] == "sea" else 0.1
        p = ow.default_params(Nx=nx, Ny=ny, Nz=nz, Lx=(nx - 1) * dx, Ly=(ny - 1) * dx if ny > 1 else 1.0, Lz=1.0, GridZ=1, **kw)
        if ny == 1:
            n, grids = nx, 1
            while (n - 1) % 2 == 0 and n > 13:
                n, grids = (n - 1) // 2 + 1, grids + 1
            p.MGmaxgrids = grids
        x, y = ow.workloads.grid_xy(p)
        if case["basin"] == "sea":      # flat, 1 m deep
            geo, h0, Hs = dict(h=np.full(len(x) * len(y), 1.0)), 1.0, 0.05
        else:                           # plane slope with three bumps
            geo = ow.serving.bathymetry(p, seed)
            h0, Hs = float(geo["h"].mean()), 0.02
        p.dt = 0.5 * dx / math.sqrt(G * float(geo["h"].max()))
        E, P = _sea(x, y, h0, Hs, 1.5, seed)
    p.g = G
    return p, geo, E, P, targets


def _regular_target(p, box, seed, nt=512):
    """A linear regular wave (T = 1 s, H = 1 cm, 0.45 m depth) over a generation zone, every half step."""
    i0, i1, j0, j1 = box
    x, _ = ow.workloads.grid_xy(p)
    xs, om = x[i0 - 1:i1], 2 * np.pi
    k = float(ow.workloads.dispersion_k(om, 0.45))
    ph = np.random.default_rng(seed).uniform(0, 2 * np.pi)
    a = k * xs[None, :] - om * (np.arange(nt) * 0.5 * p.dt)[:, None] + ph
    rows = j1 - j0 + 1
    return 0, nt, 0.5 * p.dt, np.tile(0.005 * np.cos(a), (1, rows)), np.tile(0.005 * G / om * np.sin(a), (1, rows))


class _Sim:
    """A simulation a host program keeps, with the host arrays it exchanges."""

    def __init__(self, case, seed):
        p, geo, self.E, self.P, targets = _basin(case, seed)
        self.sim = ow.Simulation(p, **geo)
        for z, t in targets.items():
            self.sim.set_relax_target(z, *(t or _regular_target(p, self.sim.zone_box(z), seed)))
        self.sim.set_state(self.E, self.P)
        self.out = [np.zeros(self.sim.C) for _ in range(3)]


def _read_surface(sim, out):
    E, P, W = out
    t = ctypes.c_double()
    d = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in out]
    st = ow.lib().ow3d_get_state(sim.h, *d, None, ctypes.byref(t))
    if st < 0:
        raise ow.OW3DError(st, "ow3d_get_state")
    return {"E": E, "P": P, "W": W}


def _surface_fields(case, seed, p):
    """A seeded sea's surface with its horizontal derivatives, as a host program hands them over (E, Ex, Exx, Ey, Eyy), and its P."""
    x, y = ow.workloads.grid_xy(p)
    E, P = _sea(x, y, 0.7, 0.02, 1.5, seed + 7)
    E2 = E.reshape(len(y), len(x))
    Ex = np.gradient(E2, x, axis=1)
    Exx = np.gradient(Ex, x, axis=1)
    Ey = np.gradient(E2, y, axis=0) if len(y) > 1 else np.zeros_like(E2)
    Eyy = np.gradient(Ey, y, axis=0) if len(y) > 1 else np.zeros_like(E2)
    return [a.ravel().copy() for a in (E2, Ex, Exx, Ey, Eyy)], P


def _rhs(p, P):
    """Right-hand side of a stage's solve: P in the free-surface rows of the interior columns, zero elsewhere."""
    nxg, nyg, nzg = ow.dims(p)
    gy = 1 if p.Ny > 1 else 0
    r = np.zeros((nyg, nxg, nzg))
    r[gy:nyg - gy, 1:nxg - 1, -1] = P.reshape(nyg, nxg)[gy:nyg - gy, 1:nxg - 1]
    return r.ravel()


def _first_guess(p, P, seed):
    """An initial guess near the solution: the potential's decay with depth, 2 % off."""
    nxg, nyg, nzg = ow.dims(p)
    sg = np.sin(np.pi * np.arange(-1, p.Nz) / (2 * (p.Nz - 1)))
    k = 1.8
    prof = np.cosh(k * np.abs(sg)) / np.cosh(k)
    eps = 1.0 + 0.02 * np.random.default_rng(seed).standard_normal(nxg * nyg)
    return ((P * eps)[:, None] * prof[None, :]).ravel()


def _batch_requests(case, seed):
    r = random.Random(case["mix"])
    out = []
    for q in range(case["count"]):
        out.append(ow.serving.Request(rid=q, arrival=0.0, Nx=r.choice((65, 129, 257)), Ny=r.choice((1, 33, 65)),
                                      Nz=r.choice((9, 13, 17)), steps=case["steps"], seed=int(seed) * 64 + q))
    return out


def prepare(case, seed):
    if case["kind"] == "step":
        s = _Sim(case, seed)
        return dict(kind="step", s=s, steps=case["steps"])
    if case["kind"] == "batch":
        backend = ow.serving.DeviceBackend(ow, coarse_cluster=True)
        sims, surf = [], []
        for req in _batch_requests(case, seed):
            sim = backend.create(req)
            _, _, E, P = ow.serving.request_case(req)
            sims.append(sim)
            surf.append((E, P, [np.zeros(sim.C) for _ in range(3)]))
        return dict(kind="batch", backend=backend, sims=sims, surf=surf, steps=case["steps"])
    p, geo, _, _, _ = _basin(case, seed)
    sim = ow.Simulation(p, **geo)
    surf, P = _surface_fields(case, seed, p)
    if case["kind"] == "solve":
        return dict(kind="solve", sim=sim, rhs=_rhs(p, P), phi0=_first_guess(p, P, seed), surf=surf)
    dev = [torch.tensor(a, device=DEV) for a in (_rhs(p, P), _first_guess(p, P, seed), *surf)]
    return dict(kind="residual", sim=sim, dev=dev, res=torch.empty_like(dev[0]))


# -------------------------------------------------------------------- run
def run(state):
    if state["kind"] == "step":
        s = state["s"]
        s.sim.put_surface(s.E, s.P)
        s.sim.step(state["steps"])
        return _read_surface(s.sim, s.out)
    if state["kind"] == "batch":
        for sim, (E, P, _) in zip(state["sims"], state["surf"]):
            sim.put_surface(E, P)
        status, _ = state["backend"].step_batch(state["sims"], [state["steps"]] * len(state["sims"]))
        if min(status) < 0:
            raise ow.OW3DError(min(status), "step_batch")
        return [_read_surface(sim, out) for sim, (_, _, out) in zip(state["sims"], state["surf"])]
    if state["kind"] == "solve":
        phi, it, st = state["sim"].solve(state["rhs"], state["phi0"], *state["surf"])
        return {"phi": phi}
    norm = ctypes.c_double()
    st = ow.lib().ow3d_residual_device_noalloc(state["sim"].h, *[t.data_ptr() for t in state["dev"]],
                                               state["res"].data_ptr(), ctypes.byref(norm))
    if st < 0:
        raise ow.OW3DError(st, "ow3d_residual_device_noalloc")
    return {"residual": state["res"], "norm": norm.value}


# ------------------------------------------------------------------- work
def work(case):
    """Each input read once and each output written once per pass; for the solves, the fields every Laplace solve must
    touch at least once (right-hand side, guess, solution and the surface) and the operator's sums once per unknown."""
    if case["kind"] == "batch":
        b = f = 0.0
        for q in _batch_requests(case, 0):
            w = work(dict(kind="step", Nx=q.Nx, Ny=q.Ny, Nz=q.Nz, steps=q.steps))
            b, f = b + w["bytes"], f + w["flops"]
        return dict(bytes=b, flops=f)
    C = (case["Nx"] + 2) * (case["Ny"] + 2 if case["Ny"] > 1 else 1)
    N = C * (case["Nz"] + 1)
    once = 8.0 * (3 * N + 10 * C)
    flops = 2.0 * 66 * N
    if case["kind"] != "step":
        return dict(bytes=once, flops=flops)
    return dict(bytes=case["steps"] * (4 * once + 8.0 * 30 * C), flops=case["steps"] * 4 * flops)


# ------------------------------------------------------------------ exact
def _window(n, i):
    return min(max(i - 3, 0), n - 7)


def _stencil(nodes, at, order):
    """Weights of the `order`-th derivative at `at` on the nodes (Vandermonde system in scaled offsets)."""
    d = np.asarray(nodes) - at
    s = np.max(np.abs(d))
    V = np.vander(d / s, len(d), increasing=True).T
    b = np.zeros(len(d))
    b[order] = math.factorial(order)
    return np.linalg.solve(V, b) / s ** order


class _Operator:
    """A(eta) phi and the 1-D derivative matrices, in torch FP64, for basins with walls."""

    def __init__(self, p, geo):
        self.nxg, self.nyg, self.nzg = ow.dims(p)
        self.three = p.Ny > 1
        x, y = ow.workloads.grid_xy(p)
        z = np.concatenate([[0.0], np.sin(np.pi * np.arange(p.Nz) / (2 * (p.Nz - 1)))])
        zn = z.copy()
        zn[0] = -z[2]
        self.sig = torch.tensor(z, device=DEV)
        self.X = [self._rows(x, o) for o in (1, 2)]
        self.Xb = self._rows(x, 1, bottom=True)
        if self.three:
            self.Y = [self._rows(y, o) for o in (1, 2)]
            self.Yb = self._rows(y, 1, bottom=True)
        self.Z = [self._rows(zn, o) for o in (1, 2)]
        shape = (self.nyg, self.nxg)
        zero = np.zeros(shape)
        self.geo = {k: torch.tensor(np.asarray(geo[k]).reshape(shape) if k in geo and geo[k] is not None else zero, device=DEV)
                    for k in ("h", "hx", "hxx", "hy", "hyy")}

    @staticmethod
    def _rows(c, order, bottom=False):
        """First node and seven weights of each position; `bottom`: windows that stay off the two ghost ends."""
        n = len(c)
        start, w = np.zeros(n, dtype=np.int64), np.zeros((n, 7))
        for i in range(n):
            s = _window(n, i)
            if bottom:
                s = s + 1 if s == 0 else (s - 1 if s + 7 == n else s)
            start[i], w[i] = s, _stencil(c[s:s + 7], c[i], order)
        return torch.tensor(start, device=DEV), torch.tensor(w, device=DEV)

    @staticmethod
    def _along(rows, f, dim):
        start, w = rows
        out = None
        for m in range(7):
            shape = [1] * f.dim()
            shape[dim] = -1
            t = f.index_select(dim, start + m) * w[:, m].reshape(shape)
            out = t if out is None else out + t
        return out

    def apply(self, phi, surf):
        """phi (..., Nyg, Nxg, Nzg); surf: E, Ex, Exx, Ey, Eyy as (Nyg, Nxg)."""
        g, (E, Ex, Exx, Ey, Eyy) = self.geo, surf
        nd = phi.dim()
        X, Y, Z = nd - 2, nd - 3, nd - 1
        px, pxx = self._along(self.X[0], phi, X), self._along(self.X[1], phi, X)
        pz, pzz = self._along(self.Z[0], phi, Z), self._along(self.Z[1], phi, Z)
        tx = px.clone()
        tx[..., 0] = self._along(self.Xb, phi[..., 0], X)
        d = g["h"] + E
        i = 1.0 / d
        om = self.sig
        s2 = (g["hx"] * i)[..., None] - om * ((g["hx"] + Ex) * i)[..., None]
        s4 = (g["hy"] * i)[..., None] - om * ((g["hy"] + Ey) * i)[..., None]
        P1 = -2 * (g["hx"] ** 2 + g["hy"] ** 2) * i * i + (g["hxx"] + g["hyy"]) * i
        P2 = 2 * (Ex * g["hx"] + Ey * g["hy"]) * i * i
        P3 = 2 * (Ex * Ex + Ey * Ey) * i * i - (Exx + Eyy) * i
        s3 = (P1 - P2)[..., None] + om * (P3 + 2 * P2 - P1)[..., None]
        cz = s2 * s2 + s4 * s4 + (i * i)[..., None]
        r = pxx + s3 * pz + 2 * s2 * self._along(self.Z[0], tx, Z) + cz * pzz
        bot = (i + g["hx"] * s2[..., 1] + g["hy"] * s4[..., 1]) * pz[..., 1] + g["hx"] * px[..., 1]
        py = None
        if self.three:
            py, pyy = self._along(self.Y[0], phi, Y), self._along(self.Y[1], phi, Y)
            ty = py.clone()
            ty[..., 0] = self._along(self.Yb, phi[..., 0], Y)
            r = r + pyy + 2 * s4 * self._along(self.Z[0], ty, Z)
            bot = bot + g["hy"] * py[..., 1]
        r[..., 0] = bot
        r[..., -1] = phi[..., -1]
        r[..., :, 0, 1:], r[..., :, -1, 1:] = px[..., :, 1, 1:], px[..., :, -2, 1:]
        r[..., :, 0, 0], r[..., :, -1, 0] = phi[..., :, 0, 0], phi[..., :, -1, 0]
        if self.three:
            for jg, ja in ((0, 1), (-1, -2)):
                r[..., jg, 1:-1, 1:] = py[..., ja, 1:-1, 1:]
                r[..., jg, 1:-1, 0] = phi[..., jg, 1:-1, 0]
                r[..., jg, 0, :], r[..., jg, -1, :] = phi[..., jg, 0, :], phi[..., jg, -1, :]
        return r

    def solve(self, rhs, surf):
        n = rhs.numel()
        A = torch.empty((n, n), dtype=torch.float64, device=DEV)
        for a in range(0, n, 512):
            b = min(n, a + 512)
            e = torch.zeros((b - a, n), dtype=torch.float64, device=DEV)
            e[torch.arange(b - a), torch.arange(a, b)] = 1.0
            A[:, a:b] = self.apply(e.reshape(b - a, *rhs.shape), surf).reshape(b - a, n).T
        return torch.linalg.solve(A, rhs.reshape(-1)).reshape(rhs.shape)

    def derivs(self, E, P):
        """Ghost values with zero wall slopes, then the surface's derivatives (E and P are changed in place)."""
        rows = slice(1, -1) if self.three else slice(None)
        st, w = self.X[0]
        for f in (E, P):
            a, b = w[1], w[-2]
            f[rows, 0] = -(f[rows, 1:7] * a[1:]).sum(-1) / a[0]
            f[rows, -1] = -(f[rows, -7:-1] * b[:-1]).sum(-1) / b[-1]
        Ex, Exx, Px = self._along(self.X[0], E, 1), self._along(self.X[1], E, 1), self._along(self.X[0], P, 1)
        if not self.three:
            zero = torch.zeros_like(E)
            return Ex, Exx, Px, zero, zero, zero
        st, w = self.Y[0]
        for f in (E, P):
            a, b = w[1], w[-2]
            f[0, 1:-1] = -(f[1:7, 1:-1] * a[1:, None]).sum(0) / a[0]
            f[-1, 1:-1] = -(f[-7:-1, 1:-1] * b[:-1, None]).sum(0) / b[-1]
        return Ex, Exx, Px, self._along(self.Y[0], E, 0), self._along(self.Y[1], E, 0), self._along(self.Y[0], P, 0)

    def march(self, p, E, P, steps):
        """`steps` RK4 steps of the free-surface conditions from E, P (W = 0), every Laplace problem solved directly."""
        shape = (self.nyg, self.nxg)
        E, P = (torch.tensor(a.reshape(shape), device=DEV) for a in (E, P))
        W = torch.zeros_like(E)
        d = self.derivs(E, P)
        dt, inner = p.dt, (slice(1, -1) if self.three else slice(None), slice(1, -1))

        def slopes(E, P, W, d):
            Ex, _, Px, Ey, _, Py = d
            s = 1 + Ex * Ex + Ey * Ey
            ke = -Ex * Px - Ey * Py + W * s
            kp = -G * E - 0.5 * (Px * Px + Py * Py - W * W * s)
            if self.three:
                for k in (ke, kp):
                    k[0, 0] = k[0, -1] = k[-1, 0] = k[-1, -1] = 0.0
            return ke, kp

        def velocity(E, P):
            d = self.derivs(E, P)
            rhs = torch.zeros((*shape, self.nzg), dtype=torch.float64, device=DEV)
            rhs[(*inner, -1)] = P[inner]
            phi = self.solve(rhs, (E, d[0], d[1], d[3], d[4]))
            w = self.Z[0][1][-1]
            return d, (phi[..., -7:] * w).sum(-1) / (self.geo["h"] + E)

        for _ in range(steps):
            ks = [slopes(E, P, W, d)]
            for c in (0.5, 0.5, 1.0):
                tE, tP = E + c * dt * ks[-1][0], P + c * dt * ks[-1][1]
                td, tW = velocity(tE, tP)
                ks.append(slopes(tE, tP, tW, td))
            E, P = (v + dt / 6 * (ks[0][q] + 2 * ks[1][q] + 2 * ks[2][q] + ks[3][q]) for q, v in ((0, E), (1, P)))
            d, W = velocity(E, P)
        return {"E": E.reshape(-1), "P": P.reshape(-1), "W": W.reshape(-1)}


def exact(case, seed):
    """The residual at any size; the step and the solve where the Laplace problem is small enough to be solved directly
    (up to 6000 unknowns, walls, no relaxation zones)."""
    if case["kind"] == "batch" or case["basin"] in ("periodic", "zones", "shoal"):
        return None
    n = (case["Nx"] + 2) * (case["Ny"] + 2 if case["Ny"] > 1 else 1) * (case["Nz"] + 1)
    if case["kind"] != "residual" and n > 6000:
        return None
    p, geo, E, P, _ = _basin(case, seed)
    op = _Operator(p, geo)
    if case["kind"] == "step":
        return op.march(p, E, P, case["steps"])
    surf, P = _surface_fields(case, seed, p)
    shape = (op.nyg, op.nxg)
    s = [torch.tensor(a.reshape(shape), device=DEV) for a in surf]
    rhs = torch.tensor(_rhs(p, P).reshape(*shape, op.nzg), device=DEV)
    if case["kind"] == "solve":
        return {"phi": op.solve(rhs, s).reshape(-1)}
    r = rhs - op.apply(torch.tensor(_first_guess(p, P, seed).reshape(*shape, op.nzg), device=DEV), s)
    return {"residual": r.reshape(-1), "norm": float(r.square().sum().sqrt())}
