"""Which multigrid levels take the fused tile kernels, and their tile geometry
(host only), with the device runs that belong to a form's limits.

The geometry is chosen when a simulation is created, so an accepted grid must
never fail there: cores hold three columns or more and cover every column, and
a launch stays within the device's limits."""
import ctypes as C

import numpy as np
import pytest

import cases

NONE, UNIFORM, CROSS = 0, 1, 2
GEO = ("ntx", "nty", "cx", "cy", "halo", "HW", "PH", "NZP", "threads", "smem")


def form(ow3d, p, geo, level, precision=0):
    L = ow3d.lib()
    p.precision = precision
    z = np.zeros_like(geo["h"])
    a = [np.ascontiguousarray(geo.get(k, z), dtype=np.float64) for k in ("h", "hx", "hxx", "hy", "hyy")]
    D = C.POINTER(C.c_double)
    n, mode = C.c_int(), C.c_int()
    down, up = (C.c_int * 10)(), (C.c_int * 10)()
    r = L.ow3d_test_tile_form(C.byref(p), *[v.ctypes.data_as(D) for v in a], level, C.byref(n), C.byref(mode), down, up)
    assert r == 0, L.ow3d_last_error()
    return n.value, (mode.value, dict(zip(GEO, down)), dict(zip(GEO, up)))


def forms(ow3d, p, geo, precision=0):
    """Per level (0 = coarsest) the mode and the two launches' geometry."""
    n, f = form(ow3d, p, geo, 0, precision)
    return [f] + [form(ow3d, p, geo, l, precision)[1] for l in range(1, n)]


def periodic(ow3d, nx, nz):
    return ow3d.workloads.periodic_wave_2d(Nx=nx, Nz=nz)


SHORT = [(9, 13), (9, 17), (17, 25), (17, 33)]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SHORT)
def test_short_periods(ow3d, n, precision):
    """A level of two distinct columns above the coarsest has no tile form (a
    core holds three or more); the longer periods above it have one."""
    p, geo, _, _, _ = periodic(ow3d, *n)
    f = forms(ow3d, p, geo, precision)
    period = [((n[0] - 1) >> (len(f) - 1 - l)) for l in range(len(f))]
    assert 2 in period[1:]
    for (mode, down, up), m in list(zip(f, period))[1:]:
        assert mode == (UNIFORM if m >= 4 else NONE), m
        if mode:
            for g in (down, up):
                assert g["ntx"] * g["cx"] >= m and 3 <= g["cx"]


@pytest.mark.parametrize("precision", [0, 1])
def test_long_in_y(ow3d, precision):
    """524289 points in y: cores of 8 rows would be 65537 blocks in y, past the
    65535 a launch may have. A launch's tiles stay within that, or the level
    has no tile form."""
    for ny, levels in ((524289, 16), (262145, 15)):
        p, geo = cases.bump_3d(Nx=7, Ny=ny, Nz=7, Lx=0.7, Ly=0.1 * ny, amp=0.0, MGmaxgrids=levels)
        n, (mode, down, up) = form(ow3d, p, dict(h=geo["h"]), levels - 1, precision)
        assert n == levels
        assert mode == (NONE if ny == 524289 else UNIFORM)
        if mode:
            assert max(down["nty"], up["nty"]) <= 65535


@pytest.mark.parametrize("field", ["h", "hxx", "hyy"])
@pytest.mark.parametrize("at", [(1, 1), (1, -2), (-2, 1), (-2, -2), (16, 20)])
def test_one_column_differs(ow3d, field, at):
    """The uniform form needs the same coefficients in every interior column:
    one that differs, the first, the last or any other, takes it from the
    level; a ghost column does not."""
    p, geo = cases.bump_3d(Nx=33, Ny=33, Nz=9, Lx=3.3, Ly=3.3, amp=0.0)
    geo = {k: np.array(v) for k, v in geo.items()}
    assert forms(ow3d, p, geo)[-1][0] == UNIFORM
    f = geo[field].reshape(35, 35)
    f[0, 0] += 0.1
    f[-1, 3] += 0.1
    assert forms(ow3d, p, geo)[-1][0] == UNIFORM
    f[at] += 1e-12
    assert forms(ow3d, p, geo)[-1][0] == NONE


@pytest.mark.gpu
@pytest.mark.parametrize("n", SHORT)
def test_short_periods_match_oracle(ow3d, oracle, n):
    """The preconditioner as in test_periodic.py (1e-10), then five steps of
    the wave. Their solves stop at the matvec limit, where the oracle itself
    answers a relative change of the initial state by one of up to 2e3 times its
    size; with the operator's and preconditioner's 1e-12 that is 2e-9: 1e-8."""
    p, geo, E0, P0, _ = periodic(ow3d, *n)
    sim = ow3d.Simulation(p, **geo)
    o = oracle.Oracle(p, **geo, mode=oracle.MODE_DEVICE)
    r = np.random.default_rng(5).standard_normal((sim.Nxg, sim.Nzg))
    r[[0, -2, -1]] = 0.0
    u, v = sim.precondition(r.ravel()), o.precond(r.ravel())
    assert np.max(np.abs(u - v)) <= 1e-10 * np.max(np.abs(v))
    for s in (sim, o):
        s.set_state(E0, P0)
        cases.run_steps(s, 5)
    for a, b in zip(sim.get_state()[:4], o.get_state()[:4]):
        assert np.max(np.abs(a - b)) <= 1e-8 * np.max(np.abs(b))
    sim.close()
