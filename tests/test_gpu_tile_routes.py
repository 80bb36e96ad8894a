"""Which kernels a V cycle launches, counted, and its result with the tile
kernels against the per-phase kernels (test_gpu_tiles.py's comparison and
tolerance), so that a level that lost its tile form cannot pass as one that
has it.

A tiled level is two launches, a per-phase one a launch per colour and bottom
pass of the two smoothing steps, residual, restriction and prolongation; the
levels of at most coop_max_points points run as one launch together unless each
of them is tiled."""
import numpy as np
import pytest

import cases
import test_tile_forms as tf

pytestmark = pytest.mark.gpu

COOP = 160000      # points below which levels run in the fused coarse kernel
DENSE = 2500       # points of the largest dense operator below the finest level


def _expected(sim, modes, mixed, coop):
    """Launches of one ow3d_precondition."""
    nl = sim.level_count()
    N = [sim.level_size(l) for l in range(nl)]
    ncolor = [sim.level_dims(l)[3] for l in range(nl)]
    ld = max([l for l in range(1, nl - 1) if N[l] <= DENSE], default=0)
    cross = [sim.cross] * nl if not sim.top_cross else [False] * (nl - 1) + [True]

    def every(l):
        return all(modes[q] != tf.NONE for q in range(ld + 1, l + 1))

    def cycle(l):
        if l == ld:
            return 1
        if N[l] <= coop and not every(l):
            return 1
        if modes[l] != tf.NONE:
            return 2 + cycle(l - 1)
        return 2 * (ncolor[l] + (2 if cross[l] else 0)) + 3 + cycle(l - 1)

    top = nl - 1
    fine = modes[top] != tf.NONE and (N[top] > coop or every(top))
    direct = fine and (not mixed or modes[top] == tf.UNIFORM)   # reads the solver's vector
    n = cycle(top) + (0 if direct else 1) + (0 if fine else 1) + (1 if mixed else 0)
    return n, [l for l in range(ld + 1, nl) if modes[l] != tf.NONE], nl - 1 - ld


def _compare(ow3d, p, geo, precision, slope=False, tiled="all", coop=COOP, top_cross=False):
    L = ow3d.lib()
    modes = [f[0] for f in tf.forms(ow3d, p, geo, precision)]
    assert p.precision == precision
    old_coop = L.ow3d_test_set_coop_max_points(coop)
    try:
        with ow3d.Simulation(p, **geo) as sim:
            sim.cross, sim.top_cross = slope, top_cross
            r = np.random.default_rng(3).standard_normal(sim.N)
            if p.periodic_x:   # image columns are identity rows with a zero right-hand side
                r3 = r.reshape(sim.Nyg, sim.Nxg, sim.Nzg)
                r3[:, [0, -2, -1]] = 0.0
            n, which, above = _expected(sim, modes, precision == 1, coop)
            off = _expected(sim, [tf.NONE] * len(modes), precision == 1, coop)[0]
            sim.precondition(r)
            c0 = L.ow3d_launch_count()
            u = sim.precondition(r)
            c1 = L.ow3d_launch_count()
            old = L.ow3d_test_set_tiles(0)
            try:
                v = sim.precondition(r)
            finally:
                L.ow3d_test_set_tiles(old)
            c2 = L.ow3d_launch_count()
    finally:
        L.ow3d_test_set_coop_max_points(old_coop)
    if tiled == "all":
        assert len(which) == above and above > 0
    elif tiled is not None:
        assert len(which) == tiled
    else:
        assert which
    assert (c1 - c0, c2 - c1) == (n, off)
    eps = 2.0 ** -53 if precision == 0 else 2.0 ** -24
    assert np.all(np.isfinite(u))
    if slope and precision == 1:
        assert np.array_equal(u, v)
    assert np.max(np.abs(u - v)) <= 4000 * eps * np.max(np.abs(v))


def _flat(n, **kw):
    p, geo = cases.bump_3d(Nx=n[0], Ny=n[1], Nz=n[2], Lx=0.1 * n[0], Ly=0.13 * n[1], amp=0.0, **kw)
    return p, dict(h=geo["h"])


def _slope(n, **kw):
    return cases.bump_3d(Nx=n[0], Ny=n[1], Nz=n[2], Lx=0.1 * n[0], Ly=0.13 * n[1], **kw)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(33, 33, 9), (97, 49, 9), (129, 17, 13), (257, 65, 17), (513, 129, 9)])
def test_flat(ow3d, n, precision):
    p, geo = _flat(n)
    _compare(ow3d, p, geo, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(33, 33, 9), (97, 49, 9), (129, 17, 13), (257, 65, 9), (513, 65, 9)])
def test_slope(ow3d, n, precision):
    """Up to 585 tiles (FP64 513x65x9): several waves."""
    p, geo = _slope(n)
    _compare(ow3d, p, geo, precision, slope=True)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(257, 9), (1025, 9), (1025, 14)])
def test_flume(ow3d, n, precision):
    kw = dict(MGmaxgrids=4) if n[1] == 14 else {}
    p, geo = cases.slope_2d(Nx=n[0], Nz=n[1], L=0.1 * n[0], **kw)
    _compare(ow3d, p, geo, precision, slope=True)
    p, geo = cases.flat_2d(Nx=n[0], Nz=n[1], L=0.1 * n[0], **kw)
    _compare(ow3d, p, geo, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(65, 9), (1025, 9), (513, 14)])
def test_periodic_flume(ow3d, n, precision):
    kw = dict(MGmaxgrids=4) if n[1] == 14 else {}
    p, geo = cases.flat_2d(Nx=n[0], Nz=n[1], L=0.1 * n[0], periodic_x=1, **kw)
    _compare(ow3d, p, geo, precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(65, 33, 9), (33, 65, 9), (17, 129, 9), (129, 17, 13), (65, 33, 10), (257, 65, 17)])
def test_periodic_basin(ow3d, n, precision):
    """Periodic x with walls in y."""
    kw = dict(MGmaxgrids=3) if n[2] == 10 else {}
    p, geo = _flat(n, periodic_x=1, **kw)
    _compare(ow3d, p, geo, precision)


@pytest.mark.parametrize("coop", [COOP, 0])
@pytest.mark.parametrize("n,tiled", [((65, 33, 25), 3), ((65, 33, 33), 1)])
def test_tall_slope_fp64(ow3d, n, tiled, coop):
    """In FP64 a sloping level of 23 or more sigma levels that is wide enough
    has no tile form: its smallest core with its halo exceeds the shared
    memory. Such a basin's levels up to coop points run fused, tiled or not;
    with coop 0 per-phase levels stand above tiled ones."""
    p, geo = _slope(n)
    _compare(ow3d, p, geo, 0, slope=True, tiled=tiled, coop=coop)


@pytest.mark.parametrize("precision", [0, 1])
def test_varying_depth_without_slopes(ow3d, precision):
    p, geo = _slope((65, 33, 9))
    _compare(ow3d, p, dict(h=geo["h"]), precision, tiled=0)


@pytest.mark.parametrize("coop", [COOP, 0])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("coarse", ["varying", "flat"])
def test_form_changes_between_levels(ow3d, coarse, precision, coop):
    """A slope at one column that the coarse grids skip: a tiled level with
    mixed-derivative terms above levels without them, which are flat and tiled,
    or of varying depth and per-phase (their iterate is cleared by the tiled
    level's way down)."""
    p, geo = _slope((257, 65, 13), **({} if coarse == "varying" else {"amp": 0.0}))
    h = np.array(geo["h"]).reshape(67, 259)
    hx = np.zeros_like(h)
    h[30, 50] *= 0.99
    hx[30, 50] = 0.05
    g = dict(h=h.ravel(), hx=hx.ravel())
    modes = [f[0] for f in tf.forms(ow3d, p, g, precision)]
    below = tf.NONE if coarse == "varying" else tf.UNIFORM
    assert modes[-1] == tf.CROSS and set(modes[1:-1]) == {below}
    _compare(ow3d, p, g, precision, tiled=1 if coarse == "varying" else "all", coop=coop, top_cross=True)


@pytest.mark.parametrize("strategy", [1, 2])
@pytest.mark.parametrize("n", [(65, 33, 17), (17, 65, 33), (33, 33, 33)])
def test_coarsening_strategies(ow3d, n, strategy):
    """Levels coarsened in one direction at a time, or in all three at once."""
    for precision in (0, 1):
        for make, slope in ((_flat, False), (_slope, True)):
            p, geo = make(n, MGCoarseningStrategy=strategy)
            _compare(ow3d, p, geo, precision, slope=slope, tiled=None, coop=0)
