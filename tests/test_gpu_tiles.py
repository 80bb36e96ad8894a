"""The fused tile kernels of the multigrid levels (mg_tile.cu) against the
per-phase kernels: one V cycle of each on the same random right-hand side.

Sizes at the edges of the tiles' range: grids smaller than one core, cores with
one column to spare, levels coarsened in x only, in sigma, odd level counts,
2-D flumes, a periodic flume, sloping and flat bottoms, both precisions, and
grids the tile form does not cover (depth varying without slopes).

Sloping levels in FP32 keep the per-phase kernels' order of every sum: bitwise
the same.

Tolerance elsewhere: the two forms sum the same terms in different orders. A V cycle is
some tens of dependent row updates per level, each a sum of fewer than 40
terms; 4000 rounding units of the largest value bound that with room
(4.4e-13 in FP64, 2.4e-4 in FP32)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

# (Nx, Ny, Nz, multigrid levels; 0: the reference's count)
FLAT3 = [(21, 11, 7, 2), (33, 33, 9, 0), (65, 33, 9, 0), (97, 49, 9, 0), (129, 17, 13, 0), (257, 65, 17, 0),
         (65, 33, 10, 3), (17, 9, 25, 0)]
SLOPE3 = FLAT3
LINE = [(17, 9, 0), (65, 9, 0), (129, 17, 0), (513, 9, 0), (1025, 13, 0), (97, 10, 4)]


def _compare(ow3d, p, geo, precision, slope=False):
    p.precision = precision
    L = ow3d.lib()
    with ow3d.Simulation(p, **geo) as sim:
        r = np.random.default_rng(3).standard_normal(sim.N)
        if p.periodic_x:   # image columns are identity rows with a zero right-hand side
            r3 = r.reshape(sim.Nyg, sim.Nxg, sim.Nzg)
            r3[:, [0, -2, -1]] = 0.0
        u = sim.precondition(r)
        old = L.ow3d_test_set_tiles(0)
        try:
            v = sim.precondition(r)
        finally:
            L.ow3d_test_set_tiles(old)
    eps = 2.0 ** -53 if precision == 0 else 2.0 ** -24
    assert np.all(np.isfinite(u))
    if slope and precision == 1:
        assert np.array_equal(u, v)
    assert np.max(np.abs(u - v)) <= 4000 * eps * np.max(np.abs(v))


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", FLAT3)
def test_flat(ow3d, n, precision):
    p, geo = cases.bump_3d(Nx=n[0], Ny=n[1], Nz=n[2], Lx=0.1 * n[0], Ly=0.13 * n[1], amp=0.0, MGmaxgrids=n[3])
    _compare(ow3d, p, dict(h=geo["h"]), precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", SLOPE3)
def test_slope(ow3d, n, precision):
    p, geo = cases.bump_3d(Nx=n[0], Ny=n[1], Nz=n[2], Lx=0.1 * n[0], Ly=0.13 * n[1], MGmaxgrids=n[3])
    _compare(ow3d, p, geo, precision, slope=True)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(513, 65, 17), (513, 129, 9)])
def test_flat_wide_cores(ow3d, n, precision):
    """Levels that take the 24x8 and 32x8 cores."""
    p, geo = cases.bump_3d(Nx=n[0], Ny=n[1], Nz=n[2], Lx=0.1 * n[0], Ly=0.13 * n[1], amp=0.0)
    _compare(ow3d, p, dict(h=geo["h"]), precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", LINE)
def test_flume(ow3d, n, precision):
    p, geo = cases.slope_2d(Nx=n[0], Nz=n[1], L=0.1 * n[0], MGmaxgrids=n[2])
    _compare(ow3d, p, geo, precision, slope=True)
    p, geo = cases.flat_2d(Nx=n[0], Nz=n[1], L=0.1 * n[0], MGmaxgrids=n[2])
    _compare(ow3d, p, geo, precision)


@pytest.mark.parametrize("n", [(65, 9), (129, 13), (257, 9)])
def test_periodic(ow3d, n):
    p, geo = cases.flat_2d(Nx=n[0], Nz=n[1], L=0.1 * n[0], periodic_x=1)
    _compare(ow3d, p, geo, 0)


@pytest.mark.parametrize("n", [(65, 65, 17), (129, 33, 13), (257, 65, 17)])
def test_slope_rounded_centre_weight(ow3d, n):
    """Spacings at which the centred difference's centre weight is not exactly
    zero (1e-16 of the others): its terms are part of the per-phase sums."""
    p, geo = cases.bump_3d(Nx=n[0], Ny=n[1], Nz=n[2], Lx=0.1 * (n[0] - 1), Ly=0.1 * (n[1] - 1))
    _compare(ow3d, p, geo, 1, slope=True)


def test_varying_depth_without_slopes(ow3d):
    """No tile form: the per-phase kernels either way, bitwise."""
    p, geo = cases.bump_3d(Nx=65, Ny=33, Nz=9, Lx=6.5, Ly=4.0)
    L = ow3d.lib()
    with ow3d.Simulation(p, geo["h"]) as sim:
        r = np.random.default_rng(3).standard_normal(sim.N)
        u = sim.precondition(r)
        old = L.ow3d_test_set_tiles(0)
        try:
            v = sim.precondition(r)
        finally:
            L.ow3d_test_set_tiles(old)
    assert np.array_equal(u, v)
