"""The per-phase kernels inside whole steps: the fused coarse cycle on the grid
against its small levels in one thread-block cluster, and the tiled colour pass
against the per-column one, with the fused tile kernels switched off.

Flat basins and basins with their slopes given take the tile kernels on every
level above the dense operator, so a solve on them launches neither of these
forms; basins with a varying depth alone, more smoothing steps or cycles, and
odd periods do. The same functions run on the same values either way: bitwise."""
import numpy as np
import pytest

import cases  # noqa: F401  (puts tests/ on the path for the package loader)

pytestmark = pytest.mark.gpu


def _shoal(ow3d, prec):
    p, geo = ow3d.workloads.shoal(Nx=257, Ny=33, Nz=9, precision=prec)
    x = np.linspace(0.0, 1.0, (p.Nx + 2) * (p.Ny + 2))
    return p, geo, 0.01 * np.sin(40 * x), np.zeros_like(x)


def _depth_only(ow3d, prec):
    p, geo, E0, P0 = _shoal(ow3d, prec)
    return p, dict(h=geo["h"]), E0, P0


def _sea(ow3d, prec):
    return ow3d.workloads.irregular_sea(Nx=257, Ny=65, Nz=17, precision=prec, seed=7)[:4]


# launches of an FP64 V cycle on the per-phase kernels (mixed: one more, the
# conversion): scaled copy and clearing, the fused cycle, and for the sea, whose
# finest level is above its size, two colours twice, residual, restriction and
# prolongation
PHASES = {"shoal": 3, "sea": 10, "depth_only": 3}
CASES = {"shoal": _shoal, "sea": _sea, "depth_only": _depth_only}


class _Knobs:
    """Test settings of the library, put back on leaving."""

    def __init__(self, ow3d, **kw):
        self.L, self.kw, self.old = ow3d.lib(), kw, {}

    def __enter__(self):
        for k, v in self.kw.items():
            self.old[k] = getattr(self.L, "ow3d_test_set_" + k)(v)

    def __exit__(self, *a):
        for k, v in self.old.items():
            getattr(self.L, "ow3d_test_set_" + k)(v)


def _vcycle_launches(ow3d, sim):
    r = np.random.default_rng(3).standard_normal(sim.N)
    sim.precondition(r)
    n0 = ow3d.lib().ow3d_launch_count()
    sim.precondition(r)
    return ow3d.lib().ow3d_launch_count() - n0


def _run(ow3d, case, prec, schedule=(None, None, None), **knobs):
    """State after the schedule's steps, matvecs, launches of one V cycle."""
    with _Knobs(ow3d, **knobs):
        p, geo, E0, P0 = CASES[case](ow3d, prec)
        with ow3d.Simulation(p, **geo) as sim:
            n = _vcycle_launches(ow3d, sim)
            sim.set_state(E0, P0)
            for on in schedule:
                if on is not None:
                    assert ow3d.lib().ow3d_set_coarse_cluster(sim.h, on) == 0
                assert sim.step(2) >= 0
            return sim.get_state()[:4], sim.stats()["total_iterations"], n


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a[0], b[0])) and a[1] == b[1]


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
@pytest.mark.parametrize("case", list(CASES))
def test_tail_cluster_is_bitwise_the_grid_cycle(ow3d, case, prec):
    # a basin of varying depth alone has no tile form: the default takes the fused cycle
    tiles = 1 if case == "depth_only" else 0
    ref = _run(ow3d, case, prec, tiles=tiles, tail_max_points=0, tail_cluster=16)
    small16 = _run(ow3d, case, prec, tiles=tiles, tail_max_points=8192, tail_cluster=16)
    small8 = _run(ow3d, case, prec, tiles=tiles, tail_max_points=8192, tail_cluster=8)
    whole = _run(ow3d, case, prec, tiles=tiles, tail_max_points=1 << 40, tail_cluster=16)
    assert ref[2] == PHASES[case] + prec
    # descent, cluster and ascent in place of one launch, or the cluster alone
    assert small16[2] == small8[2] == ref[2] + 2 and whole[2] == ref[2]
    for got in (small16, small8, whole):
        assert _same(got, ref)


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_coarse_cluster_mode_per_handle(ow3d, prec):
    """ow3d_set_coarse_cluster switched between steps, the captured graphs
    dropped and captured again."""
    runs = [_run(ow3d, "sea", prec, schedule=s, tiles=0) for s in ((0, 0, 0), (1, 1, 1), (1, 0, 1))]
    assert all(r[2] == PHASES["sea"] + prec for r in runs)
    assert _same(runs[1], runs[0]) and _same(runs[2], runs[0])


@pytest.mark.parametrize("prec", [0, 1], ids=["fp64", "mixed"])
def test_steps_with_tiled_colour_passes(ow3d, prec):
    """257 x 65 x 17: the finest level runs outside the fused coarse kernel, so
    its smoothing takes the tiled pass inside the solves."""
    on = _run(ow3d, "sea", prec, tiles=0, colour_tiles=1)
    off = _run(ow3d, "sea", prec, tiles=0, colour_tiles=0)
    assert on[2] == off[2] == PHASES["sea"] + prec
    assert _same(on, off)
