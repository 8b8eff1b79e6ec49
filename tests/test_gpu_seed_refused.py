"""Fields that ask for more particles than there is room for are refused, with
the state as it was: one cell far above the 32-bit range, one just below it,
cells whose counts add to a multiple of 2^32, and a total one above the
capacity."""
import numpy as np
import pytest

from cudadsmc_b200 import DsmcError, DSMCSolver, mesh_icosphere, settings_t

pytestmark = pytest.mark.gpu

DIM, PPC = (8, 6, 5), 9.0
CELLS = DIM[0] * DIM[1] * DIM[2]


def solver():
    s = settings_t().set(grid_min=(0, 0, 0), grid_max=tuple(0.01 * d for d in DIM), grid_dim=DIM, density=1e20,
                         fnum=1e20 * 0.01 ** 3 / PPC, temp=200.0, gas_mass=6.63e-26, gas_diam=4.17e-10,
                         gas_tref=273.0, gas_omega=0.81, rng="philox", ntc_local=1, init_kind="maxwell", seed=3,
                         wall_diffuse=1, wall_temp=300.0, sample_every=1)
    return DSMCSolver().Init(s)


def fields(sol, per_cell):
    """Fields asking for per_cell particles (an array, cell by cell)."""
    info = sol.Info()
    f = np.zeros((CELLS, 5), np.float64)
    f[:, 0] = np.asarray(per_cell, np.float64) * float(np.float32(sol.settings.cfg.fnum)) / float(
        np.float32(info.cell_volume))
    f[:, 1], f[:, 4] = 300.0, 250.0
    return f.astype(np.float32)


def crowded(kind, capacity):
    k = np.full(CELLS, 2.0)
    if kind == "outlier":
        k[77] = 1e18  # (a finite density)
    elif kind == "first_cell":
        k[0] = 1e18
    elif kind == "below_2_32":
        k[40] = 4294967295.0 * (1 + 2.0 ** -25)
    elif kind == "warp_sum":
        k[:] = 0.0
        k[64], k[70] = 2.0 ** 31, 2.0 ** 31
    elif kind == "grid_sum":
        k[:] = 0.0
        k[[5, 45, 133, 200]] = 2.0 ** 30
    else:
        k[:] = 0.0
        k[100] = capacity + 1.0
    return k


KINDS = ["outlier", "first_cell", "below_2_32", "warp_sum", "grid_sum", "one_above"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("weight", [0.0, 0.5])
def test_refused_before_the_fill(cuda, kind, weight):
    sol = solver()
    sol.InitFromFields(fields(sol, np.full(CELLS, PPC)))
    dt = 1e-6
    sol.RunSimulationStep(dt, 3)
    before = sol.DownloadState(), sol.GetCellState()[0], sol.ReadKeys()
    f = fields(sol, crowded(kind, sol.Info().capacity))
    with pytest.raises(DsmcError, match="capacity"):
        sol.InitFromFieldsTwoStream(f, weight) if weight else sol.InitFromFields(f)
    after = sol.DownloadState(), sol.GetCellState()[0], sol.ReadKeys()
    for a, b in zip(before, after):
        assert np.array_equal(a, b)
    sol.close()


def test_a_full_state_is_filled(cuda):
    sol = solver()
    k = np.zeros(CELLS)
    k[100] = sol.Info().capacity - 0.25  # either rounding fits
    n = sol.InitFromFields(fields(sol, k))
    assert sol.Info().capacity - 2 <= n <= sol.Info().capacity
    keys = sol.ReadKeys()
    assert len(keys) == n and np.all(keys == 100)
    sol.close()


@pytest.mark.parametrize("radius", [None, 0.018])
@pytest.mark.parametrize("dim,ppc", [(DIM, PPC), ((16, 16, 8), 0.6)])
def test_refused_fill_keeps_the_samples(cuda, dim, ppc, radius):
    """Dense and sparse grids: the fill's scratch lies in one place or the
    other.  What was sampled is still there after a refusal, and a fill after
    it is the one that a new solver makes."""
    cells = dim[0] * dim[1] * dim[2]

    def make():
        s = settings_t().set(grid_min=(0, 0, 0), grid_max=tuple(0.01 * d for d in dim), grid_dim=dim, density=1e20,
                             fnum=1e20 * 0.01 ** 3 / ppc, temp=200.0, stream_vel=(800.0, 0.0, 0.0),
                             gas_mass=6.63e-26, gas_diam=4.17e-10, gas_tref=273.0, gas_omega=0.81, rng="philox",
                             ntc_local=1, init_kind="maxwell", seed=3, wall_diffuse=1, wall_temp=300.0,
                             geom_nearest=1, sample_every=1)
        sol = DSMCSolver().Init(s)
        if radius:
            sol.SetModel(*mesh_icosphere(2, radius, tuple(0.005 * d for d in dim)), (8, 8, 8))
        return sol

    sol = make()
    per = float(np.float32(sol.settings.cfg.fnum)) / float(np.float32(sol.Info().cell_volume))
    f = np.tile(np.array([ppc * per, 300.0, 0, 0, 250.0], np.float32), (cells, 1))
    for weight in (0.0, 0.7):
        n = sol.InitFromFieldsTwoStream(f, weight) if weight else sol.InitFromFields(f)
        first = make()
        assert (first.InitFromFieldsTwoStream(f, weight) if weight else first.InitFromFields(f)) == n
        assert np.array_equal(first.DownloadState(), sol.DownloadState())
        first.close()
        sol.RunSimulationStep(1e-6, 3)
        sums, totals, ns = sol.SampleStatistics()
        assert ns == 3 and sums[:, 0].sum() > 2 * n
        bad = f.copy()
        bad[cells // 2, 0] = 1e30
        with pytest.raises(DsmcError, match="capacity"):
            sol.InitFromFieldsTwoStream(bad, weight) if weight else sol.InitFromFields(bad)
        again = sol.SampleStatistics()
        assert np.array_equal(sums, again[0]) and np.array_equal(totals, again[1]) and ns == again[2]
    sol.close()
