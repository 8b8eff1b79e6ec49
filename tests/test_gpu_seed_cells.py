"""The per-cell part of the fill from fields against a numpy restatement
(counts, (sigma g)max and remainders exact, the two-stream mixture by its
moments), and redrawn positions in cells that a body covers almost wholly."""
import numpy as np
import pytest

from cudadsmc_b200 import DSMCSolver, mesh_icosphere, settings_t

pytestmark = pytest.mark.gpu

M64 = (1 << 64) - 1


def unit_draws(seed, n):
    """SplitMix64 in [0, 1): draws 1..n."""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.arange(1, n + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    return (z >> np.uint64(11)).astype(np.float64) / 9007199254740992.0


def solver(dim, seed, radius=None, ppc=9.3):
    v = 0.01 ** 3
    s = settings_t().set(grid_min=(0, 0, 0), grid_max=tuple(0.01 * d for d in dim), grid_dim=dim, density=1e20,
                         fnum=1e20 * v / ppc, temp=200.0, stream_vel=(1000.0, 20.0, -5.0), gas_mass=6.63e-26,
                         gas_diam=4.17e-10, gas_tref=273.0, gas_omega=0.81, rng="philox", ntc_local=1,
                         init_kind="maxwell", seed=seed, capacity_factor=4.0, wall_diffuse=1, wall_temp=300.0,
                         geom_nearest=1, sample_every=0)
    sol = DSMCSolver().Init(s)
    if radius:
        c = tuple(0.005 * d for d in dim)
        sol.SetModel(*mesh_icosphere(3, radius, c), (8, 8, 8))
    return sol


@pytest.mark.parametrize("dim", [(1, 1, 1), (3, 5, 7), (16, 16, 8), (33, 32, 31)])
@pytest.mark.parametrize("weight", [0.0, 0.6, 1.0])
def test_counts_and_collision_state(cuda, dim, weight):
    seed = 77
    sol = solver(dim, seed)
    cells = dim[0] * dim[1] * dim[2]
    r = np.random.default_rng(cells)
    f = np.stack([1e20 * r.uniform(0, 3, cells), r.normal(500, 300, cells), r.normal(0, 100, cells),
                  r.normal(0, 100, cells), r.uniform(50, 2500, cells)], axis=1).astype(np.float32)
    f[::7, 0] = np.nan
    f[1::11, 0] = -1.0
    f[::13, 4] = np.inf
    n = sol.InitFromFieldsTwoStream(f, weight) if weight else sol.InitFromFields(f)
    info = sol.Info()
    u = unit_draws(seed ^ 0x2545F4914F6CDD1D, 2 * cells).reshape(cells, 2)
    ok = np.isfinite(f[:, 0]) & (f[:, 0] > 0)
    expect = np.where(ok, np.where(ok, f[:, 0], 0).astype(np.float64) * np.float64(np.float32(info.cell_volume)) /
                      np.float64(np.float32(sol.settings.cfg.fnum)), 0.0)
    k = np.floor(expect) + (u[:, 0] < expect - np.floor(expect))
    assert n == int(k.sum())
    keys = sol.ReadKeys()
    assert np.array_equal(np.bincount(keys, minlength=cells), k)
    mr, _ = sol.GetCellState()
    T = np.where(np.isfinite(f[:, 4]) & (f[:, 4] > 0), f[:, 4], np.float32(200.0)).astype(np.float32)
    g = np.float32(info.max_rel_vel) * np.sqrt(np.maximum(T, np.float32(200.0)) / np.float32(200.0))
    assert np.array_equal(mr[:, 0], g.astype(np.float32))
    assert np.array_equal(mr[:, 1], u[:, 1].astype(np.float32))
    # the same population again, and the cells' mean energies within noise
    a = sol.DownloadState()
    assert (sol.InitFromFieldsTwoStream(f, weight) if weight else sol.InitFromFields(f)) == n
    assert np.array_equal(a, sol.DownloadState())
    if n > 20000:
        e = (a[3:] ** 2).sum(0, dtype=np.float64).sum()
        want = (k * ((f[:, 1:4].astype(np.float64) ** 2).sum(1) + 3 * 1.3806e-23 / 6.63e-26 * T)).sum()
        assert abs(e / want - 1) < 0.02
    sol.close()


@pytest.mark.parametrize("radius", [0.043, 0.0495])
def test_redrawn_positions_stay_outside(cuda, radius):
    """Cells at the body's rim keep 1 % of their volume or less: dozens of
    redraws, and the known outside point for the rest."""
    dim = (10, 10, 10)
    sol = solver(dim, 5, radius, ppc=40.0)
    f = np.tile(np.array([1e20, 0, 0, 0, 300.0], np.float32), (1000, 1))
    n = sol.InitFromFields(f)
    a = sol.DownloadState()
    assert a.shape[1] == n and np.all(np.isfinite(a))
    r = np.linalg.norm(a[:3].astype(np.float64).T - 0.05, axis=1)
    assert np.sum(r < radius * 0.99) <= 2e-3 * n
    lo = np.floor(a[:3] / np.float32(0.01)).astype(int).clip(0, 9)
    cell = (lo[2] * 10 + lo[1]) * 10 + lo[0]
    assert np.bincount(cell, minlength=1000).max() <= 42
    b = solver(dim, 5, radius, ppc=40.0)
    assert b.InitFromFields(f) == n and np.array_equal(a, b.DownloadState())
