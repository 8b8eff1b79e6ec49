"""One crowded cell on a large grid: cells times the most particles in a cell
passes 32 bits while the particles themselves fit.  Every cell gets its
particles, with the cell's moments, outside the body; cells x most is just
below the largest product of the kernels' 32-bit form, just above it, and
above 2^32."""
import numpy as np
import pytest

from cudadsmc_b200 import DSMCSolver, mesh_icosphere, settings_t

pytestmark = pytest.mark.gpu

DIM = (64, 32, 32)
CELLS = 65536
CELL = 0.01
# A position is rounded to FP32: at coordinates up to 0.64 by up to 3e-8, which
# puts it in the next cell with a probability of 3e-6 per axis, 0.6 of 70,000
# particles on the average.
ACROSS = 8


def filled(crowd, at, radius, weight, other=None):
    s = settings_t().set(grid_min=(0, 0, 0), grid_max=tuple(CELL * d for d in DIM), grid_dim=DIM, density=1e20,
                         fnum=1e20 * CELL ** 3 / 2.0, temp=200.0, stream_vel=(900.0, 0.0, 0.0), gas_mass=6.63e-26,
                         gas_diam=4.17e-10, gas_tref=273.0, gas_omega=0.81, rng="philox", ntc_local=1,
                         init_kind="maxwell", seed=11, capacity_factor=1.6, wall_diffuse=1, wall_temp=300.0,
                         geom_nearest=1, sample_every=0)
    sol = DSMCSolver().Init(s)
    centre = tuple(0.5 * CELL * d for d in DIM)
    if radius:
        sol.SetModel(*mesh_icosphere(3, radius, centre), (8, 8, 8))
    per = float(np.float32(sol.settings.cfg.fnum)) / float(np.float32(sol.Info().cell_volume))
    f = np.zeros((CELLS, 5))
    f[:, 0], f[:, 1], f[:, 4] = 2.0 * per, 500.0, 250.0
    f[at, 0] = crowd * per
    f[at, 1:] = (-700.0, 40.0, 10.0, 800.0)
    f = f.astype(np.float32)
    if other is not None:  # another population before it
        sol.InitFromFields(other)
    n = sol.InitFromFieldsTwoStream(f, weight) if weight else sol.InitFromFields(f)
    keys, state = sol.ReadKeys(), sol.DownloadState()
    sol.close()
    return n, keys, state, centre, f


@pytest.mark.parametrize("crowd", [61000, 62000, 70000])
@pytest.mark.parametrize("at", [0, 40000, CELLS - 1])
def test_every_cell_is_filled(cuda, crowd, at):
    n, keys, state, _, f = filled(crowd, at, None, 0.0)
    count = np.bincount(keys, minlength=CELLS)
    assert len(keys) == n == state.shape[1] == count.sum()
    # rounded up or down, from a 32-bit density
    assert abs(count[at] - crowd) <= 1 + crowd * 2.0 ** -22 + ACROSS
    rest = np.delete(count, at)
    assert rest.min() >= 1 and np.sum(rest > 3) <= ACROSS
    # the positions lie in the cells they were drawn for: slots are in cell order
    assert np.sum(np.diff(keys.astype(np.int64)) < 0) <= ACROSS
    v = state[3:, keys == at].astype(np.float64)
    std = np.sqrt(1.3806e-23 * 800.0 / 6.63e-26)
    assert np.all(np.abs(v.mean(1) - [-700.0, 40.0, 10.0]) <= 6 * std / np.sqrt(crowd))
    assert np.all(np.abs(v.std(1) / std - 1) <= 6 / np.sqrt(2 * crowd))
    x = state[0, keys == at].astype(np.float64) / CELL
    x = x - np.floor(x.mean())
    assert abs(x.mean() - 0.5) <= 6 * np.sqrt(1 / 12) / np.sqrt(crowd)
    # all draws of the crowded cell differ in their streams
    assert np.unique(state[3, keys == at]).size >= crowd - 200
    # and nothing is left of a population that was there before
    other = np.tile(np.array([f[1, 0], 0.0, 0.0, 0.0, 100.0], np.float32), (CELLS, 1))
    again = filled(crowd, at, None, 0.0, other)
    assert np.array_equal(state, again[2])


@pytest.mark.parametrize("crowd", [61000, 70000])
@pytest.mark.parametrize("weight", [0.0, 0.6])
def test_redraws_of_a_crowded_cell(cuda, crowd, weight):
    # a cell that the sphere's face cuts
    radius = 0.0743
    ix, iy, iz = 32 + 7, 16, 16
    at = (iz * DIM[1] + iy) * DIM[0] + ix
    n, keys, state, centre, _ = filled(crowd, at, radius, weight)
    count = np.bincount(keys, minlength=CELLS)
    assert count.sum() == n and abs(count[at] - crowd) <= 1 + crowd * 2.0 ** -22 + ACROSS
    r = np.linalg.norm(state[:3].astype(np.float64).T - centre, axis=1)
    # outside the icosphere (its faces lie inside the sphere by less than 2 %)
    assert np.sum(r < radius * 0.98) <= 2e-3 * n
    assert r[keys == at].min() >= radius * 0.98
    assert np.mean(r[keys == at] < radius) < 0.2
