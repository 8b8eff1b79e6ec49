"""Batches on either side of a warp's 32 members, with members that have next
to no collisions and one that has most of them: each equals itself stepped
alone, however the stages' grids are cut."""
import numpy as np
import pytest

from cudadsmc_b200 import DSMCBatch, DSMCSolver, settings_t

pytestmark = pytest.mark.gpu


def member(i, heavy):
    big = i == heavy
    dim, ppc = ((9, 8, 8), 140) if big else ((4 + i % 3, 3, 3), 1 + i % 5)
    s = settings_t().set(grid_min=(0, 0, 0), grid_max=tuple(0.01 * d for d in dim), grid_dim=dim, density=1e20,
                         fnum=(2e15 if big else 2e13) / ppc, part_per_cell=ppc, temp=300.0, gas_mass=6.63e-26,
                         gas_diam=4.17e-10, gas_tref=273.0, gas_omega=0.81, ntc_local=1, periodic="n",
                         sample_every=2, rng="philox", seed=50 + i, init_kind="maxwell", dt=4e-6)
    sol = DSMCSolver().Init(s)
    sol.InitSystemState()
    return sol


@pytest.mark.parametrize("members,heavy", [(1, 0), (32, 31), (33, 32), (70, 5)])
def test_batch_of_any_size_equals_members_alone(cuda, members, heavy):
    batched = [member(i, heavy) for i in range(members)]
    batch = DSMCBatch(batched)
    batch.Step(4)
    batch.Sync()
    pairs = []
    for i, a in enumerate(batched):
        b = member(i, heavy)
        b.RunSimulationStep(4e-6, 4)
        b.Sync()
        assert np.array_equal(a.DownloadState(), b.DownloadState()), i
        assert np.array_equal(a.GetCellState()[0], b.GetCellState()[0]), i
        ta, tb = a.Totals(), b.Totals()
        assert ta[0] == tb[0] and ta[1] == tb[1], i
        assert np.array_equal(a.Fields(), b.Fields(), equal_nan=True), i
        pairs.append(ta[0])
        b.close()
    assert pairs[heavy] > 32 * 576  # its cells are above the chunk and collided by warps
    batch.close()
    for s in batched:
        s.close()
