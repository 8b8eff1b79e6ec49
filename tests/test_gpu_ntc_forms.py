"""The forms of the NTC kernel (reference streams; many light cells; many dense
cells; the others) lie on lines of cells and particles per cell: on both sides
of each, the split kernels give the states that the fused kernel gives."""
import numpy as np
import pytest

from cudadsmc_b200 import DSMCSolver, settings_t

pytestmark = pytest.mark.gpu

# 148 SMs of 16 warps: lines at 189,440 and 378,880 cells, 14 and 24 per cell
CASES = [((57, 57, 57), 5, "philox"), ((58, 58, 58), 5, "philox"), ((58, 58, 58), 14, "philox"),
         ((72, 72, 72), 24, "philox"), ((73, 73, 73), 24, "philox"), ((20, 20, 20), 24, "philox"),
         ((58, 58, 58), 5, "taus"), ((20, 20, 20), 30, "taus"), ((3, 2, 2), 90, "taus"),
         # reference streams: another form from 113,665 to 151,552 cells
         ((48, 48, 49), 9, "taus"), ((48, 48, 50), 9, "taus"), ((53, 53, 54), 9, "taus")]


@pytest.mark.parametrize("dim,ppc,rng", CASES)
def test_forms_match_the_fused_kernel(cuda, dim, ppc, rng):
    states = []
    for variant in (5, 0):
        s = settings_t().set(grid_min=(0, 0, 0), grid_max=(1, 1, 1), grid_dim=dim, density=1e20, part_per_cell=ppc,
                             fnum=1e20 / (dim[0] * dim[1] * dim[2]) / ppc, temp=200.0, init_temp2=600.0,
                             gas_mass=6.63e-26, gas_diam=4.17e-10, gas_tref=273.0,
                             gas_omega=0.5 if rng == "taus" else 0.81, rng=rng, init_kind="bimodal", periodic="n",
                             sample_every=0, seed=5)
        sol = DSMCSolver().Init(s)
        sol.SetKernelVariant(variant)
        sol.InitSystemState()
        sol.StepGraph(2e-5, 4)
        states.append((sol.DownloadState(), sol.GetCellState(), sol.Totals()))
        sol.close()
    a, b = states
    assert np.array_equal(a[0], b[0])
    assert np.array_equal(a[1][0], b[1][0]) and np.array_equal(a[1][1], b[1][1])
    assert np.array_equal(a[2][:2], b[2][:2])
