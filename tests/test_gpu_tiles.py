"""Tile sizes of the split kernels against the fused kernel."""
import numpy as np
import pytest

from cudadsmc_b200 import DSMCSolver, settings_t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,ppc", [((3, 3, 3), 30), ((8, 8, 8), 16), ((17, 13, 11), 40), ((44, 22, 22), 6),
                                     ((40, 40, 40), 9)])
@pytest.mark.parametrize("rng", ["philox", "taus"])
def test_warp_tiles_of_every_size_equal_the_fused_kernel(cuda, rng, dim, ppc):
    """The split kernels cut a grid into warp tiles of 4 to 32 cells by its
    size; the fused CTA-wide kernel computes the same step for every cell that
    fits a chunk of both."""
    states = []
    for variant in (0, 5):
        s = settings_t().set(grid_min=(0, 0, 0), grid_max=tuple(0.01 * d for d in dim), grid_dim=dim,
                                density=1e20, fnum=1e14 / ppc, part_per_cell=ppc, temp=300.0, gas_mass=6.63e-26,
                                gas_diam=4.17e-10, gas_tref=273.0, gas_omega=0.81 if rng == "philox" else 0.5,
                                ntc_local=int(rng == "philox"), periodic="n", sample_every=0, rng=rng, seed=5,
                                init_kind="maxwell")
        sol = DSMCSolver().Init(s)
        sol.SetKernelVariant(variant)
        sol.InitSystemState()
        sol.RunSimulationStep(4e-6, 4)
        states.append((sol.DownloadState(), sol.GetCellState(), sol.Totals()[:2]))
        sol.close()
    (a, ca, ta), (b, cb_, tb) = states
    assert ta[0] > 0 and ta[1] > 0
    assert np.array_equal(a, b) and np.array_equal(ta, tb)
    assert np.array_equal(ca[0], cb_[0]) and np.array_equal(ca[1], cb_[1])
