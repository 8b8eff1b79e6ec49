"""Cells above the split kernels' chunk (128 particles): a warp carries out the
selections that the fused kernel and the oracle make one after the other,
with the same numbers, its particles in shared memory up to 256 of them."""
import numpy as np
import pytest

from cudadsmc_b200 import DSMCSolver, settings_t
from oracle import oracle as O

from test_gpu_fast_parity import D_AR, M_AR, OMEGA, SEED, TREF, vhs_gref

pytestmark = pytest.mark.gpu

DT = 4e-6


def solver(ppc, variant, omega):
    s = settings_t().set(grid_min=(0, 0, 0), grid_max=(0.04, 0.03, 0.03), grid_dim=(4, 3, 3), density=1e20,
                         fnum=1.6e15 / ppc, part_per_cell=ppc, temp=300.0, gas_mass=M_AR, gas_diam=D_AR,
                         gas_tref=TREF, gas_omega=omega, ntc_local=1, periodic="n", sample_every=0, rng="philox",
                         seed=SEED, init_kind="maxwell")
    sol = DSMCSolver().Init(s)
    sol.SetKernelVariant(variant)
    sol.InitSystemState()
    return sol


@pytest.mark.parametrize("omega", [0.5, OMEGA])
@pytest.mark.parametrize("ppc", [129, 200, 256, 257, 700])
def test_giant_cells_match_the_oracle(cuda, ppc, omega):
    """One step.  Pair counts and remainders are exact; velocities agree
    within 1e-6 of their scale per collision of a particle (sincospi and the
    base-2 logarithm differ by an ulp or two from libm's), but for cells with
    an acceptance that the oracle reports as a near tie."""
    sol = solver(ppc, 5, omega)
    before, (mr, _) = sol.DownloadState(), sol.GetCellState()
    cells = mr.shape[0]
    f = O.fast_params(SEED, 1, 1.6e15 / ppc, DT, 1e-6, O.cross_section_of(D_AR), omega,
                      vhs_gref(omega), ntc_local=1, warp_cap=128)
    vo = before[3:].copy()
    start = (np.arange(cells + 1) * ppc).astype(np.uint32)
    info, _ = O.collide_fast(f, vo[0], vo[1], vo[2], start, mr)
    sol.RunSimulationStep(DT, 1)
    after, (mg, _), totals = sol.DownloadState(), sol.GetCellState(), sol.Totals()
    sol.close()
    assert info[:, 0].min() >= 32 and np.all(info[:, 2] == 3)
    assert totals[0] == info[:, 0].sum() and np.array_equal(mg[:, 1], mr[:, 1])
    ok = info[:, 3] == 0
    assert ok.sum() >= cells - 2
    if ok.all():
        assert totals[1] == info[:, 1].sum()
    assert np.allclose(mg[ok, 0], mr[ok, 0], rtol=4e-6, atol=0)
    rms = np.repeat(np.sqrt((before[3:].astype(np.float64) ** 2).sum(0).reshape(cells, ppc).mean(1)), ppc)
    scale = np.maximum(np.linalg.norm(vo.astype(np.float64), axis=0), rms)
    # (a wall turns a component's sign)
    err = np.max(np.abs(np.abs(after[3:]) - np.abs(vo)), axis=0) / scale
    bound = 1e-6 * np.repeat(np.maximum(1.0, 2.0 * info[:, 1] / ppc), ppc)
    slot = np.repeat(ok, ppc)
    assert np.all(err[slot] <= bound[slot])


@pytest.mark.parametrize("ppc", [330, 2600])
def test_giant_cells_equal_the_fused_kernel(cuda, ppc):
    """Three steps, bit for bit, against the fused kernel that does these
    cells' selections on one thread (its chunk holds 256 particles)."""
    states = []
    for variant in (3, 5):
        sol = solver(ppc, variant, OMEGA)
        sol.RunSimulationStep(DT, 3)
        states.append((sol.DownloadState(), sol.GetCellState(), sol.Totals()[:2]))
        sol.close()
    (a, ca, ta), (b, cb, tb) = states
    assert ta[1] > 0 and np.array_equal(ta, tb)
    assert np.array_equal(a, b) and np.array_equal(ca[0], cb[0])
