"""The stage kernels at the sizes where they change form: the sort's groups
of four, tiles of keys and chunks, workspaces on and off 8 bytes; the collide
stage's warp tiles, staged and unstaged dense cells; ragged counts of the
gathers, moves and sampling."""
import ctypes

import numpy as np
import pytest
import torch

from cudadsmc_b200 import lib, stages
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nkeys", [(1, 1), (31, 3), (1025, 1), (1025, 5000), (4097, 17), (100003, 4096),
                                     (70001, 130000), (300000, 37889)])
@pytest.mark.parametrize("form", ["aligned", "off4", "own", "static"])
def test_sort(cuda, n, nkeys, form):
    r = np.random.default_rng(n + nkeys)
    # runs of near-sorted keys and a tail of keys past the range, left out
    k = np.minimum((np.arange(n) * nkeys // n + r.integers(-2, 3, n)).clip(0), nkeys - 1).astype(np.int32)
    if nkeys > 1:
        k[r.random(n) < 0.02] = r.integers(0, nkeys)
    over = r.random(n) < 0.03
    k[over] = nkeys + 5
    v = r.integers(0, 1 << 31, n).astype(np.int32)
    keys, vals = torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda()
    start = torch.full((nkeys + 1,), -1, dtype=torch.int32, device="cuda")
    if form == "static":
        stages.sort_static(keys, vals, nkeys, cell_start=start)
    else:
        ws = None
        if form != "own":
            off = 4 if form == "off4" else 0
            ws = torch.empty(stages.sort_workspace_bytes(n, nkeys) + 8, dtype=torch.uint8, device="cuda")[off:]
        stages.sort(keys, vals, nkeys, cell_start=start, workspace=ws)
    live = ~over
    order = np.argsort(k[live], kind="stable")
    m = int(live.sum())
    assert np.array_equal(keys[:m].cpu().numpy(), k[live][order])
    assert np.array_equal(vals[:m].cpu().numpy(), v[live][order])
    assert np.array_equal(start.cpu().numpy(), np.searchsorted(k[live][order], np.arange(nkeys + 1)))


def test_sort_one_key_above_a_chunk(cuda):
    n = 5000  # one key's entries above the fixup's chunk, small keys around it
    k = np.concatenate([[0, 1], np.full(n - 5, 2), [3, 3, 4]]).astype(np.int32)
    k = k[np.random.default_rng(1).permutation(n)]
    for _ in range(3):
        keys, vals = torch.from_numpy(k.copy()).cuda(), torch.arange(n, dtype=torch.int32, device="cuda")
        stages.sort(keys, vals, 5)
        assert np.array_equal(vals.cpu().numpy(), np.argsort(k, kind="stable"))


@pytest.mark.parametrize("counts", [[0, 1, 2, 3] * 9, [8] * 40, [255, 256, 257, 300, 0, 40, 12] * 3,
                                    [2047, 2048, 2049, 2100, 5]])
@pytest.mark.parametrize("omega", [0.5, 0.81])
def test_collide_cell_sizes(cuda, counts, omega):
    counts = np.asarray(counts)
    ncells, n = len(counts), int(counts.sum())
    start = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint32)
    r = np.random.default_rng(n)
    vel = r.normal(0, 300, (3, n)).astype(np.float32)
    cs, fnum, volume = O.cross_section_of(4.17e-10), 1e12, 1e-6
    gref = 0.0
    if omega != 0.5:
        from math import gamma, sqrt
        gref = sqrt(4 * 1.380649e-23 * 273.0 / 6.63e-26) * gamma(2.5 - omega) ** (-1 / (2 * omega - 1))
    vmax = np.float32(cs * 1500.0)
    # a cell of 8 selects about 3 pairs, one of 12 or more is dense
    dt = float(np.float32(3.0 / (0.5 * 8 * 7 * fnum / volume * float(vmax))))
    dt = min(dt, dt * (60.0 / max(counts.max(), 60)) ** 1.5)
    mr = np.stack([np.full(ncells, vmax), r.uniform(0, 1, ncells)], axis=1).astype(np.float32)
    f = O.fast_params(9, 4, fnum, dt, volume, cs, omega, gref, ntc_local=1, warp_cap=2048)
    vo, mo = vel.copy(), mr.copy()
    info, _ = O.collide_fast(f, vo[0], vo[1], vo[2], start, mo)
    dev = [torch.from_numpy(vel[k].copy()).cuda() for k in range(3)]
    mt = torch.from_numpy(mr.copy()).cuda()
    st = torch.zeros((ncells, 4), device="cuda")
    p = stages.collide_params(ncells, volume, cs, fnum, 0.0, dt, omega=omega, vhs_gref=gref, ntc_local=1,
                              rng="philox", seed=9, step=4)
    stages.collide(p, *dev, torch.from_numpy(start.astype(np.int32)).cuda(), mt, stat4=st)
    vg, mg, sg = np.stack([t.cpu().numpy() for t in dev]), mt.cpu().numpy(), st.cpu().numpy()
    assert np.array_equal(sg[:, 0].astype(np.int64), info[:, 0].astype(np.int64))
    assert np.array_equal(mg[:, 1], mo[:, 1])
    ok = info[:, 3] == 0  # no decision within the rounding of the base-2 log and exponential
    assert ok.sum() >= ncells - 2
    assert np.array_equal(sg[ok, 1].astype(np.int64), info[ok, 1].astype(np.int64))
    # each collision rounds on the cell's velocity scale, its partners' too
    per = np.maximum(1.0, 2.0 * info[:, 1] / np.maximum(counts, 1))
    slot = np.repeat(ok, counts)
    err = np.max(np.abs(vg - vo), axis=0) / 600.0
    assert np.all(err[slot] <= 4e-6 * np.repeat(per, counts)[slot])


@pytest.mark.parametrize("n", [1, 255, 1023, 1024, 1025, 300001])
def test_gather_move_and_sample_counts(cuda, n):
    cells, dim = 64, (4, 4, 4)
    g = torch.Generator(device="cuda").manual_seed(n)
    grid = stages.make_grid((0, 0, 0), (1, 1, 1), dim)
    pos = [torch.rand(n, generator=g, device="cuda") * 0.998 + 0.001 for _ in range(3)]
    vel = [300 * torch.randn(n, generator=g, device="cuda") for _ in range(3)]
    i32 = dict(dtype=torch.int32, device="cuda")
    keys, idx = torch.empty(n, **i32), torch.empty(n, **i32)
    start, cse = torch.empty(cells + 1, **i32), torch.empty(2 * cells, **i32)
    stages.cell_index(grid, *pos, keys, idx)
    want = sum((torch.floor(pos[k].double() / 0.25).long().clamp_(0, 3)) * 4 ** k for k in range(3))
    assert torch.equal(keys.long(), want) and torch.equal(idx.long(), torch.arange(n, device="cuda"))
    stages.sort(keys, idx, cells, cell_start=start)
    dst = [torch.empty(n, device="cuda") for _ in range(6)]
    stages.bounds_reorder(keys, idx, cells, cse, pos + vel, dst)
    order = torch.sort(want, stable=True).indices
    for a, b in zip(pos + vel, dst):
        assert torch.equal(a[order], b)
    assert torch.equal(cse.view(-1, 2)[:, 1] - cse.view(-1, 2)[:, 0], start[1:] - start[:-1])
    sums = torch.zeros((cells, 5), dtype=torch.float64, device="cuda")
    stages.sample(*dst[3:], start, cells, sums)
    ref = torch.zeros_like(sums)
    q = torch.stack([torch.ones(n, device="cuda")] + dst[3:], 1).double()
    q = torch.cat([q, (q[:, 1:] ** 2).sum(1, keepdim=True)], 1)
    ref.index_add_(0, keys.long(), q)
    assert torch.all((sums - ref).abs() <= 1e-12 * n * (1 + ref.abs()))
    x0, v0 = [a.clone() for a in dst[:3]], [a.clone() for a in dst[3:]]
    stages.move(stages.move_params(grid, 1e-5), *dst)
    for k in range(3):  # specular walls: at most a reflection off either side
        free = x0[k].double() + 1e-5 * v0[k].double()
        inside = (free > 0) & (free < 1)
        assert torch.all((dst[k].double() - free)[inside].abs() <= 2.0 ** -23)
        assert torch.all(dst[k] >= 0) and torch.all(dst[k] <= 1)
        assert torch.all(dst[3 + k].abs() == v0[k].abs())
