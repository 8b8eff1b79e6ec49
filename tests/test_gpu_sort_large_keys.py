"""Stable sort with keys of up to and above the fixup's chunk (768 entries),
which are ranked by themselves, at the edges of their passes (512 entries),
beside small and empty keys."""
import numpy as np
import pytest
import torch

from cudadsmc_b200 import stages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large", [[255, 256, 256], [257, 384, 385], [300] * 40, [512, 513, 641], [767, 768, 769], [897, 1024], [1025], [1280, 1281], [1535, 1536, 1537], [1793], [2047, 2048, 2049, 3],
                                   [4096, 4097], [30000, 1100]])
@pytest.mark.parametrize("form", ["aligned", "off4", "static"])
def test_large_keys(cuda, large, form):
    r = np.random.default_rng(sum(large))
    # large keys among keys of 0 to 5 entries
    nkeys = 70
    counts = r.integers(0, 6, nkeys)
    counts[r.permutation(nkeys)[:len(large)]] = large
    k = np.repeat(np.arange(nkeys), counts).astype(np.int32)
    k = k[r.permutation(len(k))]
    n = len(k)
    v = r.integers(0, 1 << 31, n).astype(np.int32)
    keys, vals = torch.from_numpy(k).cuda(), torch.from_numpy(v).cuda()
    start = torch.empty(nkeys + 1, dtype=torch.int32, device="cuda")
    if form == "static":
        stages.sort_static(keys, vals, nkeys, cell_start=start)
    else:
        off = 4 if form == "off4" else 0
        ws = torch.empty(stages.sort_workspace_bytes(n, nkeys) + 8, dtype=torch.uint8, device="cuda")[off:]
        stages.sort(keys, vals, nkeys, cell_start=start, workspace=ws)
    order = np.argsort(k, kind="stable")
    assert np.array_equal(keys.cpu().numpy(), k[order])
    assert np.array_equal(vals.cpu().numpy(), v[order])
    assert np.array_equal(start.cpu().numpy(), np.concatenate([[0], np.cumsum(counts)]))
