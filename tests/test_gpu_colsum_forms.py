"""Column sums on both sides of the line between their two forms (16 rows; one
row per 150 columns): the same sums as adding row after row in FP32."""
import ctypes

import pytest
import torch

from cudadsmc_b200 import lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,ld", [(0, 300, 300), (1, 257, 264), (16, 512, 512), (17, 512, 520), (17, 2549, 2549),
                                          (17, 2550, 2550), (40, 6001, 6008), (40, 5999, 5999), (129, 20000, 20000)])
def test_colsum_forms(cuda, rows, cols, ld):
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn((max(rows, 1), ld), generator=g, device="cuda")
    out = torch.full((cols + 1,), 9.0, device="cuda")
    assert lib().dsmc_colsum(ctypes.c_void_p(x.data_ptr()), rows, cols, ld, ctypes.c_void_p(out.data_ptr()), None) == 0
    seq = torch.zeros(cols, device="cuda")
    for row in x[:rows, :cols]:
        seq += row
    assert torch.equal(out[:cols], seq) and out[cols] == 9
