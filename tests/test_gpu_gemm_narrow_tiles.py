"""GEMMs whose narrow (64-column) tiles outnumber the SMs, so that a CTA works
through several of them: every epilogue warp then reuses its one staging block.
Against float64 of the same BF16 values; FP32 accumulation of k products is
within (k + 2) 2^-23 sum |a| |b| of the exact sum, a BF16 result within 2^-8 of
its value beside that."""
import ctypes

import numpy as np
import pytest
import torch

from cudadsmc_b200 import lib

pytestmark = pytest.mark.gpu


def P(t):
    return ctypes.c_void_p(t.data_ptr())


# more than 148 tiles of 128 x 64 and fewer than 148 of 128 x 128: 160, 288,
# 188 and 157 tiles
@pytest.mark.parametrize("m,n,k", [(2500, 512, 136), (4600, 512, 512), (12000, 72, 64), (20000, 64, 200)])
def test_several_narrow_tiles_per_cta(cuda, m, n, k):
    g = torch.Generator(device="cuda").manual_seed(m)
    a = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn((k, n), generator=g, device="cuda").to(torch.bfloat16)
    bias = torch.linspace(-1, 1, n, device="cuda")
    z = a.double() @ b.double() + bias.double()
    t = (k + 2) * 2.0 ** -23 * (a.double().abs() @ b.double().abs()) + 2.0 ** -23 * z.abs() + 1e-30
    act = 0.5 * z * (1 + torch.erf(z / np.sqrt(2)))
    for want_c in (True, False):
        c = torch.full((m, n), float("nan"), device="cuda")
        h = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        assert lib().dsmc_gemm_bf16(m, n, k, P(a), k, 0, P(b), n, 0, P(c) if want_c else None, n, 0.0, P(bias), 1,
                                    P(h), n, 1, None) == 0
        assert lib().dsmc_gemm_check(None) == 0
        assert not want_c or torch.all((c.double() - z).abs() <= t)
        assert torch.all((h.double() - act).abs() <= 2.0 ** -8 * act.abs() + 1.2 * t + 1e-6)


def test_several_narrow_split_tiles_per_cta(cuda):
    m, n, k, split = 1200, 512, 192, 2  # 160 tiles of 128 x 64
    g = torch.Generator(device="cuda").manual_seed(9)
    a = torch.randn((m, k), generator=g, device="cuda").to(torch.bfloat16)
    b = torch.randn((k, n), generator=g, device="cuda").to(torch.bfloat16)
    z, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    t = (k + 2 + split) * 2.0 ** -23 * mag + 1e-30
    c = torch.zeros((m, n), device="cuda")
    assert lib().dsmc_gemm_bf16(m, n, k, P(a), k, 0, P(b), n, 0, P(c), n, 0.0, None, 0, None, 0, split, None) == 0
    assert lib().dsmc_gemm_check(None) == 0
    assert torch.all((c.double() - z).abs() <= t)
    ws = torch.empty(lib().dsmc_gemm_split_workspace(m, n, split) // 4, device="cuda")
    h = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    c.zero_()
    assert lib().dsmc_gemm_split_bf16(m, n, k, P(a), k, 0, P(b), n, 0, P(c), P(h), split, P(ws), None) == 0
    assert lib().dsmc_gemm_check(None) == 0
    assert torch.all((c.double() - z).abs() <= t)
    assert torch.equal(h, c.to(torch.bfloat16))
