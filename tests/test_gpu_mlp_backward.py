"""A layer's gradients in one call, and Adam over several parameters: the
kernels of each run beside one another, and give bit for bit what the single
calls give one after the other."""
import ctypes

import pytest
import torch

from cudadsmc_b200 import lib
from cudadsmc_b200._capi import AdamParam
from cudadsmc_b200.surrogate import _p

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,din,dout", [(1024, 512, 512), (8, 16, 64), (136, 72, 264), (2000, 16, 512)])
@pytest.mark.parametrize("inner", [True, False])
def test_layer_backward_equals_single_calls(cuda, batch, din, dout, inner):
    g = torch.Generator(device="cuda").manual_seed(batch)
    rn = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, w = rn(batch, din).to(torch.bfloat16), rn(din, dout).to(torch.bfloat16)
    L = lib()
    for it in range(20):
        dz = rn(batch, dout)
        dzb = dz.to(torch.bfloat16)
        dw, db, dx = (torch.full(s, 7.0, device="cuda") for s in ((din, dout), (dout,), (batch, din)))
        assert L.dsmc_layer_backward(batch, din, dout, _p(x), _p(dz), _p(dzb), _p(w), _p(dw), _p(db),
                                     _p(dx) if inner else None, None) == 0
        # at once behind it on the stream: a reader of all three
        got = [t.clone() for t in (dw, db, dx)]
        rw, rb, rx = (torch.full_like(t, 7.0) for t in (dw, db, dx))
        assert L.dsmc_gemm_bf16(din, dout, batch, _p(x), din, 1, _p(dzb), dout, 0, _p(rw), dout, 0.0, None, 0,
                                None, 0, 1, None) == 0
        assert L.dsmc_colsum(_p(dz), batch, dout, dout, _p(rb), None) == 0
        if inner:
            assert L.dsmc_gemm_bf16(batch, din, dout, _p(dzb), dout, 0, _p(w), dout, 1, _p(rx), din, 0.0, None, 0,
                                    None, 0, 1, None) == 0
        for a, b in zip(got, (rw, rb, rx)):
            assert torch.equal(a, b), it
    assert L.dsmc_gemm_check(None) == 0


def test_layer_backward_refuses(cuda):
    t = torch.zeros((16, 16), device="cuda")
    b = t.to(torch.bfloat16)
    call = lambda n, dx, w: lib().dsmc_layer_backward(n, 16, 16, _p(b), _p(t), _p(b), w, _p(t), _p(t), dx, None)
    assert call(0, None, None) != 0 and call(16, _p(t), None) != 0


@pytest.mark.parametrize("sizes", [(5,), (1, 4096, 3, 100003), (1 << 20, 64, 64, 1 << 18)])
@pytest.mark.parametrize("off", [0, 1])
def test_adam_steps_equal_single_steps(cuda, sizes, off):
    g = torch.Generator(device="cuda").manual_seed(7)
    rn = lambda n: torch.randn(n + off, generator=g, device="cuda")[off:]
    sets = []
    for n in sizes:
        w, gr, m, v = rn(n), rn(n), 0.1 * rn(n), rn(n).abs()
        sets.append((w, gr, m, v, torch.zeros(n, dtype=torch.bfloat16, device="cuda") if n % 2 else None))
    twin = [tuple(t.clone() if t is not None else None for t in s) for s in sets]
    if off:  # clones are aligned: back to an odd offset
        twin = [tuple(None if t is None else t if t.dtype == torch.bfloat16 else
                      torch.cat([t[:1], t])[1:] for t in s) for s in twin]
    hyper = (1e-3, 0.9, 0.999, 1e-8)
    for t in (1, 2, 3):
        ps = (AdamParam * len(sets))(*[AdamParam(*(_p(a) for a in s), s[0].numel(), 0.01 * i)
                                       for i, s in enumerate(sets)])
        assert lib().dsmc_adam_steps(ps, len(sets), *hyper, t, None) == 0
        for i, s in enumerate(twin):
            assert lib().dsmc_adam_step(*(_p(a) for a in s), ctypes.c_size_t(s[0].numel()), *hyper, t, 0.01 * i,
                                        None) == 0
    for a, b in zip(sets, twin):
        for q, (x, y) in enumerate(zip(a, b)):
            assert x is None or torch.equal(x, y), q
