"""The surrogate's GEMM at the edges of its tiles (128 rows, 64 / 128 / 256
columns, 64 of k), with padded and unaligned outputs, split reductions, and
the decoder with its error in one pass, against float64 of the same BF16
values.

Tolerances: FP32 accumulation of k products, each step rounded to at worst
one unit in the last place, is within (k + 2) 2^-23 sum |a| |b| of the exact
sum; a BF16 result is within 2^-8 of its value beside that."""
import ctypes

import numpy as np
import pytest
import torch

from cudadsmc_b200 import lib

pytestmark = pytest.mark.gpu


def P(t, offset=0):
    return ctypes.c_void_p(t.data_ptr() + offset) if t is not None else None


def operand(rows, cols, ld, seed):
    """A BF16 rows x cols array in rows of ld, NaN in the padding."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.full((rows, ld), float("nan"), dtype=torch.bfloat16, device="cuda")
    a[:, :cols] = torch.randn((rows, cols), generator=g, device="cuda").to(torch.bfloat16)
    return a


def gelu(z):
    return 0.5 * z * (1 + torch.erf(z / np.sqrt(2)))


@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (1, 520, 512), (100, 512, 16), (127, 192, 72), (128, 64, 64),
                                   (129, 264, 136), (200, 1000, 328), (1024, 512, 512), (96, 40000, 256)])
@pytest.mark.parametrize("at,bt", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("pad", [0, 8])
def test_gemm_shapes(cuda, m, n, k, at, bt, pad):
    if at:
        m = (m + 7) // 8 * 8
    a = operand(k, m, m + pad, 1) if at else operand(m, k, k + pad, 1)
    b = operand(n, k, k + pad, 2) if bt else operand(k, n, n + pad, 2)
    A = (a[:, :m].T if at else a[:, :k]).double()
    B = (b[:, :k].T if bt else b[:, :n]).double()
    ref, mag = A @ B, A.abs() @ B.abs()
    tol = (k + 2) * 2.0 ** -23 * mag + 1e-30
    bias = torch.linspace(-1, 1, n, dtype=torch.float32, device="cuda")
    # C and its BF16 copy by TMA (padded rows of 4 and 8) and by plain stores
    # (rows of an odd length, a base off 16 bytes), the padding kept
    for ldc, off in ((n + pad, 0), (n + 1, 4)):
        c = torch.full((m * ldc + 1,), 7.0, dtype=torch.float32, device="cuda")
        h = torch.full((m * ldc + 1,), 7.0, dtype=torch.bfloat16, device="cuda")
        st = lib().dsmc_gemm_bf16(m, n, k, P(a), a.shape[1], at, P(b), b.shape[1], bt, P(c, off), ldc, 0.0,
                                  P(bias), 1, P(h, off // 2), ldc, 1, None)
        assert st == 0
        assert lib().dsmc_gemm_check(None) == 0
        cv = c[off // 4:off // 4 + m * ldc].reshape(m, ldc)
        hv = h[off // 4:off // 4 + m * ldc].reshape(m, ldc)
        z = ref + bias.double()
        t = tol + 2.0 ** -23 * z.abs()
        assert torch.all((cv[:, :n].double() - z).abs() <= t)
        assert torch.all((hv[:, :n].double() - gelu(z)).abs() <= 2.0 ** -8 * gelu(z).abs() + 1.2 * t + 1e-6)
        assert torch.all(cv[:, n:] == 7) and torch.all(hv[:, n:] == 7)
        # beta reads C back
        st = lib().dsmc_gemm_bf16(m, n, k, P(a), a.shape[1], at, P(b), b.shape[1], bt, P(c, off), ldc, -1.0,
                                  P(bias), 0, None, 0, 1, None)
        torch.cuda.synchronize()
        assert st == 0 and torch.all(cv[:, :n].abs() <= 2 * t)
        # a split reduction adds into C
        cv[:, :n] = 1.0
        st = lib().dsmc_gemm_bf16(m, n, k, P(a), a.shape[1], at, P(b), b.shape[1], bt, P(c, off), ldc, 0.0,
                                  None, 0, None, 0, 3, None)
        torch.cuda.synchronize()
        assert st == 0
        if k > 64:  # one K step does not split: C is overwritten
            assert torch.all((cv[:, :n].double() - 1 - ref).abs() <= tol + 4 * 2.0 ** -23 * (1 + mag))
        else:
            assert torch.all((cv[:, :n].double() - ref).abs() <= tol)
        assert torch.all(cv[:, n:] == 7)


@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (8, 1000, 32), (128, 256, 64), (136, 20040, 48), (300, 40960, 256)])
@pytest.mark.parametrize("off", [0, 1])
def test_decode_mse(cuda, m, n, k, off):
    a, b = operand(m, k, k, 3), operand(k, n, n, 4)
    g = torch.Generator(device="cuda").manual_seed(5)
    bias = torch.randn(n, generator=g, device="cuda")
    t = torch.randn((m, n), generator=g, device="cuda").to(torch.bfloat16)
    t[torch.rand((m, n), generator=g, device="cuda") < 0.1] = float("nan")
    # targets on and off a 16-byte boundary
    t = torch.cat([t.new_zeros(off), t.reshape(-1)])[off:].reshape(m, n)
    y = torch.empty((m, n), device="cuda")
    dy = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    col = torch.empty(n, device="cuda")
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    scale = 0.37
    st = lib().dsmc_decode_mse(m, n, k, P(a), P(b), P(bias), P(t), scale, P(y), P(dy), P(col), P(loss), P(cnt), None)
    assert st == 0 and lib().dsmc_gemm_check(None) == 0
    A, B = a.double(), b.double()
    ref = A @ B + bias.double()
    tol = (k + 2) * 2.0 ** -23 * (A.abs() @ B.abs()) + 2.0 ** -23 * ref.abs()
    assert torch.all((y.double() - ref).abs() <= tol)
    ok = ~torch.isnan(t)
    # the error follows from the field that was written: FP32 of y - t
    e = torch.where(ok, y - t.float(), torch.zeros((), device="cuda"))
    assert int(cnt) == int(ok.sum())
    assert abs(float(loss) - float((e.double() ** 2).sum())) <= 1e-12 * float(loss) + 1e-30
    gr = np.float32(scale) * np.float32(2.0) * e
    assert torch.equal(dy, gr.to(torch.bfloat16))
    # each column added row by row
    seq = torch.zeros(n, device="cuda")
    for row in gr:
        seq += row
    assert torch.equal(col, seq)
    s = gr.double()
    assert torch.all((col.double() - s.sum(0)).abs() <= m * 2.0 ** -24 * s.abs().sum(0) + 1e-30)


@pytest.mark.parametrize("m,n,k,split", [(8, 16, 64, 1), (33, 32, 200, 3), (128, 256, 40960, 10), (1000, 192, 6400, 64)])
def test_gemm_split(cuda, m, n, k, split):
    a, b = operand(m, k, k, 6), operand(n, k, k, 7)
    ws = torch.full((lib().dsmc_gemm_split_workspace(m, n, split) // 4,), float("nan"), device="cuda")
    outs = []
    for _ in range(2):
        c = torch.empty((m, n), device="cuda")
        cb = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
        assert lib().dsmc_gemm_split_bf16(m, n, k, P(a), k, 0, P(b), k, 1, P(c), P(cb), split, P(ws), None) == 0
        outs.append((c, cb))
    assert lib().dsmc_gemm_check(None) == 0
    A, B = a.double(), b.double()
    chunk = (k + 63) // 64
    chunk = (chunk + split - 1) // split * 64
    tol = (chunk + 2) * 2.0 ** -23 * (A.abs() @ B.abs().T) + 1e-30
    assert torch.all((outs[0][0].double() - A @ B.T).abs() <= tol)
    assert torch.equal(outs[0][0], outs[1][0])
    assert torch.equal(outs[0][1], outs[0][0].to(torch.bfloat16))


@pytest.mark.parametrize("rows,cols,ld", [(1, 1, 1), (7, 33, 40), (64, 32, 32), (1024, 512, 512), (300, 70, 70), (0, 5, 5)])
def test_colsum(cuda, rows, cols, ld):
    x = torch.randn((max(rows, 1), ld), device="cuda")
    out = torch.full((cols,), 9.0, device="cuda")
    assert lib().dsmc_colsum(P(x), rows, cols, ld, P(out), None) == 0
    seq = torch.zeros(cols, device="cuda")
    for row in x[:rows, :cols]:
        seq += row
    assert torch.equal(out, seq)
    s = x[:rows, :cols].double()
    assert torch.all((out.double() - s.sum(0)).abs() <= rows * 2.0 ** -24 * s.abs().sum(0) + 1e-30)


@pytest.mark.parametrize("n,off", [(1, 0), (3, 0), (4096, 0), (4099, 0), (1001, 1)])
def test_adam_aligned_or_not(cuda, n, off):
    g = torch.Generator(device="cuda").manual_seed(n)
    w, gr, m, v = (torch.randn(n + off, generator=g, device="cuda")[off:] for _ in range(4))
    v = v.abs()
    wb = torch.empty(n + off, dtype=torch.bfloat16, device="cuda")[off:]
    w64, m64, v64 = w.double(), m.double(), v.double()
    m64 = 0.9 * m64 + 0.1 * gr.double()
    v64 = 0.999 * v64 + 0.001 * gr.double() ** 2
    upd = (m64 / (1 - 0.9 ** 3)) / ((v64 / (1 - 0.999 ** 3)).sqrt() + 1e-8)
    ref = w64 - 1e-2 * (upd + 0.1 * w64)
    assert lib().dsmc_adam_step(P(w), P(gr), P(m), P(v), P(wb), n, 1e-2, 0.9, 0.999, 1e-8, 3, 0.1, None) == 0
    # a handful of FP32 roundings, and 1 - b2^t known to 2e-5 in FP32
    assert torch.all((m.double() - m64).abs() <= 4 * 2.0 ** -23 * (m64.abs() + gr.double().abs()))
    assert torch.all((w.double() - ref).abs() <= 2.0 ** -21 * w64.abs() + 1e-2 * 4e-5 * upd.abs() + 1e-9)
    assert torch.equal(wb, w.to(torch.bfloat16))
