"""Warm-start surrogate: a small MLP that predicts the steady per-cell fields
(n, u, v, w, T) of a flow from its parameters, trained on fields that this
DSMC produces, and used to seed the particle population instead of the
free-stream fill (no counterpart in the reference).

Network: 4 inputs (zero-padded to 16) -> `depth` x `hidden` GELU layers ->
`modes` coefficients -> field = mean + coefficients x basis, the basis
(modes x cells*5) learned with the rest.  Every GEMM, activation, loss and
optimizer step runs in this library's kernels (BF16 operands, FP32
accumulation, FP32 master weights, Adam); torch only holds the device
buffers.
"""
import ctypes
import math

import numpy as np

from ._capi import AdamParam, Mlp, check, lib

_P = ctypes.c_void_p


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _stream():
    import torch
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


class WarmStartMLP:
    IN_PAD = 16

    def __init__(self, field_size, n_in=4, hidden=512, depth=4, modes=256, seed=0, device="cuda"):
        import torch
        self.torch = torch
        self.dev = torch.device(device)
        self.F, self.n_in, self.hidden, self.depth, self.modes = field_size, n_in, hidden, depth, modes
        g = np.random.default_rng(seed)
        f32 = dict(dtype=torch.float32, device=self.dev)
        self.params = {}
        dims = [self.IN_PAD] + [hidden] * depth
        for l in range(depth):
            w = np.zeros((dims[l], hidden), np.float32)
            fan_in = n_in if l == 0 else dims[l]
            w[: (n_in if l == 0 else dims[l])] = g.normal(0, math.sqrt(2.0 / fan_in),
                                                           ((n_in if l == 0 else dims[l]), hidden))
            self.params[f"W{l}"] = torch.from_numpy(w).to(**f32)
            self.params[f"b{l}"] = torch.zeros(hidden, **f32)
        self.params["Wout"] = torch.from_numpy(
            g.normal(0, math.sqrt(1.0 / hidden), (hidden, modes)).astype(np.float32)).to(**f32)
        self.params["bout"] = torch.zeros(modes, **f32)
        self.params["B"] = torch.from_numpy(
            g.normal(0, 0.02, (modes, field_size)).astype(np.float32)).to(**f32)
        self.params["mean"] = torch.zeros(field_size, **f32)
        self.bf = {k: torch.empty(v.shape, dtype=torch.bfloat16, device=self.dev)
                   for k, v in self.params.items() if k.startswith("W") or k == "B"}
        self.m = {k: torch.zeros_like(v) for k, v in self.params.items()}
        self.v = {k: torch.zeros_like(v) for k, v in self.params.items()}
        self.t = 0
        self._refresh_bf16()

    # ------------------------------------------------------------ helpers --
    def _refresh_bf16(self):
        for k, b in self.bf.items():
            check(lib().dsmc_to_bf16(_p(self.params[k]), _p(b), b.numel(), _stream()), "to_bf16")

    def _gemm(self, m, n, k, a, lda, at, b, ldb, bt, c=None, ldc=0, beta=0.0, bias=None, act=0,
              cb=None, ldcb=0, split=1):
        check(lib().dsmc_gemm_bf16(m, n, k, _p(a), lda, at, _p(b), ldb, bt, _p(c), ldc, beta, _p(bias),
                                   act, _p(cb), ldcb, split, _stream()), "gemm_bf16")

    def set_mean(self, mean):
        """Sets the field mean (the decoder bias), e.g. the training-set mean."""
        self.params["mean"].copy_(self.torch.as_tensor(mean, dtype=self.torch.float32))

    # ------------------------------------------------------------ forward --
    def _forward(self, x, cache, field):
        """One call for the whole pass: padded inputs, layers, coefficients and,
        with `field`, the field.  Returns (field or None, cache for backward or
        None): the cache holds every layer's input and pre-activation."""
        torch = self.torch
        B, H, D = len(x), self.hidden, self.depth
        xin = np.empty((B, self.n_in), np.float32)
        xin[:] = x
        ptrs = _P * max(D, 1)
        net = Mlp(self.n_in, self.IN_PAD, H, D, self.modes, self.F)
        net.w = ptrs(*[self.bf[f"W{l}"].data_ptr() for l in range(D)])
        net.b = ptrs(*[self.params[f"b{l}"].data_ptr() for l in range(D)])
        net.w_out, net.b_out = self.bf["Wout"].data_ptr(), self.params["bout"].data_ptr()
        net.basis, net.mean = self.bf["B"].data_ptr(), self.params["mean"].data_ptr()
        # 16-bit activations in one buffer (256-byte rows apart), 32-bit
        # pre-activations only where backward will ask for them
        parts = [B * self.IN_PAD] + [B * H] * D + [B * self.modes]
        offs = [0]
        for n in parts:
            offs.append(offs[-1] + (n + 127) // 128 * 128)
        act = torch.empty(offs[-1], dtype=torch.bfloat16, device=self.dev)
        base = act.data_ptr()
        ptr = [base + 2 * o for o in offs]
        h = ptrs(*ptr[1:D + 1])
        zp = z = None
        if cache:
            z = torch.empty((max(D, 1), B, H), dtype=torch.float32, device=self.dev)
            zp = ptrs(*[z.data_ptr() + 4 * B * H * l for l in range(D)])
        y = torch.empty((B, self.F), dtype=torch.float32, device=self.dev) if field else None
        check(lib().dsmc_mlp_forward(ctypes.byref(net), xin.ctypes.data, B, ptr[0], zp, h, ptr[D + 1], _p(y), _stream()),
              "mlp_forward")
        if not cache:
            return y, None
        rows = [self.IN_PAD] + [H] * D + [self.modes]
        a = [act[o:o + n].view(B, c) for o, n, c in zip(offs, parts, rows)]
        return y, {"x": a[:D], "z": [z[l] for l in range(D)], "h": a[D], "c": a[D + 1]}

    def forward(self, x):
        """x: [batch, n_in] normalized inputs.  Returns the field [batch, F]
        (FP32, on the device) and the cache for backward."""
        return self._forward(x, cache=True, field=True)

    # ----------------------------------------------------------- backward --
    def _layer_backward(self, g, w, b, x, dz, dzb, inner):
        """The gradients of weights w and bias b into g; returns the input's (`inner`) or None."""
        B, dout = dz.shape
        din = x.shape[1]
        g[w] = self.torch.empty((din, dout), dtype=self.torch.float32, device=self.dev)
        g[b] = self.torch.empty(dout, dtype=self.torch.float32, device=self.dev)
        dx = self.torch.empty((B, din), dtype=self.torch.float32, device=self.dev) if inner else None
        check(lib().dsmc_layer_backward(B, din, dout, _p(x), _p(dz), _p(dzb), _p(self.bf[w]), _p(g[w]), _p(g[b]),
                                        _p(dx), _stream()), "layer_backward")
        return dx

    def loss_and_grads(self, x, targets_bf16):
        """Masked MSE against BF16 targets [batch, F] (NaN = no target).
        Returns (loss, valid count, grads dict of FP32 tensors)."""
        torch = self.torch
        B = len(x)
        _, cache = self._forward(x, cache=True, field=False)
        y = torch.empty((B, self.F), dtype=torch.float32, device=self.dev)
        n = B * self.F
        dyb = torch.empty(y.shape, dtype=torch.bfloat16, device=self.dev)
        acc = torch.zeros(1, dtype=torch.float64, device=self.dev)
        cnt = torch.zeros(1, dtype=torch.int64, device=self.dev)
        g = {}
        g["mean"] = torch.empty(self.F, dtype=torch.float32, device=self.dev)
        check(lib().dsmc_decode_mse(B, self.F, self.modes, _p(cache["c"]), _p(self.bf["B"]),
                                    _p(self.params["mean"]), _p(targets_bf16), 1.0 / n, _p(y), _p(dyb),
                                    _p(g["mean"]), _p(acc), _p(cnt), _stream()), "decode_mse")
        g["B"] = torch.empty((self.modes, self.F), dtype=torch.float32, device=self.dev)
        self._gemm(self.modes, self.F, B, cache["c"], self.modes, 1, dyb, self.F, 0, g["B"], self.F)
        dc = torch.empty((B, self.modes), dtype=torch.float32, device=self.dev)
        dcb = torch.empty(dc.shape, dtype=torch.bfloat16, device=self.dev)
        split = max(1, min(64, self.F // 4096))
        ws = torch.empty(lib().dsmc_gemm_split_workspace(B, self.modes, split), dtype=torch.uint8,
                         device=self.dev)
        check(lib().dsmc_gemm_split_bf16(B, self.modes, self.F, _p(dyb), self.F, 0, _p(self.bf["B"]), self.F, 1,
                                         _p(dc), _p(dcb), split, _p(ws), _stream()), "gemm_split_bf16")
        dh = self._layer_backward(g, "Wout", "bout", cache["h"], dc, dcb, True)
        for l in range(self.depth - 1, -1, -1):
            z = cache["z"][l]
            dz = torch.empty_like(z)
            dzb = torch.empty(z.shape, dtype=torch.bfloat16, device=self.dev)
            check(lib().dsmc_gelu_backward(_p(z), _p(dh), _p(dz), _p(dzb), z.numel(), _stream()),
                  "gelu_backward")
            dh = self._layer_backward(g, f"W{l}", f"b{l}", cache["x"][l], dz, dzb, l > 0)
        return acc, cnt, g, y

    def adam_step(self, grads, lr=1e-3, b1=0.9, b2=0.999, eps=1e-8, weight_decay=0.0):
        self.t += 1
        ps = (AdamParam * len(self.params))(*[
            AdamParam(*(_p(a) for a in (w, grads[k], self.m[k], self.v[k], self.bf.get(k))), w.numel(),
                      weight_decay if k.startswith("W") else 0.0)
            for k, w in self.params.items()])
        check(lib().dsmc_adam_steps(ps, len(ps), lr, b1, b2, eps, self.t, _stream()), "adam_steps")

    def train(self, x, targets_bf16, epochs=200, batch=128, lr=1e-3, lr_final=1e-5, seed=0,
              log=None):
        """Mini-batch Adam over (x [N, n_in], targets_bf16 [N, F] on the
        device, rows in random order), cosine learning-rate decay; each epoch
        visits the contiguous batches in a new random order.  Returns the
        per-epoch mean loss."""
        N = len(x)
        nb = max(1, N // batch)
        rng = np.random.default_rng(seed)
        history = []
        steps = epochs * nb
        step = 0
        for ep in range(epochs):
            tot, cnt = 0.0, 0
            for i in rng.permutation(nb):
                lo, hi = i * batch, min(N, (i + 1) * batch)
                lr_now = lr_final + 0.5 * (lr - lr_final) * (1 + math.cos(math.pi * step / steps))
                acc, c, g, _ = self.loss_and_grads(x[lo:hi], targets_bf16[lo:hi])
                self.adam_step(g, lr=lr_now)
                tot += float(acc.item())
                cnt += int(c.item())
                step += 1
            history.append(tot / max(cnt, 1))
            if log and (ep % max(1, epochs // 10) == 0 or ep == epochs - 1):
                log(f"epoch {ep}: mse {history[-1]:.3e}")
        return history

    def predict(self, x):
        return self._forward(x, cache=False, field=True)[0]
