"""The surrogate's pass in one native call at the edges of its input kernels
(1,000 and 4,096 values per launch, 4 per row here): each batch against the
same layers called one by one on inputs converted by torch.  The layers' sums
do not depend on the route, so every activation is the same bit for bit."""
import numpy as np
import pytest
import torch

from cudadsmc_b200 import lib
from cudadsmc_b200.surrogate import WarmStartMLP, _p

pytestmark = pytest.mark.gpu


def layer(a, w, b, act):
    """One layer through the plain entry point: (32-bit pre-activation, BF16 output)."""
    m, k = a.shape
    n = w.shape[1]
    z = torch.empty((m, n), dtype=torch.float32, device="cuda")
    h = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    assert lib().dsmc_gemm_bf16(m, n, k, _p(a), k, 0, _p(w), n, 0, _p(z), n, 0.0, _p(b), act, _p(h), n, 1, None) == 0
    return z, h


@pytest.mark.parametrize("batch", [1, 250, 251, 1024, 1025, 2300])
def test_forward_call_matches_layers(cuda, batch):
    net = WarmStartMLP(512, hidden=128, depth=2, modes=64, seed=3)
    net.set_mean(np.linspace(-1, 1, net.F))
    x = np.random.default_rng(batch).normal(size=(batch, net.n_in))
    a = torch.zeros((batch, net.IN_PAD), dtype=torch.bfloat16, device="cuda")
    a[:, :net.n_in] = torch.as_tensor(x.astype(np.float32)).to(torch.bfloat16)
    y, cache = net.forward(x)
    plain, none = net._forward(x, cache=False, field=True)
    assert none is None and torch.equal(plain, y)
    for l in range(net.depth):
        assert torch.equal(cache["x"][l], a), l
        z, a = layer(a, net.bf[f"W{l}"], net.params[f"b{l}"], 1)
        assert torch.equal(cache["z"][l], z), l
    assert torch.equal(cache["h"], a)
    _, c = layer(a, net.bf["Wout"], net.params["bout"], 0)
    assert torch.equal(cache["c"], c)
    assert torch.equal(y, layer(c, net.bf["B"], net.params["mean"], 0)[0])
