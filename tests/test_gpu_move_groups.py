"""The move stage on both sides of the count from which a thread flies four
particles at a time: a call on all particles and calls on parts of them give
the same state (specular and periodic faces: no random numbers)."""
import pytest
import torch

from cudadsmc_b200 import stages

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1499999, 1500000, 1500003])
@pytest.mark.parametrize("periodic", ["n", "x"])
def test_whole_equals_parts(cuda, n, periodic):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = [torch.rand(n, generator=g, device="cuda") * 0.998 + 0.001 for _ in range(3)]
    v = [300 * torch.randn(n, generator=g, device="cuda") for _ in range(3)]
    mp = stages.move_params(stages.make_grid((0, 0, 0), (1, 1, 1), (8, 8, 8)), 5e-4, periodic=periodic)
    a = [t.clone() for t in x + v]
    stages.move(mp, *a)
    b = [t.clone() for t in x + v]
    cut = [0, 1, 700000, n]
    for lo, hi in zip(cut, cut[1:]):
        part = [t[lo:hi].clone() for t in b]
        stages.move(mp, *part)
        for t, q in zip(b, part):
            t[lo:hi] = q
    for s, t in zip(a, b):
        assert torch.equal(s, t)
    assert not torch.equal(a[0], x[0]) and all(bool(((t >= 0) & (t <= 1)).all()) for t in a[:3])
