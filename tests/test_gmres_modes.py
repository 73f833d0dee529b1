"""GMRES under modes that see every tensor operation: they get them all."""

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from pytential_b200 import gmres as mod

pytestmark = pytest.mark.gpu


class _Counter(TorchDispatchMode):
    count = 0

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.count += 1
        return func(*args, **(kwargs or {}))


def _solve(n=500):
    g = torch.Generator(device="cuda").manual_seed(1)
    d = 1.0 + torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(2, n, generator=g, dtype=torch.float64, device="cuda")
    return mod.gmres(lambda v: d * v, b, tol=1e-10, restart=30, maxiter=60)


def test_dispatch_mode(monkeypatch):
    want = _solve()

    def step(*args):
        raise AssertionError("the kernel ran past the mode")
    monkeypatch.setattr(mod, "_step", step)
    with _Counter() as mode:
        got = _solve()
    # two inner products, differences and products for each kept image, twice
    assert mode.count > 8 * got.iteration_count
    # the same iteration in another order of its sums
    assert got.iteration_count == want.iteration_count
    assert float((got.solution - want.solution).abs().max()) < 1e-9
