"""The GMRES iteration's kernel against the same iteration in tensor operations."""

import pytest
import torch

from pytential_b200 import gmres as mod

pytestmark = pytest.mark.gpu


def _reference(Ae, e, w, r, x, active, update_r):
    v = r
    for _ in range(2):
        for a, b in zip(Ae, e):
            d = torch.sum(a.conj() * w, dim=-1)[:, None]
            w, v = w - d * a, v - d * b
        nw = torch.linalg.norm(w, dim=-1)
        inv = torch.where(active & (nw > 0), 1.0 / nw, torch.zeros_like(nw))[:, None]
        w, v = inv * w, inv * v
    d = torch.where(active, torch.sum(w.conj() * r, dim=-1), torch.zeros_like(w[:, 0]))[:, None]
    return w, v, r - d * w if update_r else r, x + d * v


@pytest.mark.parametrize("n", [1, 255, 2049, 8191, 8192, 16384, 16385, 40001])
@pytest.mark.parametrize("nd,count,dtype", [(1, 0, torch.complex128), (3, 1, torch.float64),
                                            (7, 20, torch.complex128), (2, 64, torch.float64),
                                            (2, 65, torch.complex128), (1, 130, torch.float64)])
@pytest.mark.parametrize("update_r", [False, True])
def test_step(n, nd, count, dtype, update_r):
    count = min(count, n - 1)
    g = torch.Generator(device="cuda").manual_seed(n)

    def rand():
        return torch.randn(nd, n, generator=g, dtype=dtype, device="cuda")
    # orthonormal images, as the iteration keeps them
    q = torch.linalg.qr(torch.stack([rand() for _ in range(count)], dim=-1))[0] if count else None
    Ae = [q[..., j].contiguous() for j in range(count)]
    e = [rand() for _ in range(count)]
    w, r, x = rand(), rand(), rand()
    active = torch.ones(nd, dtype=torch.bool, device="cuda")
    if nd > 2:
        active[1] = False
    want = _reference(Ae, e, w.clone(), r.clone(), x.clone(), active, update_r)
    w0, r0, x0 = w.clone(), r.clone(), x.clone()
    got = mod._step(Ae, e, w, r, x, active, update_r)
    assert torch.equal(w, w0) and torch.equal(r, r0) and torch.equal(x, x0)
    # sums of n float64 terms over up to 130 steps, on vectors of size sqrt(n) beside an image's 1:
    # relative to the largest of the preimages' entries
    for a, b in zip(got, want):
        scale = max(float(b.abs().max()), 1.0)
        assert float((a - b).abs().max()) <= 1e-11 * scale


@pytest.mark.parametrize("n,nd,kernel", [(65536, 1, True), (65537, 1, False), (65537, 63, False),
                                         (65537, 64, True)])
def test_few_densities_of_many_unknowns(n, nd, kernel, monkeypatch):
    """The kernel's eight SMs a density are for moderate sizes or many densities; the solve
    is the same either way."""
    calls = []
    step = mod._step
    monkeypatch.setattr(mod, "_step", lambda *a: calls.append(1) or step(*a))
    g = torch.Generator(device="cuda").manual_seed(n)
    diag = 1.0 + torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
    b = torch.randn(nd, n, generator=g, dtype=torch.float64, device="cuda")
    res = mod.gmres(lambda v: diag * v, b, tol=1e-10, restart=30, maxiter=60)
    assert bool(calls) == kernel
    # |A x - b| <= 1e-10 |b| and A >= 1
    err = torch.linalg.norm(res.solution - b / diag, dim=1) / torch.linalg.norm(b, dim=1)
    assert float(err.max()) <= 1.01e-10
