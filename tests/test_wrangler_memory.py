"""The wrangler's translations when memory for their matrices or products is short."""

import numpy as np
import pytest
import torch

from pytential_b200 import fmm
from pytential_b200.workloads import laplace3d_ellipsoid

pytestmark = pytest.mark.gpu

NEVER = 1 << 50                 # words no GPU has


def _wrangler(geo, spec):
    return fmm.B200QBXExpansionWrangler(fmm.B200TreeIndependentDataForWrangler(spec), geo,
                                        np.float64, 2, lambda *a: 9)


def _drive(geo, w):
    g = np.random.default_rng(1)
    s = torch.from_numpy(g.normal(size=(1, w.dgeo.nsources))).cuda()
    return fmm.drive_fmm(None, w, [s])


@pytest.fixture(scope="module")
def problem():
    wl = laplace3d_ellipsoid(nrefine=1, nshell=100, op="S")
    geo = wl.geometry()
    return geo, wl.spec, _drive(geo, _wrangler(geo, wl.spec))


def _calls(monkeypatch):
    names = []
    call = fmm.Plan.call
    monkeypatch.setattr(fmm.Plan, "call", lambda self, name, *a: (names.append((name, a[1:2])),
                                                                  call(self, name, *a))[1])
    return names


def test_products_of_pairs(problem, monkeypatch):
    """Only M2L forms the products of the pairs: without memory for them M2M and L2L still go
    by the matrices, and M2L by pair."""
    geo, spec, want = problem
    w = _wrangler(geo, spec)
    w._scratch_words = NEVER
    names = _calls(monkeypatch)
    got = _drive(geo, w)
    stages = [a[0] for n, a in names if n == "qbxfmm_translate_boxes"]
    assert stages == [0, 2]
    assert "qbxfmm_multipole_to_local" in [n for n, _ in names]
    # the same sums in another order
    assert float((got - want).abs().max() / want.abs().max()) < 1e-13


def test_matrices(problem, monkeypatch):
    """Without memory for the matrices the wrangler translates by pair."""
    geo, spec, want = problem
    sizes = fmm.Plan.workspace_sizes
    monkeypatch.setattr(fmm.Plan, "workspace_sizes",
                        lambda self: [*sizes(self)[:6], 8 * NEVER, *sizes(self)[7:]])
    names = _calls(monkeypatch)
    w = _wrangler(geo, spec)
    got = _drive(geo, w)
    names = [n for n, _ in names]
    assert "qbxfmm_precompute_translations" not in names and "qbxfmm_translate_boxes" not in names
    assert float((got - want).abs().max() / want.abs().max()) < 1e-13
