"""2D Helmholtz: the apply on both sides of the rule that takes the expansions straight to the
QBX targets, against the wrangler's stages (the expansions always)."""

import functools

import numpy as np
import pytest
import torch

from pytential_b200 import abi, fmm
from pytential_b200.discretization import make_starfish
from pytential_b200.geometry import QBXFMMGeometryData

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _geometry(kind, nel):
    d = make_starfish(nel)
    targets = [(d.nodes, +1)]
    if kind == "points":
        v = np.random.default_rng(2).uniform(-2, 2, size=(2, 400))
        v = v[:, np.abs(np.hypot(*v) - (1 + 0.25 * np.cos(5 * np.arctan2(v[1], v[0])))) > 0.15]
        targets.append((v[:, :60], 0))
    elif kind == "many":        # several targets per center, some at the center itself
        c, r = d.interleaved_centers()
        targets += [(d.nodes + 0.3 * r[0::2] * d.normals, +2), (c[:, 1::2].copy(), +2),
                    (d.nodes[:, :37].copy(), -1)]
    return d, QBXFMMGeometryData(d, targets)


@pytest.mark.parametrize("kind,nel,nrhs,direct,q,p,k", [
    ("surface", 250, 4, False, 3, 12, 12.0), ("surface", 250, 60, True, 5, 20, 20.0),
    ("surface", 250, 9, False, 5, 20, 20.0), ("surface", 440, 5, True, 6, 16, 20.0),
    ("surface", 440, 33, True, 3, 15, 12.0), ("surface", 440, 32, False, 3, 15, 12.0),
    ("surface", 600, 4, True, 5, 20, 20.0), ("surface", 600, 1, True, 0, 1, 3.0),
    ("points", 60, 1, False, 4, 15, 10.0), ("points", 110, 1, True, 5, 20, 15.0),
    ("points", 110, 2, False, 2, 9, 10.0), ("points", 230, 2, True, 6, 16, 15.0),
    ("points", 230, 17, True, 1, 4, 5.0), ("points", 230, 33, True, 7, 19, 12.0),
    ("many", 160, 3, False, 4, 13, 8.0), ("many", 160, 4, True, 4, 13, 8.0),
    ("many", 160, 9, True, 2, 6, 4.0)])
def test_both_sides_of_the_rule(kind, nel, nrhs, direct, q, p, k):
    d, geo = _geometry(kind, nel)
    s, _ = abi.geometry_arrays(geo)
    work = (2 * q + 1) * (2 * p + 1)
    if s["nnonqbx_chunks"] > 0:
        per_sm = 1 if nrhs == 1 else 2
    elif nrhs > 4 and work >= 400:
        per_sm = 2 if nrhs > 32 else 3
    else:
        per_sm = 4 if nrhs > 32 and work >= 160 else 5
    assert direct == (per_sm * 148 <= s["ntsqbx_chunks"]
                      <= s["nqbx_chunks"] * (4 if nrhs >= 4 else 1))
    spec = fmm.SourceKernelSpec(fmm.HelmholtzKernel(2, k), charge_coeff=-1j * k, dipole_coeff=1.0)
    rng = np.random.default_rng(5)
    dens = rng.normal(size=(nrhs, d.ndofs)) + 1j * rng.normal(size=(nrhs, d.ndofs))
    ap = fmm.QBXApply(geo, spec, q, p, nrhs=nrhs)
    x = torch.from_numpy(dens).cuda()
    u = ap(x)
    ap.check_error_word()
    w = fmm.B200QBXExpansionWrangler(
        fmm.B200TreeIndependentDataForWrangler(spec), geo, np.complex128, q,
        lambda kern, args, tree, lev: p, _use_target_specific_qbx=True, nrhs=nrhs)
    st = torch.from_numpy(d.upsample_density(dens) * d.quad_weights).cuda()
    v = fmm.drive_fmm(None, w, [st])
    # the same terms in float64; sums of order-p Hankel terms larger than their result
    assert float((u - v).abs().max() / v.abs().max()) < 5e-12
    # a captured apply runs the same kernels in the same order
    ap.capture()
    assert torch.equal(ap.replay(x), u)


@pytest.mark.parametrize("kind,nel", [("surface", 40), ("points", 60), ("many", 160)])
@pytest.mark.parametrize("nrhs", [1, 4])
def test_orders_whose_expansions_do_not_fit(kind, nel, nrhs):
    """Orders 8 and 20 with up to 4 densities, whose M2QBXL needs more shared memory than there
    is: straight to the targets, however few they are; with 6 densities it fits."""
    d, geo = _geometry(kind, nel)
    k = 9.0
    spec = fmm.SourceKernelSpec(fmm.HelmholtzKernel(2, k), charge_coeff=-1j * k, dipole_coeff=1.0)
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.normal(size=(6, d.ndofs)) + 1j * rng.normal(size=(6, d.ndofs))).cuda()
    ap = fmm.QBXApply(geo, spec, 8, 20, nrhs=nrhs)
    u = ap(x[:nrhs])
    ap.check_error_word()
    v = fmm.QBXApply(geo, spec, 8, 20, nrhs=6)(x)[:nrhs]
    assert float((u - v).abs().max() / v.abs().max()) < 5e-12
