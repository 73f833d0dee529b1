"""3D Laplace stage kernels at the edges of their orders, against the checker's stages."""

import functools

import numpy as np
import pytest
import torch

from oracle.oracle import Oracle
from pytential_b200 import fmm
from pytential_b200.discretization import make_ellipsoid
from pytential_b200.geometry import QBXFMMGeometryData

pytestmark = pytest.mark.gpu

# float64 sums of at most a few thousand terms per output, as for every stage
TOL = 1e-12


@functools.lru_cache(maxsize=None)
def _geometry():
    d = make_ellipsoid(1)
    rng = np.random.default_rng(2)
    v = rng.normal(size=(3, 45))
    far = 3.0 * v / np.linalg.norm(v, axis=0)
    return d, QBXFMMGeometryData(d, [(d.nodes, +1), (far, 0)], max_leaf_refine_weight=64)


def _setup(q, p, cq, cd, nrhs=1, tsqbx=False):
    d, geo = _geometry()
    spec = fmm.SourceKernelSpec(fmm.LaplaceKernel(3), charge_coeff=cq, dipole_coeff=cd)
    w = fmm.B200QBXExpansionWrangler(
        fmm.B200TreeIndependentDataForWrangler(spec), geo, np.float64, q,
        lambda kern, args, tree, lev: p, _use_target_specific_qbx=tsqbx, nrhs=nrhs)
    o = Oracle(geo, dim=3, qbx_order=q, fmm_order=p, nrhs=nrhs, charge_coeff=cq, dipole_coeff=cd)
    s = o.tree_strengths(np.random.default_rng(3).normal(size=(nrhs, d.nquad)))
    return w, o, s


def _close(got, want):
    got = got.cpu().numpy()
    assert np.abs(want).max() > 0
    assert np.abs(got - want).max() <= TOL * np.abs(want).max()


@pytest.mark.parametrize("q", range(9))
@pytest.mark.parametrize("cq,cd", [(1.0, 0.0), (0.0, 1.0), (0.7, -1.3)])
def test_target_specific_near_field(q, cq, cd):
    """The polynomial form against the expansions formed from the same sources."""
    w, o, s = _setup(q, 5, cq, cd, nrhs=2, tsqbx=True)
    got = w.eval_target_specific_qbx_locals(None, [torch.from_numpy(s).cuda()])
    qe, want = o.zeros_qbx_exps(), o.zeros_tree_pot()
    o.stage("form_global_qbx_locals", s, qe)
    o.stage("eval_qbx_expansions", qe, want)
    _close(got, want)


@pytest.mark.parametrize("p", [1, 2, 5, 6, 7, 10, 11, 13, 14, 19, 20])
@pytest.mark.parametrize("cq,cd", [(1.0, 0.0), (0.7, -1.3)])
def test_form_locals(p, cq, cd):
    w, o, s = _setup(2, p, cq, cd)
    got = w.form_locals(None, None, None, None, None, [torch.from_numpy(s).cuda()])
    want = o.zeros_box_exps()
    o.stage("form_locals", s, want)
    _close(got, want)


@pytest.mark.parametrize("q,p", [(0, 1), (0, 20), (1, 7), (2, 2), (3, 10), (4, 12), (5, 3),
                                 (6, 15), (7, 5), (8, 20)])
def test_multipoles_to_qbx_locals(q, p):
    w, o, s = _setup(q, p, 1.0, 0.5, nrhs=2)
    mp = o.zeros_box_exps()
    o.stage("form_multipoles", s, mp)
    o.stage("coarsen_multipoles", mp)
    got = w.translate_box_multipoles_to_qbx_local(None, torch.from_numpy(mp).cuda())
    want = o.zeros_qbx_exps()
    o.stage("translate_box_multipoles_to_qbx_local", mp, want)
    _close(got, want)


def _close_by_degree(got, want, p):
    """Box expansions: every degree against its own largest coefficient."""
    got = got.cpu().numpy()
    for n in range(p + 1):
        i = slice(n * (n + 1) // 2, (n + 1) * (n + 2) // 2)
        scale = np.abs(want[..., i]).max()
        assert scale > 0
        assert np.abs(got[..., i] - want[..., i]).max() <= TOL * scale, n


@pytest.mark.parametrize("p", [1, 10, 14, 15, 20])
@pytest.mark.parametrize("matrices", [False, True])
def test_translations(p, matrices):
    w, o, s = _setup(2, p, 1.0, 0.0)
    assert w._translations is not None
    if not matrices:
        w._translations = None
    mp = o.zeros_box_exps()
    o.stage("form_multipoles", s, mp)
    _close_by_degree(w.form_multipoles(None, None, None, [torch.from_numpy(s).cuda()]), mp, p)
    x = torch.from_numpy(mp.copy()).cuda()
    o.stage("coarsen_multipoles", mp)
    _close_by_degree(w.coarsen_multipoles(None, None, None, x), mp, p)
    lo = o.zeros_box_exps()
    o.stage("multipole_to_local", mp, lo)
    x = torch.from_numpy(mp).cuda()
    _close_by_degree(w.multipole_to_local(None, None, None, None, None, x), lo, p)
    x = torch.from_numpy(lo.copy()).cuda()
    o.stage("refine_locals", lo)
    _close_by_degree(w.refine_locals(None, None, None, x), lo, p)


@pytest.mark.parametrize("p", range(11, 21))
def test_apply_orders(p):
    """The whole apply: translations by class matrices, whose row groups change with p."""
    d = make_ellipsoid(1)
    geo = QBXFMMGeometryData(d, [(d.nodes, +1)], max_leaf_refine_weight=64)
    ap = fmm.QBXApply(geo, fmm.SourceKernelSpec(fmm.LaplaceKernel(3), charge_coeff=1.0), 2, p)
    o = Oracle(geo, dim=3, qbx_order=2, fmm_order=p, nrhs=1, charge_coeff=1.0)
    dens = np.random.default_rng(3).normal(size=(1, d.ndofs))
    want = o.apply(o.tree_strengths(d.upsample_density(dens) * d.quad_weights))
    _close(ap(torch.from_numpy(dens).cuda()), want)
