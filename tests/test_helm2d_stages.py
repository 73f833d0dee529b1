"""2D Helmholtz: M2M / M2L / L2L at the edges of their orders and density counts, and the
expansions taken straight to the QBX targets."""

import functools

import numpy as np
import pytest
import torch
from scipy.special import gammaln, hankel1, jv

from pytential_b200 import fmm
from pytential_b200.discretization import make_starfish
from pytential_b200.geometry import QBXFMMGeometryData

pytestmark = pytest.mark.gpu


@functools.lru_cache(maxsize=None)
def _geometry(kind="plain"):
    d = make_starfish(20)
    rng = np.random.default_rng(2)
    targets = [(d.nodes, +1)]
    if kind == "plain":
        targets.append((rng.uniform(-2, 2, size=(2, 60)), 0))
    else:                       # several targets per center, some at the center itself
        c, r = d.interleaved_centers()
        targets += [(d.nodes + 0.3 * r[0::2] * d.normals, +2), (c[:, 1::2].copy(), +2),
                    (d.nodes[:, :37].copy(), -1)]
    return d, QBXFMMGeometryData(d, targets, max_leaf_refine_weight=32)


def _wrangler(geo, spec, q, p, nrhs):
    return fmm.B200QBXExpansionWrangler(
        fmm.B200TreeIndependentDataForWrangler(spec), geo, np.complex128, q,
        lambda kern, args, tree, lev: p, _use_target_specific_qbx=True, nrhs=nrhs)


def _pairs(geo, kind):
    """(source box, target box) of a translation stage, level by level."""
    tree, trav = geo.tree(), geo.traversal()
    if kind == "l2":
        st, li = trav.from_sep_siblings_starts, trav.from_sep_siblings_lists
        return [[(s, t) for i, t in enumerate(trav.target_or_target_parent_boxes)
                 for s in li[st[i]:st[i + 1]]]]
    par, lev = tree.box_parent_ids, tree.box_levels
    if kind == "up":
        ok = tree.box_source_counts_cumul > 0
        return [[(b, par[b]) for b in np.flatnonzero(ok & (lev == n))]
                for n in range(tree.nlevels - 1, 0, -1)]
    ok = np.zeros(tree.nboxes, bool)
    ok[trav.target_or_target_parent_boxes] = True
    return [[(par[b], b) for b in np.flatnonzero(ok & (lev == n))] for n in range(1, tree.nlevels)]


def _translate(geo, k, p, kind, exps):
    """out_m = sum of Z_{n-m}(c_out - c_in) in_n over the pairs, in the widths' scaling, and
    the sums of the terms' sizes (J's bound (x/2)^n / n! for the shifts)."""
    tree = geo.tree()
    n = np.arange(-p, p + 1)
    out = exps.copy() if kind != "l2" else np.zeros_like(exps)
    size = np.abs(out)
    for level in _pairs(geo, kind):
        for s, t in level:
            u = tree.box_centers[:, t] - tree.box_centers[:, s]
            x, th = k * np.hypot(*u), np.arctan2(u[1], u[0])
            m = n[:, None] - n[None, :]                   # [in n, out m]
            Z = hankel1(m, x) if kind == "l2" else jv(m, x)
            am = np.abs(m)
            B = np.abs(Z) if kind == "l2" else np.exp(am * np.log(x / 2) - gammaln(am + 1))
            ws, wt = tree.level_width(tree.box_levels[s]), tree.level_width(tree.box_levels[t])
            fin = ws ** (-np.abs(n) if kind == "down" else np.abs(n)).astype(float)
            fout = wt ** (-np.abs(n) if kind == "up" else np.abs(n)).astype(float)
            F = fin[:, None] * fout[None, :]
            out[t] += out[s] @ (F * Z * np.exp(1j * m * th)) if kind != "l2" else \
                exps[s] @ (F * Z * np.exp(1j * m * th))
            size[t] += (size[s] if kind != "l2" else np.abs(exps[s])) @ (F * B)
    return out, size


@pytest.mark.parametrize("p,nrhs", [(1, 1), (3, 3), (4, 5), (7, 4), (8, 9), (10, 8), (12, 16),
                                    (15, 17), (16, 2), (19, 40), (20, 1), (20, 33)])
@pytest.mark.parametrize("kind", ["up", "l2", "down"])
@pytest.mark.parametrize("tables", [False, True])
def test_translations(p, nrhs, kind, tables):
    k = 6.0
    d, geo = _geometry()
    spec = fmm.SourceKernelSpec(fmm.HelmholtzKernel(2, k), charge_coeff=-1j * k, dipole_coeff=1.0)
    w = _wrangler(geo, spec, 2, p, nrhs)
    assert w._translations is not None
    if not tables:
        w._translations = None
    rng = np.random.default_rng(p)
    shape = (geo.tree().nboxes, nrhs, 2 * p + 1)
    e = rng.normal(size=shape) + 1j * rng.normal(size=shape)
    if kind == "up":
        e[geo.tree().box_source_counts_cumul == 0] = 0
    want, size = _translate(geo, k, p, kind, e)
    x = torch.from_numpy(e).cuda()
    got = {"up": lambda: w.coarsen_multipoles(None, None, None, x),
           "l2": lambda: w.multipole_to_local(None, None, None, None, None, x),
           "down": lambda: w.refine_locals(None, None, None, x)}[kind]()
    got = got.cpu().numpy()
    assert np.abs(want).max() > 0
    # both sides: float64 sums of at most 2p + 1 terms over up to 30 boxes on a handful of
    # levels, tables by recurrences of up to 4p steps on one side, phases of 2p products:
    # (2p + 30 + 4p + 2p) roundings of a term's size, a few levels
    assert np.all(np.abs(got - want) <= 4 * (8 * p + 30) * 2.0 ** -53 * size)


@pytest.mark.parametrize("kind,q,p,nrhs,k", [
    ("plain", 5, 20, 40, 20.0), ("plain", 0, 3, 1, 2.0), ("plain", 1, 1, 2, 2.0),
    ("many", 2, 6, 3, 4.0), ("many", 3, 8, 5, 1e-2), ("many", 4, 13, 9, 8.0),
    ("plain", 6, 16, 4, 8.0), ("many", 7, 19, 17, 8.0), ("many", 8, 12, 8, 8.0)])
def test_expansions_to_targets(kind, q, p, nrhs, k):
    """The apply against the wrangler's M2QBXL, L2QBXL and QBXL2P stages."""
    d, geo = _geometry(kind)
    assert sum(len(s.lists) for s in geo.traversal().from_sep_smaller_by_level) > 0
    spec = fmm.SourceKernelSpec(fmm.HelmholtzKernel(2, k), charge_coeff=-1j * k, dipole_coeff=1.0)
    rng = np.random.default_rng(5)
    dens = rng.normal(size=(nrhs, d.ndofs)) + 1j * rng.normal(size=(nrhs, d.ndofs))
    ap = fmm.QBXApply(geo, spec, q, p, nrhs=nrhs)
    u = ap(torch.from_numpy(dens).cuda())
    ap.check_error_word()
    w = _wrangler(geo, spec, q, p, nrhs)
    s = d.upsample_density(dens) * d.quad_weights
    v = fmm.drive_fmm(None, w, [torch.from_numpy(s).cuda()])
    err = float((u - v).abs().max() / v.abs().max())
    # the same terms in float64; sums of order-p Hankel terms larger than their result
    assert err < 5e-12, err
