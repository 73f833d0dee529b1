"""3D Helmholtz: multipoles straight to the QBX targets, against the same apply through
the QBX expansions (the wrangler's M2QBXL and QBXL2P stages)."""

import numpy as np
import pytest
import torch

from pytential_b200.discretization import make_ellipsoid
from pytential_b200.geometry import QBXFMMGeometryData

pytestmark = pytest.mark.gpu


def _geometry(kind):
    d = make_ellipsoid(1)
    c, r = d.interleaved_centers()
    targets = [(d.nodes, +1)]
    if kind == "many":          # several targets per center, some at the center itself
        targets += [(d.nodes + 0.3 * r[0::2] * d.normals, +2), (c[:, 1::2].copy(), +2),
                    (d.nodes[:, :37].copy(), -1)]
    return d, QBXFMMGeometryData(d, targets, max_leaf_refine_weight=64)


@pytest.mark.parametrize("kind,q,p,nrhs,k,backend", [
    ("plain", 5, 15, 16, 10.0, "sumpy"), ("plain", 5, 17, 17, 3.0, "sumpy"),
    ("plain", 0, 3, 1, 2.0, "sumpy"), ("plain", 1, 1, 2, 2.0, "sumpy"),
    ("many", 2, 6, 3, 4.0, "sumpy"), ("many", 3, 8, 5, 4.0, "sumpy"),
    ("many", 4, 11, 8, 4.0, "sumpy"), ("many", 5, 12, 9, 1e-3, "sumpy"),
    ("plain", 5, 15, 1, 10.0, "fmmlib"), ("many", 4, 13, 6, 6.0, "fmmlib"),
    ("many", 3, 10, 2, 0.5, "fmmlib"), ("plain", 0, 5, 4, 2.0, "fmmlib"),
])
def test_multipoles_to_targets(kind, q, p, nrhs, k, backend):
    from pytential_b200 import fmm
    d, geo = _geometry(kind)
    assert sum(len(s.lists) for s in geo.traversal().from_sep_smaller_by_level) > 0
    spec = fmm.SourceKernelSpec(fmm.HelmholtzKernel(3, k), charge_coeff=-1j * k, dipole_coeff=1.0)
    rng = np.random.default_rng(5)
    dens = rng.normal(size=(nrhs, d.ndofs)) + 1j * rng.normal(size=(nrhs, d.ndofs))
    ap = fmm.QBXApply(geo, spec, q, p, nrhs=nrhs, fmm_backend=backend)
    u = ap(torch.from_numpy(dens).cuda())
    ap.check_error_word()
    w = fmm.B200QBXExpansionWrangler(
        fmm.B200TreeIndependentDataForWrangler(spec), geo, np.complex128, q,
        lambda kern, args, tree, lev: p, _use_target_specific_qbx=True, nrhs=nrhs,
        fmm_backend=backend)
    s = d.upsample_density(dens) * d.quad_weights
    v = fmm.drive_fmm(None, w, [torch.from_numpy(s).cuda()])
    err = float((u - v).abs().max() / v.abs().max())
    # both sum the same terms in float64, a few thousand per target
    assert err < 1e-12, err
