"""Transposed 3D apply at the edges of its orders (tiles of eight rows (q + 1)^2, groups of
four orders M <= p + q), with few and with many list-3 boxes."""

import numpy as np
import pytest

from pytential_b200.discretization import make_ellipsoid
from pytential_b200.geometry import QBXFMMGeometryData

from helpers import relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,p,nrefine,leaf", [
    (0, 1, 1, 64), (0, 20, 1, 64), (1, 2, 1, 64), (2, 5, 1, 64), (2, 17, 1, 64), (3, 10, 2, 24),
    (4, 12, 2, 24), (4, 20, 1, 64), (5, 7, 1, 64), (6, 14, 1, 64), (7, 9, 1, 64), (8, 12, 1, 64),
    (8, 20, 1, 64)])
def test_transposed_apply(q, p, nrefine, leaf):
    import torch

    from oracle.oracle import Oracle
    from pytential_b200 import abi
    from pytential_b200.fmm import LaplaceKernel, QBXApply, SourceKernelSpec
    from pytential_b200.transpose import QBXTransposeApply
    d = make_ellipsoid(nrefine)
    geo = QBXFMMGeometryData(d, [(d.nodes, +1)], max_leaf_refine_weight=leaf)
    tr = QBXTransposeApply(QBXApply(geo, SourceKernelSpec(LaplaceKernel(3), charge_coeff=1.0), q, p))
    r = np.random.default_rng(3).normal(size=(1, d.ndofs))
    o = Oracle(geo, dim=3, qbx_order=q, fmm_order=p, nrhs=1, charge_coeff=1.0,
               family=abi.QBXFMM_LAPLACE)
    ref = o.apply_transpose(r)[:, np.argsort(o.arrays["user_source_ids"][:o.scalars["nsources"]])]
    got = tr.kernel_transpose(torch.from_numpy(r).cuda()).cpu().numpy()
    tr.check_error_word()
    # float64 sums of a few thousand terms, as for every stage
    assert relerr(got, ref) < 1e-12
