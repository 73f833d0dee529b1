"""Transposed 3D apply with the rows of M2QBXL^T split over four, two and one CTA (the rule
counts rows times densities), for each number of row tiles of its product."""

import numpy as np
import pytest
import torch

from helpers import relerr
from oracle.oracle import Oracle
from pytential_b200 import abi
from pytential_b200.discretization import make_ellipsoid
from pytential_b200.fmm import LaplaceKernel, QBXApply, SourceKernelSpec
from pytential_b200.geometry import QBXFMMGeometryData
from pytential_b200.transpose import QBXTransposeApply

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("q,p", [(1, 3), (3, 7), (4, 12), (5, 8), (8, 10)])
@pytest.mark.parametrize("least,below", [(0, 222), (222, 518), (518, 10 ** 9)])
def test_split(q, p, least, below):
    d = make_ellipsoid(1)
    geo = QBXFMMGeometryData(d, [(d.nodes, +1)], max_leaf_refine_weight=128)
    spec = SourceKernelSpec(LaplaceKernel(3), charge_coeff=1.0)
    rows = QBXTransposeApply(QBXApply(geo, spec, q, p)).index.nlist3_rows
    nrhs = max(1, -(-least // rows))
    assert least <= rows * nrhs < below
    tr = QBXTransposeApply(QBXApply(geo, spec, q, p, nrhs=nrhs))
    r = np.random.default_rng(q).normal(size=(nrhs, d.ndofs))
    got = tr.kernel_transpose(torch.from_numpy(r).cuda()).cpu().numpy()
    tr.check_error_word()
    o = Oracle(geo, dim=3, qbx_order=q, fmm_order=p, nrhs=nrhs, charge_coeff=1.0,
               family=abi.QBXFMM_LAPLACE)
    ref = o.apply_transpose(r)[:, np.argsort(o.arrays["user_source_ids"][:o.scalars["nsources"]])]
    # float64 sums of a few thousand terms, as for every stage
    assert relerr(got, ref) < 1e-12
