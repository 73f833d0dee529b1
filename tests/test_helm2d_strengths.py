"""2D Helmholtz strengths (upsample, weight, reorder) for the densities a thread takes."""

import ctypes

import numpy as np
import pytest
import torch

from pytential_b200 import fmm
from pytential_b200.discretization import make_starfish
from pytential_b200.geometry import QBXFMMGeometryData

pytestmark = pytest.mark.gpu


# 1280 and 6400 sources: one density a thread below 36 000 (source, density) pairs, four below
# 400 000, then eight
@pytest.mark.parametrize("nel,nrhs", [(20, 1), (20, 2), (20, 28), (20, 29), (20, 312), (20, 313),
                                      (100, 1), (100, 5), (100, 6), (100, 62), (100, 63), (100, 64)])
def test_form_strengths(nel, nrhs):
    d = make_starfish(nel)
    geo = QBXFMMGeometryData(d, [(d.nodes, +1)])
    ap = fmm.QBXApply(geo, fmm.SourceKernelSpec(fmm.HelmholtzKernel(2, 3.0), charge_coeff=1.0), 1, 2,
                      nrhs=nrhs)
    ns = ap.dgeo.nsources
    rng = np.random.default_rng(nrhs)
    x = rng.normal(size=(nrhs, d.ndofs)) + 1j * rng.normal(size=(nrhs, d.ndofs))
    dens = torch.from_numpy(x).cuda()
    out = torch.full((nrhs, ns), float("nan"), dtype=torch.complex128, device="cuda")
    vp = ctypes.c_void_p
    ap.plan.call("qbxfmm_form_strengths", ctypes.byref(ap.up.struct), vp(dens.data_ptr()),
                 vp(out.data_ptr()), vp(torch.cuda.current_stream().cuda_stream))
    ids = ap.dgeo.host_arrays["user_source_ids"][:ns]
    want = (d.upsample_density(x) * d.quad_weights)[:, ids]
    # 16 products a value, summed in another order
    size = np.abs(x).max() * np.abs(d.upsample).sum(1).max()
    assert np.all(np.abs(out.cpu().numpy() - want) <= 40 * 2.0 ** -53 * size * d.quad_weights.max())
