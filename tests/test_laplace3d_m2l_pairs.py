"""3D Laplace M2L by pair at each of its thread counts (128 to 256 by the coefficients)."""

import pytest
import torch

from test_laplace3d_stages import _close_by_degree, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [13, 14, 15, 16, 17, 18, 19, 20])
def test_m2l_by_pair(p):
    w, o, s = _setup(2, p, 1.0, 0.0)
    w._translations = None
    mp, lo = o.zeros_box_exps(), o.zeros_box_exps()
    o.stage("form_multipoles", s, mp)
    o.stage("coarsen_multipoles", mp)
    o.stage("multipole_to_local", mp, lo)
    x = torch.from_numpy(mp).cuda()
    _close_by_degree(w.multipole_to_local(None, None, None, None, None, x), lo, p)
