"""Objects built on one stream and called on another."""

import numpy as np
import pytest
import torch

from pytential_b200 import fmm, transpose
from pytential_b200.discretization import make_starfish
from pytential_b200.geometry import QBXFMMGeometryData
from pytential_b200.workloads import laplace3d_ellipsoid

pytestmark = pytest.mark.gpu


def _problem(family, dim):
    if dim == 2:
        d = make_starfish(40)
        geo = QBXFMMGeometryData(d, [(d.nodes, +1)])
        if family == "laplace":
            return d, geo, fmm.SourceKernelSpec(fmm.LaplaceKernel(2), charge_coeff=1.0)
        return d, geo, fmm.SourceKernelSpec(fmm.HelmholtzKernel(2, 5.0), charge_coeff=-5j,
                                            dipole_coeff=1.0)
    wl = laplace3d_ellipsoid(nrefine=1, nshell=100, op="S")
    geo = wl.geometry()
    if family == "laplace":
        return geo.discr, geo, wl.spec
    return geo.discr, geo, fmm.SourceKernelSpec(fmm.HelmholtzKernel(3, 2.0), charge_coeff=-2j,
                                                dipole_coeff=1.0)


def _call(kind, geo, spec, d):
    """A constructor and a call of what it returns."""
    rng = np.random.default_rng(3)
    dens = rng.normal(size=(1, d.ndofs)) + (1j * rng.normal(size=(1, d.ndofs)) if spec.is_complex else 0)
    if kind == "transpose":
        ap = fmm.QBXApply(geo, spec, 2, 8)
        r = torch.from_numpy(rng.normal(size=(1, ap.nuser_targets))).cuda()
        return (lambda: transpose.QBXTransposeApply(ap)), (lambda o: o.kernel_transpose(r))
    if kind == "wrangler":
        s = torch.from_numpy(d.upsample_density(dens) * d.quad_weights).cuda()

        def make():
            return fmm.B200QBXExpansionWrangler(
                fmm.B200TreeIndependentDataForWrangler(spec), geo, dens.dtype, 2, lambda *a: 8)
        return make, lambda o: fmm.drive_fmm(None, o, [s])
    x = torch.from_numpy(dens).cuda()
    return (lambda: fmm.QBXApply(geo, spec, 2, 8)), lambda o: o(x)


@pytest.mark.parametrize("kind,family,dim", [
    ("wrangler", "laplace", 3), ("wrangler", "helmholtz", 2), ("apply", "laplace", 3),
    ("apply", "helmholtz", 2), ("apply", "helmholtz", 3), ("apply", "laplace", 2),
    ("transpose", "laplace", 3)])
def test_built_on_another_stream(kind, family, dim, monkeypatch):
    d, geo, spec = _problem(family, dim)
    make, call = _call(kind, geo, spec, d)
    want = call(make())
    torch.cuda.synchronize()
    plan_call = fmm.Plan.call

    def late(self, name, *args):       # the tables come 20 ms after the constructor asks for them
        if name == "qbxfmm_precompute_translations":
            torch.cuda._sleep(40_000_000)
        return plan_call(self, name, *args)
    monkeypatch.setattr(fmm.Plan, "call", late)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        obj = make()
        assert a.query()               # nothing of the constructor's is left to wait for
    with torch.cuda.stream(b):
        got = call(obj)
    torch.cuda.synchronize()
    assert torch.equal(got, want)
