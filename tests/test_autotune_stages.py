"""The autotuner times the stages that the apply runs."""

import pytest
import torch

from helpers import workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ts,backend,precision,idle", [
    (True, "sumpy", 0, {"m2qbxl_densities", "l2qbxl_densities"}),
    (True, "fmmlib", 0, {"m2qbxl_densities"}), (False, "sumpy", 0, {"tsqbx_densities"}),
    (True, "sumpy", 1, set())])
def test_stages(ts, backend, precision, idle):
    from pytential_b200.autotune import KNOBS, autotune
    from pytential_b200.fmm import QBXApply
    wl = workload("h3d-CF-small")
    ap = QBXApply(wl.geometry(), wl.spec, wl.qbx_order, wl.fmm_order, nrhs=wl.nrhs,
                  target_specific_qbx=ts, fmm_backend=backend, precision=precision)
    assert set(autotune(ap, reps=1)["ms"]) == set(KNOBS) - idle
    # the stages said to be idle are: the apply's expansions stay as they were
    qe = ap._ws_tensors[3]
    qe.fill_(7.0)
    ap(torch.from_numpy(wl.density).cuda())
    assert bool((qe == 7.0).all()) == (idle >= {"m2qbxl_densities", "l2qbxl_densities"})
    # asked for by name, a knob is timed all the same
    if ts:
        assert set(autotune(ap, reps=1, knobs=["m2qbxl_densities"])["ms"]) == {"m2qbxl_densities"}
