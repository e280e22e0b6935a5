"""Evaluations at atom counts around the edges of the cluster build and its work items: one partly
filled cluster, one atom into the second, the last size of the one-launch build and the first of
the general one, and sizes whose work items hold one to four clusters.

Bounds of the other fused-system tests. FP64: energy 1e-10 relative, forces 1e-8 of the largest.
Mixed: energy 1e-6 of the summed component magnitudes, forces 1e-5 RMS.
"""
import pytest
import torch

from gpu_util import oracle_water, rel, rel_max, rel_rms, t

pytestmark = pytest.mark.gpu

WATERS = [10, 11, 64, 341, 342, 600, 1100]


@pytest.fixture(scope="module")
def refs():
    from torchff_b200.water import serving_water_box

    out = {}
    for n in WATERS:
        wb = serving_water_box(n, n)
        out[n] = wb, oracle_water(wb)
    return out


@pytest.mark.parametrize("n", WATERS)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_build_and_item_sizes(refs, n, dtype):
    from torchff_b200.system import FixedChargeSystem

    wb, ref = refs[n]
    sysm = FixedChargeSystem.from_water_box(wb, dtype=dtype)
    out = sysm.evaluate(t(wb.coords, dtype), t(wb.box, dtype))
    e, f = out["energy"].item(), out["forces"]
    if dtype == torch.float64:
        assert rel(e, ref["energy"]) < 1e-10
        assert rel_max(f, -ref["grad"]) < 1e-8
    else:
        assert abs(e - ref["energy"]) < 1e-6 * ref["scale"]
        assert rel_rms(f, -ref["grad"]) < 1e-5
    assert sysm.status() == 0
