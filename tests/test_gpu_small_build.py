"""Evaluations at atom counts around the edges of the cluster build and its work items: one partly
filled cluster, one atom into the second, the last size of the one-launch build and the first of
the general one, and sizes whose work items hold one to four clusters.

Bounds of the other fused-system tests. FP64: energy 1e-10 relative, forces 1e-8 of the largest.
Mixed: energy 1e-6 of the summed component magnitudes, forces 1e-5 RMS.
"""
import numpy as np
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


# 592 clusters, the last size whose slot parameters are written beside the neighbour search, and 593
@pytest.mark.parametrize("n", [6314, 6315])
def test_slot_parameters_beside_and_after_the_search(n):
    from oracle import oracle as O
    from torchff_b200.system import FixedChargeSystem
    from torchff_b200.water import serving_water_box

    wb, k = serving_water_box(n, n), 138.935456
    pair = (wb.coords, wb.box, wb.charges, wb.atom_types, wb.sigma_table, wb.epsilon_table, wb.coulomb_exclusions,
            wb.cutoff, wb.alpha, k)
    subset = np.random.default_rng(n).choice(wb.natoms, 128, replace=False)
    e_pme, g_pme = O.pme_subset(wb.coords, wb.box, wb.charges, wb.alpha, wb.grid, subset)
    g = O.real_space_grad_subset(*pair, subset) + k * g_pme
    e_real = O.real_space_cells(*pair)
    s64 = FixedChargeSystem.from_water_box(wb, dtype=torch.float64)
    out = s64.evaluate(t(wb.coords), t(wb.box))
    assert abs(out["energy"].item() - (e_real + k * e_pme)) < 1e-12 * (abs(e_real) + abs(k * e_pme))
    assert np.max(np.abs(-out["forces"].cpu().numpy()[subset] - g)) < 1e-8 * np.max(np.abs(g))
    # mixed against FP64 on the same rounded coordinates
    x32, b32 = t(wb.coords, torch.float32), t(wb.box, torch.float32)
    ref = s64.evaluate(x32.double(), b32.double(), terms=True)
    out = FixedChargeSystem.from_water_box(wb, dtype=torch.float32).evaluate(x32, b32)
    assert abs(out["energy"].item() - ref["energy"].item()) < 1e-6 * float(ref["terms"].abs().sum())
    assert rel_rms(out["forces"], ref["forces"].cpu().numpy()) < 1e-5
