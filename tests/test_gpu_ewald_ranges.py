"""FP64 screened Coulomb over both polynomial ranges and beyond them (alpha rc of 0 to 5), and their
ends, through the pair-list operator, the fused evaluation and its derivatives; small systems
whose work items hold one neighbour cluster.

Bounds are those of the other FP64 tests: energies 1e-10, gradients 1e-8 of their largest
component, second derivatives 1e-7. A dense system does not show the relative error of distant
pairs; test_gpu_ewald_sparse.py does.
"""
import math

import numpy as np
import pytest
import torch

from gpu_util import rel, rel_max, rel_rms, t
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KC = 138.935456


def _water(n=64, rc=0.6):
    from torchff_b200.water import make_water_box

    return make_water_box(n, (n / 33.4) ** (1 / 3), math.ceil(n ** (1 / 3)), cutoff=rc, grid=16, seed=3)


# (alpha rc)^2: 0, short range, its end, just past it, long range, its end, past it, far past it
Y = [0.0, 3.0, 7.0, 7.0001, 11.0, 13.5, 13.6, 25.0]


@pytest.mark.parametrize("y", Y)
def test_pair_list_ewald(y):
    from torchff_b200 import MultipolarInteraction

    wb = _water()
    alpha = math.sqrt(y) / wb.cutoff
    pairs = O.nblist_pairs(wb.coords, wb.box, wb.cutoff, *O.exclusions_coo_to_csr(wb.nblist_exclusions, wb.natoms),
                           include_self=False)
    excl = wb.coulomb_exclusions
    e0, gx0, gq0 = O.ewald_real(wb.coords, wb.box, pairs, wb.charges, wb.cutoff, alpha, KC, excl)
    x, q = t(wb.coords, grad=True), t(wb.charges, grad=True)
    e = MultipolarInteraction(0, wb.cutoff, alpha, KC).cuda()(x, t(wb.box), t(pairs, torch.int64), q,
                                                              pairs_excl=t(excl, torch.int64))
    e.backward()
    assert rel(e.item(), e0) < 1e-11
    assert rel_max(x.grad, gx0) < 1e-10 and rel_max(q.grad, gq0) < 1e-10


@pytest.mark.parametrize("y", Y[1:])
def test_fused_fp64(y):
    from torchff_b200.system import FixedChargeSystem

    wb = _water()
    wb.alpha = math.sqrt(y) / wb.cutoff
    ref = O.fixed_charge_energy(wb.coords, wb.box, wb.charges, wb.sigma_table, wb.epsilon_table, wb.atom_types,
                                wb.nblist_exclusions, wb.coulomb_exclusions, wb.cutoff, wb.alpha, wb.grid, KC)
    sy = FixedChargeSystem.from_water_box(wb, dtype=torch.float64)
    for out in (sy.evaluate(t(wb.coords), t(wb.box), grad_charges=True), sy.evaluate_grads(t(wb.coords), t(wb.box))):
        assert rel(out["energy"].item(), ref["total"]) < 1e-10
        assert rel_max(out["forces"], -ref["grad_coords"]) < 1e-8
        assert rel_max(out["grad_charges"], ref["grad_charges"]) < 1e-8


@pytest.mark.parametrize("y", [3.0, 11.0, 25.0])
def test_hessian_vector_products(y):
    """Derivatives of u . dE/dx against double differentiation of the float64 torch oracle."""
    from oracle import torch_energy as TE
    from torchff_b200.system import FixedChargeSystem

    wb = _water()
    wb.alpha = math.sqrt(y) / wb.cutoff
    u = np.random.default_rng(1).normal(size=wb.coords.shape)
    pairs = O.nblist_pairs(wb.coords, wb.box, wb.cutoff, *O.exclusions_coo_to_csr(wb.nblist_exclusions, wb.natoms))
    leaf = {k: torch.tensor(a, requires_grad=True) for k, a in
            (("coords", wb.coords), ("charges", wb.charges), ("sigma", wb.sigma))}
    energy = TE.fixed_charge_energy(leaf["coords"], torch.tensor(wb.box), leaf["charges"], leaf["sigma"],
                                    torch.tensor(wb.epsilon), torch.tensor(pairs), torch.tensor(wb.coulomb_exclusions),
                                    wb.cutoff, wb.alpha, wb.grid)
    (gx,) = torch.autograd.grad(energy, leaf["coords"], create_graph=True)
    ref = dict(zip(leaf, torch.autograd.grad((gx * torch.tensor(u)).sum(), list(leaf.values()))))
    hv = FixedChargeSystem.from_water_box(wb, dtype=torch.float64).hvp(t(wb.coords), t(wb.box), t(u))
    for k, v in ref.items():
        assert rel_max(hv[k], v) < 1e-7, k


@pytest.mark.parametrize("n", [1, 10, 11, 43, 216, 500])
@pytest.mark.parametrize("y", [6.9, 10.0, 20.0])
def test_small_mixed_systems(n, y):
    """FP32 real space of systems with few clusters (items of one neighbour cluster) and the FP64
    exclusion correction in every range. Energy within 1e-6 of the summed magnitudes of its terms and
    force RMS within 1e-5, the bounds of the other mixed tests; a lone water's forces, which are what two
    terms of 5300 kJ/mol/nm leave, within 1e-6 of those. Exclusion energy within 1e-6: a coordinate of up to
    2.5 nm is rounded by 1.5e-7 nm, 1.5e-6 of an O-H distance, and erf(alpha r) / r, alpha r up to 1.13,
    changes by at most 0.6 of that."""
    from torchff_b200.system import FixedChargeSystem

    wb = _water(max(n, 10))
    if n < 10:  # the first waters of the box
        m = 3 * n
        for k in ("coords", "charges", "sigma", "epsilon", "atom_types"):
            setattr(wb, k, getattr(wb, k)[:m])
        wb.nblist_exclusions = wb.nblist_exclusions[: 9 * n]
        wb.coulomb_exclusions = wb.coulomb_exclusions[: 3 * n]
        wb.n_waters = n
    wb.alpha = math.sqrt(y) / wb.cutoff
    wb.coords = wb.coords.astype(np.float32).astype(np.float64)
    wb.box = wb.box.astype(np.float32).astype(np.float64)
    ref = O.fixed_charge_energy(wb.coords, wb.box, wb.charges, wb.sigma_table, wb.epsilon_table, wb.atom_types,
                                wb.nblist_exclusions, wb.coulomb_exclusions, wb.cutoff, wb.alpha, wb.grid, KC)
    out = FixedChargeSystem.from_water_box(wb, dtype=torch.float32).evaluate(
        t(wb.coords, torch.float32), t(wb.box, torch.float32), terms=True)
    scale = abs(ref["lj"]) + abs(ref["coul_real"]) + abs(KC * ref["pme_raw"])
    assert abs(out["energy"].item() - ref["total"]) < 1e-6 * scale
    if n == 1:
        assert np.abs(out["forces"].double().cpu().numpy() + ref["grad_coords"]).max() < 1e-6 * 5300.0
    else:
        assert rel_rms(out["forces"], -ref["grad_coords"]) < 1e-5
    i, j = wb.coulomb_exclusions.T
    r = np.linalg.norm(O.min_image(wb.coords[i] - wb.coords[j], wb.box), axis=1)
    excl = -KC * sum(qq * math.erf(wb.alpha * rr) / rr for qq, rr in zip(wb.charges[i] * wb.charges[j], r))
    assert rel(out["terms"][1].item(), excl) < 1e-6
