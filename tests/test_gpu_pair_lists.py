"""Pair-list kernels at the sizes and orders where their work split can go wrong: rows that share
atoms in runs (either column), scattered and repeated rows, -1 rows, warp and block remainders,
rows off a 16-byte boundary.

Energies and gradients are compared with a float64 numpy sum over the rows. FP64: 1e-12 of the
largest gradient magnitude (sums of up to ~4000 terms of one size in another order: 4000 x
1.1e-16 = 4.4e-13). FP32: 2e-5 of it (a pair term takes about ten FP32 roundings of 6e-8, its
12th power of sigma/r multiplies the distance's by 13; the sums are exact).
"""
import numpy as np
import pytest
import torch

from gpu_util import t

pytestmark = pytest.mark.gpu

K, RC, L = 138.935456, 1.0, 2.4


def _atoms(n, seed):
    """n atoms on a jittered lattice (no two closer than ~0.2 nm), every third with epsilon 0."""
    rng = np.random.default_rng(seed)
    s = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(s)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(s ** 3)[:n]]
    d = L / s
    x = (g + 0.5) * d + rng.uniform(-0.1, 0.1, (n, 3)) * d
    eps = rng.uniform(0.3, 0.8, n)
    eps[::3] = 0.0
    return x, rng.uniform(-0.8, 0.8, n), rng.uniform(0.1, 0.2, n), eps


def _reference(x, q, sig, eps, pairs, shift=True):
    p = pairs[(pairs >= 0).all(1)]
    i, j = p[:, 0], p[:, 1]
    d = x[i] - x[j]
    d -= L * np.floor(d / L + 0.5)
    r2 = (d * d).sum(1)
    ok = r2 <= RC * RC
    i, j, d, r2 = i[ok], j[ok], d[ok], r2[ok]
    r = np.sqrt(r2)
    f = 1 / r - (1 / RC if shift else 0.0)
    s, e = 0.5 * (sig[i] + sig[j]), np.sqrt(eps[i] * eps[j])
    s6 = (s / r) ** 6
    energy = np.sum(K * q[i] * q[j] * f + 4 * e * s6 * (s6 - 1))
    dr = (-K * q[i] * q[j] / r2 - 24 * e * s6 * (2 * s6 - 1) / r) / r
    gx, gq, gs, ge = np.zeros_like(x), np.zeros(len(q)), np.zeros(len(q)), np.zeros(len(q))
    np.add.at(gx, i, dr[:, None] * d)
    np.add.at(gx, j, -dr[:, None] * d)
    np.add.at(gq, i, K * q[j] * f)
    np.add.at(gq, j, K * q[i] * f)
    ds = 12 * e * s6 * (2 * s6 - 1) / s
    de = np.where(e > 0, 4 * s6 * (s6 - 1) / (2 * np.where(e > 0, e, 1)), 0.0)
    for a, b in ((i, j), (j, i)):
        np.add.at(gs, a, ds)
        np.add.at(ge, a, de * eps[b])
    return energy, gx, gq, gs, ge


def _rows(n, order, seed):
    rng = np.random.default_rng(seed)
    i, j = np.tril_indices(n, -1)
    p = np.stack([i, j], 1)
    if order == "by_j":
        p = p[np.lexsort((p[:, 0], p[:, 1]))]
    elif order == "swapped":
        p = p[:, ::-1]
    elif order == "mixed_columns":
        flip = rng.random(len(p)) < 0.5
        p = np.where(flip[:, None], p[:, ::-1], p)
    elif order == "scattered":
        p = p[rng.permutation(len(p))]
    elif order == "repeated":
        p = np.repeat(p[rng.permutation(len(p))[: len(p) // 4]], 3, axis=0)
    elif order == "padded":
        p[rng.random(len(p)) < 0.3] = -1
        p = np.concatenate([p, np.full((77, 2), -1)])
    return np.ascontiguousarray(p)


ORDERS = ["by_i", "by_j", "swapped", "mixed_columns", "scattered", "repeated", "padded"]


@pytest.mark.parametrize("order", ORDERS)
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [2, 9, 33, 90])
def test_nonbonded_sums_do_not_depend_on_the_row_order(n, dtype, order):
    from torchff_b200 import compute_nonbonded_energy_from_atom_pairs as f

    pairs = _rows(n, order, 3)
    x, q, sig, eps = (a.astype(np.float32).astype(np.float64) if dtype == torch.float32 else a for a in _atoms(n, n))
    args = [t(a, dtype, True) for a in (x, sig, eps, q)]
    e = f(args[0], t(pairs, torch.int64), t(np.eye(3) * L, dtype), args[1], args[2], args[3], K, RC, True)
    e.backward()
    ref = _reference(x, q, sig, eps, pairs)
    tol = 1e-12 if dtype == torch.float64 else 2e-5
    got = [args[0].grad, args[3].grad, args[1].grad, args[2].grad]
    for a, b in zip(got, ref[1:]):
        assert np.max(np.abs(a.double().cpu().numpy() - b)) <= tol * max(np.max(np.abs(b)), 1.0)
    scale = np.abs(ref[1]).sum() * RC + 1.0  # every pair term is below its force times the cutoff
    assert abs(e.item() - ref[0]) <= tol * scale


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("rows", [0, 1, 31, 32, 33, 255, 257, 4005])
def test_row_remainders_and_unaligned_rows(rows, dtype):
    from torchff_b200 import compute_coulomb_energy

    x, q, sig, eps = _atoms(90, 5)
    pairs = _rows(90, "scattered", 1)[:rows]
    flat = torch.full((2 * rows + 1,), -1, dtype=torch.int64, device="cuda")
    flat[1:] = t(pairs, torch.int64).reshape(-1)
    xt, qt = t(x, dtype, True), t(q, dtype, True)
    e = compute_coulomb_energy(xt, flat[1:].view(-1, 2), t(np.eye(3) * L, dtype), qt, K, RC, True)
    e.backward()
    xr, qr = (a.detach().double().cpu().numpy() for a in (xt, qt))
    ref = _reference(xr, qr, sig, np.zeros_like(eps), pairs)
    tol = 1e-12 if dtype == torch.float64 else 2e-5
    assert np.max(np.abs(xt.grad.double().cpu().numpy() - ref[1])) <= tol * max(np.max(np.abs(ref[1])), 1.0)
    assert np.max(np.abs(qt.grad.double().cpu().numpy() - ref[2])) <= tol * max(np.max(np.abs(ref[2])), 1.0)


def test_fp32_gradients_are_the_same_bits_in_any_row_order():
    from torchff_b200 import compute_nonbonded_energy_from_atom_pairs as f

    x, q, sig, eps = _atoms(90, 2)
    out = []
    for order in ("by_i", "by_j", "scattered"):
        xt = t(x, torch.float32, True)
        f(xt, t(_rows(90, order, 4), torch.int64), t(np.eye(3) * L, torch.float32), t(sig, torch.float32),
          t(eps, torch.float32), t(q, torch.float32), K, RC, True).backward()
        out.append(xt.grad)
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
