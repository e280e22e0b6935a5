"""The plane transforms of the PME solve at every kind of grid side: small ones, primes (one long
radix), a large prime factor beside a small one, squares, both sides of the sizes that go to
cuFFT; and the lane splits of the spread and the gather at atom counts around a pass.

The oracle is numpy's FFT in float64. FP64: 1e-11 (energy) and 1e-9 of the largest component, the
bounds of the other PME tests. FP32: every value is a sum of ~216 products of FP32 splines and a
grid transformed in FP32, about 6e-8 sqrt(2 R) each for radices R up to 100: 2e-5 of the largest.
"""
import numpy as np
import pytest
import torch

from gpu_util import rel, rel_max, t
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# A half spectrum and a full one differ at the Nyquist frequency of an even K in a sheared box (the
# influence function of k and of its mirror image are not equal there), which coarse grids show:
# even sides are checked in an orthorhombic box.
BOXES = (np.diag([2.4, 2.2, 2.5]), np.array([[2.4, 0.0, 0.0], [0.3, 2.2, 0.0], [-0.2, 0.4, 2.5]]))


def _case(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.random((n, 3)) * 1.6 - 0.3  # in box lengths: some atoms outside the primary cell
    q = rng.standard_normal(n)
    return x, q - q.mean()


def _check(x, q, K, alpha, dtype, etol, gtol):
    from torchff_b200.pme import PME

    box = BOXES[K % 2]
    x = x @ box
    if dtype == torch.float32:
        x, q, box = (a.astype(np.float32).astype(np.float64) for a in (x, q, box))
    e0, gx0, pot0, _ = O.pme(x, box, q, alpha, K)
    pme = PME(alpha, K, 0, use_customized_ops=True).cuda()
    xt, qt = t(x, dtype, True), t(q, dtype, True)
    e = pme(xt, t(box, dtype), qt)
    e.backward()
    assert rel(e.item(), e0) < etol
    assert rel_max(xt.grad, gx0) < gtol and rel_max(qt.grad, pot0) < gtol


# 6 2x3, 7 prime, 8 2x4, 16 4x4, 17 prime, 34 2x17, 48 6x8, 49 7x7, 64 8x8, 75 5x15, 78 6x13 (the last side
# of the planes); cuFFT: 37 (the first with a long factor), 79, 80
@pytest.mark.parametrize("K", [6, 7, 8, 11, 13, 16, 17, 31, 34, 36, 37, 48, 49, 64, 75, 78, 79, 80])
def test_fp64_grid_sides(K):
    _check(*_case(200, K), K, 3.1, torch.float64, 1e-11, 1e-9)


@pytest.mark.parametrize("K", [6, 7, 17, 34, 36, 37, 48, 70, 75, 78, 79, 80, 97])
def test_fp32_grid_sides(K):
    _check(*_case(200, K), K, 3.1, torch.float32, 2e-5, 2e-5)


# one or two atoms feel forces near the splines' interpolation error, which FP32 does not resolve
@pytest.mark.parametrize("n,dtype,etol,gtol", [(1, torch.float64, 1e-11, 1e-7)] +
                         [(n, torch.float64, 1e-11, 1e-9) for n in (2, 3, 4, 5, 9, 33, 4097)] +
                         [(n, torch.float32, 2e-5, 2e-5) for n in (3, 4, 5, 9, 33, 4097)])
def test_atom_counts(n, dtype, etol, gtol):
    x, q = _case(n, n)
    q = q + 0.5  # one atom alone would have charge zero
    _check(x, q, 20, 3.1, dtype, etol, gtol)


@pytest.mark.parametrize("K", [8, 17, 48, 64])
def test_a_batched_grid_is_a_single_system_grid(K):
    """The batch transforms a plane with the arithmetic of a single system: reciprocal forces agree
    to the rounding of FP64 sums (the systems hold one atom per ~0.1 nm^3, no pairs, so forces
    are reciprocal ones)."""
    from torchff_b200.serving import BatchEvaluator, SystemSpec
    from torchff_b200.system import FixedChargeSystem

    rng = np.random.default_rng(K)
    specs = []
    for k in range(3):
        n = 5 + 40 * k
        q = rng.standard_normal(n)
        specs.append(SystemSpec(rng.random((n, 3)) * 6.0, np.eye(3) * 6.0, q - q.mean(), np.full(n, 0.1), np.zeros(n),
                                np.zeros((0, 2), np.int64), K if k == 1 else 12 + k))
    ev = BatchEvaluator(0.05, 3.0, torch.float64, max_systems=3, max_atoms=512, max_grid_points=300000)
    e, f = ev.evaluate(specs)
    for s, en, fn in zip(specs, e, f):
        one = FixedChargeSystem(s.charges, s.sigma, s.epsilon, s.excl_pairs, 0.05, 3.0, s.pme_grid, dtype=torch.float64)
        ref = one.evaluate(t(s.coords), t(s.box))
        assert rel(en.item(), ref["energy"].item()) < 1e-12
        assert rel_max(fn, ref["forces"]) < 1e-11
