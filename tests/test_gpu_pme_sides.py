"""Grid sides of a batch that single systems leave to cuFFT (above 78, and above 36 with a long prime factor), and
even sides in a sheared box, where the transform works on half a spectrum.

The oracle is numpy's FFT in float64. FP64: 1e-11 (energy) and 1e-9 of the largest component. FP32: 2e-5 of the
largest, the bound of the other transform tests (radices up to 100); direct sums of K terms, as for K = 89, stay
below it too (6e-8 sqrt(2 K) = 8e-7 each).
"""
import math

import numpy as np
import pytest
import torch

from gpu_util import rel, rel_max, t
from oracle import oracle as O

pytestmark = pytest.mark.gpu


# 37, 53, 61, 89: one prime radix; 79: the first side above the planes of a single system; 96: the last
@pytest.mark.parametrize("dtype,sides", [(torch.float32, (37, 53, 79)), (torch.float32, (89, 96)),
                                         (torch.float64, (37, 53, 61)), (torch.float64, (58, 64))])
def test_batched_sides(dtype, sides):
    """Point charges without pairs in one batch, a side of 8 first and last: reciprocal energy and
    forces alone."""
    from torchff_b200.serving import BatchEvaluator, SystemSpec

    rng = np.random.default_rng(sides[0])
    alpha, specs = 3.0, []
    for k, K in enumerate((8, *sides, 8)):
        n = 40 + 37 * k
        # odd sides in a sheared box
        box = np.diag([6.0, 6.2, 5.9]) + (np.array([[0, 0, 0], [0.5, 0, 0], [-0.4, 0.7, 0]]) if K % 2 else 0.0)
        q = rng.standard_normal(n)
        x, q = rng.random((n, 3)) @ box, q - q.mean()
        if dtype == torch.float32:
            x, q, box = (a.astype(np.float32).astype(np.float64) for a in (x, q, box))
        specs.append(SystemSpec(x, box, q, np.full(n, 0.1), np.zeros(n), np.zeros((0, 2), np.int64), K))
    ev = BatchEvaluator(0.01, alpha, dtype, max_systems=len(specs), max_atoms=2048,
                        max_grid_points=sum(s.pme_grid ** 3 for s in specs), coul_constant=1.0)
    e, f = ev.evaluate(specs)
    etol, gtol = (2e-5, 2e-5) if dtype == torch.float32 else (1e-11, 1e-9)
    for s, en, fn in zip(specs, e, f):
        e0, gx0 = O.pme(s.coords, s.box, s.charges, alpha, s.pme_grid)[:2]
        assert rel(en.item(), e0) < etol, s.pme_grid
        assert rel_max(fn, -gx0) < gtol, s.pme_grid


def _half_spectrum_pme(x, box, q, alpha, K):
    """O.pme with the transform of real data: the influence function at kz <= K / 2 alone, the imaginary
    parts at kz = 0 and K / 2 dropped on the way back. Energy, dE/dx, dE/dq."""
    n = len(q)
    recip, m0, val, der, shifts = O._pme_stencil(x, box, K)
    idx = (m0[:, :, None] + shifts[None, None, :]) % K
    w3 = val[:, 0, :, None, None] * val[:, 1, None, :, None] * val[:, 2, None, None, :]
    flat = (idx[:, 0, :, None, None] * K * K + idx[:, 1, None, :, None] * K + idx[:, 2, None, None, :]).reshape(n, -1)
    grid = np.zeros(K ** 3)
    np.add.at(grid, flat, (q[:, None, None, None] * w3).reshape(n, -1))
    S = np.fft.rfftn(grid.reshape(K, K, K))
    f = O.signed_frequency(K).astype(float)
    m = np.stack(np.meshgrid(f, f, f[:K // 2 + 1], indexing="ij"), -1)
    ksq = np.sum((2 * np.pi * m @ np.linalg.inv(box).T) ** 2, -1)
    th = O.bspline_moduli(K)
    theta = th[:, None, None] * th[None, :, None] * th[None, None, :K // 2 + 1]
    ksq[0, 0, 0] = 1.0
    C = 4 * np.pi / abs(np.linalg.det(box)) / ksq * np.exp(-ksq / (4 * alpha * alpha)) / theta ** 2
    C[0, 0, 0] = 0.0
    kz = np.arange(K // 2 + 1)
    energy = 0.5 * np.sum(np.where((kz == 0) | (2 * kz == K), 1.0, 2.0) * C * np.abs(S) ** 2)
    loc = np.fft.irfftn(C * S, s=(K, K, K), norm="forward").reshape(-1)[flat].reshape(n, 6, 6, 6)
    a, da = val[:, 0, :, None, None], der[:, 0, :, None, None]
    b, db = val[:, 1, None, :, None], der[:, 1, None, :, None]
    c, dc = val[:, 2, None, None, :], der[:, 2, None, None, :]
    gu = np.stack([np.sum(loc * w, (1, 2, 3)) for w in (da * b * c, a * db * c, a * b * dc)], 1)
    self_ = alpha / math.sqrt(math.pi)
    return energy - self_ * np.sum(q * q), -q[:, None] * (gu @ recip), np.sum(loc * w3, (1, 2, 3)) - 2 * self_ * q


# planes: 6, 16, 34, 48, 78; cuFFT: 80
@pytest.mark.parametrize("K", [6, 16, 34, 48, 78, 80])
def test_even_sides_in_a_sheared_box(K):
    from torchff_b200.pme import PME

    rng = np.random.default_rng(K)
    box = np.array([[2.4, 0.0, 0.0], [0.3, 2.2, 0.0], [-0.2, 0.4, 2.5]])
    x, q = rng.random((200, 3)) @ box, rng.standard_normal(200)
    q -= q.mean()
    e0, gx0, pot0 = _half_spectrum_pme(x, box, q, 3.1, K)
    if K in (6, 16):  # where the dropped parts are far above the tolerance: the full spectrum gives other forces
        assert rel_max(O.pme(x, box, q, 3.1, K)[1], gx0) > 1e-7
    pme = PME(3.1, K, 0, use_customized_ops=True).cuda()
    xt, qt = t(x, grad=True), t(q, grad=True)
    e = pme(xt, t(box), qt)
    e.backward()
    assert rel(e.item(), e0) < 1e-11
    assert rel_max(xt.grad, gx0) < 1e-9 and rel_max(qt.grad, pot0) < 1e-9
