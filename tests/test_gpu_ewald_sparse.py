"""FP64 screened Coulomb and exclusion correction pair by pair: isolated pairs at 0.3 to 0.99 of the
cutoff, so that no nearer pair's larger terms hide the relative error of a distant one.

Coordinates are multiples of 2^-20 in a box of 64, so displacements are exact. Reference: the
functions in 50 decimal digits at the exact squared distance. Bounds, in units of eps = 2^-52, with
y = (alpha r)^2: erfc(alpha r) and exp(-y) multiply the relative error of y by y. The rounding of alpha^2,
r^2 and their product is 3 half units, that of a rounded alpha r squared 4 more: at most 4 y, and 8 for the
polynomial (or 5 units of erfc) and the products after it. The library's exclusion terms beyond the
polynomials' ranges cancel to 1 / y of their parts, the second derivative's twice.
"""
import math
from decimal import Decimal, getcontext

import numpy as np
import pytest
import torch

from gpu_util import t

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52
KC = 138.935456
PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494459")


def _terms(r2: Decimal, alpha: float, excluded: bool):
    """f = erfc(alpha r) / r (or -erf(alpha r) / r), g = -(1/r) df/dr, h = -(1/r) dg/dr."""
    a, r = Decimal(alpha), r2.sqrt()
    y = a * a * r2
    ex = (-y).exp()
    term = s = Decimal(1)  # erf(u) = 2 u / sqrt(pi) exp(-u^2) sum (2 u^2)^n / (2n + 1)!!
    n = 0
    while term > s * Decimal(10) ** -55:
        n += 1
        term = term * 2 * y / (2 * n + 1)
        s += term
    erf = 2 * a * r / PI.sqrt() * ex * s
    f = (-erf if excluded else 1 - erf) / r
    tx = 2 * a / PI.sqrt() * ex
    g = (f + tx) / r2
    return f, g, (3 * g + 2 * a * a * tx) / r2


def _pairs(y: float):
    """48 pairs 8 apart; (coords, charges, alpha, cutoff 1)."""
    rng = np.random.default_rng(int(100 * y))
    site = 8.0 * np.stack(np.unravel_index(rng.permutation(64)[:48], (4, 4, 4)), 1) + 0.5
    d = rng.normal(size=(48, 3))
    d *= (np.linspace(0.3, 0.99, 48) / np.linalg.norm(d, axis=1))[:, None]
    d = np.round(d * 2 ** 20) / 2 ** 20
    x = np.empty((96, 3))
    x[0::2], x[1::2] = site + d, site
    return x, d, rng.uniform(0.3, 1.0, 96), math.sqrt(y)


def _reference(d, alpha, excluded):
    getcontext().prec = 60
    out = np.empty((len(d), 3))
    y = np.empty(len(d))
    for k, v in enumerate(d):
        r2 = sum((Decimal(float(c)) ** 2 for c in v), Decimal(0))
        out[k] = [float(z) for z in _terms(r2, alpha, excluded)]
        y[k] = float(Decimal(alpha) ** 2 * r2)
    return out[:, 0], out[:, 1], out[:, 2], y


def _check(gq, gx, q, d, f, g, tol):
    """Per-atom charge and coordinate gradients of every pair."""
    qi, qj = q[0::2], q[1::2]
    gq, gx = gq.cpu().numpy(), gx.cpu().numpy()
    assert np.all(np.abs(gq[0::2] / (KC * qj * f) - 1) < tol)
    assert np.all(np.abs(gq[1::2] / (KC * qi * f) - 1) < tol)
    want = -(KC * qi * qj * g)[:, None] * d  # dE/dx_i = -k q_i q_j g r
    size = np.linalg.norm(want, axis=1)
    assert np.all(np.linalg.norm(gx[0::2] - want, axis=1) < tol * size)
    assert np.all(np.linalg.norm(gx[1::2] + want, axis=1) < tol * size)


# the polynomials' ranges (to 7 and to 13.5), past them
Y = [3.0, 7.0, 7.1, 11.0, 13.5, 25.0]


@pytest.mark.parametrize("excluded", [False, True])
@pytest.mark.parametrize("y", Y)
def test_pair_operator(y, excluded):
    from torchff_b200 import MultipolarInteraction

    x, d, q, alpha = _pairs(y)
    f, g, _, yp = _reference(d, alpha, excluded)
    rows = torch.arange(96, device="cuda").reshape(48, 2)
    none = rows[:0]
    xs, qs = t(x, grad=True), t(q, grad=True)
    e = MultipolarInteraction(0, 1.0, alpha, KC).cuda()(xs, t(64.0 * np.eye(3)), none if excluded else rows, qs,
                                                        pairs_excl=rows if excluded else none)
    e.backward()
    tol = (8 + 4 * yp + (8 / yp if excluded and y > 13.5 else 0)) * EPS
    assert abs(e.item() / (KC * np.sum(q[0::2] * q[1::2] * f)) - 1) < tol.max()
    _check(qs.grad, xs.grad, q, d, f, g, tol)


@pytest.mark.parametrize("excluded", [False, True])
@pytest.mark.parametrize("y", Y)
def test_fused_evaluation(y, excluded):
    from torchff_b200.system import FixedChargeSystem

    x, d, q, alpha = _pairs(y)
    f, g, h, yp = _reference(d, alpha, excluded)
    sy = FixedChargeSystem(q, np.ones(96), np.zeros(96), np.arange(96).reshape(48, 2) if excluded else None, 1.0,
                           alpha, 0, dtype=torch.float64)
    xs, box = t(x), t(64.0 * np.eye(3))
    tol = (8 + 4 * yp + (8 / yp if excluded and y > 13.5 else 0)) * EPS
    energy = KC * np.sum(q[0::2] * q[1::2] * f)
    for out in (sy.evaluate(xs, box, grad_charges=True), sy.evaluate_grads(xs, box)):
        assert abs(out["energy"].item() / energy - 1) < tol.max()
        _check(out["grad_charges"], -out["forces"], q, d, f, g, tol)
    # u . dE/dx: -g delta + h (r . delta) r for delta = u_i - u_j
    u = np.random.default_rng(1).normal(size=x.shape)
    delta = u[0::2] - u[1::2]
    kqq, rd = KC * q[0::2] * q[1::2], np.sum(d * delta, axis=1)
    want = (-kqq * g)[:, None] * delta + (kqq * h * rd)[:, None] * d
    size = kqq * (np.abs(g) * np.linalg.norm(delta, axis=1) + np.abs(h * rd) * np.linalg.norm(d, axis=1))
    got = sy.hvp(xs, box, t(u))["coords"].cpu().numpy()
    tol2 = tol + (16 / yp ** 2 if excluded and y > 13.5 else 0) * EPS + 8 * EPS
    assert np.all(np.linalg.norm(got[0::2] - want, axis=1) < tol2 * size)
    assert np.all(np.linalg.norm(got[1::2] + want, axis=1) < tol2 * size)
