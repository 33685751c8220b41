"""The far field's band limit on the CPU: node count, interpolation weights and conjugate nodes restated in NumPy.

exp(-i x (a sin t + b cos t)), a^2 + b^2 <= 1, sampled at 2 H equispaced nodes of the circle and interpolated
trigonometrically, against the direct sum.  The bound: every term has modulus one, so the direct sum and the
interpolated one each carry about eps (1 + x) sqrt(terms) of rounding (the phase's argument is rounded to eps x), the
weights add a Lebesgue constant below 4, and the band limit leaves less than 1e-16 of a term.
"""
import math

import numpy as np
import pytest


def node_pairs(x):
    """One past the first order whose Debye bound of J_n(x) is below 1e-17."""
    x = max(x, 1e-3)
    n = int(x) + 2
    while True:
        b = math.acosh(n / x)
        t = math.tanh(b)
        if math.exp(n * (t - b)) < 1e-17 * math.sqrt(2 * math.pi * n * t):
            return n + 1
        n += 1


def weights(H, ndir):
    nd, per = ndir - 1, 2 * H * (ndir - 1)
    W = np.ones((ndir, 2 * H))
    for d in range(ndir):
        for j in range(2 * H):
            m = int(math.fmod(d * H - j * nd, per))
            m -= per * (m > per // 2)
            m += per * (m <= -(per // 2))
            if m == 0:
                continue
            k = int(math.fmod(m, 2 * nd))
            k -= 2 * nd * (k > nd)
            k += 2 * nd * (k < -nd)
            k = nd - k if 2 * k > nd else -nd - k if 2 * k < -nd else k
            h = math.pi * m / per
            W[d, j] = math.sin(math.pi * k / nd) * math.cos(h) / (math.sin(h) * 2 * H)
    return W


@pytest.mark.parametrize("x", [1e-4, 0.3, 1.0, 5.5, 16.0, 40.0])
@pytest.mark.parametrize("ndir", [181, 100, 37, 20, 361])
def test_interpolated_sums_equal_direct_ones(x, ndir):
    H = node_pairs(x)
    rng = np.random.default_rng(int(10 * x) + ndir)
    a = rng.standard_normal((300, 3))
    a *= x / np.linalg.norm(a, axis=1, keepdims=True)
    c = rng.standard_normal(300)

    def phases(t):
        return np.exp(-1j * (np.sin(t)[:, None] * a[:, 0] + np.cos(t)[:, None] * a[:, 2]))

    half = phases(np.pi * np.arange(H) / H) @ c
    nodes = np.concatenate([half, half.conj()])  # real coefficients: the node t + pi is the conjugate one
    W = weights(H, ndir)
    assert np.abs(W).sum(axis=1).max() < 4.5
    direct = phases(np.pi * np.arange(ndir) / (ndir - 1)) @ c
    bound = 4.5 * np.finfo(float).eps * (1 + x) * np.sqrt(len(c)) * np.abs(c).max() * 2
    assert np.abs(W @ nodes - direct).max() < bound


@pytest.mark.parametrize("x", [0.3, 5.5, 16.0, 40.0])
def test_debye_bound_holds(x):
    from scipy.special import jv
    H = node_pairs(x)
    assert abs(jv(np.arange(H - 1, H + 60), x)).sum() < 1e-16
