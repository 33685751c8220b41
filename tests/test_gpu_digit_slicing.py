"""Digit planes of the int8 residual, for every digit count and for row
lengths that are no multiple of the four entries a thread slices.

With S digits an entry is kept to 2^(1-7S) of its row (column) maximum and the
dropped digit pairs weigh about as much again: a product term is good to about
2^(3-7S) max|Z| max|X|, and the bound is twice that times sqrt(2n), a random
walk over the 2n real terms, plus FP64 rounding of the same sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("digits", range(2, 9))
@pytest.mark.parametrize("n,nrhs", [(2, 1), (63, 2), (65, 5), (130, 3), (2051, 7)])
def test_every_digit_count_at_ragged_lengths(n, nrhs, digits):
    import torch
    import bem_b200 as bb
    rng = np.random.default_rng(100 * digits + n)
    Z = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    X = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
    Z[n // 2, :-1] = 0.0   # the maximum in the last, partly filled group of four
    X[0, :-1] = 0.0
    B = rng.standard_normal((nrhs, n)) + 1j * rng.standard_normal((nrhs, n))
    ctx = bb.Context(0)
    try:
        bb.set_residual_digits(ctx, digits)
        lu = bb.LU(ctx, torch.from_numpy(Z.copy()).cuda(), bb.PREC_FP32_REFINE)
        R = lu.residual(torch.from_numpy(B).cuda(), torch.from_numpy(X.copy()).cuda(), method=1).cpu().numpy()
        lu.close()
    finally:
        ctx.close()
    exact = B.astype(np.clongdouble) - X.astype(np.clongdouble) @ Z.astype(np.clongdouble).T
    err = float(np.abs(R - exact).max()) / (np.abs(Z).max() * np.abs(X).max())
    assert err < (2.0 ** (4 - 7 * digits) + 2.0 ** -51) * np.sqrt(2.0 * n), err
