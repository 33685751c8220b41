"""The block substitutions round a row once per solved row before it: their error against that of the same sums in
NumPy, product first, then one subtraction.

The systems are their own factors: a unit lower triangle whose entries (0.02) leave every product well below the sum it
is taken from.  Two roundings of the sum per product give sqrt(2) times the error (1.42 in NumPy); 1.1 is the bound.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forward(L, X, dtype):
    X = X.astype(dtype)
    for k in range(len(L) - 1):
        X[k + 1:] -= L[k + 1:, k, None].astype(dtype) * X[k]
    return X


@pytest.mark.parametrize("n", [33, 100, 256])
@pytest.mark.parametrize("nrhs", [64, 200, 600])  # one, two and eight columns a CTA
@pytest.mark.parametrize("upper", [False, True])
def test_error_of_one_rounding(n, nrhs, upper):
    import bem_b200 as bb
    import torch
    rng = np.random.default_rng(n)
    L = np.tril(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), -1) * 0.02 + np.eye(n)
    B = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    exact = _forward(L, B, np.clongdouble)
    want = np.linalg.norm((_forward(L, B, np.complex128) - exact).astype(complex))
    A, C = (L[::-1, ::-1], B[::-1]) if upper else (L, B)  # reversed rows and columns: backward substitution
    ctx = bb.Context(0)
    try:
        lu = bb.LU(ctx, torch.from_numpy(A.copy()).cuda(), bb.PREC_FP64)
        X = lu.solve(torch.from_numpy(np.ascontiguousarray(C.T)).cuda())[0].cpu().numpy().T
        lu.close()
    finally:
        ctx.close()
    got = np.linalg.norm(((X[::-1] if upper else X) - exact).astype(complex))
    assert got < 1.1 * want, got / want
