"""The pivoted LU's panels in the registers of one cluster against the
cooperative grid's, bit for bit, at the sizes where the cluster's shape
changes (1, 2, 8, 9 and 16 CTAs, more than 256 rows a CTA) and with rows that
tie, vanish or hold no candidate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,kind", [(256, "random"), (257, "ties"), (2048, "zeros"), (2080, "random"), (2310, "ties"),
                                    (4097, "random"), (300, "tiny")])
def test_same_factors_as_the_grid_panels(n, kind):
    import bem_b200 as bb
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind == "ties":          # |re| + |im| equal for many rows: the smallest row wins
        A = np.sign(A.real) + 1j * np.sign(A.imag)
        A += 3.0 * np.tri(n, k=-1).T
    elif kind == "zeros":       # a zero column inside a panel and zero rows below it
        A[:, 21] = 0.0
        A[n - 40:, :16] = 0.0
    elif kind == "tiny":        # subnormal candidates and reciprocals by division
        A[:, :16] *= 1e-309
        A[:, 16:32] *= 1e300
    ctx = bb.Context(0)
    out = {}
    try:
        for mode in (1, 0):
            bb.set_option(ctx, "panel_clusters", mode)
            out[mode] = bb.lu_factorize_cuda(ctx, A)
    finally:
        ctx.close()
    (F1, p1, i1), (F0, p0, i0) = out[1], out[0]
    assert i1 == i0
    assert np.array_equal(p1, p0)
    assert np.array_equal(F1, F0, equal_nan=True)
