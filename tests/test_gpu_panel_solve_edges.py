"""Edges of the register panel, the block solves, the GEMM tiles, the operand packing and the block inverses.

Bounds: an LU solve's backward error is a small multiple of n eps (growth included), so 1e-11 relative on these
diagonally shifted matrices (condition below 1e3); a residual in FP64 is good to K eps |Z| |X|; an FP16-part product
keeps about 21 bits of each factor, 2^-19 of |A| |B| over K terms.
"""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import bem_b200 as bb
    c = bb.Context(0)
    yield c
    c.close()


def _cplx(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


# one row, one short of / exactly / one over a panel, a warp, a CTA of 256 rows, the 8-CTA cluster's 2048 and 4096
# rows (16 CTAs beyond); pivots as LAPACK's
@pytest.mark.parametrize("n,nrhs", [(1, 1), (15, 2), (16, 3), (17, 1), (33, 9), (255, 2), (257, 300), (520, 17), (2049, 3),
                                    (4100, 2)])
def test_lu_edges_match_lapack(ctx, n, nrhs):
    import bem_b200 as bb
    import scipy.linalg as sl
    rng = np.random.default_rng(n)
    Z = _cplx(rng, n, n) + 0.5 * np.sqrt(n) * np.eye(n)
    B = _cplx(rng, n, nrhs)
    F, piv, info = bb.lu_factorize_cuda(ctx, Z)
    lu, p = sl.lu_factor(Z)
    assert info == 0 and np.array_equal(piv - 1, p)
    assert rel(F, lu) < 1e-11
    assert rel(bb.lu_solve_cuda(ctx, F, piv, B), sl.lu_solve((lu, p), B)) < 1e-11


def test_lu_zero_column_and_nonfinite_entries(ctx):
    import bem_b200 as bb
    rng = np.random.default_rng(0)
    Z = _cplx(rng, 300, 300)
    Z[:, 20] = 0
    assert bb.lu_factorize_cuda(ctx, Z)[2] == 21
    Z = _cplx(rng, 40, 40)
    Z[7, 3] = np.nan  # never a pivot candidate; it spreads through the updates, nothing hangs
    bb.lu_factorize_cuda(ctx, Z)
    # pivots outside the range of the fast reciprocal
    for s in (1e-150, 1e147):
        Z = _cplx(rng, 50, 50) * s
        F, piv, info = bb.lu_factorize_cuda(ctx, Z)
        G, qiv, _ = bb.lu_factorize_cuda(ctx, Z / s)
        assert info == 0 and np.array_equal(piv, qiv) and rel(np.triu(F) / s, np.triu(G)) < 1e-12


# FP32 pivoted LU: rows of 16 bytes (even order) and not, several widths of the right-hand side
@pytest.mark.parametrize("n,nrhs", [(301, 3), (512, 40), (1037, 310)])
def test_fp32_pivoted_lu_edges(ctx, n, nrhs):
    import bem_b200 as bb
    import torch
    rng = np.random.default_rng(n)
    Z = torch.from_numpy(_cplx(rng, n, n) + 0.5 * np.sqrt(n) * np.eye(n)).cuda()
    B = torch.from_numpy(_cplx(rng, nrhs, n)).cuda()
    bb.set_symmetric(ctx, 0)
    try:
        lu = bb.LU(ctx, Z, bb.PREC_FP32_REFINE)
        X, st = lu.solve(B)
        lu.close()
    finally:
        bb.set_symmetric(ctx, 1)
    assert st["factorization"] == 0
    assert rel(X.cpu(), torch.linalg.solve(Z, B.T).T.cpu()) < 1e-10


# tiles of 64 x 64, 32 x 32 and 32 x 8, with remainders
@pytest.mark.parametrize("n,nrhs", [(130, 1), (500, 9), (1030, 33), (1030, 200), (70, 65)])
def test_fp64_gemm_tiles(ctx, n, nrhs):
    import bem_b200 as bb
    import torch
    rng = np.random.default_rng(n + nrhs)
    Z, B, X = (torch.from_numpy(_cplx(rng, *s)).cuda() for s in ((n, n), (nrhs, n), (nrhs, n)))
    lu = bb.LU(ctx, Z, bb.PREC_FP32_REFINE)
    R = lu.residual(B, X, method=0)
    lu.close()
    bound = 8 * np.finfo(float).eps * (n * Z.abs().max() * X.abs().max())
    assert (R - (B - X @ Z.T)).abs().max() < bound


# K beyond the packing kernel's register cache, rows off the 16-byte boundary, a few items
@pytest.mark.parametrize("M,N,K,off", [(70, 33, 1500, 0), (200, 5, 1024, 1), (9, 130, 77, 1), (300, 300, 1025, 0)])
def test_fp16_part_operands(ctx, M, N, K, off):
    import bem_b200 as bb
    import torch
    rng = np.random.default_rng(M + N + K)
    A = torch.from_numpy(_cplx(rng, M, K + off).astype(np.complex64)).cuda()[:, off:]
    B = torch.from_numpy(_cplx(rng, N, K + off).astype(np.complex64)).cuda()[:, off:]
    C0 = torch.from_numpy(_cplx(rng, N, M).astype(np.complex64)).cuda()
    C = bb.cgemm_tf32x3(ctx, A, B, C0.clone(), b_rowmajor=False, c_colmajor=True)
    want = C0.to(torch.complex128) - B.to(torch.complex128) @ A.to(torch.complex128).T
    assert (C - want).abs().max() < 2.0 ** -19 * K ** 0.5 * 8 * A.abs().max() * B.abs().max()


# block inverses of 1 to 4 diagonal blocks, ragged last ones, and a solve after the option has changed
@pytest.mark.parametrize("n", [200, 256, 300, 1100, 2600])
@pytest.mark.parametrize("sb", [1, 2, 3, 4])
def test_block_inverse_solves(ctx, n, sb):
    import bem_b200 as bb
    import torch
    rng = np.random.default_rng(n + sb)
    A = _cplx(rng, n, n)
    Z = torch.from_numpy(A + A.T + 4 * np.sqrt(n) * np.eye(n)).cuda()
    B = torch.from_numpy(_cplx(rng, 7, n)).cuda()
    bb.set_option(ctx, "solve_superblock", sb)
    try:
        lu = bb.LU(ctx, Z, bb.PREC_FP32_REFINE)
        X, st = lu.solve(B)
        bb.set_option(ctx, "solve_superblock", 5 - sb)
        Y, _ = lu.solve(B)
        lu.close()
    finally:
        bb.set_option(ctx, "solve_superblock", 4)
    want = torch.linalg.solve(Z, B.T).T.cpu()
    assert st["factorization"] == 1 and st["iterations"] <= 4
    assert rel(X.cpu(), want) < 1e-10 and rel(Y.cpu(), want) < 1e-10
