"""Refined solutions with the block inverses of the default against those with inverses of single 256-row blocks.

An inverse composed of several blocks in 32 bits contracts the refinement a little less than single ones, and the error
that the last sweep leaves (1e-12 here, tolerance 2e-10) grows with that.  2N = 960: 1.037 times the error of single
blocks with three blocks, 1.065 with four; 1.05 is the bound.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_default_blocks_refine_nearly_as_exactly_as_single_ones():
    import bem_b200 as bb
    import torch
    v, t = bb.icosphere(1.0, 2)
    ctx = bb.Context(0)
    ratio = []
    try:
        g = bb.Geometry(ctx, v, t, 7)
        kx, ki, ee, ei = bb.physics(2.0, 1.3116 + 0.001j)
        Z = bb.assemble_pmchwt_dev(g, kx, ki, ee, ei)
        for seed in range(4):
            RT = np.linalg.qr(np.random.default_rng(seed).standard_normal((32, 3, 3)))[0]
            B = bb.rhs_planewave_dev(g, kx, ee, RT)
            X = torch.linalg.solve(Z, B.T).T
            X = X + torch.linalg.solve(Z, (B - X @ Z.T).T).T
            err = []
            for sb in (4, 1):  # the default, and single blocks
                bb.set_option(ctx, "solve_superblock", sb)
                lu = bb.LU(ctx, Z, bb.PREC_FP32_REFINE)
                Y, st = lu.solve(B, tol=2e-10)
                lu.close()
                assert st["factorization"] == 2
                err.append(float((Y - X).norm()))
            ratio.append(err[0] / err[1])
    finally:
        ctx.close()
    assert np.exp(np.mean(np.log(ratio))) < 1.05, ratio
