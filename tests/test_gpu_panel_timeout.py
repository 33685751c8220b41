"""A panel whose CTAs do not get their peers' candidates in time: the wait runs out (a limit of zero cycles stands for
a peer that does not send), the call returns BEM_ERR_TIMEOUT, nothing outside the matrix is touched, and the same
context then factors the same matrix."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 2, 3, 9 and 16 CTAs a cluster, 16 and 17 CTA rows apart; both precisions of the pivoted LU
@pytest.mark.parametrize("n,prec", [(257, 0), (600, 0), (2049, 0), (4097, 0), (600, 1)])
def test_timeout_leaves_the_surroundings_alone(n, prec):
    import bem_b200 as bb
    import torch
    rng = np.random.default_rng(n)
    A = torch.from_numpy(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))).cuda()
    pad, ld = 40, n + 24
    guard = torch.full((n + 2 * pad, ld), 7.5 - 2.25j, dtype=torch.complex128, device="cuda")
    buf = guard.clone()
    inside = buf[pad:pad + n, :n]
    ctx = bb.Context(0)
    L = bb.lib()
    bb.set_symmetric(ctx, 0)
    try:
        for mcycles, status in ((0, 6), (2000, 0)):
            bb.set_option(ctx, "panel_wait_mcycles", mcycles)
            inside.copy_(A)
            torch.cuda.synchronize()
            lu, info = C.c_void_p(), C.c_int()
            assert L.bem_lu_factor_dev(ctx.h, inside.data_ptr(), n, ld, prec, C.byref(lu), C.byref(info)) == status
            ctx.check(L.bem_ctx_synchronize(ctx.h))
            if status:
                assert "gave up" in L.bem_last_error(ctx.h).decode() and not lu.value
            else:
                L.bem_lu_free(lu)
            out = buf.clone()
            out[pad:pad + n, :n] = guard[pad:pad + n, :n]
            assert torch.equal(out, guard)
        if prec == 0:
            L_ = torch.tril(inside, -1)
            assert L_.abs().max() < 2 ** 0.5 * 1.0001  # pivoted: |re| + |im| of every multiplier at most that of one
    finally:
        ctx.close()


def test_timeout_in_a_batch_is_every_particles_status():
    import bem_b200 as bb
    ctx = bb.Context(0)
    try:
        parts = bb.c4_particles(3, 3, orient=(1, 1, 1))
        want = [M for M, _ in bb.batch_run(ctx, parts)]
        bb.set_option(ctx, "panel_wait_mcycles", 0)
        with pytest.raises(bb.BemError) as ei:
            bb.batch_run(ctx, parts)
        assert ei.value.status == 6
        bb.set_option(ctx, "panel_wait_mcycles", 2000)
        for M, (N, _) in zip(want, bb.batch_run(ctx, parts)):
            assert np.array_equal(M, N)
    finally:
        ctx.close()
