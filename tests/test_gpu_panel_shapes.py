"""Panels on clusters of at most 8 CTAs, as on a device that holds no larger ones: up to 4096 rows they stay in registers
(no launch more than with 16 CTAs, where the cooperative grid takes a second one per panel), with the same factors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,stays", [(2049, True), (2600, True), (4096, True), (4160, False)])
def test_eight_ctas_take_up_to_4096_rows(n, stays):
    import bem_b200 as bb
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    ctx = bb.Context(0)
    out, count = {}, {}
    try:
        for mode in (1, 8, 0):
            bb.set_option(ctx, "panel_clusters", mode)
            before = bb.lib().bem_ctx_launch_count(ctx.h)
            out[mode] = bb.lu_factorize_cuda(ctx, A)
            count[mode] = bb.lib().bem_ctx_launch_count(ctx.h) - before
    finally:
        ctx.close()
    for mode in (8, 0):
        for x, y in zip(out[1], out[mode]):
            assert np.array_equal(x, y)
    assert count[1] <= count[8] < count[0] and (count[8] == count[1]) == stays
