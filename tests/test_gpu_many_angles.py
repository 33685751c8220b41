"""Mueller matrices at more scattering angles than the interpolation's weights and their 32-bit indices hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_two_million_angles_of_a_wide_band():
    import bem_b200 as bb
    import torch
    ka, ntheta = 440.0, 2_100_001  # 527 node pairs: 2 x 527 x ntheta weights are more than 2^31
    v, t = bb.icosphere(1.0, 2)
    RT, w = np.eye(3)[None], np.ones(1)
    ctx = bb.Context(0)
    try:
        g = bb.Geometry(ctx, v, t, 4)
        X = torch.view_as_complex(torch.randn((2, g.n, 2), dtype=torch.float64, device="cuda",
                                              generator=torch.Generator("cuda").manual_seed(0)))
        M = bb.mueller_from_solutions_dev(g, X, RT, w, complex(ka), 1.0, ntheta=ntheta)
        few = bb.mueller_from_solutions_dev(g, X, RT, w, complex(ka), 1.0, ntheta=8)  # every 300000th of them
    finally:
        ctx.close()
    assert np.isfinite(M).all()
    # both: eps (1 + k r) per term, elements quadratic in them
    assert np.abs(M[:, :, ::300000] - few).max() < 2e-14 * (1 + ka) * np.abs(few).max()


def test_the_widest_band_that_is_interpolated():
    # 527 node pairs of the 533 whose sums fit shared memory, against the sums per RWG half and direction
    import bem_b200 as bb
    import torch
    ka, ntheta = 440.0, 1001
    v, t = bb.icosphere(1.0, 2)
    RT, w = np.linalg.qr(np.random.default_rng(2).standard_normal((2, 3, 3)))[0], np.array([0.4, 0.6])
    ctx = bb.Context(0)
    try:
        g = bb.Geometry(ctx, v, t, 4)
        X = torch.view_as_complex(torch.randn((4, g.n, 2), dtype=torch.float64, device="cuda",
                                              generator=torch.Generator("cuda").manual_seed(1)))
        before = bb.lib().bem_ctx_launch_count(ctx.h)
        M = bb.mueller_from_solutions_dev(g, X, RT, w, complex(ka), 1.0, ntheta=ntheta)
        launches = bb.lib().bem_ctx_launch_count(ctx.h) - before
        bb.set_option(ctx, "farfield_kernel", 1)
        D = bb.mueller_from_solutions_dev(g, X, RT, w, complex(ka), 1.0, ntheta=ntheta)
    finally:
        ctx.close()
    assert launches == 4  # weights, nodes, interpolation, average
    assert np.abs(M - D).max() < 2e-14 * (1 + ka) * np.abs(D).max()
