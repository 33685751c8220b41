"""An interior with gain (Im m < 0): its Green's function grows, in the assembly by triangle pairs and per RWG pair, in
the same-triangle terms and in the gradient."""
import numpy as np
import pytest

from conftest import rel
from oracle import bem_oracle as bo

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import bem_b200 as bb
    c = bb.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("m,q,exact", [(1.5 - 0.02j, 7, False), (1.3 - 0.3j, 4, True), (1.4 - 0.05j, 13, False)])
def test_operator_matches_oracle(ctx, kernel, m, q, exact):
    import bem_b200 as bb
    v, t = bb.icosphere(1.0, 1)
    kx, ki, ee, ei = bb.physics(2.0, m)
    rwg = bo.build_rwg(v, t.astype(np.int64), order="cpp")
    want = bo.assemble_pmchwt(rwg, v, t.astype(np.int64), kx, ki, ee, ei, q, distance="direct",
                              smooth="exact" if exact else "literal")
    bb.set_option(ctx, "assembly_kernel", kernel)
    try:
        Z = bb.assemble_pmchwt_dev(bb.Geometry(ctx, v, t, q), kx, ki, ee, ei, exact_gsmooth=exact).cpu().numpy()
    finally:
        bb.set_option(ctx, "assembly_kernel", 0)
    # the literal G_smooth at coincident points (R_s = 1e-15) steps by a unit in the last place of
    # exp(-Im k R_s) cos(Re k R_s), which is 1 here in both
    assert rel(Z, want) < 1e-12


def test_strong_gain_leaves_the_branch_free_exponential(ctx):
    # |Im k| times the extent beyond 700: the kernel per RWG pair, as with the option
    import bem_b200 as bb
    v, t = bb.icosphere(1.0, 0)
    g = bb.Geometry(ctx, v, t, 4)
    Z = [None, None]
    for kernel in (0, 1):
        bb.set_option(ctx, "assembly_kernel", kernel)
        Z[kernel] = bb.assemble_pmchwt_dev(g, 1.0 + 0j, 2.0 - 245j, 1.0, 0.7).cpu().numpy()
    bb.set_option(ctx, "assembly_kernel", 0)
    assert np.isfinite(Z[0]).all() and np.array_equal(Z[0], Z[1])


def test_gradient_follows_the_loss(ctx):
    import bem_b200 as bb
    v, t = bb.icosphere(1.0, 1)
    v = v * (1 + 0.05 * np.random.default_rng(3).standard_normal((len(v), 1)))
    target = 0.04 * (1 + np.cos(np.linspace(0, np.pi, 13)) ** 2)
    dv = np.random.default_rng(4).standard_normal(v.shape)
    kw = dict(orient=(2, 2, 1))
    m, h = 1.4 - 0.03j, 1e-4
    _, grad, _ = bb.adjoint_grad_vertices(ctx, v, t, 1.2, m, target, **kw)
    lp, lm = (bb.adjoint_grad(ctx, v + s * h * dv, t, 1.2, m, target, **kw)[0] for s in (1, -1))
    # the bound of the gradients without gain: h^2 of the third derivative and the loss's rounding over 2 h
    assert abs((grad * dv).sum() - (lp - lm) / (2 * h)) <= 1e-5 * np.abs(grad).max() * np.abs(dv).sum()
