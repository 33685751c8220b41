"""The operator term of the vertex gradient over pairs of triangles, for each
instance of its kernel: a lossless and an absorbing interior (branch-free
exponential and sine) and an interior with gain (the library's functions),
with fewer triangles than a block's threads and more, and the quadratures
with the fewest and the most points."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import bem_b200 as bb
    c = bb.Context(0)
    yield c
    c.close()


def _mesh(size, seed):
    import bem_b200 as bb
    v, t = bb.icosphere(1.0, size)
    return v * (1 + 0.05 * np.random.default_rng(seed).standard_normal((len(v), 1))), t


TARGET = 0.04 * (1 + np.cos(np.linspace(0, np.pi, 13)) ** 2)


@pytest.mark.parametrize("size,m,quad", [(0, 1.4 + 0j, 7), (1, 1.33 + 0.01j, 7), (1, 1.5 + 0j, 4), (0, 1.35 + 0.01j, 13)])
def test_gradient_along_a_displacement(ctx, size, m, quad):
    # against the central difference of the loss along a random displacement:
    # h = 1e-4 leaves h^2 of the third derivative (~1e-8 of the largest entry
    # at these sizes) plus the loss's rounding (~1e-13) over 2 h; the bound is
    # the vertex gradient's own (its same-triangle term is a central difference)
    import bem_b200 as bb
    v, t = _mesh(size, size + quad)
    dv = np.random.default_rng(size).standard_normal(v.shape)
    kw = dict(orient=(2, 2, 1), quad_order=quad)
    _, grad, _ = bb.adjoint_grad_vertices(ctx, v, t, 1.2, m, TARGET, **kw)
    h = 1e-4
    lp = bb.adjoint_grad(ctx, v + h * dv, t, 1.2, m, TARGET, **kw)[0]
    lm = bb.adjoint_grad(ctx, v - h * dv, t, 1.2, m, TARGET, **kw)[0]
    fd = (lp - lm) / (2 * h)
    scale = np.abs(grad).max() * np.abs(dv).sum()
    assert abs((grad * dv).sum() - fd) <= 1e-5 * scale, ((grad * dv).sum(), fd, scale)


@pytest.mark.parametrize("size,quad", [(0, 13), (1, 4), (2, 7)])
def test_kernel_instances_agree(ctx, size, quad):
    # |Im m| = 1e-13 changes every Green's function by ~1e-13 of itself, so
    # absorption, gain and neither are the same problem to that; the exponential
    # and sine of the instances differ by rounding (2e-16).  The condition of
    # these systems (< 1e3) multiplies both.
    import bem_b200 as bb
    v, t = _mesh(size, 3)
    kw = dict(orient=(2, 2, 1), quad_order=quad)
    g = [bb.adjoint_grad_vertices(ctx, v, t, 1.2, 1.4 + im * 1j, TARGET, **kw)[1] for im in (0.0, 1e-13, -1e-13)]
    for x in g[1:]:
        assert np.abs(x - g[0]).max() <= 1e-9 * np.abs(g[0]).max()
