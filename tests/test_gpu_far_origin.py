"""Assembly of a mesh far from the origin: the distances of its points, not of its points from the origin, decide whether
the triangle-pair kernel can take it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_shifted_mesh_keeps_the_triangle_kernel():
    import bem_b200 as bb
    v, t = bb.icosphere(1.0, 2)
    v = np.round(v * 2 ** 20) / 2 ** 20  # so that the shift is exact
    ctx = bb.Context(0)
    try:
        g = bb.Geometry(ctx, v + [2.0 ** 22, 0, 0], t, 7)
        Z = {}
        for kernel in (0, 1):
            bb.set_option(ctx, "assembly_kernel", kernel)
            Z[kernel] = bb.assemble_pmchwt_dev(g, 2.0 + 0j, 3.0 + 0.1j, 1.0, 1 / 1.5).cpu().numpy()
    finally:
        ctx.close()
    # the kernels' sums differ in their last places, and by the rounding of points near 2^22 (2^-31), linearly in them
    assert not np.array_equal(Z[0], Z[1])
    assert np.abs(Z[0] - Z[1]).max() < 1e-7 * np.abs(Z[1]).max()
