"""Band-limited far field and by-triangle right-hand sides on the device, against the direct forms."""
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


def _rotations(no, seed):
    q = np.random.default_rng(seed).standard_normal((no, 3, 3))
    return np.linalg.qr(q)[0]


# node pairs below, at and above a block of 16, one and several parts, every rule and a general one, few
# directions (the direct kernel), orientations that are reflections or scaled (not only rotations), an off-centre mesh
@pytest.mark.parametrize("ka,q,no,ntheta,scale,shift", [
    (0.02, 7, 1, 181, 1.0, 0.0), (0.9, 7, 1, 37, 1.0, 0.0), (1.0, 4, 3, 181, 1.0, 0.0), (3.0, 13, 2, 100, 1.0, 0.0),
    (9.0, 7, 40, 361, 1.0, 0.0), (2.0, 7, 2, 19, 1.0, 0.0), (2.0, 7, 2, 8, 1.0, 0.0), (2.0, 7, 3, 181, 1.7, 0.0),
    (2.0, 7, 2, 181, 1.0, 3.0)])
def test_band_limited_mueller_equals_direct(ctx, ka, q, no, ntheta, scale, shift):
    import bem_b200 as bb
    import torch
    v, t = bb.icosphere(1.0, 2)
    g = bb.Geometry(ctx, v + [shift, 0, 0], t, q)
    RT, w = scale * _rotations(no, no), np.random.default_rng(1).uniform(0.1, 1, no)
    X = torch.view_as_complex(torch.randn((2 * no, g.n, 2), dtype=torch.float64, device="cuda",
                                          generator=torch.Generator("cuda").manual_seed(no)))
    M = bb.mueller_from_solutions_dev(g, X, RT, w, complex(ka), 1.0, ntheta=ntheta)
    bb.set_option(ctx, "farfield_kernel", 1)
    D = bb.mueller_from_solutions_dev(g, X, RT, w, complex(ka), 1.0, ntheta=ntheta)
    bb.set_option(ctx, "farfield_kernel", 0)
    # both sums: eps (1 + k r) per term; elements are quadratic in them, cancelling ones against the largest
    assert np.abs(M - D).max() < 2e-14 * (1 + ka * (1 + shift) * scale) * np.abs(D).max()


def test_complex_wavenumber_and_few_directions_match_oracle(ctx):
    import bem_b200 as bb
    import torch
    v, t = bb.icosphere(1.0, 1)
    g = bb.Geometry(ctx, v, t, 7)
    RT, w = _rotations(2, 5), np.array([0.3, 0.7])
    X = torch.view_as_complex(torch.randn((4, g.n, 2), dtype=torch.float64, device="cuda",
                                          generator=torch.Generator("cuda").manual_seed(0)))
    for k, nth in ((1.5 + 0.2j, 181), (1.5 + 0j, 2)):
        M = bb.mueller_from_solutions_dev(g, X, RT, w, k, 1.0, ntheta=nth)
        bb.set_option(ctx, "farfield_kernel", 1)
        D = bb.mueller_from_solutions_dev(g, X, RT, w, k, 1.0, ntheta=nth)
        bb.set_option(ctx, "farfield_kernel", 0)
        assert rel(M, D) < 1e-13


# one orientation, one short of, exactly and one over a group of 16, several groups; every rule; a complex k
@pytest.mark.parametrize("mesh,q,no,k", [("ico", 7, 1, 2.0), ("ico", 4, 15, 2.0), ("hex", 13, 16, 3.0), ("ico", 7, 17, 0.01),
                                         ("hex", 7, 50, 5.0), ("ico", 7, 3, 2.0 + 0.3j)])
def test_plane_waves_by_triangles_match_oracle(ctx, mesh, q, no, k):
    import bem_b200 as bb
    v, t = bb.icosphere(1.0, 2) if mesh == "ico" else bb.hex_prism(0.7, 1)
    g = bb.Geometry(ctx, v, t, q)
    RT = _rotations(no, no)
    B = bb.rhs_planewave_dev(g, complex(k), 1.2, RT).cpu().numpy().T
    tt = t.astype(np.int64)
    Bo = bo.orientation_rhs(bo.build_rwg(v, tt, "cpp"), v, tt, [(r, 1.0) for r in RT], complex(k), 1.2, q)
    assert rel(B, Bo) < 1e-13
