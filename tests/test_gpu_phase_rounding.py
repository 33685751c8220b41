"""Plane-wave right-hand sides where the rounding of the phase k k_hat.r decides their error: against 80-bit sums, and
compared with the error of the plain sums over RWG halves in 64 bits (k_hat.r rounded three times, k times it once)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sums(v, t, rwg, rule, RT, k, eta, real):
    """Columns (2 no, 2 N): f.E and f.H of both polarisations, term by term in the type `real`."""
    pts, wts = rule
    N = len(rwg["length"])
    v, RT = v.astype(real), RT.astype(real)
    out = np.zeros((2 * len(RT), 2 * N, 2), real)
    for tri, free, sign in ((rwg["tri_p"], rwg["free_p_idx"], 1), (rwg["tri_m"], rwg["free_m_idx"], -1)):
        a, b, c = (v[t[tri, i]] for i in range(3))
        area = np.sqrt((np.cross(b - a, c - a) ** 2).sum(1)) / 2
        s = sign * rwg["length"].astype(real) / (2 * area)
        for (l1, l2), w in zip(pts.astype(real), wts.astype(real)):
            r = (a * (1 - l1 - l2) + b * l1) + c * l2
            f = s[:, None] * (r - v[free])
            for o, R in enumerate(RT):
                kh = R[:, 2]
                ph = real(k) * (kh[0] * r[:, 0] + kh[1] * r[:, 1] + kh[2] * r[:, 2])
                cs, sn = np.cos(ph) * area * w, np.sin(ph) * area * w
                for p in (0, 1):
                    E = R[:, p]
                    for j, F in enumerate((E, np.cross(kh, E) / real(eta))):
                        d = f[:, 0] * F[0] + f[:, 1] * F[1] + f[:, 2] * F[2]
                        out[2 * o + p, j * N:(j + 1) * N, 0] += d * cs
                        out[2 * o + p, j * N:(j + 1) * N, 1] += d * sn
    return out


@pytest.mark.parametrize("k", [30.0, 100.0])
def test_error_of_the_phase(k):
    import bem_b200 as bb
    from oracle import bem_oracle as bo
    v, t = bb.icosphere(1.0, 2)
    t = t.astype(np.int64)
    rwg = bo.build_rwg(v, t, "cpp")
    RT = np.linalg.qr(np.random.default_rng(5).standard_normal((12, 3, 3)))[0]
    # edge lengths in 80 bits as well: they come from the same vertices
    edge = [np.setdiff1d(t[a], [f]) for a, f in zip(rwg["tri_p"], rwg["free_p_idx"])]
    vl = v.astype(np.longdouble)
    rwg = dict(rwg, length=np.array([np.sqrt(((vl[i] - vl[j]) ** 2).sum()) for i, j in edge]))
    rule = bb.tri_quadrature(7)
    exact = _sums(v, t, rwg, rule, RT, k, 1.0, np.longdouble)
    plain = _sums(v, t, rwg, rule, RT, k, 1.0, np.float64)
    ctx = bb.Context(0)
    try:
        B = bb.rhs_planewave_dev(bb.Geometry(ctx, v, t.astype(np.int32), 7), complex(k), 1.0, RT).cpu().numpy()
    finally:
        ctx.close()
    e, p = (np.sqrt(((x - exact) ** 2).sum()) for x in (np.stack([B.real, B.imag], -1), plain))
    assert e < 1.03 * p, float(e / p)
