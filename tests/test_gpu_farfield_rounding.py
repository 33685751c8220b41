"""Mueller matrices from the band limit against 80-bit sums over RWG halves, at the call's angles pi i / (ntheta - 1) in
64 bits.

Bound: 4.5e-16 in the 2-norm, four units of 2^-53.  A coefficient sum carries about one unit (its terms' roundings add up
as a random walk that grouping keeps short), half a unit each from the nodes and the weights, and an element of the matrix
twice that.  Errors of a node's angle or of a weight are the same for every triangle and orientation, so one more place
lost there shows at once: 8e-16 with plain weights summed in the order of the nodes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD, CL = np.longdouble, np.clongdouble
PI = LD("3.14159265358979323846264338327950288")


def _mueller(v, t, rwg, rule, X, RT, w, k, theta):
    """(16, ntheta) of the oracle's formulas, every sum in 80 bits."""
    N, vl = rwg["N"], v.astype(LD)
    edge = np.array([np.setdiff1d(t[a], [f]) for a, f in zip(rwg["tri_p"], rwg["free_p_idx"])])
    length = np.sqrt(((vl[edge[:, 0]] - vl[edge[:, 1]]) ** 2).sum(1))
    pos, f = [], []
    for tri, free, sign in ((rwg["tri_p"], rwg["free_p_idx"], 1), (rwg["tri_m"], rwg["free_m_idx"], -1)):
        a, b, c = (vl[t[tri, i]] for i in range(3))
        for (l1, l2), wq in zip(rule[0].astype(LD), rule[1].astype(LD)):
            r = (a * (1 - l1 - l2) + b * l1) + c * l2
            pos.append(r)
            f.append((sign * length * wq / 2)[:, None] * (r - vl[free]))
    n = np.tile(np.arange(N), len(pos))
    pos, f, st, ct = np.concatenate(pos), np.concatenate(f), np.sin(theta.astype(LD)), np.cos(theta.astype(LD))
    total, k = np.zeros((16, len(theta)), LD), LD(k)
    for o, R in enumerate(RT.astype(LD)):
        x1, x2 = pos @ R[:, 0], pos @ R[:, 2]
        cur = np.concatenate([f * X[2 * o + p].astype(CL)[h * N:(h + 1) * N][n][:, None] for p in (0, 1) for h in (0, 1)], 1)
        ph = [k * (s * x1 + c * x2) for s, c in zip(st, ct)]
        S = np.stack([(np.cos(x) - 1j * np.sin(x)).astype(CL) @ cur for x in ph])
        d = st[:, None] * R[:, 0] + ct[:, None] * R[:, 2]
        e = ct[:, None] * R[:, 0] - st[:, None] * R[:, 2]
        amp = []
        for p in (0, 1):
            J, M = S[:, 6 * p:6 * p + 3], S[:, 6 * p + 3:6 * p + 6]
            F = -1j * k / (4 * PI) * ((J - d * (d * J).sum(1)[:, None]) - np.cross(d, M))
            amp += [-1j * k * (e * F).sum(1), -1j * k * (R[:, 1] * F).sum(1)]
        S2, S4, S3, S1 = amp
        a1, a2, a3, a4 = (abs(x) ** 2 for x in (S1, S2, S3, S4))
        z = lambda a, b: a * b.conj()  # noqa: E731
        total += LD(w[o]) / k ** 2 * np.stack([
            (a1 + a2 + a3 + a4) / 2, (a2 - a1 + a4 - a3) / 2, (z(S2, S3) + z(S1, S4)).real, (z(S2, S3) - z(S1, S4)).imag,
            (a2 - a1 - a4 + a3) / 2, (a2 + a1 - a4 - a3) / 2, (z(S2, S3) - z(S1, S4)).real, (z(S2, S3) + z(S1, S4)).imag,
            (z(S2, S4) + z(S1, S3)).real, (z(S2, S4) - z(S1, S3)).real, (z(S1, S2) + z(S3, S4)).real,
            (z(S2, S1) + z(S4, S3)).imag, (z(S4, S2) + z(S1, S3)).imag, (z(S4, S2) - z(S1, S3)).imag,
            (z(S1, S2) - z(S3, S4)).imag, (z(S1, S2) - z(S3, S4)).real])
    return total


@pytest.mark.parametrize("size,k,no,ntheta,quad", [(2, 1.0, 1, 61, 7), (2, 6.0, 2, 100, 4), (3, 15.0, 2, 91, 7),
                                                   (1, 3.0, 3, 37, 13)])
def test_error_of_the_interpolated_sums(size, k, no, ntheta, quad):
    import bem_b200 as bb
    import torch
    from oracle import bem_oracle as bo
    v, t = bb.icosphere(1.0, size)
    v = v * np.array([1.03, 0.97, 1.01])
    rwg = bo.build_rwg(v, t.astype(np.int64), "cpp")
    rng = np.random.default_rng(size)
    RT, w = np.linalg.qr(rng.standard_normal((no, 3, 3)))[0], rng.uniform(0.2, 1.0, no)
    # currents with the phase of their incident wave, as solutions have, and a tenth of scatter
    mid, d, N = (rwg["free_p"] + rwg["free_m"]) / 2, rwg["free_m"] - rwg["free_p"], rwg["N"]
    X = np.empty((2 * no, 2 * N), complex)
    for o, R in enumerate(RT):
        ph = np.exp(1j * k * mid @ R[:, 2])
        for p in (0, 1):
            X[2 * o + p] = np.concatenate([d @ np.cross(R[:, 2], R[:, p]) * ph, d @ R[:, p] * ph])
    X += 0.1 * np.sqrt((abs(X) ** 2).mean()) * (rng.standard_normal(X.shape) + 1j * rng.standard_normal(X.shape))
    theta = np.array([np.pi * i / (ntheta - 1) for i in range(ntheta)])
    want = _mueller(v, t.astype(np.int64), rwg, bb.tri_quadrature(quad), X, RT, w, k, theta)
    ctx = bb.Context(0)
    try:
        M = bb.mueller_from_solutions_dev(bb.Geometry(ctx, v, t, quad), torch.from_numpy(X).cuda(), RT, w, complex(k), 1.0,
                                          ntheta=ntheta)
    finally:
        ctx.close()
    err = np.sqrt(((M.reshape(16, -1) - want) ** 2).sum() / (want ** 2).sum())
    assert err < 4.5e-16, float(err)
