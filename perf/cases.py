"""The timed cases: the calls a user of the dense PMCHWT framework makes, over the sizes it is used at.

A case is one public entry point on one size: operator assembly, plane-wave right-hand sides, the far field and its
Mueller matrix, the FP64 factorisation and solve, the FP32 factorisation with FP64 refinement, GMRES, the whole
pipeline, a batch of particles and the adjoint shape gradient.  `draw` spreads the same calls over meshes of other
sizes (geodesic spheres and octahedra of any frequency give orders that are no multiple of a tile), quadrature
orders, media, orientation and column counts.  `exact` restates every path in plain torch at 64 bits.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bem-cpp_b200"))

import bem_b200 as bb  # noqa: E402

_CTX = None


def _ctx():
    """The one context of the program; the factor memory of a loop of solves is kept, as the benchmark does."""
    global _CTX
    if _CTX is None:
        _CTX = bb.Context(0)
        bb.set_option(_CTX, "cache_factor_memory", 1)
    return _CTX


# ------------------------------------------------------------------- cases
def listed():
    return [
        # a single small particle: set-up call of an interactive script, launch-bound
        {"name": "assemble-ico-960", "do": "assemble", "mesh": "ico", "size": 2, "quad": 7, "ka": 1.0, "m_re": 1.3116,
         "m_im": 0.0},
        # the operator of a large absorbing faceted particle: the main assembly kernel at full occupancy
        {"name": "assemble-hex-18432", "do": "assemble", "mesh": "hex", "size": 4, "quad": 7, "ka": 10.0, "m_re": 1.3116,
         "m_im": 0.01},
        # right-hand sides of a whole orientation average (1395 orientations, both polarisations)
        {"name": "rhs-ico-15360-o1395", "do": "rhs", "mesh": "ico", "size": 4, "quad": 7, "ka": 10.0, "no": 1395},
        # Mueller matrix of a mid-size prism from its 128 solutions
        {"name": "mueller-hex-4608-o64", "do": "mueller", "mesh": "hex", "size": 3, "quad": 7, "ka": 5.0, "no": 64,
         "ntheta": 181},
        # Mueller matrix of a large sphere over 512 orientations
        {"name": "mueller-ico-15360-o512", "do": "mueller", "mesh": "ico", "size": 4, "quad": 7, "ka": 15.0, "no": 512,
         "ntheta": 181},
        # the reference's LU path: FP64 partial pivoting and 128 right-hand sides
        {"name": "lu64-hex-4608-r128", "do": "lu64", "mesh": "hex", "size": 3, "ka": 5.0, "m_re": 1.3116, "m_im": 0.001,
         "nrhs": 128},
        # FP32 factors + FP64 refinement of an orientation average
        {"name": "refine-ico-15360-r2790", "do": "refine", "mesh": "ico", "size": 4, "ka": 10.0, "m_re": 1.3116,
         "m_im": 0.001, "nrhs": 2790},
        # the same on the largest system of a set, an order that is no multiple of a block
        {"name": "refine-geo-29040-r1024", "do": "refine", "mesh": "geo", "size": 22, "ka": 15.0, "m_re": 1.3116,
         "m_im": 0.001, "nrhs": 1024},
        # iterative solve with the exterior operator as preconditioner
        {"name": "gmres-ico-3840-r32", "do": "gmres", "mesh": "ico", "size": 3, "ka": 5.0, "m_re": 1.3116, "m_im": 0.0001,
         "nrhs": 32},
        # host mesh to host Mueller matrix of one small particle in one orientation (latency)
        {"name": "dense-ico-960-single", "do": "dense", "mesh": "ico", "size": 2, "ka": 1.0, "m_re": 1.3116, "m_im": 0.0,
         "na": 1, "nb": 1, "single": True, "fp32": False},
        # a batch of seeded prisms of both sizes, as a particle-population study runs them
        {"name": "batch-hex-16", "do": "batch", "count": 16, "na": 4, "nb": 4},
        # gradient of the M11 misfit in every vertex coordinate: one step of a shape inversion
        {"name": "grad-ico-3840", "do": "grad", "mesh": "ico", "size": 3, "ka": 5.0, "m_re": 1.5, "m_im": 0.01, "na": 8,
         "nb": 8},
    ]


def _order(mesh, size):
    """2N: three edges for two triangles, two unknowns per edge."""
    return 2 * 3 * _triangles(mesh, size) // 2


def _triangles(mesh, size):
    return {"ico": 20 * 4 ** size, "geo": 20 * size * size, "oct": 8 * size * size, "hex": 24 * 4 ** size}[mesh]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _some_mesh(rng, lo, hi):
    """A mesh whose order 2N lies in [lo, hi], spread over its logarithm."""
    for _ in range(200):
        n = _log(rng, lo, hi)
        mesh = rng.choice(["geo", "geo", "oct", "hex"])
        size = (round(math.sqrt(n / 60)) if mesh == "geo" else round(math.sqrt(n / 24)) if mesh == "oct"
                else round(math.log(n / 72, 4)))
        if size >= 1 and lo <= _order(mesh, size) <= hi:
            return mesh, size
    return "geo", max(1, round(math.sqrt(lo / 60)))


def draw(rng):
    do = rng.choice(["assemble", "assemble", "rhs", "mueller", "mueller", "lu64", "lu64", "refine", "refine", "gmres",
                     "dense", "dense", "batch", "grad"])
    if do == "batch":
        return {"do": do, "count": rng.randint(2, 20), "na": rng.randint(1, 5), "nb": rng.randint(1, 5)}
    span = {"assemble": (240, 18432), "rhs": (240, 15360), "mueller": (240, 15360), "lu64": (240, 7000),
            "refine": (500, 25000), "gmres": (240, 4000), "dense": (240, 5000), "grad": (240, 3840)}[do]
    mesh, size = _some_mesh(rng, *span)
    n = _order(mesh, size)
    # a discretisation that resolves the wave: at least about six edges a wavelength inside
    ka = round(_log(rng, 0.5, max(0.6, min(15.0, 0.06 * math.sqrt(n)))), 3)
    absorbing = rng.random() < 0.6
    m_re, m_im = round(rng.uniform(1.3, 1.6), 4), round(_log(rng, 1e-5, 1e-1), 6) if absorbing else 0.0
    c = {"do": do, "mesh": mesh, "size": size, "ka": ka}
    if do in ("assemble", "rhs", "mueller"):
        c["quad"] = rng.choice([7, 7, 4, 13])
    if do == "rhs":
        c["no"] = round(_log(rng, 1, 1395))
    elif do == "mueller":
        c["no"], c["ntheta"] = round(_log(rng, 1, 512)), rng.choice([181, 181, 91, 37, 100, 361])
    else:
        c["m_re"], c["m_im"] = m_re, m_im
    if do == "lu64":
        c["nrhs"] = round(_log(rng, 1, 256))
    elif do == "refine":
        c["nrhs"] = round(_log(rng, 1, 1024 if n > 15360 else 2790))
    elif do == "gmres":
        c["nrhs"] = round(_log(rng, 1, 48))
    elif do in ("dense", "grad"):
        single = rng.random() < 0.3
        c["na"], c["nb"] = (1, 1) if single else (rng.randint(1, 8), rng.randint(1, 8))
        if do == "dense":
            c["single"], c["fp32"] = single, rng.random() < 0.5
    return c


# ------------------------------------------------------------------ inputs
def _geodesic(base, f):
    """The sphere of a triangulated convex solid with every face split into f * f triangles."""
    if base == "geo":
        g = (1 + 5 ** 0.5) / 2
        V = np.array([[-1, g, 0], [1, g, 0], [-1, -g, 0], [1, -g, 0], [0, -1, g], [0, 1, g], [0, -1, -g], [0, 1, -g],
                      [g, 0, -1], [g, 0, 1], [-g, 0, -1], [-g, 0, 1]], dtype=float)
        F = np.array([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2],
                      [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5],
                      [2, 4, 11], [6, 2, 10], [8, 6, 7], [9, 8, 1]])
    else:
        V = np.array([[1, 0, 0], [-1, 0, 0], [0, 1, 0], [0, -1, 0], [0, 0, 1], [0, 0, -1]], dtype=float)
        F = np.array([[0, 2, 4], [2, 1, 4], [1, 3, 4], [3, 0, 4], [2, 0, 5], [1, 2, 5], [3, 1, 5], [0, 3, 5]])
    pts, tris, at = [], [], 0
    for a, b, c in F:
        idx = {}
        for i in range(f + 1):
            for j in range(f + 1 - i):
                idx[i, j] = at
                pts.append((V[a] * (f - i - j) + V[b] * i + V[c] * j) / f)
                at += 1
        for i in range(f):
            for j in range(f - i):
                tris.append((idx[i, j], idx[i + 1, j], idx[i, j + 1]))
                if j < f - i - 1:
                    tris.append((idx[i + 1, j], idx[i + 1, j + 1], idx[i, j + 1]))
    pts = np.array(pts)
    _, first, inv = np.unique(np.round(pts, 9), axis=0, return_index=True, return_inverse=True)
    v = pts[first]
    return v / np.linalg.norm(v, axis=1, keepdims=True), inv.reshape(-1)[np.array(tris)].astype(np.int32)


def _mesh(case, seed):
    """The particle of a seed: a slightly deformed sphere, or a prism of some aspect ratio."""
    rng = np.random.default_rng(seed)
    if case["mesh"] == "hex":
        return bb.hex_prism(float(rng.uniform(0.5, 2.0)), case["size"])
    v, t = bb.icosphere(1.0, case["size"]) if case["mesh"] == "ico" else _geodesic(case["mesh"], case["size"])
    a = rng.uniform(0.95, 1.05, 3)
    r = 1.0 + 0.02 * np.sin(v @ rng.uniform(-3, 3, 3) + rng.uniform(0, 6))
    return v * r[:, None] * a, t


def _directions(no, seed):
    """`no` seeded orientations (uniform over rotations) with weights that add up to one."""
    q = np.random.default_rng(seed + 1).standard_normal((no, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    R = np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                  1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                  1 - 2 * (x * x + y * y)], axis=1)
    return R.reshape(no, 3, 3), np.full(no, 1.0 / no)


def _target(case, seed):
    """The measured M11 a shape inversion fits: a forward-peaked curve with a seeded ripple."""
    rng = np.random.default_rng(seed + 2)
    th = np.linspace(0.0, np.pi, 181)
    return 0.3 * case["ka"] ** 2 * np.exp(-th * rng.uniform(1, 3)) * (1 + 0.1 * np.cos(rng.uniform(3, 9) * th))


def _particles(case, seed):
    return bb.c4_particles(seed, case["count"], orient=(case["na"], case["nb"], 1))


def prepare(case, seed):
    ctx, do = _ctx(), case["do"]
    s = {"case": case, "ctx": ctx, "seed": seed}
    if do == "batch":
        s["particles"] = _particles(case, seed)
        return s
    s["verts"], s["tris"] = _mesh(case, seed)
    s["m"] = complex(case.get("m_re", 1.3116), case.get("m_im", 0.0))
    s["kx"], s["ki"], s["ee"], s["ei"] = bb.physics(case["ka"], s["m"])
    if do == "grad":
        s["target"] = _target(case, seed)
    if do in ("dense", "grad"):
        return s
    s["geom"] = bb.Geometry(ctx, s["verts"], s["tris"], case.get("quad", 7))
    n = s["geom"].n
    if do == "assemble":
        s["Z"] = torch.empty((n, n), dtype=torch.complex128, device="cuda")
    elif do == "rhs":
        s["RT"], _ = _directions(case["no"], seed)
        s["B"] = torch.empty((2 * case["no"], n), dtype=torch.complex128, device="cuda")
    elif do == "mueller":
        s["RT"], s["w"] = _directions(case["no"], seed)
        # surface currents with the phase of their incident wave, as solutions have, and a seeded tenth of scatter
        X = bb.rhs_planewave_dev(s["geom"], s["kx"], s["ee"], s["RT"])
        g = torch.Generator("cuda").manual_seed(seed)
        noise = torch.randn((2 * case["no"], n, 2), generator=g, dtype=torch.float64, device="cuda")
        s["X"] = X + 0.1 * X.abs().pow(2).mean().sqrt() * torch.view_as_complex(noise)
    else:
        s["Z"] = bb.assemble_pmchwt_dev(s["geom"], s["kx"], s["ki"], s["ee"], s["ei"])
        RT, _ = _directions((case["nrhs"] + 1) // 2, seed)
        s["B"] = bb.rhs_planewave_dev(s["geom"], s["kx"], s["ee"], RT)[:case["nrhs"]].contiguous()
        s["X"] = torch.empty_like(s["B"])
        if do == "lu64":
            s["work"] = torch.empty_like(s["Z"])
    return s


def run(s):
    case, ctx, do = s["case"], s["ctx"], s["case"]["do"]
    if do == "assemble":
        return bb.assemble_pmchwt_dev(s["geom"], s["kx"], s["ki"], s["ee"], s["ei"], Z=s["Z"])
    if do == "rhs":
        return bb.rhs_planewave_dev(s["geom"], s["kx"], s["ee"], s["RT"], B=s["B"])
    if do == "mueller":
        return bb.mueller_from_solutions_dev(s["geom"], s["X"], s["RT"], s["w"], s["kx"], s["ee"], ntheta=case["ntheta"])
    if do == "lu64":
        s["work"].copy_(s["Z"])  # the factors replace the matrix
        lu = bb.LU(ctx, s["work"], bb.PREC_FP64)
        X, _ = lu.solve(s["B"], X=s["X"])
        lu.close()
        return X
    if do == "refine":
        lu = bb.LU(ctx, s["Z"], bb.PREC_FP32_REFINE)
        X, _ = lu.solve(s["B"], X=s["X"], tol=2e-10)
        lu.close()
        return X
    if do == "gmres":
        M, _ = bb.build_aext_preconditioner(s["geom"], s["kx"], s["ee"])
        X, info = bb.gmres(ctx, s["Z"], s["B"], M, tol=1e-8, restart=200, maxiter=200)
        M.close()
        return X
    if do == "dense":
        M, _ = bb.dense_run(ctx, s["verts"], s["tris"], case["ka"], s["m"], single=case["single"],
                            orient=(case["na"], case["nb"], 1), precision=bb.PREC_FP32_REFINE if case["fp32"] else bb.PREC_FP64)
        return M
    if do == "batch":
        return [M for M, _ in bb.batch_run(ctx, s["particles"])]
    loss, grad, M = bb.adjoint_grad_vertices(ctx, s["verts"], s["tris"], case["ka"], s["m"], s["target"],
                                             orient=(case["na"], case["nb"], 1))
    return {"loss": loss, "grad": grad, "mueller": M}


# --------------------------------------------------------- work, tolerance
def work(case):
    """Unavoidable traffic and arithmetic: a complex multiply-add is 8, a complex exponential about 40 operations."""
    do = case["do"]
    if do == "batch":
        # half of the seeded prisms have order 1152, half 4608
        per = [_solve_work(n, 2 * case["na"] * case["nb"], False) for n in (1152, 4608)]
        return {k: case["count"] * (per[0][k] + per[1][k]) / 2 for k in ("bytes", "flops")}
    n, t, q = _order(case["mesh"], case["size"]), _triangles(case["mesh"], case["size"]), case.get("quad", 7)
    if do == "assemble":  # each unordered pair of triangles, both media: the exponential and 18 complex moments
        return {"bytes": 16.0 * n * n, "flops": t * (t + 1) / 2 * q * q * 2 * (40 + 18 * 4)}
    if do == "rhs":
        return {"bytes": 16.0 * n * 2 * case["no"], "flops": case["no"] * t * (q * 50.0 + 100)}
    if do == "mueller":
        return {"bytes": 16.0 * n * 2 * case["no"], "flops": case["no"] * case["ntheta"] * t * (q * 50.0 + 100)}
    if do in ("lu64", "refine"):
        return _solve_work(n, case["nrhs"], do == "refine")
    if do == "gmres":
        return {"bytes": 2 * 16.0 * n * n, "flops": 8 / 3 * n ** 3 + 20 * 16.0 * n * n * case["nrhs"]}
    cols = 2 if case.get("single") else 2 * case["na"] * case["nb"]
    a = work(dict(case, do="assemble"))
    f = work(dict(case, do="mueller", no=max(1, cols // 2), ntheta=181))
    b = _solve_work(n, cols, case.get("fp32", False))
    times = 2 if do == "grad" else 1
    return {k: a[k] * times + f[k] * times + b[k] * (1.25 if do == "grad" else 1) for k in ("bytes", "flops")}


def _solve_work(n, nrhs, fp32):
    # partial pivoting: 8/3 n^3; the symmetric FP32 factors: 4/3 n^3, then two residuals and three solves
    if fp32:
        return {"bytes": 16.0 * n * n + 32.0 * n * nrhs, "flops": 4 / 3 * n ** 3 + 5 * 8.0 * n * n * nrhs}
    return {"bytes": 32.0 * n * n + 32.0 * n * nrhs, "flops": 8 / 3 * n ** 3 + 8.0 * n * n * nrhs}


def tolerance(case):
    # about four times the largest error against exact() over the ranges.  Assembly: the finite difference of the
    # singular term (step 1e-6) amplifies the rounding of its quadrature; solves: the condition of the operator times
    # the unit roundoff; refinement and GMRES: the tolerance that the call asks for; gradient: its same-triangle
    # differences (step 1e-4 of an edge)
    do = case["do"]
    if do == "dense":
        return {"rel": 1e-10 if case["fp32"] else 1e-12}
    return {"rel": {"assemble": 4e-12, "rhs": 1e-14, "mueller": 1e-14, "lu64": 4e-12, "refine": 2e-10, "gmres": 1e-8,
                    "batch": 1e-12, "grad": 1e-9}[do]}


# ------------------------------------------------ the same in plain torch
def _rule(order):
    p, w = bb.tri_quadrature(order)  # the published barycentric tables
    return np.column_stack([1 - p.sum(axis=1), p]), w


class _Surface:
    """Points, weights and the three basis halves of every triangle of a closed surface, in 64 bits."""

    def __init__(self, v, t, order):
        v, t = np.asarray(v, dtype=np.float64), np.asarray(t, dtype=np.int64)
        lam, wq = _rule(order)
        T = len(t)
        e = np.stack([t, np.roll(t, -1, axis=1)], axis=2).reshape(-1, 2)  # edge j of triangle i at 3 i + j
        lo, hi = e.min(axis=1), e.max(axis=1)
        o = np.lexsort((np.arange(3 * T), hi, lo))
        assert np.array_equal(lo[o[::2]], lo[o[1::2]]) and np.array_equal(hi[o[::2]], hi[o[1::2]])
        self.N, self.T, self.q = len(o) // 2, T, len(wq)
        n_of, sign = np.empty(3 * T, dtype=np.int64), np.empty(3 * T)
        n_of[o], sign[o] = np.repeat(np.arange(self.N), 2), np.tile([1.0, -1.0], self.N)
        area = 0.5 * np.linalg.norm(np.cross(v[t[:, 1]] - v[t[:, 0]], v[t[:, 2]] - v[t[:, 0]]), axis=1)
        length = np.linalg.norm(v[hi] - v[lo], axis=1).reshape(T, 3)
        s = sign.reshape(T, 3) * length / (2 * area[:, None])
        cu = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda() if torch.cuda.is_available() else torch.from_numpy(np.ascontiguousarray(x))  # noqa: E731
        self.n = cu(n_of.reshape(T, 3))
        self.tv, self.free, self.s, self.div = cu(v[t]), cu(v[np.roll(t, -2, axis=1)]), cu(s), cu(2 * s)
        self.w, self.area, self.lam, self.wq = cu(area[:, None] * wq), cu(area), cu(lam), cu(wq)
        self.r = torch.einsum("ql,tlx->tqx", self.lam, self.tv)
        self.f = self.s[:, :, None, None] * (self.r[:, None] - self.free[:, :, None])  # (T, 3, q, xyz)
        self.fw = self.f * self.w[:, None, :, None]
        self.dw = self.div[:, :, None] * self.w[:, None, :]
        self.cw = torch.linalg.cross(self.fw, self.r[:, None].expand_as(self.fw))

    def rows(self, x):
        """Sparse (N, points) matrix of per-half point values x (T, 3, q)."""
        at = torch.arange(self.T * self.q, device=x.device).reshape(self.T, 1, self.q).expand(self.T, 3, self.q)
        i = torch.stack([self.n[:, :, None].expand_as(at).reshape(-1), at.reshape(-1)])
        return torch.sparse_coo_tensor(i, x.reshape(-1).to(torch.complex128), (self.N, self.T * self.q)).coalesce().to_sparse_csr()

    def singular(self):
        """Symmetrised same-triangle corrections (A, B) of the scalar and vector potentials, (N, N) real."""
        v, r = self.tv, self.r
        nh = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
        nh = nh / nh.norm(dim=1, keepdim=True)
        P = torch.zeros(self.T, self.q, dtype=torch.float64, device=r.device)
        for i in range(3):
            a, b = v[:, i], v[:, (i + 1) % 3]
            th = (b - a) / (b - a).norm(dim=1, keepdim=True)
            d = ((r - a[:, None]) * torch.linalg.cross(nh, th)[:, None]).sum(-1)
            sp, sm = ((b[:, None] - r) * th[:, None]).sum(-1), ((a[:, None] - r) * th[:, None]).sum(-1)
            P += d * torch.log(((b[:, None] - r).norm(dim=-1) + sp) / ((a[:, None] - r).norm(dim=-1) + sm))
        eps, gw = 1e-6, []
        for x in range(3):
            off = torch.zeros(3, dtype=torch.float64, device=r.device)
            off[x] = eps
            W = [self.area[:, None] * ((r[:, None] - (r + sg * off)[:, :, None]).norm(dim=-1) * self.wq).sum(-1) for sg in (1, -1)]
            gw.append((W[0] - W[1]) / (2 * eps))
        V = r * P[..., None] - torch.stack(gw, dim=-1)
        src = self.s[:, :, None, None] * (V[:, None] - self.free[:, :, None] * P[:, None, :, None])
        A = torch.einsum("ta,tb,t->tab", self.div, self.div, (P * self.w).sum(1)) / (4 * math.pi)
        B = torch.einsum("taqx,tbqx->tab", self.fw, src) / (4 * math.pi)
        out = []
        for x in (A, B):
            S = torch.zeros(self.N * self.N, dtype=torch.float64, device=r.device)
            S.index_add_(0, (self.n[:, :, None] * self.N + self.n[:, None, :]).reshape(-1), x.reshape(-1))
            S = S.reshape(self.N, self.N)
            out.append((S + S.T) / 2)
        return out

    def operators(self, ks):
        """[(L, K)] of each wavenumber of ks."""
        P, dev = self.T * self.q, self.r.device
        rows = [self.rows(self.fw[..., x]) for x in range(3)] + [self.rows(self.cw[..., x]) for x in range(3)] + [self.rows(self.dw)]
        c128 = dict(dtype=torch.complex128, device=dev)
        out = [(torch.zeros(self.N, self.N, **c128), torch.zeros(self.N, self.N, **c128)) for _ in ks]
        r, step = self.r.reshape(P, 3), max(1, min(self.T, int(4e7 / P / self.q)))
        for t0 in range(0, self.T, step):
            t1 = min(self.T, t0 + step)
            c, cols = slice(t0, t1), slice(t0 * self.q, t1 * self.q)
            R = (r[:, None, 0] - r[None, cols, 0]).square_()
            for x in (1, 2):
                R += (r[:, None, x] - r[None, cols, x]).square_()
            R = R.sqrt_().clamp_(min=1e-15)
            tri = torch.arange(P, device=dev) // self.q
            same = tri[:, None] == tri[None, cols]
            back = lambda H, w: torch.einsum("ntq,taq->nta", H.reshape(self.N, t1 - t0, self.q), w.to(torch.complex128)).reshape(self.N, -1)  # noqa: E731
            at = self.n[c].reshape(-1)
            for (L, K), k in zip(out, ks):
                amp = torch.exp(-k.imag * R) / (4 * math.pi * R) if k.imag else 1 / (4 * math.pi * R)
                G = torch.polar(amp, k.real * R)
                g = torch.where(same, torch.zeros((), **c128), G * (1j * k * R - 1) / (R * R))
                G = torch.where(same, G - 1 / (4 * math.pi * R), G)
                add = sum(1j * k * back(rows[x] @ G, self.fw[c][..., x]) for x in range(3)) - 1j / k * back(rows[6] @ G, self.dw[c])
                L.index_add_(1, at, add)
                add = sum(back(rows[3 + x] @ g, self.fw[c][..., x]) + back(rows[x] @ g, self.cw[c][..., x]) for x in range(3))
                K.index_add_(1, at, add)
        A, B = self.singular()
        for (L, _), k in zip(out, ks):
            L += -1j / k * A + 1j * k * B
        return out

    def pmchwt(self, kx, ki, ee, ei):
        (Le, Ke), (Li, Ki) = self.operators([kx, ki])
        K = Ke + Ki
        return torch.cat([torch.cat([ee * Le + ei * Li, -K], 1), torch.cat([K, Le / ee + Li / ei], 1)], 0)

    def plane_waves(self, kx, ee, RT):
        """(2 no, 2 N): E and H of both polarisations tested with the basis."""
        RT = torch.from_numpy(np.ascontiguousarray(RT)).to(self.r.device)
        r, rows, out = self.r.reshape(-1, 3), [self.rows(self.fw[..., x]) for x in range(3)], []
        for o in range(0, len(RT), 64):
            R = RT[o:o + 64]
            kh = R[:, :, 2]
            ph = torch.polar(torch.ones((), dtype=torch.float64, device=r.device), kx.real * (r @ kh.T))
            F = torch.stack([x @ ph for x in rows])  # (3, N, o)
            for p in (0, 1):
                E = R[:, :, p]
                H = torch.linalg.cross(kh, E) / ee
                out.append(torch.cat([torch.einsum("xno,ox->on", F, e.to(F.dtype)) for e in (E, H)], 1))
        blocks = [torch.stack([out[i], out[i + 1]], 1).reshape(-1, 2 * self.N) for i in range(0, len(out), 2)]
        return torch.cat(blocks)

    def mueller(self, X, RT, w, kx, ee, ntheta):
        """(4, 4, ntheta): the weighted Mueller matrix over |k|^2 from solutions X (2 no, 2 N)."""
        dev = self.r.device
        th = torch.linspace(0, math.pi, ntheta, dtype=torch.float64, device=dev)
        st, ct = torch.sin(th), torch.cos(th)
        fw, r = self.fw.to(torch.complex128), self.r.reshape(-1, 3)
        total = torch.zeros(16, ntheta, dtype=torch.float64, device=dev)
        for o in range(len(RT)):
            R = torch.from_numpy(np.ascontiguousarray(RT[o])).to(dev)
            d = st[:, None] * R[:, 0] + ct[:, None] * R[:, 2]
            ph = torch.polar(torch.ones((), dtype=torch.float64, device=dev), -kx.real * (d @ r.T))
            c = X[2 * o:2 * o + 2].reshape(2, 2, self.N)  # (pol, J / M, N)
            cur = torch.einsum("pjta,taqx->tqpjx", c[:, :, self.n], fw).reshape(-1, 12)
            S = (ph @ cur).reshape(ntheta, 2, 2, 3)
            dd = d.to(torch.complex128)
            e = torch.stack([ct[:, None] * R[:, 0] - st[:, None] * R[:, 2], R[:, 1].expand(ntheta, 3)], 1).to(torch.complex128)
            amp = []
            for p in (0, 1):
                J, M = S[:, p, 0], S[:, p, 1]
                F = -1j * kx / (4 * math.pi) * (ee * (J - dd * (dd * J).sum(1, keepdim=True)) - torch.linalg.cross(dd, M))
                amp.append(-1j * kx * (e * F[:, None]).sum(-1))
            S2, S4, S3, S1 = amp[0][:, 0], amp[0][:, 1], amp[1][:, 0], amp[1][:, 1]
            a1, a2, a3, a4 = (x.abs() ** 2 for x in (S1, S2, S3, S4))
            z = lambda a, b: a * b.conj()  # noqa: E731
            m = [(a1 + a2 + a3 + a4) / 2, (a2 - a1 + a4 - a3) / 2, (z(S2, S3) + z(S1, S4)).real, (z(S2, S3) - z(S1, S4)).imag,
                 (a2 - a1 - a4 + a3) / 2, (a2 + a1 - a4 - a3) / 2, (z(S2, S3) - z(S1, S4)).real, (z(S2, S3) + z(S1, S4)).imag,
                 (z(S2, S4) + z(S1, S3)).real, (z(S2, S4) - z(S1, S3)).real, (z(S1, S2) + z(S3, S4)).real,
                 (z(S2, S1) + z(S4, S3)).imag, (z(S4, S2) + z(S1, S3)).imag, (z(S4, S2) - z(S1, S3)).imag,
                 (z(S1, S2) - z(S3, S4)).imag, (z(S1, S2) - z(S3, S4)).real]
            total += w[o] / abs(kx) ** 2 * torch.stack(m)
        return total.reshape(4, 4, ntheta).cpu().numpy()


def _orientations(na, nb):
    """The reference's average: uniform alpha, Gauss-Legendre cos(beta)."""
    return bb.generate_orientations(na, nb, 1, sort_nearest=True)


def _whole(v, t, ka, m, RT, w):
    s = _Surface(v, t, 7)
    kx, ki, ee, ei = complex(ka), complex(ka) * m, 1.0, 1.0 / abs(m)
    X = torch.linalg.solve(s.pmchwt(kx, ki, ee, ei), s.plane_waves(kx, ee, RT).T).T.contiguous()
    return s.mueller(X, RT, w, kx, ee, 181)


def exact(case, seed):
    do = case["do"]
    if do == "batch":
        out = []
        for p in _particles(case, seed):
            out.append(_whole(p["verts"], p["tris"], p["ka"], p["m"], *_orientations(case["na"], case["nb"])))
        return out
    if do in ("dense", "grad"):
        v, t = _mesh(case, seed)
        m = complex(case["m_re"], case["m_im"])
        RT, w = (np.eye(3)[None], np.ones(1)) if case.get("single") else _orientations(case["na"], case["nb"])
        M = _whole(v, t, case["ka"], m, RT, w)
        if do == "dense":
            return M
        # the gradient of 3 nv coordinates has no cheap 64-bit counterpart (2 * 3 nv solves)
        return {"loss": float(((M[0, 0] - _target(case, seed)) ** 2).sum()), "grad": None, "mueller": M}
    s = prepare(case, seed)
    if do in ("lu64", "refine", "gmres"):
        return torch.linalg.solve(s["Z"], s["B"].T).T.contiguous()
    surface = _Surface(s["verts"], s["tris"], case["quad"])
    if do == "assemble":
        if case["quad"] * _triangles(case["mesh"], case["size"]) > 50000:
            return None
        return surface.pmchwt(s["kx"], s["ki"], s["ee"], s["ei"])
    if do == "rhs":
        return surface.plane_waves(s["kx"], s["ee"], s["RT"])
    return surface.mueller(s["X"], s["RT"], s["w"], s["kx"], s["ee"], case["ntheta"])
