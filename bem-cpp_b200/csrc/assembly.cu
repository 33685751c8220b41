// PMCHWT assembly on the device (FP64).
//
// Restates assemble_LK_kernel (assembly.cu:14-135), precompute_half
// (assembly.cu:150-201), apply_singular_corrections (assembly.cu:208-321),
// the symmetrisation (assembly.cu:494-502) and the block fill of
// assemble_pmchwt (pmchwt.cu:36-51) as one device pipeline:
//
//   1. graglia_kernel     -- per (triangle, point): Graglia P and the
//                            finite-difference vector potential V (FP64).
//   2. assemble_kernel    -- per 16x16 tile of RWG pairs (m <= n tiles only):
//                            all four half pairs, both media, quadrature part of
//                            L and K, written straight into the four Z blocks and
//                            mirrored (L and K are symmetric).
//   3. singular_fixup     -- per RWG pair sharing a triangle: the symmetrised
//                            same-triangle correction (S[m,n] + S[n,m])/2.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "asm_device.cuh"
#include "bem_internal.h"

namespace bem {


// ------------------------------------------------------------ geometry upload
bool host_mesh_from(const double* verts, int nv, const int* tris, int nt, HostMesh* m);

// Position-dependent geometry arrays (everything the vertex coordinates
// enter): per-half quadrature points, basis values, weights, divergences,
// free vertices; triangle vertices; per-triangle centroid-relative data.
struct PosArrays {
    std::vector<double> px, py, pz, fx, fy, fz, cx, cy, cz, jw, div, coef, frx, fry, frz, tv, tc, tu, tjw, hpi;
    std::vector<int> tri;
};

static void position_arrays(const bem_geom* g, PosArrays& A) {
    const HostMesh& m = g->mesh;
    const HostRWG& r = g->rwg;
    const Quad& q = g->quad;
    const int N = r.N, Nq = q.n, nt = m.nt();
    const size_t P = (size_t)2 * N * Nq;
    auto& px = A.px; auto& py = A.py; auto& pz = A.pz; auto& fx = A.fx; auto& fy = A.fy; auto& fz = A.fz;
    auto& cx = A.cx; auto& cy = A.cy; auto& cz = A.cz; auto& jw = A.jw;
    for (auto* v : {&px, &py, &pz, &fx, &fy, &fz, &cx, &cy, &cz, &jw}) v->assign(P, 0.0);
    auto& div = A.div; auto& coef = A.coef; auto& frx = A.frx; auto& fry = A.fry; auto& frz = A.frz;
    for (auto* v : {&div, &coef, &frx, &fry, &frz}) v->assign(2 * N, 0.0);
    auto& tri = A.tri;
    tri.assign(2 * N, 0);
    for (int h = 0; h < 2; h++) {
        int sign = h == 0 ? 1 : -1;
        for (int n = 0; n < N; n++) {
            int t = h == 0 ? r.tri_p[n] : r.tri_m[n];
            V3 fr = h == 0 ? r.free_p[n] : r.free_m[n];
            double area = h == 0 ? r.area_p[n] : r.area_m[n];
            double c = sign * r.length[n] / (2.0 * area);
            int hn = h * N + n;
            div[hn] = sign * r.length[n] / area;
            coef[hn] = c;
            frx[hn] = fr.x, fry[hn] = fr.y, frz[hn] = fr.z;
            tri[hn] = t;
            V3 v0 = m.verts[m.tris[3 * t]], v1 = m.verts[m.tris[3 * t + 1]],
               v2 = m.verts[m.tris[3 * t + 2]];
            for (int k = 0; k < Nq; k++) {
                double l1 = q.l1[k], l2 = q.l2[k], l0 = 1.0 - l1 - l2;
                // r = v0 l0 + v1 l1 + v2 l2, evaluated left to right as the reference
                double rx = (v0.x * l0 + v1.x * l1) + v2.x * l2;
                double ry = (v0.y * l0 + v1.y * l1) + v2.y * l2;
                double rz = (v0.z * l0 + v1.z * l1) + v2.z * l2;
                double ffx = (rx - fr.x) * c, ffy = (ry - fr.y) * c, ffz = (rz - fr.z) * c;
                size_t i = (size_t)hn * Nq + k;
                px[i] = rx, py[i] = ry, pz[i] = rz;
                fx[i] = ffx, fy[i] = ffy, fz[i] = ffz;
                cx[i] = ffy * rz - ffz * ry;
                cy[i] = ffz * rx - ffx * rz;
                cz[i] = ffx * ry - ffy * rx;
                jw[i] = area * q.w[k];
            }
        }
    }
    auto& tv = A.tv;
    tv.assign(9 * (size_t)nt, 0.0);
    for (int t = 0; t < nt; t++)
        for (int j = 0; j < 3; j++) {
            V3 v = m.verts[m.tris[3 * t + j]];
            tv[9 * t + 3 * j] = v.x, tv[9 * t + 3 * j + 1] = v.y, tv[9 * t + 3 * j + 2] = v.z;
        }
    // triangle-pair assembly data: per triangle the centroid, the quadrature
    // points relative to it (the same points as the halves') and area x
    // weight; per half the free vertex relative to its triangle's centroid
    auto& tc = A.tc; auto& tu = A.tu; auto& tjw = A.tjw; auto& hpi = A.hpi;
    tc.assign(3 * (size_t)nt, 0.0);
    tu.assign(3 * (size_t)nt * Nq, 0.0);
    tjw.assign((size_t)nt * Nq, 0.0);
    hpi.assign(3 * (size_t)2 * N, 0.0);
    std::vector<double> tarea(nt, -1.0);
    for (int h = 0; h < 2; h++)
        for (int n = 0; n < N; n++) {
            const int t = h == 0 ? r.tri_p[n] : r.tri_m[n];
            if (tarea[t] < 0) tarea[t] = h == 0 ? r.area_p[n] : r.area_m[n];
        }
    for (int t = 0; t < nt; t++) {
        V3 v0 = m.verts[m.tris[3 * t]], v1 = m.verts[m.tris[3 * t + 1]], v2 = m.verts[m.tris[3 * t + 2]];
        const double cx0 = (v0.x + v1.x + v2.x) / 3.0, cy0 = (v0.y + v1.y + v2.y) / 3.0,
                     cz0 = (v0.z + v1.z + v2.z) / 3.0;
        tc[3 * t] = cx0, tc[3 * t + 1] = cy0, tc[3 * t + 2] = cz0;
        for (int k = 0; k < Nq; k++) {
            double l1 = q.l1[k], l2 = q.l2[k], l0 = 1.0 - l1 - l2;
            double rx = (v0.x * l0 + v1.x * l1) + v2.x * l2;
            double ry = (v0.y * l0 + v1.y * l1) + v2.y * l2;
            double rz = (v0.z * l0 + v1.z * l1) + v2.z * l2;
            size_t i = ((size_t)t * Nq + k) * 3;
            tu[i] = rx - cx0, tu[i + 1] = ry - cy0, tu[i + 2] = rz - cz0;
            tjw[(size_t)t * Nq + k] = (tarea[t] > 0 ? tarea[t] : 0.0) * q.w[k];
        }
    }
    for (int h = 0; h < 2; h++)
        for (int n = 0; n < N; n++) {
            const int t = h == 0 ? r.tri_p[n] : r.tri_m[n];
            const V3 fr = h == 0 ? r.free_p[n] : r.free_m[n];
            size_t i = ((size_t)h * N + n) * 3;
            hpi[i] = fr.x - tc[3 * t], hpi[i + 1] = fr.y - tc[3 * t + 1], hpi[i + 2] = fr.z - tc[3 * t + 2];
        }
}

// g->rmax and g->extent: the largest |r| and a bound of |r - r'| (the diagonal
// of the bounding box, which unlike 2 rmax does not grow with the distance from
// the origin) over the vertices and so over all quadrature points.
static void mesh_bounds(bem_geom* g) {
    double r2 = 0.0, lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (const V3& v : g->mesh.verts) {
        const double x[3] = {v.x, v.y, v.z};
        r2 = std::max(r2, x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
        for (int i = 0; i < 3; i++) lo[i] = std::min(lo[i], x[i]), hi[i] = std::max(hi[i], x[i]);
    }
    g->rmax = std::sqrt(r2);
    g->extent = std::sqrt((hi[0] - lo[0]) * (hi[0] - lo[0]) + (hi[1] - lo[1]) * (hi[1] - lo[1]) +
                          (hi[2] - lo[2]) * (hi[2] - lo[2]));
}

// RWG order of the assembly tiles (ASM_TILE consecutive ones each): patches
// grown over shared triangles.  A tile starts at the first triangle along the
// Morton order that still has RWGs to place, and takes in turn an RWG whose
// two triangles it already has, else the one whose other triangle has the
// fewest RWGs left outside the patch (it would be left behind otherwise), the
// nearest to the patch's centre among equals.  15.5-15.8 distinct triangles
// per 16 RWGs on spheres and prisms against 17.1 along the Morton curve
// itself: 18 % fewer triangle pairs in the assembly.
static std::vector<int> patch_order(const HostRWG& r, int nt, const std::vector<double>& tc,
                                    const std::vector<int>& torder) {
    const int N = r.N;
    std::vector<int> first(nt + 1, 0), on(2 * (size_t)N), left(nt, 0);
    for (int n = 0; n < N; n++) first[r.tri_p[n] + 1]++, first[r.tri_m[n] + 1]++;
    for (int t = 0; t < nt; t++) left[t] = first[t + 1], first[t + 1] += first[t];
    {
        std::vector<int> at(first.begin(), first.end() - 1);
        for (int n = 0; n < N; n++) on[at[r.tri_p[n]]++] = n, on[at[r.tri_m[n]]++] = n;
    }
    std::vector<char> used(N, 0);
    std::vector<int> in_cand(N, -1), in_tile(nt, -1), cand, perm;
    perm.reserve(N);
    int ptr = 0, tile = 0, cnt = 0, ntri = 0;
    double sum[3] = {0, 0, 0};
    auto add_tri = [&](int t) {
        in_tile[t] = tile;
        ntri++;
        for (int j = 0; j < 3; j++) sum[j] += tc[3 * (size_t)t + j];
        for (int i = first[t]; i < first[t + 1]; i++)
            if (!used[on[i]] && in_cand[on[i]] != tile) in_cand[on[i]] = tile, cand.push_back(on[i]);
    };
    while ((int)perm.size() < N) {
        if (cand.empty()) {
            while (left[torder[ptr]] == 0) ptr++;
            add_tri(torder[ptr]);
        }
        size_t best = 0;
        int best_key = 1 << 30;
        double best_d = 0.0;
        for (size_t i = 0; i < cand.size(); i++) {
            const int n = cand[i], ta = r.tri_p[n], tb = r.tri_m[n];
            const bool ha = in_tile[ta] == tile, hb = in_tile[tb] == tile;
            if (ha && hb) {
                best = i;
                break;
            }
            const int t = ha ? tb : ta;
            int key = 0;
            for (int k = first[t]; k < first[t + 1]; k++)
                if (!used[on[k]]) key += in_cand[on[k]] == tile ? -1 : 1;
            if (key > best_key) continue;
            double d = 0.0;
            for (int j = 0; j < 3; j++) {
                const double x = tc[3 * (size_t)t + j] - sum[j] / ntri;
                d += x * x;
            }
            if (key < best_key || d < best_d) best = i, best_key = key, best_d = d;
        }
        const int n = cand[best];
        cand.erase(cand.begin() + best);
        used[n] = 1;
        perm.push_back(n);
        for (int t : {r.tri_p[n], r.tri_m[n]}) {
            left[t]--;
            if (in_tile[t] != tile) add_tri(t);
        }
        if (++cnt == ASM_TILE) {
            cnt = ntri = 0;
            sum[0] = sum[1] = sum[2] = 0.0;
            tile++;
            cand.clear();
        }
    }
    return perm;
}

int geom_upload(bem_ctx* ctx, bem_geom* g) {
    const HostMesh& m = g->mesh;
    mesh_bounds(g);
    const HostRWG& r = g->rwg;
    const Quad& q = g->quad;
    const int N = r.N, Nq = q.n, nt = m.nt();
    const size_t P = (size_t)2 * N * Nq;
    PosArrays A;
    position_arrays(g, A);
    auto& px = A.px; auto& py = A.py; auto& pz = A.pz; auto& fx = A.fx; auto& fy = A.fy; auto& fz = A.fz;
    auto& cx = A.cx; auto& cy = A.cy; auto& cz = A.cz; auto& jw = A.jw;
    auto& div = A.div; auto& coef = A.coef; auto& frx = A.frx; auto& fry = A.fry; auto& frz = A.frz;
    auto& tri = A.tri; auto& tv = A.tv; auto& tc = A.tc; auto& tu = A.tu; auto& tjw = A.tjw; auto& hpi = A.hpi;
    // singular pairs: halves per triangle, ordered (test, source) items per
    // unordered RWG pair
    // (half h N + n of each triangle in that order, triangle by triangle)
    std::vector<int> tfirst((size_t)nt + 1, 0), on_tri(2 * (size_t)N);
    for (int n = 0; n < N; n++) tfirst[r.tri_p[n] + 1]++, tfirst[r.tri_m[n] + 1]++;
    for (int t = 0; t < nt; t++) tfirst[t + 1] += tfirst[t];
    {
        std::vector<int> at(tfirst.begin(), tfirst.end() - 1);
        for (int n = 0; n < N; n++) on_tri[at[r.tri_p[n]]++] = n;
        for (int n = 0; n < N; n++) on_tri[at[r.tri_m[n]]++] = N + n;
    }
    // one entry per (triangle, test, source), sorted by (m <= n) and, for one
    // pair, in the order above: a bucket per m and an insertion sort by n in it
    struct Item {
        int n, t, a, b;
    };
    std::vector<int> mfirst((size_t)N + 1, 0);
    auto each = [&](auto&& f) {
        for (int t = 0; t < nt; t++)
            for (int i = tfirst[t]; i < tfirst[t + 1]; i++)
                for (int k = tfirst[t]; k < tfirst[t + 1]; k++) {
                    const int mm = on_tri[i] % N, nn = on_tri[k] % N;
                    f(std::min(mm, nn), Item{std::max(mm, nn), t, on_tri[i], on_tri[k]});
                }
    };
    each([&](int mm, const Item&) { mfirst[mm + 1]++; });
    for (int i = 0; i < N; i++) mfirst[i + 1] += mfirst[i];
    std::vector<Item> items(mfirst[N]);
    {
        std::vector<int> at(mfirst.begin(), mfirst.end() - 1);
        each([&](int mm, const Item& x) {
            int i = at[mm]++;
            for (; i > mfirst[mm] && items[i - 1].n > x.n; i--) items[i] = items[i - 1];
            items[i] = x;
        });
    }
    std::vector<int> pair_mn, item_ptr{0}, item;
    item.reserve(3 * items.size());
    for (int mm = 0; mm < N; mm++)
        for (int i = mfirst[mm]; i < mfirst[mm + 1]; i++) {
            if (i == mfirst[mm] || items[i].n != items[i - 1].n) {
                if (!pair_mn.empty()) item_ptr.push_back((int)item.size() / 3);
                pair_mn.push_back(mm);
                pair_mn.push_back(items[i].n);
            }
            item.insert(item.end(), {items[i].t, items[i].a, items[i].b});
        }
    if (!pair_mn.empty()) item_ptr.push_back((int)item.size() / 3);
    g->sing.npairs = (int)pair_mn.size() / 2;
    g->sing.nitems = (int)item.size() / 3;

    // triangles in the Morton order of their centroids, along which patch_order starts the tiles
    std::vector<int> torder(nt);
    {
        double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
        for (int t = 0; t < nt; t++)
            for (int j = 0; j < 3; j++) lo[j] = std::min(lo[j], tc[3 * t + j]), hi[j] = std::max(hi[j], tc[3 * t + j]);
        const double span = std::max(std::max(hi[0] - lo[0], hi[1] - lo[1]), std::max(hi[2] - lo[2], 1e-300));
        std::vector<uint64_t> key(nt);
        for (int t = 0; t < nt; t++) {
            uint64_t code = 0;
            uint64_t c3[3];
            for (int j = 0; j < 3; j++) {
                double f = (tc[3 * t + j] - lo[j]) / span;
                c3[j] = (uint64_t)std::min(2097151.0, std::max(0.0, f * 2097151.0));
            }
            for (int b = 20; b >= 0; b--)
                for (int j = 0; j < 3; j++) code = (code << 1) | ((c3[j] >> b) & 1u);
            key[t] = code;
        }
        for (int t = 0; t < nt; t++) torder[t] = t;
        std::stable_sort(torder.begin(), torder.end(), [&](int x, int y) { return key[x] < key[y]; });
    }
    std::vector<int> tri_half(3 * (size_t)nt, -1);
    for (int h = 0; h < 2; h++)
        for (int n = 0; n < N; n++) {
            const int t = h == 0 ? r.tri_p[n] : r.tri_m[n];
            int j = 0;
            while (j < 3 && tri_half[3 * (size_t)t + j] >= 0) j++;
            if (j == 3) return fail(ctx, BEM_ERR_INVALID, "triangle %d carries more than 3 RWG halves", t);
            tri_half[3 * (size_t)t + j] = h * N + n;
        }
    const int ntile = (N + ASM_TILE - 1) / ASM_TILE;
    const std::vector<int> perm = patch_order(r, nt, tc, torder);
    std::vector<int> pos(N);
    for (int i = 0; i < N; i++) pos[perm[i]] = i;
    std::vector<int> tile_rwg((size_t)ntile * ASM_TILE, -1), tile_tri((size_t)ntile * ASM_TRI_MAX, -1), tile_ntri(ntile, 0);
    std::vector<unsigned char> tile_ent((size_t)ntile * ASM_TRI_MAX * 3, 0xff);
    for (int tl = 0; tl < ntile; tl++) {
        int cnt = 0;
        for (int sl = 0; sl < ASM_TILE && tl * ASM_TILE + sl < N; sl++) {
            const int n = perm[tl * ASM_TILE + sl];
            tile_rwg[(size_t)tl * ASM_TILE + sl] = n;
            for (int h = 0; h < 2; h++) {
                const int t = h == 0 ? r.tri_p[n] : r.tri_m[n];
                int li = 0;
                while (li < cnt && tile_tri[(size_t)tl * ASM_TRI_MAX + li] != t) li++;
                if (li == cnt) tile_tri[(size_t)tl * ASM_TRI_MAX + cnt++] = t;
                unsigned char* e = &tile_ent[((size_t)tl * ASM_TRI_MAX + li) * 3];
                int j = 0;
                while (j < 3 && e[j] != 0xff) j++;
                if (j == 3) return fail(ctx, BEM_ERR_INVALID, "triangle %d carries more than 3 RWG halves", t);
                e[j] = (unsigned char)(sl * 2 + h);
            }
        }
        tile_ntri[tl] = cnt;
    }

    // one device allocation, 256-byte aligned sub-arrays
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += (bytes + 255) & ~(size_t)255;
        return o;
    };
    size_t o_pt[10];
    for (int i = 0; i < 10; i++) o_pt[i] = take(P * 8);
    size_t o_div = take(2 * N * 8), o_coef = take(2 * N * 8), o_fr = take(3 * 2 * N * 8);
    size_t o_tri = take(2 * N * 4);
    size_t o_pmn = take(pair_mn.size() * 4), o_iptr = take(item_ptr.size() * 4),
           o_item = take(item.size() * 4);
    size_t o_P = take((size_t)nt * Nq * 8), o_V = take((size_t)nt * Nq * 3 * 8),
           o_tv = take(tv.size() * 8);
    size_t o_tc = take(tc.size() * 8), o_tu = take(tu.size() * 8), o_tjw = take(tjw.size() * 8),
           o_hpi = take(hpi.size() * 8), o_trwg = take(tile_rwg.size() * 4), o_pos = take((size_t)N * 4),
           o_ttri = take(tile_tri.size() * 4), o_tntri = take((size_t)ntile * 4), o_tent = take(tile_ent.size()),
           o_tflag = take((size_t)ntile), o_rrec = take((size_t)N), o_thalf = take(tri_half.size() * 4);
    g->dmem = devmem_alloc(ctx->device, off, ctx);
    if (!g->dmem) return fail(ctx, BEM_ERR_OOM, "geometry arrays (%zu bytes)", off);
    g->dmem_bytes = off;
    char* base = (char*)g->dmem;
    // the arrays side by side on the host as on the device, in one copy
    std::vector<char> stage(off, 0);
    auto put = [&](void* dst, const void* src, size_t bytes) { std::memcpy(stage.data() + ((char*)dst - base), src, bytes); };
    double** pts[10] = {&g->half.px, &g->half.py, &g->half.pz, &g->half.fx, &g->half.fy,
                        &g->half.fz, &g->half.cx, &g->half.cy, &g->half.cz, &g->half.jw};
    std::vector<double>* src[10] = {&px, &py, &pz, &fx, &fy, &fz, &cx, &cy, &cz, &jw};
    for (int i = 0; i < 10; i++) {
        *pts[i] = (double*)(base + o_pt[i]);
        put(*pts[i], src[i]->data(), P * 8);
    }
    g->half.div = (double*)(base + o_div);
    g->half.tri = (int*)(base + o_tri);
    double* d_coef = (double*)(base + o_coef);
    double* d_fr = (double*)(base + o_fr);
    put(g->half.div, div.data(), 2 * N * 8);
    put(d_coef, coef.data(), 2 * N * 8);
    put(d_fr, frx.data(), 2 * N * 8);
    put(d_fr + 2 * N, fry.data(), 2 * N * 8);
    put(d_fr + 4 * N, frz.data(), 2 * N * 8);
    put(g->half.tri, tri.data(), 2 * N * 4);
    g->sing.pair_mn = (int*)(base + o_pmn);
    g->sing.item_ptr = (int*)(base + o_iptr);
    g->sing.item = (int*)(base + o_item);
    g->sing.P = (double*)(base + o_P);
    g->sing.V = (double*)(base + o_V);
    g->sing.tv = (double*)(base + o_tv);
    put(g->sing.pair_mn, pair_mn.data(), pair_mn.size() * 4);
    put(g->sing.item_ptr, item_ptr.data(), item_ptr.size() * 4);
    put(g->sing.item, item.data(), item.size() * 4);
    put(g->sing.tv, tv.data(), tv.size() * 8);
    DevTriAsm& ta = g->tri;
    ta.c = (double*)(base + o_tc);
    ta.u = (double*)(base + o_tu);
    ta.jw = (double*)(base + o_tjw);
    ta.pi = (double*)(base + o_hpi);
    ta.tile_rwg = (int*)(base + o_trwg);
    ta.pos = (int*)(base + o_pos);
    ta.tile_tri = (int*)(base + o_ttri);
    ta.tile_ntri = (int*)(base + o_tntri);
    ta.tile_ent = (unsigned char*)(base + o_tent);
    ta.tile_flag = (unsigned char*)(base + o_tflag);
    ta.rwg_rec = (unsigned char*)(base + o_rrec);
    ta.ntile = ntile;
    ta.tri_half = (int*)(base + o_thalf);
    put(ta.tri_half, tri_half.data(), tri_half.size() * 4);
    put(ta.c, tc.data(), tc.size() * 8);
    put(ta.u, tu.data(), tu.size() * 8);
    put(ta.jw, tjw.data(), tjw.size() * 8);
    put(ta.pi, hpi.data(), hpi.size() * 8);
    put(ta.tile_rwg, tile_rwg.data(), tile_rwg.size() * 4);
    put(ta.pos, pos.data(), (size_t)N * 4);
    put(ta.tile_tri, tile_tri.data(), tile_tri.size() * 4);
    put(ta.tile_ntri, tile_ntri.data(), (size_t)ntile * 4);
    put(ta.tile_ent, tile_ent.data(), tile_ent.size());
    BEM_TRY(h2d(ctx, base, stage.data(), off));
    // half coefficient and free vertex live right after div (see fixup kernel)
    (void)d_coef;
    (void)d_fr;
    g->sing_coef = d_coef;
    g->sing_free = d_fr;
    return BEM_OK;
}

int geom_set_vertices(bem_ctx* ctx, bem_geom* g, const double* verts) {
    HostRWG& r = g->rwg;
    HostMesh& m = g->mesh;
    if (!verts || r.edge_lo.size() != (size_t)r.N || r.vfree_p.size() != (size_t)r.N)
        return fail(ctx, BEM_ERR_INVALID, "vertex update needs a geometry built from its mesh");
    for (int i = 0; i < m.nv(); i++) m.verts[i] = {verts[3 * i], verts[3 * i + 1], verts[3 * i + 2]};
    rwg_refresh(m, r);
    mesh_bounds(g);
    PosArrays A;
    position_arrays(g, A);
    const int N = r.N;
    const size_t P = A.px.size();
    cudaStream_t st = ctx->stream;
    double* dst[10] = {g->half.px, g->half.py, g->half.pz, g->half.fx, g->half.fy,
                       g->half.fz, g->half.cx, g->half.cy, g->half.cz, g->half.jw};
    const std::vector<double>* src[10] = {&A.px, &A.py, &A.pz, &A.fx, &A.fy, &A.fz, &A.cx, &A.cy, &A.cz, &A.jw};
    for (int i = 0; i < 10; i++)
        BEM_TRY_CUDA(ctx, cudaMemcpyAsync(dst[i], src[i]->data(), P * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->half.div, A.div.data(), 2 * (size_t)N * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->sing_coef, A.coef.data(), 2 * (size_t)N * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->sing_free, A.frx.data(), 2 * (size_t)N * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->sing_free + 2 * N, A.fry.data(), 2 * (size_t)N * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->sing_free + 4 * N, A.frz.data(), 2 * (size_t)N * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->sing.tv, A.tv.data(), A.tv.size() * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->tri.c, A.tc.data(), A.tc.size() * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->tri.u, A.tu.data(), A.tu.size() * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->tri.jw, A.tjw.data(), A.tjw.size() * 8, cudaMemcpyHostToDevice, st));
    BEM_TRY_CUDA(ctx, cudaMemcpyAsync(g->tri.pi, A.hpi.data(), A.hpi.size() * 8, cudaMemcpyHostToDevice, st));
    return BEM_OK;
}

// One thread per (triangle, point): P and V = r P - grad W (central
// differences, eps = 1e-6) -- graglia.h:90-112.
__global__ void graglia_kernel(const double* __restrict__ tv, int nt, TriQ q,
                               double* __restrict__ P, double* __restrict__ V) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nt * q.n) return;
    int t = i / q.n, k = i % q.n;
    double v[9];
    for (int j = 0; j < 9; j++) v[j] = tv[9 * t + j];
    graglia_point(v, q.l1[k], q.l2[k], q, &P[i], &V[3 * i]);
}

// ------------------------------------------------------------ main assembly
constexpr int TILE = 16;
static_assert(TILE == ASM_TILE, "assembly band width");
constexpr int MAXQ = 13;

struct AsmArgs {
    DevHalf h;
    int N, Nq;
    int ntile;       // tiles per side
    Medium med[2];   // ext, int (only med[0] when nmed == 1)
    double eta_e, eta_i;
    unsigned flags;
    // outputs
    double2* Z;      // row-major 2N x 2N: PMCHWT (nmed == 2) or A_ext (nmed == 1)
    int64_t ldz;
    double2* L;      // row-major N x N (nmed == 1, Z null)
    double2* K;
    int64_t ld;
    // optional: only tile pairs with a flagged row or column tile are computed
    const unsigned char* tile_flag;
    const double* coef;  // (2N) sign*l/(2A) per half (triangle-pair kernel)
};

template <int NMED>
__global__ void __launch_bounds__(256) assemble_kernel(AsmArgs a) {
    // upper-triangular tile index -> (tile row bi, tile col bj), bi <= bj
    int64_t lin = blockIdx.x;
    int T = a.ntile;
    // row bi starts at offset bi*T - bi*(bi-1)/2
    int bi = (int)floor((2.0 * T + 1.0 - sqrt((2.0 * T + 1.0) * (2.0 * T + 1.0) - 8.0 * (double)lin)) * 0.5);
    if (bi < 0) bi = 0;
    while (bi > 0 && (int64_t)bi * T - (int64_t)bi * (bi - 1) / 2 > lin) bi--;
    while ((int64_t)(bi + 1) * T - (int64_t)(bi + 1) * bi / 2 <= lin) bi++;
    int bj = bi + (int)(lin - ((int64_t)bi * T - (int64_t)bi * (bi - 1) / 2));

    const int N = a.N, Nq = a.Nq;
    const int tx = threadIdx.x % TILE, ty = threadIdx.x / TILE;
    if (a.tile_flag && !a.tile_flag[bi] && !a.tile_flag[bj]) return;  // a tile the caller keeps
    const int m0 = bi * TILE, n0 = bj * TILE;

    // source data of the tile's columns: [half][q][col]
    __shared__ double s_px[2][MAXQ][TILE], s_py[2][MAXQ][TILE], s_pz[2][MAXQ][TILE];
    __shared__ double s_fx[2][MAXQ][TILE], s_fy[2][MAXQ][TILE], s_fz[2][MAXQ][TILE];
    __shared__ double s_cx[2][MAXQ][TILE], s_cy[2][MAXQ][TILE], s_cz[2][MAXQ][TILE];
    __shared__ double s_jw[2][MAXQ][TILE];
    __shared__ double s_div[2][TILE];
    __shared__ int s_tri[2][TILE];
    for (int i = threadIdx.x; i < 2 * Nq * TILE; i += blockDim.x) {
        int col = i % TILE, q = (i / TILE) % Nq, h = i / (TILE * Nq);
        int n = min(n0 + col, N - 1);
        size_t p = ((size_t)(h * N + n)) * Nq + q;
        s_px[h][q][col] = a.h.px[p];
        s_py[h][q][col] = a.h.py[p];
        s_pz[h][q][col] = a.h.pz[p];
        s_fx[h][q][col] = a.h.fx[p];
        s_fy[h][q][col] = a.h.fy[p];
        s_fz[h][q][col] = a.h.fz[p];
        s_cx[h][q][col] = a.h.cx[p];
        s_cy[h][q][col] = a.h.cy[p];
        s_cz[h][q][col] = a.h.cz[p];
        s_jw[h][q][col] = a.h.jw[p];
    }
    if (threadIdx.x < 2 * TILE) {
        int h = threadIdx.x / TILE, col = threadIdx.x % TILE;
        int n = min(n0 + col, N - 1);
        s_div[h][col] = a.h.div[h * N + n];
        s_tri[h][col] = a.h.tri[h * N + n];
    }
    __syncthreads();

    const int m = min(m0 + ty, N - 1);
    const bool exact = (a.flags & BEM_ASM_GSMOOTH_EXACT) != 0;
    cplx Lv[NMED], Ls[NMED], Kk[NMED];
    for (int e = 0; e < NMED; e++) Lv[e] = Ls[e] = Kk[e] = {0.0, 0.0};

    for (int th = 0; th < 2; th++) {
        const int thn = th * N + m;
        const int ttri = a.h.tri[thn];
        const double tdiv = a.h.div[thn];
        for (int sh = 0; sh < 2; sh++) {
            const bool sing = (ttri == s_tri[sh][tx]);
            const double dd = tdiv * s_div[sh][tx];
            cplx Lsb[NMED];
            for (int e = 0; e < NMED; e++) Lsb[e] = {0.0, 0.0};
            for (int q = 0; q < Nq; q++) {
                size_t tp = (size_t)thn * Nq + q;
                const double tpx = a.h.px[tp], tpy = a.h.py[tp], tpz = a.h.pz[tp];
                const double tfx = a.h.fx[tp], tfy = a.h.fy[tp], tfz = a.h.fz[tp];
                const double tcx = a.h.cx[tp], tcy = a.h.cy[tp], tcz = a.h.cz[tp];
                const double tjw = a.h.jw[tp];
                for (int qs = 0; qs < Nq; qs++) {
                    double dx = tpx - s_px[sh][qs][tx];
                    double dy = tpy - s_py[sh][qs][tx];
                    double dz = tpz - s_pz[sh][qs][tx];
                    double R = sqrt(dx * dx + dy * dy + dz * dz);
                    double Rs = fmax(R, 1e-15);
                    double invR = 1.0 / Rs;
                    // rounded on its own: the literal G_smooth subtracts it
                    // from G, and a multiply-add fused across the two would
                    // leave its rounding error (~0.01 at R_s = 1e-15)
                    double i4R = __dmul_rn(INV4PI_D, invR);
                    double jwp = tjw * s_jw[sh][qs][tx];
                    double fdot = tfx * s_fx[sh][qs][tx] + tfy * s_fy[sh][qs][tx] + tfz * s_fz[sh][qs][tx];
                    // f_t . ((r_t - r_s) x f_s) = (f_t x r_t).f_s + f_t.(f_s x r_s)
                    double trip = (tcx * s_fx[sh][qs][tx] + tcy * s_fy[sh][qs][tx] + tcz * s_fz[sh][qs][tx]) +
                                  (tfx * s_cx[sh][qs][tx] + tfy * s_cy[sh][qs][tx] + tfz * s_cz[sh][qs][tx]);
                    bool kval = !sing && R > 1e-12;
#pragma unroll
                    for (int e = 0; e < NMED; e++) {
                        const Medium k = a.med[e];
                        double s, c;
                        sincos(k.kr * Rs, &s, &c);
                        double ea = (k.ki != 0.0) ? exp_decay(k.ki * Rs) : 1.0;
                        cplx G = {ea * c * i4R, ea * s * i4R};
                        cplx Gu = G;
                        if (sing) {
                            if (exact) Gu = g_smooth_exact(k, R);
                            else Gu.re -= i4R;
                        }
                        cplx Gj = {Gu.re * jwp, Gu.im * jwp};
                        Lv[e].re += fdot * Gj.re;
                        Lv[e].im += fdot * Gj.im;
                        Lsb[e].re += Gj.re;
                        Lsb[e].im += Gj.im;
                        if (kval) {
                            // grad G coefficient (ik - 1/R)/R
                            cplx gc = cmul(G, cplx{(-k.ki - invR) * invR, k.kr * invR});
                            double w = jwp * trip;
                            Kk[e].re += gc.re * w;
                            Kk[e].im += gc.im * w;
                        }
                    }
                }
            }
            for (int e = 0; e < NMED; e++) {
                Ls[e].re += dd * Lsb[e].re;
                Ls[e].im += dd * Lsb[e].im;
            }
        }
    }
    const int n = n0 + tx;
    const int mm = m0 + ty;
    if (mm >= N || n >= N) return;
    // L = ik Lvec - (i/k) sum(div div Lscl)
    cplx Lf[NMED];
    for (int e = 0; e < NMED; e++) {
        Medium k = a.med[e];
        cplx ik = {-k.ki, k.kr};
        double k2 = k.kr * k.kr + k.ki * k.ki;
        cplx iok = {k.ki / k2, k.kr / k2};  // i/k
        cplx t1 = cmul(ik, Lv[e]), t2 = cmul(iok, Ls[e]);
        Lf[e] = {t1.re - t2.re, t1.im - t2.im};
    }
    // L and K are symmetric: in a diagonal tile only the thread of the upper
    // entry writes, to both positions, so the stored blocks are exactly
    // symmetric (as after the reference's (X + X^T)/2, assembly.cu:494-502)
    if (bi == bj && n < mm) return;
    const bool mirror = (n != mm);
    if (a.Z) {
        // PMCHWT blocks; with one medium the exterior-only A_ext
        // [[eta_e L_e, -K_e], [K_e, L_e / eta_e]] (bem_core.py:1071-1090)
        cplx TL, BR, Ks;
        if constexpr (NMED == 2) {
            TL = {a.eta_e * Lf[0].re + a.eta_i * Lf[1].re, a.eta_e * Lf[0].im + a.eta_i * Lf[1].im};
            BR = {Lf[0].re / a.eta_e + Lf[1].re / a.eta_i, Lf[0].im / a.eta_e + Lf[1].im / a.eta_i};
            Ks = {Kk[0].re + Kk[1].re, Kk[0].im + Kk[1].im};
        } else {
            TL = {a.eta_e * Lf[0].re, a.eta_e * Lf[0].im};
            BR = {Lf[0].re / a.eta_e, Lf[0].im / a.eta_e};
            Ks = Kk[0];
        }
        double2* Z = a.Z;
        int64_t ld = a.ldz;
        Z[(int64_t)mm * ld + n] = make_double2(TL.re, TL.im);
        Z[(int64_t)mm * ld + N + n] = make_double2(-Ks.re, -Ks.im);
        Z[(int64_t)(N + mm) * ld + n] = make_double2(Ks.re, Ks.im);
        Z[(int64_t)(N + mm) * ld + N + n] = make_double2(BR.re, BR.im);
        if (mirror) {
            Z[(int64_t)n * ld + mm] = make_double2(TL.re, TL.im);
            Z[(int64_t)n * ld + N + mm] = make_double2(-Ks.re, -Ks.im);
            Z[(int64_t)(N + n) * ld + mm] = make_double2(Ks.re, Ks.im);
            Z[(int64_t)(N + n) * ld + N + mm] = make_double2(BR.re, BR.im);
        }
    } else {
        a.L[(int64_t)mm * a.ld + n] = make_double2(Lf[0].re, Lf[0].im);
        a.K[(int64_t)mm * a.ld + n] = make_double2(Kk[0].re, Kk[0].im);
        if (mirror) {
            a.L[(int64_t)n * a.ld + mm] = make_double2(Lf[0].re, Lf[0].im);
            a.K[(int64_t)n * a.ld + mm] = make_double2(Kk[0].re, Kk[0].im);
        }
    }
}


// ------------------------------------------------- triangle-pair assembly
// The same quadrature sums as assemble_kernel, organised by triangle pairs:
// every RWG half on triangle a paired with every half on triangle b uses the
// same 7 x 7 Green's function values, so each (a, b) of a tile pair computes
// them once and keeps moments in coordinates relative to the centroids
// (u = r - c_a, v = r' - c_b, D = c_a - c_b, d = r - r' = D + u - v):
//   L: M0 = sum G, Mu = sum G u, Mv = sum G v, Muv = sum G u.v
//   K: S0 = sum g, A = sum g u, B = sum g v, C = sum g u x v, from which
//      (D being constant over the pair) P1 = sum g u.(D x v) = -D.C,
//      Q2 = sum g (u x D - u x v) = A x D - C, Q3 = sum g (D x v + u x v)
//      = D x B + C and Q4 = sum g d = D S0 + A - B
// (G, g with the weights jw jw').  With f_m = s_m (r - p_m) = s_m (u - pi_m),
// f_n = s_n (v - nu_n):
//   sum G f_m.f_n  = s_m s_n (Muv - pi.Mv - nu.Mu + pi.nu M0)
//   sum g f_m.(d x f_n) = s_m s_n (P1 - nu.Q2 - pi.Q3 + pi.(Q4 x nu))
// The quadrature sum over the points of b is formed first, sum_q G w_q (1, v)
// and sum_q g w_q (1, v): four complex sums per point of a and kernel, from
// which the moments take u once per point of a instead of once per pair of
// points (16 multiply-adds per point pair and medium fewer).  One thread does
// both media of a triangle pair: they share the distance and the K moments
// (only K_e + K_i is needed).
// Each (RWG pair, half pair) term lands in its own shared-memory slot and the
// four half pairs of an entry are summed in a fixed order, so the result does
// not depend on the tiling.  RWGs are tiled in patches grown over shared
// triangles (geom_upload), ~15.5 distinct triangles per 16 RWGs.
//
// Bound by the FP64 pipe, ~100 operations per point pair for two lossless
// media, ~120 with one absorbing, which is 58 % busy: the 52 accumulators of a
// thread leave room for two blocks of four warps an SM.  2N = 18432, one
// medium absorbing: 29.3 ms, 64.3 ms before (moments per point pair and medium,
// 17.1 triangles a tile).  Measured against it, at 28.6 ms with a sine of three
// operations less: three blocks of 128 at 168 registers 31.2 ms, 96 threads
// 37.9 ms, 160 threads 36.8 ms, the inner loop unrolled 7 times 29.3 ms, not at
// all 32.0 ms.  A tile pair's ~240 triangle
// pairs are two rounds of 128 threads.
constexpr int ASM_THREADS = 128;
// points of a triangle in shared memory: Nq x (u, weight), padded to an odd
// number of 16-byte units so that the triangles of neighbouring lanes do not conflict
__host__ __device__ constexpr int asm_pt_pitch(int Nq) { return 4 * Nq + 2; }
constexpr size_t tri_smem_bytes(int Nq) {
    return (size_t)256 * 4 * 3 * sizeof(double2) +
           sizeof(double) * (2 * ASM_TRI_MAX * asm_pt_pitch(Nq) + 2 * ASM_TRI_MAX * 3 + 2 * TILE * 2 * 5) +
           sizeof(int) * (2 * ASM_TRI_MAX + 2) + 2 * ASM_TRI_MAX * 3;
}

__device__ __forceinline__ void cfma(cplx& a, cplx b, double s) { a.re += b.re * s, a.im += b.im * s; }

// One medium's or the media's combined outputs of the half pairs of a
// triangle pair, from the moments.  LM: L moments per medium (M0, Muv, Mu,
// Mv); KM: K moments (S0, A, B, C); null LM[e].k: no K (the same triangle).
struct LMoments {
    cplx M0, Muv, Mu[3], Mv[3];
};
struct KMoments {
    cplx S0, A[3], B[3], C[3];
};

// term(x, y) of the half pairs into their slots: (TL, BR, K) for Z, (L, K) for one operator.
template <int NMED>
__device__ __forceinline__ void store_half_pairs(const AsmArgs& a, const LMoments* L, const KMoments& K, double Dx,
                                                 double Dy, double Dz, const unsigned char* ea,
                                                 const unsigned char* eb, const double* ssig, const double* sdiv,
                                                 const double* spi, double2* slots) {
    // scalar part: sum_e c_e (i / k_e) M0_e; vector part's factor c_e i k_e; c_e = eta_e (TL), 1 / eta_e (BR)
    cplx s1 = {0, 0}, s2 = {0, 0}, v1[NMED], v2[NMED];
#pragma unroll
    for (int e = 0; e < NMED; e++) {
        const Medium k = a.med[e];
        const double c1 = a.Z ? (e ? a.eta_i : a.eta_e) : 1.0, c2 = 1.0 / c1, k2 = k.kr * k.kr + k.ki * k.ki;
        const cplx t = cmul(cplx{k.ki / k2, k.kr / k2}, L[e].M0);
        cfma(s1, t, c1), cfma(s2, t, c2);
        v1[e] = {-k.ki * c1, k.kr * c1}, v2[e] = {-k.ki * c2, k.kr * c2};
    }
    // P1 = -D.C, Q2 = A x D - C, Q3 = D x B + C, Q4 = D S0 + A - B
    const double DD[3] = {Dx, Dy, Dz};
    cplx P1 = {0, 0}, Q2[3], Q3[3], Q4[3];
#pragma unroll
    for (int j = 0; j < 3; j++) {
        const int j1 = (j + 1) % 3, j2 = (j + 2) % 3;
        cfma(P1, K.C[j], -DD[j]);
        Q2[j] = {K.A[j1].re * DD[j2] - K.A[j2].re * DD[j1] - K.C[j].re,
                 K.A[j1].im * DD[j2] - K.A[j2].im * DD[j1] - K.C[j].im};
        Q3[j] = {DD[j1] * K.B[j2].re - DD[j2] * K.B[j1].re + K.C[j].re,
                 DD[j1] * K.B[j2].im - DD[j2] * K.B[j1].im + K.C[j].im};
        Q4[j] = {DD[j] * K.S0.re + K.A[j].re - K.B[j].re, DD[j] * K.S0.im + K.A[j].im - K.B[j].im};
    }
    for (int x = 0; x < 3; x++) {
        const int er = ea[x];
        if (er == 0xff) break;
        const int r = er >> 1;
        const double sr = ssig[er], dr = sdiv[er];
        const double p[3] = {spi[er * 3], spi[er * 3 + 1], spi[er * 3 + 2]};
        // over the test half: Muv - p.Mv, Mu - p M0; P1 - p.Q3, Q2 - p x Q4
        cplx qx[NMED], ux[NMED][3], kx = P1, wx[3];
#pragma unroll
        for (int e = 0; e < NMED; e++) {
            qx[e] = L[e].Muv;
#pragma unroll
            for (int j = 0; j < 3; j++) {
                cfma(qx[e], L[e].Mv[j], -p[j]);
                ux[e][j] = L[e].Mu[j];
                cfma(ux[e][j], L[e].M0, -p[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 3; j++) {
            const int j1 = (j + 1) % 3, j2 = (j + 2) % 3;
            cfma(kx, Q3[j], -p[j]);
            wx[j] = {Q2[j].re - (p[j1] * Q4[j2].re - p[j2] * Q4[j1].re),
                     Q2[j].im - (p[j1] * Q4[j2].im - p[j2] * Q4[j1].im)};
        }
        for (int y = 0; y < 3; y++) {
            const int ec = eb[y];
            if (ec == 0xff) break;
            const int c = ec >> 1;
            const double ss = sr * ssig[2 * TILE + ec], dd = dr * sdiv[2 * TILE + ec];
            const double* nu = spi + (2 * TILE + ec) * 3;
            cplx o1 = {0, 0}, o2 = {0, 0}, kv = kx;
#pragma unroll
            for (int e = 0; e < NMED; e++) {
                cplx lv = qx[e];
#pragma unroll
                for (int j = 0; j < 3; j++) cfma(lv, ux[e][j], -nu[j]);
                const cplx t1 = cmul(v1[e], lv), t2 = cmul(v2[e], lv);
                o1.re += t1.re, o1.im += t1.im, o2.re += t2.re, o2.im += t2.im;
            }
#pragma unroll
            for (int j = 0; j < 3; j++) cfma(kv, wx[j], -nu[j]);
            double2* out = slots + ((r * TILE + c) * 4 + (er & 1) * 2 + (ec & 1)) * 3;
            out[0] = make_double2(ss * o1.re - dd * s1.re, ss * o1.im - dd * s1.im);
            out[1] = make_double2(ss * o2.re - dd * s2.re, ss * o2.im - dd * s2.im);
            out[2] = make_double2(ss * kv.re, ss * kv.im);
        }
    }
}

// DAMP: bit e set when medium e absorbs (k_im != 0).  NQ: points of the rule (0: a.Nq).
template <int NMED, int DAMP, int NQ>
__global__ void __launch_bounds__(ASM_THREADS, 2) assemble_tri_kernel(AsmArgs a, DevTriAsm ta) {
    int64_t lin = blockIdx.x;
    const int T = a.ntile;
    int bi = (int)floor((2.0 * T + 1.0 - sqrt((2.0 * T + 1.0) * (2.0 * T + 1.0) - 8.0 * (double)lin)) * 0.5);
    if (bi < 0) bi = 0;
    while (bi > 0 && (int64_t)bi * T - (int64_t)bi * (bi - 1) / 2 > lin) bi--;
    while ((int64_t)(bi + 1) * T - (int64_t)(bi + 1) * bi / 2 <= lin) bi++;
    const int bj = bi + (int)(lin - ((int64_t)bi * T - (int64_t)bi * (bi - 1) / 2));
    if (a.tile_flag && !a.tile_flag[bi] && !a.tile_flag[bj]) return;  // a tile the caller keeps
    const int N = a.N, Nq = NQ > 0 ? NQ : a.Nq, tid = threadIdx.x, pitch = asm_pt_pitch(Nq);

    extern __shared__ __align__(16) unsigned char tri_smem[];
    double2* slots = reinterpret_cast<double2*>(tri_smem);         // [256 entries][4 half pairs][3]
    double* spt = reinterpret_cast<double*>(slots + 256 * 4 * 3);  // [2][TRI_MAX][pitch]: u, weight per point
    double* sc = spt + 2 * ASM_TRI_MAX * pitch;                    // [2][TRI_MAX][3]
    double* ssig = sc + 2 * ASM_TRI_MAX * 3;                       // [2][TILE][2]
    double* sdiv = ssig + 2 * TILE * 2;                            // [2][TILE][2]
    double* spi = sdiv + 2 * TILE * 2;                             // [2][TILE][2][3]
    int* stri = reinterpret_cast<int*>(spi + 2 * TILE * 2 * 3);    // [2][TRI_MAX]
    unsigned char* sent = reinterpret_cast<unsigned char*>(stri + 2 * ASM_TRI_MAX);  // [2][TRI_MAX][3]

    const int na = ta.tile_ntri[bi], nb = ta.tile_ntri[bj];
    for (int i = tid; i < na + nb; i += ASM_THREADS) {
        const int sl = i < na ? i : ASM_TRI_MAX + i - na;
        const int t = ta.tile_tri[(size_t)(i < na ? bi : bj) * ASM_TRI_MAX + sl % ASM_TRI_MAX];
        stri[sl] = t;
        for (int j = 0; j < 3; j++) sc[sl * 3 + j] = ta.c[(size_t)t * 3 + j];
    }
    for (int i = tid; i < (na + nb) * Nq; i += ASM_THREADS) {
        const int q = i % Nq, l = i / Nq, sl = l < na ? l : ASM_TRI_MAX + l - na;
        const int t = ta.tile_tri[(size_t)(l < na ? bi : bj) * ASM_TRI_MAX + sl % ASM_TRI_MAX];
        const size_t src = (size_t)t * Nq + q;
        double* d = spt + sl * pitch + 4 * q;
        for (int j = 0; j < 3; j++) d[j] = ta.u[src * 3 + j];
        d[3] = ta.jw[src];
    }
    for (int i = tid; i < 2 * ASM_TRI_MAX * 3; i += ASM_THREADS)
        sent[i] = ta.tile_ent[(size_t)(i >= ASM_TRI_MAX * 3 ? bj : bi) * ASM_TRI_MAX * 3 + i % (ASM_TRI_MAX * 3)];
    for (int i = tid; i < 2 * TILE * 2; i += ASM_THREADS) {
        const int side = i / (TILE * 2), slot = (i / 2) % TILE, h = i % 2;
        const int n = ta.tile_rwg[(size_t)(side ? bj : bi) * TILE + slot];
        const int hn = h * N + (n >= 0 ? n : 0);
        ssig[i] = n >= 0 ? a.coef[hn] : 0.0;
        sdiv[i] = n >= 0 ? a.h.div[hn] : 0.0;
        for (int j = 0; j < 3; j++) spi[i * 3 + j] = n >= 0 ? ta.pi[(size_t)hn * 3 + j] : 0.0;
    }
    __syncthreads();

    for (int it = tid; it < na * nb; it += ASM_THREADS) {
        const int ia = it / nb, ib = ASM_TRI_MAX + it - ia * nb;
        if (stri[ia] == stri[ib]) continue;  // the same triangle: below
        const double Dx = sc[ia * 3] - sc[ib * 3], Dy = sc[ia * 3 + 1] - sc[ib * 3 + 1],
                     Dz = sc[ia * 3 + 2] - sc[ib * 3 + 2];
        LMoments L[NMED];
        KMoments K;
#pragma unroll
        for (int e = 0; e < NMED; e++) {
            L[e].M0 = L[e].Muv = {0, 0};
#pragma unroll
            for (int j = 0; j < 3; j++) L[e].Mu[j] = L[e].Mv[j] = {0, 0};
        }
        K.S0 = {0, 0};
#pragma unroll
        for (int j = 0; j < 3; j++) K.A[j] = K.B[j] = K.C[j] = {0, 0};
#pragma unroll 1
        for (int qa = 0; qa < Nq; qa++) {
            const double2 uxy = *(const double2*)(spt + ia * pitch + 4 * qa),
                          uzw = *(const double2*)(spt + ia * pitch + 4 * qa + 2);
            const double ex = Dx + uxy.x, ey = Dy + uxy.y, ez = Dz + uzw.x, wa = uzw.y * INV4PI_D;
            cplx T0[NMED], Tv[NMED][3], s0 = {0, 0}, sv[3];
#pragma unroll
            for (int j = 0; j < 3; j++) sv[j] = {0, 0};
#pragma unroll
            for (int e = 0; e < NMED; e++) {
                T0[e] = {0, 0};
#pragma unroll
                for (int j = 0; j < 3; j++) Tv[e][j] = {0, 0};
            }
#pragma unroll 2
            for (int qb = 0; qb < Nq; qb++) {
                const double2 vxy = *(const double2*)(spt + ib * pitch + 4 * qb),
                              vzw = *(const double2*)(spt + ib * pitch + 4 * qb + 2);
                const double dx = ex - vxy.x, dy = ey - vxy.y, dz = ez - vzw.x;
                const double R2 = fmax(dx * dx + dy * dy + dz * dz, 1e-30);  // R clamped at 1e-15
                const double invR = rsqrt_normal(R2), R = R2 * invR, iw = invR * vzw.y;
                cplx g = {0, 0};  // sum_e G_e (i k_e - 1/R)
#pragma unroll
                for (int e = 0; e < NMED; e++) {
                    const Medium k = a.med[e];
                    double sn, cs;
                    sincos_bounded(k.kr * R, &sn, &cs);
                    double am = iw;
                    if ((DAMP >> e) & 1) am *= exp_decay_bounded(k.ki * R);
                    const cplx G = {am * cs, am * sn};
                    T0[e].re += G.re, T0[e].im += G.im;
                    cfma(Tv[e][0], G, vxy.x), cfma(Tv[e][1], G, vxy.y), cfma(Tv[e][2], G, vzw.x);
                    const double f = ((DAMP >> e) & 1) ? -k.ki - invR : -invR;
                    g.re += G.re * f - G.im * k.kr;
                    g.im += G.im * f + G.re * k.kr;
                }
                const double gr = R2 > 1e-24 ? invR : 0.0;  // coincident points of distinct triangles: no K
                g.re *= gr, g.im *= gr;
                s0.re += g.re, s0.im += g.im;
                cfma(sv[0], g, vxy.x), cfma(sv[1], g, vxy.y), cfma(sv[2], g, vzw.x);
            }
            const double wu[3] = {wa * uxy.x, wa * uxy.y, wa * uzw.x};
#pragma unroll
            for (int e = 0; e < NMED; e++) {
                cfma(L[e].M0, T0[e], wa);
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    cfma(L[e].Mu[j], T0[e], wu[j]);
                    cfma(L[e].Mv[j], Tv[e][j], wa);
                    cfma(L[e].Muv, Tv[e][j], wu[j]);
                }
            }
            cfma(K.S0, s0, wa);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                const int j1 = (j + 1) % 3, j2 = (j + 2) % 3;
                cfma(K.A[j], s0, wu[j]);
                cfma(K.B[j], sv[j], wa);
                K.C[j].re += wu[j1] * sv[j2].re - wu[j2] * sv[j1].re;
                K.C[j].im += wu[j1] * sv[j2].im - wu[j2] * sv[j1].im;
            }
        }
        store_half_pairs<NMED>(a, L, K, Dx, Dy, Dz, sent + ia * 3, sent + ib * 3, ssig, sdiv, spi, slots);
    }
    // the same triangle on both sides: G_smooth in the literal or the exact
    // form with the library's functions, no K (few per tile pair: thread per
    // row triangle)
    const bool exact = (a.flags & BEM_ASM_GSMOOTH_EXACT) != 0;
    for (int ia = tid; ia < na; ia += ASM_THREADS) {
        int ib = -1;
        for (int l = 0; l < nb; l++)
            if (stri[ASM_TRI_MAX + l] == stri[ia]) ib = ASM_TRI_MAX + l;
        if (ib < 0) continue;
        LMoments L[NMED];
        KMoments K;
        K.S0 = {0, 0};
        for (int j = 0; j < 3; j++) K.A[j] = K.B[j] = K.C[j] = {0, 0};
#pragma unroll 1
        for (int e = 0; e < NMED; e++) {
            const Medium k = a.med[e];
            LMoments S;
            S.M0 = S.Muv = {0, 0};
            for (int j = 0; j < 3; j++) S.Mu[j] = S.Mv[j] = {0, 0};
#pragma unroll 1
            for (int p = 0; p < Nq * Nq; p++) {
                const double* u = spt + ia * pitch + 4 * (p / Nq);
                const double* v = spt + ib * pitch + 4 * (p % Nq);
                const double w = u[3] * v[3];
                const double dx = u[0] - v[0], dy = u[1] - v[1], dz = u[2] - v[2];
                const double R2 = fmax(dx * dx + dy * dy + dz * dz, 1e-30);
                const double invR = rsqrt(R2), Rs = R2 * invR;
                const double i4R = __dmul_rn(INV4PI_D, invR);  // rounded alone, as in assemble_kernel
                double sn, cs;
                sincos(k.kr * Rs, &sn, &cs);
                const double eav = (k.ki != 0.0) ? exp_decay(k.ki * Rs) : 1.0;
                cplx G = {eav * cs * i4R, eav * sn * i4R};
                if (exact) G = g_smooth_exact(k, Rs);
                else G.re -= i4R;
                G.re *= w, G.im *= w;
                S.M0.re += G.re, S.M0.im += G.im;
                cfma(S.Muv, G, u[0] * v[0] + u[1] * v[1] + u[2] * v[2]);
                for (int j = 0; j < 3; j++) cfma(S.Mu[j], G, u[j]), cfma(S.Mv[j], G, v[j]);
            }
#pragma unroll
            for (int e2 = 0; e2 < NMED; e2++)
                if (e2 == e) L[e2] = S;
        }
        store_half_pairs<NMED>(a, L, K, 0.0, 0.0, 0.0, sent + ia * 3, sent + ib * 3, ssig, sdiv, spi, slots);
    }
    __syncthreads();

    for (int en = tid; en < TILE * TILE; en += ASM_THREADS) {
        const int r = en / TILE, c = en % TILE;
        const int mm = ta.tile_rwg[(size_t)bi * TILE + r], n = ta.tile_rwg[(size_t)bj * TILE + c];
        if (mm < 0 || n < 0) continue;
        if (bi == bj && c < r) continue;  // diagonal tile pair: the upper entry writes both positions
        double2 o[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double2* sl = slots + en * 12 + k;
            o[k] = make_double2(((sl[0].x + sl[3].x) + sl[6].x) + sl[9].x, ((sl[0].y + sl[3].y) + sl[6].y) + sl[9].y);
        }
        const bool mirror = (n != mm);
        if (a.Z) {
            const double2 TL = o[0], BR = o[1], Ks = o[2], Km = make_double2(-o[2].x, -o[2].y);
            double2* Z = a.Z;
            const int64_t ld = a.ldz;
            Z[(int64_t)mm * ld + n] = TL;
            Z[(int64_t)mm * ld + N + n] = Km;
            Z[(int64_t)(N + mm) * ld + n] = Ks;
            Z[(int64_t)(N + mm) * ld + N + n] = BR;
            if (mirror) {
                Z[(int64_t)n * ld + mm] = TL;
                Z[(int64_t)n * ld + N + mm] = Km;
                Z[(int64_t)(N + n) * ld + mm] = Ks;
                Z[(int64_t)(N + n) * ld + N + mm] = BR;
            }
        } else {
            a.L[(int64_t)mm * a.ld + n] = o[0];
            a.K[(int64_t)mm * a.ld + n] = o[2];
            if (mirror) {
                a.L[(int64_t)n * a.ld + mm] = o[0];
                a.K[(int64_t)n * a.ld + mm] = o[2];
            }
        }
    }
}

template <int NMED, int DAMP>
static int launch_assemble_tri(bem_ctx* ctx, const bem_geom* g, const AsmArgs& a, unsigned ntiles) {
    auto kern = g->Nq == 7   ? assemble_tri_kernel<NMED, DAMP, 7>
                : g->Nq == 4 ? assemble_tri_kernel<NMED, DAMP, 4>
                             : assemble_tri_kernel<NMED, DAMP, 0>;
    const size_t smem = tri_smem_bytes(g->Nq);
    BEM_TRY_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<ntiles, ASM_THREADS, smem, ctx->stream>>>(a, g->tri);
    return BEM_OK;
}

// Tiles to recompute from an RWG mask (tile_rwg null: tiles of 16
// consecutive RWGs), and per RWG whether its tile is recomputed.
__global__ void mask_tiles_kernel(const unsigned char* __restrict__ mask, const int* __restrict__ tile_rwg, int N,
                                  int ntile, unsigned char* __restrict__ flag) {
    const int tl = blockIdx.x * blockDim.x + threadIdx.x;
    if (tl >= ntile) return;
    unsigned char f = 0;
    for (int sl = 0; sl < TILE; sl++) {
        const int n = tile_rwg ? tile_rwg[(size_t)tl * TILE + sl] : tl * TILE + sl;
        if (n >= 0 && n < N && mask[n]) f = 1;
    }
    flag[tl] = f;
}

__global__ void mask_rec_kernel(const unsigned char* __restrict__ flag, const int* __restrict__ pos, int N,
                                unsigned char* __restrict__ rec) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= N) return;
    rec[n] = flag[(pos ? pos[n] : n) / TILE];
}

// ------------------------------------------------------------ singular fixup
struct FixArgs {
    DevHalf h;
    DevSingular s;
    const double* coef;  // (2N) sign*l/(2A)
    const double* fr;    // (3*2N) free vertex: x block, y block, z block
    int N, Nq, nmed;
    Medium med[2];
    double eta_e, eta_i;
    double2* Z;
    int64_t ldz;
    double2* L;
    int64_t ld;
    const unsigned char* rec;   // optional: RWGs whose assembly tiles were recomputed
};

// One thread per unordered RWG pair {m, n} sharing a triangle.  For every
// (triangle t, test half a, source half b) item:
//   A = div_a div_b sum_q P_q jw_a,q / (4 pi)
//   B = sum_q f_a,q . coef_b (V_q - r_free,b P_q) jw_a,q / (4 pi)
// and S = -(i/k) A + i k B (assembly.cu:290-317).  The symmetrised
// correction (S[m,n] + S[n,m])/2 is added to both L entries.
__global__ void singular_fixup_kernel(FixArgs a) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.s.npairs) return;
    const int N = a.N, Nq = a.Nq;
    int m = a.s.pair_mn[2 * p], n = a.s.pair_mn[2 * p + 1];
    if (a.rec && !a.rec[m] && !a.rec[n]) return;
    double SA = 0.0, SB = 0.0;
    for (int it = a.s.item_ptr[p]; it < a.s.item_ptr[p + 1]; it++) {
        int t = a.s.item[3 * it], ha = a.s.item[3 * it + 1], hb = a.s.item[3 * it + 2];
        double sbase = 0.0, vec = 0.0;
        double cb = a.coef[hb];
        double frx = a.fr[hb], fry = a.fr[2 * N + hb], frz = a.fr[4 * N + hb];
        for (int q = 0; q < Nq; q++) {
            size_t ip = (size_t)ha * Nq + q;
            size_t tq = (size_t)t * Nq + q;
            double P = a.s.P[tq];
            double jw = a.h.jw[ip];
            sbase += P * jw;
            double gx = cb * (a.s.V[3 * tq] - frx * P);
            double gy = cb * (a.s.V[3 * tq + 1] - fry * P);
            double gz = cb * (a.s.V[3 * tq + 2] - frz * P);
            vec += (a.h.fx[ip] * gx + a.h.fy[ip] * gy + a.h.fz[ip] * gz) * jw;
        }
        SA += a.h.div[ha] * a.h.div[hb] * (sbase * INV4PI_D);
        SB += vec * INV4PI_D;
    }
    if (m != n) {
        SA *= 0.5;
        SB *= 0.5;
    }
    cplx dL[2];
    for (int e = 0; e < a.nmed; e++) {
        Medium k = a.med[e];
        double k2 = k.kr * k.kr + k.ki * k.ki;
        cplx iok = {k.ki / k2, k.kr / k2};
        cplx ik = {-k.ki, k.kr};
        dL[e] = {-iok.re * SA + ik.re * SB, -iok.im * SA + ik.im * SB};
    }
    if (a.Z) {
        cplx TL, BR;
        if (a.nmed == 2) {
            TL = {a.eta_e * dL[0].re + a.eta_i * dL[1].re, a.eta_e * dL[0].im + a.eta_i * dL[1].im};
            BR = {dL[0].re / a.eta_e + dL[1].re / a.eta_i, dL[0].im / a.eta_e + dL[1].im / a.eta_i};
        } else {
            TL = {a.eta_e * dL[0].re, a.eta_e * dL[0].im};
            BR = {dL[0].re / a.eta_e, dL[0].im / a.eta_e};
        }
        double2* z;
        z = &a.Z[(int64_t)m * a.ldz + n];
        z->x += TL.re, z->y += TL.im;
        z = &a.Z[(int64_t)(N + m) * a.ldz + N + n];
        z->x += BR.re, z->y += BR.im;
        if (m != n) {
            z = &a.Z[(int64_t)n * a.ldz + m];
            z->x += TL.re, z->y += TL.im;
            z = &a.Z[(int64_t)(N + n) * a.ldz + N + m];
            z->x += BR.re, z->y += BR.im;
        }
    } else {
        double2* z = &a.L[(int64_t)m * a.ld + n];
        z->x += dL[0].re, z->y += dL[0].im;
        if (m != n) {
            z = &a.L[(int64_t)n * a.ld + m];
            z->x += dL[0].re, z->y += dL[0].im;
        }
    }
}

// mode 2: PMCHWT into Z; mode 1: L and K of medium 0 into L, K; mode 3: the
// exterior-only PMCHWT A_ext of medium 0 into Z.
int assemble_dev(bem_ctx* ctx, const bem_geom* g, double ke_re, double ke_im, double ki_re,
                 double ki_im, double eta_e, double eta_i, unsigned flags, int mode, void* Z,
                 int64_t ldz, void* L, void* K, const unsigned char* rwg_mask) {
    const int N = g->N;
    if (N < 1) return fail(ctx, BEM_ERR_INVALID, "empty basis");
    if ((mode == 2 || mode == 3) && (!Z || ldz < 2 * N)) return fail(ctx, BEM_ERR_INVALID, "bad Z / ldz");
    if (mode == 1 && (!L || !K || ldz < N)) return fail(ctx, BEM_ERR_INVALID, "bad L/K / ld");
    if (!(ke_re != 0.0 || ke_im != 0.0) || (mode == 2 && !(ki_re != 0.0 || ki_im != 0.0)))
        return fail(ctx, BEM_ERR_INVALID, "zero wavenumber");
    if (mode == 2 && (!(eta_e > 0) || !(eta_i > 0))) return fail(ctx, BEM_ERR_INVALID, "eta <= 0");
    if (mode == 3 && !(eta_e > 0)) return fail(ctx, BEM_ERR_INVALID, "eta <= 0");
    const int nmed = mode == 2 ? 2 : 1;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->stream;
    // 1. Graglia P, V per (triangle, point)
    TriQ tq;
    tq.n = g->quad.n;
    for (int i = 0; i < 25; i++) tq.l1[i] = g->quad.l1[i], tq.l2[i] = g->quad.l2[i], tq.w[i] = g->quad.w[i];
    int nthr = g->nt * g->Nq;
    graglia_kernel<<<(nthr + 127) / 128, 128, 0, st>>>(g->sing.tv, g->nt, tq, g->sing.P, g->sing.V);
    BEM_LAUNCHED(ctx);
    // 2. quadrature part, upper tiles
    AsmArgs a;
    a.h = g->half;
    a.N = N;
    a.Nq = g->Nq;
    a.ntile = (N + TILE - 1) / TILE;
    a.med[0] = {ke_re, ke_im};
    a.med[1] = {ki_re, ki_im};
    a.eta_e = eta_e;
    a.eta_i = eta_i;
    a.flags = flags;
    a.Z = mode == 1 ? nullptr : (double2*)Z;
    a.ldz = ldz;
    a.L = (double2*)L;
    a.K = (double2*)K;
    a.ld = ldz;
    a.coef = g->sing_coef;
    a.tile_flag = nullptr;
    // triangle pairs, unless a phase could leave the range of sincos_bounded
    // (|r - r'| <= extent): then the per-RWG kernel with the library's sine and cosine
    const double kmax = std::max(std::fabs(ke_re), mode == 2 ? std::fabs(ki_re) : 0.0);
    // or a medium's gain the range of exp_decay_bounded
    const double gain = std::max(-ke_im, mode == 2 ? -ki_im : 0.0);
    const bool tri = ctx->asm_kernel == 0 && kmax * g->extent < SINCOS_MAX && !(gain * g->extent > 700.0);
    const unsigned char* rec = nullptr;
    if (rwg_mask) {
        // tiles holding a flagged RWG, and the RWGs of those tiles
        mask_tiles_kernel<<<(a.ntile + 127) / 128, 128, 0, st>>>(rwg_mask, tri ? g->tri.tile_rwg : nullptr, N,
                                                                 a.ntile, g->tri.tile_flag);
        BEM_LAUNCHED(ctx);
        mask_rec_kernel<<<(N + 255) / 256, 256, 0, st>>>(g->tri.tile_flag, tri ? g->tri.pos : nullptr, N,
                                                         g->tri.rwg_rec);
        BEM_LAUNCHED(ctx);
        a.tile_flag = g->tri.tile_flag;
        rec = g->tri.rwg_rec;
    }
    int64_t ntiles = (int64_t)a.ntile * (a.ntile + 1) / 2;
    if (ntiles > 0x7fffffffLL) return fail(ctx, BEM_ERR_INVALID, "too many tiles");
    if (g->Nq > MAXQ) return fail(ctx, BEM_ERR_INVALID, "quadrature of %d points (at most %d)", g->Nq, MAXQ);
    cudaEvent_t ev = ctx->prof_begin(PROF_ASSEMBLY);
    if (tri) {
        const int damp = (ke_im != 0.0 ? 1 : 0) | (mode == 2 && ki_im != 0.0 ? 2 : 0);
        const unsigned nb = (unsigned)ntiles;
        if (mode == 2)
            BEM_TRY(damp == 0   ? (launch_assemble_tri<2, 0>(ctx, g, a, nb))
                    : damp == 2 ? (launch_assemble_tri<2, 2>(ctx, g, a, nb))
                                : (launch_assemble_tri<2, 3>(ctx, g, a, nb)));
        else
            BEM_TRY(damp == 0 ? (launch_assemble_tri<1, 0>(ctx, g, a, nb)) : (launch_assemble_tri<1, 1>(ctx, g, a, nb)));
    } else if (mode == 2) {
        assemble_kernel<2><<<(unsigned)ntiles, 256, 0, st>>>(a);
    } else {
        assemble_kernel<1><<<(unsigned)ntiles, 256, 0, st>>>(a);
    }
    BEM_LAUNCHED(ctx);
    // algorithmic unit: one quadrature-pair evaluation per medium, every
    // ordered RWG pair (no symmetry credit): 64 flop + sincos + exp each
    if (ev)
        ctx->prof_end(PROF_ASSEMBLY, ev, 64.0 * nmed * 4.0 * N * (double)N * g->Nq * g->Nq,
                      (mode == 1 ? 32.0 : 64.0) * (double)N * N);
    // 3. singular correction
    if (g->sing.npairs > 0) {
        FixArgs f;
        f.h = g->half;
        f.s = g->sing;
        f.coef = g->sing_coef;
        f.fr = g->sing_free;
        f.N = N;
        f.Nq = g->Nq;
        f.nmed = nmed;
        f.med[0] = {ke_re, ke_im};
        f.med[1] = {ki_re, ki_im};
        f.eta_e = eta_e;
        f.eta_i = eta_i;
        f.Z = a.Z;
        f.ldz = ldz;
        f.L = (double2*)L;
        f.ld = ldz;
        f.rec = rec;
        singular_fixup_kernel<<<(g->sing.npairs + 127) / 128, 128, 0, st>>>(f);
        BEM_LAUNCHED(ctx);
    }
    return BEM_OK;
}

}  // namespace bem

using namespace bem;

extern "C" {

int bem_geom_create(bem_ctx* ctx, const double* verts, int nv, const int* tris, int nt,
                    int quad_order, bem_geom** out, int* N) {
    if (!ctx || !out) return BEM_ERR_INVALID;
    *out = nullptr;
    bem_geom* g = new bem_geom();
    g->ctx = ctx;
    g->device = ctx->device;
    if (!host_mesh_from(verts, nv, tris, nt, &g->mesh)) {
        delete g;
        return fail(ctx, BEM_ERR_INVALID, "bad mesh arrays");
    }
    if (!quadrature(quad_order, &g->quad)) {
        delete g;
        return fail(ctx, BEM_ERR_INVALID, "quadrature order %d unsupported (4, 7, 13)", quad_order);
    }
    g->quad_order = quad_order;
    g->rwg = build_rwg(g->mesh);
    g->N = g->rwg.N;
    g->Nq = g->quad.n;
    g->nv = nv;
    g->nt = nt;
    if (g->N < 1) {
        delete g;
        return fail(ctx, BEM_ERR_INVALID, "mesh has no interior edges");
    }
    int s = cudaSetDevice(ctx->device) == cudaSuccess ? geom_upload(ctx, g) : BEM_ERR_CUDA;
    if (s != BEM_OK) {
        if (g->dmem) devmem_free(ctx->device, g->dmem, g->dmem_bytes, ctx);
        delete g;
        return s;
    }
    *out = g;
    if (N) *N = g->N;
    return BEM_OK;
}

int bem_geom_create_rwg(bem_ctx* ctx, const double* verts, int nv, const int* tris, int nt, int N,
                        const int* tri_p, const int* tri_m, const double* free_p, const double* free_m,
                        const double* length, const double* area_p, const double* area_m, int quad_order,
                        bem_geom** out) {
    if (!ctx || !out || N < 1 || !tri_p || !tri_m || !free_p || !free_m || !length || !area_p || !area_m)
        return BEM_ERR_INVALID;
    *out = nullptr;
    bem_geom* g = new bem_geom();
    g->ctx = ctx;
    g->device = ctx->device;
    if (!host_mesh_from(verts, nv, tris, nt, &g->mesh) || !quadrature(quad_order, &g->quad)) {
        delete g;
        return fail(ctx, BEM_ERR_INVALID, "bad mesh arrays or quadrature order");
    }
    HostRWG& r = g->rwg;
    r.N = N;
    for (int n = 0; n < N; n++) {
        if (tri_p[n] < 0 || tri_p[n] >= nt || tri_m[n] < 0 || tri_m[n] >= nt) {
            delete g;
            return fail(ctx, BEM_ERR_INVALID, "RWG %d refers to a missing triangle", n);
        }
        r.tri_p.push_back(tri_p[n]);
        r.tri_m.push_back(tri_m[n]);
        r.vfree_p.push_back(-1);
        r.vfree_m.push_back(-1);
        r.free_p.push_back({free_p[3 * n], free_p[3 * n + 1], free_p[3 * n + 2]});
        r.free_m.push_back({free_m[3 * n], free_m[3 * n + 1], free_m[3 * n + 2]});
        r.length.push_back(length[n]);
        r.area_p.push_back(area_p[n]);
        r.area_m.push_back(area_m[n]);
    }
    g->quad_order = quad_order;
    g->N = N;
    g->Nq = g->quad.n;
    g->nv = nv;
    g->nt = nt;
    int s = cudaSetDevice(ctx->device) == cudaSuccess ? geom_upload(ctx, g) : BEM_ERR_CUDA;
    if (s != BEM_OK) {
        if (g->dmem) devmem_free(ctx->device, g->dmem, g->dmem_bytes, ctx);
        delete g;
        return s;
    }
    *out = g;
    return BEM_OK;
}

int bem_geom_free(bem_geom* g) {
    if (!g) return BEM_OK;
    if (g->dmem) {
        cudaSetDevice(g->device);
        // last used on the creating context's stream (or the device waits)
        devmem_free(g->device, g->dmem, g->dmem_bytes, g->ctx);
    }
    delete g;
    return BEM_OK;
}

int bem_geom_size(const bem_geom* g) { return g ? g->N : 0; }

int bem_geom_set_vertices(bem_ctx* ctx, bem_geom* g, const double* verts) {
    if (!ctx || !g || !verts) return BEM_ERR_INVALID;
    BEM_TRY_CUDA(ctx, cudaSetDevice(ctx->device));
    return geom_set_vertices(ctx, g, verts);
}

int bem_assemble_pmchwt_dev(bem_ctx* ctx, const bem_geom* g, double kext_re, double kext_im,
                            double kint_re, double kint_im, double eta_ext, double eta_int,
                            unsigned flags, void* Z_dev, int64_t ldz) {
    if (!ctx || !g) return BEM_ERR_INVALID;
    return assemble_dev(ctx, g, kext_re, kext_im, kint_re, kint_im, eta_ext, eta_int, flags, 2,
                        Z_dev, ldz, nullptr, nullptr);
}

int bem_assemble_aext_dev(bem_ctx* ctx, const bem_geom* g, double kext_re, double kext_im, double eta_ext,
                          unsigned flags, void* Z_dev, int64_t ldz) {
    if (!ctx || !g) return BEM_ERR_INVALID;
    return assemble_dev(ctx, g, kext_re, kext_im, 0, 0, eta_ext, 1, flags, 3, Z_dev, ldz, nullptr, nullptr);
}

int bem_assemble_LK_dev(bem_ctx* ctx, const bem_geom* g, double k_re, double k_im,
                        unsigned flags, void* L_dev, void* K_dev, int64_t ld) {
    if (!ctx || !g) return BEM_ERR_INVALID;
    return assemble_dev(ctx, g, k_re, k_im, 0, 0, 1, 1, flags, 1, nullptr, ld, L_dev, K_dev);
}

}  // extern "C"
