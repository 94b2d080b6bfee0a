// ct_clip.cuh -- the Sutherland-Hodgman clip area (ct_geom.cuh) of small
// polygons, for the per-pair area kernels.
//
// Same values and vertex order as clip_area (and so upstream,
// algorithms/sutherland_hodgman.py:83-148), restricted to what nearly every
// pair is: a clip edge's line leaves the subject polygon whole, removes it,
// or crosses it twice, and at most 8 vertices are held.  Anything else
// (another number of crossings, a crossing with N.V == 0, non-finite or
// subnormal values, more vertices) returns false and the caller runs the
// general form.
//
// What bounds it: the general form spent 83 % of the float64 unit's time with
// 1.3 instructions issued per cycle and its polygons in local memory (4.3 KB
// per thread, 300 B of DRAM traffic per pair).  Here
//   * the vertices lie in shared memory, one column per thread (no bank
//     conflicts whatever slot each lane reads), and the polygon's order is a
//     word of 4-bit slot numbers, so kept vertices never move;
//   * the inside flags come from float32 coordinates relative to the first
//     clipper vertex, those of a new vertex from its edge's (no float64);
//   * division and part of the products run on the integer pipes
//     (ct_sf64.cuh) beside the float64 unit's additions.
// Zonal areas of 91M (box, mixed cell) pairs: 34.9 -> 20 ms, 1.6M (triangle,
// quad) pairs of two regridded meshes 1.55 -> 0.85 ms.  What bounds it now:
// the float64 unit's additions (about 90 per pair of a quad, 20 cycles each
// per warp) with the integer pipe at 70 % beside it.
#pragma once

#include "ct_geom.cuh"
#include "ct_sf64.cuh"

constexpr int CL_SLOTS = 8;   // vertices held per thread
constexpr int CL_THREADS = 128;

template <int KT>
struct ClipCols {
    double2 v[CL_SLOTS][CL_THREADS];
    float2 f[CL_SLOTS][CL_THREADS];
    double2 c[KT][CL_THREADS];
};

// x truncated to float (0 below the normal range, infinite above it)
__device__ __forceinline__ float cl_float(double x) {
    const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
    const uint32_t e = ((h >> 20) & 0x7ffu) - 897u;  // of a normal float: < 254
    const uint32_t t = (((__funnelshift_l(l, h, 3)) + 0x40000000u) & 0x7fffffffu);
    const uint32_t m = e < 254u ? t : (int)e < 0 ? 0u : 0x7f800000u;
    return __uint_as_float(m | (h & 0x80000000u));
}

__device__ __forceinline__ float cl_max2(float2 f) { return fmaxf(fabsf(f.x), fabsf(f.y)); }

// N.W or N.V and the like: one product on the integer pipes, one on the
// float64 unit, each rounded on its own
__device__ __forceinline__ double cl_dot(dpt a, dpt b, bool* bad) {
    return sf_mul(a.x, b.x, bad) + sf_mul(a.y, b.y, bad);
}

// Whether two vertices are equal, looked at in float64 only when their
// float32 coordinates (errors up to ed) allow it.
__device__ __forceinline__ bool cl_equal(float2 fa, float2 fb, float ed, double2 a, double2 b) {
    return fabsf(fa.x - fb.x) + fabsf(fa.y - fb.y) <= 4.1f * ed && a.x == b.x && a.y == b.y;
}

struct ClipCross {
    dpt p;
    float2 f;
    float e;  // error of f
    bool ok;
};

// sh_intersection of edge a -> b with the line through r with normal N.
// BOX: the subject began as a box, and when all lanes' edges are parallel to an
// axis (what is left of the box's sides: half of the crossings of a cell
// inside it) the products with the zero component are left out: they add a
// zero.  5 additions of the float64 unit instead of 8, 4 integer products
// instead of 6.  Pairs known to have the cell inside come together
// (ct_box_pair_order), so that whole warps take this path: 91M pairs 20.8 ->
// 19.9 ms (the order alone 20.6).
template <bool BOX>
__device__ __forceinline__ ClipCross cl_cross(double2 a2, double2 b2, float2 fa, float2 fb, dpt r, dpt N, float ed,
                                              float dabs) {
    const float u24 = 5.9604644775390625e-08f;
    const dpt a = mkp(a2.x, a2.y), b = mkp(b2.x, b2.y);
    const dpt W = mkp(r.x - a.x, r.y - a.y);
    bool bad = false, general = true;
    double nw = cl_dot(N, W, &bad), nv, t;
    ClipCross c;
    if (BOX) {
        const bool up = dbits(a.x) == dbits(b.x), flat = dbits(a.y) == dbits(b.y);
        if (!__any_sync(__activemask(), !(up || flat))) {
            general = false;
            const double am = up ? a.y : a.x, Vm = (up ? b.y : b.x) - am;
            nv = sf_mul(up ? N.y : N.x, Vm, &bad);
            t = sf_div(nw, nv, &bad);
            const double pm = am + sf_mul(t, Vm, &bad);
            c.p = up ? mkp(a.x, pm) : mkp(pm, a.y);
        }
    }
    if (general || bad) {
        const dpt V = mkp(b.x - a.x, b.y - a.y);
        double tx, ty;
        if (!bad) {
            nv = cl_dot(N, V, &bad);
            t = sf_div(nw, nv, &bad);
            tx = sf_mul(t, V.x, &bad);
            ty = sf_mul(t, V.y, &bad);
        }
        if (bad) {  // subnormal, overflow or N.V == 0: the hardware's operators
            nw = dotp(N, W);
            nv = dotp(N, V);
            t = nw / nv;
            tx = t * V.x;
            ty = t * V.y;
        }
        c.p = mkp(a.x + tx, a.y + ty);
    }
    const float tf = cl_float(t);
    const float2 fv = make_float2(fb.x - fa.x, fb.y - fa.y);
    c.f = make_float2(__fmaf_rn(tf, fv.x, fa.x), __fmaf_rn(tf, fv.y, fa.y));
    // for t in [0, 1] the errors of fa and fb combine to at most ed; then the
    // conversion of t (2 u), the subtraction and the sum's roundings, and the
    // float64 roundings of the vertex itself
    c.e = 1.03f * ed + 6.0f * u24 * cl_max2(fv) + 2.0f * u24 * cl_max2(c.f) + dabs;
    c.ok = !g_zero(nv) && tf >= -0.01f && tf <= 1.01f;
    return c;
}

// The clipped polygon: slots of its L (0: nothing left) vertices in order,
// with OWN the edge each vertex's outgoing edge lies on (subject edge k, from
// its vertex k, or 8 + i, the clipper's edge to its vertex i), and the error
// of its float32 coordinates.
struct ClipPoly {
    uint32_t list, own;
    int L;
    float ed;
};

// The subject's n_poly (<= CL_SLOTS) vertices in S.v and the clipper's n_clip
// in S.c (column of the thread).  False: not handled here (with OWN also
// clippers with an edge of no length).
template <int KT, bool BOX, bool OWN>
__device__ __forceinline__ bool clip_small(ClipCols<KT>& S, int tid, int n_poly, int n_clip, ClipPoly* C) {
    const float u24 = 5.9604644775390625e-08f;
    const double2 O = S.c[0][tid];
    float mx = 0.0f;
    if (BOX) {  // (x0, y0), (x1, y0), (x1, y1), (x0, y1)
        const double2 lo = S.v[0][tid], hi = S.v[2][tid];
        const float2 a = make_float2(cl_float(lo.x - O.x), cl_float(lo.y - O.y));
        const float2 b = make_float2(cl_float(hi.x - O.x), cl_float(hi.y - O.y));
        S.f[0][tid] = a;
        S.f[1][tid] = make_float2(b.x, a.y);
        S.f[2][tid] = b;
        S.f[3][tid] = make_float2(a.x, b.y);
        mx = fmaxf(cl_max2(a), cl_max2(b));
    } else {
        for (int k = 0; k < n_poly; k++) {
            const double2 v = S.v[k][tid];
            const float2 f = make_float2(cl_float(v.x - O.x), cl_float(v.y - O.y));
            S.f[k][tid] = f;
            mx = fmaxf(mx, cl_max2(f));
        }
    }
    double2 r = S.c[n_clip - 1][tid];
    float2 fr = make_float2(cl_float(r.x - O.x), cl_float(r.y - O.y));
    const float om = fmaxf(fabsf(cl_float(O.x)), fabsf(cl_float(O.y)));
    // ed, er: errors of the subject's float32 coordinates and of fr
    // (truncation to float, 2 u, and the float64 rounding of the difference)
    float ed = 2.01f * u24 * mx + 1e-37f, er = 2.01f * u24 * cl_max2(fr) + 1e-37f;
    const float dabs = 4.5e-16f * (om + 2.0f * mx) + 1e-37f;
    if (!(mx < 1e15f && om < 1e25f)) return false;
    uint32_t list = 0x76543210u;
    int L = n_poly;
    if (L < CL_SLOTS) list &= (1u << (4 * L)) - 1u;
    uint32_t own = list;
    C->L = 0;
    for (int k = 0, p = n_poly - 1; k < n_poly; p = k, k++)
        if (cl_equal(S.f[k][tid], S.f[p][tid], ed, S.v[k][tid], S.v[p][tid])) return false;
    for (int i = 0; i < n_clip; i++) {
        const double2 s = S.c[i][tid];
        const dpt U = mkp(s.x - r.x, s.y - r.y);
        if (g_zero(U.x) && g_zero(U.y)) {
            if (OWN) return false;
            continue;
        }
        const float2 uf = make_float2(cl_float(U.x), cl_float(U.y));
        if (!(cl_max2(uf) < 1e15f && cl_max2(fr) < 1e15f)) return false;
        // Inside test U.x (b.y - r.y) > U.y (b.x - r.x) in float32: with W =
        // f - fr, |W| <= M, errors ew = ed + er + u M of W and eU of U, the
        // estimate is off by at most 2 eU Mx + Nu ew + 4 u Nu Mx (float32
        // products and sum) + 2^-52 Nu Mx (float64 products), Mx = M + ew
        const float eU = 2.01f * u24 * cl_max2(uf) + 1e-37f, e2 = ed + er;
        const float Nu = fabsf(uf.x) + fabsf(uf.y) + 2.0f * eU;
        const float k1 = 1.03f * (2.0f * eU + 5.2f * u24 * Nu);
        const float k0 = 1.03f * (e2 * (2.0f * eU + 4.2f * u24 * Nu) + e2 * Nu) + 1e-37f;
        uint32_t in = 0, unsure = 0;
        for (int j = 0; j < L; j++) {
            const float2 f = S.f[(list >> (4 * j)) & 7u][tid];
            const float wx = f.x - fr.x, wy = f.y - fr.y;
            const float est = __fmaf_rn(uf.x, wy, -(uf.y * wx));
            const float thr = __fmaf_rn(fabsf(wx) + fabsf(wy), k1, k0);
            in |= (est > 0.0f ? 1u : 0u) << j;
            unsure |= (fabsf(est) > thr ? 0u : 1u) << j;
        }
        while (unsure) {
            const int j = __ffs(unsure) - 1;
            unsure &= unsure - 1u;
            const double2 b = S.v[(list >> (4 * j)) & 7u][tid];
            const double lhs = U.x * (b.y - r.y), rhs = U.y * (b.x - r.x);
            in = (in & ~(1u << j)) | ((lhs > rhs ? 1u : 0u) << j);
        }
        const uint32_t full = (1u << L) - 1u;
        if (in == 0u) return true;
        if (in != full) {
            const uint32_t prev = ((in << 1) | (in >> (L - 1))) & full;
            const uint32_t enter = in & ~prev, leave = prev & ~in;
            const int kept = __popc(in);
            if ((enter & (enter - 1u)) || kept + 2 > CL_SLOTS) return false;
            const int je = __ffs(enter) - 1, jl = __ffs(leave) - 1;
            uint32_t used = 0;
            for (uint32_t m = in; m; m &= m - 1u) used |= 1u << ((list >> (4 * (__ffs(m) - 1))) & 7u);
            const int je0 = je ? je - 1 : L - 1, jl0 = jl ? jl - 1 : L - 1;
            const uint32_t ea = (list >> (4 * je0)) & 7u, eb = (list >> (4 * je)) & 7u;
            const uint32_t la = (list >> (4 * jl0)) & 7u, lb = (list >> (4 * jl)) & 7u;
            const dpt N = mkp(sf_value(sf_bits(U.y) ^ 0x8000000000000000ull), U.x), rr = mkp(r.x, r.y);
            const ClipCross E = cl_cross<BOX>(S.v[ea][tid], S.v[eb][tid], S.f[ea][tid], S.f[eb][tid], rr, N, ed, dabs);
            const ClipCross X = cl_cross<BOX>(S.v[la][tid], S.v[lb][tid], S.f[la][tid], S.f[lb][tid], rr, N, ed, dabs);
            if (!(E.ok && X.ok)) return false;
            ed = fmaxf(ed, fmaxf(E.e, X.e));
            const double2 Ep = make_double2(E.p.x, E.p.y), Xp = make_double2(X.p.x, X.p.y);
            if (cl_equal(E.f, X.f, ed, Ep, Xp) || cl_equal(E.f, S.f[eb][tid], ed, Ep, S.v[eb][tid]) ||
                cl_equal(X.f, S.f[la][tid], ed, Xp, S.v[la][tid]))
                return false;
            const uint32_t s0 = __ffs(~used) - 1, s1 = __ffs(~used & ~(1u << s0)) - 1;
            S.v[s0][tid] = Ep;
            S.f[s0][tid] = E.f;
            S.v[s1][tid] = Xp;
            S.f[s1][tid] = X.f;
            // the walk's output order: a run of kept vertices je .. between
            // its two crossings, or, when the last vertex is kept, those up
            // to jl, the two crossings, those from je
            const uint32_t oe = (own >> (4 * je0)) & 15u, ol = 8u + (uint32_t)i;
            auto next = [&](uint32_t x, uint32_t e, uint32_t l) -> uint32_t {
                if ((in >> (L - 1)) & 1u)
                    return (x & ((1u << (4 * jl)) - 1u)) | (l << (4 * jl)) | (e << (4 * jl + 4)) |
                           ((x >> (4 * je)) << (4 * jl + 8));
                return e | (((x >> (4 * je)) & ((1u << (4 * kept)) - 1u)) << 4) | (l << (4 * kept + 4));
            };
            list = next(list, s0, s1);
            if (OWN) own = next(own, oe, ol);
            L = kept + 2;
        }
        // fs = fr + U: one rounding, and the errors of both
        r = s;
        fr = make_float2(fr.x + uf.x, fr.y + uf.y);
        er += eU + u24 * cl_max2(fr);
    }
    C->list = list;
    C->own = own;
    C->L = L < 3 ? 0 : L;
    C->ed = ed;
    return true;
}

template <int KT, bool BOX>
__device__ __forceinline__ bool clip_area_small(ClipCols<KT>& S, int tid, int n_poly, int n_clip, double* area) {
    ClipPoly C;
    if (!clip_small<KT, BOX, false>(S, tid, n_poly, n_clip, &C)) return false;
    const uint32_t list = C.list;
    *area = 0.0;
    if (C.L == 0) return true;
    // polygon_area geometry_utils.py:82-95
    const double2 a = S.v[list & 7u][tid], b = S.v[(list >> 4) & 7u][tid];
    dpt U = mkp(b.x - a.x, b.y - a.y);
    double sum = 0.0;
    bool bad = false;
    for (int j = 2; j < C.L; j++) {
        const double2 c = S.v[(list >> (4 * j)) & 7u][tid];
        const dpt V = mkp(a.x - c.x, a.y - c.y);
        double p = sf_mul(U.x, V.y, &bad), q = sf_mul(U.y, V.x, &bad);
        if (bad) {
            p = U.x * V.y;
            q = U.y * V.x;
        }
        sum += fabs(p - q);
        U = V;
    }
    *area = 0.5 * sum;
    return true;
}
