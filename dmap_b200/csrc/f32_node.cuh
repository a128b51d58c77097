// Outward-rounded FP32 node tests of the displaced-surface walk, shared by
// the FP32 kernels (walk32.cu describes the scheme). Every quantity lives in
// named scalars: no array is indexed by a run-time value, so nothing spills
// to the stack frame.
#pragma once
#include "device_types.cuh"
#include "f64_math.cuh"
#include "f64_leaf.cuh"
#include "f64_node.cuh"
#include "launch.h"

namespace d32
{
using dmapdev::AssetDev;
using dmapdev::TriDev;
using dmapdev::TriDev32;

constexpr float G = 9.5367431640625e-07f;     // 2^-20: bound factor for the roundings of one step
constexpr float U2 = 1.1920928955078125e-07f; // 2^-23

__device__ __forceinline__ float ru_add(float x, float y) { return __fadd_ru(x, y); }
__device__ __forceinline__ float rd_add(float x, float y) { return __fadd_rd(x, y); }
__device__ __forceinline__ float ru_mul(float x, float y) { return __fmul_ru(x, y); }
__device__ __forceinline__ float rd_mul(float x, float y) { return __fmul_rd(x, y); }
__device__ __forceinline__ float ru_fma(float x, float y, float z) { return __fmaf_ru(x, y, z); }
// 2^e exactly, -126 <= e <= 127
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }

struct Node32 { float h0, gu, gv, r, mn, mx; };

// First cell of level l of a pyramid over 2^L x 2^L leaf cells: the sum of
// 4^(L - m) over m < l, that is 4^(L + 1 - l) (4^l - 1) / 3.
__device__ __forceinline__ int64_t level_first(int L, int l)
{
    return (int64_t)((0x5555555555555555ull & ((1ull << (2 * l)) - 1ull)) << (2 * (L + 1 - l)));
}

// TaylorPyramid::node (taylor_pyramid.cpp:259-274) on the FP32 pyramid of
// 2^L x 2^L leaf cells: wrapped indices (the level's width is a power of
// two), above the root the root's height range as a min-max node.
__device__ __forceinline__ Node32 fetch_node(const float *pyr32, int L, int level, int i, int j)
{
    Node32 n;
    const bool above = level > L;
    const int lv = above ? L : level;
    const int m1 = (1 << (L - lv)) - 1;
    const int64_t at = level_first(L, lv) + (((int64_t)(j & m1)) << (L - lv)) + (i & m1);
    const float4 *p = reinterpret_cast<const float4 *>(pyr32 + 8 * at);
    const float4 q0 = __ldg(p), q1 = __ldg(p + 1);
    n.h0 = q0.x;
    n.gu = q0.y;
    n.gv = q0.z;
    n.r = q0.w;
    n.mn = q1.z;
    n.mx = q1.w;
    if (above) {
        n.h0 = 0.5f * (n.mn + n.mx);
        n.r = fmaxf(__fsub_ru(n.mx, n.h0), __fsub_ru(n.h0, n.mn));
        n.gu = n.gv = 0.0f;
    }
    return n;
}

// What the node test and the walk's domain test read of a triangle's FP32
// record, loaded as nine 16-byte words.
struct Walk32
{
    float4 n[3]; // per axis: a0, au, av, rowsum
    float qc, q1, q2, q11, q12, q22;
    float lox, loy, hix, hiy;
    float ux[3], uy[3], udm[3];
    float nerr[3], qerr;
    int log2n;
};

__device__ __forceinline__ Walk32 load_walk(const TriDev32 &T)
{
    const float4 *p = reinterpret_cast<const float4 *>(&T);
    const float4 a = __ldg(p + 3), b = __ldg(p + 4), c = __ldg(p + 5), d = __ldg(p + 6), f = __ldg(p + 8), g = __ldg(p + 9);
    Walk32 w;
    w.n[0] = __ldg(p);
    w.n[1] = __ldg(p + 1);
    w.n[2] = __ldg(p + 2);
    w.qc = a.x, w.q1 = a.y, w.q2 = a.z, w.q11 = a.w;
    w.q12 = b.x, w.q22 = b.y;
    w.lox = b.z, w.loy = b.w, w.hix = c.x, w.hiy = c.y;
    w.ux[0] = c.z, w.uy[0] = c.w, w.ux[1] = d.x, w.uy[1] = d.y, w.ux[2] = d.z, w.uy[2] = d.w;
    w.nerr[0] = f.x, w.nerr[1] = f.y, w.nerr[2] = f.z, w.qerr = f.w;
    w.udm[0] = g.x, w.udm[1] = g.y, w.udm[2] = g.z;
    w.log2n = __float_as_int(g.w);
    return w;
}

// The tangent-space ray (o, d), its reciprocal directions and the widening
// E that covers its rounding from the double ray.
struct Ray32 { float ox, oy, oz, dx, dy, dz, ix, iy, iz, ex, ey, ez; };

struct Cell32 { int level, i, j; };

__device__ __forceinline__ int fdiv2(int x) { return x >> 1; } // arithmetic shift: floor division by 2
__device__ __forceinline__ void cell_next(Cell32 &c, int si, int sj, int root_level)
{
    // displaced_intersector.cpp:99-121
    for (;;) {
        int code = 2 * ((c.i + si) & 1) + ((c.j + sj) & 1);
        if (code == 1) {
            c.j += sj ? 1 : -1;
            c.i += si ? -1 : 1;
            return;
        }
        if (code == 3) {
            ++c.level;
            c.i = fdiv2(c.i);
            c.j = fdiv2(c.j);
            if (c.level > root_level)
                return;
            continue;
        }
        c.j += sj ? -1 : 1;
        return;
    }
}

// classify_square (uv_clip.cpp:27-44) reporting Outside only when the
// separation exceeds the rounding of the test: of a footprint's cell, with
// the bound of that rounding in udm, ...
__device__ __forceinline__ bool cell_meets_domain(const Walk32 &T, float cx, float cy, float s)
{
    if (cx + s <= T.lox || cx - s >= T.hix || cy + s <= T.loy || cy - s >= T.hiy)
        return false;
    bool out = false;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        out = out || __fmaf_rn(fabsf(T.ux[k]) + fabsf(T.uy[k]), s, __fmaf_rn(T.uy[k], cy, T.ux[k] * cx)) <= T.udm[k];
    return !out;
}

// ... and of a leaf's sub-square, with the bound taken where it is.
__device__ __forceinline__ bool square_meets_domain(const TriDev32 &T, float cx, float cy, float s)
{
    if (cx + s <= T.lo[0] || cx - s >= T.hi[0] || cy + s <= T.lo[1] || cy - s >= T.hi[1])
        return false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float proj = __fmaf_rn(T.un[k][1], cy, T.un[k][0] * cx);
        float ext = (fabsf(T.un[k][0]) + fabsf(T.un[k][1])) * s;
        float slack = G * (fabsf(T.un[k][0] * cx) + fabsf(T.un[k][1] * cy) + fabsf(T.ud[k]) + ext);
        if (proj + ext + slack <= T.ud[k])
            return false;
    }
    return true;
}

struct Iv { float lo, hi; };
__device__ __forceinline__ Iv iv_scale(float s, Iv a)
{
    return s >= 0.0f ? Iv{rd_mul(s, a.lo), ru_mul(s, a.hi)} : Iv{rd_mul(s, a.hi), ru_mul(s, a.lo)};
}
__device__ __forceinline__ Iv iv_add(Iv a, Iv b) { return {rd_add(a.lo, b.lo), ru_add(a.hi, b.hi)}; }
__device__ __forceinline__ Iv iv_mul(Iv a, Iv b)
{
    float p0 = rd_mul(a.lo, b.lo), p1 = rd_mul(a.lo, b.hi), p2 = rd_mul(a.hi, b.lo), p3 = rd_mul(a.hi, b.hi);
    float q0 = ru_mul(a.lo, b.lo), q1 = ru_mul(a.lo, b.hi), q2 = ru_mul(a.hi, b.lo), q3 = ru_mul(a.hi, b.hi);
    return {fminf(fminf(p0, p1), fminf(p2, p3)), fmaxf(fmaxf(q0, q1), fmaxf(q2, q3))};
}
__device__ __forceinline__ float iv_mag(Iv a) { return fmaxf(fabsf(a.lo), fabsf(a.hi)); }

__device__ __forceinline__ float tol32(float t) { return G * fmaxf(1.0f, fabsf(t)); }

// One axis of Aabb3::clip (node_bounds.cpp:25-44).
__device__ __forceinline__ void clip_axis(float o, float d, float inv, float lo, float hi, float &t0, float &t1,
                                          bool &ok)
{
    if (d != 0.0f) {
        float ta = (lo - o) * inv, tb = (hi - o) * inv;
        t0 = fmaxf(t0, fminf(ta, tb));
        t1 = fminf(t1, fmaxf(ta, tb));
    } else if (o < lo || o > hi) {
        ok = false;
    }
}

// The range of 1/|N| over the rectangle [cx +- hx] x [cy +- hy], with
// |N(s,t)|^2 = qc + 2 s q1 + 2 t q2 + s^2 q11 + 2 s t q12 + t^2 q22, as
// midpoint rm and radius rr; false when |N| may vanish there. The roundings
// of the centre value and of the spread are at most some ten units in the
// last place of the sum of the terms' magnitudes, whose bound over the domain
// gives qerr.
__device__ __forceinline__ bool inv_norm_range(const Walk32 &T, float cx, float cy, float hx, float hy, float &rm,
                                               float &rr)
{
    const float gs = __fmaf_rn(cy, T.q12, __fmaf_rn(cx, T.q11, T.q1));
    const float gt = __fmaf_rn(cy, T.q22, __fmaf_rn(cx, T.q12, T.q2));
    const float qv = __fmaf_rn(cy, T.q2 + gt, __fmaf_rn(cx, T.q1 + gs, T.qc));
    const float hx2 = hx + hx, hy2 = hy + hy;
    const float quad = ru_fma(hx * hx, fabsf(T.q11), ru_mul(hy * hy, fabsf(T.q22)));
    const float spread = ru_add(ru_fma(hx2, ru_fma(hy, fabsf(T.q12), fabsf(gs)), ru_mul(hy2, fabsf(gt))), T.qerr);
    const float q_lo = __fsub_rd(qv, spread), q_hi = ru_add(ru_add(qv, spread), quad);
    if (!(q_lo > 0.0f) || !(q_hi < INFINITY))
        return false;
    const float up = 1.0f + 9.5367431640625e-07f, dn = 1.0f - 9.5367431640625e-07f;
    float r_lo = rd_mul(rsqrtf(q_hi), dn), r_hi = ru_mul(rsqrtf(q_lo), up);
    rm = 0.5f * (r_lo + r_hi);
    rr = fmaxf(__fsub_ru(r_hi, rm), __fsub_ru(rm, r_lo));
    return true;
}

// One component of the tangent normal's enclosure m_k = (A N)_k / |N|: the
// affine form of (A N)_k = a0 + s au + t av over the rectangle (its
// coefficients rounded from double, their rounding and the evaluation's in
// nerr) times the interval rm +- rr. Then the box coordinate p_k + h m_k with
// h = mid +- hh and the base point's form (pc, pa, pb), hulled outward and
// widened by E: the ray's own rounding and the base point's.
// With s1 = |nc| + |na| + |nb|: m = c + a eu + b ev + rho, |rho| <= k =
// rr (s1 + nerr) + rm (G s1 + nerr), |c| + |a| + |b| + k <= V = rm' s1 + k,
// rm' = rm (1 + G); h m + p has the remainder |mid| (k + G V) + hh V.
__device__ __forceinline__ void box_axis(const float4 &n, float nerr, float cx, float cy, float hx, float hy, bool ok,
                                         float rm, float rmu, float rr, float mid, float hh, float pc, float pa,
                                         float pb, float E, float &lo, float &hi, float &mc, float &mh)
{
    const float nc = __fmaf_rn(cy, n.z, __fmaf_rn(cx, n.y, n.x));
    const float na = hx * n.y, nb = hy * n.z;
    const float s1 = ru_add(ru_add(fabsf(na), fabsf(nb)), fabsf(nc));
    const float c = rm * nc, a = rm * na, b = rm * nb;
    float k = ru_fma(rr, ru_add(s1, nerr), ru_mul(rm, ru_fma(G, s1, nerr)));
    // |N| can vanish over the rectangle (rm = rr = 0): a unit normal maps into |m_k| <= sum_j |A_kj|
    k = ok ? k : n.w;
    const float V = ru_fma(rmu, s1, k);
    mc = c;
    mh = ru_add(ru_add(fabsf(a), fabsf(b)), k);
    const float tc = __fmaf_rn(mid, c, pc), ta = __fmaf_rn(mid, a, pa), tb = __fmaf_rn(mid, b, pb);
    const float sk = ru_fma(hh, V, ru_fma(fabsf(mid), ru_fma(G, V, k), E));
    const float e = ru_add(ru_add(fabsf(ta), fabsf(tb)), sk);
    const float w = ru_fma(G, ru_add(fabsf(tc), e), e); // and the clip's own rounding
    lo = __fsub_rd(tc, w);
    hi = __fadd_ru(tc, w);
}

// a / b as a product with the hardware's reciprocal (rcp.approx: within 1
// ulp), rounded up / down past its error, for |b| between 1e-30 and 1e30,
// whose reciprocal is a normal float.
__device__ __forceinline__ bool quot_ok(float b) { return fabsf(b) > 1e-30f && fabsf(b) < 1e30f; }
__device__ __forceinline__ float approx_rcp(float b)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
}
__device__ __forceinline__ float quot_up(float a, float b)
{
    const float q = a * approx_rcp(b);
    return __fmaf_ru(fabsf(q), 4.76837158203125e-07f, q);
}
__device__ __forceinline__ float quot_dn(float a, float b)
{
    const float q = a * approx_rcp(b);
    return __fmaf_rd(-fabsf(q), 4.76837158203125e-07f, q);
}

// The node test of one cell (node_bounds.cpp:83-211): the box, and at levels
// <= slab_max_level the slab, both enclosing their double counterparts. Its
// roundings are bounded by constants of the triangle where a bound over the
// domain is as good as one at the cell (a box coordinate took 52 operations
// with every magnitude summed, 33 to 35 so: walk rounds of 2.80M rays on 96 x
// 2048^2 maps 14.6 -> 13.6 ms).
__device__ __forceinline__ bool node_test32(const Walk32 &T, const float *pyr32, const Ray32 &r, int level, int i,
                                            int j, float t_min, float t_max, int bound, int slab_max_level)
{
    Node32 n = fetch_node(pyr32, T.log2n, level, i, j);
    float w = pow2f(level - T.log2n);
    float u0 = ((float)i + 0.5f) * w, v0 = ((float)j + 0.5f) * w;
    float rlx = fmaxf((float)i * w, T.lox), rly = fmaxf((float)j * w, T.loy);
    float rhx = fminf((float)(i + 1) * w, T.hix), rhy = fminf((float)(j + 1) * w, T.hiy);
    float cx = 0.5f * (rlx + rhx), cy = 0.5f * (rly + rhy);
    float hx = fmaxf(fmaxf(__fsub_ru(rhx, cx), __fsub_ru(cx, rlx)), 0.0f);
    float hy = fmaxf(fmaxf(__fsub_ru(rhy, cy), __fsub_ru(cy, rly)), 0.0f);
    float rm = 0.0f, rr = 0.0f;
    bool ok = inv_norm_range(T, cx, cy, hx, hy, rm, rr);
    const float rmu = ru_mul(rm, 1.0f + G);
    float mid = 0.5f * (n.mn + n.mx);
    float hh = fmaxf(__fsub_ru(n.mx, mid), __fsub_ru(mid, n.mn));
    float lx, hx_, ly, hy_, lz, hz, mxc, mxh, myc, myh, mzc, mzh;
    // The base point's roundings (of the cell's corners past 2^24 cells, of
    // the rectangle's centre, of the sums with h m) are a few 2^-24 of its own
    // coordinate. Bounded over the domain instead, a chart of 12,000 tiles
    // admitted six times the leaf cells near its origin.
    const float ex = ru_fma(G, ru_add(fabsf(cx), hx), r.ex), ey = ru_fma(G, ru_add(fabsf(cy), hy), r.ey);
    box_axis(T.n[0], T.nerr[0], cx, cy, hx, hy, ok, rm, rmu, rr, mid, hh, cx, hx, 0.0f, ex, lx, hx_, mxc, mxh);
    box_axis(T.n[1], T.nerr[1], cx, cy, hx, hy, ok, rm, rmu, rr, mid, hh, cy, 0.0f, hy, ey, ly, hy_, myc, myh);
    box_axis(T.n[2], T.nerr[2], cx, cy, hx, hy, ok, rm, rmu, rr, mid, hh, 0.0f, 0.0f, 0.0f, r.ez, lz, hz, mzc, mzh);
    bool read_slab = level <= slab_max_level;
    float b0 = t_min, b1 = t_max;
    if (bound != 1 || !read_slab) {
        bool okc = true;
        clip_axis(r.ox, r.dx, r.ix, lx, hx_, b0, b1, okc);
        clip_axis(r.oy, r.dy, r.iy, ly, hy_, b0, b1, okc);
        clip_axis(r.oz, r.dz, r.iz, lz, hz, b0, b1, okc);
        if (!okc || b0 > b1 + tol32(fmaxf(fabsf(b0), fabsf(b1))))
            return false;
        if (bound == 0 || !read_slab)
            return true;
    }
    // slab (node_bounds.cpp:111-122, 137-179) in outward interval arithmetic
    float c0 = t_min, c1 = t_max;
    bool okc = true;
    clip_axis(r.ox, r.dx, r.ix, lx, hx_, c0, c1, okc);
    clip_axis(r.oy, r.dy, r.iy, ly, hy_, c0, c1, okc);
    if (!okc || c0 > c1 + tol32(fmaxf(fabsf(c0), fabsf(c1))))
        return false;
    Iv mx = {__fsub_rd(mxc, mxh), __fadd_ru(mxc, mxh)}, my = {__fsub_rd(myc, myh), __fadd_ru(myc, myh)},
       mz = {__fsub_rd(mzc, mzh), __fadd_ru(mzc, mzh)};
    Iv A = iv_add(iv_add(Iv{1.0f, 1.0f}, iv_scale(n.gu, mx)), iv_scale(n.gv, my));
    Iv B = iv_scale(-n.gu, mz), C = iv_scale(-n.gv, mz);
    float p1lo = rd_mul(n.gu, u0), p1hi = ru_mul(n.gu, u0), p2lo = rd_mul(n.gv, v0), p2hi = ru_mul(n.gv, v0);
    Iv P0 = {__fsub_rd(__fsub_rd(n.h0, p1hi), p2hi), __fsub_ru(__fsub_ru(n.h0, p1lo), p2lo)};
    Iv D = iv_mul(Iv{-P0.hi, -P0.lo}, mz);
    // the FP32 plane's gradient rounding, |dgu| s + |dgv| s, joins the remainder
    float reff = ru_fma(U2 * (0.5f * w), ru_add(fabsf(n.gu), fabsf(n.gv)), n.r);
    float R = ru_mul(reff, iv_mag(mz));
    // the ray's rounding, and the cell centre's (two roundings past 2^23 cells)
    const float eu = ru_fma(0x1p-22f, fabsf(u0), 2.0f * r.ex), ev = ru_fma(0x1p-22f, fabsf(v0), 2.0f * r.ey);
    R = ru_fma(iv_mag(A), 2.0f * r.ez, ru_fma(iv_mag(B), eu, ru_fma(iv_mag(C), ev, R)));
    float ax = __fmaf_rn(c0, r.dx, r.ox), ay = __fmaf_rn(c0, r.dy, r.oy), az = __fmaf_rn(c0, r.dz, r.oz);
    float span = c1 - c0;
    Iv F0 = iv_add(iv_add(iv_add(iv_scale(az, A), iv_scale(ax, B)), iv_scale(ay, C)), D);
    Iv F1 = iv_add(iv_add(iv_scale(r.dz, A), iv_scale(r.dx, B)), iv_scale(r.dy, C));
    // the quotients of the interval test as products with a reciprocal within
    // 2^-23, widened by 2^-21; a divisor out of its range bounds nothing
    float s0 = 0.0f, s1 = span;
    const float ql = __fsub_ru(R, F0.lo), qh = __fsub_rd(-R, F0.hi);
    if (quot_ok(F1.lo)) {
        if (F1.lo > 0.0f)
            s1 = fminf(s1, quot_up(ql, F1.lo));
        else
            s0 = fmaxf(s0, quot_dn(ql, F1.lo));
    } else if (F1.lo == 0.0f && F0.lo > R) {
        return false;
    }
    if (quot_ok(F1.hi)) {
        if (F1.hi > 0.0f)
            s0 = fmaxf(s0, quot_dn(qh, F1.hi));
        else
            s1 = fminf(s1, quot_up(qh, F1.hi));
    } else if (F1.hi == 0.0f && F0.hi < -R) {
        return false;
    }
    if (s0 > s1 + tol32(fabsf(c0) + span))
        return false;
    if (bound == 1)
        return true;
    float t0 = fmaxf(b0, c0 + s0), t1 = fminf(b1, c0 + s1);
    return !(t0 > t1 + tol32(fmaxf(fabsf(t0), fabsf(t1))));
}

template <typename R>
__device__ __forceinline__ void load_ray(const R *rays, int64_t k, double *o, double *d, double &t_min, double &t_max)
{
    const R *r = rays + 8 * k;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        o[a] = (double)r[a];
        d[a] = (double)r[3 + a];
    }
    t_min = (double)r[6];
    t_max = (double)r[7];
    dmapdev::sanitize_ray(o, d, t_min, t_max);
}

// The same for a ray record type chosen at run time (QueryOpts::ray_dtype).
__device__ __forceinline__ void load_ray(const void *rays, int ray_dtype, int64_t k, double *o, double *d,
                                         double &t_min, double &t_max)
{
    if (ray_dtype == 2)
        load_ray(static_cast<const double *>(rays), k, o, d, t_min, t_max);
    else
        load_ray(static_cast<const float *>(rays), k, o, d, t_min, t_max);
}

template <typename H, typename Fp>
__device__ __forceinline__ void store_hit(H *hits, int64_t k, bool found, const d64::hit64 &h, int tri, int flags)
{
    H out;
    if (found) {
        out.t = (Fp)h.t;
        out.st[0] = (Fp)h.st.x;
        out.st[1] = (Fp)h.st.y;
        out.bary[0] = (Fp)h.bary.x;
        out.bary[1] = (Fp)h.bary.y;
        out.ng[0] = (Fp)h.ng.x;
        out.ng[1] = (Fp)h.ng.y;
        out.ng[2] = (Fp)h.ng.z;
        out.tri = tri;
        out.i = (int32_t)h.i;
        out.j = (int32_t)h.j;
        out.flags = flags;
    } else {
        out.t = (Fp)INFINITY;
        out.st[0] = out.st[1] = out.bary[0] = out.bary[1] = (Fp)0;
        out.ng[0] = out.ng[1] = out.ng[2] = (Fp)0;
        out.tri = -1;
        out.i = out.j = 0;
        out.flags = flags;
    }
    hits[k] = out;
}

// The same for a hit record type chosen at run time (QueryOpts::hit_dtype).
__device__ __forceinline__ void store_hit(void *hits, int hit_dtype, int64_t k, bool found, const d64::hit64 &h,
                                          int tri, int flags)
{
    if (hit_dtype == 2)
        store_hit<dmapdev::Hit64, double>(static_cast<dmapdev::Hit64 *>(hits), k, found, h, tri, flags);
    else
        store_hit<dmapdev::Hit32, float>(static_cast<dmapdev::Hit32 *>(hits), k, found, h, tri, flags);
}

// A leaf cell the FP32 walk reached: first the reference's own node test of
// the cell in double (the FP32 tests, widened by the ray's rounding, admit
// more leaf cells than the FP64 walk; a cell the FP64 walk rejects has no
// leaf there), then the certified Newton leaf.
__device__ __noinline__ inline bool leaf64(const TriDev &T, const AssetDev &g, const double *o, const double *d,
                                           double t_min, double t_max, int i, int j, d64::hit64 &h, int64_t *st,
                                           const dmapk::QueryOpts &opt)
{
    d64::v3 O = d64::V3(o[0], o[1], o[2]), D = d64::V3(d[0], d[1], d[2]);
    if (!d64::leaf_cell_admitted(T, g, O, D, t_min, t_max, i, j, opt))
        return false;
    return d64::intersect_newton(T, g, O, D, t_min, t_max, i, j, h, st);
}

} // namespace d32
