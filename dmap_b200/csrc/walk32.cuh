// The FP32 query path: the reference's walk (displaced_intersector.cpp:175-237)
// with every node test evaluated in FP32 and widened outward (f32_node.cuh),
// so that a cell the double-precision test admits is admitted here too;
// leaves run the reference's certified Newton leaf in double (f64_leaf.cuh),
// which makes every reported hit the reference's own FP64 root.
//
// Conservative FP32 arithmetic. A form is c + a eu + b ev + rho with
// |rho| <= k; c, a, b are rounded to nearest and k is an upper bound kept
// with round-up operations. Every operation adds to k a bound on the
// rounding of the coefficients it produced: G * (sum of the magnitudes of
// the terms that entered them), G = 2^-20 (16 units in the last place, more
// than the few roundings of each step), and every input rounded from double
// (the triangle's frame, normals, pyramid nodes) carries its own rounding
// into k the same way. The reciprocal norm is bounded with directed rounding
// around rsqrtf's documented 2-ulp error. The box of a cell is the outward
// interval hull; the tangent-space ray (transformed in double, then rounded)
// is covered by widening every box by the ray's own rounding error over the
// triangle's t range. Slab tests use directed-rounding interval arithmetic.
//
// Two schedules:
//  - simple: one thread per ray, one launch (the plain per-request kernel).
//    Its lanes serialize on divergence: each lane walks its own triangles
//    while the others wait (measured 1.6 active threads per warp
//    instruction on the cube-sphere workload).
//  - wavefront (default): rounds of two persistent kernels. The walk kernel
//    gives each ray four lanes, which test the four cells of a sibling group
//    together: a ray that reaches leaves writes a leaf job, parks its walk
//    state and its lanes take the next ray; the leaf kernel runs the parked
//    leaves, a job per quad of lanes, and queues their rays to resume.
//    After `rounds` rounds a last walk runs the few remaining rays with
//    their leaves inline. Every ray still visits its cells in the
//    reference's order with the reference's t_max, so its hit is the one
//    the simple schedule finds.
//
// The kernels live in this header and are instantiated by two translation
// units (walk32_launch.h lists which launches each one owns):
//  - walk32.cu, compiled with FMA contraction: the walk rounds, whose
//    arithmetic is conservative by its error bounds, so a fused multiply-add
//    (one rounding instead of two) stays inside them, and whose rounding
//    never reaches a result (every leaf cell is re-tested in FP64);
//  - walk32_exact.cu, compiled with -fmad=false: everything that must round
//    like the reference or the same way wherever it runs: the simple
//    schedule, the last walk with leaves inline, the leaf rounds of both
//    leaves and the FP64 re-test of parked cells.
// FP32 code asks for fused multiply-adds explicitly (fmaf) where its bounds
// are written for one.
#pragma once
#include "walk32_launch.h"
#include "f32_node.cuh"
#include "bvh.cuh"
#include "leaf32.cuh"
#include "leaf_quad.cuh"
#include "order.cuh"
#include "filter.cuh"
#include "instance.cuh"

namespace
{
using namespace d32;
using dmapdev::AssetDev;
using dmapdev::TriDev;
using dmapdev::TriDev32;

// Resident 128-thread CTAs per SM the walk rounds are compiled for (register
// budget: 65536 / (128 x blocks) per thread; 96 registers at 5). 2.80M rays on
// the sphere of 96 x 2048^2 maps, walk rounds at 4 / 5 / 6: 18.3 / 16.3 / 16.2
// ms; 20,011 rays on 512^2 maps 0.43 / 0.45 / 0.49.
#ifndef DMAP_WALK_MIN_BLOCKS
#define DMAP_WALK_MIN_BLOCKS 5
#endif
#ifndef DMAP_WALK_TREE_MIN_BLOCKS
#define DMAP_WALK_TREE_MIN_BLOCKS 5
#endif
// Node tests a ray may run past its first collected leaf before it parks.
#ifndef DMAP_STALE_CAP
#define DMAP_STALE_CAP 32
#endif

constexpr int kMaskWords = 8; // scenes of up to 256 triangles take the object-box candidate mask
constexpr unsigned FULL = 0xffffffffu;

// The tangent-space ray of a triangle: transformed in double, rounded to
// float, and E covering, for t in [0, t_far], the distance between the float
// ray and the reference's double ray (A (o - q0), A d in its own operation
// order): the rounding to float, at most 2^-24 of each coordinate (2^-22
// taken), plus the difference of two double evaluations of the transform,
// a few units of 2^-53 of the sums of the terms' magnitudes (2^-40 taken of
// the row's magnitude sum times the largest component). tangent_row: axis a.
__device__ __forceinline__ void tangent_row(const TriDev32 &T, int a, const double *o, const double *d, float t_far,
                                            float &ro, float &rd, float &e)
{
    const double A0 = T.A[a][0], A1 = T.A[a][1], A2 = T.A[a][2];
    const double u0 = o[0] - T.q0[0], u1 = o[1] - T.q0[1], u2 = o[2] - T.q0[2];
    const double d0 = d[0], d1 = d[1], d2 = d[2];
    ro = (float)__fma_rn(A2, u2, __fma_rn(A1, u1, A0 * u0));
    rd = (float)__fma_rn(A2, d2, __fma_rn(A1, d1, A0 * d0));
    const float um = fmaxf(fmaxf(fabsf((float)u0), fabsf((float)u1)), fabsf((float)u2));
    const float dm = fmaxf(fmaxf(fabsf((float)d0), fabsf((float)d1)), fabsf((float)d2));
    const float sum = ru_mul(__double2float_ru(fabs(A0) + fabs(A1) + fabs(A2)), ru_fma(t_far, dm, um));
    e = ru_fma(0x1p-22f, ru_fma(t_far, fabsf(rd), fabsf(ro)), ru_mul(0x1.1p-40f, sum));
}

__device__ __forceinline__ void tangent_ray(const TriDev32 &T, const double *o, const double *d, float t_far,
                                            Ray32 &r)
{
    tangent_row(T, 0, o, d, t_far, r.ox, r.dx, r.ex);
    tangent_row(T, 1, o, d, t_far, r.oy, r.dy, r.ey);
    tangent_row(T, 2, o, d, t_far, r.oz, r.dz, r.ez);
    r.ix = r.dx != 0.0f ? __frcp_rn(r.dx) : 0.0f;
    r.iy = r.dy != 0.0f ? __frcp_rn(r.dy) : 0.0f;
    r.iz = r.dz != 0.0f ? __frcp_rn(r.dz) : 0.0f;
}

__device__ __forceinline__ float far_bound(float t1) { return ru_add(ru_mul(t1, 1.0f + 4.0f * G), G); }

// Position of the k-th set bit (k from 0) of m, or -1.
__device__ __forceinline__ int nth_bit(unsigned m, int k)
{
#pragma unroll 1
    for (; k > 0; --k)
        m &= m - 1u;
    return __ffs((int)m) - 1;
}
// m without its k lowest set bits.
__device__ __forceinline__ unsigned drop_bits(unsigned m, int k)
{
#pragma unroll 1
    for (; k > 0; --k)
        m &= m - 1u;
    return m;
}

// ---- simple schedule: one thread per ray ----------------------------------

// A leaf cell the FP32 walk reached, in the simple schedule and the
// inline-leaf walk: the cell's FP64 node test, then the certified leaf in the
// query's leaf precision (FP64: the reference's leaf; FP32: leaf32.cuh).
// flags: DMAP_HIT_* of the root.
__device__ __noinline__ bool leaf_cell(const TriDev32 &T32, const TriDev &T, const AssetDev &g, const double *o,
                                       const double *d, double t_min, double t_max, int i, int j, d64::hit64 &h,
                                       int &flags, int64_t *st, const dmapk::QueryOpts &opt)
{
    // an instanced triangle meets the ray in its object space (instance.cuh)
    double oo[3], od[3];
    if (T.inst) {
        dmapdev::object_ray(opt.inst_xf + dmapdev::kInstDoubles * (T.inst - 1), o, d, oo, od);
        o = oo;
        d = od;
    }
    bool ok;
    if (opt.leaf_precision != 1) {
        flags = DMAP_HIT_FP64_LEAF;
        ok = leaf64(T, g, o, d, t_min, t_max, i, j, h, st, opt);
    } else {
        d64::v3 O = d64::V3(o[0], o[1], o[2]), D = d64::V3(d[0], d[1], d[2]);
        ok = d64::leaf_cell_admitted(T, g, O, D, t_min, t_max, i, j, opt) &&
             l32::intersect_newton32(T, T32, g, O, D, t_min, t_max, i, j, opt.polish_cond, h, flags, st);
    }
    if (ok && T.inst)
        dmapdev::world_normal(opt.inst_xf + dmapdev::kInstDoubles * (T.inst - 1), h.ng);
    return ok;
}

// DisplacedIntersector::intersect with the FP32 node test.
__device__ bool triangle_walk32(const TriDev32 &T, const TriDev &T64, const AssetDev &g, const double *o,
                                const double *d, double t_min, double &t_max, const dmapk::QueryOpts &opt,
                                d64::hit64 &hit, int &hflags, int64_t *st, float t_far, unsigned *status,
                                bool &capped)
{
    Ray32 r;
    tangent_ray(T, o, d, t_far, r);
    int si = r.dx < 0.0f, sj = r.dy < 0.0f;
    float tmin_f = __double2float_rd(t_min);
    bool found = false;
    int64_t nah = 0, lah = 0;
    const Walk32 W = load_walk(T);
    for (int q = 0; q < T.n_roots; ++q) {
        Cell32 cur = {T.root_level, T.roots_i[q], T.roots_j[q]}, end = cur;
        cell_next(end, si, sj, T.root_level);
        int guard = 0;
        while (!(cur.level == end.level && cur.i == end.i && cur.j == end.j)) {
            if (++guard > opt.guard_cap) { // a finite tree: the cap guards corrupt records
                atomicOr(status, dmapdev::kStatusCapped);
                capped = true;
                break;
            }
            float w = pow2f(cur.level - W.log2n);
            if (!cell_meets_domain(W, ((float)cur.i + 0.5f) * w, ((float)cur.j + 0.5f) * w, 0.5f * w)) {
                cell_next(cur, si, sj, T.root_level);
                continue;
            }
            if (st) {
                ++st[DMAP_ST_NODE];
                ++nah;
            }
            float tmax_f = __double2float_ru(t_max);
            if (!node_test32(W, T.pyr32, r, cur.level, cur.i, cur.j, tmin_f, tmax_f, opt.bound,
                             opt.slab_max_level)) {
                cell_next(cur, si, sj, T.root_level);
                continue;
            }
            if (cur.level > 0) {
                --cur.level;
                cur.i = 2 * cur.i + si;
                cur.j = 2 * cur.j + sj;
                continue;
            }
            if (st) {
                ++st[DMAP_ST_LEAF];
                ++lah;
            }
            d64::hit64 lh;
            int lf = 0;
            if (leaf_cell(T, T64, g, o, d, t_min, t_max, cur.i, cur.j, lh, lf, st, opt) && lh.t < t_max) {
                hit = lh;
                hflags = lf;
                t_max = lh.t;
                found = true;
                nah = lah = 0;
                if (opt.mode == 1 && !opt.op_mask) // a filter judges the nearest crossing
                    return true;
            }
            cell_next(cur, si, sj, T.root_level);
        }
    }
    if (st && found) {
        st[DMAP_ST_NAH] += nah;
        st[DMAP_ST_LAH] += lah;
    }
    return found;
}

template <typename R, typename H, typename Fp>
__global__ void __launch_bounds__(128) walk32_simple(const TriDev32 *__restrict__ tris32,
                                                     const TriDev *__restrict__ tris64, int n_tri,
                                                     const AssetDev *__restrict__ assets, const R *__restrict__ rays,
                                                     int64_t n, dmapk::QueryOpts opt, H *__restrict__ hits,
                                                     int64_t *__restrict__ stats, unsigned *status,
                                                     const int *__restrict__ ray_list = nullptr,
                                                     const unsigned long long *list_n = nullptr)
{
    int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (ray_list) {
        // the rays a filtered wavefront query hands back (check_crossing)
        if ((unsigned long long)k >= *list_n)
            return;
        k = ray_list[k];
    } else if (k >= n || (opt.n_dev && k >= *opt.n_dev)) {
        return;
    }
    double o[3], d[3], t_min, t_max;
    load_ray(rays, k, o, d, t_min, t_max);
    float of[3], df[3], invf[3];
    for (int a = 0; a < 3; ++a) {
        of[a] = (float)o[a];
        df[a] = (float)d[a];
        invf[a] = df[a] != 0.0f ? __frcp_rn(df[a]) : 0.0f;
    }
    int64_t st[DMAP_ST_N] = {0, 0, 0, 0, 0, 0, 0, 0};
    int64_t *sp = stats ? st : nullptr;
    d64::hit64 best;
    int best_tri = -1, best_flags = 0;
    bool found = false, capped = false;
    // the next triangle: the smallest (key, index) past the cursor among the
    // candidates the ray still reaches, the key being the index (index
    // order) or the box entry (nearest)
    double inv[3], ckey = -INFINITY;
    int cidx = -1;
    d64::ray_inverse(d, inv);
    // scenes of more than 256 triangles: the triangle tree (bvh.cuh)
    const d32::BvhView bvh = {opt.bvh_nodes, opt.bvh_tri, opt.bvh_range, opt.bvh_n_nodes};
    d32::NearBuf nbuf;
    nbuf.n = -1;
    nbuf.pos = 0;
    for (int step = 0; step < n_tri; ++step) {
        int t = step;
        float t1 = __double2float_ru(t_max);
        if (bvh.nodes) {
            bool err = false;
            const float tmin_f = __double2float_rd(t_min);
            t = opt.order == 1 ? d32::near_next<true>(nbuf, bvh, tris32, tris64, o, d, inv, t_min, of, df, invf,
                                                      tmin_f, t1, ckey, cidx, t1, err)
                               : d32::near_next<false>(nbuf, bvh, tris32, tris64, o, d, inv, t_min, of, df, invf,
                                                       tmin_f, t1, ckey, cidx, t1, err);
            if (err)
                atomicOr(status, dmapdev::kStatusCapped);
            if (t < 0)
                break;
        } else if (opt.order == 1) {
            const float tmf = t1;
            double bk = 0.0;
            int bt = -1;
            for (int q = 0; q < n_tri; ++q) {
                const double key = d64::entry_key(tris64[q], o, d, inv, t_min);
                if (!d64::after_cursor(key, q, ckey, cidx) || !d64::before_best(key, q, bk, bt))
                    continue;
                float tt = tmf;
                if (!object_box(tris32[q], of, df, invf, __double2float_rd(t_min), tt))
                    continue;
                bk = key;
                bt = q;
                t1 = tt;
            }
            if (bt < 0)
                break;
            t = bt;
            ckey = bk;
            cidx = bt;
        } else if (!object_box(tris32[t], of, df, invf, __double2float_rd(t_min), t1)) {
            continue;
        }
        const TriDev32 &T = tris32[t];
        if (sp)
            ++st[DMAP_ST_TRI];
        d64::hit64 h;
        int hf = 0;
        bool got = false;
        // the callbacks' filter passes (displaced_geometry.cpp:53-106); no filter: one walk
        double t_lo = t_min;
        for (int pass = 0; pass < (opt.op_mask ? dmapdev::kFilterPasses : 1); ++pass) {
            double tm = t_max;
            if (!triangle_walk32(T, tris64[t], assets[T.asset], o, d, t_lo, tm, opt, h, hf, sp, far_bound(t1), status,
                                 capped))
                break;
            if (dmapdev::crossing_opaque(opt, tris64[t], t, h.bary.x, h.bary.y)) {
                got = true;
                break;
            }
            t_lo = h.t;
        }
        if (got) {
            best = h;
            best_flags = hf;
            best_tri = t;
            t_max = h.t;
            found = true;
            if (opt.mode == 1)
                break;
        }
    }
    store_hit<H, Fp>(hits, k, found, best, best_tri, (found ? best_flags : 0) | (capped ? DMAP_HIT_CAPPED : 0));
    if (stats)
        for (int q = 0; q < DMAP_ST_N; ++q)
            stats[DMAP_ST_N * k + q] = st[q];
}

// ---- wavefront schedule ---------------------------------------------------------

// One bit per cell of a stackless walk's open sibling groups: child k of the
// group at level l (k counts the siblings in the ray's visiting order) is bit
// 4 l + k, so the lowest bit is the next cell of the depth-first order. The
// walk has one open group per level, and the roots are the group of the root
// level. 64 bits hold root levels up to 15; scenes with a higher one (repeat
// charts over many tiles, maps beyond 32768 texels) take DEEP, up to 31.
template <bool DEEP>
struct CellBits
{
    unsigned long long lo, hi;
    __device__ __forceinline__ bool any() const { return DEEP ? (lo | hi) != 0ull : lo != 0ull; }
    __device__ __forceinline__ int first() const
    {
        return !DEEP || lo ? __ffsll((long long)lo) - 1 : 63 + __ffsll((long long)hi);
    }
    __device__ __forceinline__ unsigned group(int l) const
    {
        return (unsigned)((!DEEP || l < 16 ? lo : hi) >> (4 * (l & 15))) & 15u;
    }
    __device__ __forceinline__ void set_group(int l, unsigned nib)
    {
        const int sh = 4 * (l & 15);
        if (!DEEP || l < 16)
            lo = (lo & ~(15ull << sh)) | ((unsigned long long)nib << sh);
        else
            hi = (hi & ~(15ull << sh)) | ((unsigned long long)nib << sh);
    }
    // bits 0 .. p of a word (p = 63: all)
    static __device__ __forceinline__ unsigned long long upto(int p) { return (2ull << p) - 1ull; }
    __device__ __forceinline__ void clear_bit(int p)
    {
        if (!DEEP || p < 64)
            lo &= ~(1ull << (p & 63));
        else
            hi &= ~(1ull << (p & 63));
    }
    __device__ __forceinline__ void clear_upto(int p)
    {
        if (!DEEP || p < 64) {
            lo &= ~upto(p & 63);
        } else {
            lo = 0ull;
            hi &= ~upto(p & 63);
        }
    }
    __device__ __forceinline__ int count_upto(int p) const
    {
        if (!DEEP || p < 64)
            return __popcll(lo & upto(p & 63));
        return __popcll(lo) + __popcll(hi & upto(p & 63));
    }
    __device__ __forceinline__ int count() const { return DEEP ? __popcll(lo) + __popcll(hi) : __popcll(lo); }
    __device__ __forceinline__ bool has(int p) const
    {
        return (((!DEEP || p < 64 ? lo : hi) >> (p & 63)) & 1ull) != 0ull;
    }
};

// The cells of the open groups that come after cell (l, i, j) in walk order:
// its later siblings and those of the cells above it. The walk counts a
// group's cells when it tests them, all at once; less those still ahead this
// is what the one-cell walk has visited, which opt.guard_cap bounds. Called
// out of line it cost the walk 1% (14.06 -> 14.18 ms at 2.80M rays).
__device__ __forceinline__ int cells_ahead(const TriDev32 &T, int l, int i, int j, int si, int sj)
{
    const int up = T.root_level - l, m = (int)((1u << up) - 1u);
    int k = 0;
    while (k + 1 < T.n_roots && (T.roots_i[k] != i >> up || T.roots_j[k] != j >> up))
        ++k;
    return T.n_roots - 1 - k + 3 * up - 2 * __popc((i ^ -si) & m) - __popc((j ^ -sj) & m);
}

// A parked walk: the ray's position in ObjectIntersector's triangle loop and
// in DisplacedIntersector's walk (the cell last taken and the open groups'
// bits), its current t_max and result, its candidate mask and the counters
// of the triangle in progress.
struct RayState
{
    double t_max;
    double ckey; // triangle tree, nearest first: the cursor (key, index) of the last triangle taken
    int cidx;
    int tri, best_tri, flags;
    int cl, ci, cj;
    int nah, lah, pad;
    unsigned long long todo[2], dom[2];
    union {
        unsigned long long mask[4]; // per lane of the ray's four
        // scenes of more than 256 triangles: the buffered candidates, kept
        // across parks so a resumed ray does not walk the tree again
        d32::NearBuf buf;
    };
};
// Up to kCollect consecutive leaves of one triangle's walk, in walk order.
// The walk goes on past a leaf with the t_max it has (it cannot know the
// leaf's result yet), so it may also reach leaves the reference prunes with
// the smaller t_max of a hit; the leaf kernel runs them with that smaller
// t_max, where they cannot report a nearer root than the one found, so the
// ray's hit is unchanged.
constexpr int kCollect = 4; // leaf slots of a job
// Leaves a ray collects before it parks (at most kCollect).
#ifndef DMAP_COLLECT
#define DMAP_COLLECT 4
#endif
static_assert(DMAP_COLLECT >= 1 && DMAP_COLLECT <= kCollect, "leaf slots");
struct LeafJob
{
    int ray, tri, n;
    int keep; // the cells the FP64 node test admits, a bit each (wave_filter)
    int i[kCollect], j[kCollect];
};
// RayState.flags
constexpr int kFoundInTri = 1; // a hit was taken in the triangle in progress
constexpr int kShrunk = 2;     // the leaves of the last job shrank t_max: the cells still open are tested again
constexpr int kExpand = 16;   // parked with the last cell taken still to expand
constexpr int kCapped = 4;     // a triangle walk of this ray ran out of its cell-visit cap (DMAP_HIT_CAPPED)
constexpr int kRerun = 8;      // listed for the filter's schedule (it took a crossing the filter rejects)

// A filtered scene's wavefront query commits crossings as it finds them,
// without the filter's passes. A ray whose every committed crossing the
// filter accepts has the answer the passes give (each triangle's first pass
// finds the crossing it committed, with the same t_max); a ray that took a
// crossing the filter rejects is listed once, and the filter's own schedule
// (walk32_simple) answers it again after the query.
__device__ __forceinline__ void check_crossing(const dmapk::QueryOpts &opt, const TriDev &T, int tri,
                                               const d64::hit64 &h, int ray, int &flags, unsigned long long *ctr,
                                               int *rerun)
{
    if (!opt.op_mask || (flags & kRerun) || dmapdev::crossing_opaque(opt, T, tri, h.bary.x, h.bary.y))
        return;
    flags |= kRerun;
    rerun[atomicAdd(ctr + 4 * (dmapk::kMaxRounds + 1), 1ull)] = ray;
}

// Counter slots of one round: the walk's fetch counter, the leaf queue's
// length, the leaf kernel's fetch counter, the resume queue's length.
__device__ __forceinline__ unsigned long long *round_ctr(unsigned long long *c, int round, int k)
{
    return c + 4 * round + k;
}

// Ray k as triangle T meets it: in the object space of an instanced one
// (instance.cuh). One copy of its code for the leaf kernels.
__device__ __noinline__ void leaf_ray(const void *rays, int ray_dtype, int64_t k, const double *inst_xf, int inst,
                                      d64::v3 &O, d64::v3 &D, double &t_min, double &t_max)
{
    double o[3], d[3], oo[3], od[3];
    load_ray(rays, ray_dtype, k, o, d, t_min, t_max);
    dmapdev::ray_for(inst_xf, inst, o, d, oo, od);
    O = d64::V3(oo[0], oo[1], oo[2]);
    D = d64::V3(od[0], od[1], od[2]);
}

// A leaf cell the last walk reached, by the four lanes of its ray's quad: the
// cell's FP64 node test, then the certified leaf in the query's precision.
// A nearer root is stored as the ray's hit; returns the ray's t_max.
template <class P, bool ST>
__device__ __noinline__ double quad_leaf(const TriDev32 &T32, const TriDev &T, const AssetDev *assets, const void *rays,
                                         int ray, int tri, double t_max, int i, int j, const dmapk::QueryOpts &opt,
                                         void *hits, double *stack_mem, unsigned long long *ctr, int *rerun, int &flags,
                                         int64_t *stl)
{
    const int lane = threadIdx.x & 31;
    const lq::Quad Q = {0xfu << (lane & 28), lane & 28, lane & 3};
    const AssetDev &g = assets[T.asset];
    typename P::Ent *stack = reinterpret_cast<typename P::Ent *>(stack_mem);
    double t_min, t_ray;
    d64::v3 O, D;
    leaf_ray(rays, opt.ray_dtype, ray, opt.inst_xf, T.inst, O, D, t_min, t_ray);
    if (!d64::leaf_cell_admitted(T, g, O, D, t_min, t_max, i, j, opt))
        return t_max;
    typename P::Bound L;
    P::setup(T, g, O, D, i, j, L);
    auto ray_of = [&](d64::v3 &ro, d64::v3 &rd) {
        ro = O;
        rd = D;
    };
    // the last root taken, in the lane that took it
    lq::Found best;
    double mine = -INFINITY;
    auto on_root = [&](const lq::Found &f) {
        best = f;
        mine = f.t;
    };
    const double t_start = t_max;
    typename P::Ent e = lq::root_entry<P>();
    int sp = 0;
    int64_t subs = 0, iters = 0;
    do {
        lq::Child<P> c;
        lq::bound_children<P>(Q, e, T32, T, L, t_min, t_max, c);
        if (ST)
            subs += 4;
        if (e.depth + 1 < lq::kDepth)
            lq::push_children<P>(Q, c, e.depth + 1, stack, sp);
        else if (c.n > 0) // the leaf's nearest root, in an occlusion query too: the simple schedule's record
            lq::newton_children<P, ST>(Q, c, T, g, L, ray_of, t_min, t_max, i, j, opt.polish_cond, false, iters, on_root);
    } while (lq::pop<P>(stack, sp, t_max, e));
    if (mine == t_max && t_max < t_start) {
        d64::hit64 h;
        d64::root_record_shared(T, g, best.t, best.st, i, j, h);
        if (T.inst)
            dmapdev::world_normal(opt.inst_xf + dmapdev::kInstDoubles * (T.inst - 1), h.ng);
        store_hit(hits, opt.hit_dtype, ray, true, h, tri, best.flags | ((flags & kCapped) ? DMAP_HIT_CAPPED : 0));
        check_crossing(opt, T, tri, h, ray, flags, ctr, rerun);
    }
    __syncwarp(Q.mask);
    flags = (int)__reduce_or_sync(Q.mask, (unsigned)flags);
    if (ST) {
        iters += __shfl_xor_sync(Q.mask, iters, 1);
        iters += __shfl_xor_sync(Q.mask, iters, 2);
        stl[DMAP_ST_SUB] += subs;
        stl[DMAP_ST_NEWTON] += iters;
    }
    return t_max;
}

// A ray in work or fetched ahead, as its picks read it.
struct RaySlot
{
    double o[3], d[3], inv[3], t_min, t_max; // inv: d64::ray_inverse
    float of[3], df[3], invf[3];
    int ray;
};

// An empty slab range beyond the FP32 tolerance (box_range's test; with wide
// 2 and t_lo the range's start, node_range's).
__device__ __forceinline__ bool misses(float t0, float t1, float wide, float t_lo)
{
    return t0 > t1 + wide * tol32(fmaxf(fmaxf(fabsf(t0), fabsf(t1)), fabsf(t_lo)));
}

// The slabs of a box against a ray (d32::box_range, or with wide 2 and t_lo
// node_range), out of line: one copy of its code serves every place of the
// walk that tests a box. Component c of the box is box[c * stride]. Not ok:
// the ray misses it; t1 is the exit bound either way.
struct Span
{
    float t0, t1;
    bool ok;
};
__device__ __noinline__ Span box_span(const float *box, int stride, const RaySlot &S, float t0, float t1,
                                      float wide = 1.0f, float t_lo = 0.0f)
{
    Span r = {t0, t1, true};
#pragma unroll
    for (int c = 0; c < 3; ++c)
        r.ok = box_slab(box[c * stride], box[(3 + c) * stride], S.of[c], S.df[c], S.invf[c], r.t0, r.t1) && r.ok;
    r.ok = r.ok && !misses(r.t0, r.t1, wide, t_lo);
    return r;
}

// d64::entry_key of a box (lo, then hi), out of line.
__device__ __noinline__ double box_key(const double *lo, const RaySlot &S)
{
    double key = S.t_min;
#pragma unroll 1
    for (int a = 0; a < 3; ++a)
        if (S.d[a] != 0.0) {
            const double o = S.o[a], inv = S.inv[a];
            key = d64::dmax(key, d64::dmin((lo[a] - o) * inv, (lo[3 + a] - o) * inv));
        }
    return key;
}

// Four lanes walk one ray (a quad; eight rays per warp), so that the four
// cells of a sibling group are tested together, one per lane. A lane per ray
// ran one node test per step with 19.6 of 32 lanes in it, the others being in
// a pick or between cells; and a ray's tests, one after the other, set the
// time of small batches and of every launch's tail. Walk rounds and last walk
// before and after: 64 rays on a quad 212 -> 63 us, 20,011 rays on the sphere
// of 96 x 512^2 maps 2.80 -> 0.69 ms, 2.80M rays on 96 x 2048^2 34.1 -> 27.2
// ms.
//
// The loop's code is kept small: at 53 KB (the box test in four places, the
// park in four, the ray transform and the ray's load in two each) 2.7 of 8.6
// cycles per issued instruction were instruction fetch, at 84 KB 7.2 of 13.
// Each now stands in one place (40 KB), and rays are fetched ahead, a lane
// per ray, into shared memory: the walk rounds above take 16.4 ms from 22.5.
// Per quad and step: take
// the next cell of the open groups (its lowest bit), descend into it by
// testing its four children, or collect it when it is a leaf.
//
// The order, the tests and the leaf jobs are those of the walk that visits
// one cell at a time: t_max does not change between a group's test and the
// cells taken from it, except where a job's leaves or a leaf run inline
// shrink it, and then every group still open is tested again before a cell
// is taken from it (`stale`).
//
// The walk rounds are compiled for DMAP_WALK_MIN_BLOCKS (mask) or
// DMAP_WALK_TREE_MIN_BLOCKS (tree) CTAs per SM; the last walk (INLINE_LEAF),
// which runs the few rays left with their leaves inline, for
// DMAP_DRAIN_MIN_BLOCKS, so that the leaf it calls is not squeezed into the
// rounds' register budget.
// In a round that keeps the quads busy (32 rays and more per warp), the warp
// makes its picks when DMAP_PICK_QUADS of its quads (TREE:
// DMAP_TREE_PICK_QUADS) need one, or none has a group to test: a pick costs
// about as much as a group's test and served 1.9 quads. Over the tree, whose
// refills cost several times that, fetches wait too. 2.80M rays on 96 x
// 2048^2 maps, walk rounds at 1 / 2 / 3 / 4: 15.9 / 15.3 / 15.0 / 15.1 ms;
// 12,288 triangles 6.2 / 5.4 / 5.2 / 5.1. In the last walk a leaf waits for
// DMAP_DRAIN_QUADS: 1 / 2 / 3 / 4 / 6: 3.6 / 3.0 / 2.8 / 2.6 / 2.6 ms, and in
// index order with the FP64 leaf (100,003 rays) 3.5 / 3.0 / 2.7 / 2.6 / 2.3.
// Small rounds, where a ray's own chain sets the time, wait for nothing.
#ifndef DMAP_PICK_QUADS
#define DMAP_PICK_QUADS 3
#endif
#ifndef DMAP_TREE_PICK_QUADS
#define DMAP_TREE_PICK_QUADS 4
#endif
#ifndef DMAP_DRAIN_QUADS
#define DMAP_DRAIN_QUADS 6
#endif
#ifndef DMAP_DRAIN_MIN_BLOCKS
#define DMAP_DRAIN_MIN_BLOCKS 2
#endif
template <bool ST, bool INLINE_LEAF, bool TREE, bool NEAR, bool DEEP>
__global__ void __launch_bounds__(128, INLINE_LEAF ? DMAP_DRAIN_MIN_BLOCKS
                                                  : (TREE ? DMAP_WALK_TREE_MIN_BLOCKS : DMAP_WALK_MIN_BLOCKS))
    wave_walk(const TriDev32 *__restrict__ tris32, const TriDev *__restrict__ tris64, int n_tri,
              const AssetDev *__restrict__ assets, const void *__restrict__ rays, int64_t n, dmapk::QueryOpts opt,
              void *__restrict__ hits, int64_t *__restrict__ stats, RayState *__restrict__ states,
              const int *__restrict__ q_in, int round, LeafJob *__restrict__ q_leaf, unsigned long long *ctr,
              unsigned *status, int *__restrict__ rerun)
{
    enum : int { NEED = 0, TOP = 1, WALK = 2, DONE = 3, LEAF = 4 }; // LEAF: the last walk, at a leaf cell
    const int lane = threadIdx.x & 31, sub = lane & 3, lead = lane & 28;
    // the candidates: scenes of up to 256 triangles take a mask of one bit
    // per triangle whose box the ray meets (built by the warp at the ray's
    // start; triangle t is bit t / 4 of the quad's lane t % 4), larger scenes
    // (TREE) the triangle tree (bvh.cuh), in either order; the launcher takes
    // the mask only for up to 256 triangles, so its loops are never compiled
    // into the kernels of larger scenes
    const d32::BvhView bvh = {opt.bvh_nodes, opt.bvh_tri, opt.bvh_range, opt.bvh_n_nodes};
    // scenes of up to 256 triangles: their outward FP32 boxes in shared
    // memory, component c of triangle t at c * kStaged + t
    constexpr int kStaged = TREE ? 1 : 32 * kMaskWords;
    __shared__ float s_box32[6 * kStaged];
    if (!TREE) {
        for (int k = threadIdx.x; k < 6 * n_tri; k += blockDim.x) {
            const int t = k / 6, c = k - 6 * t;
            s_box32[c * kStaged + t] = c < 3 ? tris32[t].box_lo[c] : tris32[t].box_hi[c - 3];
        }
        __syncthreads();
    }
    // boxes around runs of 8 triangles, for the candidates' first test
    constexpr int kRuns = TREE ? 1 : 32;
    __shared__ float s_run[6 * kRuns];
    if (!TREE) {
        for (int k = threadIdx.x; k < 6 * kRuns; k += blockDim.x) {
            const int c = k >> 5, first = 8 * (k & 31);
            float v = c < 3 ? INFINITY : -INFINITY;
            for (int t = first; t < first + 8 && t < n_tri; ++t)
                v = c < 3 ? fminf(v, s_box32[c * kStaged + t]) : fmaxf(v, s_box32[c * kStaged + t]);
            s_run[k] = v;
        }
        __syncthreads();
    }
    // the box entries of a lane's candidates: of mask bit b at b * 128 + thread
    extern __shared__ float s_entry[];
    // the rays in work and those the warp has fetched ahead
    constexpr int kRaySlots = 16, kRayBatch = 8; // per warp: eight in work, eight ahead
    __shared__ RaySlot s_ray[4][kRaySlots];
    // the quads' rays in their triangles' frames: per axis origin, direction,
    // its reciprocal, widening (Ray32)
    __shared__ float4 s_frame[32][3];
    // the last walk: the leaf search's stacks, per quad
    __shared__ double s_stack[INLINE_LEAF ? 32 : 1][INLINE_LEAF ? lq::kStack * sizeof(lq::P64::Ent) / 8 : 1];
    // items of this round: every ray in round 0, else the resume queue
    unsigned long long count = round == 0 ? (unsigned long long)n : *round_ctr(ctr, round - 1, 3);
    if (round == 0 && opt.n_dev && (unsigned long long)*opt.n_dev < count)
        count = *opt.n_dev < 0 ? 0ull : (unsigned long long)*opt.n_dev;
    unsigned long long *fetch = round_ctr(ctr, round, 0);
    // a round of fewer rays than the grid has quads spreads them over all
    // its warps, so that fewer of them share a warp
    const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
    int phase = (unsigned long long)(lane >> 2) * warps < count ? NEED : DONE;
    // rays fetched at once: a fill of the warp's quads while at least two
    // fills per warp are to come, else a quarter of the warp's share, so that
    // no warp is left with several long rays (20,011 rays, 7 per warp: the
    // walk rounds take 0.43 ms, with half of the share at once 0.45; 65,536
    // rays on one quad, 22 per warp: 156 us with a fill, 171 with a quarter)
    const int batch = count >= 2ull * kRayBatch * warps ? kRayBatch : (int)max(1ull, count / (4ull * warps));
    const bool full = !INLINE_LEAF && count >= 32ull * warps;
    const int pick_quads = full ? (TREE ? DMAP_TREE_PICK_QUADS : DMAP_PICK_QUADS) : 1;
    bool more = count > 0ull; // rays may be left in the queue
    unsigned ready = 0u;      // slots with a ray no quad has taken
    const int wi = threadIdx.x >> 5;
    RaySlot *const slots = s_ray[wi];
    int slot = 0; // the quad's ray
    int ray = 0;
    double t_max = 0.0;
    float tmin_f = 0.0f, tmax_f = 0.0f;
    int tri = 0, best_tri = -1, si = 0, sj = 0, nah = 0, lah = 0, flags = 0, guard = 0;
    double ckey = -INFINITY;
    int cidx = -1;
    // the triangle tree (TREE): the buffered candidates, held by the quad's
    // first lane, refilled from the ray's cursor for a fresh ray, kept in the
    // ray's state across parks
    d32::NearBuf nbuf;
    nbuf.n = -1;
    nbuf.pos = 0;
    float4 *const frame = s_frame[threadIdx.x >> 2];
    const float *pyr = nullptr;
    Cell32 cur = {0, 0, 0};
    CellBits<DEEP> todo = {0ull, 0ull}, dom = {0ull, 0ull}; // cells that passed; cells in the domain, not yet gone past
    unsigned stale = 0u;                                   // levels whose group must be tested again
    unsigned long long mask = 0ull; // the lane's candidates
    bool entries = false;           // their box entries are in s_entry
    int64_t stl[DMAP_ST_N];
    int nl = 0, li = 0, lj = 0; // collected leaves, the lane's own
    int since = 0;              // node tests since the first collected leaf

    auto flush_stats = [&]() {
        if (ST && sub == 0)
            for (int q = 0; q < DMAP_ST_N; ++q)
                stats[DMAP_ST_N * (int64_t)ray + q] += stl[q];
    };
    // Park the ray: its collected leaves become one job, its walk state
    // waits for the next round.
    auto park = [&]() {
        RayState &s = states[ray];
        unsigned long long slot = 0;
        if (sub == 0) {
            s.t_max = t_max;
            s.tri = tri;
            s.best_tri = best_tri;
            s.flags = flags;
            s.cl = cur.level, s.ci = cur.i, s.cj = cur.j;
            s.todo[0] = todo.lo;
            s.dom[0] = dom.lo;
            if (DEEP) {
                s.todo[1] = todo.hi;
                s.dom[1] = dom.hi;
            }
            if (ST) {
                s.nah = nah;
                s.lah = lah;
            }
            if (TREE) {
                s.ckey = ckey;
                s.cidx = cidx;
                s.buf = nbuf;
            }
            slot = atomicAdd(round_ctr(ctr, round, 1), 1ull);
        }
        if (!TREE)
            s.mask[sub] = mask;
        slot = __shfl_sync(0xfu << lead, slot, lead);
        LeafJob &job = q_leaf[slot];
        if (sub == 0) {
            job.ray = ray;
            job.tri = tri;
            job.n = nl;
        }
        job.i[sub] = li;
        job.j[sub] = lj;
        nl = 0;
        since = 0;
        flush_stats();
        phase = NEED;
    };
    // the ray transform into triangle T's tangent frame, a row per lane
    auto enter_frame = [&](const TriDev32 &T, const double *o, const double *d, float t_far) {
        const unsigned quad = 0xfu << lead;
        if (sub < 3) {
            float4 f;
            tangent_row(T, sub, o, d, t_far, f.x, f.y, f.w);
            f.z = f.y != 0.0f ? __frcp_rn(f.y) : 0.0f;
            frame[sub] = f;
        }
        __syncwarp(quad);
        si = frame[0].y < 0.0f;
        sj = frame[1].y < 0.0f;
        pyr = T.pyr32;
    };

    for (;;) {
        // 1. quads without work take a ray that is ready; when none is, the
        // warp fetches the next ones of the round, a lane per ray
        bool fresh = false;
        bool enter = false;  // the quad's lanes need the ray in triangle tri's frame
        bool expand = false; // a resumed ray whose last cell's children come next
        unsigned need;
        while ((need = __ballot_sync(FULL, phase == NEED) & 0x11111111u) != 0u) {
            if (TREE && __popc(need) < pick_quads && __any_sync(FULL, phase == WALK || phase == TOP || phase == LEAF))
                break;
            if (!ready) {
                if (!more) {
                    if (phase == NEED)
                        phase = DONE;
                    break;
                }
                unsigned long long base = 0;
                if (lane == 0)
                    base = atomicAdd(fetch, (unsigned long long)batch);
                base = __shfl_sync(FULL, base, 0);
                more = base + batch < count;
                const unsigned taken = __reduce_or_sync(FULL, phase != NEED && phase != DONE ? 1u << slot : 0u);
                const bool get = lane < batch && base + lane < count;
                const int to = get ? nth_bit(~taken, lane) : 0;
                if (get) {
                    RaySlot &S = slots[to];
                    const int k = round == 0 ? (int)(base + lane) : q_in[base + lane];
                    double o[3], d[3], t0, t1;
                    load_ray(rays, opt.ray_dtype, k, o, d, t0, t1);
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        S.o[a] = o[a];
                        S.d[a] = d[a];
                        S.of[a] = (float)o[a];
                        S.df[a] = (float)d[a];
                    }
#pragma unroll 1
                    for (int a = 0; a < 3; ++a) {
                        S.inv[a] = S.d[a] != 0.0 ? 1.0 / S.d[a] : 0.0; // d64::ray_inverse
                        S.invf[a] = S.df[a] != 0.0f ? __frcp_rn(S.df[a]) : 0.0f;
                    }
                    S.t_min = t0;
                    S.t_max = t1;
                    S.ray = k;
                }
                __syncwarp();
                ready = __reduce_or_sync(FULL, get ? 1u << to : 0u);
                continue;
            }
            const int k = __popc(need & ((1u << lead) - 1u)), want = __popc(need);
            if (phase == NEED && k < __popc(ready)) {
                slot = nth_bit(ready, k);
                const RaySlot &S = slots[slot];
                ray = S.ray;
                tmin_f = __double2float_rd(S.t_min);
                nbuf.n = -1;
                entries = round == 0;
                if (ST)
                    for (int q = 0; q < DMAP_ST_N; ++q)
                        stl[q] = 0;
                if (round == 0) {
                    t_max = S.t_max;
                    tri = 0;
                    ckey = -INFINITY;
                    cidx = -1;
                    best_tri = -1;
                    flags = 0;
                    mask = 0ull;
                    tmax_f = __double2float_ru(t_max);
                    fresh = true;
                    phase = TOP;
                } else {
                    const RayState &s = states[ray];
                    t_max = s.t_max;
                    tri = s.tri;
                    best_tri = s.best_tri;
                    flags = s.flags;
                    cur = {s.cl, s.ci, s.cj};
                    todo.lo = s.todo[0];
                    dom.lo = s.dom[0];
                    if (DEEP) {
                        todo.hi = s.todo[1];
                        dom.hi = s.dom[1];
                    }
                    if (ST) {
                        nah = s.nah;
                        lah = s.lah;
                    }
                    if (TREE) {
                        ckey = s.ckey;
                        cidx = s.cidx;
                        if (sub == 0)
                            nbuf = s.buf;
                    } else {
                        mask = s.mask[sub];
                    }
                    // back into the walk just after the leaves (displaced_intersector.cpp:229)
                    tmax_f = __double2float_ru(t_max);
                    enter = true;
                    stale = (flags & kShrunk) ? ~0u : 0u;
                    expand = (flags & kExpand) != 0;
                    flags &= ~(kShrunk | kExpand);
                    nl = 0;
                    phase = WALK;
                }
            }
            ready = drop_bits(ready, want);
            __syncwarp();
        }
        // round 0: the warp finds the fresh rays' candidate triangles
        // together: the runs the ray meets, then the boxes of four runs per
        // ballot, lane 8 q + 2 i + k of a ballot triangle 4 k + q of its
        // i-th run, so that byte q is the candidates of the quad's lane q
        if (!TREE) {
            unsigned left = __ballot_sync(FULL, fresh) & 0x11111111u;
            while (left) {
                const int src = __ffs(left) - 1;
                left &= left - 1;
                const RaySlot &S = slots[__shfl_sync(FULL, slot, src)];
                const float s_tmin = __shfl_sync(FULL, tmin_f, src), s_tmax = __shfl_sync(FULL, tmax_f, src);
                unsigned runs = __ballot_sync(FULL, 8 * lane < n_tri && box_span(s_run + lane, kRuns, S, s_tmin, s_tmax,
                                                                                 2.0f, s_tmin).ok);
#pragma unroll 1
                while (runs) {
                    const int run = nth_bit(runs, (lane & 7) >> 1), b = 2 * run + (lane & 1), t = 4 * b + (lane >> 3);
                    bool ok = false;
                    if (run >= 0 && t < n_tri) {
                        const Span x = box_span(s_box32 + t, kStaged, S, s_tmin, s_tmax);
                        ok = x.ok;
                        if (ok)
                            s_entry[b * 128 + (threadIdx.x & ~31) + src + (lane >> 3)] = x.t0;
                    }
                    const unsigned bits = __ballot_sync(FULL, ok);
                    const unsigned own = lead == src ? (bits >> (8 * sub)) & 255u : 0u;
#pragma unroll 1
                    for (int i = 0; i < 8 && runs; i += 2, runs &= runs - 1u)
                        mask |= (unsigned long long)((own >> i) & 3u) << (2 * (__ffs((int)runs) - 1));
                }
            }
            __syncwarp();
        }
        if (__all_sync(FULL, phase == DONE))
            break;

        // 2. the next triangle whose object box the ray meets (intersect_flat's loop)
        float t1 = tmax_f; // the exit bound of the triangle's box
        bool test = false, roots = false, again = false; // a group to test: the roots; one tested before
        const unsigned top = __ballot_sync(FULL, phase == TOP) & 0x11111111u;
        const bool pick = __popc(top) >= pick_quads || !__any_sync(FULL, phase == WALK);
        if (phase == TOP && pick) {
            const unsigned quad = 0xfu << lead;
            const RaySlot &S = slots[slot];
            const double *o = S.o, *d = S.d, *inv = S.inv;
            const float *of = S.of, *df = S.df, *invf = S.invf;
            const double t_min = S.t_min;
            int bt = -1;
            if (TREE) {
                if (sub == 0) {
                    bool err = false;
                    if (NEAR) {
                        bt = d32::near_next<true>(nbuf, bvh, tris32, tris64, o, d, inv, t_min, of, df, invf, tmin_f,
                                                  tmax_f, ckey, cidx, t1, err);
                    } else {
                        // index order: the smallest index from tri on whose
                        // box the ray still meets
                        double ck = tri - 1;
                        int ci = tri - 1;
                        bt = d32::near_next<false>(nbuf, bvh, tris32, tris64, o, d, nullptr, t_min, of, df, invf,
                                                   tmin_f, tmax_f, ck, ci, t1, err);
                    }
                    if (err)
                        atomicOr(status, dmapdev::kStatusCapped);
                }
                bt = __shfl_sync(quad, bt, lead);
                t1 = __shfl_sync(quad, t1, lead);
                ckey = __shfl_sync(quad, ckey, lead);
                cidx = __shfl_sync(quad, cidx, lead);
            } else {
                // the entries of a resumed ray's candidates; those whose box
                // no longer passes are dropped for good (t_max only shrinks)
                if (!entries) {
#pragma unroll 1
                    for (unsigned long long m = mask; m; m &= m - 1ull) {
                        const int b = __ffsll((long long)m) - 1;
                        const Span x = box_span(s_box32 + 4 * b + sub, kStaged, S, tmin_f, tmax_f);
                        s_entry[b * 128 + threadIdx.x] = x.t0;
                        if (!x.ok)
                            mask &= ~(1ull << b);
                    }
                    entries = true;
                }
#pragma unroll 1
                for (;;) {
                    // the quad's first candidate: in the nearest order the
                    // smallest box entry, a lower bound of its key; in the
                    // index order the smallest index
                    float be = INFINITY;
                    bt = -1;
#pragma unroll 1
                    for (unsigned long long m = mask; m; m &= m - 1ull) {
                        const int b = __ffsll((long long)m) - 1;
                        const float e = s_entry[b * 128 + threadIdx.x];
                        if (e >= 0.0f && tmax_f >= 0.0f && e > tmax_f + tol32(fmaxf(e, tmax_f)))
                            mask &= ~(1ull << b); // past t_max
                        else if (bt < 0 || (NEAR && e < be)) {
                            be = e;
                            bt = 4 * b + sub;
                        }
                    }
                    __syncwarp(quad);
#pragma unroll 1
                    for (int x = 1; x < 4; x <<= 1) {
                        const int ot = __shfl_xor_sync(quad, bt, x);
                        const float oe = __shfl_xor_sync(quad, be, x);
                        if (ot >= 0 && (bt < 0 || (NEAR && oe < be) || ((!NEAR || oe == be) && ot < bt))) {
                            be = oe;
                            bt = ot;
                        }
                    }
                    if (bt < 0)
                        break;
                    // it leaves the candidates, and is the next triangle if
                    // its box passes with the current t_max
                    const int first = bt;
                    if ((bt & 3) == sub)
                        mask &= ~(1ull << (bt >> 2));
                    const Span x = box_span(s_box32 + bt, kStaged, S, tmin_f, tmax_f);
                    t1 = x.t1;
                    if (!x.ok)
                        continue;
                    if (!NEAR)
                        break;
                    // another candidate comes before it only if its entry is
                    // not past this one's key: then their keys decide
                    double bk = box_key(tris64[bt].box_lo, S);
                    const double fk = bk;
#pragma unroll 1
                    for (unsigned long long m = mask; m; m &= m - 1ull) {
                        const int b = __ffsll((long long)m) - 1, t = 4 * b + sub;
                        if ((double)s_entry[b * 128 + threadIdx.x] > fk)
                            continue;
                        const Span y = box_span(s_box32 + t, kStaged, S, tmin_f, tmax_f);
                        const double k = box_key(tris64[t].box_lo, S);
                        if (y.ok && d64::before_best(k, t, bk, bt)) {
                            bk = k;
                            bt = t;
                            t1 = y.t1;
                        }
                    }
                    __syncwarp(quad);
                    if (__any_sync(quad, bt != first)) {
#pragma unroll 1
                        for (int q = 1; q < 4; q <<= 1) {
                            const int ot = __shfl_xor_sync(quad, bt, q);
                            const float o1 = __shfl_xor_sync(quad, t1, q);
                            const double ok = __shfl_xor_sync(quad, bk, q);
                            if (d64::before_best(ok, ot, bk, bt)) {
                                bk = ok;
                                bt = ot;
                                t1 = o1;
                            }
                        }
                        // the taken one leaves, the first one stays
                        if ((first & 3) == sub)
                            mask |= 1ull << (first >> 2);
                        if ((bt & 3) == sub)
                            mask &= ~(1ull << (bt >> 2));
                    }
                    break;
                }
            }
            if (bt < 0) {
                if (sub == 0) {
                    if (best_tri < 0) {
                        d64::hit64 none;
                        store_hit(hits, opt.hit_dtype, ray, false, none, -1, (flags & kCapped) ? DMAP_HIT_CAPPED : 0);
                    } else if (flags & kCapped) {
                        // the stored hit is final: this quad owns the ray
                        if (opt.hit_dtype == 2)
                            static_cast<dmapdev::Hit64 *>(hits)[ray].flags |= DMAP_HIT_CAPPED;
                        else
                            static_cast<dmapdev::Hit32 *>(hits)[ray].flags |= DMAP_HIT_CAPPED;
                    }
                }
                flush_stats();
                phase = NEED;
            } else {
                tri = bt;
                enter = true;
                todo = {0ull, 0ull};
                dom = {0ull, 0ull};
                stale = 0u;
                guard = 0;
                flags &= ~kFoundInTri;
                nah = lah = 0;
                if (ST)
                    ++stl[DMAP_ST_TRI];
                phase = WALK;
                test = roots = true;
            }
        }
        if (enter) {
            const TriDev32 &T = tris32[tri];
            if (!test) {
                // a resumed ray: the exit bound with the current t_max
                const Span x = box_span(T.box_lo, 1, slots[slot], tmin_f, tmax_f);
                t1 = fmaxf(x.t1, tmin_f);
            }
            enter_frame(T, slots[slot].o, slots[slot].d, far_bound(t1));
            if (!test)
                guard = cells_ahead(T, cur.level, cur.i, cur.j, si, sj);
        }
        __syncwarp();

        // 3a. the next cell of the open groups: a leaf is collected, another
        // cell's children are the group to test
        int tl = 0, pi = 0, pj = 0; // the group: its level, its parent cell
        unsigned cells = 15u;
        if (phase == WALK) {
            const int root_level = tris32[tri].root_level;
            if (roots) {
                tl = root_level;
                cells = (1u << tris32[tri].n_roots) - 1u;
                if (DEEP && tl > 31) { // beyond the bits of the open groups
                    atomicOr(status, dmapdev::kStatusCapped);
                    flags |= kCapped;
                    ++tri;
                    phase = TOP;
                    test = false;
                }
            }
            if (expand) {
                tl = cur.level - 1;
                pi = cur.i;
                pj = cur.j;
                test = true;
            }
            bool parking = false;
            while (!test && phase == WALK && !parking) {
                if (!todo.any()) {
                    // the end of the triangle's walk
                    if (guard > opt.guard_cap) { // a finite tree: the cap guards corrupt records
                        atomicOr(status, dmapdev::kStatusCapped);
                        flags |= kCapped;
                    }
                    if (ST) {
                        // with leaves collected, at most the tests before a park
                        int left = dom.count();
                        if (nl > 0 && since + left > DMAP_STALE_CAP)
                            left = DMAP_STALE_CAP + 1 - since;
                        stl[DMAP_ST_NODE] += left;
                        nah += left;
                        for (; left > 0; --left)
                            dom.clear_bit(dom.first());
                    } else {
                        dom = {0ull, 0ull};
                    }
                    if (!INLINE_LEAF && nl > 0) {
                        // the collected leaves decide this triangle's t_max before the next one
                        parking = true;
                    } else {
                        if (ST && (flags & kFoundInTri)) {
                            stl[DMAP_ST_NAH] += nah;
                            stl[DMAP_ST_LAH] += lah;
                        }
                        ++tri;
                        phase = TOP;
                    }
                    break;
                }
                const int p = todo.first(), l = p >> 2, k = p & 3, sh = l + 1 - cur.level;
                const bool at_root = l == root_level;
                pi = at_root ? 0 : cur.i >> sh;
                pj = at_root ? 0 : cur.j >> sh;
                if ((stale >> l) & 1u) {
                    // its group was tested with a t_max that has shrunk since
                    tl = l;
                    cells = todo.group(l);
                    roots = at_root;
                    test = again = true;
                    break;
                }
                // the tests the one-cell walk makes from the last cell taken
                // to this one: the cells in the domain between them that
                // failed, and this one (unless it was counted before a park)
                const int n_in = dom.count_upto(p);
                if (!INLINE_LEAF && nl > 0) {
                    const int before = n_in - (dom.has(p) ? 1 : 0);
                    if (since + before > DMAP_STALE_CAP) {
                        // the ray holds collected leaves and walked on for
                        // DMAP_STALE_CAP tests with the t_max it had before
                        // them: park, so that they can shrink it
                        if (ST) {
                            for (int q = DMAP_STALE_CAP + 1 - since; q > 0; --q) {
                                dom.clear_bit(dom.first());
                                ++stl[DMAP_ST_NODE];
                                ++nah;
                            }
                        }
                        parking = true;
                        break;
                    }
                    since += n_in;
                }
                if (ST) {
                    stl[DMAP_ST_NODE] += n_in;
                    nah += n_in;
                }
                dom.clear_upto(p);
                todo.clear_bit(p);
                const TriDev32 &T = tris32[tri];
                cur.level = l;
                cur.i = at_root ? T.roots_i[k] : 2 * pi + ((k >> 1) ^ si);
                cur.j = at_root ? T.roots_j[k] : 2 * pj + ((k & 1) ^ sj);
                if (guard > opt.guard_cap &&
                    guard - cells_ahead(T, cur.level, cur.i, cur.j, si, sj) > opt.guard_cap) {
                    todo = {0ull, 0ull}; // gives up before this cell
                    dom = {0ull, 0ull};
                    continue;
                }
                if (l > 0) {
                    tl = l - 1;
                    pi = cur.i;
                    pj = cur.j;
                    test = true;
                    if (!INLINE_LEAF && nl > 0 && since > DMAP_STALE_CAP) {
                        flags |= kExpand; // its children are tested after the resume
                        parking = true;
                        test = false;
                    }
                    break;
                }
                if (ST) {
                    ++stl[DMAP_ST_LEAF];
                    ++lah;
                }
                if (INLINE_LEAF) {
                    phase = LEAF;
                    break;
                }
                // collect the leaf; park once DMAP_COLLECT are held
                if (sub == nl) {
                    li = cur.i;
                    lj = cur.j;
                }
                if (nl == 0)
                    since = 1;
                if (++nl == DMAP_COLLECT || since > DMAP_STALE_CAP)
                    parking = true;
            }
            if (!INLINE_LEAF && parking)
                park();
        }
        __syncwarp();

        if (INLINE_LEAF) {
            // the last round: the few remaining rays finish here. A leaf
            // waits until DMAP_DRAIN_QUADS quads of the warp have one, or no
            // other has anything else to do.
            const int wait = __popc(__ballot_sync(FULL, phase == LEAF) & 0x11111111u);
            const bool others = __any_sync(FULL, phase == TOP || phase == WALK);
            if (phase == LEAF && (wait >= DMAP_DRAIN_QUADS || !others)) {
                phase = WALK;
                const double t_old = t_max;
                t_max = opt.leaf_precision == 1
                            ? quad_leaf<lq::P32, ST>(tris32[tri], tris64[tri], assets, rays, ray, tri, t_max, cur.i, cur.j,
                                                     opt, hits, s_stack[threadIdx.x >> 2], ctr, rerun, flags, stl)
                            : quad_leaf<lq::P64, ST>(tris32[tri], tris64[tri], assets, rays, ray, tri, t_max, cur.i, cur.j,
                                                     opt, hits, s_stack[threadIdx.x >> 2], ctr, rerun, flags, stl);
                if (t_max < t_old) {
                    tmax_f = __double2float_ru(t_max);
                    best_tri = tri;
                    flags |= kFoundInTri;
                    nah = lah = 0;
                    stale = ~0u;
                    if (opt.mode == 1) {
                        flush_stats();
                        phase = NEED;
                    }
                }
            }
            __syncwarp();
        }

        // 3b. the group's cells, one per lane, all quads together
        bool in = false, pass = false;
        if (test && ((cells >> sub) & 1u)) {
            const TriDev32 &T = tris32[tri];
            const Walk32 W = load_walk(T);
            const int ci = roots ? T.roots_i[sub] : 2 * pi + ((sub >> 1) ^ si);
            const int cj = roots ? T.roots_j[sub] : 2 * pj + ((sub & 1) ^ sj);
            const float w = pow2f(tl - W.log2n);
            in = cell_meets_domain(W, ((float)ci + 0.5f) * w, ((float)cj + 0.5f) * w, 0.5f * w);
            const float4 fx = frame[0], fy = frame[1], fz = frame[2];
            const Ray32 r = {fx.x, fy.x, fz.x, fx.y, fy.y, fz.y, fx.z, fy.z, fz.z, fx.w, fy.w, fz.w};
            if (in)
                pass = node_test32(W, pyr, r, tl, ci, cj, tmin_f, tmax_f, opt.bound, opt.slab_max_level);
        }
        const unsigned b_in = __ballot_sync(FULL, in), b_pass = __ballot_sync(FULL, pass);
        if (test) {
            todo.set_group(tl, (b_pass >> lead) & 15u);
            stale &= ~(1u << tl);
            if (!again) {
                dom.set_group(tl, (b_in >> lead) & 15u);
                if (roots)
                    cur = {tl + 1, 0, 0};
                guard += __popc(cells);
            }
        }
    }
}

// The parked leaves of a round, a quad per job: the cells the filter kept are
// searched in walk order, all four lanes together (leaf_quad.cuh), one entry
// per step, quads at the same kind of step side by side. A ray whose walk has
// cells left goes back to the resume queue.
//
// The leaf setups (some 800 double operations each) are made by the warp for
// up to sixteen jobs at a time, a lane per cell, ahead of the quads that take
// them: shared memory holds the setups of the cells in work and of those made
// ready, up to 32 a warp, and the search reads them there (in registers they
// spilled). Newton runs wait until DMAP_NEWTON_QUADS of a warp's quads have
// some, and the hit records of the roots found (some 200 double operations
// behind two chains of loads) until the warp has a batch of them. Each quad
// making its own setups and records as they came, with one or two of the
// warp's lanes in it, spent most of the kernel there. Leaf rounds of 2.80M
// rays on the sphere of 96 x 2048^2 maps: a lane per job 9.1 ms, quads 19.7,
// with setups of eight jobs at a time 15.1, batched Newton runs and records
// 10.0, setups in shared memory 8.1, less code around the ray's load 7.0,
// setups of sixteen jobs and 32 records at a time 5.8; of 20,011 rays on
// 512^2 maps 0.72 -> 0.27 ms. The kernel issues in a quarter of its cycles at
// 3 warps per scheduler; instruction fetch and loads hold it up about alike.
// Resident CTAs per SM the leaf kernels are compiled for: 6 for the FP32 leaf
// (168 registers; 5, 7 and 8 are 1-12% slower), 4 for the FP64 leaf.
#ifndef DMAP_LEAF32_MIN_BLOCKS
#define DMAP_LEAF32_MIN_BLOCKS 6
#endif
#ifndef DMAP_LEAF_MIN_BLOCKS
#define DMAP_LEAF_MIN_BLOCKS 4
#endif
// Quads of a warp with Newton runs waiting before the warp makes them (1M
// shadow rays, leaf rounds at 4 / 5 / 6 / 7: 4.05 / 3.96 / 3.89 / 3.90 ms).
#ifndef DMAP_NEWTON_QUADS
#define DMAP_NEWTON_QUADS 6
#endif
constexpr int kLeafThreads = 64;
constexpr int kLeafBlocks = DMAP_LEAF32_MIN_BLOCKS;
template <bool ST, class P>
__global__ void __launch_bounds__(kLeafThreads,
                                  sizeof(typename P::Real) == 4 ? DMAP_LEAF32_MIN_BLOCKS : DMAP_LEAF_MIN_BLOCKS)
    wave_leaf(const TriDev32 *__restrict__ tris32, const TriDev *__restrict__ tris64,
              const AssetDev *__restrict__ assets, const void *__restrict__ rays, dmapk::QueryOpts opt,
              void *__restrict__ hits, int64_t *__restrict__ stats, RayState *__restrict__ states,
              const LeafJob *__restrict__ q_leaf, int round, int *__restrict__ q_out, unsigned long long *ctr,
              int *__restrict__ rerun)
{
    using namespace d64;
    typedef typename P::Ent Ent;
    typedef typename P::Bound Bound;
    enum : int { NEED = 0, SEARCH = 1, NEWTON = 2, DONE = 3 };
    constexpr int kSlots = 32; // jobs per warp, in work or ready
    constexpr int kBatch = 16; // jobs fetched at once
    constexpr int kRecs = 32;  // leaf setups per warp
    constexpr int kReps = 32;  // hit records per warp still to be made
    __shared__ Bound s_rec[kLeafThreads / 32][kRecs];
    struct Slot { double t_min; int ray, tri, keep, i[kCollect], j[kCollect]; unsigned char rec[kCollect]; };
    __shared__ Slot s_job[kLeafThreads / 32][kSlots];
    __shared__ Ent s_stack[kLeafThreads / 4][lq::kStack];
    // the root each quad's job holds, and the roots of finished jobs whose
    // records are still to be made
    struct Rep { double t, s, v; int ray, tri, i, j, flags, pad; };
    __shared__ Rep s_best[kLeafThreads / 4], s_rep[kLeafThreads / 32][kReps];
    const int lane = threadIdx.x & 31, wi = threadIdx.x >> 5, qi = threadIdx.x >> 2;
    const lq::Quad Q = {0xfu << (lane & 28), lane & 28, lane & 3};
    const unsigned long long count = *round_ctr(ctr, round, 1);
    unsigned long long *fetch = round_ctr(ctr, round, 2);
    // as the walk: a round of few jobs spreads them over all warps
    const unsigned long long warps = (unsigned long long)gridDim.x * (kLeafThreads / 32);
    const int share = (int)min(64ull, (count + warps - 1ull) / warps);
    const int batch = share >= 4 * kBatch ? kBatch : min(8, share); // 16 of a long queue, which leaves no lane idle
    int phase = (lane >> 2) < share ? NEED : DONE;
    unsigned long long next = 0, last = 0; // items of the queue this warp holds and has not set up
    bool more = batch > 0;                 // items may be left in the queue
    unsigned ready = 0u;                   // slots with a job set up and not yet taken
    unsigned recs = 0u;                    // setups in use
    int slot = 0, rec = -1;                // the quad's job, the setup of its cell
    int ray = 0, tri = 0, ci = 0, cj = 0, sp = 0;
    unsigned keep = 0u; // the job's cells not yet searched
    bool answered = false, found = false;
    int n_rep = 0;
    double t_min = 0.0, t_max = 0.0;
    lq::Child<P> c;
    c.pass = false;
    c.n = 0;
    int64_t subs = 0, iters = 0;

    // the job's ray, in its triangle's space
    auto ray_of = [&](v3 &O, v3 &D) {
        double t0, t1;
        leaf_ray(rays, opt.ray_dtype, ray, opt.inst_xf, tris64[tri].inst, O, D, t0, t1);
    };
    // the records of the roots found, a lane per root
    auto report = [&]() {
        __syncwarp();
        if (lane < n_rep) {
            const Rep &r = s_rep[wi][lane];
            const TriDev &T = tris64[r.tri];
            hit64 h;
            root_record_shared(T, assets[T.asset], r.t, V2(r.s, r.v), r.i, r.j, h);
            if (T.inst)
                dmapdev::world_normal(opt.inst_xf + dmapdev::kInstDoubles * (T.inst - 1), h.ng);
            RayState &s = states[r.ray];
            store_hit(hits, opt.hit_dtype, r.ray, true, h, r.tri, r.flags | ((s.flags & kCapped) ? DMAP_HIT_CAPPED : 0));
            check_crossing(opt, T, r.tri, h, r.ray, s.flags, ctr, rerun);
        }
        n_rep = 0;
        __syncwarp();
    };

    for (;;) {
        // quads without a job take one that is ready; when none is, the warp
        // sets up the next ones of the queue
        unsigned need;
        while ((need = __ballot_sync(FULL, phase == NEED) & 0x11111111u) != 0u) {
            if (ready) {
                const int k = __popc(need & ((1u << Q.lead) - 1u)), have = __popc(ready), want = __popc(need);
                if (phase == NEED && k < have) {
                    slot = nth_bit(ready, k);
                    const Slot &J = s_job[wi][slot];
                    ray = J.ray;
                    tri = J.tri;
                    keep = (unsigned)J.keep;
                    t_min = J.t_min;
                    t_max = states[ray].t_max;
                    sp = 0;
                    subs = iters = 0;
                    answered = found = false;
                    phase = SEARCH;
                }
                ready = drop_bits(ready, want);
                __syncwarp();
                continue;
            }
            if (next == last) {
                if (!more) {
                    if (phase == NEED)
                        phase = DONE;
                    break;
                }
                if (lane == 0)
                    next = atomicAdd(fetch, (unsigned long long)batch);
                next = __shfl_sync(FULL, next, 0);
                last = min(next + batch, count);
                more = last < count;
                if (next >= last) {
                    next = last = 0;
                    continue;
                }
            }
            // the next jobs whose cells the free setups hold, a lane per job
            const unsigned long long item = next + lane;
            const bool here = lane < kBatch && item < last;
            unsigned cells = 0u;
            int jr = 0, jt = 0;
            if (here) {
                const LeafJob &J = q_leaf[item];
                cells = (unsigned)J.keep;
                jr = J.ray;
                jt = J.tri;
            }
            int upto = __popc(cells); // cells of the jobs up to this one
#pragma unroll 1
            for (int x = 1; x < kBatch; x <<= 1) {
                const int below = __shfl_up_sync(FULL, upto, x);
                upto += lane >= x ? below : 0;
            }
            const bool fits = here && upto <= kRecs - __popc(recs);
            const unsigned took = __ballot_sync(FULL, fits);
            if (!took)
                break; // the jobs in work hold them
            // the slots no quad's job is in
            const unsigned taken = __reduce_or_sync(FULL, phase == SEARCH || phase == NEWTON ? 1u << slot : 0u);
            const int to = nth_bit(~taken, lane & (kBatch - 1));
            if (fits) {
                Slot &S = s_job[wi][to];
                S.ray = jr;
                S.tri = jt;
                S.keep = (int)cells;
                if (!cells) // the filter rejected every cell of the job: the walk goes on
                    q_out[atomicAdd(round_ctr(ctr, round, 3), 1ull)] = jr;
            }
            // their setups, a lane per cell: the job whose cells reach past the lane
            int job = 0;
#pragma unroll 1
            for (int x = kBatch / 2; x > 0; x >>= 1)
                job += __shfl_sync(FULL, upto, job + x - 1) <= lane ? x : 0;
            const int total = __shfl_sync(FULL, upto, __popc(took) - 1);
            const unsigned jc = __shfl_sync(FULL, cells, job);
            const int q = nth_bit(jc, lane - (__shfl_sync(FULL, upto, job) - __popc(jc)));
            const int cs = __shfl_sync(FULL, to, job), cr = __shfl_sync(FULL, jr, job), ct = __shfl_sync(FULL, jt, job);
            unsigned mine = 0u;
            if (lane < total) {
                Slot &S = s_job[wi][cs];
                const LeafJob &J = q_leaf[next + job];
                const int li = J.i[q], lj = J.j[q], at = nth_bit(~recs, lane);
                S.i[q] = li;
                S.j[q] = lj;
                S.rec[q] = (unsigned char)at;
                mine = 1u << at;
                double t0, t1;
                v3 O, D;
                const TriDev &T = tris64[ct];
                leaf_ray(rays, opt.ray_dtype, cr, opt.inst_xf, T.inst, O, D, t0, t1);
                S.t_min = t0; // the same from every lane of the job
                P::setup(T, assets[T.asset], O, D, li, lj, s_rec[wi][at]);
            }
            next += __popc(took);
            __syncwarp();
            recs |= __reduce_or_sync(FULL, mine);
            ready = __reduce_or_sync(FULL, fits && cells ? 1u << to : 0u);
        }
        if (__all_sync(FULL, phase == DONE))
            break;
        // the next entry of the search, the next cell's root, or the job is done
        bool have = false;
        unsigned done = 0u;
        Ent e = lq::root_entry<P>();
        if (phase == SEARCH) {
            have = lq::pop<P>(s_stack[qi], sp, t_max, e);
            if (!have && rec >= 0) {
                done = 1u << rec; // the cell's setup is free again
                rec = -1;
            }
            if (answered) // the cells left are not searched
                for (; keep; keep &= keep - 1u)
                    done |= 1u << s_job[wi][slot].rec[__ffs(keep) - 1];
            if (!have && keep) {
                const int q = __ffs(keep) - 1;
                keep &= keep - 1u;
                ci = s_job[wi][slot].i[q];
                cj = s_job[wi][slot].j[q];
                rec = s_job[wi][slot].rec[q];
                e = lq::root_entry<P>();
                have = true;
            }
            if (!have) {
                if (ST) {
                    iters += __shfl_xor_sync(Q.mask, iters, 1);
                    iters += __shfl_xor_sync(Q.mask, iters, 2);
                }
                if (Q.sub == 0) {
                    if (ST) {
                        stats[DMAP_ST_N * (int64_t)ray + DMAP_ST_SUB] += subs;
                        stats[DMAP_ST_N * (int64_t)ray + DMAP_ST_NEWTON] += iters;
                    }
                    if (found) {
                        RayState &s = states[ray];
                        s.t_max = t_max;
                        s.best_tri = tri;
                        s.flags |= kFoundInTri | kShrunk;
                        s.nah = s.lah = 0;
                    }
                    if (!answered)
                        q_out[atomicAdd(round_ctr(ctr, round, 3), 1ull)] = ray;
                }
                phase = NEED;
            }
        }
        recs &= ~__reduce_or_sync(FULL, done);
        // finished jobs' roots join the batch
        const unsigned fin = __ballot_sync(FULL, phase == NEED && found) & 0x11111111u;
        if (fin) {
            if (phase == NEED && found) {
                if (Q.sub == 0)
                    s_rep[wi][n_rep + __popc(fin & ((1u << Q.lead) - 1u))] = s_best[qi];
                found = false;
            }
            n_rep += __popc(fin);
            if (n_rep > kReps - 8)
                report();
        }
        if (have) {
            const TriDev &T = tris64[tri];
            lq::bound_children<P>(Q, e, tris32[tri], T, s_rec[wi][rec], t_min, t_max, c);
            if (ST)
                subs += 4;
            if (e.depth + 1 < lq::kDepth)
                lq::push_children<P>(Q, c, e.depth + 1, s_stack[qi], sp);
            else if (c.n > 0)
                phase = NEWTON;
        }
        __syncwarp();
        const unsigned wait = __ballot_sync(FULL, phase == NEWTON) & 0x11111111u;
        if (__popc(wait) >= DMAP_NEWTON_QUADS || (wait && !__any_sync(FULL, phase == SEARCH))) {
            if (phase == NEWTON) {
                const TriDev &T = tris64[tri];
                auto on_root = [&](const lq::Found &f) {
                    s_best[qi] = {f.t, f.st.x, f.st.y, ray, tri, ci, cj, f.flags, 0};
                };
                const double t_old = t_max;
                phase = SEARCH;
                if (lq::newton_children<P, ST>(Q, c, T, assets[T.asset], s_rec[wi][rec], ray_of, t_min, t_max, ci, cj,
                                               opt.polish_cond, opt.mode == 1, iters, on_root)) {
                    // occlusion: any hit answers the query (one that an opacity
                    // mask rejects hands the ray to the filter's schedule)
                    answered = true;
                    sp = 0;
                }
                found = found || t_max < t_old;
            }
            __syncwarp();
        }
    }
    report();
}

// Dynamic shared memory of the walk: the candidates' box entries.
size_t entry_bytes(int n_tri) { return n_tri > 32 * kMaskWords ? 0 : (size_t)(n_tri + 3) / 4 * 128 * sizeof(float); }
// The opt-in to as much of it as the largest scene that takes the mask needs,
// whatever the scene at hand: the attribute is the kernel's, and another
// thread's launch over a larger scene may stand between this thread's opt-in
// and its launch. Made at every launch over the mask, not only past the 48 KB
// that need none, so that no size has to know the kernels' static share (the
// last walk passes them at 157 triangles, the walk rounds at 253); a query's
// three opt-ins take less than the 0.3 us by which its enqueueing scatters.
template <class Kernel>
cudaError_t allow_entries(Kernel *kernel)
{
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)entry_bytes(32 * kMaskWords));
}

int sm_count()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    }
    return sms;
}

} // namespace
