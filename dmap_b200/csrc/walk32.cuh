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
//    state and its lanes take the next ray; the leaf kernel runs the parked leaves, one job per lane, each
//    lane taking the next job when its own is done, and queues their rays
//    to resume. After `rounds` rounds a last walk runs the few
//    remaining rays with their leaves inline. Every ray still visits its
//    cells in the reference's order with the reference's t_max, so its hit
//    is the one the simple schedule finds.
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
#include "order.cuh"
#include "filter.cuh"
#include "instance.cuh"

namespace
{
using namespace d32;
using dmapdev::AssetDev;
using dmapdev::TriDev;
using dmapdev::TriDev32;

// Resident 128-thread CTAs per SM the walk and leaf kernels are compiled for
// (register budget: 65536 / (128 x blocks) per thread). The walk rounds over
// the per-ray candidate mask (scenes of up to 256 triangles) take 4 (119
// registers, no spills: faster than 5 at 96 registers with spills); over the
// triangle tree, whose candidate buffer lives in local memory either way, 5.
#ifndef DMAP_WALK_MIN_BLOCKS
#define DMAP_WALK_MIN_BLOCKS 4
#endif
#ifndef DMAP_WALK_TREE_MIN_BLOCKS
#define DMAP_WALK_TREE_MIN_BLOCKS 5
#endif
#ifndef DMAP_LEAF_MIN_BLOCKS
#define DMAP_LEAF_MIN_BLOCKS 1
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
// a few units of 2^-53 of the sums of the terms' magnitudes (2^-40 taken).
__device__ __forceinline__ void tangent_row(const TriDev32 &T, int a, const double *o, const double *d, float t_far,
                                            float &ro, float &rd, float &e)
{
    const double A0 = T.A[a][0], A1 = T.A[a][1], A2 = T.A[a][2];
    double u0 = o[0] - T.q0[0], u1 = o[1] - T.q0[1], u2 = o[2] - T.q0[2];
    double x = A0 * u0;
    x = __fma_rn(A1, u1, x);
    x = __fma_rn(A2, u2, x);
    double y = __fma_rn(A2, d[2], __fma_rn(A1, d[1], A0 * d[0]));
    double mx = fabs(A0 * u0) + fabs(A1 * u1) + fabs(A2 * u2);
    double my = fabs(A0 * d[0]) + fabs(A1 * d[1]) + fabs(A2 * d[2]);
    ro = (float)x;
    rd = (float)y;
    float sum = ru_add(__double2float_ru(mx), ru_mul(t_far, __double2float_ru(my)));
    e = ru_add(ru_mul(0x1p-22f, ru_add(fabsf(ro), ru_mul(t_far, fabsf(rd)))), ru_mul(0x1p-40f, sum));
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
            if (!square_meets_domain(W, ((float)cur.i + 0.5f) * w, ((float)cur.j + 0.5f) * w, 0.5f * w)) {
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
    unsigned long long mask[4]; // per lane of the ray's four
    // scenes of more than 256 triangles: the buffered candidates, kept
    // across parks so a resumed ray does not walk the tree again
    d32::NearBuf buf;
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
    int ray, tri, n, pad;
    int i[kCollect], j[kCollect];
};
// RayState.flags
constexpr int kFoundInTri = 1; // a hit was taken in the triangle in progress
constexpr int kShrunk = 2;     // the leaves of the last job shrank t_max: the cells still open are tested again
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

// Four lanes walk one ray (a quad; eight rays per warp), so that the four
// cells of a sibling group are tested together, one per lane. A lane per ray
// ran one node test per step with 19.6 of 32 lanes in it, the others being in
// a pick or between cells; and a ray's tests, one after the other, set the
// time of small batches and of every launch's tail. Walk rounds and last walk
// before and after: 64 rays on a quad 212 -> 63 us, 20,011 rays on the sphere
// of 96 x 512^2 maps 2.80 -> 0.69 ms, 2.80M rays on 96 x 2048^2 34.1 -> 27.2
// ms. Per quad and step: take
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
    enum : int { NEED = 0, TOP = 1, WALK = 2, DONE = 3 };
    const int lane = threadIdx.x & 31, sub = lane & 3, lead = lane & 28;
    // the candidates: scenes of up to 256 triangles take a mask of one bit
    // per triangle whose box the ray meets (built by the warp at the ray's
    // start; triangle t is bit t / 4 of the quad's lane t % 4), larger scenes
    // (TREE) the triangle tree (bvh.cuh), in either order; the launcher takes
    // the mask only for up to 256 triangles, so its loops are never compiled
    // into the kernels of larger scenes
    const d32::BvhView bvh = {opt.bvh_nodes, opt.bvh_tri, opt.bvh_range, opt.bvh_n_nodes};
    // scenes of up to 256 triangles: their object boxes in shared memory
    // (outward FP32 for the box tests, FP64 for the nearest order's keys),
    // which every candidate test of the CTA reads; component c of triangle t
    // at c * kStaged + t
    constexpr int kStaged = TREE ? 1 : 32 * kMaskWords;
    __shared__ float s_box32[6 * kStaged];
    __shared__ double s_box64[(NEAR ? 6 : 1) * kStaged];
    if (!TREE) {
        for (int k = threadIdx.x; k < 6 * n_tri; k += blockDim.x) {
            const int t = k / 6, c = k - 6 * t;
            s_box32[c * kStaged + t] = c < 3 ? tris32[t].box_lo[c] : tris32[t].box_hi[c - 3];
            if (NEAR)
                s_box64[c * kStaged + t] = c < 3 ? tris64[t].box_lo[c] : tris64[t].box_hi[c - 3];
        }
        __syncthreads();
    }
    auto box32 = [&](int t, float *lo, float *hi) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = s_box32[c * kStaged + t];
            hi[c] = s_box32[(3 + c) * kStaged + t];
        }
    };
    // items of this round: every ray in round 0, else the resume queue
    unsigned long long count = round == 0 ? (unsigned long long)n : *round_ctr(ctr, round - 1, 3);
    if (round == 0 && opt.n_dev && (unsigned long long)*opt.n_dev < count)
        count = *opt.n_dev < 0 ? 0ull : (unsigned long long)*opt.n_dev;
    unsigned long long *fetch = round_ctr(ctr, round, 0);
    // a round of fewer rays than the grid has quads spreads them over all
    // its warps, so that fewer of them share a warp
    const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
    int phase = (unsigned long long)(lane >> 2) * warps < count ? NEED : DONE;
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
    Ray32 r;
    const float *pyr = nullptr;
    Cell32 cur = {0, 0, 0};
    CellBits<DEEP> todo = {0ull, 0ull}, dom = {0ull, 0ull}; // cells that passed; cells in the domain, not yet gone past
    unsigned stale = 0u;                                   // levels whose group must be tested again
    unsigned long long mask = 0ull;
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
            job.pad = 0;
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
        float ro, rd, e;
        tangent_row(T, sub < 3 ? sub : 0, o, d, t_far, ro, rd, e);
        const float inv = rd != 0.0f ? __frcp_rn(rd) : 0.0f;
        r.ox = __shfl_sync(quad, ro, lead), r.oy = __shfl_sync(quad, ro, lead + 1), r.oz = __shfl_sync(quad, ro, lead + 2);
        r.dx = __shfl_sync(quad, rd, lead), r.dy = __shfl_sync(quad, rd, lead + 1), r.dz = __shfl_sync(quad, rd, lead + 2);
        r.ix = __shfl_sync(quad, inv, lead), r.iy = __shfl_sync(quad, inv, lead + 1), r.iz = __shfl_sync(quad, inv, lead + 2);
        r.ex = __shfl_sync(quad, e, lead), r.ey = __shfl_sync(quad, e, lead + 1), r.ez = __shfl_sync(quad, e, lead + 2);
        si = r.dx < 0.0f;
        sj = r.dy < 0.0f;
        pyr = T.pyr32;
    };

    for (;;) {
        // 1. quads without work take the next items, one atomic per warp
        const unsigned need = __ballot_sync(FULL, phase == NEED) & 0x11111111u;
        bool fresh = false;
        float of[3], df[3], invf[3]; // the ray in float, while it is fetched or picks
        if (need) {
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader)
                base = atomicAdd(fetch, (unsigned long long)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (phase == NEED) {
                unsigned long long item = base + (unsigned long long)__popc(need & ((1u << lead) - 1u));
                if (item >= count) {
                    phase = DONE;
                } else {
                    ray = round == 0 ? (int)item : q_in[item];
                    double o[3], d[3], t_min;
                    load_ray(rays, opt.ray_dtype, ray, o, d, t_min, t_max);
                    nbuf.n = -1;
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        of[a] = (float)o[a];
                        df[a] = (float)d[a];
                        invf[a] = df[a] != 0.0f ? __frcp_rn(df[a]) : 0.0f;
                    }
                    tmin_f = __double2float_rd(t_min);
                    if (ST)
                        for (int q = 0; q < DMAP_ST_N; ++q)
                            stl[q] = 0;
                    if (round == 0) {
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
                        const TriDev32 &T = tris32[tri];
                        float t1 = tmax_f;
                        object_box(T, of, df, invf, tmin_f, t1);
                        enter_frame(T, o, d, far_bound(fmaxf(t1, tmin_f)));
                        stale = (flags & kShrunk) ? ~0u : 0u;
                        flags &= ~kShrunk;
                        guard = 0;
                        nl = 0;
                        phase = WALK;
                    }
                }
            }
        }
        // round 0: the warp finds the fresh rays' candidate triangles
        // together, 32 boxes per ballot; byte q of a ballot is the triangles
        // of lane q
        if (!TREE) {
            unsigned left = __ballot_sync(FULL, fresh) & 0x11111111u;
            while (left) {
                const int src = __ffs(left) - 1;
                left &= left - 1;
                float so[3], sd[3], sv[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    so[a] = __shfl_sync(FULL, of[a], src);
                    sd[a] = __shfl_sync(FULL, df[a], src);
                    sv[a] = __shfl_sync(FULL, invf[a], src);
                }
                const float s_tmin = __shfl_sync(FULL, tmin_f, src), s_tmax = __shfl_sync(FULL, tmax_f, src);
#pragma unroll 1
                for (int w = 0; w < ((n_tri + 31) >> 5); ++w) {
                    const int t = 32 * w + 4 * (lane & 7) + (lane >> 3);
                    float t1 = s_tmax, lo[3], hi[3];
                    bool pass = t < n_tri;
                    if (pass) {
                        box32(t, lo, hi);
                        pass = box_pass(lo, hi, so, sd, sv, s_tmin, t1);
                    }
                    const unsigned bits = __ballot_sync(FULL, pass);
                    if (lead == src)
                        mask |= (unsigned long long)((bits >> (8 * sub)) & 255u) << (8 * w);
                }
            }
        }
        if (__all_sync(FULL, phase == DONE))
            break;

        // 2. the next triangle whose object box the ray meets (intersect_flat's loop)
        bool test = false, roots = false, again = false; // a group to test: the roots; one tested before
        if (phase == TOP) {
            const unsigned quad = 0xfu << lead;
            double o[3], d[3], t_min, t_ray;
            load_ray(rays, opt.ray_dtype, ray, o, d, t_min, t_ray);
            if (!fresh) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    of[a] = (float)o[a];
                    df[a] = (float)d[a];
                    invf[a] = df[a] != 0.0f ? __frcp_rn(df[a]) : 0.0f;
                }
            }
            float t1 = 0.0f;
            int bt = -1;
            double inv[3];
            if (NEAR) {
                // 1 / d in double, an axis per lane
                const double da = sub == 0 ? d[0] : sub == 1 ? d[1] : d[2];
                const double ia = da != 0.0 ? 1.0 / da : 0.0;
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    inv[a] = __shfl_sync(quad, ia, lead + a);
            }
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
                // the best of each lane's candidates (nearest order: the
                // smallest (key, index); index order: the smallest index),
                // then of the quad's; each box is re-tested with the current
                // t_max first, and a bit whose box no longer passes is
                // cleared for good (t_max only shrinks). The taken triangle's
                // bit is cleared too, so every bit left is past it.
                double bk = 0.0;
                unsigned long long m = mask;
                while (m) {
                    const int b = __ffsll((long long)m) - 1;
                    m &= m - 1ull;
                    const int t = 4 * b + sub;
                    float e = tmin_f, tt = tmax_f, lo[3], hi[3];
                    box32(t, lo, hi);
                    if (!box_range(lo, hi, of, df, invf, e, tt)) {
                        mask &= ~(1ull << b);
                        continue;
                    }
                    if (!NEAR) {
                        bt = t;
                        t1 = tt;
                        break;
                    }
                    if (bt >= 0 && (double)e > bk)
                        continue; // its key (at least e) is past the best
                    double dlo[3], dhi[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        dlo[c] = s_box64[c * kStaged + t];
                        dhi[c] = s_box64[(3 + c) * kStaged + t];
                    }
                    const double key = d64::entry_key(dlo, dhi, o, d, inv, t_min);
                    if (!d64::before_best(key, t, bk, bt))
                        continue;
                    bk = key;
                    bt = t;
                    t1 = tt;
                }
                __syncwarp(quad);
#pragma unroll
                for (int x = 1; x < 4; x <<= 1) {
                    const int ot = __shfl_xor_sync(quad, bt, x);
                    const float o1 = __shfl_xor_sync(quad, t1, x);
                    const double ok = NEAR ? __shfl_xor_sync(quad, bk, x) : (double)ot;
                    if (ot >= 0 && (NEAR ? d64::before_best(ok, ot, bk, bt) : (bt < 0 || ot < bt))) {
                        bk = ok;
                        bt = ot;
                        t1 = o1;
                    }
                }
                if (bt >= 0 && (bt & 3) == sub)
                    mask &= ~(1ull << (bt >> 2));
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
                enter_frame(tris32[tri], o, d, far_bound(t1));
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
        __syncwarp();

        // 3a. the next cell of the open groups: a leaf is collected, another
        // cell's children are the group to test
        int tl = 0, pi = 0, pj = 0; // the group: its level, its parent cell
        unsigned cells = 15u;
        bool leaf = false;
        if (phase == WALK) {
            const int root_level = tris32[tri].root_level;
            if (test) {
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
            while (!test && phase == WALK) {
                if (!todo.any()) {
                    // the end of the triangle's walk
                    if (ST) {
                        const int left = dom.count();
                        stl[DMAP_ST_NODE] += left;
                        nah += left;
                    }
                    dom = {0ull, 0ull};
                    if (!INLINE_LEAF && nl > 0) {
                        // the collected leaves decide this triangle's t_max before the next one
                        park();
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
                        park();
                        break;
                    }
                    since += n_in;
                }
                if (ST) {
                    stl[DMAP_ST_NODE] += n_in;
                    nah += n_in;
                }
                dom.clear_upto(p);
                if (l > 0 && nl > 0 && since > DMAP_STALE_CAP) {
                    park(); // the cell is taken (and its group tested) again after the resume
                    break;
                }
                todo.clear_bit(p);
                const TriDev32 &T = tris32[tri];
                cur.level = l;
                cur.i = at_root ? T.roots_i[k] : 2 * pi + ((k >> 1) ^ si);
                cur.j = at_root ? T.roots_j[k] : 2 * pj + ((k & 1) ^ sj);
                if (l > 0) {
                    tl = l - 1;
                    pi = cur.i;
                    pj = cur.j;
                    test = true;
                    break;
                }
                if (ST) {
                    ++stl[DMAP_ST_LEAF];
                    ++lah;
                }
                if (INLINE_LEAF) {
                    leaf = true;
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
                    park();
            }
        }
        __syncwarp();

        if (INLINE_LEAF) {
            // the last round: the few remaining rays finish here
            int got = 0;
            if (leaf && sub == 0) {
                double o[3], d[3], t_min, t_ray;
                load_ray(rays, opt.ray_dtype, ray, o, d, t_min, t_ray);
                d64::hit64 lh;
                int lf = 0;
                if (leaf_cell(tris32[tri], tris64[tri], assets[tris32[tri].asset], o, d, t_min, t_max, cur.i, cur.j, lh,
                              lf, ST ? stl : nullptr, opt) &&
                    lh.t < t_max) {
                    t_max = lh.t;
                    got = 1;
                    store_hit(hits, opt.hit_dtype, ray, true, lh, tri, lf | ((flags & kCapped) ? DMAP_HIT_CAPPED : 0));
                    check_crossing(opt, tris64[tri], tri, lh, ray, flags, ctr, rerun);
                }
            }
            __syncwarp();
            got = __shfl_sync(FULL, got, lead);
            t_max = __shfl_sync(FULL, t_max, lead);
            flags = __shfl_sync(FULL, flags, lead);
            if (leaf && got) {
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

        // 3b. the group's cells, one per lane, all quads together
        bool in = false, pass = false;
        if (test && ((cells >> sub) & 1u)) {
            const TriDev32 &T = tris32[tri];
            const Walk32 W = load_walk(T);
            const int ci = roots ? T.roots_i[sub] : 2 * pi + ((sub >> 1) ^ si);
            const int cj = roots ? T.roots_j[sub] : 2 * pj + ((sub & 1) ^ sj);
            const float w = pow2f(tl - W.log2n);
            in = square_meets_domain(W, ((float)ci + 0.5f) * w, ((float)cj + 0.5f) * w, 0.5f * w);
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
                if (guard > opt.guard_cap) { // a finite tree: the cap guards corrupt records
                    atomicOr(status, dmapdev::kStatusCapped);
                    flags |= kCapped;
                    todo = {0ull, 0ull};
                    dom = {0ull, 0ull};
                }
            }
        }
    }
}

// The leaf cells of a round's jobs through the reference's own node test in
// double (node_bounds.cpp:83-211 at level 0, the node computed from the
// grid): the FP32 walk, widened by its roundings, reaches more leaf cells
// than the FP64 walk, and a cell the FP64 walk rejects has no leaf there.
// The ray's t_max is the one it parked with; earlier leaves of the same job
// can only shrink it, so a cell kept here may still be rejected by the FP64
// walk at that point, and its search then finds nothing the reference
// would not. Cells are compacted in walk order; a job may end up empty.
// Kept apart from the leaf kernel so that kernel's code stays small.
template <typename R>
__global__ void __launch_bounds__(128)
    wave_filter(const TriDev *__restrict__ tris64, const AssetDev *__restrict__ assets, const R *__restrict__ rays,
                dmapk::QueryOpts opt, const RayState *__restrict__ states, LeafJob *__restrict__ q_leaf, int round,
                const unsigned long long *ctr)
{
    const unsigned long long count = *round_ctr(const_cast<unsigned long long *>(ctr), round, 1);
    for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < count;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        LeafJob job = q_leaf[k];
        double o[3], d[3], t_min, t_max;
        load_ray(rays, job.ray, o, d, t_min, t_max);
        t_max = states[job.ray].t_max;
        const TriDev &T = tris64[job.tri];
        const AssetDev &g = assets[T.asset];
        if (T.inst) {
            double oo[3], od[3];
            dmapdev::object_ray(opt.inst_xf + dmapdev::kInstDoubles * (T.inst - 1), o, d, oo, od);
            for (int a = 0; a < 3; ++a) {
                o[a] = oo[a];
                d[a] = od[a];
            }
        }
        d64::tray r = d64::tangent_ray64(T, d64::V3(o[0], o[1], o[2]), d64::V3(d[0], d[1], d[2]), t_min, t_max);
        int m = 0;
#pragma unroll 1
        for (int q = 0; q < job.n; ++q) {
            if (d64::leaf_cell_admitted(T, g, r, job.i[q], job.j[q], opt)) {
                job.i[m] = job.i[q];
                job.j[m] = job.j[q];
                ++m;
            }
        }
        if (m != job.n) {
            job.n = m;
            q_leaf[k] = job;
        }
    }
}

// The parked leaves of a round (the certified leaf, d64::intersect_newton,
// displaced_intersector.cpp:239-323). Each lane holds one job at a time and
// takes the next one as soon as its own is done, so a warp's lanes stay busy
// however long their leaves run. A step of the loop runs, for the lanes that
// need it: the leaf setup, one sub-square expansion (four bounds, the sort,
// the push) or one Newton run, with the warp reconverged between blocks.
// Each lane's search is intersect_newton's, in the same order with the same
// arithmetic, so each ray's result equals it bit for bit. A ray whose walk
// has cells left goes back to the resume queue.
template <bool ST, typename R, typename H, typename Fp>
__global__ void __launch_bounds__(128, DMAP_LEAF_MIN_BLOCKS)
    wave_leaf(const TriDev *__restrict__ tris64, const AssetDev *__restrict__ assets, const R *__restrict__ rays,
              dmapk::QueryOpts opt, H *__restrict__ hits, int64_t *__restrict__ stats, RayState *__restrict__ states,
              const LeafJob *__restrict__ q_leaf, int round, int *__restrict__ q_out, unsigned long long *ctr,
              int *__restrict__ rerun)
{
    using namespace d64;
    constexpr int kDepth = 5; // subdivision_depth
    enum : int { NEED = 0, SETUP = 1, SEARCH = 2, DONE = 3 };
    const int lane = threadIdx.x & 31;
    const unsigned long long count = *round_ctr(ctr, round, 1);
    unsigned long long *fetch = round_ctr(ctr, round, 2);
    int phase = NEED;
    unsigned long long item = 0;
    int ray = 0, tri = 0, n_leaves = 0, q = 0, li = 0, lj = 0, sp = 0;
    bool first = false, answered = false;
    double t_min = 0.0, t_max = 0.0;
    v3 O = V3(0.0, 0.0, 0.0), D = O;
    leafbound L;
    leafent stack[4 * kDepth + 4];
    int64_t subs = 0, iters = 0;

    for (;;) {
        // lanes without a job take the next ones, one atomic per warp
        unsigned need = __ballot_sync(FULL, phase == NEED);
        if (need) {
            int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader)
                base = atomicAdd(fetch, (unsigned long long)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (phase == NEED) {
                item = base + (unsigned long long)__popc(need & ((1u << lane) - 1u));
                if (item >= count) {
                    phase = DONE;
                } else {
                    const LeafJob &J = q_leaf[item];
                    ray = J.ray;
                    tri = J.tri;
                    n_leaves = J.n;
                    q = 0;
                    if (n_leaves == 0) {
                        // the filter rejected every cell of the job: the walk goes on
                        unsigned long long slot = atomicAdd(round_ctr(ctr, round, 3), 1ull);
                        q_out[slot] = ray;
                    } else {
                        double o[3], d[3];
                        load_ray(rays, ray, o, d, t_min, t_max);
                        if (tris64[tri].inst) {
                            double oo[3], od[3];
                            dmapdev::object_ray(opt.inst_xf + dmapdev::kInstDoubles * (tris64[tri].inst - 1), o, d,
                                                oo, od);
                            for (int a = 0; a < 3; ++a) {
                                o[a] = oo[a];
                                d[a] = od[a];
                            }
                        }
                        O = V3(o[0], o[1], o[2]);
                        D = V3(d[0], d[1], d[2]);
                        t_max = states[ray].t_max;
                        answered = false;
                        subs = iters = 0;
                        phase = SETUP;
                    }
                }
            }
        }
        if (__all_sync(FULL, phase == DONE))
            break;
        const TriDev &T = tris64[tri];
        const AssetDev &g = assets[T.asset];
        // leaf q of the job (a cell wave_filter kept): the texel's corners,
        // its normal form and the ray's plane basis (:239-264)
        if (phase == SETUP) {
            li = q_leaf[item].i[q];
            lj = q_leaf[item].j[q];
            sp = 0;
            phase = SEARCH;
            L.w = cell_width(g, 0);
            L.lo = {li * L.w, lj * L.w};
            L.h00 = grid_h(g, L.lo.x, L.lo.y);
            L.h10 = grid_h(g, L.lo.x + L.w, L.lo.y);
            L.h01 = grid_h(g, L.lo.x, L.lo.y + L.w);
            L.h11 = grid_h(g, L.lo.x + L.w, L.lo.y + L.w);
            v2 c = add2(L.lo, V2(0.5 * L.w, 0.5 * L.w));
            double hw = 0.5 * L.w;
            L.N_hat = AF3(add3(add3(L3(T.m0), mul3(c.x, L3(T.Mu))), mul3(c.y, L3(T.Mv))), mul3(hw, L3(T.Mu)),
                          mul3(hw, L3(T.Mv)));
            normalize(L.N_hat);
            L.o = O;
            L.d_len = norm3(D);
            L.dn = div3(D, L.d_len);
            plane_basis(L.dn, L.d1, L.d2);
            stack[sp++] = {0.5, 0.5, -INFINITY, 0};
            first = true;
        }
        // the next live entry of the search (a pop is a call of search_leaf;
        // an entry at or beyond t_max is the sorted loop's break)
        bool expand = false, newton = false;
        leafent e = {0.0, 0.0, 0.0, 0};
        if (phase == SEARCH) {
            while (sp > 0) {
                e = stack[--sp];
                if (first || e.t_lo < t_max) {
                    first = false;
                    newton = e.depth == kDepth;
                    expand = !newton;
                    break;
                }
            }
            if (!expand && !newton) {
                // the leaf is done; the next of the job, or the job is done
                if (++q < n_leaves && !answered) {
                    phase = SETUP;
                } else {
                    if (ST) {
                        stats[DMAP_ST_N * (int64_t)ray + DMAP_ST_SUB] += subs;
                        stats[DMAP_ST_N * (int64_t)ray + DMAP_ST_NEWTON] += iters;
                    }
                    if (!answered) {
                        unsigned long long slot = atomicAdd(round_ctr(ctr, round, 3), 1ull);
                        q_out[slot] = ray;
                    }
                    phase = NEED;
                }
            }
        }
        __syncwarp();
        if (expand) {
            double r = 0.5 * ldexp(0.5, -e.depth);
            leafent ch[4];
            int n = 0;
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                double ca = e.a + ((k & 1) ? r : -r), cb = e.b + ((k & 2) ? r : -r), t_lo;
                ++subs;
                if (sub_square_bound(T, L, ca, cb, r, t_min, t_max, t_lo))
                    ch[n++] = {ca, cb, t_lo, e.depth + 1};
            }
            for (int p = 1; p < n; ++p)
                for (int k = p; k > 0 && ch[k].t_lo < ch[k - 1].t_lo; --k) {
                    leafent x = ch[k];
                    ch[k] = ch[k - 1];
                    ch[k - 1] = x;
                }
            for (int k = n - 1; k >= 0; --k)
                stack[sp++] = ch[k];
        }
        __syncwarp();
        if (newton) {
            hit64 h;
            if (newton_from(T, g, O, D, t_min, t_max, li, lj, add2(L.lo, mul2(L.w, V2(e.a, e.b))), h, iters)) {
                // a nearer root of this leaf (each later one is nearer still)
                t_max = h.t;
                RayState &s = states[ray];
                s.t_max = h.t;
                s.best_tri = tri;
                s.flags |= kFoundInTri | kShrunk;
                s.nah = s.lah = 0;
                if (tris64[tri].inst)
                    dmapdev::world_normal(opt.inst_xf + dmapdev::kInstDoubles * (tris64[tri].inst - 1), h.ng);
                store_hit<H, Fp>(hits, ray, true, h, tri,
                                 DMAP_HIT_FP64_LEAF | ((s.flags & kCapped) ? DMAP_HIT_CAPPED : 0));
                check_crossing(opt, tris64[tri], tri, h, ray, s.flags, ctr, rerun);
                if (opt.mode == 1) { // occlusion: any hit answers the query
                    answered = true;
                    sp = 0;
                }
            }
        }
        __syncwarp();
    }
}

// The parked leaves of a round with the FP32 certified leaf (leaf32.cuh):
// wave_leaf's schedule (one job per lane, a lane takes the next job when its
// own is done, one search step per loop iteration) over the FP32 leaf state.
#ifndef DMAP_LEAF32_MIN_BLOCKS
#define DMAP_LEAF32_MIN_BLOCKS 1
#endif
template <bool ST, typename R, typename H, typename Fp>
__global__ void __launch_bounds__(128, DMAP_LEAF32_MIN_BLOCKS)
    wave_leaf32(const TriDev32 *__restrict__ tris32, const TriDev *__restrict__ tris64,
                const AssetDev *__restrict__ assets, const R *__restrict__ rays, dmapk::QueryOpts opt,
                H *__restrict__ hits, int64_t *__restrict__ stats, RayState *__restrict__ states,
                const LeafJob *__restrict__ q_leaf, int round, int *__restrict__ q_out, unsigned long long *ctr,
                int *__restrict__ rerun)
{
    using namespace d64;
    constexpr int kDepth = 5; // subdivision_depth
    enum : int { NEED = 0, SETUP = 1, SEARCH = 2, DONE = 3 };
    const int lane = threadIdx.x & 31;
    const unsigned long long count = *round_ctr(ctr, round, 1);
    unsigned long long *fetch = round_ctr(ctr, round, 2);
    int phase = NEED;
    unsigned long long item = 0;
    int ray = 0, tri = 0, n_leaves = 0, q = 0, li = 0, lj = 0, sp = 0;
    bool first = false, answered = false;
    double t_min = 0.0, t_max = 0.0;
    v3 O = V3(0.0, 0.0, 0.0), D = O;
    l32::Leaf32 L;
    l32::Ent32 stack[4 * kDepth + 4];
    int64_t subs = 0, iters = 0;

    for (;;) {
        unsigned need = __ballot_sync(FULL, phase == NEED);
        if (need) {
            int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if (lane == leader)
                base = atomicAdd(fetch, (unsigned long long)__popc(need));
            base = __shfl_sync(FULL, base, leader);
            if (phase == NEED) {
                item = base + (unsigned long long)__popc(need & ((1u << lane) - 1u));
                if (item >= count) {
                    phase = DONE;
                } else {
                    const LeafJob &J = q_leaf[item];
                    ray = J.ray;
                    tri = J.tri;
                    n_leaves = J.n;
                    q = 0;
                    if (n_leaves == 0) {
                        unsigned long long slot = atomicAdd(round_ctr(ctr, round, 3), 1ull);
                        q_out[slot] = ray;
                    } else {
                        double o[3], d[3];
                        load_ray(rays, ray, o, d, t_min, t_max);
                        if (tris64[tri].inst) {
                            double oo[3], od[3];
                            dmapdev::object_ray(opt.inst_xf + dmapdev::kInstDoubles * (tris64[tri].inst - 1), o, d,
                                                oo, od);
                            for (int a = 0; a < 3; ++a) {
                                o[a] = oo[a];
                                d[a] = od[a];
                            }
                        }
                        O = V3(o[0], o[1], o[2]);
                        D = V3(d[0], d[1], d[2]);
                        t_max = states[ray].t_max;
                        answered = false;
                        subs = iters = 0;
                        phase = SETUP;
                    }
                }
            }
        }
        if (__all_sync(FULL, phase == DONE))
            break;
        const TriDev &T = tris64[tri];
        const AssetDev &g = assets[T.asset];
        if (phase == SETUP) {
            li = q_leaf[item].i[q];
            lj = q_leaf[item].j[q];
            l32::leaf_setup32(T, g, O, D, li, lj, L);
            sp = 0;
            stack[sp++] = {0.5f, 0.5f, -INFINITY, 0};
            first = true;
            phase = SEARCH;
        }
        bool expand = false, newton = false;
        l32::Ent32 e = {0.0f, 0.0f, 0.0f, 0};
        if (phase == SEARCH) {
            while (sp > 0) {
                e = stack[--sp];
                if (first || (double)e.t_lo < t_max) {
                    first = false;
                    newton = e.depth == kDepth;
                    expand = !newton;
                    break;
                }
            }
            if (!expand && !newton) {
                if (++q < n_leaves && !answered) {
                    phase = SETUP;
                } else {
                    if (ST) {
                        stats[DMAP_ST_N * (int64_t)ray + DMAP_ST_SUB] += subs;
                        stats[DMAP_ST_N * (int64_t)ray + DMAP_ST_NEWTON] += iters;
                    }
                    if (!answered) {
                        unsigned long long slot = atomicAdd(round_ctr(ctr, round, 3), 1ull);
                        q_out[slot] = ray;
                    }
                    phase = NEED;
                }
            }
        }
        __syncwarp();
        if (expand) {
            const TriDev32 &T32 = tris32[tri];
            float r = __int_as_float((125 - e.depth) << 23); // half of the entry's rho = 0.5 * 2^-depth
            l32::Ent32 ch[4];
            int n = 0;
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                float ca = e.a + ((k & 1) ? r : -r), cb = e.b + ((k & 2) ? r : -r), tl;
                ++subs;
                if (l32::sub_square_bound32(T32, L, ca, cb, r, t_min, t_max, tl))
                    ch[n++] = {ca, cb, tl, e.depth + 1};
            }
            for (int p = 1; p < n; ++p)
                for (int k = p; k > 0 && ch[k].t_lo < ch[k - 1].t_lo; --k) {
                    l32::Ent32 x = ch[k];
                    ch[k] = ch[k - 1];
                    ch[k - 1] = x;
                }
            for (int k = n - 1; k >= 0; --k)
                stack[sp++] = ch[k];
        }
        __syncwarp();
        if (newton) {
            l32::Root32 root;
            hit64 h;
            int fl = 0;
            if (l32::newton32(T, L, e.a, e.b, root, iters) &&
                l32::accept_root(T, g, L.lo_s, L.lo_t, L.w, L.Q3, L.inv_dlen, O, D, t_min, t_max, li, lj, root,
                                 opt.polish_cond, h, fl, iters)) {
                t_max = h.t;
                RayState &s = states[ray];
                s.t_max = h.t;
                s.best_tri = tri;
                s.flags |= kFoundInTri | kShrunk;
                s.nah = s.lah = 0;
                if (tris64[tri].inst)
                    dmapdev::world_normal(opt.inst_xf + dmapdev::kInstDoubles * (tris64[tri].inst - 1), h.ng);
                store_hit<H, Fp>(hits, ray, true, h, tri, fl | ((s.flags & kCapped) ? DMAP_HIT_CAPPED : 0));
                check_crossing(opt, tris64[tri], tri, h, ray, s.flags, ctr, rerun);
                if (opt.mode == 1) {
                    answered = true;
                    sp = 0;
                }
            }
        }
        __syncwarp();
    }
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
