// The certified leaf's search (displaced_intersector.cpp:239-323,
// intersect_newton and search_leaf) by the four lanes of a quad: the four
// children of a sub-square are bounded together, one per lane, and the
// Newton runs of a last expansion's children run together too. The search
// visits what the recursive one visits, in its order, with its arithmetic:
// the children that pass are pushed in sorted order (ties to the lower
// child), an entry at or beyond t_max is dropped when it comes off the
// stack, and roots are taken in sorted order, each judged against the t_max
// the earlier ones left. So every leaf finds the roots that one lane
// searching alone finds, bit for bit, in a quarter of the steps: a lane per
// leaf left a warp waiting for its longest search.
//
// Two leaves: P64, the reference's in double (f64_leaf.cuh), and P32, the
// FP32 leaf (leaf32.cuh).
#pragma once
#include "leaf32.cuh"

namespace lq
{
using dmapdev::AssetDev;
using dmapdev::TriDev;
using dmapdev::TriDev32;
using d64::hit64;
using d64::v3;

constexpr int kDepth = 5;  // subdivision_depth
// Entries of the search's stack: below the last depth at most three siblings
// wait per level, and four after an expansion; children at the last depth
// are not pushed.
constexpr int kStack = 16;
static_assert(3 * (kDepth - 2) + 4 <= kStack, "search stack");

// An accepted root; the hit record follows from it (d64::root_record), once
// the search is over.
struct Found { double t; d64::v2 st; int flags; };

struct P32
{
    using Real = float;
    using Bound = l32::Leaf32;
    using Root = l32::Root32;
    struct Ent { float a, b, t_lo; int depth; };
    static __device__ __forceinline__ void setup(const TriDev &T, const AssetDev &g, v3 o, v3 d, int i, int j, Bound &L)
    {
        l32::leaf_setup32_shared(T, g, o, d, i, j, L);
    }
    static __device__ __forceinline__ bool bound(const TriDev32 &T32, const TriDev &, const Bound &L, float a, float b,
                                                 float rho, double t_min, double t_max, float &t_lo)
    {
        return l32::sub_square_bound32(T32, L, a, b, rho, t_min, t_max, t_lo);
    }
    template <class Ray>
    static __device__ __forceinline__ bool newton(const TriDev &T, const AssetDev &, const Bound &L, const Ray &, double,
                                                  double, int, int, float a, float b, Root &r, int64_t &iters)
    {
        return l32::newton32(T, L, a, b, r, iters);
    }
    template <class Ray>
    static __device__ __forceinline__ bool judge(const TriDev &T, const AssetDev &g, const Bound &L, const Ray &ray,
                                                 double t_min, double t_max, int i, int j, const Root &r,
                                                 double polish_cond, Found &f, int64_t &iters)
    {
        return l32::judge_root(T, g, L, ray, t_min, t_max, i, j, r, polish_cond, f.t, f.st, f.flags, iters);
    }
};

struct P64
{
    using Real = double;
    using Bound = d64::leafbound;
    using Root = hit64;
    struct Ent { double t_lo; float a, b; int depth; }; // a, b: multiples of 2^-6, exact
    static __device__ __forceinline__ void setup(const TriDev &T, const AssetDev &g, v3 o, v3 d, int i, int j, Bound &L)
    {
        d64::leaf_setup_shared(T, g, o, d, i, j, L);
    }
    static __device__ __forceinline__ bool bound(const TriDev32 &, const TriDev &T, const Bound &L, float a, float b,
                                                 float rho, double t_min, double t_max, double &t_lo)
    {
        return d64::sub_square_bound(T, L, a, b, rho, t_min, t_max, t_lo);
    }
    template <class Ray>
    static __device__ __forceinline__ bool newton(const TriDev &T, const AssetDev &g, const Bound &L, const Ray &ray,
                                                  double t_min, double t_max, int i, int j, float a, float b, Root &r,
                                                  int64_t &iters)
    {
        v3 o, d;
        ray(o, d);
        return d64::newton_from(T, g, o, d, t_min, t_max, i, j,
                                d64::add2(L.lo, d64::mul2(L.w, d64::V2((double)a, (double)b))), r, iters);
    }
    template <class Ray>
    static __device__ __forceinline__ bool judge(const TriDev &, const AssetDev &, const Bound &, const Ray &, double,
                                                 double t_max, int, int, const Root &r, double, Found &f, int64_t &)
    {
        // newton_from judged it with the t_max of the runs' start; the nearer roots found since count too
        if (r.t >= t_max)
            return false;
        f.t = r.t;
        f.st = r.st;
        f.flags = DMAP_HIT_FP64_LEAF;
        return true;
    }
};

// The quad's lanes: its mask, its first lane and the lane's number in it.
struct Quad { unsigned mask; int lead, sub; };

template <class P>
__device__ __forceinline__ typename P::Ent root_entry()
{
    typename P::Ent e;
    e.a = e.b = 0.5f;
    e.t_lo = -INFINITY;
    e.depth = 0;
    return e;
}

// The next entry of the search off its stack (an entry at or beyond t_max is
// the sorted loop's break).
template <class P>
__device__ __forceinline__ bool pop(const typename P::Ent *stack, int &sp, double t_max, typename P::Ent &e)
{
    while (sp > 0) {
        e = stack[--sp];
        if ((double)e.t_lo < t_max)
            return true;
    }
    return false;
}

// A lane's child of an expanded entry: its centre, its t_lo, whether it
// passed, its place among the children that passed (sorted by t_lo, ties to
// the lower child), and how many passed.
template <class P>
struct Child
{
    float a, b;
    typename P::Real t_lo;
    bool pass;
    int rank, n;
};

// The children of an entry, bounded by the four lanes together.
template <class P>
__device__ __forceinline__ void bound_children(const Quad &Q, const typename P::Ent &e, const TriDev32 &T32,
                                               const TriDev &T, const typename P::Bound &L, double t_min, double t_max,
                                               Child<P> &c)
{
    typedef typename P::Real Real;
    const float r = __int_as_float((125 - e.depth) << 23); // half of the entry's rho = 0.5 * 2^-depth
    c.a = e.a + ((Q.sub & 1) ? r : -r);
    c.b = e.b + ((Q.sub & 2) ? r : -r);
    c.t_lo = 0;
    c.pass = P::bound(T32, T, L, c.a, c.b, r, t_min, t_max, c.t_lo);
    __syncwarp(Q.mask);
    const unsigned pm = (__ballot_sync(Q.mask, c.pass) >> Q.lead) & 15u;
    c.rank = 0;
    c.n = __popc(pm);
#pragma unroll
    for (int x = 1; x < 4; ++x) {
        const Real o = __shfl_xor_sync(Q.mask, c.t_lo, x);
        const int os = Q.sub ^ x;
        c.rank += ((pm >> os) & 1u) && (o < c.t_lo || (o == c.t_lo && os < Q.sub)) ? 1 : 0;
    }
}

// The children that passed onto the stack, the nearest on top.
template <class P>
__device__ __forceinline__ void push_children(const Quad &Q, const Child<P> &c, int depth, typename P::Ent *stack,
                                              int &sp)
{
    if (c.pass) {
        typename P::Ent k;
        k.a = c.a;
        k.b = c.b;
        k.t_lo = c.t_lo;
        k.depth = depth;
        stack[sp + c.n - 1 - c.rank] = k;
    }
    sp += c.n;
    __syncwarp(Q.mask);
}

// The Newton runs of a last expansion's children, together, and their roots
// taken in sorted order. `ray(o, d)` gives the ray; the lane that holds a
// nearer root hands it to on_root(found), and its t becomes t_max for the
// whole quad. Returns true when `any_hit` and a root was taken.
template <class P, bool ST, class Ray, class OnRoot>
__device__ __forceinline__ bool newton_children(const Quad &Q, const Child<P> &c, const TriDev &T, const AssetDev &g,
                                                const typename P::Bound &L, const Ray &ray, double t_min, double &t_max,
                                                int i, int j, double polish_cond, bool any_hit, int64_t &iters,
                                                const OnRoot &on_root)
{
    typename P::Root root;
    int64_t it = 0;
    const bool conv = c.pass && P::newton(T, g, L, ray, t_min, t_max, i, j, c.a, c.b, root, it);
    __syncwarp(Q.mask);
    if (!ST && !__any_sync(Q.mask, conv))
        return false;
    for (int k = 0; k < c.n; ++k) {
        bool got = false;
        double t_new = 0.0;
        if (c.pass && c.rank == k && (double)c.t_lo < t_max) {
            if (ST)
                iters += it;
            Found f;
            if (conv && P::judge(T, g, L, ray, t_min, t_max, i, j, root, polish_cond, f, iters)) {
                t_new = f.t;
                got = true;
                on_root(f);
            }
        }
        __syncwarp(Q.mask);
        const unsigned w = __ballot_sync(Q.mask, got);
        if (w) {
            // a nearer root of this leaf (each later one is nearer still)
            t_max = __shfl_sync(Q.mask, t_new, __ffs(w) - 1);
            if (any_hit)
                return true;
        }
    }
    return false;
}

} // namespace lq
