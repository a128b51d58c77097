// The FP32 query's launches that must round like the reference, or the same
// way wherever they run (compiled with -fmad=false): the simple schedule, the
// last walk with its leaves inline, the FP64 re-test of parked cells, and the
// leaf rounds of both leaves (the FP32 leaf also runs inline in the last
// walk, so both places round alike and a ray's answer does not depend on the
// round it finishes in).
#include "walk32.cuh"

namespace
{
// The leaf cells of a round's jobs through the reference's own node test in
// double (node_bounds.cpp:83-211 at level 0, the node computed from the
// grid), a lane per cell: the FP32 walk, widened by its roundings, reaches
// more leaf cells than the FP64 walk, and a cell the FP64 walk rejects has no
// leaf there. The ray's t_max is the one it parked with; earlier leaves of
// the same job can only shrink it, so a cell kept here may still be rejected
// by the FP64 walk at that point, and its search then finds nothing the
// reference would not. Kept apart from the leaf kernel so that kernel's code
// stays small.
__global__ void __launch_bounds__(128)
    wave_filter(const TriDev *__restrict__ tris64, const AssetDev *__restrict__ assets, const void *__restrict__ rays,
                dmapk::QueryOpts opt, const RayState *__restrict__ states, LeafJob *__restrict__ q_leaf, int round,
                const unsigned long long *ctr)
{
    const unsigned long long count = 4ull * *round_ctr(const_cast<unsigned long long *>(ctr), round, 1);
    const int lead = threadIdx.x & 28, sub = threadIdx.x & 3;
    for (unsigned long long k = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; k < count;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        LeafJob &job = q_leaf[k >> 2];
        bool admitted = false;
        if (sub < job.n) {
            double t_min, t_max;
            d64::v3 O, D;
            const TriDev &T = tris64[job.tri];
            leaf_ray(rays, opt.ray_dtype, job.ray, opt.inst_xf, T.inst, O, D, t_min, t_max);
            t_max = states[job.ray].t_max;
            admitted = d64::leaf_cell_admitted(T, assets[T.asset], O, D, t_min, t_max, job.i[sub], job.j[sub], opt);
        }
        const unsigned quad = 0xfu << lead;
        __syncwarp(quad);
        const unsigned keep = __ballot_sync(quad, admitted);
        if (sub == 0)
            job.keep = (int)((keep >> lead) & 15u);
    }
}

} // namespace

namespace dmapk
{
namespace w32
{

template <typename R, typename H, typename Fp>
cudaError_t simple(const Args &a, cudaStream_t stream)
{
    const int threads = 128;
    const int64_t blocks = (a.n + threads - 1) / threads;
    walk32_simple<R, H, Fp><<<(unsigned)blocks, threads, 0, stream>>>(
        a.t32, a.t64, a.n_tri, a.assets, static_cast<const R *>(a.rays), a.n, a.opt, static_cast<H *>(a.hits),
        a.stats, a.status);
    return cudaGetLastError();
}

template <typename R, typename H, typename Fp>
cudaError_t simple_rerun(const Args &a, cudaStream_t stream)
{
    const int threads = 128;
    const int64_t blocks = (a.n + threads - 1) / threads;
    walk32_simple<R, H, Fp><<<(unsigned)blocks, threads, 0, stream>>>(
        a.t32, a.t64, a.n_tri, a.assets, static_cast<const R *>(a.rays), a.n, a.opt, static_cast<H *>(a.hits),
        a.stats, a.status, a.rerun, a.counters + 4 * (kMaxRounds + 1));
    return cudaGetLastError();
}

cudaError_t walk_drain(const Args &a, const int *q_in, int round, cudaStream_t stream)
{
    const bool nearest = a.opt.order == 1, tree = a.n_tri > 32 * kMaskWords;
    RayState *states = static_cast<RayState *>(a.states);
    LeafJob *leaves = static_cast<LeafJob *>(a.leaves);
    const size_t bytes = entry_bytes(a.n_tri);
    cudaError_t e = cudaSuccess;
    auto run = [&](auto *kernel, int64_t *stats) {
        e = bytes > 0 ? allow_entries(kernel) : cudaSuccess;
        if (e == cudaSuccess)
            kernel<<<a.grid, 128, bytes, stream>>>(a.t32, a.t64, a.n_tri, a.assets, a.rays, a.n, a.opt, a.hits, stats,
                                                   states, q_in, round, leaves, a.counters, a.status, a.rerun);
    };
#define DMAP_DRAIN(ST_, TR_, NR_, DP_) run(wave_walk<ST_, true, TR_, NR_, DP_>, ST_ ? a.stats : nullptr)
#define DMAP_DRAIN_DEEP(ST_, TR_, NR_)                                                                              \
    (ST_ || a.opt.deep ? DMAP_DRAIN(ST_, TR_, NR_, true) : DMAP_DRAIN(false, TR_, NR_, false))
#define DMAP_DRAIN_MODE(ST_)                                                                                        \
    (tree ? (nearest ? DMAP_DRAIN_DEEP(ST_, true, true) : DMAP_DRAIN_DEEP(ST_, true, false))                        \
          : (nearest ? DMAP_DRAIN_DEEP(ST_, false, true) : DMAP_DRAIN_DEEP(ST_, false, false)))
    if (a.stats)
        DMAP_DRAIN_MODE(true);
    else
        DMAP_DRAIN_MODE(false);
#undef DMAP_DRAIN_MODE
#undef DMAP_DRAIN_DEEP
#undef DMAP_DRAIN
    return e != cudaSuccess ? e : cudaGetLastError();
}

cudaError_t filter(const Args &a, int round, cudaStream_t stream)
{
    wave_filter<<<a.filter_grid, 128, 0, stream>>>(a.t64, a.assets, a.rays, a.opt, static_cast<RayState *>(a.states),
                                                   static_cast<LeafJob *>(a.leaves), round, a.counters);
    return cudaGetLastError();
}

cudaError_t leaves(const Args &a, int round, int *q_out, cudaStream_t stream)
{
    RayState *states = static_cast<RayState *>(a.states);
    const LeafJob *jobs = static_cast<const LeafJob *>(a.leaves);
#define DMAP_LEAVES(ST_, P_)                                                                                        \
    wave_leaf<ST_, P_><<<a.leaf_grid, kLeafThreads, 0, stream>>>(a.t32, a.t64, a.assets, a.rays, a.opt, a.hits,     \
                                                                 ST_ ? a.stats : nullptr, states, jobs, round,      \
                                                                 q_out, a.counters, a.rerun)
    if (a.opt.leaf_precision == 1) // the FP32 certified leaf
        a.stats ? DMAP_LEAVES(true, lq::P32) : DMAP_LEAVES(false, lq::P32);
    else
        a.stats ? DMAP_LEAVES(true, lq::P64) : DMAP_LEAVES(false, lq::P64);
#undef DMAP_LEAVES
    return cudaGetLastError();
}

#define DMAP_W32_EXACT(R, H, Fp)                                                                                    \
    template cudaError_t simple<R, H, Fp>(const Args &, cudaStream_t);                                              \
    template cudaError_t simple_rerun<R, H, Fp>(const Args &, cudaStream_t);
DMAP_W32_EXACT(float, dmapdev::Hit32, float)
DMAP_W32_EXACT(float, dmapdev::Hit64, double)
DMAP_W32_EXACT(double, dmapdev::Hit32, float)
DMAP_W32_EXACT(double, dmapdev::Hit64, double)
#undef DMAP_W32_EXACT

} // namespace w32
} // namespace dmapk
