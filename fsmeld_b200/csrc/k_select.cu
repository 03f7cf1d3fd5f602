// Candidate selection for the top-k `cutoff` command (src/fsmeld.cpp:185-569).
//
// The reference scans candidates in index order with a k-element max-heap of
// (distance, index) pairs and a threshold that tightens as the heap fills;
// since replacement needs a strictly smaller distance and indices arrive in
// increasing order, its result is exactly the k lexicographically smallest
// (distance, index) pairs among valid candidates.  The device form reaches
// the same set without the serial scan:
//  1. LB_IP per window (k_lbip with z output);
//  2. seeds: the windows with the smallest LB of each stretch of each segment
//     (k_seed, ceil(2k/S) stretches per segment, eight on short targets, at
//     most 32, so that there are at least k seeds unless k > 32 S); the k-th
//     smallest exact distance among the seeds is an upper bound tau on the
//     k-th smallest distance overall (with fewer than k seeds there is no
//     bound and every candidate is evaluated); the windows around the best
//     seeds lower it (k_tau_block, k_tau_refine), to the k-th distance itself
//     when the best matches are neighbours of theirs.  Without that step the
//     filters and the DP ran at a bound that left tens of times the
//     candidates;
//  3. every valid window whose LB does not exceed tau (k_lb_filter) goes
//     through GLB at tau and then the exact DP; any window whose distance is
//     at most the true k-th distance survives both admissible bounds;
//  4. a lexicographic sort of the surviving (distance, index) pairs gives the
//     ranking and the threshold.
#include <cfloat>

#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

__global__ void __launch_bounds__(256) k_lb_filter(Geom g, const double* __restrict__ z,
                                                   const double* __restrict__ SIG,
                                                   const double* __restrict__ cutoff_dev, int metric,
                                                   long long* out, unsigned long long* n_out, long long cap) {
    const double cutoff = *cutoff_dev;
    const int lane = threadIdx.x & 31;
    for (long long base = (long long)blockIdx.x * blockDim.x; base < g.tsn;
         base += (long long)gridDim.x * blockDim.x) {
        const long long gi = base + threadIdx.x;
        bool keep = false;
        if (gi < g.tsn) {
            long long s;
            int j;
            g.locate(gi, &s, &j);
            const double sg = SIG[s * g.kml + j];
            keep = !window_invalid(sg, g, gi) && !lbip_exceeds(z[s * g.kml + j], cutoff, metric);
        }
        const unsigned mask = __ballot_sync(0xffffffffu, keep);
        if (mask) {
            unsigned long long o = 0;
            const int leader = __ffs(mask) - 1;
            if (lane == leader) o = atomicAdd(n_out, (unsigned long long)__popc(mask));
            o = __shfl_sync(0xffffffffu, o, leader) + __popc(mask & ((1u << lane) - 1));
            if (keep && o < (unsigned long long)cap) out[o] = gi;
        }
    }
}

struct MinZ {
    double z;
    long long gi;
};
struct MinZOp {
    __device__ MinZ operator()(const MinZ& a, const MinZ& b) const {
        if (a.z < b.z) return a;
        if (b.z < a.z) return b;
        return (a.gi <= b.gi) ? a : b;
    }
};

// One block per segment, cut into per_seg stretches of windows: the valid
// window with the smallest LB of each stretch (ties: lowest index), one pass
// over the bounds.
__global__ void __launch_bounds__(256) k_seed(Geom g, const double* __restrict__ z,
                                              const double* __restrict__ SIG, int per_seg,
                                              long long* out, unsigned long long* n_out, long long cap) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long s = blockIdx.x; s < g.S; s += gridDim.x) {
        const int lo = g.lo(s), len = (g.kml - lo + per_seg - 1) / per_seg;
        for (int p = warp; p < per_seg; p += 8) {
            const int j0 = lo + p * len, j1 = min(g.kml, j0 + len);
            MinZ best{INFINITY, -1};
            for (int j = j0 + lane; j < j1; j += 32) {
                const long long gi = g.gidx(s, j);
                if (window_invalid(SIG[s * g.kml + j], g, gi)) continue;
                const double zz = z[s * g.kml + j];
                const MinZ c{isnan(zz) ? INFINITY : zz, gi};
                best = best.gi < 0 ? c : MinZOp()(best, c);
            }
            for (int o = 16; o; o >>= 1) {
                const MinZ c{__shfl_xor_sync(0xffffffffu, best.z, o), __shfl_xor_sync(0xffffffffu, best.gi, o)};
                if (c.gi >= 0) best = best.gi < 0 ? c : MinZOp()(best, c);
            }
            if (lane == 0 && best.gi >= 0) {
                const unsigned long long o = atomicAdd(n_out, 1ull);
                if (o < (unsigned long long)cap) out[o] = best.gi;
            }
        }
    }
}

namespace {

// (key, index) pairs of shared memory in ascending order, n2 a power of two
template <typename Less>
__device__ void bitonic(int n2, Less less, double* __restrict__ d, long long* __restrict__ x) {
    for (int k = 2; k <= n2; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < n2; i += blockDim.x) {
                const int o = i ^ j;
                if (o > i) {
                    const double da = d[i], db = d[o];
                    const long long xa = x[i], xb = x[o];
                    if (less(db, xb, da, xa) == ((i & k) == 0)) {
                        d[i] = db; d[o] = da;
                        x[i] = xb; x[o] = xa;
                    }
                }
            }
            __syncthreads();
        }
}

}  // namespace

// The end of a query in one block: up to kFinishSort results in their order (by
// index, or by distance and index), in place, the first kFinishOut of them and
// the counters also in host memory the device can write, so that the host waits
// once and copies nothing.  More results are left as they are (the host sorts
// them by radix).
__global__ void __launch_bounds__(kFinishThreads) k_finish(const unsigned long long* __restrict__ cnt, int ncnt,
                                                           int out_slot, long long cap, int lex,
                                                           long long* __restrict__ idx, double* __restrict__ dist,
                                                           FinishOut* __restrict__ host) {
    extern __shared__ __align__(16) unsigned char fin_smem[];
    double* d = (double*)fin_smem;
    long long* x = (long long*)(d + kFinishSort);
    for (int i = threadIdx.x; i < ncnt; i += blockDim.x) host->cnt[i] = cnt[i];
    const unsigned long long n_all = cnt[out_slot];
    const int n = n_all < (unsigned long long)cap ? (int)min(n_all, (unsigned long long)kFinishSort + 1)
                                                  : (int)min(cap, (long long)kFinishSort + 1);
    if (n > kFinishSort) return;
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (int i = threadIdx.x; i < n2; i += blockDim.x) {
        d[i] = i < n ? (dist ? dist[i] : 0.0) : INFINITY;
        x[i] = i < n ? idx[i] : 0x7fffffffffffffffLL;
    }
    __syncthreads();
    if (lex)
        bitonic(n2, [](double da, long long xa, double db, long long xb) { return da < db || (da == db && xa < xb); },
                d, x);
    else
        bitonic(n2, [](double, long long xa, double, long long xb) { return xa < xb; }, d, x);
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        idx[i] = x[i];
        if (dist) dist[i] = d[i];
        if (i < kFinishOut) {
            host->idx[i] = x[i];
            host->dist[i] = d[i];
        }
    }
}

// The bound tau (the k-th smallest seed distance, DBL_MAX with fewer than k
// seeds) and the windows to refine it with.  Seeds lie at the smallest bound of
// their stretch; the windows next to a good match are good matches too, and
// most of the ranking usually, so the kRefineReach windows on either side of
// the best seeds are evaluated next.  The seeds taken lie more than twice the
// reach apart, so no window is listed twice and the k-th smallest of their
// distances is a bound again (k_tau_refine).  sorted: the seeds are in
// ascending order, else there are at most kFinishSort of them.
__global__ void __launch_bounds__(kFinishThreads) k_tau_block(const double* __restrict__ dist,
                                                              const long long* __restrict__ idx, int sorted,
                                                              const unsigned long long* __restrict__ n_seed,
                                                              long long cap, long long k, long long tsn, int picks,
                                                              double* tau, long long* __restrict__ list,
                                                              unsigned long long* __restrict__ n_list) {
    extern __shared__ __align__(16) unsigned char tau_smem[];
    __shared__ long long s_pick[kRefinePicks];
    __shared__ int s_np, s_n;
    double* d = (double*)tau_smem;
    long long* x = (long long*)(d + kFinishSort);
    const long long n_all = min((long long)*n_seed, cap);
    const int n = (int)min(n_all, (long long)kFinishSort);
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (int i = threadIdx.x; i < n2; i += blockDim.x) {
        d[i] = i < n ? dist[i] : INFINITY;
        x[i] = i < n ? idx[i] : 0x7fffffffffffffffLL;
    }
    if (threadIdx.x == 0) s_np = s_n = 0;
    __syncthreads();
    if (!sorted)
        bitonic(n2, [](double da, long long xa, double db, long long xb) { return da < db || (da == db && xa < xb); },
                d, x);
    if (threadIdx.x == 0) *tau = k <= n_all ? (k <= n ? d[k - 1] : dist[k - 1]) : DBL_MAX;
    if (!picks) return;
    if (threadIdx.x < 32) {
        int np = 0;
        for (int i = 0; i < min(n, 8 * kRefinePicks) && np < picks; ++i) {
            bool clash = false;
            for (int q = threadIdx.x; q < np; q += 32) {
                const long long gap = x[i] - s_pick[q];
                clash = clash || (gap <= 2 * kRefineReach && gap >= -2 * kRefineReach);
            }
            if (__any_sync(0xffffffffu, clash)) continue;
            if (threadIdx.x == 0) s_pick[np] = x[i];
            ++np;
            __syncwarp();
        }
        if (threadIdx.x == 0) s_np = np;
    }
    __syncthreads();
    constexpr int kSpan = 2 * kRefineReach + 1;
    for (int e = threadIdx.x; e < s_np * kSpan; e += blockDim.x) {
        const long long w = s_pick[e / kSpan] + e % kSpan - kRefineReach;
        if (w >= 0 && w < tsn) list[atomicAdd(&s_n, 1)] = w;
    }
    __syncthreads();
    if (threadIdx.x == 0) *n_list = (unsigned long long)s_n;
}

// tau lowered to the k-th smallest of the refining distances
__global__ void __launch_bounds__(kFinishThreads) k_tau_refine(const double* __restrict__ dist,
                                                               const unsigned long long* __restrict__ n_dist,
                                                               long long k, double* tau) {
    extern __shared__ __align__(16) unsigned char ref_smem[];
    double* d = (double*)ref_smem;
    long long* x = (long long*)(d + kFinishSort);
    const int n = (int)min(*n_dist, (unsigned long long)kFinishSort);
    if (k > n) return;
    int n2 = 1;
    while (n2 < n) n2 <<= 1;
    for (int i = threadIdx.x; i < n2; i += blockDim.x) {
        d[i] = i < n ? dist[i] : INFINITY;
        x[i] = 0;
    }
    __syncthreads();
    bitonic(n2, [](double da, long long, double db, long long) { return da < db; }, d, x);
    if (threadIdx.x == 0 && d[k - 1] < *tau) *tau = d[k - 1];
}

}  // namespace fsm
