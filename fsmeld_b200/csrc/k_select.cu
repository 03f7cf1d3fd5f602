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
//     at most the true k-th distance survives both admissible bounds.  Where
//     a bound equals the distance (narrow bands, flat runs) its sum, taken in
//     another order, can round above it, so tau is the k-th distance and a
//     little more (raise);
//  4. a lexicographic sort of the surviving (distance, index) pairs gives the
//     ranking and the threshold.
#include <cfloat>

#include <cub/block/block_merge_sort.cuh>

#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

// A block takes 2048 windows and appends its survivors, in order, with one
// atomic: one per warp (2^23 windows: 262,144 on one address) took 0.15 ms where
// reading the bounds takes 0.02.
__global__ void __launch_bounds__(256) k_lb_filter(Geom g, const double* __restrict__ z,
                                                   const double* __restrict__ SIG,
                                                   const double* __restrict__ cutoff_dev, int metric,
                                                   long long* out, unsigned long long* n_out, long long cap) {
    constexpr int kPer = 8;
    __shared__ unsigned s_mask[kPer * 8];
    __shared__ unsigned long long s_base;
    const double cutoff = *cutoff_dev;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (long long base = (long long)blockIdx.x * 256 * kPer; base < g.tsn; base += (long long)gridDim.x * 256 * kPer) {
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const long long gi = base + u * 256 + threadIdx.x;
            bool keep = false;
            if (gi < g.tsn) {
                long long s;
                int j;
                g.locate(gi, &s, &j);
                const double sg = SIG[s * g.kml + j];
                keep = !window_invalid(sg, g, gi) && !lbip_exceeds(z[s * g.kml + j], cutoff, metric);
            }
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) s_mask[u * 8 + warp] = mask;
        }
        __syncthreads();
        // survivors before each of the 64 words
        const int c0 = __popc(s_mask[2 * lane]), c1 = __popc(s_mask[2 * lane + 1]);
        int inc = c0 + c1;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        const int total = __shfl_sync(0xffffffffu, inc, 31);
        if (threadIdx.x == 0) s_base = total ? atomicAdd(n_out, (unsigned long long)total) : 0ull;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int wd = u * 8 + warp;
            const int before = __shfl_sync(0xffffffffu, inc - c0 - c1, wd >> 1) +
                               ((wd & 1) ? __shfl_sync(0xffffffffu, c0, wd >> 1) : 0);
            const unsigned mask = s_mask[wd];
            if (mask >> lane & 1u) {
                const unsigned long long o = s_base + before + __popc(mask & ((1u << lane) - 1));
                if (o < (unsigned long long)cap) out[o] = base + u * 256 + threadIdx.x;
            }
        }
        __syncthreads();
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
    __shared__ MinZ s_best[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // few stretches: the whole block on each, else a warp each
    const bool whole = per_seg < 8;
    const int t0 = whole ? (int)threadIdx.x : lane, step = whole ? 256 : 32;
    for (long long s = blockIdx.x; s < g.S; s += gridDim.x) {
        const int lo = g.lo(s), len = (g.kml - lo + per_seg - 1) / per_seg;
        for (int p = whole ? 0 : warp; p < per_seg; p += whole ? 1 : 8) {
            const int j0 = lo + p * len, j1 = min(g.kml, j0 + len);
            MinZ best{INFINITY, -1};
            for (int j = j0 + t0; j < j1; j += step) {
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
            if (whole) {
                if (lane == 0) s_best[warp] = best;
                __syncthreads();
                for (int i = 0; i < 8; ++i) {
                    const MinZ c = s_best[i];
                    if (c.gi >= 0) best = best.gi < 0 ? c : MinZOp()(best, c);
                }
                __syncthreads();
            }
            if (lane == 0 && (!whole || warp == 0) && best.gi >= 0) {
                const unsigned long long o = atomicAdd(n_out, 1ull);
                if (o < (unsigned long long)cap) out[o] = best.gi;
            }
        }
    }
}

namespace {

struct Pair {
    double d;
    long long x;
};
struct PairLess {
    __device__ bool operator()(const Pair& a, const Pair& b) const { return a.d < b.d || (a.d == b.d && a.x < b.x); }
};
using PairSort = cub::BlockMergeSort<Pair, kFinishThreads, kFinishSort / kFinishThreads>;

// n pairs of shared memory in ascending (distance, index) order: up to 1024 by
// counting the smaller ones of each (no barriers; 6 us at 1024), a merge sort of
// all kFinishSort slots beyond (45 us).  Pairs are distinct.
__device__ void sort_pairs(Pair* __restrict__ v, int n, PairSort::TempStorage& tmp) {
    constexpr int kPer = kFinishSort / kFinishThreads;
    if (n > 2 * kFinishThreads) {
        Pair own[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            const int i = threadIdx.x * kPer + k;
            own[k] = i < n ? v[i] : Pair{INFINITY, 0x7fffffffffffffffLL};
        }
        __syncthreads();
        PairSort(tmp).Sort(own, PairLess());
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) v[threadIdx.x * kPer + k] = own[k];
        __syncthreads();
        return;
    }
    const int i0 = threadIdx.x, i1 = i0 + kFinishThreads;
    const Pair a = i0 < n ? v[i0] : Pair{INFINITY, 0}, b = i1 < n ? v[i1] : Pair{INFINITY, 0};
    int ra = 0, rb = 0;
    if ((i0 & ~31) < n)
        for (int j = 0; j < n; ++j) {
            const Pair c = v[j];
            ra += PairLess()(c, a) ? 1 : 0;
            rb += PairLess()(c, b) ? 1 : 0;
        }
    __syncthreads();
    if (i0 < n) v[ra] = a;
    if (i1 < n) v[rb] = b;
    __syncthreads();
}

// A bound for the filters from a distance: more than the roundings that a lower
// bound's sum of up to 2 m terms may lie above the distance's by (2^-30 is over a
// hundred times that at m = 16384; the absolute term covers squares that underflow).
__device__ double raise(double d) { return d < 1e300 ? d * (1.0 + 0x1p-30) + 1e-150 : d; }

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
    Pair* v = (Pair*)fin_smem;
    PairSort::TempStorage& tmp = *reinterpret_cast<PairSort::TempStorage*>(v + kFinishSort);
    for (int i = threadIdx.x; i < ncnt; i += blockDim.x) host->cnt[i] = cnt[i];
    const unsigned long long n_all = cnt[out_slot];
    const int n = n_all < (unsigned long long)cap ? (int)min(n_all, (unsigned long long)kFinishSort + 1)
                                                  : (int)min(cap, (long long)kFinishSort + 1);
    if (n > kFinishSort) return;
    // by index: the distances ride along in idx order (a second read)
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = Pair{lex ? dist[i] : 0.0, lex ? idx[i] : idx[i] << 13 | i};
    __syncthreads();
    sort_pairs(v, n, tmp);
    double keep[kFinishSort / kFinishThreads];
    if (!lex) {
#pragma unroll
        for (int u = 0; u < kFinishSort / kFinishThreads; ++u) {
            const int i = threadIdx.x + u * kFinishThreads;
            keep[u] = i < n && dist ? dist[v[i].x & 8191] : 0.0;
        }
        __syncthreads();  // every distance is read before its place is written
    }
#pragma unroll
    for (int u = 0; u < kFinishSort / kFinishThreads; ++u) {
        const int i = threadIdx.x + u * kFinishThreads;
        if (i >= n) continue;
        const long long x = lex ? v[i].x : v[i].x >> 13;
        const double d = lex ? v[i].d : keep[u];
        idx[i] = x;
        if (dist) dist[i] = d;
        if (i < kFinishOut) {
            host->idx[i] = x;
            host->dist[i] = d;
        }
    }
}

// Up to kFinishSort matches in window order into the caller's buffers; *total
// is their number, or kFinishSort + 1 or more when they are left as they are.
__global__ void __launch_bounds__(kFinishThreads) k_order(const unsigned long long* __restrict__ n_in,
                                                          const long long* __restrict__ idx,
                                                          const double* __restrict__ dist,
                                                          long long* __restrict__ out_idx,
                                                          double* __restrict__ out_dist, long long cap,
                                                          unsigned long long* __restrict__ total) {
    extern __shared__ __align__(16) unsigned char ord_smem[];
    Pair* v = (Pair*)ord_smem;
    PairSort::TempStorage& tmp = *reinterpret_cast<PairSort::TempStorage*>(v + kFinishSort);
    const unsigned long long n_all = *n_in;
    if (threadIdx.x == 0) *total = n_all;
    if (n_all > (unsigned long long)kFinishSort) return;
    const int n = (int)n_all;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = Pair{0.0, idx[i] << 13 | i};
    __syncthreads();
    sort_pairs(v, n, tmp);
    for (int i = threadIdx.x; i < n && i < cap; i += blockDim.x) {
        out_idx[i] = v[i].x >> 13;
        out_dist[i] = dist[v[i].x & 8191];
    }
}

// The bound tau (the k-th smallest seed distance, raised; DBL_MAX with fewer than k
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
    Pair* v = (Pair*)tau_smem;
    PairSort::TempStorage& tmp = *reinterpret_cast<PairSort::TempStorage*>(v + kFinishSort);
    const long long n_all = min((long long)*n_seed, cap);
    const int n = (int)min(n_all, (long long)kFinishSort);
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = Pair{dist[i], idx[i]};
    if (threadIdx.x == 0) s_np = s_n = 0;
    __syncthreads();
    if (!sorted) sort_pairs(v, n, tmp);
    if (threadIdx.x == 0) *tau = k <= n_all ? raise(k <= n ? v[k - 1].d : dist[k - 1]) : DBL_MAX;
    if (!picks) return;
    if (threadIdx.x < 32) {
        // best first, 32 seeds at a time: those that clash with no pick so far,
        // then the first of them again and again
        int np = 0;
        const int lane = threadIdx.x;
        for (int i0 = 0; i0 < min(n, 8 * kRefinePicks) && np < picks; i0 += 32) {
            const bool in = i0 + lane < n;
            const long long x = in ? v[i0 + lane].x : 0;
            auto near = [&](long long c) { return x - c <= 2 * kRefineReach && c - x <= 2 * kRefineReach; };
            bool free = in;
            for (int q = 0; q < np; ++q) free = free && !near(s_pick[q]);
            unsigned left = __ballot_sync(0xffffffffu, free);
            while (left && np < picks) {
                const long long c = __shfl_sync(0xffffffffu, x, __ffs(left) - 1);
                if (lane == 0) s_pick[np] = c;
                ++np;
                free = free && !near(c);
                left = __ballot_sync(0xffffffffu, free);
            }
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
    Pair* v = (Pair*)ref_smem;
    PairSort::TempStorage& tmp = *reinterpret_cast<PairSort::TempStorage*>(v + kFinishSort);
    const int n = (int)min(*n_dist, (unsigned long long)kFinishSort);
    if (k > n) return;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v[i] = Pair{dist[i], i};
    __syncthreads();
    sort_pairs(v, n, tmp);
    if (threadIdx.x == 0) *tau = fmin(*tau, raise(v[k - 1].d));
}

size_t finish_smem_bytes() { return sizeof(Pair) * kFinishSort + sizeof(PairSort::TempStorage) + 16; }

}  // namespace fsm
