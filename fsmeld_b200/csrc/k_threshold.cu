// LB_IP threshold selection per macro segment and side
// (src/find_t_lp.cpp: find_tl_lp_dtw 218-287, find_tl_lp 288-398,
//  find_tl_lp_erp 510-582, find_tu_lp_erp 583-654, find_tu_lp_dtw 655-724,
//  find_tu_lp 726-825; dispatch src/fsmeld.cpp:778-790).
//
// The reference: run-length dedup of the envelope core U/L_normal[m-1 ..
// m_k-m] (consecutive equal values only), sort, then one sequential sweep
// that moves pointers over the sorted query, updates running power sums m_p
// and a penalty sum C, and scores LB[i] = h(t_i) * g_i; the argmax gives t.
//
// Here one CTA handles one (segment, side):
//  1. dedup with a block scan, then the runs are sorted (total order: value,
//     NaN last, ties by position): every run is counted into one of two
//     buckets per run slot, equal in width over the values' range, and ranked
//     by comparison with the few other runs of its bucket.  That took half of
//     the kernel as a block merge sort of (64-bit key, run) pairs, which
//     stays for values bunched in a few buckets (over kBucketMost in one);
//  2. every pointer move of the sweep becomes an op with the sweep step at
//     which it fires (a binary search over the sorted values); ops are
//     ordered by (step, stream, rank) -- the order the reference's loops
//     perform them in;
//  3. the ops are replayed in that order, so m_p and C carry the reference's
//     rounding bit for bit: lane j of warp 0 owns accumulator j (m_0..m_2, C)
//     and adds each op's operand, pre-signed for it, recording the state
//     after each op;
//  4. every candidate reads its state, scores LB in parallel, and a block
//     reduction takes the first maximum (NaN at index 0 wins, as in
//     findMaxIndex, src/find_t_lp.cpp:206-216).
// Several blocks per SM hide each other's serial phases (the sums before the
// sweep and the replay, 11 cycles an add); the sort is a quarter of what is left.
// Measured, five queries on 2^24 points (m = 256): 11.5 ms with the merge sort,
// predicated chains and a quadratic op order for ERP; 5.9 ms with buckets; 4.5 ms
// with the runs found by ballots, a bucket's values side by side and the counts
// of ops kept for every 32nd step.  20 queries of mixed length on 2^22 points,
// most with 8192-point segments that used to lie in global scratch: 17.6, 8.9,
// 7.3 ms.
// ERP's priority queues pop equal keys in an order the C++ library leaves
// to its heap layout; here equal keys pop by query index.  The threshold is
// the same unless two candidates' scores tie to the last bit.
#include <climits>
#include <cub/block/block_merge_sort.cuh>
#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>

#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

namespace {

constexpr int kNever = INT_MAX;
constexpr int kBucketMost = 24;  // runs of one bucket that are ranked by comparison

// Order-preserving key of a double: ascending values map to ascending keys,
// -0 and +0 to one key (they compare equal), NaN to the largest key (sorted
// last); desc reverses the order of the non-NaN values.
__device__ __forceinline__ unsigned long long order_key(double x, int desc) {
    if (isnan(x)) return ~0ull;
    const unsigned long long u = (unsigned long long)__double_as_longlong(x == 0.0 ? 0.0 : x);
    const unsigned long long k = (u >> 63) ? ~u : (u | 0x8000000000000000ull);
    return desc ? ~k : k;
}

struct KeyLess {
    __device__ __forceinline__ bool operator()(const unsigned long long& a, const unsigned long long& b) const {
        return a < b;
    }
};

struct ArgMax {
    double v;
    int i;
    int ok;  // 0 for NaN scores (never selected unless at index 0)
};
struct ArgMaxOp {
    __device__ ArgMax operator()(const ArgMax& a, const ArgMax& b) const {
        if (!a.ok) return b;
        if (!b.ok) return a;
        if (a.v > b.v) return a;
        if (b.v > a.v) return b;
        return (a.i <= b.i) ? a : b;
    }
};

enum Cmp { LE, LT, GE, GT };

// first i in [0, n) with tv[i] (cmp) x, or kNever; tv is monotone so the
// predicate is false..false true..true
__device__ __forceinline__ int first_step(const double* tv, int n, Cmp c, double x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const double t = tv[mid];
        bool p;
        switch (c) {
            case LE: p = t <= x; break;
            case LT: p = t < x; break;
            case GE: p = t >= x; break;
            default: p = t > x; break;
        }
        if (p) hi = mid; else lo = mid + 1;
    }
    return lo < n ? lo : kNever;
}

// prefix length of an index-ordered table whose keys satisfy pred (monotone)
template <typename F>
__device__ __forceinline__ int prefix_count(int n, F pred) {
    int lo = 0, hi = n;
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (pred(mid)) lo = mid + 1; else hi = mid; }
    return lo;
}

__device__ __forceinline__ double f_p(double mp0, double mp1, double mp2, int p, double t) {
    // src/find_t_lp.cpp:187-199 (p == 0 only occurs for EDR/LCSS, which return 0)
    if (p == 0) return 0.0;
    if (p == 1) return dsub(mp1, dmul(mp0, t));
    return dadd(dsub(mp2, dmul(dmul(mp1, t), 2.0)), dmul(mp0, dmul(t, t)));
}

// Stream plan of one (metric, side): op element, step, payload kind.
struct Plan {
    int kind;      // 0 DTW, 1 general (MSM, EDR, LCSS), 2 ERP
    int upper;
    int idx1, idx2, kA0, kB0;
    int nA, nB;
    int p;
};

}  // namespace

// Block working set: region R, the runs (values and starts) and, in the same
// place once the runs are in registers, the sorted values and counts; region Z,
// the sort's temporaries and after it the sweep (op steps, op order,
// operand/state slots).  Segments of up to 8192 core values keep both in shared
// memory; longer ones keep R in global scratch with a second area for the
// sorted values, and Z in shared memory when it fits.
__host__ __device__ constexpr size_t thr_round16(size_t b) { return (b + 15) & ~size_t(15); }
// counts and the bucket sort's counters are walked in runs of a few per thread:
// one spare slot in 32 puts the walks on distinct banks
__host__ __device__ constexpr int thr_pad(int i) { return i + (i >> 5); }
__host__ __device__ constexpr size_t thr_r_bytes(int cap) {
    return thr_round16((size_t)cap * 8 + ((size_t)thr_pad(cap) + 2) * 4);
}
constexpr int kChainPad = 32;  // slots past the last op: a whole chunk and the loads ahead
__host__ __device__ inline size_t thr_z_bytes(int m) { return (size_t)m * 24 + 16 + (size_t)(2 * m + kChainPad) * 32; }
__host__ __device__ constexpr size_t thr_bucket_bytes(int cap, int nb) {
    return thr_round16(((size_t)thr_pad(nb) + 1) * 4 + (size_t)cap * 2);
}
__host__ __device__ constexpr int thr_buckets(int cap, bool gw) { return gw ? cap : 2 * cap; }

// acc plus n operands in order, 4 doubles apart, the sum left in each operand's
// place if STORE; operands up to the next multiple of 16 leave the sum as it
// is.  A serial chain of additions: 8 operands are loaded under the 8 additions
// before theirs, at fixed distances and without a test, up to 8 past the end.
// (Strides and ends known only at run time cost 22 cycles an addition, these 11.)
template <bool STORE>
__device__ __forceinline__ double chain(double acc, double* p, int n) {
    double a[8], b[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) a[u] = p[4 * u];
#pragma unroll 1
    for (int i = 0; i < n; i += 16, p += 64) {
#pragma unroll
        for (int u = 0; u < 8; ++u) b[u] = p[4 * (u + 8)];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            acc = dadd(acc, a[u]);
            if (STORE) p[4 * u] = acc;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) a[u] = p[4 * (u + 16)];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            acc = dadd(acc, b[u]);
            if (STORE) p[4 * (u + 8)] = acc;
        }
    }
    return acc;
}

// The runs sorted by a block merge sort (thread t on runs t IPT ..) into the
// sorted values and counts; in a function of its own for its registers.
template <int T, int IPT>
__device__ __noinline__ void merge_runs(typename cub::BlockMergeSort<unsigned long long, T, IPT, int>::TempStorage& tmp,
                                        const double* rval, const int* rstart, double* tv, int* gp, int nr,
                                        int upper) {
    const int t = threadIdx.x;
    unsigned long long keys[IPT];
    int rid[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int r = t * IPT + k;
        keys[k] = r < nr ? order_key(rval[r], upper ? 0 : 1) : ~0ull;  // padding after every run
        rid[k] = r;
    }
    __syncthreads();
    cub::BlockMergeSort<unsigned long long, T, IPT, int>(tmp).StableSort(keys, rid, KeyLess());
    __syncthreads();
    double rv[IPT];
#pragma unroll
    for (int k = 0; k < IPT; ++k) {
        const int r = t * IPT + k < nr ? rid[k] : 0;
        rv[k] = rval[r];
        rid[k] = rstart[r + 1] - rstart[r];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < IPT; ++k)
        if (t * IPT + k < nr) {
            tv[t * IPT + k] = rv[k];
            gp[thr_pad(t * IPT + k)] = rid[k];
        }
}

// 1024 / T blocks per SM: at most 64 registers a thread, so that several
// blocks hide each other's serial phases
template <int T, int IPT, bool GW>
__global__ void __launch_bounds__(T, 1024 / T) k_threshold(Geom g, ThrJob job, unsigned char* gwork,
                                                                   long long slot_stride, int z_shared) {
    using Sort = cub::BlockMergeSort<unsigned long long, T, IPT, int>;
    using IScan = cub::BlockScan<int, T>;
    using AReduce = cub::BlockReduce<ArgMax, T>;
    constexpr int CAP = T * IPT, NW = T / 32;

    extern __shared__ __align__(16) unsigned char thr_smem[];
    __shared__ typename IScan::TempStorage iscan_tmp;
    __shared__ typename AReduce::TempStorage red_tmp;
    __shared__ int s_nfin, s_best, s_nops;
    __shared__ int s_cnt[2];
    __shared__ unsigned s_ext[64];
    __shared__ int s_wc[NW * IPT];
    __shared__ int s_lo[CAP / 32 + 2];

    const QueryDev& q = job.q;
    const int m = q.m, mk = g.m_k;
    const int cnt = mk - 2 * m + 2;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;

    // GW: region R in global scratch; otherwise provably shared memory
    constexpr size_t RB = thr_r_bytes(CAP);
    unsigned char* base = GW ? gwork + (long long)blockIdx.x * slot_stride
                                : thr_smem;
    double* rval = (double*)base;                        // [CAP]
    int* rstart = (int*)(base + (size_t)CAP * 8);        // [CAP + 1]
    double* tv = (double*)(GW ? base + RB : base);       // [CAP] sorted values, over the runs
    int* gp = (int*)((GW ? base + RB : base) + (size_t)CAP * 8);  // [thr_pad(CAP)] inclusive count sums
    unsigned char* zb = GW ? (z_shared ? thr_smem : base + 2 * RB) : thr_smem + RB;
    // the sorts' temporaries (shared memory in every form)
    unsigned char* sortb = GW ? thr_smem : thr_smem + RB;
    typename Sort::TempStorage& sort_tmp = *reinterpret_cast<typename Sort::TempStorage*>(sortb);
    constexpr int NB = thr_buckets(CAP, GW);
    int* bcnt = (int*)sortb;                                            // [thr_pad(NB) + 1]
    unsigned short* bslot = (unsigned short*)(bcnt + thr_pad(NB) + 1);  // [CAP]
    int* sA = (int*)zb;                                 // [m]
    int* sB = sA + m;                                   // [m]
    int* opdesc = sB + m;                               // [2m]
    int* opstep = opdesc + 2 * m;                       // [2m]
    double* st = (double*)(((uintptr_t)(opstep + 2 * m) + 15) & ~uintptr_t(15));  // [(2m + kChainPad) * 4]

    const int p = q.p;
    const int kind = (q.metric == DTW) ? 0 : (q.metric == ERP ? 2 : 1);

    for (long long bid = blockIdx.x; bid < 2 * g.S; bid += gridDim.x) {
        const long long s = bid >> 1;
        const int upper = (int)(bid & 1);
        const double* env = (upper ? job.Un : job.Ln) + s * mk + (m - 1);

        // ---- 1. run-length dedup (src/find_t_lp.cpp:53-67), value t + k T per
        // thread; the extremes of the finite values as the upper words of their
        // order keys
        double v[IPT];
        unsigned fl = 0, kmn = ~0u, kmx = 0;
#pragma unroll
        for (int k = 0; k < IPT; ++k) v[k] = t + k * T < cnt ? env[t + k * T] : 0.0;
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int i = t + k * T;
            double prev = __shfl_up_sync(0xffffffffu, v[k], 1);
            if (lane == 0 && i > 0 && i < cnt) prev = env[i - 1];
            const bool f = i < cnt && (i == 0 || v[k] != prev);
            const unsigned hw = (unsigned)__double2hiint(v[k]);
            if (i < cnt && (hw & 0x7ff00000u) != 0x7ff00000u) {
                const unsigned key = (hw >> 31) ? ~hw : hw | 0x80000000u;
                kmn = min(kmn, key);
                kmx = max(kmx, key);
            }
            fl |= f ? 1u << k : 0u;
            const int c = __popc(__ballot_sync(0xffffffffu, f));
            if (lane == 0) s_wc[k * NW + wid] = c;
        }
        kmn = __reduce_min_sync(0xffffffffu, kmn);
        kmx = __reduce_max_sync(0xffffffffu, kmx);
        if (lane == 0) { s_ext[wid] = kmn; s_ext[32 + wid] = kmx; }
        for (int i = t; i <= thr_pad(NB); i += T) bcnt[i] = 0;
        __syncthreads();
        kmn = __reduce_min_sync(0xffffffffu, s_ext[min(lane, NW - 1)]);
        kmx = __reduce_max_sync(0xffffffffu, s_ext[32 + min(lane, NW - 1)]);
        int wbase, nr;
        IScan(iscan_tmp).ExclusiveSum(t < NW * IPT ? s_wc[t] : 0, wbase, nr);
        if (t < NW * IPT) s_wc[t] = wbase;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const bool f = (fl >> k) & 1;
            const unsigned bal = __ballot_sync(0xffffffffu, f);
            if (f) {
                const int o = s_wc[k * NW + wid] + __popc(bal & ((1u << lane) - 1));
                rstart[o] = t + k * T;
                rval[o] = v[k];
            }
        }
        if (t == 0) rstart[nr] = cnt;
        __syncthreads();

        // ---- 2. sort runs (src/find_t_lp.cpp:68-81): ascending keys, ties by
        // run; run t + k T is this thread's k-th
        double rv[IPT];
        int rank[IPT], rc[IPT], bk[IPT];
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int r = t + k * T;
            rv[k] = r < nr ? rval[r] : dnan();
            rc[k] = r < nr ? rstart[r + 1] - rstart[r] : 0;
        }
        // buckets of equal width over the finite values (the infinities in the
        // outer ones, NaN in the last): the range and the width are rounded, the
        // order of the buckets is that of the values all the same
        const double vmn = __hiloint2double((int)((kmn >> 31) ? kmn ^ 0x80000000u : ~kmn), (kmn >> 31) ? 0 : -1);
        const double vmx = __hiloint2double((int)((kmx >> 31) ? kmx ^ 0x80000000u : ~kmx), (kmx >> 31) ? -1 : 0);
        const double width = vmx > vmn ? (NB - 1) / (vmx - vmn) : 0.0;
        const double scale = isfinite(width) ? width : 0.0;
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            bk[k] = thr_pad(NB - 1);
            rank[k] = 0;
            if (t + k * T < nr) {
                if (!isnan(rv[k])) {
                    const int bu = isfinite(rv[k]) ? min(NB - 2, (int)dmul(dsub(rv[k], vmn), scale))
                                                   : (rv[k] < 0.0 ? 0 : NB - 2);
                    bk[k] = thr_pad(upper ? bu : NB - 2 - bu);
                }
                rank[k] = atomicAdd(&bcnt[bk[k]], 1);  // place inside the bucket, any order
            }
        }
        __syncthreads();
        constexpr int PER = NB / T;
        int most = 0, bsum = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            const int x = bcnt[thr_pad(t * PER + i)];
            most = max(most, x);
            bsum += x;
        }
        if (t == T - 1) s_nfin = nr - bcnt[thr_pad(NB - 1)];  // the last bucket holds the NaN
        int bbase;
        IScan(iscan_tmp).ExclusiveSum(bsum, bbase);
        if (!__syncthreads_or(most > kBucketMost)) {
#pragma unroll
            for (int i = 0; i < PER; ++i) {
                const int x = bcnt[thr_pad(t * PER + i)];
                bcnt[thr_pad(t * PER + i)] = bbase;
                bbase += x;
            }
            __syncthreads();
            // the runs by buckets, values over the unsorted ones
#pragma unroll
            for (int k = 0; k < IPT; ++k)
                if (t + k * T < nr) {
                    const int pos = bcnt[bk[k]] + rank[k];
                    tv[pos] = rv[k];
                    bslot[pos] = (unsigned short)(t + k * T);
                }
            __syncthreads();
            // rank inside the bucket by comparison with its runs, four runs'
            // buckets side by side
            constexpr int G = IPT < 4 ? IPT : 4;
#pragma unroll
            for (int k0 = 0; k0 < IPT; k0 += G) {
                int lo[G], num[G], less[G], eq[G], most_here = 0;
#pragma unroll
                for (int u = 0; u < G; ++u) {
                    const int k = k0 + u;
                    less[u] = eq[u] = lo[u] = num[u] = 0;
                    if (t + k * T < nr) {
                        lo[u] = bcnt[bk[k]];
                        const int nb = bk[k] + (bk[k] % 33 == 31 ? 2 : 1);  // the next bucket's slot
                        num[u] = (bk[k] < thr_pad(NB - 1) ? bcnt[nb] : nr) - lo[u];
                    }
                    most_here = max(most_here, num[u]);
                }
                most_here = __reduce_max_sync(0xffffffffu, most_here);
                if (most_here > 1)
#pragma unroll 1
                    for (int i = 0; i < most_here; ++i) {
#pragma unroll
                        for (int u = 0; u < G; ++u) {
                            if (i >= num[u]) continue;
                            const double vo = tv[lo[u] + i];
                            less[u] += (upper ? vo < rv[k0 + u] : vo > rv[k0 + u]) ? 1 : 0;
                            eq[u] += vo == rv[k0 + u] ? 1 : 0;
                        }
                    }
#pragma unroll
                for (int u = 0; u < G; ++u) {
                    if (num[u] > 1 && eq[u] != 1) {  // equal values or NaN: by run
                        const double x = rv[k0 + u];
                        less[u] = 0;
                        for (int i = 0; i < num[u]; ++i) {
                            const double vo = tv[lo[u] + i];
                            const bool before = upper ? vo < x : vo > x, after = upper ? vo > x : vo < x;
                            less[u] += before || (!after && (int)bslot[lo[u] + i] < t + (k0 + u) * T) ? 1 : 0;
                        }
                    }
                    rank[k0 + u] = lo[u] + less[u];
                }
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < IPT; ++k) {
                if (t + k * T < nr) {
                    tv[rank[k]] = rv[k];
                    gp[thr_pad(rank[k])] = rc[k];
                }
            }
        } else {  // values bunched in a few buckets
            merge_runs<T, IPT>(sort_tmp, rval, rstart, tv, gp, nr, upper);
        }
        __syncthreads();

        // ---- 3. cumulative counts g_i, finite prefix length
        int csum = 0;
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int i = t * IPT + k;
            if (i < nr) csum += gp[thr_pad(i)];
        }
        int cbase;
        IScan(iscan_tmp).ExclusiveSum(csum, cbase);
#pragma unroll
        for (int k = 0; k < IPT; ++k) {
            const int i = t * IPT + k;
            if (i < nr) {
                cbase += gp[thr_pad(i)];
                gp[thr_pad(i)] = cbase;
            }
        }
        if (t == 0) { s_cnt[0] = 0; s_cnt[1] = 0; }
        __syncthreads();
        const int nfin = s_nfin;
        double* out = job.thr + s * 2 + upper;
        if (nfin == 0) {  // every score is NaN: index 0 wins
            if (t == 0) *out = tv[0];
            __syncthreads();
            continue;
        }

        // ---- 4. stream plan, src/find_t_lp.cpp init loops: the pointer
        // scans stop at the partition point of a monotone table (sorted
        // query, t_l/t_u of the sorted query, the ERP pop orders), found here
        // as a block-wide count
        const double t0 = tv[0];
        {
            int c0 = 0, c1 = 0;
            for (int j = t; j < m; j += T) {
                if (kind == 0) {
                    c0 += upper ? (q.qs[j] <= t0) : (q.qs[j] < t0);
                } else if (kind == 1) {
                    if (!upper) { c0 += q.qs[j] < t0; c1 += q.tlq[j] < t0; }
                    else { c0 += q.qs[j] <= t0; c1 += q.tuq[j] <= t0; }
                } else {
                    if (!upper) { c0 += q.otl[q.ordA_l[j]] >= t0; c1 += q.qn[q.ordB_l[j]] >= t0; }
                    else { c0 += q.otu[q.ordA_u[j]] <= t0; c1 += q.qn[q.ordB_u[j]] <= t0; }
                }
            }
            for (int o = 16; o; o >>= 1) {
                c0 += __shfl_xor_sync(0xffffffffu, c0, o);
                c1 += __shfl_xor_sync(0xffffffffu, c1, o);
            }
            if ((t & 31) == 0) { atomicAdd(&s_cnt[0], c0); atomicAdd(&s_cnt[1], c1); }
        }
        __syncthreads();
        Plan pl;
        pl.kind = kind; pl.upper = upper; pl.p = p;
        pl.idx1 = pl.idx2 = pl.kA0 = pl.kB0 = 0;
        pl.nA = pl.nB = 0;
        {
            const int c0 = s_cnt[0], c1 = s_cnt[1];
            if (kind == 0) {
                if (!upper) { pl.idx1 = c0 - 1; pl.nB = pl.idx1 + 1; }
                else { pl.idx1 = c0; pl.nB = m - pl.idx1; }
            } else if (kind == 1) {
                if (!upper) {
                    pl.idx1 = c0 - 1;
                    pl.idx2 = min(pl.idx1, c1 - 1);
                    pl.nA = pl.idx2 + 1;
                    pl.nB = pl.idx1 + 1;
                } else {
                    pl.idx1 = c0;
                    pl.idx2 = max(pl.idx1, c1);
                    pl.nA = m - pl.idx2;
                    pl.nB = m - pl.idx1;
                }
            } else {
                pl.kA0 = c0;
                pl.kB0 = c1;
                pl.nA = m - pl.kA0;
                pl.nB = m - pl.kB0;
            }
        }

        // ---- 5. firing step of every op
        for (int r = t; r < pl.nA; r += T) {
            int st_ = kNever;
            if (kind == 1) {
                if (!upper) { const int j = pl.idx2 - r; st_ = first_step(tv, nfin, LE, q.tlq[j]); }
                else { const int j = pl.idx2 + r; st_ = first_step(tv, nfin, GE, q.tuq[j]); }
            } else if (kind == 2) {
                if (!upper) { const int e = q.ordA_l[pl.kA0 + r]; st_ = first_step(tv, nfin, LE, q.otl[e]); }
                else { const int e = q.ordA_u[pl.kA0 + r]; st_ = first_step(tv, nfin, GE, q.otu[e]); }
            }
            sA[r] = st_;
        }
        for (int r = t; r < pl.nB; r += T) {
            int st_ = kNever;
            if (kind == 0) {
                if (!upper) st_ = first_step(tv, nfin, LE, q.qs[pl.idx1 - r]);
                else st_ = first_step(tv, nfin, GT, q.qs[pl.idx1 + r]);
            } else if (kind == 1) {
                if (!upper) {
                    const int j = pl.idx1 - r;
                    st_ = first_step(tv, nfin, LT, q.qs[j]);
                    if (j <= pl.idx2 && st_ != kNever) st_ = max(st_, first_step(tv, nfin, LE, q.tlq[j]));
                } else {
                    const int j = pl.idx1 + r;
                    st_ = first_step(tv, nfin, GT, q.qs[j]);
                    if (j >= pl.idx2 && st_ != kNever) st_ = max(st_, first_step(tv, nfin, GE, q.tuq[j]));
                }
            } else {
                if (!upper) {
                    const int e = q.ordB_l[pl.kB0 + r];
                    st_ = first_step(tv, nfin, LE, q.qn[e]);
                    if (q.otl[e] < t0 && st_ != kNever) st_ = max(st_, first_step(tv, nfin, LE, q.otl[e]));
                } else {
                    const int e = q.ordB_u[pl.kB0 + r];
                    st_ = first_step(tv, nfin, GE, q.qn[e]);
                    if (q.otu[e] > t0 && st_ != kNever) st_ = max(st_, first_step(tv, nfin, GE, q.otu[e]));
                }
            }
            sB[r] = st_;
        }
        __syncthreads();

        // ---- 6. op order: (step, stream A before B, rank)
        // valid ops form a prefix of each stream (steps never go from finite to kNever and back)
        const int nAv = prefix_count(pl.nA, [&](int r) { return sA[r] != kNever; });
        const int nBv = prefix_count(pl.nB, [&](int r) { return sB[r] != kNever; });
        // ERP's steps of stream B ascend too (both the query points and their
        // t_l / t_u ascend), unless rounding of t_l, t_u breaks it
        int falls = 0;
        if (kind == 2)
            for (int r = t; r + 1 < nBv; r += T) falls |= sB[r] > sB[r + 1] ? 1 : 0;
        const bool b_sorted = !__syncthreads_or(falls);
        for (int k = t; k < nAv + nBv; k += T) opdesc[k] = -1;
        __syncthreads();
        for (int r = t; r < nAv; r += T) {
            const int sa = sA[r];
            int blt;  // valid B ops with step < sa
            if (b_sorted) {
                blt = prefix_count(nBv, [&](int k) { return sB[k] < sa; });
            } else {
                blt = 0;
                for (int k = 0; k < nBv; ++k) blt += (sB[k] < sa) ? 1 : 0;
            }
            const int pos = r + blt;
            opdesc[pos] = r;
            opstep[pos] = sa;
        }
        for (int r = t; r < nBv; r += T) {
            const int sb = sB[r];
            int bbefore;
            if (b_sorted) {
                bbefore = r;
            } else {
                bbefore = 0;
                for (int k = 0; k < nBv; ++k) {
                    const int sk = sB[k];
                    bbefore += (sk < sb || (sk == sb && k < r)) ? 1 : 0;
                }
            }
            const int ale = prefix_count(nAv, [&](int k) { return sA[k] <= sb; });
            const int pos = bbefore + ale;
            opdesc[pos] = 0x40000000 | r;
            opstep[pos] = sb;
        }
        if (t == 0) s_nops = nAv + nBv;
        __syncthreads();
        const int nops = s_nops;

        // ---- 7. replay: initial sums then every op, in the reference's order.
        // Every thread first gathers the operands into shared memory, already
        // signed for the accumulator they go to, so that the replaying lanes
        // only add: x - y is x + (-y) in IEEE arithmetic, and an element or op
        // that leaves an accumulator unchanged contributes -0.0 (x + -0.0 == x
        // for every x, signed zeros included).
        const double* pw0 = (kind == 2) ? q.opw : q.pw;
        const double* Dt = (kind == 2) ? q.oD : q.Dq;
        // (the power sums' elements and the penalty sum's, in the order they are
        // added; past the last one no change, to a whole number of chunks)
        int em = 0, dm = 1, lm = m, ec = 0, lc = m;
        if (kind == 0) {
            em = upper ? pl.idx1 : 0;
            lm = upper ? m - pl.idx1 : pl.idx1 + 1;
            lc = 0;
        } else if (kind == 1) {
            em = pl.idx1;
            dm = upper ? 1 : -1;
            lm = upper ? pl.idx2 - pl.idx1 : pl.idx1 - pl.idx2;
            ec = upper ? pl.idx2 : 0;
            lc = upper ? m - pl.idx2 : pl.idx2 + 1;
        }
        const int ninit = (max(lm, lc) + 15) & ~15;
        for (int i = t; i < ninit; i += T) {
            bool in_m = i < lm, in_c = i < lc;
            if (kind == 2 && i < m) {  // which initial sum the element enters, if any
                const double qv = q.qn[i];
                int cd;
                if (!upper) cd = (qv >= t0) ? 0 : (q.otl[i] >= t0 ? 1 : 2);
                else cd = (qv <= t0) ? 0 : (q.otu[i] <= t0 ? 1 : 2);
                in_m = cd == 1;
                in_c = cd == 2;
            }
            const int jm = em + dm * i;
            double* o = st + 4 * i;
            o[0] = in_m ? pw0[jm] : -0.0;
            o[1] = in_m ? pw0[m + jm] : -0.0;
            o[2] = in_m ? pw0[2 * m + jm] : -0.0;
            o[3] = in_c ? Dt[ec + i] : -0.0;
        }
        __syncthreads();
        // initial sums: lane j of one warp (a different one in each block, so that
        // co-resident blocks' chains sit on different sub-partitions) owns
        // accumulator j (the power sums m_0..m_2 for j < 3, the penalty sum C
        // for j = 3) and adds its elements in the reference's order
        const int jl = t - 32 * (int)(blockIdx.x % (T / 32));
        double acc = 0.0;
        if (jl >= 0 && jl < 4) acc = chain<false>(acc, st + jl, ninit);
        __syncthreads();
        // ops before every 32nd step
        for (int b = t; b <= (nr + 31) / 32; b += T) s_lo[b] = prefix_count(nops, [&](int k) { return opstep[k] < 32 * b; });
        // op payloads into the state slots the replay overwrites: op B
        // subtracts the element's powers, op A adds them and subtracts its
        // penalty
        for (int k = t; k < ((nops + 15) & ~15); k += T) {
            const int d = k < nops ? opdesc[k] : -1;
            double* o = st + 4 * (k + 1);
            if (d < 0) {  // past the last op: no change
                o[0] = o[1] = o[2] = o[3] = -0.0;
                continue;
            }
            const int r = d & 0x3fffffff;
            const bool op_b = (d & 0x40000000) != 0;
            int x;  // table index of the op's query element
            if (kind == 2) x = op_b ? (upper ? q.ordB_u : q.ordB_l)[pl.kB0 + r]
                                    : (upper ? q.ordA_u : q.ordA_l)[pl.kA0 + r];
            else if (op_b) x = upper ? pl.idx1 + r : pl.idx1 - r;
            else x = upper ? pl.idx2 + r : pl.idx2 - r;
            x = min(max(x, 0), m - 1);
            const double a0 = pw0[x], a1 = pw0[m + x], a2 = pw0[2 * m + x], a3 = Dt[x];
            o[0] = op_b ? -a0 : a0;
            o[1] = op_b ? -a1 : a1;
            o[2] = op_b ? -a2 : a2;
            o[3] = op_b ? -0.0 : -a3;
        }
        __syncthreads();
        // replay: lane j adds every op's operand to its accumulator j and
        // stores the state after each op in the operand's place
        if (jl >= 0 && jl < 4) {
            st[jl] = acc;
            chain<true>(acc, st + 4 + jl, nops);
        }
        __syncthreads();

        // ---- 8. scores and first maximum
        ArgMax best{0.0, INT_MAX, 0};
        int nan0 = 0;
        // the number of ops with step <= i lies between the counts at the ends of
        // the step's 32
        for (int i = t; i < nr; i += T) {
            int lo = s_lo[i >> 5], hi = s_lo[(i >> 5) + 1];
            while (lo < hi) { const int mid = (lo + hi) >> 1; if (opstep[mid] <= i) lo = mid + 1; else hi = mid; }
            const double* sv = st + 4 * lo;
            const double tt = tv[i];
            const double f = f_p(sv[0], sv[1], sv[2], p, tt);
            double h;
            if (kind == 0) h = upper ? f : fabs(f);
            else h = dadd(sv[3], upper ? f : fabs(f));
            const double lb = dmul(h, (double)gp[thr_pad(i)]);
            if (isnan(lb)) {
                if (i == 0) nan0 = 1;  // findMaxIndex never leaves a NaN at index 0
            } else {
                best = ArgMaxOp()(best, ArgMax{lb, i, 1});
            }
        }
        const int any_nan0 = __syncthreads_or(nan0);
        const ArgMax r = AReduce(red_tmp).Reduce(best, ArgMaxOp());
        if (t == 0) s_best = any_nan0 ? 0 : (r.ok ? r.i : 0);
        __syncthreads();
        if (t == 0) *out = tv[s_best];
        __syncthreads();
    }
}

template <int T, int IPT>
ThrMem threshold_mem(int m, size_t smem_optin) {
    using Sort = cub::BlockMergeSort<unsigned long long, T, IPT, int>;
    constexpr int CAP = T * IPT;
    const size_t r = thr_r_bytes(CAP), z = thr_z_bytes(m), sort = sizeof(typename Sort::TempStorage);
    auto most = [](size_t a, size_t b) { return a > b ? a : b; };
    ThrMem mem;
    mem.gw = false;
    mem.z_shared = 1;
    mem.smem = r + most(z, most(sort, thr_bucket_bytes(CAP, thr_buckets(CAP, false)))) + 16;
    mem.gbytes = 0;
    if (mem.smem + 8192 <= smem_optin) return mem;
    const size_t sorts = most(sort, thr_bucket_bytes(CAP, thr_buckets(CAP, true)));
    mem.gw = true;
    mem.z_shared = most(z, sorts) + 16 + 8192 <= smem_optin;
    mem.smem = (mem.z_shared ? most(z, sorts) : sorts) + 16;
    mem.gbytes = 2 * r + (mem.z_shared ? 0 : z + 16);
    return mem;
}

#define FSM_THR_INST(T, IPT)                                                                 \
    template __global__ void k_threshold<T, IPT, false>(Geom, ThrJob, unsigned char*,  \
                                                        long long, int);              \
    template __global__ void k_threshold<T, IPT, true>(Geom, ThrJob, unsigned char*,   \
                                                       long long, int);               \
    template ThrMem threshold_mem<T, IPT>(int, size_t);
FSM_THR_INST(128, 4)
FSM_THR_INST(256, 4)
FSM_THR_INST(256, 8)
FSM_THR_INST(512, 8)
FSM_THR_INST(1024, 8)
FSM_THR_INST(1024, 16)

}  // namespace fsm
