// Exact EDR and LCSS distances (src/ElasticMeasures.cpp) of candidate windows
// as bit-vector recurrences: one lane per candidate, one candidate point per
// step, the whole band of the step in one to sixteen machine words.
//
// Both measures only ask of a pair of points whether |x - y| <= eps, and
// their values count unit steps, so the differences between neighbouring
// cells are 0 or 1 (LCSS) or -1, 0, 1 (EDR), band cells included, and fit in
// bits (G. Myers, J. ACM 46(3), 1999; H. Hyyro, Nordic J. Computing 10(1),
// 2003, for the band that moves along the diagonal; M. Crochemore et al.,
// Inf. Process. Lett. 80(6), 2001 and Hyyro 2004 for LCSS).  Everything is
// integer arithmetic on exact comparisons: the results are the banded
// recurrences' values, whatever the operand magnitudes.
//
// Bit d of a vector at candidate point t is query point i = t - w + d
// (0 <= d <= 2w), so the band slides by one bit per step.
//
// Matches: for a query point x the doubles y with fl(|x - y|) <= eps are an
// interval [a, b] (rounding is monotone), found exactly by the host.  Over
// all query points the 2m ends cut the line into 2m + 1 ranges on each of
// which the set of matching query points is constant: a table of 2m + 1 bit
// rows (k_bit_table).  A candidate point takes its range from the sorted ends
// (a grid of buckets gives the place to start, then a short forward walk, or a
// bisection where a bucket is crowded) and
// reads the 2w+1 bits around its own position from the range's row: the 2w+1
// comparisons of the cell-by-cell DP become one lookup.
//
// Early abandon, as in the cell-by-cell DP but along the candidate:
//   EDR: the band's minimum after point t plus, for the points to come, at
//     least one for every point that meets no query point in its band.  GLB's
//     T->Q sum counts points that meet none (it tests the envelope of the same
//     band), so that sum less the empty lookups so far is a lower bound.
//   LCSS: the band's maximum plus the points to come that may match: at most
//     GLB's T->Q count less the non-empty lookups so far.
// These are integers, so no slack is needed.  The band minimum takes a pass
// over the differences by nibbles; it is taken only when the centre cell alone
// would already abandon.
//
// What bounds it: instruction issue, about 90 instructions per point and lane
// at w <= 15 (normalisation 6 FP64 operations, the lookup 30, the update 15)
// where the cell-by-cell DP issues 20 to 60 per cell.  A warp takes 32
// consecutive entries of the candidate list and steps them together: neighbours
// read neighbouring points (coalesced) and mostly abandon within a few points
// of each other, and every index into the band is uniform.  Measured on the
// five-metric workload (2^24 points, m = 256, w = 13; the candidates left by
// GLB): EDR 29.8 ms cell by cell, 4.5 ms here; LCSS 7.1 and 0.81 ms; the exact
// scan of 400,009 points by LCSS (m = 160, w = 8) 1.27 and 0.17 ms.
#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

namespace {

constexpr int kSteps = 4;  // points loaded and normalised together

// rank of y among the sorted ends E[0..ne) (E[ne] = +inf): the number <= y.  deep:
// some bucket holds more than kBitDeep ends (an outlier among the query's points
// stretches the buckets), so the place in the bucket is bisected.  Stepping there
// took a query of 1100 points with spikes 30 times as long.
__device__ __forceinline__ int bit_rank(double y, const double* __restrict__ E, const unsigned short* __restrict__ grid,
                                        double e0, double elast, double scale, int ne, bool deep) {
    const double c = y < e0 ? e0 : (y > elast ? elast : y);
    // 1.5 * 2^52 added: the low word holds the bucket, rounded to nearest (the
    // host places the ends with the same operations)
    const double v = dadd(dmul(dsub(c, e0), scale), 6755399441055744.0);
    const int b = __double2loint(v);
    int r = grid[b];
    if (deep) {
        for (int hi = b < kBitBuckets ? grid[b + 1] : ne; r < hi;) {
            const int mid = (r + hi) >> 1;
            if (E[mid] <= y) r = mid + 1;
            else hi = mid;
        }
    }
    while (E[r] <= y) ++r;
    return r;
}

}  // namespace

// row r, word j of the table: bit b is query point 32 (j - pad) + b
__global__ void __launch_bounds__(256) k_bit_table(const int* __restrict__ pa, const int* __restrict__ pb, int m,
                                                   int pad, int rs, unsigned* __restrict__ table) {
    const long long total = (long long)(2 * m + 1) * rs;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(k / rs), i0 = ((int)(k % rs) - pad) * 32;
        unsigned v = 0;
        for (int b = 0; b < 32; ++b) {
            const int i = i0 + b;
            if (i >= 0 && i < m && pa[i] < r && r <= pb[i]) v |= 1u << b;
        }
        table[k] = v;
    }
}

template <int METRIC, int NW>
__global__ void __launch_bounds__(kBitThreads) k_bitdp(Geom g, DpJob job, BitTab bt) {
    extern __shared__ __align__(16) unsigned char bit_smem[];
    __shared__ short s_nib[256];  // EDR: (minimum prefix sum, sum) of four differences
    const QueryDev& q = job.q;
    const int m = q.m, w = q.w, W2 = 2 * w + 1, ne = 2 * m;
    double* E = (double*)bit_smem;
    unsigned short* grid = (unsigned short*)(E + ne + 1);
    unsigned* stab = (unsigned*)(bit_smem + bit_table_offset(m));
    for (int i = threadIdx.x; i <= ne; i += kBitThreads) E[i] = bt.E[i];
    for (int i = threadIdx.x; i <= kBitBuckets; i += kBitThreads) grid[i] = bt.grid[i];
    const int rs = bt.rs;
    if (bt.in_smem)
        for (int i = threadIdx.x; i < (ne + 1) * rs; i += kBitThreads) stab[i] = bt.table[i];
    for (int i = threadIdx.x; i < 256; i += kBitThreads) {
        int sum = 0, mn = 0;
        for (int b = 0; b < 4; ++b) {
            sum += ((i >> b) & 1) - ((i >> (4 + b)) & 1);
            mn = min(mn, sum);
        }
        s_nib[i] = (short)((mn << 8) | (sum & 0xff));
    }
    __syncthreads();
    const unsigned* __restrict__ table = bt.in_smem ? stab : bt.table;
    const double e0 = bt.e0, elast = bt.elast, scale = bt.scale;
    const bool deep = bt.most > kBitDeep;

    const unsigned long long n_all = job.list ? *job.n_list : (unsigned long long)job.n_windows;
    const unsigned long long n =
        (job.list && n_all > (unsigned long long)job.list_cap) ? job.list_cap : n_all;
    const double cut = job.cutoff_ptr ? *job.cutoff_ptr : job.cutoff;
    const int lane = threadIdx.x & 31;
    // the largest EDR value, the smallest LCSS count, that is kept
    int lim;
    if (METRIC == EDR) {
        lim = cut >= 1e9 ? 1000000000 : (cut >= 0.0 ? (int)cut : -1);
    } else {
        int lo = 0, hi = m + 1;  // first count whose distance is <= cut (monotone)
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (dsub(1.0, ddiv((double)mid, (double)m)) <= cut) hi = mid;
            else lo = mid + 1;
        }
        lim = lo;
    }
    constexpr unsigned kAll = 0xffffffffu;
    const unsigned top = (W2 & 31) ? (1u << (W2 & 31)) - 1u : kAll;  // bits of the last word
    const int cw = w >> 5, cb = w & 31;                              // the centre bit
    const int off0 = 32 * bt.pad - w;                                // bit offset of d = 0 at t = 0

    unsigned long long valid_count = 0, cells = 0;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(job.next, 32ull);
        base = __shfl_sync(kAll, base, 0);
        if (base >= n) break;
        const unsigned long long item = base + lane;
        bool active = item < n;
        long long gi = 0;
        double mu = 0.0, sg = 1.0;
        int S = -1;  // GLB's T->Q sum, -1: none
        if (active) {
            gi = job.list ? job.list[item] : (long long)item;
            long long s;
            int j;
            g.locate(gi, &s, &j);
            mu = job.MU[s * g.kml + j];
            sg = job.SIG[s * g.kml + j];
            active = !window_invalid(sg, g, gi);
            if (active && job.list_t) {
                const double v = job.list_t[item];
                if (v >= 0.0) S = (int)v;
            }
        }
        if (active) ++valid_count;
        else { mu = 0.0; sg = 1.0; gi = 0; }
        const double inv = ddiv(1.0, sg);
        const bool rok = rcp_div_in_range(sg);
        const double* tp = job.target + gi;

        unsigned P[NW], N[NW];  // EDR: +1 / -1 differences; LCSS: P = zero differences
        int c = 0, c0 = w;      // EDR: centre and lowest band cell; LCSS: c0 = value below the band
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            if (METRIC == EDR) {  // D(i, 0) = |i|
                const int a = w - 32 * k;
                N[k] = a >= 32 ? kAll : (a <= 0 ? 0u : (1u << a) - 1u);
                P[k] = ~N[k];
            } else {
                P[k] = kAll;
                N[k] = 0u;
            }
        }
        P[NW - 1] &= top;
        if (METRIC == LCSS) c0 = 0;
        int seen = 0;  // EDR: empty lookups; LCSS: non-empty ones
        int t = 0;
        double nx[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; ++u) nx[u] = (active && u < m) ? tp[u] : 0.0;
        for (; t < m; t += kSteps) {
            double y[kSteps];
            bool good = rok;
#pragma unroll
            for (int u = 0; u < kSteps; ++u) {
                const double a = dsub(nx[u], mu);
                const double q0 = rcp_div_estimate(a, inv);
                good = good & (rcp_div_in_range_bits(q0) != 0);
                y[u] = rcp_div_finish(a, sg, inv, q0);
            }
            if (!good) {
#pragma unroll
                for (int u = 0; u < kSteps; ++u) y[u] = ddiv(dsub(nx[u], mu), sg);
            }
#pragma unroll
            for (int u = 0; u < kSteps; ++u)
                nx[u] = (active && t + kSteps + u < m) ? tp[t + kSteps + u] : 0.0;
#pragma unroll
            for (int u = 0; u < kSteps; ++u) {
                if (t + u >= m) break;
                const int r = bit_rank(y[u], E, grid, e0, elast, scale, ne, deep);
                const int o = off0 + t + u;  // uniform
                const unsigned* row = table + r * rs + (o >> 5);
                unsigned Eq[NW], any = 0, w0 = row[0];
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    const unsigned w1 = row[k + 1];
                    Eq[k] = __funnelshift_r(w0, w1, o & 31);
                    if (k == NW - 1) Eq[k] &= top;
                    any |= Eq[k];
                    w0 = w1;
                }
                if (METRIC == EDR) {
                    unsigned D0[NW], HP[NW], HN[NW];
                    unsigned long long carry = 0;
#pragma unroll
                    for (int k = 0; k < NW; ++k) {
                        carry += (unsigned long long)(Eq[k] & P[k]) + P[k];
                        D0[k] = ((unsigned)carry ^ P[k]) | Eq[k] | N[k];
                        carry >>= 32;
                        HP[k] = N[k] | ~(D0[k] | P[k]);
                        HN[k] = D0[k] & P[k];
                    }
                    c0 += 1 - (int)(D0[0] & 1u);
                    D0[NW - 1] &= top;
#pragma unroll
                    for (int k = 0; k < NW; ++k) {
                        if (k == cw) c += 1 - (int)((D0[k] >> cb) & 1u);
                        const unsigned X = k + 1 < NW ? __funnelshift_r(D0[k], D0[k < NW - 1 ? k + 1 : k], 1) : D0[k] >> 1;
                        P[k] = HN[k] | ~(X | HP[k]);
                        N[k] = HP[k] & X;
                    }
                    P[NW - 1] &= top;
                    seen += any ? 0 : 1;
                } else {
                    // the band moves up: the lowest cell's difference joins the value below
                    if (t + u) {
                        c0 += 1 - (int)(P[0] & 1u);
#pragma unroll
                        for (int k = 0; k < NW; ++k)
                            P[k] = k + 1 < NW ? __funnelshift_r(P[k], P[k < NW - 1 ? k + 1 : k], 1)
                                              : (P[k] >> 1) | (top & ~(top >> 1));
                    }
                    unsigned long long carry = 0;
#pragma unroll
                    for (int k = 0; k < NW; ++k) {
                        carry += (unsigned long long)(P[k] & Eq[k]) + P[k];
                        P[k] = (unsigned)carry | (P[k] & ~Eq[k]);
                        carry >>= 32;
                    }
                    P[NW - 1] &= top;
                    seen += any ? 1 : 0;
                }
            }
            // abandon
            const int done = min(t + kSteps, m);
            cells += active ? (unsigned long long)W2 * (done - t) : 0ull;
            bool stop = !active;
            if (METRIC == EDR) {
                const int rest = max(0, S - seen);  // S = -1: 0
                if (active && done < m && c + rest > lim) {
                    int sum = c0, mn = c0;
#pragma unroll
                    for (int k = 0; k < NW; ++k)
#pragma unroll
                        for (int b = 0; b < 32; b += 4) {
                            const int v = s_nib[((P[k] >> b) & 15u) | (((N[k] >> b) & 15u) << 4)];
                            mn = min(mn, sum + (v >> 8));
                            sum += (int)(signed char)(v & 0xff);
                        }
                    // differences past the band's last cell are +1 or 0: no lower value
                    stop = mn + rest > lim;
                }
            } else {
                int v = c0 + W2;
#pragma unroll
                for (int k = 0; k < NW; ++k) v -= __popc(P[k]);
                int rest = m - done;
                if (S >= 0) rest = min(rest, max(0, S - seen));
                if (v + rest < lim) stop = true;
            }
            if (stop) active = false;
            if (!__any_sync(kAll, active)) break;
        }
        if (active) {
            double dist;
            if (METRIC == EDR) {
                dist = (double)c;
            } else {
                int v = c0;  // cell (m-1, m-1): differences of bits 0..w
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    const int b = w + 1 - 32 * k;
                    const unsigned keep = b >= 32 ? kAll : (b <= 0 ? 0u : (1u << b) - 1u);
                    v += __popc(~P[k] & keep);
                }
                dist = dsub(1.0, ddiv((double)v, (double)m));
            }
            if (dist <= cut && isfinite(dist)) {
                const unsigned long long o = atomicAdd(job.n_out, 1ull);
                if (o < (unsigned long long)job.out_cap) {
                    job.out_idx[o] = gi;
                    job.out_dist[o] = dist;
                }
            }
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) {
        valid_count += __shfl_xor_sync(kAll, valid_count, o);
        cells += __shfl_xor_sync(kAll, cells, o);
    }
    if (lane == 0) {
        if (job.n_valid && valid_count) atomicAdd(job.n_valid, valid_count);
        if (job.n_cells && cells) atomicAdd(job.n_cells, cells);
    }
}

#define FSM_BIT_INST(NW)                                                \
    template __global__ void k_bitdp<EDR, NW>(Geom, DpJob, BitTab);     \
    template __global__ void k_bitdp<LCSS, NW>(Geom, DpJob, BitTab);
FSM_BIT_INST(1)
FSM_BIT_INST(2)
FSM_BIT_INST(3)
FSM_BIT_INST(4)
FSM_BIT_INST(5)
FSM_BIT_INST(6)
FSM_BIT_INST(7)
FSM_BIT_INST(8)
FSM_BIT_INST(9)
FSM_BIT_INST(10)
FSM_BIT_INST(11)
FSM_BIT_INST(12)
FSM_BIT_INST(13)
FSM_BIT_INST(14)
FSM_BIT_INST(15)
FSM_BIT_INST(16)

int bit_words(int w) {
    const int need = (2 * w + 1 + 31) / 32;
    return need <= 16 ? need : 0;
}

template <int M>
static const void* bit_for(int nw) {
    switch (nw) {
        case 1: return (const void*)k_bitdp<M, 1>;
        case 2: return (const void*)k_bitdp<M, 2>;
        case 3: return (const void*)k_bitdp<M, 3>;
        case 4: return (const void*)k_bitdp<M, 4>;
        case 5: return (const void*)k_bitdp<M, 5>;
        case 6: return (const void*)k_bitdp<M, 6>;
        case 7: return (const void*)k_bitdp<M, 7>;
        case 8: return (const void*)k_bitdp<M, 8>;
        case 9: return (const void*)k_bitdp<M, 9>;
        case 10: return (const void*)k_bitdp<M, 10>;
        case 11: return (const void*)k_bitdp<M, 11>;
        case 12: return (const void*)k_bitdp<M, 12>;
        case 13: return (const void*)k_bitdp<M, 13>;
        case 14: return (const void*)k_bitdp<M, 14>;
        case 15: return (const void*)k_bitdp<M, 15>;
        case 16: return (const void*)k_bitdp<M, 16>;
        default: return nullptr;
    }
}

const void* bitdp_kernel(int metric, int w) {
    return metric == EDR ? bit_for<EDR>(bit_words(w)) : metric == LCSS ? bit_for<LCSS>(bit_words(w)) : nullptr;
}

}  // namespace fsm
