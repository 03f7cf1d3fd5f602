// Per-segment envelopes: min/max of window means and sigmas over trailing
// windows (src/lower_upper_lemire.cpp:94-126), the centred radius-w envelope
// of the segment (src/lower_upper_lemire.cpp:8-44), and the conservative
// z-normalised envelopes U_normal, L_normal (src/lb_normalize.cpp:9-32).
//
// The reference uses monotone deques.  Their outputs have a closed form that
// this kernel computes in parallel:
//  * with no NaN in the window: the window minimum (maximum); among equal
//    values the deque keeps the most recent one, which only matters for the
//    sign of a zero (window means and sigmas are never -0; a target's -0 and
//    +0 give the same U_normal / L_normal comparisons and penalties);
//  * with a NaN in the window: a NaN blocks every pop behind it, so the
//    front is the extremum of the points before the first NaN, or NaN when
//    the window starts with NaN.
//
// A block takes a tile of consecutive outputs of one segment.  Trailing
// windows of m points (m >= 17): the tile and its m - 1 points to the left are
// cut into runs of eight; a thread takes a run and leaves the extremum from
// the run's start to each point and from each point to its end (van Herk, Gil
// and Werman's blocks, but eight long whatever m is), and the runs' own
// extrema are doubled to stretches of 2^L runs, 2^L the largest power that
// fits between a window's two end runs.  A window is then four reads: its
// first point's rest of run, its last point's start of run, and two stretches
// that cover the runs between.  Shorter windows are read point by point.
// Positions outside [0, n) hold NaN, which no comparison takes, so clipped
// windows need no case of their own.  Centred windows of the raw points are the
// min/max of two forward windows of the target (k_fwd_env) that lie inside the
// segment.  Windows that do hold a NaN (a bit per position, only looked at
// when the tile has any) end before the first one.
//
// What bounds it: shared-memory accesses, about 8 eight-byte ones per point,
// series and extremum, and three reads of MU and SIG each (one from HBM).
// Doubling over single points took log2(m) passes of the whole segment with a
// block barrier each, one block per SM, and global scratch from 8192 points
// on.  Measured: 2^24 points, m = 256: 1.89 -> 0.67 ms; 2^22 points, m = 64 ..
// 1024 (19 lengths, most with 8192-point segments): 17.3 -> 3.9 ms; 2^21 points,
// m = 1850: 0.86 -> 0.12 ms.
#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

namespace {

constexpr int kRun = 8;

// one spare slot after every run, so threads on neighbouring runs meet
// different banks
__host__ __device__ __forceinline__ int px(int i) { return i + (i >> 3); }

template <bool MAX>
__device__ __forceinline__ double ext(double a, double b) {  // b unless NaN or worse
    return MAX ? (b > a ? b : a) : (b < a ? b : a);
}

// first set bit at or after i and before n, or n
__device__ __forceinline__ int next_bit(const unsigned* __restrict__ bits, int i, int n) {
    while (i < n) {
        const unsigned v = bits[i >> 5] >> (i & 31);
        if (v) return min(n, i + __ffs(v) - 1);
        i = (i | 31) + 1;
    }
    return n;
}

struct EnvWork {
    double *P, *S;        // [px(len)] start of run .. point, point .. end of run
    double *R0, *Ra, *Rb;  // [runs] run extrema; doubled stretches
    unsigned* bits;        // [len / 32] NaN positions
};

// Extrema of src over [o - m + 1, o] for the tile's outputs o0 + t + k T,
// clipped to [0, n).  Local position l is o0 - m + 1 + l.
template <int T, int OPT, bool MAX>
__device__ void trailing(const double* __restrict__ src, int n, int m, int o0, int nout, const EnvWork& wk,
                         double (&out)[OPT]) {
    constexpr double kNone = MAX ? -INFINITY : INFINITY;
    const int t = threadIdx.x, b0 = o0 - (m - 1);
    const int len = nout + m - 1, runs = (len + kRun - 1) / kRun, plen = (runs * kRun + 31) & ~31;
    int local_nan = 0;
    for (int l = t; l < plen; l += T) {
        const int p = b0 + l;
        const bool in = l < len && p >= 0 && p < n;
        const double v = in ? src[p] : dnan();
        if (l < runs * kRun) wk.P[px(l)] = v;
        const unsigned bad = __ballot_sync(0xffffffffu, in && isnan(v));
        if ((l & 31) == 0) wk.bits[l >> 5] = bad;
        local_nan |= bad != 0u;
    }
    const int any_nan = __syncthreads_or(local_nan);
    const bool by_runs = m > 2 * kRun;
    int L = 0;
    const double* Rt = wk.R0;
    if (by_runs) {
        for (int r = t; r < runs; r += T) {
            double v[kRun];
#pragma unroll
            for (int u = 0; u < kRun; ++u) v[u] = wk.P[px(r * kRun) + u];
            double e = kNone;
#pragma unroll
            for (int u = kRun - 1; u >= 0; --u) {
                e = ext<MAX>(e, v[u]);
                wk.S[px(r * kRun) + u] = e;
            }
            wk.R0[r] = e;
            e = kNone;
#pragma unroll
            for (int u = 0; u < kRun; ++u) {
                e = ext<MAX>(e, v[u]);
                wk.P[px(r * kRun) + u] = e;
            }
        }
        __syncthreads();
        // whole runs between a window's end runs: (m-1)/8 - 1 or one more
        L = 31 - __clz((m - 1) / kRun - 1);
        double* w0 = wk.Ra;
        double* w1 = wk.Rb;
        for (int lv = 1; lv <= L; ++lv) {
            const int s = 1 << (lv - 1);
            for (int r = t; r < runs; r += T) w0[r] = r + s < runs ? ext<MAX>(Rt[r], Rt[r + s]) : Rt[r];
            __syncthreads();
            Rt = w0;
            double* x = w0; w0 = w1; w1 = x;
        }
    }
#pragma unroll
    for (int k = 0; k < OPT; ++k) {
        const int a = t + k * T;
        out[k] = kNone;
        if (a >= nout) continue;
        int b = a + m - 1;
        if (any_nan) {
            const int first = max(a, -b0), last = min(b, n - 1 - b0);  // inside [0, n)
            const int f = next_bit(wk.bits, first, last + 1);
            if (f <= last) {  // only the points before the first NaN
                double e = kNone;
                if (f == first) {
                    e = dnan();
                } else if (!by_runs || (f - 1) / kRun == first / kRun) {
                    for (int l = first; l < f; ++l) e = ext<MAX>(e, src[b0 + l]);
                } else {
                    e = ext<MAX>(wk.S[px(first)], wk.P[px(f - 1)]);
                    for (int r = first / kRun + 1; r < (f - 1) / kRun; ++r) e = ext<MAX>(e, wk.R0[r]);
                }
                out[k] = e;
                continue;
            }
        }
        double e;
        if (by_runs) {
            const int ra = a / kRun + 1, rb = b / kRun - (1 << L);
            e = ext<MAX>(ext<MAX>(wk.S[px(a)], wk.P[px(b)]), ext<MAX>(Rt[ra], Rt[rb]));
        } else {
            e = kNone;
            for (; b >= a; --b) e = ext<MAX>(e, wk.P[px(b)]);
        }
        out[k] = e;
    }
    __syncthreads();
}

}  // namespace

template <int T, int OPT>
__global__ void __launch_bounds__(T) k_envelope(const double* __restrict__ target, const double* __restrict__ Lraw,
                                                const double* __restrict__ Uraw, const double* __restrict__ MU,
                                                const double* __restrict__ SIG, Geom g, int w, int tiles,
                                                double* __restrict__ Un, double* __restrict__ Ln) {
    extern __shared__ __align__(16) unsigned char env_smem[];
    constexpr int O = T * OPT;
    const int mk = g.m_k, kml = g.kml, m = g.m, t = threadIdx.x;
    const int runs = (O + m - 1 + kRun - 1) / kRun;
    EnvWork wk;
    wk.P = (double*)env_smem;
    wk.S = wk.P + px(runs * kRun);
    wk.R0 = wk.S + px(runs * kRun);
    wk.Ra = wk.R0 + runs;
    wk.Rb = wk.Ra + runs;
    wk.bits = (unsigned*)(wk.Rb + runs);
    const long long s = blockIdx.x / tiles;
    const int o0 = (int)(blockIdx.x % tiles) * O, nout = min(O, mk - o0);
    double simn[OPT], simx[OPT], mumn[OPT], mumx[OPT];
    trailing<T, OPT, false>(SIG + s * kml, kml, m, o0, nout, wk, simn);
    trailing<T, OPT, true>(SIG + s * kml, kml, m, o0, nout, wk, simx);
    trailing<T, OPT, false>(MU + s * kml, kml, m, o0, nout, wk, mumn);
    trailing<T, OPT, true>(MU + s * kml, kml, m, o0, nout, wk, mumx);
    // centred windows of the raw segment: NaN positions o0 - w + l
    const long long off = g.off(s);
    const double* __restrict__ seg = target + off;
    const int c0 = o0 - w, clen = (nout + 2 * w + 31) & ~31;
    int local_nan = 0;
    for (int l = t; l < clen; l += T) {
        const int p = c0 + l;
        const unsigned bad = __ballot_sync(0xffffffffu, p >= 0 && p < mk && isnan(seg[min(max(p, 0), mk - 1)]));
        if ((l & 31) == 0) wk.bits[l >> 5] = bad;
        local_nan |= bad != 0u;
    }
    const int any_nan = __syncthreads_or(local_nan);
    const double* __restrict__ lf = Lraw + off;
    const double* __restrict__ uf = Uraw + off;
#pragma unroll
    for (int k = 0; k < OPT; ++k) {
        const int x = t + k * T, o = o0 + x;
        if (x >= nout) continue;
        const int ws = max(0, o - w), we = min(mk - 1, o + w);
        const int p1 = we - w;  // the forward windows at ws and we - w cover [ws, we]
        double lmn = lf[ws], lmx = uf[ws];
        lmn = ext<false>(lmn, lf[p1]);
        lmx = ext<true>(lmx, uf[p1]);
        if (any_nan) {
            const int f = next_bit(wk.bits, ws - c0, we - c0 + 1) + c0;
            if (f <= we) {
                lmn = f == ws ? dnan() : INFINITY;
                lmx = f == ws ? dnan() : -INFINITY;
                for (int p = ws; p < f; ++p) {
                    lmn = ext<false>(lmn, seg[p]);
                    lmx = ext<true>(lmx, seg[p]);
                }
            }
        }
        const double nu = dsub(lmx, mumn[k]);
        const double un = (nu >= 0) ? ddiv(nu, simn[k]) : ddiv(nu, simx[k]);
        const double nl = dsub(lmn, mumx[k]);
        const double ln = (nl <= 0) ? ddiv(nl, simn[k]) : ddiv(nl, simx[k]);
        Un[s * mk + o] = un;
        Ln[s * mk + o] = ln;
    }
}

size_t envelope_smem_bytes(int tile, int m, int w) {
    const int runs = (tile + m - 1 + kRun - 1) / kRun;
    const size_t bits = (size_t)(runs * kRun > tile + 2 * w ? runs * kRun : tile + 2 * w) / 32 + 2;
    return (2 * (size_t)px(runs * kRun) + 3 * (size_t)runs) * 8 + bits * 4;
}

#define FSM_ENV_INST(T, OPT)                                                                                    \
    template __global__ void k_envelope<T, OPT>(const double*, const double*, const double*, const double*,    \
                                                const double*, Geom, int, int, double*, double*);
FSM_ENV_INST(128, 4)
FSM_ENV_INST(256, 4)
FSM_ENV_INST(512, 4)

}  // namespace fsm
