// FP32 screen before the exact FP64 DP (DTW, ERP, MSM): drops candidates whose
// banded distance provably exceeds the cutoff and hands the others on.  No
// result is computed here: every kept candidate is evaluated by the exact DP,
// and a dropped one is one that the exact DP would discard.
//
// The proof per candidate.  x, y, g are rounded to FP32; a point difference
// computed in FP32 is off by at most delta = 2^-22 (A + Y + |g|), A = max|x|,
// Y the limit on |y| below (two roundings of the operands, one of the
// difference; MSM's distance of a point to an interval is 1-Lipschitz in each
// argument, which delta covers twice over).  Sums of non-negative terms and
// minima of them carry a relative error of 2^-24 per operation, at most 4m + 4
// on a path of at most 2m + 2 cells: the factor G.
//   MSM: a path of true cost D costs at most (D + (2m+2) delta_c) G here
//     (delta_c = delta + 2^-23 c).
//     Where the query's points lie close together against c (on average within
//     c/2), a first pass takes c alone for the steps up and left: at most the
//     true cost, so what it drops is dropped for certain, and what it keeps runs
//     through the second pass with the intervals.  Its slots hold a cell plus c;
//     the two roundings of a cell's sums stay relative, that of |x-y| - c and c's
//     share of the slot's (2^-24 (|x-y| + 2 c)) lie in delta, which has twice
//     what the difference needs.
//   DTW, ERP: at most (sqrt(D) + delta sqrt(2m+2))^2 G (Cauchy-Schwarz over
//     the path's differences); for D <= R <= s^2 that is at most
//     (R + 2 e s + e^2) G with e = delta sqrt(2m+2).
// So the computed minimum V over a row proves D > R when V > (R + E) G.  R is
// the cutoff (squared for DTW, ERP; with the 1e-9 slack of the exact DP's
// abandon test) less what the rows to come must still add: GLB's Q->T sum
// less an upper bound of the terms of the rows done (FP32 on an envelope
// narrowed by 2^-21 Y).  A candidate with a point beyond Y = 2A + 8 (raw
// series of values below 1: Y = 10A) is dropped when that point alone costs more than
// the cutoff and else kept.  A point y is matched with some x (DTW, ERP: at least
// (|y| - A)^2; ERP may take it out: (|y| - |g|)^2).  MSM reaches y's column from the
// diagonal, which costs at least |y| - A, or from the left at the distance of y to
// [x, y'], which makes up what y' itself did not cost: at least |y| - A as well.
// Raw walks far above and below the query, 1.4 million windows, MSM, m = 249, w = 12,
// all windows evaluated: 2.9 ms a call while the exact DP got such candidates, 0.57 now.
// Points outside the matrix are +-1e15: every path through them costs at least
// about 1e15, and the screen is skipped unless (R + E) G < 1e12.
//
// Points and centred windows come in FP32 relative to the segment (k_rel) where
// there are such rows and the warp's windows allow it, else in FP64: two loads and
// conversions less a row; the query's points in FP32 from shared memory.
//
// One lane per candidate, the band row and the candidate points in shared
// memory [slot][lane].  A warp takes 32 consecutive list entries and steps
// them together, so every index is uniform and neighbours read neighbouring
// points.  R rows (2, 4 or 8) are computed per pass: cell d of the first and cell
// d-u of row u lie in the same column, so a pass reads each band cell and each
// point once and writes one cell for R computed, tests and loads once for R rows,
// and R chains of dependent operations interleave.
//
// What bounds it: instruction issue (a cell takes 3 operations for DTW, 5 and 12
// for MSM without and with the intervals, and a share of the pass; the exact DP
// spends 30 to 110 on FP64 selects and compares).  Measured on the five-metric
// workload (2^24 points, m = 256, w = 13), a query with 16 million candidates: MSM
// 82 ms by the exact DP alone; screen 36 ms with intervals only, 29 with the first
// pass (which steps 95 rows of a candidate instead of 77), 28 with FP32 points, 22
// with four rows a pass instead of two, and 0.2 ms exact; ERP 2.6 -> 0.95 + 0.1 ms;
// 8 top-k queries (DTW, m = 512) 3.9 ms with two rows and FP64 points, 2.1 now.
// DTW and ERP run best with 120 registers (8% slower at 80), MSM with 80 and six
// blocks an SM (3% slower at 72).  A warp steps until its last candidate is
// dropped: 1.5 (MSM) to 1.9 (ERP, DTW) lane rows per useful one.
#include <cfloat>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

namespace {

constexpr float kOut = 1e15f;    // candidate points outside the matrix
constexpr float kBlock = 1e30f;  // band cells outside the band

__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(fminf(a, b), c); }

struct Row {
    float x, c0, s;  // ERP: c0 = (x-g)^2; MSM: c0 = |x-x'| + c, s = sign(x-x')
};

struct Col {
    float y, gy, ady;  // ERP: gy = (y-g)^2; MSM: ady = |y-y'|
    unsigned flip;     // MSM: sign bit that turns x-y into the side of the step
};

template <int METRIC>
__device__ __forceinline__ Col make_col(float y, float yprev, float arg) {
    Col c;
    c.y = y;
    c.gy = c.ady = 0.f;
    c.flip = 0u;
    if (METRIC == ERP) {
        const float d = y - arg;
        c.gy = d * d;
    }
    if (METRIC == MSM) {
        const float dy = y - yprev;
        c.ady = fabsf(dy);
        c.flip = ~__float_as_uint(dy) & 0x80000000u;
    }
    return c;
}

// What a band slot holds of a cell: its value, or (MSM without the intervals)
// its value plus the cost of a step, which up and left moves read as it is and
// a diagonal move takes off again under |x - y|.
template <bool FULL>
__device__ __forceinline__ float slot(float v, float arg) {
    return FULL ? v : v + arg;
}

// one cell from the slots above (up), diagonal and left
template <int METRIC, bool FULL>
__device__ __forceinline__ float cell(float up, float diag, float left, const Row& r, const Col& c, float arg) {
    const float d = r.x - c.y;
    if (METRIC == DTW) return fmaf(d, d, min3(up, diag, left));
    if (METRIC == ERP) return min3(fmaf(d, d, diag), left + c.gy, up + r.c0);
    if (!FULL) return min3(up, left, diag + (fabsf(d) - arg));
    // MSM: C(x, x', y) = c + the distance of x to [x', y], C(y, x, y') likewise
    const float e2 = fmaxf(arg, fminf(r.c0, fmaf(r.s, d, arg)));
    const float e3 = fmaxf(0.f, fminf(c.ady, __uint_as_float(__float_as_uint(d) ^ c.flip)));
    return min3(up + e2, (left + arg) + e3, diag + fabsf(d));
}

}  // namespace

double mean_step(const double* x, int m) {
    double s = 0.0;
    for (int i = 1; i < m; ++i) s += fabs(x[i] - x[i - 1]);
    return m > 1 ? s / (m - 1) : 0.0;
}

// The screen costs a fifth to a quarter (DTW, ERP) or two fifths (MSM, two passes)
// of the lane-per-candidate DP on windows it drops none of, so a scan that keeps
// over 75% (60%) of its windows does better without.  No z-scored DTW or ERP distance
// lies above twice the query's spread, hardly an MSM distance above 1.5 times; below
// that and from about the spread on a strided sample of the windows is screened
// first (screen_sampled): random walks, z-scored, m = 64 to 600, have their median
// at 0.8 to 1.5 of the spread (DTW), 0.7 to 1.2 (ERP, MSM), their 80th percentile at
// 1.07 to 1.73 and 0.81 to 1.33.  131,072 windows of m = 200, w = 6 at a cutoff that keeps
// all: MSM 1.38 ms with the screen, 0.97 without.
double screen_loose(int metric, double spread, bool raw) { return raw ? DBL_MAX : (metric == MSM ? 1.5 : 2.0) * spread; }

// A sample takes the time of one candidate's full band: scans of seven waves at least.
bool screen_sampled(const DpJob& job, int sm_count) {
    return !job.list && job.n_windows >= 7 * 32LL * sm_count &&
           job.cutoff >= (job.q.metric == DTW ? 1.0 : 0.78) * job.q.spread && job.cutoff < job.q.loose;
}

double query_spread(int metric, const double* x, int m) {
    double mean = 0.0, s = 0.0;
    for (int i = 0; i < m; ++i) mean += x[i] / m;
    for (int i = 0; i < m; ++i) s += metric == MSM ? fabs(x[i] - mean) : (x[i] - mean) * (x[i] - mean);
    return metric == MSM ? s : sqrt(s);
}

// Lists that go on whole.  A warp of the screen steps its 32 candidates one row after
// another, so one with a match in it takes (2w+1) m cells however short the list is,
// while the wavefront's abandon test ends most candidates of a GLB list early.  On
// searches of random walks (rank 10 and 300; m = 2.6 w to 21 w) the two are even at lists of
// 15,000 to 20,000 (w = 6), 16,000 to 30,000 (w = 13), 20,000 to 45,000 (w = 31), 30,000
// to 60,000 (w = 67), 20,000 to 115,000 (w = 96), 30,000 to 180,000 (w = 129; DTW over
// 200,000): MSM, m = 676, w = 129, 21,748 candidates 6.6 ms screened, 1.5 whole;
// 64,861 of a looser cutoff 15 and 25; 973,569 91 and 224.  Past 0.4 of the spread the
// cutoff ends them later and the line falls with it (19,793 windows, m = 126, w = 3, MSM,
// all near the cutoff: 0.26 ms screened, 0.41 whole).  A scan of every window ends
// early too, in proportion to the cutoff: even at 5000 to 11,000 windows of full
// length and, at rank 25 (0.05 to 0.3 of the query's spread), at 46,000 to 230,000 for
// DTW, 60,000 to 124,000 ERP, 20,000 to 114,000 MSM (m = 200, 800).  MSM, m = 800,
// w = 31, 65,536 windows at rank 25: 2.1 ms screened, 1.1 whole.
long long screen_few(const DpJob& job, int sm_count) {
    const int metric = job.q.metric, w = job.q.w;
    const long long wave = 32LL * sm_count;
    // DTW past w = 128: four rows a pass instead of eight
    double waves = metric == MSM ? 4.0 + w / 15.0 : (1.8 + w / 20.0) * (metric == DTW && w > 128 ? 4.0 : 1.0);
    if (!job.lraw) {
        const double most = waves * (metric == MSM ? 2.0 : 3.0), full = w >= 13 ? 2.0 : 1.2;
        const double by_cut = job.cutoff * most <= full * job.q.spread ? most : full * job.q.spread / job.cutoff;
        waves = by_cut > full ? by_cut : full;
    }
    return (long long)(waves * (double)wave);
}

// Rows a pass: four from w = 4 on (ERP's row -4 lies inside the band), DTW eight
// from w = 12.  A pass of R rows has R - 1 columns more than the band at half
// their work.  Measured with two, four and eight rows: DTW w = 13 0.20, 0.148,
// 0.119 ms, w = 26 (8 queries) 3.6, 2.46, 2.07; ERP w = 13 1.13, 0.95, 1.01; MSM
// w = 13 27.9, 21.9, 24.0 (registers).  The widest bands keep two rows, whose
// points still fit a third of an SM's shared memory (up to w = 150).
static int screen_rows(int metric, int w) {
    return w < 4 || w > 149 ? 2 : metric == DTW && w >= 12 && w <= 128 ? 8 : 4;
}

size_t screen_warp_bytes(int metric, int w) {
    return (size_t)(2 * w + 2 + 2 * w + screen_rows(metric, w)) * 32 * sizeof(float);
}

size_t screen_smem_bytes(int metric, int w, int m, int warps) {
    return screen_warp_bytes(metric, w) * warps + (size_t)m * sizeof(float);
}

template <int METRIC, int R>
__global__ void __launch_bounds__(kScreenThreads, METRIC == MSM ? 6 : 1) k_screen(Geom g, DpJob job, long long* __restrict__ out,
                                                           unsigned long long* __restrict__ n_out, long long few) {
    extern __shared__ __align__(16) float scr_smem[];
    const QueryDev& q = job.q;
    const int m = q.m, w = q.w, NR = 2 * w + R;  // points of a pass's columns
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr unsigned kAll = 0xffffffffu;
    float* const A = scr_smem + (size_t)warp * (2 * w + 2 + NR) * 32 + lane;  // band row A[d * 32], d in [0, 2w+1]
    float* const Yr = A + (2 * w + 2) * 32;                                   // points, slot p - (k0-w) + 1 (mod NR)
    float* const X = scr_smem + (size_t)(blockDim.x >> 5) * (2 * w + 2 + NR) * 32;  // [m] query points
    const unsigned long long n_all = job.list ? *job.n_list : (unsigned long long)job.n_windows;
    const unsigned long long n =
        (job.list && n_all > (unsigned long long)job.list_cap) ? job.list_cap : n_all;
    const double cut = job.cutoff_ptr ? *job.cutoff_ptr : job.cutoff;
    const float arg = (float)q.arg;

    const double xm = fmax(-q.qlo, q.qhi);
    const double ymax = 2.0 * xm + (g.raw ? fmin(8.0, 8.0 * xm) : 8.0);
    const double cut_s = cut + 1e-9 * (1.0 + fabs(cut));
    // FP32 points (RelMap's range test below): off by 2^-17 + 2^-23 Y more
    const double rel_err = job.rel ? 0x1.02p-17 + 0x1p-23 * ymax : 0.0;
    const double delta = 0x1p-22 * (xm + ymax + fabs(q.arg)) * 1.01 + rel_err;
    const double G = 1.0 + (2.0 * m + 16.0) * 0x1p-23 * 1.01;
    double Rc, Eb;
    if (METRIC == MSM) {
        Rc = cut_s;
        Eb = (2.0 * m + 2.0) * (delta + 0x1p-23 * fabs(q.arg));
    } else {
        const double e = delta * sqrt(2.0 * m + 2.0);
        Rc = cut_s * cut_s * (1.0 + 0x1p-50);
        Eb = 2.0 * e * cut_s + e * e;
    }
    const double lim_all = (Rc + Eb) * G * (1.0 + 0x1p-20);
    // nothing to gain (a short list, shorter at cutoffs past 0.4 of the spread, where
    // the wavefront ends a GLB list later; a scan's loose cutoff, a sample that stayed)
    // or no proof possible (distances past FP32's exact range; points far from zero
    // that lie closer together than FP32 tells apart): every valid candidate goes on
    bool pass = (n <= (unsigned long long)few && !(job.lraw && (double)n * cut > 0.4 * q.spread * (double)few)) ||
                (!job.list && cut >= q.loose) || !(lim_all < 1e12) || !(xm + ymax + fabs(q.arg) < 1e9) ||
                !(Eb < (METRIC == MSM ? q.spread : q.spread * q.spread));
    if (job.sample) pass = pass || 20 * job.sample[1] >= (METRIC == MSM ? 12 : 15) * job.sample[0];
    const float ylim = (float)ymax, narrow = (float)(0x1p-21 * ymax + 1.01 * rel_err);
    const float far_lim = (float)(((METRIC == MSM ? fmax(Rc, 0.0) : sqrt(Rc)) +
                                   fmax(xm, METRIC == ERP ? fabs(q.arg) : 0.0) + 2.0 * delta) * (1.0 + 0x1p-19));
    const float grow = (float)(1.0 + (m + 16.0) * 0x1p-23);

    // MSM: the intervals add at most |x - x'| to a step's cost c; a mean of c/2
    // keeps the first pass's cells within about a half of the second's
    const bool rough = METRIC == MSM && q.step <= 0.5 * q.arg;
    if (!pass) {
        for (int i = threadIdx.x; i < m; i += blockDim.x) X[i] = (float)q.qn[i];
        __syncthreads();
    }
    unsigned long long valid_count = 0, cells = 0;
    const int erp = METRIC == ERP ? 1 : 0;
    // first row of the first pass: row 0 (ERP: -1, the empty prefix), earlier when
    // that makes the number of rows a multiple of R
    const int k0 = -erp - (R - (m + erp) % R) % R;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(job.next, 32ull);
        base = __shfl_sync(kAll, base, 0);
        if (base >= n) break;
        const unsigned long long item = base + lane;
        bool active = item < n;
        long long gi = 0, s = 0;
        int j = 0;
        double mu = 0.0, sg = 1.0, S = 0.0;
        bool casc = false;
        if (active) {
            gi = job.list ? job.list[item] : (long long)item * (job.stride ? job.stride : 1);
            g.locate(gi, &s, &j);
            mu = job.MU[s * g.kml + j];
            sg = job.SIG[s * g.kml + j];
            active = !window_invalid(sg, g, gi);
            if (active) ++valid_count;
            if (active && job.list_s && job.lraw) {
                S = job.list_s[item];
                casc = S >= 0.0;
            }
        }
        if (!active) gi = 0;
        bool keep = active;
        float far = 0.f;  // the furthest of the points so far (a NaN stays)
        auto run = [&](auto full_c) {
            constexpr bool FULL = decltype(full_c)::value;
            const double inv = 1.0 / sg;
            const double* __restrict__ tp = job.target + gi;
            const double* __restrict__ lr = job.lraw + gi;
            const double* __restrict__ ur = job.uraw + gi;
            const bool warp_casc = __any_sync(kAll, casc);
            // FP32 points relative to the segment while its half range and the
            // mean's place in it stay below 64 sigma
            float ra = 0.f, rb = 0.f;
            bool rel_ok = !active;
            const float* rp = nullptr;
            if (job.rel) {
                rp = job.rel + (s * g.m_k + j);
                if (active) {
                    const double2 sr = job.rseg[s];
                    ra = (float)inv;
                    const double p = (sr.x - mu) * (double)ra;
                    rb = (float)p;
                    rel_ok = inv > 1e-30 && inv < 1e30 && sr.y < 1e30 && sr.y * inv <= 64.0 && fabs(p) <= 64.0;
                }
            }
            const bool fast = job.rel && __all_sync(kAll, rel_ok);
            const long long N = g.S * g.m_k;
            auto pack = [](float v) { return __hiloint2double(0, __float_as_int(v)); };
            auto unpack = [&](double v) { return fmaf(__int_as_float(__double2loint(v)), ra, rb); };
            auto inner = [&](int k) { return fast && k >= max(w, 1) && k + R - 1 <= min(m - 1 - w, m - 2); };
            // (R - S + Pre + E) G: the part known before the first row, rounded up
            const float lim0 = (float)((Rc - (casc ? S : 0.0) + Eb) * G + 0x1p-20 * lim_all);
            const float limg = (float)(G * (1.0 + 0x1p-22)) * grow;
            float pre = 0.f;
            // ring: point k0 - w in slot 1, so a pass's columns R-1, R start on an even slot
            auto point = [&](int p, double raw) {
                float y = p < 0 ? -kOut : kOut;
                if (p >= 0 && p < m) {
                    y = fast ? unpack(raw) : (float)((raw - mu) * inv);
                    asm("max.NaN.f32 %0, %0, %1;" : "+f"(far) : "f"(fabsf(y)));
                }
                return y;
            };
            for (int d = 0; d < 2 * w + 2; ++d) A[d * 32] = kBlock;
            // the cell that the first row grows from (see the rows above the matrix below)
            A[(w + (erp ? -k0 : 0)) * 32] = slot<FULL>(0.f, arg);
            for (int i = 0; i < NR; ++i) {
                const int p = k0 - w + i;
                const bool in = active && p >= 0 && p < m;
                const double raw = !in ? 0.0 : fast ? pack(rp[p]) : tp[p];
                Yr[((i + 1) % NR) * 32] = point(p, raw);
            }
            int b = 1;  // slot of the pass's first column
            auto ring = [&](int i) { return b + i >= NR ? b + i - NR : b + i; };
            // points of the next pass, loaded a pass ahead
            double nx[R];
            auto load = [&](int k) {
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    const int p = k + w + u;
                    const bool in = active && p >= 0 && p < m;
                    nx[u] = !in ? 0.0 : fast ? pack(rp[p]) : tp[p];
                }
            };
            // the term of row k on its narrowed window
            auto term = [&](float lo, float up, float x) {
                const float e = fmaxf(fmaxf((lo + narrow) - x, x - (up - narrow)), 0.f);
                if (METRIC == MSM) return fminf(e, arg * (1.f + 0x1p-22f));
                if (METRIC == ERP) return fminf(e * e, (fabsf(x - arg) + narrow) * (fabsf(x - arg) + narrow));
                return e * e;
            };
            float yl0 = -kOut;  // the point left of the pass's first column (MSM)
            for (int k = k0; k < m; k += R) {
                // rows above the matrix: x = -1e15 matches the padding left of it
                // at no cost and nothing else, so the zero travels down the
                // diagonal (DTW, MSM) or straight down (ERP, whose row -1 then
                // gathers the deletions of the prefix) to the first real row
                Row r[R];
#pragma unroll
                for (int u = 0; u < R; ++u) {
                    const int kk = k + u;
                    const float x = kk >= 0 ? X[kk] : -kOut;
                    r[u].x = x;
                    r[u].c0 = r[u].s = 0.f;
                    if (METRIC == ERP) r[u].c0 = kk >= 0 ? (x - arg) * (x - arg) : 0.f;
                    if (METRIC == MSM && FULL) {
                        const float xp = kk >= 1 ? X[kk - 1] : -kOut;
                        r[u].c0 = fabsf(x - xp) + arg;
                        r[u].s = x >= xp ? 1.f : -1.f;
                    }
                }
                if (k + R < m) load(k + R);
                float el[R], eu[R];  // the rows' centred windows, for the test at the pass's end
                const bool mid = warp_casc && inner(k);
                if (mid) {
#pragma unroll
                    for (int u = 0; u < R; ++u) {
                        el[u] = casc ? rp[N + k + u] : 0.f;
                        eu[u] = casc ? rp[2 * N + k + u] : 0.f;
                    }
                }
                // the pass, column by column: row u's cell there is band cell c - u
                float ext = kBlock, pv[R];
#pragma unroll
                for (int u = 0; u < R; ++u) pv[u] = kBlock;
                float yp = yl0, pd = A[0];
                auto column = [&](float y, float diag0, float up0, int lo, int hi) {  // rows lo .. hi
                    const Col c = make_col<METRIC>(y, yp, arg);
                    float diag = diag0, up = up0, last = kBlock;
#pragma unroll
                    for (int u = 0; u < R; ++u) {
                        if (u < lo || u > hi) {
                            diag = pv[u];
                            pv[u] = up = kBlock;
                            continue;
                        }
                        const float v = cell<METRIC, FULL>(up, diag, pv[u], r[u], c, arg);
                        diag = pv[u];
                        pv[u] = up = slot<FULL>(v, arg);
                        last = v;
                    }
                    yp = y;
                    return last;
                };
                // columns 0 .. R-2: the upper rows only
#pragma unroll
                for (int c = 0; c < R - 1; ++c) {
                    const float pn = A[(c + 1) * 32];
                    column(Yr[ring(c) * 32], pd, pn, 0, c);
                    pd = pn;
                }
                // columns R-1 .. 2w, two at a time (even slots: no wrap inside a two)
                const int all = w - R / 2 + 1;
                int sl = ring(R - 1), d = R - 1;
                const int first = min(all, (NR - sl) >> 1);
#pragma unroll 1
                for (int part = 0; part < 2; ++part) {
                    const int cnt = part ? all - first : first;
                    const float* yptr = Yr + sl * 32;
                    float* aptr = A + d * 32;
#pragma unroll 2
                    for (int t = 0; t < cnt; ++t) {
                        const float ya = yptr[0], yb = yptr[32];
                        const float pna = aptr[32], pnb = aptr[64];
                        const float l1 = column(ya, pd, pna, 0, R - 1);
                        aptr[-32 * (R - 1)] = pv[R - 1];
                        const float l2 = column(yb, pna, pnb, 0, R - 1);
                        aptr[-32 * (R - 2)] = pv[R - 1];
                        ext = min3(ext, l1, l2);
                        pd = pnb;
                        yptr += 64;
                        aptr += 64;
                    }
                    sl = 0;
                    d += 2 * cnt;
                }
                // columns 2w+1 .. 2w+R-1: the lower rows only
#pragma unroll
                for (int c = 1; c < R; ++c) {
                    const float l1 = column(Yr[ring(2 * w + c) * 32], kBlock, kBlock, c, R - 1);
                    A[(2 * w + c - R + 1) * 32] = pv[R - 1];
                    ext = fminf(ext, l1);
                }
                cells += active ? (unsigned long long)(2 * w + 1) * R : 0ull;
                // the next pass starts R columns on: the slots of this pass's
                // first R columns take its last R points
                if (METRIC == MSM && FULL) yl0 = Yr[ring(R - 1) * 32];
                if (k + R < m) {
#pragma unroll
                    for (int u = 0; u < R; ++u) Yr[ring(u) * 32] = point(k + R + w + u, nx[u]);
                    b += R;
                    if (b >= NR) b -= NR;
                }
                // terms of the pass's rows
                if (mid) {
#pragma unroll
                    for (int u = 0; u < R; ++u)
                        pre += casc ? term(fmaf(el[u], ra, rb), fmaf(eu[u], ra, rb), r[u].x) : 0.f;
                } else if (warp_casc) {
                    for (int u = 0; u < R; ++u) {
                        const int kk = k + u;
                        if (!(casc && active && kk >= 1 && kk <= m - 2)) continue;
                        const int p0 = qt_p0(kk, w), p1 = qt_p1(kk, m, w);
                        const double a = lr[p0] < lr[p1] ? lr[p0] : lr[p1], c = ur[p0] > ur[p1] ? ur[p0] : ur[p1];
                        pre += term((float)((a - mu) * inv), (float)((c - mu) * inv), X[kk]);
                    }
                }
                if (!(far <= ylim)) {  // the rows' bound does not cover it
                    if (far > far_lim && far <= FLT_MAX) keep = false;
                    active = false;
                } else if (active && ext > fmaf(pre, limg, lim0)) {
                    active = keep = false;
                }
                if (!__any_sync(kAll, active)) break;
            }
            // the last row's cell (m-1, m-1)
            const double last = FULL ? (double)A[w * 32] : (double)A[w * 32] * (1.0 - 0x1p-22) - (double)arg;
            if (active && last > lim_all) keep = false;
        };
        if (!pass && __any_sync(kAll, active)) {
            if (METRIC == MSM && rough) {
                run(std::false_type{});
                active = keep && far <= ylim;
                __syncwarp();
            }
            if (__any_sync(kAll, active)) run(std::true_type{});
        }
        const unsigned mask = __ballot_sync(kAll, keep);
        if (mask) {
            unsigned long long o = 0;
            if (lane == 0) o = atomicAdd(n_out, (unsigned long long)__popc(mask));
            o = __shfl_sync(kAll, o, 0) + __popc(mask & ((1u << lane) - 1));
            if (keep) out[o] = gi;
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

const void* screen_kernel(int metric, int w) {
    const int rows = screen_rows(metric, w);
    switch (metric) {
        case DTW:
            return rows == 8 ? (const void*)k_screen<DTW, 8>
                 : rows == 4 ? (const void*)k_screen<DTW, 4> : (const void*)k_screen<DTW, 2>;
        case ERP: return rows == 4 ? (const void*)k_screen<ERP, 4> : (const void*)k_screen<ERP, 2>;
        case MSM: return rows == 4 ? (const void*)k_screen<MSM, 4> : (const void*)k_screen<MSM, 2>;
        default: return nullptr;
    }
}

}  // namespace fsm
