// GLB second filter (src/glb.cpp:200-373), split in the reference's own two
// directions:
//  * k_glb_tq: one lane per LB_IP survivor, the boundary term and the T->Q sum
//    (candidate points against the query's envelope);
//  * k_glb_qt: one lane per T->Q survivor, the Q->T sum (query points against
//    the candidate's envelope).  The candidate envelope (lower_upper_lemire of
//    the z-normalised window, src/glb.cpp:302-304) is never materialised:
//    z-normalisation x -> (x - mu) / sigma is monotone even after rounding, so
//    the minimum of the normalised points equals the normalised minimum of the
//    raw points, bit for bit; every envelope point is the min/max of two
//    forward windows of the target, an interior one (w <= k <= m-1-w) a value
//    of the centred windows (k_rel).  On short lists 8 lanes share a candidate:
//    one lane's chain of loads is what such a launch waits for.
// What GLB decides is whether boundary + T->Q and boundary + Q->T stay within
// the cutoff (LCSS: whether both counts reach it): running sums never decrease
// and rounding is monotone, so glb <= cutoff exactly when both hold, and when
// a sum is abandoned makes no difference.
//
// So the sums are taken in fixed point and single precision with a proven
// margin, and only a candidate whose sum falls within the margin of the limit
// is decided by the reference's FP64 operations (exact_tq, exact_qt).
//   * One FP64 fused multiply-add turns a raw point into a fixed-point number
//     and an FP32 one at once: v = fl(t A + B), A = 2^K / sigma, B = M - mu A,
//     with M = 1.5 2^52 + 0x4b400000.  The low word of v is then the bit
//     pattern of the float F = 1.5 2^23 + n, n the integer next to y 2^K, off
//     the reference's normalised point by at most 1.01 units of 2^-K (0.5 from
//     B, 0.5 from v).  No conversion instruction (14 a cycle and SM against 64
//     for the multiply-add).  K is the largest with |y| 2^K < 2^22 for
//     |y| <= sqrt(m) (raw mode: four times the query's half range around its
//     middle, which M then carries); a point outside shows in the upper bits,
//     and its candidate is decided in FP64.
//   * Differences of such floats are exact integers; with the query's side
//     rounded to units too, each is off by less than 2 units (ERP with a gap
//     far outside: by its FP32 rounding more).
//   * DTW, ERP: the sum of squares is the squared norm of the differences
//     (boundary terms among them), so its root is off by at most 2 sqrt(m+2)
//     units (triangle inequality); MSM: the sum by 2 (m+4) units (its boundary
//     is continuous in its arguments); the FP32 sums by a relative (m+16) 2^-23.
//   * EDR, LCSS: terms are 0 or 1; those within 2 units of the tolerance count
//     as 0 in one total and as 1 in the other.
//   * From 2^18 points on the points come in FP32, relative to the middle of
//     their segment's range (k_rel): one FP32 multiply-add gives F, from half the
//     bytes and without a range test (RelMap).  A warp with a window whose sigma
//     is small against that range takes the FP64 points.
// What bounds it: instruction issue, about 8 instructions a point (T->Q; 14 with
// FP64 points) and 11 (Q->T; 18, with the L1 path 84% busy) where the FP64 sums
// took 45 and 90 issue slots.  Measured on the five-metric workload (2^24 points,
// m = 256, w = 13), T->Q and Q->T of all five queries: 19.3 and 14.6 ms with FP64
// sums, 10.1 and 6.5 ms with fixed point, 7.9 and 5.2 ms with FP32 points (and
// 0.1 ms for k_rel); 8 top-k queries (m = 512, 2^23 points) 18.6 and 7.6, 4.5 and
// 1.4, 3.4 and 1.2 ms.  Q->T of 20 queries of mixed length with some thousand
// candidates each: 1.5 ms a lane per candidate, 1.05 ms 8 lanes.
#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

namespace {

__device__ __forceinline__ double edr_sub(double a, double b, double eps) {
    return (fabs(dsub(a, b)) <= eps) ? 0.0 : 1.0;
}
__device__ __forceinline__ double dminv(double a, double b) { return (a < b) ? a : b; }  // MIN macro
__device__ __forceinline__ double dmaxv(double a, double b) { return (a > b) ? a : b; }  // MAX macro

// warp-aggregated append; returns nothing, writes entry via functor
template <typename F>
__device__ __forceinline__ void warp_append(bool pred, unsigned long long* counter, F write) {
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (!mask) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) write(base + __popc(mask & ((1u << lane) - 1)));
}

// N quotients dividend(u) / sg (zdiv) with one range test for the group: a
// group with any estimate outside the reciprocal method's range (zero
// dividends, extreme scales) is divided directly -- the same bits either way,
// one branch per group instead of one per point.  The rare direct path
// evaluates the dividends again rather than keeping them live.
template <int N, typename F>
__device__ __forceinline__ void zdiv_group(F dividend, double sg, double inv, bool ok, double (&z)[N]) {
    bool good = ok;
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const double a = dividend(u);
        const double q0 = rcp_div_estimate(a, inv);
        good = good & (rcp_div_in_range_bits(q0) != 0);
        z[u] = rcp_div_finish(a, sg, inv, q0);
    }
    if (!good) {
#pragma unroll
        for (int u = 0; u < N; ++u) z[u] = ddiv(dividend(u), sg);
    }
}

// T->Q term of normalised candidate point t against the query envelope
// [lo, hi] at the same index (src/glb.cpp:230-300), written with selects so
// lanes never split on the data.  lo <= hi, so at most one of t < lo, t > hi
// holds: the side is selected first and one distance computed to it.
template <int METRIC>
__device__ __forceinline__ double tq_term(double t, double lo, double hi, double arg) {
    const bool below = t < lo, above = t > hi;
    const double e = above ? hi : lo;  // the nearer side when outside
    if (METRIC == DTW) {
        const double a = dsq(t, e);
        return (below || above) ? a : 0.0;
    } else if (METRIC == ERP) {
        const double a = dminv(dsq(t, e), dsq(t, arg));
        return (below || above) ? a : 0.0;
    } else if (METRIC == EDR) {
        const double a = edr_sub(t, e, arg);
        return (below || above) ? a : 0.0;
    } else if (METRIC == LCSS) {  // match indicator: lo - t or t - hi within eps
        const bool a = dsub(below ? lo : t, below ? t : hi) <= arg;
        return ((below || above) ? a : true) ? 1.0 : 0.0;
    } else {  // MSM
        const double a = dminv(fabs(dsub(t, e)), arg);
        return (below || above) ? a : 0.0;
    }
}

// boundary term in the reference's operations (src/glb.cpp:200-230)
template <int METRIC>
__device__ __forceinline__ double boundary_exact(const double* __restrict__ Q, int m, double arg,
                                                 const double* __restrict__ tp, double mu, double sg, double inv,
                                                 bool rok) {
    if (METRIC == LCSS) return 0.0;
#define TN(k) zdiv_i(dsub(tp[(k)], mu), sg, inv, rok)
    const double T0 = TN(0), TL = TN(m - 1);
    if (METRIC == DTW) {
        return dadd(dsq(T0, Q[0]), dsq(TL, Q[m - 1]));
    } else if (METRIC == ERP) {
        return dmin3(dsq(Q[m - 1], TL), dsq(Q[m - 1], arg), dsq(TL, arg));
    } else if (METRIC == EDR) {
        return dminv(edr_sub(Q[m - 1], TL, arg), 1.0);
    } else if (METRIC == MSM) {
        const double T2 = TN(m - 2);
        const double q0 = Q[0], ql = Q[m - 1], ql2 = Q[m - 2];
        if ((T2 >= TL && TL >= ql) || (T2 <= TL && TL <= ql) || (ql2 <= ql && ql <= TL) ||
            (ql2 >= ql && ql >= TL)) {
            return dadd(fabs(dsub(q0, T0)), dminv(fabs(dsub(ql, TL)), arg));
        } else {
            return dadd(fabs(dsub(q0, T0)),
                            dmin3(fabs(dsub(ql, TL)), dadd(arg, fabs(dsub(TL, T2))),
                                  dadd(arg, fabs(dsub(ql, ql2)))));
        }
    }
#undef TN
    return 0.0;
}

// boundary term and T->Q sum in the reference's operations; false: abandoned
template <int METRIC>
__device__ __noinline__ bool exact_tq(const double* __restrict__ Q, const double* __restrict__ LQ,
                                      const double* __restrict__ UQ, int m, double arg,
                                      const double* __restrict__ tp, double mu, double sg, double bsf,
                                      double& boundary_out, double& tq_out) {
    double boundary, tq;
    const double inv = __drcp_rn(sg);
    const bool rok = rcp_div_in_range(sg);
    const double lim = (METRIC == DTW || METRIC == ERP) ? dmul(bsf, bsf) : bsf;  // src/glb.cpp:28-31
    bool alive = true;
    boundary = tq = 0.0;
#define TN(k) zdiv_i(dsub(tp[(k)], mu), sg, inv, rok)
    boundary = boundary_exact<METRIC>(Q, m, arg, tp, mu, sg, inv, rok);
    if (METRIC == LCSS) {
        // every point, no abandon (src/glb.cpp:238-252)
        const double min_len = (double)m;
        int k = 0;
        for (; k + 4 <= m; k += 4) {
            double z4[4], t4[4];
            zdiv_group([&](int u) { return dsub(tp[k + u], mu); }, sg, inv, rok, z4);
#pragma unroll
            for (int u = 0; u < 4; ++u) t4[u] = tq_term<LCSS>(z4[u], LQ[k + u], UQ[k + u], arg);
#pragma unroll
            for (int u = 0; u < 4; ++u) tq = dadd(tq, t4[u]);
        }
        for (; k < m; ++k) tq = dadd(tq, tq_term<LCSS>(TN(k), LQ[k], UQ[k], arg));
        if (dmax0(dsub(1.0, ddiv(tq, min_len))) > bsf) alive = false;
    } else {
        // points 1..m-2 four at a time: the four normalisations are
        // independent, the sum takes them in the reference's order, and
        // the abandon test runs once per group -- the sum never
        // decreases, so a sum past the limit anywhere in the group is
        // past it at the group's end (the same decision)
        int k = 1;
        for (; k + 4 <= m - 1; k += 4) {
            double z4[4], t4[4];
            zdiv_group([&](int u) { return dsub(tp[k + u], mu); }, sg, inv, rok, z4);
#pragma unroll
            for (int u = 0; u < 4; ++u) t4[u] = tq_term<METRIC>(z4[u], LQ[k + u], UQ[k + u], arg);
#pragma unroll
            for (int u = 0; u < 4; ++u) tq = dadd(tq, t4[u]);
            if (dadd(boundary, tq) > lim) { alive = false; break; }
        }
        if (alive) {
            for (; k < m - 1; ++k) tq = dadd(tq, tq_term<METRIC>(TN(k), LQ[k], UQ[k], arg));
            if (m > 2 && dadd(boundary, tq) > lim) alive = false;  // m = 2 has no inner point to test at
        }
    }
#undef TN
    boundary_out = boundary;
    tq_out = tq;
    return alive;
}

// the Q->T sum in the reference's operations and order
template <int METRIC>
__device__ __noinline__ double exact_qt(const double* __restrict__ Q, int m, int w, double arg,
                                        const double* __restrict__ lf, const double* __restrict__ uf, double mu,
                                        double sg) {
    const double inv = __drcp_rn(sg);
    const bool rok = rcp_div_in_range(sg);
    double qt = 0.0;
    const int k0 = (METRIC == LCSS) ? 0 : 1, k1 = (METRIC == LCSS) ? m - 1 : m - 2;
    // the terms are independent (unrolled so their loads and divisions
    // overlap); only the sum is sequential, in the reference's order.
    // Interior points (w <= k <= m-1-w) read the windows at k-w and k
    // directly; the edges take the clamped indices.
    const int i0 = max(k0, w), i1 = min(k1, m - 1 - w);
    int k = k0;
    for (; k <= k1 && k < i0; ++k) qt = dadd(qt, qt_term(METRIC, Q[k], k, m, w, lf, uf, mu, sg, inv, rok, arg));
    for (; k + 1 <= i1; k += 2) {  // two points, four quotients, one range test
        double z4[4];
        zdiv_group(
            [&](int u) {
                const int kk = k + (u & 1);
                if (u < 2) { const double a0 = lf[kk - w], a1 = lf[kk]; return dsub((a1 < a0) ? a1 : a0, mu); }
                const double b0 = uf[kk - w], b1 = uf[kk];
                return dsub((b0 < b1) ? b1 : b0, mu);
            },
            sg, inv, rok, z4);
        qt = dadd(qt, qt_term_norm(METRIC, Q[k], z4[0], z4[2], arg));
        qt = dadd(qt, qt_term_norm(METRIC, Q[k + 1], z4[1], z4[3], arg));
    }
    for (; k <= i1; ++k) {
        const double a0 = lf[k - w], a1 = lf[k], b0 = uf[k - w], b1 = uf[k];
        qt = dadd(qt, qt_term_env(METRIC, Q[k], (a1 < a0) ? a1 : a0, (b0 < b1) ? b1 : b0, mu, sg, inv, rok,
                                  arg));
    }
    for (; k <= k1; ++k) qt = dadd(qt, qt_term(METRIC, Q[k], k, m, w, lf, uf, mu, sg, inv, rok, arg));
    return qt;
}

// The same two sums with a warp per candidate, every lane with the same
// arguments and the same results: the terms of 32 points at a time, added in
// the reference's order.  One lane alone waits for each of its loads; most
// warps that come here have one candidate to decide.
template <int METRIC>
__device__ __noinline__ bool warp_tq(const double* __restrict__ Q, const double* __restrict__ LQ,
                                     const double* __restrict__ UQ, int m, double arg,
                                     const double* __restrict__ tp, double mu, double sg, double bsf,
                                     double& boundary_out, double& tq_out) {
    const int lane = threadIdx.x & 31;
    const double inv = __drcp_rn(sg);
    const bool rok = rcp_div_in_range(sg);
    const double lim = (METRIC == DTW || METRIC == ERP) ? dmul(bsf, bsf) : bsf;
    double boundary = boundary_exact<METRIC>(Q, m, arg, tp, mu, sg, inv, rok), tq = 0.0;
    bool alive = true;
    const int kb = METRIC == LCSS ? 0 : 1, ke = METRIC == LCSS ? m : m - 1;
    for (int k0 = kb; k0 < ke && alive; k0 += 32) {
        const int k = min(k0 + lane, ke - 1);
        const double term = tq_term<METRIC>(zdiv_i(dsub(tp[k], mu), sg, inv, rok), LQ[k], UQ[k], arg);
        for (int j = 0; j < min(32, ke - k0); ++j) tq = dadd(tq, __shfl_sync(0xffffffffu, term, j));
        if (METRIC != LCSS && dadd(boundary, tq) > lim) alive = false;
    }
    if (METRIC == LCSS) {
        if (dmax0(dsub(1.0, ddiv(tq, (double)m))) > bsf) alive = false;
    } else if (m > 2 && dadd(boundary, tq) > lim) {
        alive = false;
    }
    boundary_out = boundary;
    tq_out = tq;
    return alive;
}

template <int METRIC>
__device__ __noinline__ double warp_qt(const double* __restrict__ Q, int m, int w, double arg,
                                       const double* __restrict__ lf, const double* __restrict__ uf, double mu,
                                       double sg) {
    const int lane = threadIdx.x & 31;
    const double inv = __drcp_rn(sg);
    const bool rok = rcp_div_in_range(sg);
    const int kb = METRIC == LCSS ? 0 : 1, ke = METRIC == LCSS ? m : m - 1;
    double qt = 0.0;
    for (int k0 = kb; k0 < ke; k0 += 32) {
        const int k = min(k0 + lane, ke - 1);
        const double term = qt_term(METRIC, Q[k], k, m, w, lf, uf, mu, sg, inv, rok, arg);
        for (int j = 0; j < min(32, ke - k0); ++j) qt = dadd(qt, __shfl_sync(0xffffffffu, term, j));
    }
    return qt;
}
constexpr int kWarpExact = 6;  // candidates of a warp decided one after another by the whole warp

// ------------------------------------------------ fixed point and FP32 sums

constexpr double kM = 6755399441055744.0 + (double)0x4b400000;  // 1.5 * 2^52 + the bits of the float 1.5 * 2^23
constexpr unsigned kMHi = 0x43380000u;             // upper word of every in-range v

// Scale and limits of one query at one cutoff, in units of 2^-K.
struct Fix {
    double scale;     // 2^K
    double mid;       // units of the middle of the range
    double eta;       // how far a sum (its root) may be off
    float hi, lo;     // a total above hi exceeds the limit, one of at most lo does not
    float a;          // ERP: the gap as F; MSM: the cost
    float e1, e0;     // EDR, LCSS: a distance above e1 misses for certain, one below e0 matches
    int most;         // EDR, LCSS: the misses the cutoff allows
    bool exact;       // everything in FP64
};

template <int METRIC>
__device__ __forceinline__ Fix make_fix(const QueryDev& q, double bsf, bool raw, bool rel) {
    Fix f;
    const int m = q.m;
    const double xl = q.qlo, xh = q.qhi;
    const double ymax = raw ? 2.0 * (xh - xl) + 1.0 : fmax(fmax(xh, -xl), sqrt((double)m)) * 1.01 + 1.0;
    f.exact = !(ymax < 1e200) || !(bsf < kGlbMax);
    int K = f.exact ? 0 : 21 - ilogb(ymax);  // ymax 2^K < 2^22
    // FP32 points need H 2^K / sigma <= 2^21 (H: half the segment's range): K no
    // larger than leaves room for H up to 64 (32) sigma, which one warp of 32
    // neighbouring windows in 1000 exceeds on random walks; a unit stays far
    // below what separates candidates (the linear sums and counts take more)
    if (rel && !f.exact) K = raw ? K - 5 : min(K, METRIC == DTW || METRIC == ERP ? 15 : 16);
    f.scale = scalbn(1.0, K);
    f.mid = raw && !f.exact ? rint(0.5 * (xl + xh) * f.scale) : 0.0;
    f.exact |= !(fabs(f.mid) < 0x1p50);
    const double U = bsf * f.scale, arg = q.arg * f.scale;
    const double rho = (m + 16.0) * 0x1p-23;
    f.hi = f.lo = f.a = f.e1 = f.e0 = 0.f;
    f.eta = 0.0;
    f.most = 0;
    if (METRIC == DTW || METRIC == ERP || METRIC == MSM) {
        double hi, lo;
        if (METRIC == MSM) {
            const double eta = 2.0 * (m + 4.0);
            f.eta = eta;
            hi = (U + eta) * (1.0 + rho);
            lo = (U - eta) * (1.0 - rho);
            f.a = (float)arg;
            f.exact |= !(arg < 1e30);
        } else {
            double unit = 2.0;
            if (METRIC == ERP) {
                const double ga = rint(arg - f.mid);
                if (!(fabs(ga) < 0x1p22)) unit += (fabs(ga) + 0x1p24) * 0x1p-22;
                f.a = (float)(12582912.0 + ga);
                f.exact |= !(fabs(ga) < 0x1p60);
            }
            const double eta = unit * sqrt(m + 2.0);
            hi = (U + eta) * (U + eta) * (1.0 + rho);
            lo = U > eta ? (U - eta) * (U - eta) * (1.0 - rho) : -1.0;
            f.eta = eta;
        }
        f.hi = __double2float_ru(hi);
        f.lo = __double2float_rd(lo);
        f.exact |= !(hi < 1e37);
    } else {
        f.e1 = __double2float_ru(arg * (1.0 + 0x1p-22) + 2.0);
        f.e0 = __double2float_rd(arg * (1.0 - 0x1p-22) - 2.0);
        if (METRIC == EDR) {
            f.most = f.exact ? 0 : (int)bsf;
        } else {  // the fewest matches whose bound does not exceed the cutoff
            int a = 0, b = m;
            while (a < b) {
                const int mid = (a + b) >> 1;
                if (dmax0(dsub(1.0, ddiv((double)mid, (double)m))) > bsf) a = mid + 1;
                else b = mid;
            }
            f.most = m - a;
        }
    }
    return f;
}

// One candidate's map from raw points to F, with the upper bits collected.
struct FixMap {
    double A, B;
    unsigned badh, badl;
    __device__ __forceinline__ bool init(double mu, double sg, const Fix& f) {
        A = __drcp_rn(sg) * f.scale;
        const double p = mu * A;
        B = fma(-mu, A, kM - f.mid);
        badh = badl = 0u;
        return fabs(p) < 0x1p51 && A < 0x1p900 && A > 0x1p-900;
    }
    __device__ __forceinline__ float at(double t) {  // with range check
        const double v = fma(t, A, B);
        const unsigned l = (unsigned)__double2loint(v);
        badh |= (unsigned)__double2hiint(v) ^ kMHi;
        badl |= l ^ 0x4b000000u;
        return __uint_as_float(l);
    }
    __device__ __forceinline__ float at_checked(double t) const {  // T->Q has checked every point of the window
        return __uint_as_float((unsigned)__double2loint(fma(t, A, B)));
    }
    __device__ __forceinline__ bool bad() const { return (badh | (badl & 0xff800000u)) != 0u; }
};

// One candidate's map from FP32 points relative to its segment to F: off by
// less than 1.4 units where the segment allows it (ok), 0.125 from the point,
// 0.25 from A, 0.5 from B, 0.5 from the sum, and always in range.
struct RelMap {
    float A, B;
    bool ok;
    __device__ __forceinline__ RelMap() : A(0.f), B(0.f), ok(false) {}
    __device__ __forceinline__ RelMap(double a, double mu, double2 seg, double mid) {
        constexpr double kMost = 0x1p21 * (1.0 - 0x1p-10);
        A = (float)a;
        const double p = fma(mu - seg.x, (double)A, mid);
        B = (float)(12582912.0 - p);
        ok = A > 1e-30f && A < 1e30f && seg.y < 1e30 && seg.y * (double)A <= kMost && fabs(p) <= kMost;
    }
    __device__ __forceinline__ float at(float t) const { return fmaf(t, A, B); }
};

// Sum (DTW, ERP, MSM) or certain / possible misses (EDR, LCSS).
struct Acc {
    float s = 0.f;
    int c1 = 0, c2 = 0;
};

// the term of x against [lo, up]; gap: ERP's distance to the gap value
template <int METRIC>
__device__ __forceinline__ void acc_add(Acc& a, float x, float lo, float up, float gap, const Fix& f) {
    if (METRIC == EDR || METRIC == LCSS) {
        const float e = fmaxf(lo - x, x - up);  // signed: inside is certain for small tolerances too
        a.c1 += e > f.e1 ? 1 : 0;
        a.c2 += e >= f.e0 ? 1 : 0;
        return;
    }
    float e = fmaxf(fmaxf(lo - x, x - up), 0.f);
    if (METRIC == DTW) {
        a.s = fmaf(e, e, a.s);
    } else if (METRIC == ERP) {
        e = fminf(e, fabsf(gap));
        a.s = fmaf(e, e, a.s);
    } else {
        a.s += fminf(e, f.a);
    }
}

// the boundary terms of points 0 and m-1 (and m-2), src/glb.cpp:200-230
template <int METRIC>
__device__ __forceinline__ Acc acc_boundary(FixMap& map, const double* __restrict__ tp, const float2* __restrict__ Qx,
                                            int m, const Fix& f) {
    Acc a;
    if (METRIC == LCSS) return a;
    const float TL = map.at(tp[m - 1]), ql = Qx[m - 1].x;
    // EDR and ERP have no term of point 0, but Q->T's envelopes hold it: its range
    // is checked with the others'
    if (METRIC == EDR || METRIC == ERP) map.at(tp[0]);
    if (METRIC == EDR) {
        const float e = fabsf(ql - TL);
        a.c1 = e > f.e1 ? 1 : 0;
        a.c2 = e >= f.e0 ? 1 : 0;
    } else if (METRIC == ERP) {
        const float d = fminf(fabsf(ql - TL), fminf(fabsf(ql - f.a), fabsf(TL - f.a)));
        a.s = d * d;
    } else {
        const float d0 = map.at(tp[0]) - Qx[0].x, dl = fabsf(ql - TL);
        if (METRIC == DTW) {
            a.s = fmaf(d0, d0, dl * dl);
        } else {
            const float T2 = map.at(tp[m - 2]), ql2 = Qx[m - 2].x;
            float b = fminf(dl, f.a);
            if (!((T2 >= TL && TL >= ql) || (T2 <= TL && TL <= ql) || (ql2 <= ql && ql <= TL) ||
                  (ql2 >= ql && ql >= TL)))
                b = fminf(dl, fminf(f.a + fabsf(TL - T2), f.a + fabsf(ql - ql2)));
            a.s = fabsf(d0) + b;
        }
    }
    return a;
}

// the sums of the 8 lanes that share a candidate
__device__ __forceinline__ Acc group_sum(Acc a) {
    for (int o = 4; o; o >>= 1) {
        a.s += __shfl_xor_sync(0xffffffffu, a.s, o);
        a.c1 += __shfl_xor_sync(0xffffffffu, a.c1, o);
        a.c2 += __shfl_xor_sync(0xffffffffu, a.c2, o);
    }
    return a;
}
// candidates per resident group of 8 lanes up to which they share (57,000 on 148
// SMs; T->Q lists are rarely that short, and its kernel has no registers to spare:
// the same there made long lists 5% slower)
constexpr unsigned long long kGrouped = 4;

template <int METRIC>
__device__ __forceinline__ bool acc_dead(const Acc& a, const Fix& f) {
    return (METRIC == EDR || METRIC == LCSS) ? a.c1 > f.most : a.s > f.hi;
}
template <int METRIC>
__device__ __forceinline__ bool acc_alive(const Acc& a, const Fix& f) {
    return (METRIC == EDR || METRIC == LCSS) ? a.c2 <= f.most : a.s <= f.lo;
}

__device__ __forceinline__ float fix_units(double x, const Fix& f) {
    return (float)(12582912.0 + rint(x * f.scale - f.mid));
}

}  // namespace

// Five blocks an SM (48 registers, the exact path spills): a list of a few hundred
// thousand candidates is as much latency as issue.  32 DTW queries (m = 128, 2^22
// points) 2.75, 2.40, 2.27 ms at three, four and five, 2.23 at six, where MSM loses 2%.
template <int METRIC>
__global__ void __launch_bounds__(256, 5) k_glb_tq(Geom g, GlbJob job) {
    extern __shared__ __align__(16) float2 gtq_smem[];
    const QueryDev& q = job.q;
    const int m = q.m;
    constexpr int kb = METRIC == LCSS ? 0 : 1;
    float2* LU = gtq_smem + kb;       // [m] query envelope as F, points kb, kb + 1 16-byte aligned
    float2* Qx = gtq_smem + m + 1;    // [m] query points as F (x)
    const double bsf = job.cutoff_ptr ? *job.cutoff_ptr : q.cutoff;
    __shared__ Fix s_fix;  // one thread's divisions and roots serve the block
    if (threadIdx.x == 0) s_fix = make_fix<METRIC>(q, bsf, g.raw != 0, job.rel != nullptr);
    __syncthreads();
    const Fix f = s_fix;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        LU[i] = make_float2(fix_units(q.LQ[i], f), fix_units(q.UQ[i], f));
        Qx[i] = make_float2(fix_units(q.qn[i], f), 0.f);
    }
    __syncthreads();
    const int ke = METRIC == LCSS ? m : m - 1;
    const unsigned long long n_in = *job.n_in;
    const unsigned long long n_lim = n_in < (unsigned long long)job.in_cap ? n_in : job.in_cap;
    for (unsigned long long base = (unsigned long long)blockIdx.x * blockDim.x; base < n_lim;
         base += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned long long idx = base + threadIdx.x;
        const bool active = idx < n_lim;
        long long gi = 0, s = 0;
        double mu = 0.0, sg = 1.0;
        int j = 0;
        if (active) {
            gi = job.in[idx];
            g.locate(gi, &s, &j);
            mu = job.MU[s * g.kml + j];
            sg = job.SIG[s * g.kml + j];
        }
        const double* __restrict__ tp = job.target + gi;
        FixMap map;
        bool bad = !map.init(mu, sg, f) || f.exact;
        bool dead = !active;
        Acc a;
        int inner = 0;  // certain misses without the boundary (the T->Q sum)
        if (__any_sync(0xffffffffu, !dead && !bad)) {
            RelMap rm;
            if (job.rel && active) rm = RelMap(map.A, mu, job.rseg[s], f.mid);
            const bool fast = __all_sync(0xffffffffu, !active || (rm.ok && !bad));
            a = acc_boundary<METRIC>(map, tp, Qx, m, f);
            inner = a.c1;
            auto add = [&](int k, float F) {
                const float2 e = LU[k];
                acc_add<METRIC>(a, F, e.x, e.y, F - f.a, f);
            };
            if (fast) {
                const float* __restrict__ rp = job.rel + (s * g.m_k + j);
                for (int k = kb; k < ke; k += 8) {
                    if (k + 8 <= ke) {
                        float t[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) t[u] = rp[k + u];
#pragma unroll
                        for (int u = 0; u < 8; u += 2) {
                            const float4 e = *(const float4*)(LU + k + u);
                            const float F0 = rm.at(t[u]), F1 = rm.at(t[u + 1]);
                            acc_add<METRIC>(a, F0, e.x, e.y, F0 - f.a, f);
                            acc_add<METRIC>(a, F1, e.z, e.w, F1 - f.a, f);
                        }
                    } else {
                        for (int u = 0; k + u < ke; ++u) add(k + u, rm.at(rp[k + u]));
                    }
                    dead = dead || acc_dead<METRIC>(a, f);
                    if (!__any_sync(0xffffffffu, !dead)) break;
                }
            } else {
                for (int k = kb; k < ke; k += 8) {
                    if (k + 8 <= ke) {
                        double t[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) t[u] = tp[k + u];
#pragma unroll
                        for (int u = 0; u < 8; ++u) add(k + u, map.at(t[u]));
                    } else {
                        for (int u = 0; k + u < ke; ++u) add(k + u, map.at(tp[k + u]));
                    }
                    bad = bad || map.bad();
                    dead = dead || (!bad && acc_dead<METRIC>(a, f));
                    if (!__any_sync(0xffffffffu, !dead && !bad)) break;
                }
            }
            bad = bad || map.bad();  // no inner point: the boundary's own
            dead = dead || (!bad && acc_dead<METRIC>(a, f));
            inner = a.c1 - inner;
        }
        bool alive = !dead && !bad && acc_alive<METRIC>(a, f);
        double ob = dnan();  // certified: nothing to hand on but the T->Q count
        double ot = METRIC == LCSS ? (double)(m - inner) : (double)inner;
        // within the margin or out of range: the reference's operations
        const unsigned open = __ballot_sync(0xffffffffu, !dead && !alive);
        if (__popc(open) <= kWarpExact) {
            for (unsigned left = open; left; left &= left - 1) {
                const int L = __ffs(left) - 1;
                const long long gL = __shfl_sync(0xffffffffu, gi, L);
                const double muL = __shfl_sync(0xffffffffu, mu, L), sgL = __shfl_sync(0xffffffffu, sg, L);
                double b, t;
                const bool on = warp_tq<METRIC>(q.qn, q.LQ, q.UQ, m, q.arg, job.target + gL, muL, sgL, bsf, b, t);
                if ((threadIdx.x & 31) == L) {
                    alive = on;
                    ob = b;
                    ot = t;
                }
            }
            if ((open >> (threadIdx.x & 31) & 1u) && !alive && kGlbMax <= bsf) { alive = true; ob = -1.0; }
        } else if (!dead && !alive) {
            alive = exact_tq<METRIC>(q.qn, q.LQ, q.UQ, m, q.arg, tp, mu, sg, bsf, ob, ot);
            // abandoned: GLB returns MAX_VAL (src/glb.cpp:221 etc.); it survives only if
            // MAX_VAL <= cutoff (marker -1)
            if (!alive && kGlbMax <= bsf) { alive = true; ob = -1.0; }
        }
        warp_append(alive, job.n_out, [&](unsigned long long o) {
            if (o < (unsigned long long)job.out_cap) {
                job.out[o] = gi;
                job.out_b[o] = ob;
                job.out_t[o] = ot;
            }
        });
    }
}

// Forward windows of the raw target: lo/up[p] = min/max(t[p .. min(n-1, p+w)])
// with fmin/fmax (NaN ignored unless the whole window is NaN; only windows
// inside valid candidate windows, which hold no NaN, are ever read).
//
// Doubling in shared memory: after pass k, M[i] = min(t[i .. i + 2^k - 1]);
// a window of length L = w+1 is the union of the two length-2^K runs at its
// ends (2^K <= L < 2^(K+1)), min(M[p], M[p + L - 2^K]) -- the same set, so
// the same value as a direct scan.  log2(L) passes of one min per element
// replace the L reads per output of a direct scan, so the cost no longer
// grows with the radius.  A CTA produces kFwdTile outputs per tile from the
// tile plus its w-point halo, ping-ponging between two shared buffers.
//
__global__ void __launch_bounds__(kFwdThreads) k_fwd_env(const double* __restrict__ t, long long n, int w,
                                                        double* __restrict__ lo, double* __restrict__ up) {
    extern __shared__ double fw_smem[];
    const int ext = kFwdTile + w;  // tile plus halo
    double* An = fw_smem;
    double* Ax = An + ext;
    double* Bn = Ax + ext;
    double* Bx = Bn + ext;
    const int L = w + 1;
    int K = 0;
    while ((2 << K) <= L) ++K;  // 2^K <= L < 2^(K+1)
    const int off = L - (1 << K);
    for (long long p0 = (long long)blockIdx.x * kFwdTile; p0 < n; p0 += (long long)gridDim.x * kFwdTile) {
        const int cnt = (int)((n - p0) < ext ? (n - p0) : ext);
        for (int i = threadIdx.x; i < ext; i += kFwdThreads) {
            const double v = i < cnt ? t[p0 + i] : NAN;
            An[i] = v;
            Ax[i] = v;
        }
        __syncthreads();
        for (int k = 0; k < K; ++k) {
            const int s = 1 << k;
            for (int i = threadIdx.x; i < ext; i += kFwdThreads) {
                const bool in = i + s < ext;
                Bn[i] = in ? fmin(An[i], An[i + s]) : An[i];
                Bx[i] = in ? fmax(Ax[i], Ax[i + s]) : Ax[i];
            }
            __syncthreads();
            double* tn = An; An = Bn; Bn = tn;
            double* tx = Ax; Ax = Bx; Bx = tx;
        }
        for (int i = threadIdx.x; i < kFwdTile; i += kFwdThreads) {
            const long long p = p0 + i;
            if (p >= n) break;
            double mn, mx;
            if (p + w <= n - 1) {
                mn = fmin(An[i], An[i + off]);
                mx = fmax(Ax[i], Ax[i + off]);
            } else {  // the last w points: the window is clipped at the end of the target
                mn = t[p];
                mx = t[p];
                for (long long j = p + 1; j < n; ++j) {
                    mn = fmin(mn, t[j]);
                    mx = fmax(mx, t[j]);
                }
            }
            lo[p] = mn;
            up[p] = mx;
        }
        __syncthreads();
    }
}

size_t fwd_env_smem_bytes(int w) { return sizeof(double) * 4 * (size_t)(kFwdTile + w); }

// The points and the centred windows min/max(t[p-w .. p+w]) of every macro
// segment in FP32, relative to the middle of the segment's range, for GLB: half
// the bytes, and one FP32 multiply-add makes F of them.  A block per segment:
// its extremes (finite points), then the three rows (the windows where they lie
// inside the segment).  Bound by memory: 24 bytes read (two of the three reads
// twice, from L2) and 12 written per point.
__global__ void k_rel(const double* __restrict__ t, const double* __restrict__ lraw, const double* __restrict__ uraw,
                      Geom g, int w, float* __restrict__ rel, double2* __restrict__ seg) {
    __shared__ double s_mn[32], s_mx[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5, mk = g.m_k;
    const long long N = g.S * mk;
    for (long long s = blockIdx.x; s < g.S; s += gridDim.x) {
        const long long off = g.off(s);
        double mn = INFINITY, mx = -INFINITY;
        for (int p = tid; p < mk; p += blockDim.x) {
            const double v = t[off + p];
            if (isfinite(v)) {
                mn = fmin(mn, v);
                mx = fmax(mx, v);
            }
        }
        for (int o = 16; o; o >>= 1) {
            mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if (lane == 0) { s_mn[warp] = mn; s_mx[warp] = mx; }
        __syncthreads();
        for (int i = 0; i < nw; ++i) { mn = fmin(mn, s_mn[i]); mx = fmax(mx, s_mx[i]); }
        const double c = mn <= mx ? 0.5 * mn + 0.5 * mx : 0.0;
        if (tid == 0) seg[s] = make_double2(c, mn <= mx ? fmax(mx - c, c - mn) * (1.0 + 0x1p-40) : INFINITY);
        for (int p = tid; p < mk; p += blockDim.x) {
            const long long o = s * mk + p;
            rel[o] = (float)(t[off + p] - c);
            if (p >= w && p < mk - w) {
                rel[N + o] = (float)(fmin(lraw[off + p - w], lraw[off + p]) - c);
                rel[2 * N + o] = (float)(fmax(uraw[off + p - w], uraw[off + p]) - c);
            }
        }
        __syncthreads();
    }
}

template <int METRIC>
__global__ void __launch_bounds__(256, 3) k_glb_qt(Geom g, GlbJob job) {
    extern __shared__ __align__(16) float2 gqt_smem[];
    const QueryDev& q = job.q;
    const int m = q.m, w = q.w;
    float2* Qx = gqt_smem;  // [m] query points as F, and (ERP) their distance to the gap
    const double bsf = job.cutoff_ptr ? *job.cutoff_ptr : q.cutoff;
    __shared__ Fix s_fix;
    if (threadIdx.x == 0) s_fix = make_fix<METRIC>(q, bsf, g.raw != 0, job.rel != nullptr);
    __syncthreads();
    const Fix f = s_fix;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const float x = fix_units(q.qn[i], f);
        Qx[i] = make_float2(x, x - f.a);
    }
    __syncthreads();
    const double inv_scale = 1.0 / f.scale;
    const double rho = (m + 16.0) * 0x1p-23;
    constexpr int kb = METRIC == LCSS ? 0 : 1;
    const int ke = METRIC == LCSS ? m : m - 1;
    // interior points: the centred windows
    const int in0 = min(max(kb, w), ke), in1 = max(in0, min(ke, m - w));
    const unsigned long long n_in = *job.n_in;
    const unsigned long long n_lim = n_in < (unsigned long long)job.in_cap ? n_in : job.in_cap;
    // short lists: 8 lanes per candidate, each every eighth point
    const bool grouped = n_lim <= kGrouped * (unsigned long long)gridDim.x * blockDim.x / 8;
    const int share = grouped ? 3 : 0, sub = grouped ? threadIdx.x & 7 : 0;
    const unsigned per_block = blockDim.x >> share;
    for (unsigned long long base = (unsigned long long)blockIdx.x * per_block; base < n_lim;
         base += (unsigned long long)gridDim.x * per_block) {
        const unsigned long long c = base + (threadIdx.x >> share);
        bool active = c < n_lim;
        long long gi = 0, s = 0;
        double mu = 0.0, sg = 1.0, boundary = 0.0, tq = 0.0;
        int j = 0;
        if (active) {
            gi = job.in[c];
            boundary = job.in_b[c];
            tq = job.in_t[c];
            g.locate(gi, &s, &j);
            mu = job.MU[s * g.kml + j];
            sg = job.SIG[s * g.kml + j];
        }
        const double* __restrict__ lf = job.lraw + gi;
        const double* __restrict__ uf = job.uraw + gi;
        FixMap map;
        bool keep = false;
        const bool certified = map.init(mu, sg, f) && isnan(boundary);  // its points are in range
        bool dead = !active || !certified;  // not certified: decided below
        Acc a;
        int edge = 0;
        if (__any_sync(0xffffffffu, !dead)) {
            RelMap rm;
            if (job.rel && active) rm = RelMap(map.A, mu, job.rseg[s], f.mid);
            const bool fast = __all_sync(0xffffffffu, dead || rm.ok);
            const int i0 = fast ? in0 : ke, i1 = fast ? in1 : ke;
            if (sub == 0) a = acc_boundary<METRIC>(map, job.target + gi, Qx, m, f);
            edge = a.c1;
            auto term = [&](int k, float lo, float up) {
                const float2 x = Qx[k];
                acc_add<METRIC>(a, x.x, lo, up, x.y, f);
            };
            auto ends = [&](int k) {
                const int p0 = qt_p0(k, w), p1 = qt_p1(k, m, w);
                term(k, fminf(map.at_checked(lf[p0]), map.at_checked(lf[p1])),
                     fmaxf(map.at_checked(uf[p0]), map.at_checked(uf[p1])));
            };
            auto done = [&] {
                dead = dead || acc_dead<METRIC>(a, f);
                return !__any_sync(0xffffffffu, !dead);
            };
            const float* __restrict__ cl = job.rel + (g.S * g.m_k + s * g.m_k + j);
            const float* __restrict__ cu = cl + g.S * g.m_k;
            bool stop = false;
            if (grouped) {
                auto some = [&](int b, int e) {  // points of [b, e), which holds no interior point or only those
                    const bool inner = b == i0 && e == i1;
                    for (int k = b + sub; k - sub < e && !stop; k += inner ? 64 : 16) {
                        if (inner) {
                            float lo[8], up[8];
#pragma unroll
                            for (int u = 0; u < 8; ++u) {
                                const int kk = min(k + 8 * u, e - 1);
                                lo[u] = cl[kk];
                                up[u] = cu[kk];
                            }
#pragma unroll
                            for (int u = 0; u < 8; ++u)
                                if (k + 8 * u < e) term(k + 8 * u, rm.at(lo[u]), rm.at(up[u]));
                        } else {
#pragma unroll
                            for (int u = 0; u < 2; ++u)
                                if (k + 8 * u < e) ends(k + 8 * u);
                        }
                        Acc t = group_sum(a);
                        dead = dead || acc_dead<METRIC>(t, f);
                        stop = !__any_sync(0xffffffffu, !dead);
                    }
                };
                some(kb, i0);
                some(i0, i1);
                some(i1, ke);
                a = group_sum(a);
                edge = __shfl_sync(0xffffffffu, edge, threadIdx.x & 24);
            } else {
                for (int k = kb; k < i0 && !stop; k += 4) {
                    if (k + 4 <= i0) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) ends(k + u);
                    } else {
                        for (int u = 0; k + u < i0; ++u) ends(k + u);
                    }
                    stop = done();
                }
                for (int k = i0; k < i1 && !stop; k += 8) {
                    if (k + 8 <= i1) {
                        float lo[8], up[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) { lo[u] = cl[k + u]; up[u] = cu[k + u]; }
#pragma unroll
                        for (int u = 0; u < 8; ++u) term(k + u, rm.at(lo[u]), rm.at(up[u]));
                    } else {
                        for (int u = 0; k + u < i1; ++u) term(k + u, rm.at(cl[k + u]), rm.at(cu[k + u]));
                    }
                    stop = done();
                }
                for (int k = i1; k < ke && !stop; k += 4) {
                    if (k + 4 <= ke) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) ends(k + u);
                    } else {
                        for (int u = 0; k + u < ke; ++u) ends(k + u);
                    }
                    stop = done();
                }
            }
            dead = dead || acc_dead<METRIC>(a, f);
        }
        active = active && sub == 0;  // the first lane decides
        // what the abandon tests of the exact distances take: a lower bound of
        // the Q->T sum (LCSS: an upper bound of the count), the T->Q count
        double os, ot = tq;
        if (METRIC == LCSS) os = (double)(m - (a.c1 - edge));
        else if (METRIC == EDR) os = (double)(a.c1 - edge);
        else {
            // the boundary is part of a.s: taken off at its upper end
            Acc b;
            if (!dead) b = acc_boundary<METRIC>(map, job.target + gi, Qx, m, f);
            const double v = fmax(0.0, ((double)a.s - (double)b.s * (1.0 + rho)) - (double)a.s * rho);
            if (METRIC == MSM) os = fmax(0.0, v - f.eta) * inv_scale;
            else {
                const double r = fmax(0.0, sqrt(v) - f.eta) * inv_scale;
                os = r * r * (1.0 - 0x1p-40);
            }
        }
        keep = active && certified && !dead && acc_alive<METRIC>(a, f);
        const bool want = active && !keep && !(certified && dead);
        const unsigned open = __ballot_sync(0xffffffffu, want);
        if (open) {
            double qt = 0.0;
            bool on = true;
            if (__popc(open) <= kWarpExact) {
                for (unsigned left = open; left; left &= left - 1) {
                    const int L = __ffs(left) - 1;
                    const long long gL = __shfl_sync(0xffffffffu, gi, L);
                    const double muL = __shfl_sync(0xffffffffu, mu, L), sgL = __shfl_sync(0xffffffffu, sg, L);
                    double bL = __shfl_sync(0xffffffffu, boundary, L), tL = __shfl_sync(0xffffffffu, tq, L);
                    bool onL = true;
                    if (__shfl_sync(0xffffffffu, (int)certified, L))
                        onL = warp_tq<METRIC>(q.qn, q.LQ, q.UQ, m, q.arg, job.target + gL, muL, sgL, bsf, bL, tL);
                    double v = 0.0;
                    if (bL != -1.0 && onL)
                        v = warp_qt<METRIC>(q.qn, m, w, q.arg, job.lraw + gL, job.uraw + gL, muL, sgL);
                    if ((threadIdx.x & 31) == L) {
                        boundary = bL;
                        tq = tL;
                        on = onL;
                        qt = v;
                    }
                }
            } else if (want) {
                if (certified)
                    on = exact_tq<METRIC>(q.qn, q.LQ, q.UQ, m, q.arg, job.target + gi, mu, sg, bsf, boundary, tq);
                if (boundary != -1.0 && on) qt = exact_qt<METRIC>(q.qn, m, w, q.arg, lf, uf, mu, sg);
            }
            if (want) {
                double glb;
                if (boundary == -1.0 || !on) {
                    glb = kGlbMax;  // abandoned in T->Q but MAX_VAL <= cutoff
                } else if (METRIC == LCSS) {
                    glb = dmax0(dsub(1.0, ddiv(dminv(tq, qt), (double)m)));
                } else {
                    const double tot = dadd(boundary, qt);
                    if (METRIC == DTW || METRIC == ERP)
                        glb = (m > 2 && tot > dmul(bsf, bsf)) ? kGlbMax : dsqrt(dmax0(dadd(boundary, dmaxv(tq, qt))));
                    else
                        glb = (m > 2 && tot > bsf) ? kGlbMax : dadd(boundary, dmaxv(tq, qt));
                }
                keep = glb <= bsf;
                os = boundary == -1.0 ? -1.0 : qt;
                ot = boundary == -1.0 ? -1.0 : tq;
            }
        }
        warp_append(keep, job.n_out, [&](unsigned long long o) {
            if (o < (unsigned long long)job.out_cap) {
                job.out[o] = gi;
                if (job.out_t) job.out_t[o] = os;
                if (job.out_b) job.out_b[o] = ot;
            }
            if (job.segc && s < g.forsize) atomicAdd((unsigned long long*)&job.segc[3 * s + 2], 1ull);
        });
    }
}

#define FSM_GLB_INST(M)                                       \
    template __global__ void k_glb_tq<M>(Geom, GlbJob);       \
    template __global__ void k_glb_qt<M>(Geom, GlbJob);
FSM_GLB_INST(DTW)
FSM_GLB_INST(ERP)
FSM_GLB_INST(EDR)
FSM_GLB_INST(LCSS)
FSM_GLB_INST(MSM)

}  // namespace fsm
