// LB_IP for every window of a macro segment, fused with the prune test and
// survivor compaction.
//
// Reference: penalties q_to_h_{l,u} (src/q_to_h.cpp:11-134), masks
// s_to_g_{l,u} (src/lb.cpp:18-34), sliding inner products through real FFTs
// of length m_k (src/sip.cpp:16-52 as sequenced at src/fsmeld.cpp:792-806),
// trans (src/fsmeld.cpp:84-106 and the tail variant 912-921), and the prune
// test fsmeld_lbip_exceeds_cutoff (include/fsmeld_internal.h:9-19).
//
// z_l[m-1+j] + z_u[m-1+j] = sum_k h_l[k] g_l[j+k] + h_u[k] g_u[j+k] for the
// kml windows j.  Three ways:
//  * k_lbip_runs, DTW, ERP, MSM with 100 (w+1) >= m: the masks g come from
//    envelopes of radius w and change value rarely, so with H[k] = h[0] + .. +
//    h[k-1] an inner product is a signed sum of H over the changes inside the
//    window (summation by parts): a few adds per window instead of a
//    transform.  A run in which the radius-w maximum exceeds a level is at least
//    2w+1 long, so a window has about m / (w+1) changes a side at most; at the
//    limit of the rule, 200 for both, that costs what the transform does.
//    Measured on 2^24 points (m = 256, w = 13): DTW 1.16 -> 0.65 ms; 20 mixed queries on
//    2^22 points (m to 1024) 7.5 -> 2.7 ms with the popcounts below (0.75 -> 0.28 ms
//    for LCSS on the 2^24 points).  H is in fixed point, 64 bits over the most that
//    it can be: differences of it are exact, so the many changes of a noisy window
//    cost nothing, and a product is off by the rounding of its h alone, at most
//    m/2 units of 2^-60 m h_max, and the last conversion.  Against the products in
//    extended precision (walks, noise, bursts, spikes, raw series; m = 16 to 1024, 300
//    combinations) its largest error is 3.2e-16 of H[m] and below the transform's
//    (8.6e-16) in each; FP64 sums of H, at the same time, were up to 30 times
//    the transform's (4.9e-15).
//  * k_lbip_runs, EDR and LCSS: h and g are 0/1, so the products are popcounts
//    of bit masks: exact integers.
//  * k_lbip, narrower bands: one complex FFT packs (g_l + i g_u), one packs the
//    reversed penalties, the two real spectra of each are separated, the
//    products are summed, and one inverse FFT gives z_l + z_u directly
//    (3 complex FFTs of length P >= m_k instead of the reference's 6 real
//    FFTs).  FP64 Stockham autosort FFT in shared memory, radix 16/8/4/2
//    passes with a padded layout (one pad every 16 points) so strided
//    stores are bank-conflict free.  Rounding differs from FFTW's at the
//    1e-13 level; the prune test's 1e-9 guard makes the decision the same.
#include <cub/block/block_reduce.cuh>
#include <cub/block/block_scan.cuh>

#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

__constant__ double2 c_w16[16];  // exp(-2*pi*i*k/16)

namespace {

__device__ __forceinline__ int padi(int i) { return i + (i >> 4); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

__host__ __device__ constexpr int bitrev(int x, int bits) {
    int r = 0;
    for (int i = 0; i < bits; ++i) r |= ((x >> i) & 1) << (bits - 1 - i);
    return r;
}
template <int R> struct Log2;
template <> struct Log2<2> { static constexpr int v = 1; };
template <> struct Log2<4> { static constexpr int v = 2; };
template <> struct Log2<8> { static constexpr int v = 3; };
template <> struct Log2<16> { static constexpr int v = 4; };

// in-register DFT of size R (radix-2 decimation in time, natural order out)
template <int R>
__device__ __forceinline__ void dft_reg(double2 (&v)[R], bool inv) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int j = bitrev(i, Log2<R>::v);
        if (i < j) { const double2 tmp = v[i]; v[i] = v[j]; v[j] = tmp; }
    }
#pragma unroll
    for (int len = 2; len <= R; len <<= 1) {
#pragma unroll
        for (int s = 0; s < R; s += len) {
#pragma unroll
            for (int k = 0; k < len / 2; ++k) {
                double2 w = c_w16[k * (16 / len)];
                if (inv) w.y = -w.y;
                const double2 a = v[s + k];
                const double2 b = cmul(v[s + k + len / 2], w);
                v[s + k] = cadd(a, b);
                v[s + k + len / 2] = csub(a, b);
            }
        }
    }
}

// one Stockham radix-R pass: a -> b (both padded layout)
template <int R, int T>
__device__ __forceinline__ void fft_pass(const double2* __restrict__ a, double2* __restrict__ b, int P,
                                         int Ns, const double2* __restrict__ W, bool inv) {
    const int nb = P / R;
    for (int j = threadIdx.x; j < nb; j += T) {
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = a[padi(j + r * nb)];
        const int jm = j & (Ns - 1);
        if (Ns > 1) {
            const int stride = P / (Ns * R);
#pragma unroll
            for (int r = 1; r < R; ++r) {
                double2 w = __ldg(&W[jm * r * stride]);
                if (inv) w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        dft_reg<R>(v, inv);
        const int idxD = (j - jm) * R + jm;
#pragma unroll
        for (int r = 0; r < R; ++r) b[padi(idxD + r * Ns)] = v[r];
    }
}

// Full FFT of length P = 2^logP; returns the buffer holding the result.
template <int T>
__device__ double2* fft_run(double2* a, double2* b, int P, int logP, const double2* W, bool inv) {
    const int passes = (logP + 3) / 4;
    int rem = logP, Ns = 1;
    for (int ps = 0; ps < passes; ++ps) {
        const int left = passes - ps;
        const int bits = (rem + left - 1) / left;  // spread bits evenly, larger radices first
        switch (bits) {
            case 4: fft_pass<16, T>(a, b, P, Ns, W, inv); break;
            case 3: fft_pass<8, T>(a, b, P, Ns, W, inv); break;
            case 2: fft_pass<4, T>(a, b, P, Ns, W, inv); break;
            default: fft_pass<2, T>(a, b, P, Ns, W, inv); break;
        }
        __syncthreads();
        double2* tmp = a; a = b; b = tmp;
        Ns <<= bits;
        rem -= bits;
    }
    return a;
}

// src/q_to_h.cpp:11-64 (lower) / 84-134 (upper)
__device__ __forceinline__ double q_to_h(int metric, bool upper, double x, double t, double C) {
    if (!upper) {
        switch (metric) {
            case MSM: return (x < t) ? ((dsub(t, x) < C) ? dsub(t, x) : C) : 0.0;
            case DTW: return (x < t) ? dsq(t, x) : 0.0;
            case ERP: return (x < t) ? ((dsq(x, t) > dsq(x, C)) ? dsq(x, C) : dsq(x, t)) : 0.0;
            default: return (x < dsub(t, C)) ? 1.0 : 0.0;
        }
    }
    switch (metric) {
        case MSM: return (x > t) ? ((dsub(x, t) < C) ? dsub(x, t) : C) : 0.0;
        case DTW: return (x > t) ? dsq(x, t) : 0.0;
        case ERP: return (x > t) ? ((dsq(x, t) > dsq(x, C)) ? dsq(x, C) : dsq(x, t)) : 0.0;
        default: return (x > dadd(t, C)) ? 1.0 : 0.0;
    }
}

__device__ __forceinline__ unsigned long long bits64(const unsigned long long* w, int b) {
    const int q = b >> 6, r = b & 63;
    return r ? ((w[q] >> r) | (w[q + 1] << (64 - r))) : w[q];
}

}  // namespace

template <int T, bool GW>
__global__ void __launch_bounds__(T) k_lbip(Geom g, LbJob job, const double2* __restrict__ W, int P,
                                            int logP) {
    using IScan = cub::BlockScan<int, T>;
    using IReduce = cub::BlockReduce<int, T>;
    extern __shared__ __align__(16) unsigned char lb_smem[];
    __shared__ typename IScan::TempStorage scan_tmp;
    __shared__ typename IReduce::TempStorage red_tmp;
    __shared__ unsigned long long s_base;
    __shared__ double s_tl, s_tu;

    const QueryDev& q = job.q;
    const int m = q.m, mk = g.m_k, kml = g.kml, metric = q.metric;
    const int tid = threadIdx.x;
    const int Pp = P + (P >> 4) + 1;
    unsigned char* lbase = GW ? job.gwork + (long long)blockIdx.x * job.slot_stride : lb_smem;
    double2* bufA = (double2*)lbase;
    double2* bufB = bufA + Pp;
    double2* bufC = bufB + Pp;
    for (long long s = blockIdx.x; s < g.S; s += gridDim.x) {
        if (tid == 0) { s_tl = job.thr[2 * s]; s_tu = job.thr[2 * s + 1]; }
        __syncthreads();
        const double tl = s_tl, tu = s_tu;
        const double* Ln = job.Ln + s * mk;
        const double* Un = job.Un + s * mk;
        const double* zsrc;
        // X = g_l + i g_u, Y = reversed h_l + i reversed h_u (src/sip.cpp:16-29)
        for (int i = tid; i < P; i += T) {
            double2 x = make_double2(0.0, 0.0), y = make_double2(0.0, 0.0);
            if (i < mk) x = make_double2(Ln[i] >= tl ? 1.0 : 0.0, Un[i] <= tu ? 1.0 : 0.0);
            if (i < m) {
                const double qv = q.qn[m - 1 - i];
                y = make_double2(q_to_h(metric, false, qv, tl, q.arg), q_to_h(metric, true, qv, tu, q.arg));
            }
            bufA[padi(i)] = x;
            bufC[padi(i)] = y;
        }
        __syncthreads();
        double2* X = fft_run<T>(bufA, bufB, P, logP, W, false);
        double2* freeb = (X == bufA) ? bufB : bufA;
        double2* Y = fft_run<T>(bufC, freeb, P, logP, W, false);
        double2* Zb = (Y == bufC) ? freeb : bufC;  // the buffer holding neither X nor Y
        const double half = 0.5;
        for (int k = tid; k < P; k += T) {
            const int kn = (P - k) & (P - 1);
            const double2 xk = X[padi(k)], xn = X[padi(kn)];
            const double2 yk = Y[padi(k)], yn = Y[padi(kn)];
            // split two real spectra packed in one complex FFT
            const double2 gl = make_double2(half * (xk.x + xn.x), half * (xk.y - xn.y));
            const double2 gu = make_double2(half * (xk.y + xn.y), -half * (xk.x - xn.x));
            const double2 hl = make_double2(half * (yk.x + yn.x), half * (yk.y - yn.y));
            const double2 hu = make_double2(half * (yk.y + yn.y), -half * (yk.x - yn.x));
            Zb[padi(k)] = cadd(cmul(gl, hl), cmul(gu, hu));
        }
        __syncthreads();
        double2* Z = fft_run<T>(Zb, X, P, logP, W, true);
        const double invP = 1.0 / (double)P;
        // z_l + z_u for window j sits at m-1+j; stash it in the free buffer as doubles
        double* zs = (double*)((Z == Zb) ? X : Zb);
        for (int j = tid; j < kml; j += T) zs[j] = Z[padi(m - 1 + j)].x * invP;
        __syncthreads();
        zsrc = zs;

        // trans + validity + prune, in window order
        const int lo = g.lo(s);
        const int nwin = kml - lo;
        const int c = (nwin + T - 1) / T;
        const int wlo = lo + tid * c, whi = min(kml, wlo + c);
        int nvalid = 0, nsurv = 0;
        for (int j = wlo; j < whi; ++j) {
            const long long gi = g.gidx(s, j);
            const double sg = job.SIG[s * kml + j];
            if (window_invalid(sg, g, gi)) {
                if (job.zout) job.zout[s * kml + j] = dnan();
                continue;
            }
            ++nvalid;
            const double zz = zsrc[j];
            double z;
            if (metric == DTW || metric == ERP) z = dsqrt(dmax0(zz));
            else z = zz;
            if (job.zout) job.zout[s * kml + j] = z;
            if (job.surv && !lbip_exceeds(z, q.cutoff, metric)) ++nsurv;
        }
        if (!job.surv) {
            const int tv = IReduce(red_tmp).Sum(nvalid);
            if (tid == 0 && tv) atomicAdd(job.nvalid, (unsigned long long)tv);
        } else {
            int off, total;
            IScan(scan_tmp).ExclusiveSum(nsurv, off, total);
            if (tid == 0) s_base = total ? atomicAdd(job.nsurv, (unsigned long long)total) : 0ull;
            __syncthreads();
            unsigned long long o = s_base + off;
            if (nsurv) {
                for (int j = wlo; j < whi; ++j) {
                    const long long gi = g.gidx(s, j);
                    const double sg = job.SIG[s * kml + j];
                    if (window_invalid(sg, g, gi)) continue;
                    const double zz = zsrc[j];
                    double z;
                    if (metric == DTW || metric == ERP) z = dsqrt(dmax0(zz));
                    else z = zz;
                    if (!lbip_exceeds(z, q.cutoff, metric)) {
                        if (o < (unsigned long long)job.surv_cap) job.surv[o] = gi;
                        ++o;
                    }
                }
            }
            const int tv = IReduce(red_tmp).Sum(nvalid);
            if (tid == 0 && tv) atomicAdd(job.nvalid, (unsigned long long)tv);
            if (tid == 0 && job.segc) {
                job.segc[3 * s] = tv;
                job.segc[3 * s + 1] = total;
                job.segc[3 * s + 2] = 0;
            }
        }
        __syncthreads();
    }
}

// One block per segment.  POPC: EDR, LCSS.
template <int T, bool POPC>
__global__ void __launch_bounds__(T) k_lbip_runs(Geom g, LbJob job, double keep_max) {
    using LScan = cub::BlockScan<long long, T>;
    using IScan = cub::BlockScan<int, T>;
    extern __shared__ __align__(16) unsigned char lr_smem[];
    __shared__ typename LScan::TempStorage lscan_tmp;
    __shared__ typename IScan::TempStorage iscan_tmp;
    __shared__ unsigned long long s_base;
    __shared__ int s_cnt[2], s_off[T / 32 + 1];
    constexpr unsigned kAll = 0xffffffffu;
    const QueryDev& q = job.q;
    const int m = q.m, mk = g.m_k, kml = g.kml, metric = q.metric;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gw = (mk + 63) / 64 + 2, hw = (m + 63) / 64;
    // mask words of the two sides, survivor bits of the windows, then either
    // the penalty words (POPC) or H of the two sides, the changes and, per mask
    // word, the number of changes before it
    unsigned long long* G[2] = {(unsigned long long*)lr_smem, (unsigned long long*)lr_smem + gw};
    unsigned* keepw = (unsigned*)(G[1] + gw);
    unsigned char* rest = (unsigned char*)keepw + (((size_t)(kml + 31) / 32 * 4 + 15) & ~size_t(15));
    unsigned long long* Hb[2] = {(unsigned long long*)rest, (unsigned long long*)rest + hw};
    long long* H[2] = {(long long*)rest, (long long*)rest + (m + 1)};
    int* pre[2] = {(int*)(H[1] + m + 1), (int*)(H[1] + m + 1) + gw};
    unsigned short* edge[2] = {(unsigned short*)(pre[1] + gw), (unsigned short*)(pre[1] + gw) + mk};

    for (long long s = blockIdx.x; s < g.S; s += gridDim.x) {
        const double tl = job.thr[2 * s], tu = job.thr[2 * s + 1];
        const double* __restrict__ Ln = job.Ln + s * mk;
        const double* __restrict__ Un = job.Un + s * mk;
        for (int base = warp * 32; base < gw * 64; base += T) {
            const int i = base + lane;
            const unsigned bl = __ballot_sync(kAll, i < mk && Ln[min(i, mk - 1)] >= tl);
            const unsigned bu = __ballot_sync(kAll, i < mk && Un[min(i, mk - 1)] <= tu);
            if (lane == 0) {
                ((unsigned*)G[0])[base >> 5] = bl;
                ((unsigned*)G[1])[base >> 5] = bu;
            }
        }
        bool plain = true;  // every penalty finite
        double unit[2] = {1.0, 1.0};  // of H
        if (POPC) {
            for (int base = warp * 32; base < hw * 64; base += T) {
                const int k = base + lane;
                const double qv = (k < m) ? q.qn[k] : 0.0;
                const unsigned bl = __ballot_sync(kAll, k < m && q_to_h(metric, false, qv, tl, q.arg) != 0.0);
                const unsigned bu = __ballot_sync(kAll, k < m && q_to_h(metric, true, qv, tu, q.arg) != 0.0);
                if (lane == 0) {
                    ((unsigned*)Hb[0])[base >> 5] = bl;
                    ((unsigned*)Hb[1])[base >> 5] = bu;
                }
            }
            __syncthreads();
        } else {
            // H: each thread's own stretch, then a block scan
            const int per = (m + T - 1) / T, k0 = min(m, tid * per), k1 = min(m, k0 + per);
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const double far = side ? q.qhi - tu : tl - q.qlo;  // of the query's points from the threshold
                double hmax = !(far > 0.0) ? 0.0 : metric == MSM ? fmin(far, q.arg) : far * far;
                if (metric == ERP) hmax = fmin(hmax, fmax(dsq(q.qlo, q.arg), dsq(q.qhi, q.arg)));
                plain = plain && isfinite(hmax);
                // m hmax scale < 2^62
                const int e = hmax > 0.0 && isfinite(hmax) ? min(1000, 60 - ilogb(hmax) - ilogb((double)m)) : 0;
                const double scale = scalbn(1.0, e);
                unit[side] = scalbn(1.0, -e);
                auto fixed = [&](int k) {
                    return __double2ll_rn(q_to_h(metric, side == 1, q.qn[k], side ? tu : tl, q.arg) * scale);
                };
                long long sum = 0, off;
                for (int k = k0; k < k1; ++k) sum += fixed(k);
                LScan(lscan_tmp).ExclusiveSum(sum, off);
                for (int k = k0; k < k1; ++k) {
                    H[side][k] = off;
                    off += fixed(k);
                }
                if (k1 == m && k0 < m) H[side][m] = off;
                __syncthreads();
            }
            // changes: positions p with g[p] != g[p-1]; even ones start a run
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                int before = 0;  // gw <= 258 words: one or two rounds
                for (int w0 = 0; w0 < gw; w0 += T) {
                    const int wi = w0 + tid;
                    unsigned long long x = 0;
                    if (wi < gw) x = G[side][wi] ^ ((G[side][wi] << 1) | (wi ? G[side][wi - 1] >> 63 : 0ull));
                    int off, tot;
                    IScan(iscan_tmp).ExclusiveSum(__popcll(x), off, tot);
                    __syncthreads();
                    if (wi < gw) {
                        off += before;
                        pre[side][wi] = off;
                        while (x) {
                            const int b = __ffsll((long long)x) - 1;
                            x &= x - 1;
                            if (wi * 64 + b < mk) edge[side][off++] = (unsigned short)(wi * 64 + b);
                        }
                    }
                    before += tot;
                }
            }
            __syncthreads();
        }

        // windows in order: warp by warp stretches of whole 32-window words
        const int lo = g.lo(s), words = (kml + 31) / 32, wper = (words + T / 32 - 1) / (T / 32);
        const int wd0 = min(words, warp * wper), wd1 = min(words, wd0 + wper);
        int nvalid = 0, nsurv = 0;
        for (int wd = wd0; wd < wd1; ++wd) {
            const int j = wd * 32 + lane;
            const bool in = j < kml && j >= lo;
            const long long gi = in ? g.gidx(s, j) : 0;
            const bool ok = in && !window_invalid(job.SIG[s * kml + j], g, gi);
            bool keep = false;
            double zz = 0.0;
            if (ok) {
                if (POPC) {
                    int cnt = 0;
                    for (int i = 0; i < hw; ++i) {
                        cnt += __popcll(Hb[0][i] & bits64(G[0], j + 64 * i));
                        cnt += __popcll(Hb[1][i] & bits64(G[1], j + 64 * i));
                    }
                    zz = (double)cnt;
                } else if (plain) {
#pragma unroll
                    for (int side = 0; side < 2; ++side) {
                        // changes at most x, x = j and j+m-1: those of the words before and of the word itself
                        const unsigned long long* Gs = G[side];
                        auto upto = [&](int x) {
                            const int wi = x >> 6;
                            const unsigned long long c =
                                Gs[wi] ^ ((Gs[wi] << 1) | (wi ? Gs[wi - 1] >> 63 : 0ull));
                            return pre[side][wi] + __popcll(c & (~0ull >> (63 - (x & 63))));
                        };
                        int e = upto(j);
                        const int e1 = upto(j + m - 1);
                        const unsigned short* __restrict__ E = edge[side];
                        const long long* __restrict__ Hs = H[side] - j;
                        // an odd change ends a run (+H), an even one starts it (-H); H[0] = 0
                        long long z0 = 0, z1 = 0;
                        if ((e & 1) && e < e1) { z0 = Hs[E[e]]; ++e; }
                        for (; e + 1 < e1; e += 2) {
                            z1 += Hs[E[e]];
                            z0 += Hs[E[e + 1]];
                        }
                        if (e < e1) z1 += Hs[E[e]];
                        if (e1 & 1) z0 += Hs[j + m];
                        zz += (double)(z0 - z1) * unit[side];
                    }
                } else {
                    zz = dnan();  // as the transform of infinite penalties
                }
                ++nvalid;
                keep = !(zz > keep_max && zz <= 1.7976931348623157e308);
            }
            if (job.zout && in) {
                double z;
                if (metric == DTW || metric == ERP) z = dsqrt(dmax0(zz));
                else if (metric == LCSS) z = dmax0(ddiv(zz, (double)m));
                else z = zz;
                job.zout[s * kml + j] = ok ? z : dnan();
            }
            const unsigned mask = __ballot_sync(kAll, keep);
            if (lane == 0) keepw[wd] = mask;
            nsurv += __popc(mask);  // the same in every lane
        }
        for (int o = 16; o; o >>= 1) nvalid += __shfl_xor_sync(kAll, nvalid, o);
        if (lane == 0) s_off[warp] = nsurv;
        if (tid == 0) s_cnt[0] = 0;
        __syncthreads();
        if (lane == 0 && nvalid) atomicAdd(&s_cnt[0], nvalid);
        int off = 0, total = 0;
        for (int i = 0; i < T / 32; ++i) {
            if (i < warp) off += s_off[i];
            total += s_off[i];
        }
        __syncthreads();
        if (tid == 0) {
            if (s_cnt[0]) atomicAdd(job.nvalid, (unsigned long long)s_cnt[0]);
            if (job.surv) s_base = total ? atomicAdd(job.nsurv, (unsigned long long)total) : 0ull;
            if (job.surv && job.segc) {
                job.segc[3 * s] = s_cnt[0];
                job.segc[3 * s + 1] = total;
                job.segc[3 * s + 2] = 0;
            }
        }
        __syncthreads();
        if (job.surv) {
            unsigned long long o = s_base + off;
            for (int wd = wd0; wd < wd1; ++wd) {
                const unsigned mask = keepw[wd];
                if (mask >> lane & 1u) {
                    const unsigned long long at = o + __popc(mask & ((1u << lane) - 1));
                    if (at < (unsigned long long)job.surv_cap) job.surv[at] = g.gidx(s, wd * 32 + lane);
                }
                o += __popc(mask);
            }
        }
        __syncthreads();
    }
}

size_t lbip_smem_bytes(int P) {
    const size_t Pp = (size_t)P + (P >> 4) + 1;
    return 3 * Pp * sizeof(double2) + 64;
}

size_t lbip_runs_smem_bytes(int m_k, int kml, int m, bool popc) {
    const size_t gw = (m_k + 63) / 64 + 2, hw = (m + 63) / 64;
    const size_t keep = (((size_t)(kml + 31) / 32 * 4) + 15) & ~size_t(15);
    return 2 * gw * 8 + keep + (popc ? 2 * hw * 8 : 2 * ((size_t)m + 1) * 8 + 2 * gw * 4 + 2 * (size_t)m_k * 2) + 64;
}

int lbip_set_w16() {
    double2 w[16];
    for (int k = 0; k < 16; ++k) {
        const double ang = 6.283185307179586476925286766559 * k / 16.0;
        w[k] = make_double2(cos(ang), -sin(ang));
    }
    FSM_CUDA_TRY(cudaMemcpyToSymbol(c_w16, w, sizeof(w)));
    return 0;
}

template __global__ void k_lbip<256, false>(Geom, LbJob, const double2*, int, int);
template __global__ void k_lbip<256, true>(Geom, LbJob, const double2*, int, int);
template __global__ void k_lbip_runs<256, false>(Geom, LbJob, double);
template __global__ void k_lbip_runs<256, true>(Geom, LbJob, double);

}  // namespace fsm
