// LB_IP for a group of queries of equal (m, w) as one tensor-core
// contraction (tcgen05.mma, BF16 operands, FP32 accumulation in TMEM).
//
// LB_IP's sliding inner products (src/sip.cpp:16-52; z[m-1+j] = sum_k
// h[k] g[j+k], src/fsmeld.cpp:792-806) have a product form: the window masks
// g depend on the target envelopes and a threshold t, the penalties h on the
// query and t (src/lb.cpp:18-34, src/q_to_h.cpp:11-134).  When every query
// of a group uses the same thresholds (t_l, t_u), the masks are shared and
// the inner products of all windows with all queries are one matrix product
//
//     Z[j][q] = sum_k A[j][k] B[q][k],   A[j][k] = g[j+k] (Hankel, 0/1),
//                                        B[q][k] = h_q[k],
//
// per side (lower, upper).  A is exact in BF16 (0 or 1).  Each h_q is split
// on the host into three BF16 terms h0 + h1 + h2 (h0 = bf16(h), h1 =
// bf16(h - h0), h2 = bf16(h - h0 - h1)); the three products accumulate into
// one FP32 accumulator, so Z carries the FP32 accumulation error and the
// split's residual.  The host bounds both per query and side (margin =
// residual + 4 n 2^-23 sum_k(|h0|+|h1|+|h2|), n = the accumulated terms)
// and the epilogue lowers each Z by its margin before the bound is formed,
// so the bound stays a true lower bound of the exact FP64 inner product and
// the pruning is admissible (the exact DP decides every match).  Any
// threshold gives a valid bound (the reference picks one per segment and
// query to make it tight; here one pair serves the whole group).
//
// Tiles: a CTA of 256 threads takes kTiles 128-window tiles of one segment at a
// time.  The group's window masks g (one bit per segment position and side)
// are computed once before the product (k_gemm_masks, one ballot per 32
// positions).  Row r of A is g[j0 + r ...], so the eight elements of row r and
// K group kg depend on r + 8 kg alone: in the canonical no-swizzle K-major
// layout (8-row x 16-byte core matrices) with 128 bytes from row group to row
// group and also from K group to K group, all tiles' rows and K groups lie in
// one array, 16 bytes per position (the operand that is read repeats, the one
// that is stored does not).  B is arranged on the host in the operand layout
// and stays in shared memory where it and A leave room for two CTAs per SM
// (NQ m up to about 7000); otherwise a chunk of 64 K elements at a time is staged.  One
// thread issues kTiles x 4 K-steps x 2 sides x 3 splits of
// tcgen05.mma.cta_group::1.kind::f16 (M = 128, N = NQ, K = 16) per chunk into
// the TMEM accumulators (per tile columns [0, NQ) lower, [NQ, 2 NQ) upper) and
// commits them to an mbarrier.  The epilogue: a warp reads its TMEM lanes (32
// windows) with tcgen05.ld, 16 queries at a time, forms each query's inner
// product and compares it with the largest one the prune test keeps
// (src/fsmeld.cpp:84-106, include/fsmeld_internal.h:9-19; the host's bisection);
// lane i collects query i's ballot and sets the survivors' bits in the query's
// window bit mask; k_bits_to_list turns a mask into the survivor list the GLB
// stage reads.
//
// What bounds it: instruction issue of the epilogue (about 25 instructions per
// query and 32 windows) beside the MMAs' operand reads (4 KB of A per MMA).
// Writing A out per chunk (16 KB and 16 expanded bytes a thread and side) and
// counting by shared-memory atomics took 1.64 ms for 32 queries of m = 128 on 2^22
// points, this takes 0.60.
//
// Waits are bounded (about a second of clock cycles): on a timeout the
// kernel records an error flag, waits once more for its MMAs, frees its
// TMEM and returns; the host reports FSMELD_E_CUDA.
#include <cute/arch/mma_sm100_desc.hpp>

#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

namespace {

constexpr int kGemmThreads = 256;
constexpr int kKChunk = 64;                         // K elements per chunk
constexpr size_t kResident = 104 * 1024;            // operands of two CTAs per SM
constexpr long long kWaitCycles = 2000000000LL;     // ~1 s at 2 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    cute::UMMA::SmemDescriptor d;
    d.start_address_ = static_cast<uint16_t>(saddr >> 4);
    d.leading_byte_offset_ = static_cast<uint16_t>(lbo >> 4);
    d.stride_byte_offset_ = static_cast<uint16_t>(sbo >> 4);
    d.version_ = 1;  // Blackwell descriptor
    d.lbo_mode_ = 0;
    d.base_offset_ = 0;
    d.layout_type_ = static_cast<uint8_t>(cute::UMMA::LayoutType::SWIZZLE_NONE);
    return d.desc_;
}

template <int NQ>
__host__ __device__ constexpr uint32_t gemm_idesc() {
    // kind::f16: D F32, A and B BF16, both K-major, M = 128, N = NQ
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NQ >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

// bounded wait for phase `parity` of the mbarrier; false on timeout
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok = 0;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > kWaitCycles) return false;
    }
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

// eight 0/1 mask bits -> eight BF16 values (1.0 = 0x3F80) packed in 16 bytes:
// bits 2i and 2i+1 are brought 16 apart and multiplied by 0x3F80 >> 2i
__device__ __forceinline__ uint4 bits_to_bf16x8(uint32_t b) {
    const uint32_t t = b * 0x8001u;
    return make_uint4((t & 0x00010001u) * 0x3F80u, (t & 0x00040004u) * 0x0FE0u, (t & 0x00100010u) * 0x03F8u,
                      (t & 0x00400040u) * 0x00FEu);
}

// one query's limits in the epilogue
struct __align__(16) Limits {
    double ml, mu;    // margins of the two inner products
    double keep_max;
    double unused;
};

}  // namespace

size_t lbgemm_smem_bytes(int nq_pad, int m, int* resident) {
    const size_t kpad = (size_t)(m + kKChunk - 1) / kKChunk * kKChunk;
    const size_t rows = 128 * (size_t)lbgemm_tiles(nq_pad), fixed = nq_pad * (sizeof(Limits) + 8);
    const size_t all = 2 * (rows + kpad) * 16 + 12 * (size_t)nq_pad * kpad + fixed;
    *resident = all <= kResident;
    return *resident ? all : 2 * (rows + kKChunk) * 16 + 12 * (size_t)nq_pad * kKChunk + fixed;
}

template <int NQ>
__global__ void __launch_bounds__(kGemmThreads, NQ <= 64 ? 3 : 2) k_lbgemm(Geom g, GemmJob job) {
    constexpr int kTiles = lbgemm_tiles(NQ);
    constexpr int kBlocks = NQ / 16;                        // 16-query blocks of the epilogue
    constexpr int kOwn = kBlocks > 1 ? kBlocks / 2 : 1;     // those of one warpgroup
    constexpr int kBChunk = 12 * NQ * kKChunk;              // bytes of a B chunk
    extern __shared__ __align__(1024) unsigned char gm_smem[];
    const int kc = job.resident ? job.kchunks : 1;          // K chunks staged at a time
    const int rows = 128 * kTiles + kc * kKChunk;           // A positions staged at a time
    unsigned char* As = gm_smem;                            // [2 sides][rows] eight elements per position
    unsigned char* Bs = As + 2 * rows * 16;                 // [kc] B chunks
    Limits* lim = (Limits*)(Bs + kc * kBChunk);             // [NQ]
    int* s_cnt = (int*)(lim + NQ);                          // [NQ] survivors, [NQ] valid windows
    int* s_valid = s_cnt + NQ;
    __shared__ __align__(8) unsigned long long s_bar;
    __shared__ uint32_t s_tmem;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int half = warp >> 2;                             // warpgroup
    const int m = job.m, kml = g.kml;
    const int per_seg = (kml + 128 * kTiles - 1) / (128 * kTiles);
    const long long items = g.S * per_seg;
    constexpr uint32_t kCols = lbgemm_cols(NQ);
    const uint32_t idesc = gemm_idesc<NQ>();
    const uint32_t bar = smem_u32(&s_bar);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    bool ex = false;
    for (int q = tid; q < NQ; q += kGemmThreads) {
        const bool in = q < job.nq;
        lim[q] = Limits{in ? job.margin_l[q] : 0.0, in ? job.margin_u[q] : 0.0, in ? job.keep_max[q] : 0.0, 0.0};
        s_cnt[q] = s_valid[q] = 0;
        ex = ex || (in && job.excl_b[q] >= 0);
    }
    if (job.resident)
        for (int i = tid; i < kc * (kBChunk / 16); i += kGemmThreads) ((uint4*)Bs)[i] = job.B[i];
    asm volatile("tcgen05.fence::before_thread_sync;");
    const bool any_excl = __syncthreads_or(ex) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = s_tmem;
    uint32_t phase = 0;
    bool failed = false;
    int cnt[kOwn], val[kOwn];  // lane i: query i of each own block
#pragma unroll
    for (int b = 0; b < kOwn; ++b) cnt[b] = val[b] = 0;

    for (long long it = blockIdx.x; it < items && !failed; it += gridDim.x) {
        const long long s = it / per_seg;
        const int j0 = (int)(it - s * per_seg) * 128 * kTiles;
        const unsigned* ml = job.mask_l + s * (long long)job.mask_words;
        const unsigned* mu = job.mask_u + s * (long long)job.mask_words;
        for (int c = 0; c < job.kchunks; c += kc) {
            // A: positions j0 + 64 c + i, eight mask bits each (0 past the segment)
            for (int i = tid; i < rows; i += kGemmThreads) {
                const int p = j0 + c * kKChunk + i, w = p >> 5;
                const unsigned l0 = w < job.mask_words ? ml[w] : 0u, l1 = w + 1 < job.mask_words ? ml[w + 1] : 0u;
                const unsigned u0 = w < job.mask_words ? mu[w] : 0u, u1 = w + 1 < job.mask_words ? mu[w + 1] : 0u;
                ((uint4*)As)[i] = bits_to_bf16x8(__funnelshift_r(l0, l1, p & 31) & 0xFFu);
                ((uint4*)As)[rows + i] = bits_to_bf16x8(__funnelshift_r(u0, u1, p & 31) & 0xFFu);
            }
            if (!job.resident) {
                const uint4* src = job.B + (size_t)c * (kBChunk / 16);
                for (int i = tid; i < kBChunk / 16; i += kGemmThreads) ((uint4*)Bs)[i] = src[i];
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncthreads();
            if (tid == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;");
                for (int ks = 0; ks < kc * (kKChunk / 16); ++ks) {
                    const unsigned char* bk = Bs + (ks / (kKChunk / 16)) * kBChunk + 2 * (ks % (kKChunk / 16)) * (NQ * 16);
#pragma unroll
                    for (int side = 0; side < 2; ++side) {
#pragma unroll
                        for (int t = 0; t < kTiles; ++t) {
                            const uint64_t ad =
                                umma_desc(smem_u32(As + (side * rows + t * 128 + ks * 16) * 16), 128, 128);
#pragma unroll
                            for (int sp = 0; sp < 3; ++sp) {
                                const uint64_t bd =
                                    umma_desc(smem_u32(bk + (side * 3 + sp) * NQ * kKChunk * 2), NQ * 16, 128);
                                mma_bf16(tmem + (2 * t + side) * NQ, ad, bd, idesc, (c > 0 || ks > 0 || sp > 0) ? 1u : 0u);
                            }
                        }
                    }
                }
                mma_commit(bar);
            }
            const bool done = mbar_wait(bar, phase);
            phase ^= 1;
            failed = __syncthreads_or(!done) != 0;  // block-uniform
            if (failed) {
                if (tid == 0) atomicExch(job.err, 1u);
                break;
            }
        }
        if (failed) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        // epilogue: warp w <-> TMEM lanes 32 (w mod 4) ...; a warpgroup takes every
        // second block of 16 queries (every second tile where there is one block)
#pragma unroll 1
        for (int t = kBlocks > 1 ? 0 : half; t < kTiles; t += kBlocks > 1 ? 1 : 2) {
            const int jw = j0 + 128 * t + 32 * (warp & 3), j = jw + lane;
            if (jw >= kml) break;
            const bool inwin = j < kml && j >= g.lo(s);
            const long long gi = inwin ? g.gidx(s, j) : 0;
            const double sg = inwin ? job.SIG[s * kml + j] : 0.0;
            const bool sig_ok = inwin && isfinite(sg) && sg > kSigmaFloor;
            const unsigned valid = __ballot_sync(0xffffffffu, sig_ok);
            // survivor bits of this warp's 32 consecutive windows: positions p0 .. p0+31
            const long long p0 = s * (long long)kml + jw - g.lo(s);
            const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 2 * t * NQ;
#pragma unroll
            for (int b = 0; b < kOwn; ++b) {
                const int q0 = 16 * (kBlocks > 1 ? 2 * b + half : 0);
                if (q0 >= job.nq) continue;
                uint32_t rl[16], ru[16];
                tmem_ld16(trow + q0, rl);
                tmem_ld16(trow + NQ + q0, ru);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                auto bound = [&](int i) {  // the inner product, lowered by its margins
                    const Limits& L = lim[q0 + i];
                    return dadd(dmax0(dsub((double)__uint_as_float(rl[i]), L.ml)),
                                dmax0(dsub((double)__uint_as_float(ru[i]), L.mu)));
                };
                unsigned mine = 0, mine_v = valid;
#pragma unroll
                for (int i = 0; i < 16; ++i) {  // the prune test, without its square roots
                    const unsigned bk = __ballot_sync(0xffffffffu, !(bound(i) > lim[q0 + i].keep_max));
                    if (lane == i) mine = bk;
                }
                if (any_excl) {
                    for (int i = 0; i < 16 && q0 + i < job.nq; ++i) {
                        const long long eb = job.excl_b[q0 + i], ee = job.excl_e[q0 + i];
                        const unsigned out = __ballot_sync(0xffffffffu, eb >= 0 && gi >= eb && gi < ee);
                        if (lane == i) mine_v &= ~out;
                    }
                }
                mine &= mine_v;
                if (job.zout) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const bool ok = __shfl_sync(0xffffffffu, mine_v, i) >> lane & 1u;
                        if (q0 + i >= job.nq || j >= kml) continue;
                        const int metric = job.metric[q0 + i];
                        double z = bound(i);
                        if (metric == DTW || metric == ERP) z = dsqrt(z);
                        else if (metric == LCSS) z = ddiv(z, (double)m);
                        job.zout[(size_t)(q0 + i) * job.zstride + s * kml + j] = ok ? z : dnan();
                    }
                }
                if (lane < 16 && q0 + lane < job.nq) {
                    val[b] += __popc(mine_v);
                    if (mine && job.bits) {
                        cnt[b] += __popc(mine);
                        unsigned* bq = job.bits + (size_t)(q0 + lane) * job.bit_words;
                        const long long w0 = p0 >> 5;  // floor for negative p0 (short targets' tail)
                        const int sh = (int)(p0 & 31);
                        const unsigned lo_bits = mine << sh;
                        if (w0 >= 0 && lo_bits) atomicOr(bq + w0, lo_bits);
                        if (sh && (mine >> (32 - sh))) atomicOr(bq + w0 + 1, mine >> (32 - sh));
                    }
                }
            }
        }
        // the accumulators are read: the next tile may overwrite them
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
    }
    if (failed) mbar_wait(bar, phase ^ 1);  // let issued MMAs drain (bounded) before freeing TMEM
#pragma unroll
    for (int b = 0; b < kOwn; ++b) {
        const int q = 16 * (kBlocks > 1 ? 2 * b + half : 0) + lane;
        if (lane < 16 && val[b]) atomicAdd(&s_valid[q], val[b]);
        if (lane < 16 && cnt[b]) atomicAdd(&s_cnt[q], cnt[b]);
    }
    __syncthreads();
    for (int q = tid; q < job.nq; q += kGemmThreads) {
        if (s_cnt[q]) atomicAdd(job.nsurv + q, (unsigned long long)s_cnt[q]);
        if (s_valid[q]) atomicAdd(job.nvalid + q, (unsigned long long)s_valid[q]);
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
}

// One warp per 32 positions: the ballot of the threshold tests is the word.
__global__ void __launch_bounds__(256) k_gemm_masks(Geom g, const double* __restrict__ Ln,
                                                    const double* __restrict__ Un, double t_l, double t_u,
                                                    unsigned* __restrict__ mask_l, unsigned* __restrict__ mask_u,
                                                    int words) {
    const int lane = threadIdx.x & 31;
    const long long total = g.S * (long long)words;
    const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
    for (long long it = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < total; it += nwarps) {
        const long long s = it / words;
        const int p = (int)(it - s * words) * 32 + lane;
        const bool in = p < g.m_k;
        const long long o = s * (long long)g.m_k + (in ? p : 0);
        const unsigned bl = __ballot_sync(0xffffffffu, in && Ln[o] >= t_l);
        const unsigned bu = __ballot_sync(0xffffffffu, in && Un[o] <= t_u);
        if (lane == 0) {
            mask_l[it] = bl;
            mask_u[it] = bu;
        }
    }
}

// survivor bit mask -> list of window indices (ascending within a block of
// 8192 windows; blocks append in any order).  A warp takes 32 words: their
// counts by a shuffle scan, then a word at a time, a lane per bit, so the
// stores are coalesced.
__global__ void __launch_bounds__(256) k_bits_to_list(const unsigned* __restrict__ bits, long long words,
                                                      long long* __restrict__ out, long long cap,
                                                      unsigned long long* __restrict__ n) {
    __shared__ int s_cnt[8];
    __shared__ unsigned long long s_off;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (long long b0 = (long long)blockIdx.x * 256; b0 < words; b0 += (long long)gridDim.x * 256) {
        const long long wi = b0 + tid;
        const unsigned v = wi < words ? bits[wi] : 0u;
        const int c = __popc(v);
        int inc = c;
        for (int d = 1; d < 32; d <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += x;
        }
        if (lane == 31) s_cnt[warp] = inc;
        __syncthreads();
        int before = 0, total = 0;
        for (int i = 0; i < 8; ++i) {
            before += i < warp ? s_cnt[i] : 0;
            total += s_cnt[i];
        }
        if (tid == 0) s_off = total ? atomicAdd(n, (unsigned long long)total) : 0ull;
        __syncthreads();
        const unsigned long long o = s_off + before;
        const unsigned below = (1u << lane) - 1;
        for (int i = 0; i < 32; ++i) {
            const unsigned x = __shfl_sync(0xffffffffu, v, i);
            const int at = __shfl_sync(0xffffffffu, inc - c, i);
            if (x >> lane & 1u) {
                const unsigned long long p = o + at + __popc(x & below);
                if (p < (unsigned long long)cap) out[p] = (b0 + warp * 32 + i) * 32 + lane;
            }
        }
        __syncthreads();
    }
}

template __global__ void k_lbgemm<16>(Geom, GemmJob);
template __global__ void k_lbgemm<32>(Geom, GemmJob);
template __global__ void k_lbgemm<64>(Geom, GemmJob);
template __global__ void k_lbgemm<128>(Geom, GemmJob);

const void* lbgemm_kernel(int nq_pad) {
    switch (nq_pad) {
        case 16: return (const void*)k_lbgemm<16>;
        case 32: return (const void*)k_lbgemm<32>;
        case 64: return (const void*)k_lbgemm<64>;
        case 128: return (const void*)k_lbgemm<128>;
        default: return nullptr;
    }
}

}  // namespace fsm
