// Rolling window mean / standard deviation per macro segment.
//
// Follows src/mvmean.cpp:9-46 operation for operation: the running sums are
// restarted at every macro segment (src/fsmeld.cpp:753, 861) and updated by
// `sum = sum - outgoing + incoming` with non-finite points replaced by 0.0;
// a window containing a non-finite point gets NaN statistics.  The sums are
// a serial recurrence whose rounding decides validity (sigma <= 1e-12) and
// every z-normalised candidate, so each segment is one sequential chain: one
// lane per segment, up to 16 segments per block.
//
// What bounds it: the chain, two dependent FP64 adds (16 cycles) per point and
// segment, m_k points long whatever the target's length (24 cycles a point
// with its shared-memory accesses), next to about 35 FP64 operations per window
// for mean and sigma; from a few hundred blocks on also
// the HBM traffic (one read of the target with the m-1 halo per segment, the
// outgoing points again from L2, 16 bytes written per window).  So one warp of
// the block does nothing but the chain: its operands lie ready in shared
// memory and its loop is 32 unrolled steps without a branch, and the other
// eight warps do the rest a tile of 32 points ahead or behind:
//   * the incoming points t[k] and the outgoing points t[k-m] (0 before the
//     first full window) of tile t + 3 into registers, those of tile t + 1
//     from registers into shared memory, non-finite points as 0.0 and one bit
//     in a mask per segment (x - 0.0 and x + 0.0 leave every sum as it is, so
//     the first m points and the skipped ones need no case of their own);
//   * mean and sigma of the windows that end in tile t - 1 (two divisions by
//     m, each a multiply by RN(1/m) and FMA corrections that give the
//     correctly rounded quotient, and a square root), written coalesced.
// One block barrier per tile.  Short targets take fewer segments per block
// (mvmean_segments), so that their windows' divisions spread over more SMs.
// Measured against one warp that loads, chains and stages: m_k = 16384 2.39 ->
// 0.33 ms, 2^20 points with m_k = 1024 0.162 -> 0.046 ms, 2^24 points with
// m_k = 2048 (585 blocks) 0.320 -> 0.165 to 0.18 ms = 2.3 to 2.6 TB/s.
//
// Raw (non-normalised) mode (g.raw): a window is valid iff its points are all
// finite, and its statistics are mean 0 and sigma 1, so every later stage
// sees the raw values ((t - 0) / 1 = t exactly) with the same code.
#include "common.cuh"
#include "kernels.cuh"

namespace fsm {

namespace {
constexpr int kTile = 32;
constexpr int kPitch = kTile + 1;  // padded rows: lane-strided smem reads hit distinct banks
constexpr int kRows = 16;          // segments per block at most
constexpr int kTileDoubles = kRows * kPitch;
constexpr int kMaskTiles = 4;      // tiles whose non-finite masks are kept (tile t - 1 .. t + 1)
constexpr int kHelpers = kMvmeanThreads / 32 - 1;  // two rows of a tile each
static_assert(2 * kHelpers == kRows, "helpers take rows h and h + kHelpers");
}

__global__ void __launch_bounds__(kMvmeanThreads, 4) k_mvmean(const double* __restrict__ target, Geom g,
                                                              double* __restrict__ mu, double* __restrict__ sig,
                                                              int seg, int sms) {
    extern __shared__ __align__(16) double sm[];
    double* tin = sm;                                     // [2][kRows][kPitch] incoming points t[k], by tile parity
    double* tout = tin + 2 * kTileDoubles;                // [2][kRows][kPitch] outgoing points t[k-m]
    double* S1 = tout + 2 * kTileDoubles;                 // [2][kRows][kPitch] sums after each point
    double* S2 = S1 + 2 * kTileDoubles;                   // [2][kRows][kPitch] sums of squares
    unsigned* IM = (unsigned*)(S2 + 2 * kTileDoubles);    // [kMaskTiles][kRows] non-finite incoming points of a row
    unsigned* OM = IM + kMaskTiles * kRows;                  // [kMaskTiles][kRows] the same of the outgoing points
    int* NF = (int*)(OM + kMaskTiles * kRows);               // [2][kRows] non-finite points in the window before the tile
    const int lane = threadIdx.x & 31;
    // the chain warps of the blocks resident on one SM sit on different
    // sub-partitions (blocks are handed out to the SMs in turn)
    const int id = threadIdx.x >> 5, cw = (int)(blockIdx.x / (unsigned)sms) & 3;
    const bool chain = id == cw;
    const int h = id - (id > cw ? 1 : 0);  // helper: rows h and h + kHelpers
    const long long s0 = (long long)blockIdx.x * seg;  // seg <= kRows segments
    const int m = g.m, mk = g.m_k, kml = g.kml;
    const int ntiles = (mk + kTile - 1) / kTile;
    const bool row[2] = {h < seg && s0 + h < g.S, h + kHelpers < seg && s0 + h + kHelpers < g.S};
    const double* tp[2] = {target + g.off(row[0] ? s0 + h : 0) + lane, target + g.off(row[1] ? s0 + h + kHelpers : 0) + lane};

    // helpers: this thread's points of tile t (row h + kHelpers u, point lane)
    struct Points { double in[2], out[2]; };
    auto load_tile = [&](int t, Points& p) {
        if (h >= seg) return;
        const int k0 = t * kTile, k = k0 + lane;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool in = row[u] && k < mk;
            p.in[u] = in ? tp[u][k0] : 0.0;
            p.out[u] = in && k >= m ? tp[u][k0 - m] : 0.0;
        }
    };
    auto stage_tile = [&](int t, const Points& p) {
        if (h >= seg) return;
        const int b = (t & (kMaskTiles - 1)) * kRows, st = (t & 1) * kTileDoubles;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int r = h + kHelpers * u, o = st + r * kPitch + lane;
            const bool bi = !isfinite(p.in[u]), bo = !isfinite(p.out[u]);
            const unsigned mi = __ballot_sync(0xffffffffu, bi), mo = __ballot_sync(0xffffffffu, bo);
            if (r >= seg) continue;
            tin[o] = bi ? 0.0 : p.in[u];
            tout[o] = bo ? 0.0 : p.out[u];
            if (lane == 0) {
                IM[b + r] = mi;
                OM[b + r] = mo;
            }
        }
    };
    // helpers: mean and sigma of the windows that end in tile t
    const double dm = (double)m;
    const double invm = ddiv(1.0, dm);  // S / m by the reciprocal method (correctly rounded)
    auto finish_tile = [&](int t) {
        const int k = t * kTile + lane;
        const int b = t & 1, ms = (t & (kMaskTiles - 1)) * kRows;
        if (k < m - 1 || k >= mk) return;
        const unsigned upto = 0xffffffffu >> (31 - lane);
        double mean[2] = {}, sd[2] = {};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int r = h + kHelpers * u, o = b * kTileDoubles + r * kPitch + lane;
            if (!row[u]) continue;
            const bool bad = NF[b * kRows + r] + __popc(IM[ms + r] & upto) - __popc(OM[ms + r] & upto) != 0;
            mean[u] = 0.0;
            sd[u] = 1.0;  // raw mode: valid iff every point is finite
            if (!g.raw) {
                // both quotients by the reciprocal method with one range test
                const double a1 = S1[o], a2 = S2[o];
                const double e1 = rcp_div_estimate(a1, invm), e2 = rcp_div_estimate(a2, invm);
                double z1 = rcp_div_finish(a1, dm, invm, e1), z2 = rcp_div_finish(a2, dm, invm, e2);
                if (!(rcp_div_in_range_bits(e1) & rcp_div_in_range_bits(e2))) {
                    z1 = ddiv(a1, dm);
                    z2 = ddiv(a2, dm);
                }
                mean[u] = z1;
                sd[u] = dsqrt(dsub(z2, dmul(z1, z1)));
            }
            if (bad) mean[u] = sd[u] = dnan();
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (!row[u]) continue;
            const long long w = (s0 + h + kHelpers * u) * kml + (k - m + 1);
            mu[w] = mean[u];
            sig[w] = sd[u];
        }
    };

    double s1 = 0.0, s2 = 0.0;
    int nonfinite = 0;
    Points p1{}, p2{};
    if (!chain) {
        load_tile(0, p1);
        stage_tile(0, p1);
        load_tile(1, p1);
        load_tile(2, p2);
    }
    __syncthreads();
    const int first = (m - 1) / kTile;  // the first tile that a window ends in
    for (int t = 0; t <= ntiles; ++t) {
        if (chain) {
            if (t < ntiles && lane < seg) {
                const int b = t & 1, ms = (t & (kMaskTiles - 1)) * kRows, o = b * kTileDoubles + lane * kPitch;
                const double *in = tin + o, *out = tout + o;
                double *q1 = S1 + o, *q2 = S2 + o;
                NF[b * kRows + lane] = nonfinite;
                nonfinite += __popc(IM[ms + lane]) - __popc(OM[ms + lane]);
                // src/mvmean.cpp:16-27 (outgoing 0.0) and 32-44; operands in
                // registers four steps ahead of the adds
                double vi[4], vo[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) { vi[u] = in[u]; vo[u] = out[u]; }
#pragma unroll
                for (int x0 = 0; x0 < kTile; x0 += 4) {
                    double ni[4] = {}, no[4] = {};
                    if (x0 + 4 < kTile) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) { ni[u] = in[x0 + 4 + u]; no[u] = out[x0 + 4 + u]; }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        s1 = dadd(dsub(s1, vo[u]), vi[u]);
                        s2 = dadd(dsub(s2, dmul(vo[u], vo[u])), dmul(vi[u], vi[u]));
                        q1[x0 + u] = s1;
                        q2[x0 + u] = s2;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) { vi[u] = ni[u]; vo[u] = no[u]; }
                }
            }
        } else {
            if (t + 1 < ntiles) stage_tile(t + 1, p1);
            p1 = p2;
            load_tile(t + 3, p2);
            if (t > first) finish_tile(t - 1);
        }
        // tile t's sums are staged, tile t-1's consumed, tile t+1's points are there
        __syncthreads();
    }
}

size_t mvmean_smem_bytes() {
    return sizeof(double) * 8 * kTileDoubles + sizeof(unsigned) * (2 * kMaskTiles + 2) * kRows;
}

// Segments per block: the fewest for which all blocks are resident at once,
// one chain on every sub-partition of an SM at most (the chain of a block takes
// the same time for one segment as for kRows)
int mvmean_segments(long long S, int sm_count) {
    int seg = 2;
    while (seg < kRows && (S + seg - 1) / seg > 4LL * sm_count) seg *= 2;
    return seg;
}

}  // namespace fsm
