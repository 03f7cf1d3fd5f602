// Kernel entry points and their job descriptors.
#pragma once

#include "common.cuh"

namespace fsm {

struct ThrJob {
    QueryDev q;
    const double* Un;  // [S][m_k]
    const double* Ln;
    double* thr;       // [S][2]: (t_l, t_u) per segment
};

struct LbJob {
    QueryDev q;
    const double* Un;
    const double* Ln;
    const double* thr;
    const double* SIG;          // window sigmas [S][kml] (validity)
    double* zout;               // optional: LB per window [S][kml] (NaN if invalid)
    long long* surv;            // optional: LB survivors (global window index)
    long long surv_cap;
    unsigned long long* nsurv;
    unsigned long long* nvalid; // valid, non-excluded windows
    long long* segc;            // optional: per segment (valid, after LB, after GLB)
    unsigned char* gwork;       // global scratch when the FFT buffers exceed shared memory
    long long slot_stride;
};

struct GlbJob {
    QueryDev q;
    const double* target;
    const double* lraw;         // forward windows min / max(t[p .. p+w]) of the raw target
    const double* uraw;
    const float* rel;           // optional: [3][S m_k] FP32 relative to the segment (k_rel)
    const double2* rseg;        // [S] what it is relative to, and how far a point is off at most
    const double* MU;
    const double* SIG;
    const long long* in;
    const double* in_b;         // stage 2 input: boundary terms (NaN: T->Q decided without them, -1: abandoned)
    const double* in_t;         // stage 2 input: T->Q sums (LCSS: T->Q reward)
    const unsigned long long* n_in;
    long long in_cap;
    long long* out;
    double* out_b;
    double* out_t;
    unsigned long long* n_out;
    long long out_cap;
    long long* segc;
    const double* cutoff_ptr;   // when set: the cutoff in device memory (read at kernel start)
};

struct DpJob {
    QueryDev q;
    const double* target;
    const double* lraw;         // forward windows of the raw target (cascading abandon terms)
    const double* uraw;
    const float* rel;           // optional: FP32 points and windows by segment (k_screen)
    const double2* rseg;
    const double* MU;
    const double* SIG;
    const long long* list;      // candidates, or null for windows [0, n_windows)
    const double* list_s;       // optional: GLB Q->T sum per candidate (cascading abandon)
    const double* list_t;       // optional: GLB T->Q sum per candidate (k_bitdp)
    const unsigned long long* n_list;
    long long list_cap;
    long long n_windows;
    int mode;                   // 0: keep dist <= cutoff; 1: keep every finite dist
    double cutoff;
    long long* out_idx;
    double* out_dist;
    unsigned long long* n_out;
    long long out_cap;
    unsigned long long* n_valid;
    unsigned long long* next;   // work counter (zeroed before the launch)
    double* gwork;              // global band scratch when shared memory is too small
    int force_exact;            // every candidate in the DP's exact boundary mode
    unsigned long long* n_cells;  // band cells computed (optional)
    const double* cutoff_ptr;   // when set: the cutoff in device memory (read at kernel start)
    long long* screened;        // when set: room for the candidates an FP32 screen leaves
    unsigned long long* n_screened;
    int few;                    // the screen will leave few (a ranking at a refined bound)
    long long stride;           // without a list: window of item i (0: i itself)
    const unsigned long long* sample;  // optional: valid and kept windows of a sample that was screened before
    long long run_from, run_to; // runs on lists of [run_from, run_to) candidates only (run_to 0: no upper limit)
};

// LB_IP of a group of queries of equal (m, w) with shared thresholds as one
// tensor-core product (k_lbgemm); per-query arrays are indexed by query
struct GemmJob {
    const double* Un;           // [S][m_k]
    const double* Ln;
    const double* SIG;          // [S][kml]
    double t_l, t_u;            // the group's thresholds
    const uint4* B;             // BF16 penalty operand, per K chunk [side][split][NQ x 64] (operand layout)
    int m, nq, kchunks, resident;
    const double* margin_l;     // rounding-error margins of the lower / upper inner products
    const double* margin_u;
    const int* metric;
    const double* keep_max;     // the largest inner product the prune test keeps
    const long long* excl_b;    // exclusion interval per query (-1: none)
    const long long* excl_e;
    double* zout;               // optional: bound per window, [q][zstride]
    long long zstride;
    unsigned* bits;             // survivors per query: bit g of bits[q * bit_words ...] (zeroed by the caller)
    long long bit_words;
    unsigned long long* nsurv;  // [nq]
    unsigned long long* nvalid; // [nq]
    unsigned int* err;          // set when a bounded wait gave up
    const unsigned* mask_l;     // window masks g of the group (k_gemm_masks): [S][mask_words] 32-bit words,
    const unsigned* mask_u;     // bit p of a segment = position p (0 at and past m_k)
    int mask_words;
};
template <int NQ>
__global__ void k_lbgemm(Geom g, GemmJob job);
// bit p of segment s: Ln[s][p] >= t_l (mask_l), Un[s][p] <= t_u (mask_u); 0 for p >= m_k
__global__ void k_gemm_masks(Geom g, const double* __restrict__ Ln, const double* __restrict__ Un, double t_l,
                             double t_u, unsigned* __restrict__ mask_l, unsigned* __restrict__ mask_u, int words);
const void* lbgemm_kernel(int nq_pad);  // NQ in {16, 32, 64, 128}
__global__ void k_bits_to_list(const unsigned* __restrict__ bits, long long words, long long* __restrict__ out,
                               long long cap, unsigned long long* __restrict__ n);
// shared memory a CTA, and whether all of B stays in it
size_t lbgemm_smem_bytes(int nq_pad, int m, int* resident);
// 128-window tiles of a CTA at a time, and their TMEM columns
__host__ __device__ constexpr int lbgemm_tiles(int nq_pad) { return nq_pad >= 64 ? 1 : 64 / nq_pad; }
__host__ __device__ constexpr int lbgemm_cols(int nq_pad) { return lbgemm_tiles(nq_pad) * 2 * nq_pad; }
constexpr int kLbGemmThreads = 256;
constexpr int kLbGemmKChunk = 64;

// window statistics: one block per seg (mvmean_segments) segments, one warp runs the running sums
// and eight load the points and derive mean and sigma
constexpr int kMvmeanThreads = 288;
__global__ void k_mvmean(const double* __restrict__ target, Geom g, double* __restrict__ mu,
                         double* __restrict__ sig, int seg, int sms);
int mvmean_segments(long long S, int sm_count);
// one block per tile of T * OPT outputs of a segment
template <int T, int OPT>
__global__ void k_envelope(const double* __restrict__ target, const double* __restrict__ Lraw,
                           const double* __restrict__ Uraw, const double* __restrict__ MU,
                           const double* __restrict__ SIG, Geom g, int w, int tiles, double* __restrict__ Un,
                           double* __restrict__ Ln);
template <int T, int IPT, bool GW>
__global__ void k_threshold(Geom g, ThrJob job, unsigned char* gwork, long long slot_stride, int z_shared);
template <int T, bool GW>
__global__ void k_lbip(Geom g, LbJob job, const double2* __restrict__ W, int P, int logP);
// LB_IP by the changes of the masks (DTW, ERP, MSM) or by popcounts (EDR,
// LCSS); keep_max: the largest inner product the prune test keeps
template <int T, bool POPC>
__global__ void k_lbip_runs(Geom g, LbJob job, double keep_max);
size_t lbip_runs_smem_bytes(int m_k, int kml, int m, bool popc);
template <int METRIC>
__global__ void k_glb_tq(Geom g, GlbJob job);
template <int METRIC>
__global__ void k_glb_qt(Geom g, GlbJob job);
// forward windows min/max(t[p .. p+w]) by doubling in shared memory, kFwdTile
// outputs per CTA and tile
constexpr int kFwdThreads = 256;
constexpr int kFwdTile = 2048;
__global__ void k_fwd_env(const double* __restrict__ t, long long n, int w, double* __restrict__ lo,
                          double* __restrict__ up);
size_t fwd_env_smem_bytes(int w);
// FP32 points and centred windows by segment, relative to its middle (GLB)
__global__ void k_rel(const double* __restrict__ t, const double* __restrict__ lraw, const double* __restrict__ uraw,
                      Geom g, int w, float* __restrict__ rel, double2* __restrict__ seg);
template <int METRIC, bool GW>
__global__ void k_dp(Geom g, DpJob job);
// the DP kernel for a metric, with its band in shared memory or in job.gwork
const void* dp_kernel(int metric, bool gw);
// wide-band DP: one warp per candidate, one anti-diagonal per step, the band
// in registers (K chunks of 64 band offsets per warp, 2w+1 <= 64 K)
// INNER: with the fast steps away from the matrix's corners
template <int METRIC, int K, bool INNER>
__global__ void k_dpw(Geom g, DpJob job);
constexpr int kDpwThreads = 32;  // one warp: a short list spreads over the SMs
constexpr int kDpwMaxChunks = 8;  // w <= 255
// the wavefront kernel for (metric, w), or null when the band is too wide
const void* dpw_kernel(int metric, int w);
// shared memory: the query plus, per warp, its candidate and the row-block
// suffix sums of the abandon bound
__host__ __device__ size_t dpw_warp_doubles(int m);
size_t dpw_smem_bytes(int m, int warps);
// the exact DP for lists of `from` candidates and more behind the screen (kernel
// null: the wavefront kernel for every length)
struct LongDp {
    const void* kernel;
    long long from;
    int threads, blocks;  // threads a block, blocks an SM
    size_t smem;
    bool lane;
};
LongDp long_dp(const DpJob& job, bool screened, int sm_count);
// whether a list of n candidates is outside job's lengths
__host__ __device__ inline bool other_length(const DpJob& job, unsigned long long n) {
    return n < (unsigned long long)job.run_from || (job.run_to && n >= (unsigned long long)job.run_to);
}
// EDR and LCSS as bit vectors: the query's matching table (BitTab in
// common.cuh), one lane per candidate
constexpr int kBitThreads = 256;
constexpr int kBitMaxM = 2048;
// row r of the table: the query points that match candidate points of rank r
__global__ void k_bit_table(const int* __restrict__ pa, const int* __restrict__ pb, int m, int pad, int rs,
                            unsigned* __restrict__ table);
template <int METRIC, int NW>
__global__ void k_bitdp(Geom g, DpJob job, BitTab bt);
// the kernel for (metric, w), or null when the band is wider than 16 words
const void* bitdp_kernel(int metric, int w);
int bit_words(int w);
// byte offset of the table in shared memory, after the ends and the grid
__host__ __device__ inline size_t bit_table_offset(int m) {
    return ((size_t)(2 * m + 1) * 8 + (kBitBuckets + 1) * 2 + 15) & ~size_t(15);
}
// FP32 screen before the exact DP (DTW, ERP, MSM): the candidates it cannot
// drop, to out; lists of at most `few` entries go on whole
constexpr int kScreenThreads = 128;
template <int METRIC, int R>
__global__ void k_screen(Geom g, DpJob job, long long* __restrict__ out, unsigned long long* __restrict__ n_out,
                         long long few);
const void* screen_kernel(int metric, int w);
long long screen_few(const DpJob& job, int sm_count);
constexpr long long kScreenSample = 2048;
bool screen_sampled(const DpJob& job, int sm_count);
size_t screen_warp_bytes(int metric, int w);
size_t screen_smem_bytes(int metric, int w, int m, int warps);
double mean_step(const double* x, int m);  // QueryDev::step
double query_spread(int metric, const double* x, int m);       // QueryDev::spread
double screen_loose(int metric, double spread, bool raw);      // QueryDev::loose
__global__ void k_lb_filter(Geom g, const double* __restrict__ z, const double* __restrict__ SIG,
                            const double* __restrict__ cutoff, int metric, long long* out,
                            unsigned long long* n_out, long long cap);
// results of a query that k_finish leaves in host memory
constexpr int kFinishThreads = 512;
constexpr int kFinishSort = 4096;  // results sorted in one block
constexpr int kFinishOut = 1024;   // results copied
size_t finish_smem_bytes();
struct FinishOut {
    unsigned long long cnt[16];
    long long idx[kFinishOut];
    double dist[kFinishOut];
};
__global__ void k_finish(const unsigned long long* __restrict__ cnt, int ncnt, int out_slot, long long cap, int lex,
                         long long* __restrict__ idx, double* __restrict__ dist, FinishOut* __restrict__ host);
__global__ void k_order(const unsigned long long* __restrict__ n_in, const long long* __restrict__ idx,
                        const double* __restrict__ dist, long long* __restrict__ out_idx,
                        double* __restrict__ out_dist, long long cap, unsigned long long* __restrict__ total);
// top-k: tau from the seeds, and the windows around the best of them
constexpr int kRefineReach = 15;
constexpr int kRefinePicks = 132;  // 132 x 31 windows fit kFinishSort
__global__ void k_tau_block(const double* __restrict__ dist, const long long* __restrict__ idx, int sorted,
                            const unsigned long long* __restrict__ n_seed, long long cap, long long k, long long tsn,
                            int picks, double* tau, long long* __restrict__ list,
                            unsigned long long* __restrict__ n_list);
__global__ void k_tau_refine(const double* __restrict__ dist, const unsigned long long* __restrict__ n_dist,
                             long long k, double* tau);
__global__ void k_seed(Geom g, const double* __restrict__ z, const double* __restrict__ SIG, int per_seg,
                       long long* out, unsigned long long* n_out, long long cap);

// raise a kernel's dynamic shared-memory limit on a device to at least `bytes`
// (process-wide, never lowered; the device must be current)
cudaError_t raise_smem_limit(const void* kernel, int device, size_t bytes);

size_t mvmean_smem_bytes();
size_t envelope_smem_bytes(int tile, int m, int w);
// where a block of k_threshold keeps its working set
struct ThrMem {
    bool gw;         // runs and sorted values in global scratch
    int z_shared;    // the sweep in shared memory
    size_t smem;     // dynamic shared memory
    size_t gbytes;   // global scratch per block
};
template <int T, int IPT>
ThrMem threshold_mem(int m, size_t smem_optin);
size_t lbip_smem_bytes(int P);
int lbip_set_w16();
// DP block size (2 warps: the per-warp band scratch sets the occupancy)
constexpr int kDpThreads = 64;
// DP per-warp scratch: band row (2w+1 cells + one out-of-band cell) and the
// candidate ring (power of two >= 2w+2 points), 32 lanes each
__host__ __device__ int dp_ring(int w);
__host__ __device__ size_t dp_warp_doubles(int w);

}  // namespace fsm
