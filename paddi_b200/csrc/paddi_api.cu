// paddi_api.cu -- host side of libpaddi: contexts, the per-attempt pipeline,
// the PD3 and PALMAD drivers and the exported C ABI (include/paddi.h).
//
// One attempt (one length m, one threshold r) is
//   witnesses   k_witness_check   (PALMAD: neighbours known from the length before)
//   phase 1     k_phase1          (reference: gpu_local_candidate_select +
//                                  gpu_local_define_candidates, src/PD3.cuh:18-29)
//   compaction  k_compact         (get_node_candidates_num + local_candidates_union,
//                                  src/sets_processing.hpp:49-113)
//   refine      k_refine_*        (gpu_local_discords_refine + gpu_global_discords_refine,
//                                  src/PD3.cuh:31-50)
//   selection   k_finalize, k_recheck, k_select
//                                 (get_node_discords_num + find_top1_discord,
//                                  src/sets_processing.hpp:11-87)
// all on one stream as a chain of launches; the selection writes a small result
// record to pinned host memory.  The r-schedules are restated from src/main.cu:136-233 in the
// same float arithmetic as the reference, so equal distances give equal
// thresholds.
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <algorithm>
#include <atomic>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "../../include/paddi.h"
#include "paddi_internal.cuh"

cudaError_t paddi_raise_smem_limit(const void *func, size_t bytes)
{
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> set;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(mu);
    size_t &cur = set[{dev, func}];
    if (bytes <= cur) return cudaSuccess;
    e = cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) cur = bytes;
    return e;
}

#define PADDI_API extern "C" __attribute__((visibility("default")))

struct paddi_ctx {
    paddi_opts opts;
    int device = 0;
    int num_sms = 0;
    cudaStream_t st = nullptr;
    cudaEvent_t ev[4] = {}; // ordering against a caller's stream (0, 1), autotuner (2, 3)
    // PADDI_TRACE=1 in the environment: one stderr line per attempt with the
    // candidates entering every refine round
    bool trace = false;
    PaddiAttemptDev *h_trace = nullptr;
    std::string err;
    size_t cap_n = 0; // series capacity (values)
    int32_t rc_cap = 0; // FP64 recheck capacity (windows)
    // device buffers
    float *d_x = nullptr;
    float4 *d_wst = nullptr;
    float *d_mu = nullptr;
    double2 *d_ms64 = nullptr; // {FP64 mean, FP64 inverse norm}
    uint8_t *d_flat = nullptr, *d_alive = nullptr, *d_pruned = nullptr;
    int32_t *d_cand = nullptr, *d_rcslot = nullptr, *d_recheck = nullptr;
    int32_t *d_list[2] = {nullptr, nullptr};
    int32_t *d_pc = nullptr;  // range-discord profile output (allocated on first use)
    float *d_pn = nullptr;
    uint16_t *d_bq = nullptr; // tensor-core refine: split series slices per tile block
    uint32_t *d_bmax = nullptr; // tensor-core refine: block maxima (bmax_cap entries)
    int64_t bmax_cap = 0;
    float4 *d_wdq = nullptr;  // tensor-core refine: epilogue window data per tile block
    // r guidance: exact FP64 nn of the bound window, kept incrementally
    PaddiGuide *d_guide = nullptr, *h_guide = nullptr; // state + result (h: pinned)
    double *d_G = nullptr;                  // shifted dot products, two buffers (on first use)
    size_t G_cap = 0;                       // windows per buffer
    // witnesses of the current PALMAD run (allocated on first use): the length
    // they stand at (0: none in use) and the steps taken so far
    PaddiWitness W = {};
    void *W_mem = nullptr; // one allocation
    size_t W_cap = 0;      // windows
    int wit_m = 0;
    PaddiWitnessRun wit = {};
    int wit_edge = 0, wit_steps = 0; // steps between wit_edge and wit_edge + 1 so far
    // learned r predictor
    bool model_ok = false;
    float model_margin = 1.f;
    float *d_model = nullptr;               // FP32 parameters
    void *d_model_bf16 = nullptr;           // BF16 copy used for inference
    float *d_feat = nullptr, *d_pred = nullptr;
    float *h_feat = nullptr;                // pinned: features [12] then prediction
    uint32_t *d_rho = nullptr;
    unsigned long long *d_nn64 = nullptr;
    // state of the current attempt: one of two, the selection of each attempt
    // clears the other (dirty: an attempt broke off before that)
    PaddiAttemptDev *d_att = nullptr, *d_att2[2] = {nullptr, nullptr};
    bool att_dirty = false;
    bool alive_used = false; // d_alive is not all ones: written from witnesses, not reset
    unsigned long long *d_tprep = nullptr; // time stamps of the current length's preparation
    PaddiAttemptResult *d_res = nullptr;
    // {flat windows, flat span (2), fragile windows} of the current length: one of
    // two, the statistics of each length clear the other
    int32_t *d_flatcount = nullptr, *d_flat2[2] = {nullptr, nullptr};
    int prep_launches = 0;          // kernels of the current length's preparation
    int32_t *d_frag = nullptr;      // fragile windows of the current length
    PaddiAttemptResult *h_res = nullptr;
    bool umma_ok = false;
    // test hooks (paddi_debug_set): fail the k-th next device allocation; the
    // refine's barrier-wait limit; withhold one refine pipeline stage
    int64_t fail_alloc = 0;
    long long wait_cycles = 0;
    int32_t withhold = 0;
    int32_t last_passes = 0; // selection passes of the last attempt
    // the small buffers above live in one device and one pinned block
    void *d_small = nullptr, *h_small = nullptr;
    // worker contexts of paddi_palmad_batched, kept for the next call: as many as
    // the last call used, while they hold at most kWorkerPoints points together;
    // destroyed with the context, after a failed call, or when an allocation of this
    // context needs their memory
    std::vector<paddi_ctx *> workers;
};

namespace {

const char *kStatusText[] = {"ok",
                             "invalid argument",
                             "CUDA error",
                             "out of device memory",
                             "r-schedule did not converge within the attempt cap",
                             "no sm_100 CUDA device",
                             "internal capacity exceeded",
                             "unsupported option"};

paddi_status fail(paddi_ctx *c, paddi_status s, const std::string &msg)
{
    if (c) c->err = msg;
    return s;
}

#define CK(call)                                                                            \
    do {                                                                                    \
        cudaError_t e_ = (call);                                                            \
        if (e_ != cudaSuccess)                                                              \
            return fail(ctx, e_ == cudaErrorMemoryAllocation ? PADDI_ERR_OUT_OF_MEMORY      \
                                                             : PADDI_ERR_CUDA,              \
                        std::string(#call) + ": " + cudaGetErrorString(e_));                \
    } while (0)

// Points that kept workers may hold, in all: about 1 GB of buffers (120 bytes a
// point).  A call on four streams, lengths 32..55, with kept workers and without: 32
// series of 2^14..2^17 points 55 and 75 ms, 16 of 2^18..2^20 507 and 548, 8 of
// 2^20..2^21 1215 and 1324 to 1400.  Longer ones take longer still and would hold
// memory that others on the device may need.
constexpr size_t kWorkerPoints = (size_t)1 << 23;

void drop_workers(paddi_ctx *ctx, size_t keep = 0)
{
    while (ctx->workers.size() > keep) {
        paddi_ctx_destroy(ctx->workers.back());
        ctx->workers.pop_back();
    }
}

template <typename T>
void dfree(T *&p)
{
    if (p) cudaFree((void *)p);
    p = nullptr;
}

void free_witness(paddi_ctx *ctx)
{
    dfree(ctx->W_mem);
    ctx->W = {};
    ctx->W_cap = 0;
    ctx->wit_m = 0;
}

// Every device allocation of a context goes through here, so a test can have
// one refused (PADDI_DEBUG_FAIL_ALLOC) and check that PADDI_ERR_OUT_OF_MEMORY
// reaches the caller.  What the context holds only to be faster is given up
// before that: idle workers, the witnesses (a run goes on without them) and the
// block maxima (the recheck then scans the whole series).
template <typename T>
cudaError_t dmalloc(paddi_ctx *ctx, T **p, size_t bytes)
{
    const bool refuse = ctx->fail_alloc > 0 && --ctx->fail_alloc == 0;
    cudaError_t e = refuse ? cudaErrorMemoryAllocation : cudaMalloc((void **)p, bytes);
    if (e == cudaErrorMemoryAllocation && !ctx->workers.empty()) {
        cudaGetLastError();
        drop_workers(ctx);
        e = cudaMalloc((void **)p, bytes);
    }
    if (e == cudaErrorMemoryAllocation && ctx->W_mem) {
        cudaGetLastError();
        free_witness(ctx); // (cudaFree waits for the kernels that use them)
        e = cudaMalloc((void **)p, bytes);
    }
    if (e == cudaErrorMemoryAllocation && ctx->d_bmax) {
        cudaGetLastError();
        dfree(ctx->d_bmax); // (as above)
        ctx->bmax_cap = 0;
        e = cudaMalloc((void **)p, bytes);
    }
    if (e != cudaSuccess) cudaGetLastError(); // reported by this call alone
    return e;
}

void free_buffers(paddi_ctx *ctx)
{
    dfree(ctx->d_x);
    dfree(ctx->d_wst);
    dfree(ctx->d_mu);
    dfree(ctx->d_ms64);
    dfree(ctx->d_flat);
    dfree(ctx->d_alive);
    dfree(ctx->d_pruned);
    dfree(ctx->d_cand);
    dfree(ctx->d_rcslot);
    dfree(ctx->d_recheck);
    dfree(ctx->d_rho);
    dfree(ctx->d_nn64);
    dfree(ctx->d_list[0]);
    dfree(ctx->d_list[1]);
    dfree(ctx->d_frag);
    dfree(ctx->d_bq);
    dfree(ctx->d_wdq);
    dfree(ctx->d_bmax);
    dfree(ctx->d_pc);
    dfree(ctx->d_pn);
    dfree(ctx->d_G);
    ctx->G_cap = 0;
    free_witness(ctx);
    ctx->cap_n = 0;
    ctx->rc_cap = 0;
}

// A recheck queue of `cap` windows in place of the present one, which stays when the
// memory is refused.  No kernel that uses it may be in flight.
cudaError_t set_recheck_cap(paddi_ctx *ctx, int32_t cap)
{
    int32_t *q = nullptr;
    unsigned long long *v = nullptr;
    cudaError_t e = dmalloc(ctx, &q, sizeof(int32_t) * (size_t)cap);
    if (e == cudaSuccess) e = dmalloc(ctx, &v, sizeof(unsigned long long) * (size_t)cap);
    if (e != cudaSuccess) {
        dfree(q);
        return e;
    }
    dfree(ctx->d_recheck);
    dfree(ctx->d_nn64);
    ctx->d_recheck = q;
    ctx->d_nn64 = v;
    ctx->rc_cap = cap;
    return cudaSuccess;
}

paddi_status ensure_capacity(paddi_ctx *ctx, size_t n)
{
    if (n <= ctx->cap_n) return PADDI_OK;
    CK(cudaSetDevice(ctx->device));
    CK(cudaStreamSynchronize(ctx->st));
    free_buffers(ctx);
    const size_t W = n + PADDI_PAD_WIN + 64; // windows (upper bound) incl. the zeroed tail
    CK(dmalloc(ctx, &ctx->d_x, sizeof(float) * (n + 64)));
    CK(dmalloc(ctx, &ctx->d_wst, sizeof(float4) * W));
    CK(dmalloc(ctx, &ctx->d_mu, sizeof(float) * W));
    CK(dmalloc(ctx, &ctx->d_ms64, sizeof(double2) * W));
    CK(dmalloc(ctx, &ctx->d_flat, W));
    CK(dmalloc(ctx, &ctx->d_alive, W));
    CK(dmalloc(ctx, &ctx->d_pruned, W));
    CK(dmalloc(ctx, &ctx->d_cand, sizeof(int32_t) * W));
    CK(dmalloc(ctx, &ctx->d_rcslot, sizeof(int32_t) * W));
    CK(dmalloc(ctx, &ctx->d_rho, sizeof(uint32_t) * W));
    CK(dmalloc(ctx, &ctx->d_list[0], sizeof(int32_t) * W));
    CK(dmalloc(ctx, &ctx->d_list[1], sizeof(int32_t) * W));
    CK(dmalloc(ctx, &ctx->d_frag, sizeof(int32_t) * W));
    if (ctx->umma_ok) {
        const int64_t blocks = paddi_tile_blocks((int64_t)n);
        CK(dmalloc(ctx, &ctx->d_bq, sizeof(uint16_t) * (size_t)(blocks * paddi_tile_block_elems_max())));
        CK(dmalloc(ctx, &ctx->d_wdq, sizeof(float4) * (size_t)(blocks * paddi_tile_wd_entries())));
    }
    CK(set_recheck_cap(ctx, PADDI_MAX_RECHECK));
    if (ctx->umma_ok) {
        // a row of block maxima for 2048 candidates of a long series, and for all
        // that an attempt commonly leaves of a short one; without memory for them
        // the recheck scans the whole series
        const int64_t blocks = paddi_tile_blocks((int64_t)n);
        ctx->bmax_cap = std::min<int64_t>((int64_t)n * 2 * blocks,
                                          std::max<int64_t>(2 * (int64_t)W, 1 << 21));
        if (dmalloc(ctx, &ctx->d_bmax, sizeof(uint32_t) * (size_t)ctx->bmax_cap) != cudaSuccess)
            ctx->bmax_cap = 0;
    }
    CK(cudaMemsetAsync(ctx->d_wst, 0, sizeof(float4) * W, ctx->st));
    CK(cudaMemsetAsync(ctx->d_mu, 0, sizeof(float) * W, ctx->st));
    ctx->cap_n = n;
    return PADDI_OK;
}

float ms_between(unsigned long long a, unsigned long long b)
{
    return a && b > a ? (float)((double)(b - a) * 1e-6) : 0.f;
}

struct AttemptOut {
    PaddiAttemptResult res;
    float ms_stats = 0, ms_guide = 0; // the preparation of the length
    float ms_phase1 = 0, ms_refine = 0, ms_select = 0, ms_total = 0;
    float ms_refine_kernel = 0; // the refine launches alone
    int launches = 0;
    int kernel = PADDI_DIST_FP32;
    int p1_rows = 0; // rows per phase-1 task
};

// Refine kernel for length m: the tensor-core split where the length fits
// its shared-memory budget, else FP32 CUDA cores.
int refine_kernel_for(const paddi_ctx *ctx, int m)
{
    const int k = ctx->opts.distance_kernel;
    if (k == PADDI_DIST_FP32 || !ctx->umma_ok || m > paddi_umma_max_m()) return PADDI_DIST_FP32;
    return k == PADDI_DIST_SPLIT_BF16 ? PADDI_DIST_SPLIT_BF16 : PADDI_DIST_SPLIT_FP16;
}

// The message of a refine that gave up on a wait.
std::string refine_timeout(int kernel, int m)
{
    return std::string(kernel == PADDI_DIST_FP32 ? "FP32 refine" : "tensor-core refine") +
           ": a barrier wait timed out (m=" + std::to_string(m) + ")";
}

// Guard band, in correlation units: the largest per-window rounding bound a
// bounded refine kernel accepts, and the half-width of the FP64 recheck band.
float guard_of(const paddi_ctx *ctx, int kernel)
{
    if (ctx->opts.guard > 0.f) return ctx->opts.guard;
    // the largest per-window rounding bound the bounded kernels accept (above it
    // a window is fragile and goes to the FP64 pass), and the band of the FP64
    // recheck: 2e-4 balances the two on the headline series (1e-4 left 35k
    // fragile windows per attempt, 4e-4 doubled the rechecks)
    return kernel == PADDI_DIST_SPLIT_BF16 ? 1e-3f : 2e-4f;
}

// Statistics of length m for the series in `x` (n values) and the refine's
// per-length data: its tiles (tensor cores) and the windows whose rounding
// bound exceeds the guard band (both refine kernels).  chained: the stream's
// previous operation is a kernel of this context.
paddi_status run_stats(paddi_ctx *ctx, const float *x, size_t n, int m, bool chained = false)
{
    const int cur = ctx->d_flatcount == ctx->d_flat2[0] ? 1 : 0;
    ctx->d_flatcount = ctx->d_flat2[cur];
    ctx->alive_used = false;
    PaddiStatsExtra ex;
    ex.alive = ctx->d_alive;
    ex.next = ctx->d_flat2[cur ^ 1];
    ex.guide = ctx->d_guide;
    ex.t = ctx->d_tprep + PADDI_T_STATS_B;
    unsigned long long *t_end = ctx->d_tprep + PADDI_T_STATS_E;
    const int kernel = refine_kernel_for(ctx, m);
    const float guard = guard_of(ctx, kernel);
    if (kernel != PADDI_DIST_FP32) {
        CK(paddi_launch_prep(kernel == PADDI_DIST_SPLIT_BF16, x, (int64_t)n, m, ctx->d_wst,
                             ctx->d_mu, ctx->d_ms64, ctx->d_flat, ctx->d_flatcount, ctx->d_bq,
                             ctx->d_wdq, guard, ctx->d_frag, ctx->st, chained, ex, t_end));
        ctx->prep_launches = 1;
    } else {
        CK(paddi_launch_stats(x, (int64_t)n, m, ctx->d_wst, ctx->d_mu, ctx->d_ms64, ctx->d_flat,
                              ctx->d_flatcount, ctx->st, ctx->d_flatcount + 1, chained, ex));
        CK(paddi_launch_fragile_scan_fp32(x, ctx->d_wst, ctx->d_mu, (int32_t)(n - m + 1), m, guard,
                                          ctx->d_frag, ctx->d_flatcount + 3, ctx->num_sms, ctx->st,
                                          t_end));
        ctx->prep_launches = 2;
    }
    return PADDI_OK;
}

// Starts a run's witnesses: no window has one.  Without memory for them (16 bytes a
// window) the run goes on without (wit_m stays 0): every attempt then runs phase 1.
paddi_status start_witness(paddi_ctx *ctx, const float *x, size_t n, int m0)
{
    const size_t W = ctx->cap_n + PADDI_PAD_WIN + 64;
    ctx->wit = {m0, 0, 0.0};
    if (ctx->W_cap < W) {
        free_witness(ctx);
        const size_t Wa = (W + 63) & ~(size_t)63; // 256-byte steps
        if (dmalloc(ctx, &ctx->W_mem, 16 * Wa + 256) != cudaSuccess) return PADDI_OK;
        ctx->W.wc = (double *)ctx->W_mem;
        ctx->W.wit = (int32_t *)(ctx->W.wc + Wa);
        ctx->W.wrho = (float *)(ctx->W.wit + Wa);
        ctx->W.scal = (uint32_t *)(ctx->W.wrho + Wa);
        ctx->W_cap = W;
    }
    CK(paddi_launch_witness_start(x, (int64_t)n, (int32_t)(n - m0 + 1), ctx->W, ctx->num_sms,
                                  ctx->st));
    ctx->wit_m = m0;
    ctx->wit_edge = ctx->wit_steps = 0;
    return PADDI_OK;
}

// Advances the run's witnesses to length m, whose statistics are current.
paddi_status witness_to(paddi_ctx *ctx, const float *x, size_t n, int m)
{
    if (ctx->wit_m == 0 || ctx->wit_m == m) return PADDI_OK;
    const int edge = std::min(ctx->wit_m, m);
    if (edge != ctx->wit_edge) {
        ctx->wit_edge = edge;
        ctx->wit_steps = 0;
    }
    ctx->wit.steps2 += 2.0 * ctx->wit_steps + 1.0; // (c + 1)^2 - c^2
    ++ctx->wit_steps;
    ctx->wit.returns = ctx->wit_steps / 2; // forward, back, forward, ...
    CK(paddi_launch_witness_step(x, ctx->d_ms64, (int32_t)(n - m + 1), m, ctx->wit_m, ctx->wit,
                                 ctx->W, ctx->d_list[1], ctx->num_sms, ctx->st,
                                 ctx->d_tprep + PADDI_T_STATS_E));
    ctx->prep_launches += 2;
    ctx->wit_m = m;
    return PADDI_OK;
}

// Queues the statistics of length m and the bound (see the definition).
// known_w >= 0 (in the attempt functions): window whose exact FP64 nn at this
// length is already known (its ordered image known_ord, from the guide
// kernel); the recheck skips it.
paddi_status enqueue_prep(paddi_ctx *ctx, const float *x, size_t n, int m, bool guided,
                          int32_t w_host, bool chained);

// Phase-1 rows per task for `rows` rows: at most the segment length (the
// reference's SEGMENT_N; validated at the ABI, rounded up to a multiple of 8),
// and few enough to give every resident warp of the GPU a task.  Both attempts
// of a PD3 search, phase 1 only, us (the segment length alone decided before):
//   n = 131072, m = 128: 64 rows 118, 128 135, 256 186, 4096 1582
//   n = 131072, m = 600: 64 rows 237, 128 224, 256 241 (start dot products: m per
//                        diagonal and task)
//   n = 600000, m = 500: 64 rows 587, 128 461, 256 473
//   n = 1500007, m = 300: 128 rows 737, 192 715, 256 726, 1024 1580
int p1_rows_of(const paddi_ctx *ctx, int64_t rows, int m)
{
    int R = (int)ctx->opts.segment_len;
    if (R <= 0) R = 256;
    R = (R + 7) & ~7;
    // one-warp tasks that are resident at once: 15 a SM at 256 rows and m = 300 (the
    // launcher asks for the occupancy of the rows chosen here)
    const int64_t tasks = 15ll * ctx->num_sms;
    const int fit = rows <= 64 * tasks && m <= 256 ? 64 : rows <= 512 * tasks ? 128 : 512;
    return std::min(R, fit);
}

// Windows without a proving witness: up to wit_limit of them look for a new
// one, one warp each; phase 1 runs when more than wit_enough are left.
int32_t wit_limit(int32_t N) { return std::max(4096, N / 16); }
int32_t wit_enough(int32_t N) { return std::max(1024, N / 512); }

// The correlation threshold of r^2 at length m: d < r^2 <=> rho > thr.
float thr_of(float r2, int m) { return (float)(1.0 - (double)r2 / (2.0 * (double)m)); }

// The refine's block maxima for N windows, or none: the FP32 refine keeps none,
// nor does a refine of a part of the windows.
PaddiBlockMax block_max(const paddi_ctx *ctx, int kernel, int32_t N, bool whole)
{
    PaddiBlockMax B = {};
    if (kernel != PADDI_DIST_FP32 && whole && ctx->d_bmax) {
        B.v = ctx->d_bmax;
        B.cap = ctx->bmax_cap;
        B.halves = 2 * (int32_t)paddi_tile_blocks(N);
    }
    return B;
}

// Refine of the compacted candidates against the windows [col_lo, col_hi)
// (col_lo on the refine's grid), then the FP64 pass over the fragile windows of
// that range.  It runs in rounds over growing window ranges (1/16, 1/4, 1/2,
// all of the range; a sweep of 4 to 8 rounds picked 4); survivors are
// re-compacted between rounds so every tile is dense with live candidates.
paddi_status refine_rounds(paddi_ctx *ctx, const float *x, int32_t N, int m, int kernel,
                           float thr, float guard, int32_t col_lo, int32_t col_hi, int *launches)
{
    cudaStream_t st = ctx->st;
    const PaddiWitness *W = ctx->wit_m == m ? &ctx->W : nullptr;
    const PaddiBlockMax B = block_max(ctx, kernel, N, col_lo == 0 && col_hi == N);
    if (kernel != PADDI_DIST_FP32)
        CK(paddi_launch_refine_umma(kernel == PADDI_DIST_SPLIT_BF16, x, ctx->d_wst, ctx->d_mu,
                                    ctx->d_cand, ctx->d_list[0], ctx->d_list[1], ctx->d_bq,
                                    ctx->d_wdq, ctx->d_att, ctx->d_rho, ctx->d_pruned, N, m,
                                    col_lo, col_hi, thr, ctx->num_sms, st, ctx->wait_cycles,
                                    ctx->withhold, ctx->opts.tile_rows == 64, W, &B, guard));
    else
        CK(paddi_launch_refine_fp32(x, ctx->d_wst, ctx->d_mu, ctx->d_cand, ctx->d_list[0],
                                    ctx->d_list[1], ctx->d_att, ctx->d_rho, ctx->d_pruned, N, m,
                                    col_lo, col_hi, thr, guard, ctx->num_sms, st,
                                    ctx->wait_cycles, W));
    ++*launches;
    // the fragile windows (skipped by the refine: their rounding bound exceeds
    // the guard band) against the candidates of the last round's list that are
    // still unpruned, in FP64 (the kernel returns at once when there are none)
    CK(paddi_launch_fragile(x, ctx->d_ms64, ctx->d_cand, ctx->d_list[0], ctx->d_list[1],
                            ctx->d_att, ctx->d_pruned, ctx->d_rho, ctx->d_frag,
                            ctx->d_flatcount + 3, m, thr, col_lo, col_hi, ctx->num_sms, st, &B,
                            guard));
    *launches += 1;
    return PADDI_OK;
}

// Classification, FP64 recheck and top-k selection of the refined
// candidates, redone (at most 6 passes) when the recheck queue overflows or a
// pick lacks an exact value.  kept: the refine has stored block maxima.
// next_m > 0: the statistics (and, with next_guided, the bound) of length next_m
// are queued behind the first pass, before its result is synced; *spec tells
// whether they were.
paddi_status select_passes(paddi_ctx *ctx, const float *x, size_t n, int m, float r2,
                           float guard, bool kept, int top_k, int32_t known_w,
                           unsigned long long known_ord, int next_m, bool next_guided,
                           bool *spec, int *launches)
{
    const int32_t N = (int32_t)(n - m + 1);
    const float thr = thr_of(r2, m);
    cudaStream_t st = ctx->st;
    *spec = false;
    float widen = 2.f;
    const int kernel = refine_kernel_for(ctx, m);
    for (int pass = 0; pass < 6; ++pass) {
        // (a pass that grew the recheck queue may have given up the block maxima)
        const PaddiBlockMax B = block_max(ctx, kernel, N, kept);
        CK(paddi_launch_finalize(ctx->d_cand, ctx->d_att, ctx->d_rho, ctx->d_pruned, m, r2, thr,
                                 guard, widen, top_k, ctx->d_flat, ctx->rc_cap, ctx->d_recheck,
                                 ctx->d_rcslot, ctx->d_nn64, ctx->d_res, known_w, known_ord, st));
        CK(paddi_launch_recheck(x, ctx->d_ms64, ctx->d_flat, N, m, ctx->d_cand,
                                ctx->d_recheck, ctx->d_att, ctx->d_nn64, ctx->num_sms, known_w,
                                st, ctx->d_rho, &B, guard));
        CK(paddi_launch_select(ctx->d_cand, ctx->d_att, ctx->d_rho, ctx->d_pruned,
                               ctx->d_recheck, ctx->d_rcslot, ctx->d_nn64, m, r2, thr, guard,
                               top_k, ctx->d_flat, ctx->d_flatcount, ctx->d_tprep,
                               ctx->d_att2[ctx->d_att == ctx->d_att2[0]], ctx->d_res, ctx->h_res,
                               st));
        *launches += 3;
        if (ctx->trace)
            CK(cudaMemcpyAsync(ctx->h_trace, ctx->d_att, sizeof(PaddiAttemptDev),
                               cudaMemcpyDeviceToHost, st));
        if (pass == 0 && next_m > 0) {
            paddi_status s = enqueue_prep(ctx, x, n, next_m, next_guided, -1, !ctx->trace);
            if (s != PADDI_OK) return s;
            *spec = true;
        }
        CK(cudaStreamSynchronize(st));
        ctx->att_dirty = false;
        ctx->last_passes = pass + 1;
        if (ctx->h_res->status == 3) // a refine wait ran out: no redo can help
            return fail(ctx, PADDI_ERR_CUDA, refine_timeout(kernel, m));
        if (ctx->h_res->status == 1) {
            // more windows need the exact value than the queue holds: grow it and redo
            int32_t cap = ctx->rc_cap;
            while (cap < ctx->h_res->n_recheck) cap *= 2;
            CK(set_recheck_cap(ctx, cap));
        } else if (ctx->h_res->status == 2) {
            // a pick had no exact value: queue everything up to the cut and redo
            widen = 1e30f;
        } else {
            break;
        }
        if (*spec) { // the redo needs this length's statistics back
            paddi_status s = run_stats(ctx, x, n, m);
            if (s != PADDI_OK) return s;
            *spec = false;
        }
        CK(cudaMemsetAsync(&ctx->d_att->recheck_next, 0, sizeof(int32_t), st));
        CK(cudaMemsetAsync(&ctx->d_att->status, 0, sizeof(int32_t), st));
    }
    if (ctx->h_res->status == 1)
        return fail(ctx, PADDI_ERR_INTERNAL_LIMIT,
                    "more windows than the FP64 recheck capacity fall inside the guard band (m=" +
                        std::to_string(m) + ", r2=" + std::to_string(r2) +
                        ", phase-1 candidates=" + std::to_string(ctx->h_res->n_p1) +
                        ", certain=" + std::to_string(ctx->h_res->n_cand) +
                        ", queued>=" + std::to_string(ctx->h_res->n_recheck) +
                        ", widen=" + std::to_string(widen) + ")");
    if (ctx->h_res->status != 0)
        return fail(ctx, PADDI_ERR_INTERNAL_LIMIT, "top-k selection did not settle");
    return PADDI_OK;
}

// One (m, r2) attempt on the statistics currently in the context.
// next_m > 0: the statistics (and, with next_guided, the bound) of length
// next_m are queued behind the attempt, before its result is synced, so the
// host waits once per length; *spec_out then tells whether the statistics
// now hold next_m (not when the selection had to be redone).
paddi_status run_attempt(paddi_ctx *ctx, const float *x, size_t n, int m, float r2, int top_k,
                         AttemptOut *out, int32_t known_w = -1, unsigned long long known_ord = 0,
                         int next_m = 0, bool next_guided = false, bool *spec_out = nullptr)
{
    const int32_t N = (int32_t)(n - m + 1);
    const int kernel = refine_kernel_for(ctx, m);
    const float guard = guard_of(ctx, kernel);
    const float thr = thr_of(r2, m);
    const int R = p1_rows_of(ctx, N, m);
    const int chunks = ctx->opts.phase1_chunks ? (int)ctx->opts.phase1_chunks : 12;
    cudaStream_t st = ctx->st;
    // the attempt's state and the alive flags are clean: the previous attempt's
    // selection, the statistics and the compaction leave them so
    ctx->d_att = ctx->d_att2[ctx->d_att == ctx->d_att2[0]];
    if (ctx->att_dirty) CK(cudaMemsetAsync(ctx->d_att, 0, sizeof(PaddiAttemptDev), st));
    ctx->att_dirty = true;
    int launches = 0;
    const bool wit = ctx->wit_m == m;
    if (!wit && ctx->alive_used) // the witnesses were given up since the last attempt
        CK(cudaMemsetAsync(ctx->d_alive, 1, (size_t)N, st));
    ctx->alive_used = wit;
    if (wit) {
        CK(paddi_launch_witness_check(ctx->d_ms64, x, N, m, thr, ctx->wit, ctx->W,
                                      ctx->d_alive, ctx->d_list[0], ctx->d_att, wit_limit(N),
                                      ctx->num_sms, st));
        launches += 2;
    }
    CK(paddi_launch_phase1_dev(x, ctx->d_wst, ctx->d_mu, ctx->d_ms64, ctx->d_alive, N, m, R,
                               chunks, thr, 0, N, ctx->d_att, ctx->num_sms, st,
                               wit ? &ctx->W : nullptr, wit_enough(N)));
    ++launches;
    CK(paddi_launch_compact(ctx->d_alive, !wit, N, ctx->d_cand, ctx->d_rho, ctx->d_pruned,
                            ctx->d_rcslot, ctx->d_att, ctx->d_flat, ctx->d_flatcount + 1, m,
                            r2 > 0.f, thr >= 0.f, st));
    ++launches;
    out->kernel = kernel;
    out->p1_rows = R;
    paddi_status s = refine_rounds(ctx, x, N, m, kernel, thr, guard, 0, N, &launches);
    if (s != PADDI_OK) return s;
    bool spec = false;
    s = select_passes(ctx, x, n, m, r2, guard, true, top_k, known_w, known_ord, next_m,
                      next_guided, &spec, &launches);
    if (s != PADDI_OK) return s;
    out->res = *ctx->h_res;
    out->launches = launches;
    if (spec_out) *spec_out = spec;
    const unsigned long long *T = out->res.t, *P = out->res.t_prep;
    out->ms_stats = ms_between(P[PADDI_T_STATS_B], P[PADDI_T_STATS_E]);
    out->ms_guide = ms_between(P[PADDI_T_GUIDE_B], P[PADDI_T_GUIDE_E]);
    out->ms_phase1 = ms_between(T[PADDI_T_BEGIN], T[PADDI_T_COMPACT]);
    out->ms_refine = ms_between(T[PADDI_T_COMPACT], T[PADDI_T_SELECT]);
    out->ms_refine_kernel = ms_between(T[PADDI_T_REFINE_B], T[PADDI_T_REFINE_E]);
    out->ms_select = ms_between(T[PADDI_T_SELECT], T[PADDI_T_END]);
    out->ms_total = ms_between(T[PADDI_T_BEGIN], T[PADDI_T_END]);
    if (ctx->trace) {
        const PaddiAttemptDev &t = *ctx->h_trace;
        const float fms = ms_between(T[PADDI_T_FRAGILE], T[PADDI_T_SELECT]);
        std::fprintf(stderr,
                     "paddi-trace m=%d r2=%f unproven=%d-%d p1=%d p1_tasks=%dx%d/%f "
                     "rounds: %d %d %d %d/%f fragile=%d/%f recheck=%d disc=%lld pairs=%llu live=%llu\n",
                     m, r2, t.n_fail, t.n_rescued, t.n_cand_p1, t.p1_walked, R, out->ms_phase1,
                     t.n_cand_p1, t.list_count[1], t.list_count[2], t.list_count[3],
                     out->ms_refine_kernel, ctx->h_res->n_fragile, fms, ctx->h_res->n_recheck,
                     (long long)ctx->h_res->n_disc, t.n_pairs, t.n_live);
    }
    return PADDI_OK;
}

void fill_log(paddi_attempt_log *L, int m, float r, float r2, int top_k, const AttemptOut &a,
              float ms_stats)
{
    std::memset(L, 0, sizeof(*L));
    L->m = m;
    L->r = r;
    L->r2 = r2;
    L->n_cand = a.res.n_cand;
    L->n_disc = a.res.n_disc;
    L->n_phase1 = a.res.n_p1;
    L->n_recheck = a.res.n_recheck;
    L->found = a.res.n_sel >= top_k && a.res.n_sel > 0;
    if (a.res.n_sel > 0) {
        L->top.ind = a.res.sel_ind[0];
        L->top.dist = a.res.sel_dist[0];
    } else {
        L->top.ind = -1;
        L->top.dist = -FLT_MAX;
    }
    L->ms_stats = ms_stats;
    L->ms_phase1 = a.ms_phase1;
    L->ms_refine = a.ms_refine;
    L->ms_select = a.ms_select;
    L->ms_total = a.ms_total + ms_stats;
    L->refine_pairs = (int64_t)a.res.n_pairs;
    L->refine_live_pairs = (int64_t)a.res.n_live;
    L->p1_pairs = (int64_t)a.res.p1_walked * (int64_t)a.p1_rows * 256;
    L->ms_refine_kernel = a.ms_refine_kernel;
    L->n_fragile = a.res.n_fragile;
    L->n_launches = a.launches;
    L->refine_kernel = a.kernel;
    L->r_source = 0;
    L->ms_guide = 0.f;
}

// Phase-1 segment lengths this build runs: 0 (default 256) or 64..4096 rows.
// The reference caps SEGMENT_N at its 1024-thread block (src/PD3.cuh:20); here
// a segment is a task of one warp, so longer segments only cost occupancy.
bool segment_len_ok(uint32_t seg) { return seg == 0 || (seg >= 64 && seg <= 4096); }

bool valid_lengths(size_t n, uint32_t minL, uint32_t maxL)
{
    return minL >= 3 && maxL >= minL && maxL <= 1024 && n >= 2 * (size_t)maxL &&
           n < (size_t)INT32_MAX - PADDI_PAD_WIN - 64;
}

// What is known about one length before its first attempt: its flat-window
// count and, for the guided r policies, the exact FP64 nn of the bound window
// (the previous length's top-1 window).
struct Prep {
    int m = 0;                        // length prepared (0: none)
    int32_t flatcount = 0;
    int32_t known_w = -1;             // bound window with a finite exact nn (-1: none)
    unsigned long long known_ord = 0; // its ordered image
    double lb = 0.0;                  // its nn
};

// Queues the statistics of length m and, with `guided`, the bound window's
// exact nn (window w_host; w_host < 0: the top-1 window of the attempt result
// on the device, so this can be queued before the host has read it).  No
// sync: read_prep collects the values after the next one.
paddi_status enqueue_prep(paddi_ctx *ctx, const float *x, size_t n, int m, bool guided,
                          int32_t w_host, bool chained)
{
    paddi_status s = run_stats(ctx, x, n, m, chained);
    if (s != PADDI_OK) return s;
    s = witness_to(ctx, x, n, m);
    if (s != PADDI_OK) return s;
    if (guided) {
        CK(paddi_launch_guide(x, ctx->d_ms64, ctx->d_flat, (int32_t)(n - m + 1), m, ctx->d_res,
                              w_host, ctx->d_guide, ctx->d_G, ctx->G_cap, ctx->num_sms, ctx->st,
                              ctx->h_guide, ctx->d_flatcount, ctx->d_tprep));
        ctx->prep_launches += 2;
    }
    return PADDI_OK;
}

// After a sync that covers enqueue_prep(m, guided = true).
void read_prep(paddi_ctx *ctx, int m, Prep *p)
{
    *p = Prep();
    p->m = m;
    p->flatcount = ctx->h_guide->n_flat;
    const unsigned long long u = ctx->h_guide->nn_ord;
    const unsigned long long bits = (u & 0x8000000000000000ull) ? (u & 0x7fffffffffffffffull) : ~u;
    double d;
    std::memcpy(&d, &bits, sizeof(d));
    if (ctx->h_guide->w_used >= 0 && std::isfinite(d)) {
        p->known_w = ctx->h_guide->w_used;
        p->known_ord = u;
        p->lb = d;
    }
    if (ctx->trace)
        std::fprintf(stderr, "paddi-guide m=%d w=%d mode=%d\n", m, ctx->h_guide->w_used,
                     ctx->h_guide->mode);
}

// MERLIN's first r for length minL + j (src/main.cu:38, 171, 202-214): a pure
// function of the previous top-1 distances; S is the decrement of :230.
float merlin_first_r(const paddi_discord *out, int j, uint32_t minL, float *S_out)
{
    float S = 0.f, r;
    if (j == 0) {
        r = (float)(2.0 * std::sqrt((double)minL)); // sqrt of an unsigned int: double
    } else if (j < 5) {
        r = (float)((double)std::sqrt(out[j - 1].dist) * 0.99); // :171
    } else {
        float M = 0.f;
        for (int k = j - 5; k < j; ++k) M += std::sqrt(out[k].dist); // :205-206
        M = (float)((double)M * 0.2);                               // :208
        for (int k = j - 5; k < j; ++k)
            S = (float)((double)S + std::pow((double)(std::sqrt(out[k].dist) - M), 2.0));
        S = (float)std::sqrt((double)S * 0.2); // :213
        r = M - 2 * S;                         // :214
    }
    if (S_out) *S_out = S;
    return r;
}

// MERLIN's lowering of r after an attempt without discords (:155, :187, :230).
float merlin_lower(float r, int j, float S)
{
    if (j == 0) return (float)(0.5 * (double)r);
    if (j < 5) return (float)(0.99 * (double)r);
    return r - S;
}

// Largest float r with r*r < v (v > 0).
float r_below(float v)
{
    float r = std::sqrt(v);
    while (r > 0.f && r * r >= v) r = std::nextafter(r, 0.f);
    return r;
}

void r_features_impl(const paddi_discord *out, int j, uint32_t minL, float lb, float flat_frac,
                     int prev_attempts, float *f)
{
    const int m = (int)minL + j;
    auto d = [&](int k) { return (double)std::fmax(out[k].dist, 1e-6f); };
    auto lr = [&](int a, int b) { return (float)std::log(d(a) / d(b)); };
    for (int k = 0; k < MLP_NFEAT; ++k) f[k] = 0.f;
    f[0] = (float)m / 1024.f;
    if (j >= 1) f[1] = (float)std::log(d(j - 1) / (2.0 * m));
    if (j >= 2) f[2] = lr(j - 1, j - 2);
    if (j >= 3) f[3] = lr(j - 2, j - 3);
    if (j >= 4) f[4] = lr(j - 3, j - 4);
    if (j >= 1 && lb > 0.f) f[5] = (float)std::log((double)lb / d(j - 1));
    if (j >= 2) f[6] = out[j - 1].ind != out[j - 2].ind ? 1.f : 0.f;
    f[7] = (float)std::min(std::max(prev_attempts - 1, 0), 10) / 10.f;
    if (j >= 1) {
        float S = 0.f;
        const float r0 = merlin_first_r(out, j, minL, &S);
        f[8] = (float)std::log(std::fmax((double)r0 * r0, 1e-6) / d(j - 1));
        if (j >= 5) f[10] = (float)std::log(std::fmax((double)S, 1e-6) / std::fmax((double)std::fabs(r0) + 2.0 * S, 1e-6));
    }
    f[9] = flat_frac;
    if (j >= 5) f[11] = 0.25f * lr(j - 1, j - 5);
}

// Prediction of the learned model for one feature vector (BF16 weights).
paddi_status model_predict1(paddi_ctx *ctx, const float *f, float *y)
{
    std::memcpy(ctx->h_feat, f, sizeof(float) * MLP_NFEAT);
    CK(cudaMemcpyAsync(ctx->d_feat, ctx->h_feat, sizeof(float) * MLP_NFEAT,
                       cudaMemcpyHostToDevice, ctx->st));
    CK(paddi_launch_mlp_forward(ctx->d_feat, 1, ctx->d_model_bf16, true, ctx->d_pred, ctx->st));
    CK(cudaMemcpyAsync(ctx->h_feat + MLP_NFEAT, ctx->d_pred, sizeof(float),
                       cudaMemcpyDeviceToHost, ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
    *y = ctx->h_feat[MLP_NFEAT];
    return PADDI_OK;
}

// PALMAD on a series already on the device.
// Range-discord profile of the length's final attempt into prof (host, N
// entries): the nnDist layout of paddi_do_pd3.
paddi_status attempt_profile(paddi_ctx *ctx, int m, int32_t N, float r2, std::vector<float> &prof)
{
    if (!ctx->d_pc) {
        const size_t W = ctx->cap_n + PADDI_PAD_WIN + 64;
        CK(dmalloc(ctx, &ctx->d_pc, sizeof(int32_t) * W));
        CK(dmalloc(ctx, &ctx->d_pn, sizeof(float) * W));
    }
    CK(paddi_launch_scatter(ctx->d_cand, ctx->d_att, ctx->d_rho, ctx->d_pruned, ctx->d_rcslot,
                            ctx->d_nn64, ctx->d_flat, N, m, r2, ctx->d_pc, ctx->d_pn, ctx->st));
    prof.resize((size_t)N);
    CK(cudaMemcpyAsync(prof.data(), ctx->d_pn, sizeof(float) * (size_t)N, cudaMemcpyDeviceToHost,
                       ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
    return PADDI_OK;
}

paddi_status palmad_impl(paddi_ctx *ctx, const float *x, size_t n, uint32_t minL, uint32_t maxL,
                         paddi_discord *out, paddi_attempt_log *log, uint32_t log_cap,
                         uint32_t *n_log, paddi_profile_fn prof_fn = nullptr,
                         void *prof_user = nullptr)
{
    std::vector<float> prof;
    const int L = (int)(maxL - minL + 1);
    const int iter_cap = ctx->opts.iter_cap ? (int)ctx->opts.iter_cap : 200;
    const int policy = ctx->opts.r_policy;
    if (policy == PADDI_R_LEARNED && !ctx->model_ok)
        return fail(ctx, PADDI_ERR_INVALID_ARG, "r_policy LEARNED needs paddi_model_set first");
    const bool want_lb = policy != PADDI_R_MERLIN || (ctx->opts.flags & PADDI_FLAG_LOG_BOUND);
    uint32_t nl = 0;
    for (int j = 0; j < L; ++j) {
        out[j].ind = -1;
        out[j].dist = -FLT_MAX;
    }
    int prev_attempts = 0;
    const bool guided = want_lb || policy == PADDI_R_LEARNED;
    // with the profile callback every length's statistics must stay current
    // until its profile is written: no statistics are queued ahead then
    const bool ahead = guided && !prof_fn;
    if (guided) {
        const size_t W = ctx->cap_n + PADDI_PAD_WIN + 64;
        if (ctx->G_cap < W) {
            dfree(ctx->d_G);
            ctx->G_cap = 0;
            CK(dmalloc(ctx, &ctx->d_G, sizeof(double) * 2 * W)); // two buffers
            ctx->G_cap = W;
        }
        // the dot products of an earlier call belong to another series
        CK(cudaMemsetAsync(ctx->d_guide, 0, sizeof(PaddiGuide), ctx->st));
    }
    // one length: nothing to carry over
    struct EndWitness {
        paddi_ctx *c;
        ~EndWitness() { c->wit_m = 0; }
    } end_witness{ctx};
    if (L > 1) {
        paddi_status s = start_witness(ctx, x, n, (int)minL);
        if (s != PADDI_OK) return s;
    }
    Prep pre; // the length whose statistics (and bound) are current, if queued ahead
    for (int j = 0; j < L; ++j) {
        const int m = (int)minL + j;
        const int32_t N = (int32_t)(n - m + 1);
        paddi_status s;
        // ---- statistics and the bound: queued ahead by the previous length's
        //      last attempt, or here (the previous length's top-1 window,
        //      evaluated exactly at this length: its nn is a lower bound on
        //      this length's top-1 distance)
        const bool g_here = guided && j >= 1 && out[j - 1].ind >= 0;
        if (pre.m != m) {
            const int32_t w = g_here ? (out[j - 1].ind < N ? out[j - 1].ind : N - 1) : -1;
            s = enqueue_prep(ctx, x, n, m, g_here, w, false);
            if (s != PADDI_OK) return s;
            if (g_here) {
                CK(cudaStreamSynchronize(ctx->st));
                read_prep(ctx, m, &pre);
            } else {
                pre = Prep(); // nothing is known before the first attempt
            }
        }
        const int prep_launches = ctx->prep_launches;
        Prep cur = pre; // the next length's values may replace pre during the attempts
        pre.m = 0;
        float S = 0.f;
        float r = merlin_first_r(out, j, minL, &S);
        // ---- guidance: the bound and / or the model's prediction
        float lbf = 0.f, lbm = 0.f; // lbm: largest r^2 below the bound
        int source = 0;
        if (cur.known_w >= 0 && cur.lb > 0.0) {
            lbf = (float)std::fmin(cur.lb, (double)FLT_MAX);
            const float rb = r_below(lbf);
            lbm = rb * rb;
        }
        const float flat_frac = (float)cur.flatcount / (float)N;
        if (policy == PADDI_R_BOUND && lbm > 0.f && lbm > r * r) {
            // tighter than MERLIN's first r and certain to find a discord (a window
            // that was flat at m-1 may have a small nn at m: then MERLIN leads)
            r = r_below(lbf);
            source = 2;
        } else if (policy == PADDI_R_LEARNED && j >= 1 && lbm > 0.f && lbm > r * r) {
            // the bound beats MERLIN's first r: start just below it (certain to find a
            // discord, and exact whenever the previous top window stays on top, which
            // is the common case); the model is for the lengths where it is weak
            r = r_below(lbf);
            source = 2;
        } else if (policy == PADDI_R_LEARNED && j >= 1) {
            float f[MLP_NFEAT];
            r_features_impl(out, j, minL, lbf, flat_frac, prev_attempts, f);
            float y = 0.f;
            s = model_predict1(ctx, f, &y);
            if (s != PADDI_OK) return s;
            double r2 = (double)std::fmax(out[j - 1].dist, 1e-6f) * std::exp((double)y) *
                        (double)ctx->model_margin;
            if (lbm > 0.f && r2 < (double)lbm) r2 = lbm; // never looser than the bound
            if (std::isfinite(r2) && r2 > 0.0) {
                r = r_below((float)std::fmin(r2 * (1.0 + 1e-7), (double)FLT_MAX));
                if (lbm > 0.f && r * r < lbm) r = r_below(lbf);
                source = 1;
            }
        }
        // ---- attempts
        int it = 0;
        bool first = true;
        bool stale = false; // the statistics hold the next length (queued ahead)
        bool spec = false;
        while (out[j].dist < 0) {
            if (it++ >= iter_cap)
                return fail(ctx, PADDI_ERR_ITER_CAP,
                            "length " + std::to_string(m) + ": no discord after " +
                                std::to_string(iter_cap) + " attempts");
            if (stale) { // a miss after the next length was queued: restore this one
                s = run_stats(ctx, x, n, m);
                if (s == PADDI_OK) s = witness_to(ctx, x, n, m);
                if (s != PADDI_OK) return s;
                stale = false;
            }
            const float r2 = r * r;
            AttemptOut a;
            const int next_m = ahead && j + 1 < L ? m + 1 : 0;
            s = run_attempt(ctx, x, n, m, r2, 1, &a, cur.known_w, cur.known_ord, next_m, guided,
                            &spec);
            if (s != PADDI_OK) return s;
            stale = spec;
            cur.flatcount = a.res.n_flat;
            if (a.res.n_sel > 0) {
                out[j].ind = a.res.sel_ind[0];
                out[j].dist = a.res.sel_dist[0];
            }
            if (log && nl < log_cap) {
                fill_log(&log[nl], m, r, r2, 1, a, first ? a.ms_stats : 0.f);
                log[nl].r_source = source;
                log[nl].lb = lbf;
                log[nl].flat_frac = (float)cur.flatcount / (float)N;
                if (first) {
                    if (g_here) log[nl].ms_guide = a.ms_guide;
                    log[nl].ms_total += log[nl].ms_guide;
                    log[nl].n_launches += prep_launches + (source == 1 ? 1 : 0);
                }
            }
            ++nl;
            first = false;
            if (out[j].dist >= 0) break;
            // no discord: MERLIN lowers r by its own schedule (src/main.cu:216-233).
            // The guided policies lower r^2 by at least 15% (30% from the second
            // miss on): after a sudden drop of the top-1 distance (a flat run that
            // ends) MERLIN's decrement S is tiny and would take dozens of attempts.
            // They never go below the bound, where a discord is certain.
            r = merlin_lower(r, j, S);
            source = 0;
            if (policy != PADDI_R_MERLIN) {
                const float q = it == 1 ? 0.85f : 0.7f;
                const float rg = r2 > 0.f ? r_below(q * r2) : 0.f;
                if (rg < r) r = rg;
                if (lbm > 0.f && r * r < lbm) {
                    r = r_below(lbf);
                    source = 2;
                }
            }
        }
        if (spec) { // the last attempt queued the next length
            read_prep(ctx, m + 1, &pre);
        }
        prev_attempts = it;
        if (prof_fn) {
            s = attempt_profile(ctx, m, N, r * r, prof);
            if (s != PADDI_OK) return s;
            prof_fn(prof_user, (uint32_t)m, prof.data(), (size_t)N);
        }
    }
    if (n_log) *n_log = nl;
    return PADDI_OK;
}

} // namespace

// ====================================================================== ABI
PADDI_API int32_t paddi_abi_version(void) { return PADDI_ABI_VERSION; }

PADDI_API const char *paddi_status_string(paddi_status s)
{
    const int i = (int)s;
    if (i < 0 || i >= (int)(sizeof(kStatusText) / sizeof(kStatusText[0]))) return "unknown status";
    return kStatusText[i];
}

PADDI_API void paddi_opts_default(paddi_opts *o)
{
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->struct_size = sizeof(paddi_opts);
    o->distance_kernel = PADDI_DIST_AUTO;
    o->r_policy = PADDI_R_MERLIN;
    o->segment_len = 256;
    o->phase1_chunks = 12;
    o->iter_cap = 200;
    o->guard = 0.f;
}

PADDI_API paddi_status paddi_ctx_create(paddi_ctx **out, const paddi_opts *opts)
{
    if (!out) return PADDI_ERR_INVALID_ARG;
    *out = nullptr;
    paddi_ctx *ctx = new paddi_ctx();
    paddi_opts_default(&ctx->opts);
    if (opts) {
        if (opts->struct_size != sizeof(paddi_opts)) {
            delete ctx;
            return PADDI_ERR_INVALID_ARG;
        }
        ctx->opts = *opts;
        if (!segment_len_ok(ctx->opts.segment_len) ||
            (ctx->opts.tile_rows != 0 && ctx->opts.tile_rows != 64)) {
            delete ctx;
            return PADDI_ERR_UNSUPPORTED;
        }
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= ctx->opts.device ||
        ctx->opts.device < 0) {
        cudaGetLastError();
        delete ctx;
        return PADDI_ERR_NO_DEVICE;
    }
    ctx->device = ctx->opts.device;
    int major = 0;
    if (cudaSetDevice(ctx->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, ctx->device) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, ctx->device) !=
            cudaSuccess ||
        major < 10) {
        cudaGetLastError();
        delete ctx;
        return PADDI_ERR_NO_DEVICE;
    }
    ctx->umma_ok = paddi_umma_supported(ctx->device);
    if ((ctx->opts.distance_kernel == PADDI_DIST_SPLIT_BF16 ||
         ctx->opts.distance_kernel == PADDI_DIST_SPLIT_FP16) &&
        !ctx->umma_ok) {
        delete ctx;
        return PADDI_ERR_UNSUPPORTED;
    }
    bool ok = cudaStreamCreateWithFlags(&ctx->st, cudaStreamNonBlocking) == cudaSuccess;
    for (auto &e : ctx->ev) ok = ok && cudaEventCreate(&e) == cudaSuccess;
    {
        const char *tr = std::getenv("PADDI_TRACE");
        ctx->trace = tr && tr[0] && tr[0] != '0';
    }
    // small buffers, in one allocation each (256-byte steps), zeroed
    size_t dn = 0, hn = 0;
    auto place = [](size_t &off, size_t bytes) {
        const size_t at = off;
        off += (bytes + 255) & ~(size_t)255;
        return at;
    };
    const size_t o_att[2] = {place(dn, sizeof(PaddiAttemptDev)), place(dn, sizeof(PaddiAttemptDev))};
    const size_t o_flat[2] = {place(dn, 4 * sizeof(int32_t)), place(dn, 4 * sizeof(int32_t))};
    const size_t o_res = place(dn, sizeof(PaddiAttemptResult));
    const size_t o_tp = place(dn, PADDI_T_PREP * sizeof(unsigned long long));
    const size_t o_guide = place(dn, sizeof(PaddiGuide));
    const size_t o_model = place(dn, sizeof(float) * MLP_NPARAM);
    const size_t o_bf16 = place(dn, 2 * MLP_NPARAM);
    const size_t o_feat = place(dn, sizeof(float) * 16), o_pred = place(dn, sizeof(float) * 4);
    const size_t p_res = place(hn, sizeof(PaddiAttemptResult)), p_guide = place(hn, sizeof(PaddiGuide));
    const size_t p_feat = place(hn, sizeof(float) * 16), p_trace = place(hn, sizeof(PaddiAttemptDev));
    ok = ok && cudaMalloc(&ctx->d_small, dn) == cudaSuccess;
    ok = ok && cudaMemset(ctx->d_small, 0, dn) == cudaSuccess;
    ok = ok && cudaMallocHost(&ctx->h_small, hn) == cudaSuccess;
    if (ok) {
        char *d = (char *)ctx->d_small, *h = (char *)ctx->h_small;
        for (int k = 0; k < 2; ++k) {
            ctx->d_att2[k] = (PaddiAttemptDev *)(d + o_att[k]);
            ctx->d_flat2[k] = (int32_t *)(d + o_flat[k]);
        }
        ctx->d_att = ctx->d_att2[0];
        ctx->d_flatcount = ctx->d_flat2[0];
        ctx->d_res = (PaddiAttemptResult *)(d + o_res);
        ctx->d_tprep = (unsigned long long *)(d + o_tp);
        ctx->d_guide = (PaddiGuide *)(d + o_guide);
        ctx->d_model = (float *)(d + o_model);
        ctx->d_model_bf16 = d + o_bf16;
        ctx->d_feat = (float *)(d + o_feat);
        ctx->d_pred = (float *)(d + o_pred);
        ctx->h_res = (PaddiAttemptResult *)(h + p_res);
        ctx->h_guide = (PaddiGuide *)(h + p_guide);
        ctx->h_feat = (float *)(h + p_feat);
        ctx->h_trace = (PaddiAttemptDev *)(h + p_trace);
    }
    if (!ok) {
        cudaGetLastError();
        paddi_ctx_destroy(ctx);
        return PADDI_ERR_CUDA;
    }
    *out = ctx;
    return PADDI_OK;
}

PADDI_API paddi_status paddi_ctx_destroy(paddi_ctx *ctx)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    cudaSetDevice(ctx->device);
    if (ctx->st) cudaStreamSynchronize(ctx->st);
    drop_workers(ctx);
    free_buffers(ctx);
    if (ctx->d_small) cudaFree(ctx->d_small);
    if (ctx->h_small) cudaFreeHost(ctx->h_small);
    for (auto &e : ctx->ev)
        if (e) cudaEventDestroy(e);
    if (ctx->st) cudaStreamDestroy(ctx->st);
    delete ctx;
    return PADDI_OK;
}

PADDI_API const char *paddi_last_error(const paddi_ctx *ctx)
{
    return ctx ? ctx->err.c_str() : "null context";
}

PADDI_API void *paddi_ctx_stream(paddi_ctx *ctx) { return ctx ? (void *)ctx->st : nullptr; }

PADDI_API paddi_status paddi_ctx_reserve(paddi_ctx *ctx, size_t n, uint32_t maxL)
{
    if (!ctx || n < 2 || maxL > 1024) return PADDI_ERR_INVALID_ARG;
    CK(cudaSetDevice(ctx->device));
    return ensure_capacity(ctx, n);
}

PADDI_API paddi_status paddi_palmad_device(paddi_ctx *ctx, const float *d_series, size_t n,
                                           uint32_t minL, uint32_t maxL, paddi_discord *out,
                                           paddi_attempt_log *log, uint32_t log_cap,
                                           uint32_t *n_log)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!d_series || !out || !valid_lengths(n, minL, maxL))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "invalid series, lengths or output pointer");
    if (n_log) *n_log = 0;
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    return palmad_impl(ctx, d_series, n, minL, maxL, out, log, log_cap, n_log);
}

PADDI_API paddi_status paddi_palmad(paddi_ctx *ctx, const float *series, size_t n, uint32_t minL,
                                    uint32_t maxL, paddi_discord *out, paddi_attempt_log *log,
                                    uint32_t log_cap, uint32_t *n_log)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!series || !out || !valid_lengths(n, minL, maxL))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "invalid series, lengths or output pointer");
    if (n_log) *n_log = 0;
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    CK(cudaMemcpyAsync(ctx->d_x, series, sizeof(float) * n, cudaMemcpyHostToDevice, ctx->st));
    return palmad_impl(ctx, ctx->d_x, n, minL, maxL, out, log, log_cap, n_log);
}

PADDI_API paddi_status paddi_palmad_profiled(paddi_ctx *ctx, const float *series, size_t n,
                                             uint32_t minL, uint32_t maxL, paddi_discord *out,
                                             paddi_attempt_log *log, uint32_t log_cap,
                                             uint32_t *n_log, paddi_profile_fn fn, void *user)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!series || !out || !fn || !valid_lengths(n, minL, maxL))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "invalid series, lengths, output or callback");
    if (n_log) *n_log = 0;
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    CK(cudaMemcpyAsync(ctx->d_x, series, sizeof(float) * n, cudaMemcpyHostToDevice, ctx->st));
    return palmad_impl(ctx, ctx->d_x, n, minL, maxL, out, log, log_cap, n_log, fn, user);
}

PADDI_API paddi_status paddi_pd3(paddi_ctx *ctx, const float *series, size_t n, uint32_t m,
                                 uint32_t segment_len, uint32_t top_k, float r,
                                 paddi_discord *out, uint32_t *n_out, paddi_attempt_log *log,
                                 uint32_t log_cap, uint32_t *n_log)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!series || !out || !n_out || top_k < 1 || top_k > PADDI_MAX_TOPK ||
        !valid_lengths(n, m, m))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "invalid series, length, top_k or output");
    if (!segment_len_ok(segment_len))
        return fail(ctx, PADDI_ERR_UNSUPPORTED,
                    "segment_len " + std::to_string(segment_len) + " outside 64..4096");
    *n_out = 0;
    if (n_log) *n_log = 0;
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    const uint32_t saved_seg = ctx->opts.segment_len;
    if (segment_len) ctx->opts.segment_len = segment_len;
    CK(cudaMemcpyAsync(ctx->d_x, series, sizeof(float) * n, cudaMemcpyHostToDevice, ctx->st));
    s = run_stats(ctx, ctx->d_x, n, (int)m);
    if (s != PADDI_OK) {
        ctx->opts.segment_len = saved_seg;
        return s;
    }
    const bool halving = !(r > 0.f);
    float rr = halving ? (float)(2.0 * std::sqrt((double)m)) : r;
    const int iter_cap = ctx->opts.iter_cap ? (int)ctx->opts.iter_cap : 200;
    uint32_t nl = 0;
    AttemptOut a;
    for (int it = 0;; ++it) {
        if (it >= iter_cap) {
            ctx->opts.segment_len = saved_seg;
            return fail(ctx, PADDI_ERR_ITER_CAP, "no discords after the attempt cap");
        }
        const float r2 = rr * rr;
        s = run_attempt(ctx, ctx->d_x, n, (int)m, r2, (int)top_k, &a);
        if (s != PADDI_OK) {
            ctx->opts.segment_len = saved_seg;
            return s;
        }
        if (log && nl < log_cap) {
            fill_log(&log[nl], (int)m, rr, r2, (int)top_k, a, it == 0 ? a.ms_stats : 0.f);
            if (it == 0) log[nl].n_launches += ctx->prep_launches;
        }
        ++nl;
        const bool found = a.res.n_sel >= (int)top_k;
        if (!halving || found || r2 == 0.f) break; // r2 == 0 admits every nn > 0
        rr = (float)(0.5 * (double)rr);
    }
    ctx->opts.segment_len = saved_seg;
    *n_out = (uint32_t)a.res.n_sel;
    for (int q = 0; q < a.res.n_sel; ++q) {
        out[q].ind = a.res.sel_ind[q];
        out[q].dist = a.res.sel_dist[q];
    }
    if (n_log) *n_log = nl;
    return PADDI_OK;
}

PADDI_API paddi_status paddi_compute_statistics(paddi_ctx *ctx, const float *d_T, float *d_mean,
                                                float *d_std, size_t n, uint32_t m, void *stream)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!d_T || !d_mean || !d_std || !valid_lengths(n, m, m))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "invalid pointers or length");
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    cudaStream_t user = stream ? (cudaStream_t)stream : ctx->st;
    if (user != ctx->st) { // order the context stream after the caller's
        CK(cudaEventRecord(ctx->ev[0], user));
        CK(cudaStreamWaitEvent(ctx->st, ctx->ev[0], 0));
    }
    CK(paddi_launch_mean_std(d_T, (int64_t)n, (int32_t)m, d_mean, d_std, ctx->st));
    if (user != ctx->st) {
        CK(cudaEventRecord(ctx->ev[1], ctx->st));
        CK(cudaStreamWaitEvent(user, ctx->ev[1], 0));
    }
    return PADDI_OK;
}

PADDI_API paddi_status paddi_do_pd3(paddi_ctx *ctx, const float *d_T, size_t n, uint32_t m,
                                    float r2, int32_t *d_is_cand, float *d_nnDist,
                                    int64_t *n_cand, void *stream)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!d_T || !d_is_cand || !d_nnDist || !valid_lengths(n, m, m) || !(r2 >= 0.f))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "invalid pointers, length or threshold");
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    cudaStream_t user = stream ? (cudaStream_t)stream : ctx->st;
    if (user != ctx->st) {
        CK(cudaEventRecord(ctx->ev[0], user));
        CK(cudaStreamWaitEvent(ctx->st, ctx->ev[0], 0));
    }
    s = run_stats(ctx, d_T, n, (int)m);
    if (s != PADDI_OK) return s;
    AttemptOut a;
    s = run_attempt(ctx, d_T, n, (int)m, r2, 1, &a);
    if (s != PADDI_OK) return s;
    CK(paddi_launch_scatter(ctx->d_cand, ctx->d_att, ctx->d_rho, ctx->d_pruned, ctx->d_rcslot,
                            ctx->d_nn64, ctx->d_flat, (int32_t)(n - m + 1), (int)m, r2, d_is_cand,
                            d_nnDist, ctx->st));
    if (user != ctx->st) {
        CK(cudaEventRecord(ctx->ev[1], ctx->st));
        CK(cudaStreamWaitEvent(user, ctx->ev[1], 0));
    } else {
        CK(cudaStreamSynchronize(ctx->st));
    }
    if (n_cand) *n_cand = a.res.n_cand;
    return PADDI_OK;
}

// ==================================================================== shards
PADDI_API paddi_status paddi_shard_phase1(paddi_ctx *ctx, const float *d_series, size_t n,
                                          uint32_t m, float r2, size_t row_lo, size_t row_hi,
                                          uint8_t *d_alive)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!d_series || !d_alive || !valid_lengths(n, m, m) || !(r2 >= 0.f))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "shard_phase1: invalid series, length or r2");
    const size_t N = n - m + 1;
    if (row_lo >= row_hi || row_hi > N)
        return fail(ctx, PADDI_ERR_INVALID_ARG, "shard_phase1: empty or out-of-range rows");
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    s = run_stats(ctx, d_series, n, (int)m);
    if (s != PADDI_OK) return s;
    cudaStream_t st = ctx->st;
    CK(cudaMemsetAsync(d_alive, 1, N, st));
    CK(cudaMemsetAsync(ctx->d_att, 0, sizeof(PaddiAttemptDev), st));
    const int chunks = ctx->opts.phase1_chunks ? (int)ctx->opts.phase1_chunks : 12;
    CK(paddi_launch_phase1_dev(d_series, ctx->d_wst, ctx->d_mu, ctx->d_ms64, d_alive, (int32_t)N,
                               (int)m, p1_rows_of(ctx, (int64_t)(row_hi - row_lo), (int)m), chunks, thr_of(r2, (int)m),
                               (int32_t)row_lo, (int32_t)row_hi, ctx->d_att, ctx->num_sms, st));
    CK(cudaStreamSynchronize(st));
    return PADDI_OK;
}

PADDI_API paddi_status paddi_shard_refine(paddi_ctx *ctx, const float *d_series, size_t n,
                                          uint32_t m, float r2, const uint8_t *d_alive,
                                          size_t col_lo, size_t col_hi, int32_t *d_ind,
                                          uint32_t *d_rho, uint8_t *d_pruned, uint32_t cap,
                                          uint32_t *n_cand)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!d_series || !d_alive || !d_ind || !d_rho || !d_pruned || !n_cand ||
        !valid_lengths(n, m, m) || !(r2 >= 0.f))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "shard_refine: invalid argument");
    const size_t N = n - m + 1;
    const size_t grid = (size_t)paddi_tile_width();
    if (col_lo >= col_hi || col_hi > N || col_lo % grid || (col_hi % grid && col_hi != N))
        return fail(ctx, PADDI_ERR_INVALID_ARG,
                    "shard_refine: columns must be [a, b) with a, b multiples of 2048 (b or N)");
    if (ctx->cap_n < n)
        return fail(ctx, PADDI_ERR_INVALID_ARG, "shard_refine: run paddi_shard_phase1 first");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->st;
    const int kernel = refine_kernel_for(ctx, (int)m);
    const float thr = thr_of(r2, (int)m);
    CK(cudaMemsetAsync(ctx->d_att, 0, sizeof(PaddiAttemptDev), st));
    CK(paddi_launch_compact(const_cast<uint8_t *>(d_alive), false, (int32_t)N, ctx->d_cand, ctx->d_rho, ctx->d_pruned,
                            ctx->d_rcslot, ctx->d_att, ctx->d_flat, ctx->d_flatcount + 1, (int)m,
                            r2 > 0.f, false, st));
    int launches = 0;
    paddi_status s = refine_rounds(ctx, d_series, (int32_t)N, (int)m, kernel, thr,
                                   guard_of(ctx, kernel), (int32_t)col_lo, (int32_t)col_hi,
                                   &launches);
    if (s != PADDI_OK) return s;
    CK(cudaMemcpyAsync(&ctx->h_res->n_p1, &ctx->d_att->n_cand_p1, sizeof(int32_t),
                       cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(&ctx->h_res->status, &ctx->d_att->status, sizeof(int32_t),
                       cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (ctx->h_res->status == 3) // the arrays miss pairs
        return fail(ctx, PADDI_ERR_CUDA, refine_timeout(kernel, (int)m));
    const int32_t C = ctx->h_res->n_p1;
    *n_cand = (uint32_t)C;
    if ((uint32_t)C > cap)
        return fail(ctx, PADDI_ERR_INTERNAL_LIMIT,
                    "shard_refine: " + std::to_string(C) + " candidates, room for " +
                        std::to_string(cap));
    if (C > 0) {
        CK(cudaMemcpyAsync(d_ind, ctx->d_cand, sizeof(int32_t) * C, cudaMemcpyDeviceToDevice, st));
        CK(cudaMemcpyAsync(d_rho, ctx->d_rho, sizeof(uint32_t) * C, cudaMemcpyDeviceToDevice, st));
        CK(cudaMemcpyAsync(d_pruned, ctx->d_pruned, C, cudaMemcpyDeviceToDevice, st));
    }
    CK(cudaStreamSynchronize(st));
    return PADDI_OK;
}

PADDI_API paddi_status paddi_shard_select(paddi_ctx *ctx, const float *d_series, size_t n,
                                          uint32_t m, float r2, const int32_t *d_ind,
                                          const uint32_t *d_rho, const uint8_t *d_pruned,
                                          uint32_t count, uint32_t top_k, paddi_discord *out,
                                          uint32_t *n_out, paddi_attempt_log *log)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!d_series || (count && (!d_ind || !d_rho || !d_pruned)) || !out || !n_out ||
        top_k < 1 || top_k > PADDI_MAX_TOPK || !valid_lengths(n, m, m) || !(r2 >= 0.f))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "shard_select: invalid argument");
    const size_t N = n - m + 1;
    if (count > N || ctx->cap_n < n)
        return fail(ctx, PADDI_ERR_INVALID_ARG, "shard_select: count or context out of range");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->st;
    const int kernel = refine_kernel_for(ctx, (int)m);
    // the merged candidates become this context's candidate arrays
    CK(cudaMemsetAsync(ctx->d_att, 0, sizeof(PaddiAttemptDev), st));
    if (count > 0) {
        CK(cudaMemcpyAsync(ctx->d_cand, d_ind, sizeof(int32_t) * count, cudaMemcpyDeviceToDevice,
                           st));
        CK(cudaMemcpyAsync(ctx->d_rho, d_rho, sizeof(uint32_t) * count, cudaMemcpyDeviceToDevice,
                           st));
        CK(cudaMemcpyAsync(ctx->d_pruned, d_pruned, count, cudaMemcpyDeviceToDevice, st));
        CK(cudaMemsetAsync(ctx->d_rcslot, 0xff, sizeof(int32_t) * count, st)); // -1
    }
    ctx->h_res->n_p1 = (int32_t)count;
    CK(cudaMemcpyAsync(&ctx->d_att->n_cand_p1, &ctx->h_res->n_p1, sizeof(int32_t),
                       cudaMemcpyHostToDevice, st));
    int launches = 0;
    bool spec = false;
    paddi_status s = select_passes(ctx, d_series, n, (int)m, r2, guard_of(ctx, kernel), false,
                                   (int)top_k, -1, 0, 0, false, &spec, &launches);
    if (s != PADDI_OK) return s;
    AttemptOut a;
    a.res = *ctx->h_res;
    a.launches = launches;
    a.kernel = kernel;
    a.ms_select = ms_between(a.res.t[PADDI_T_SELECT], a.res.t[PADDI_T_END]);
    a.ms_total = a.ms_select;
    *n_out = (uint32_t)a.res.n_sel;
    for (int q = 0; q < a.res.n_sel; ++q) {
        out[q].ind = a.res.sel_ind[q];
        out[q].dist = a.res.sel_dist[q];
    }
    if (log) fill_log(log, (int)m, std::sqrt(r2), r2, (int)top_k, a, 0.f);
    return PADDI_OK;
}

PADDI_API float paddi_merlin_first_r(const paddi_discord *out, uint32_t j, uint32_t minL, float *S)
{
    if (j > 0 && !out) return 0.f;
    return merlin_first_r(out, (int)j, minL, S);
}

PADDI_API float paddi_merlin_lower(float r, uint32_t j, float S)
{
    return merlin_lower(r, (int)j, S);
}

// ================================================================ test hooks
PADDI_API paddi_status paddi_debug_set(paddi_ctx *ctx, int32_t key, int64_t value)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    switch (key) {
    case PADDI_DEBUG_FAIL_ALLOC:
        if (value < 0) break;
        ctx->fail_alloc = value;
        return PADDI_OK;
    case PADDI_DEBUG_WAIT_CYCLES:
        if (value < 0) break;
        ctx->wait_cycles = (long long)value;
        return PADDI_OK;
    case PADDI_DEBUG_WITHHOLD_STAGE:
        ctx->withhold = value != 0;
        return PADDI_OK;
    case PADDI_DEBUG_RECHECK_CAP: {
        if (value < 1 || value > (1 << 24) || !ctx->d_recheck) break;
        CK(cudaSetDevice(ctx->device));
        CK(cudaStreamSynchronize(ctx->st));
        CK(set_recheck_cap(ctx, (int32_t)value));
        return PADDI_OK;
    }
    default:
        break;
    }
    return fail(ctx, PADDI_ERR_INVALID_ARG, "paddi_debug_set: unknown key or bad value");
}

PADDI_API paddi_status paddi_debug_get(paddi_ctx *ctx, int32_t key, int64_t *value)
{
    if (!ctx || !value) return PADDI_ERR_INVALID_ARG;
    switch (key) {
    case PADDI_DEBUG_FAIL_ALLOC: *value = ctx->fail_alloc; return PADDI_OK;
    case PADDI_DEBUG_WAIT_CYCLES: *value = ctx->wait_cycles; return PADDI_OK;
    case PADDI_DEBUG_WITHHOLD_STAGE: *value = ctx->withhold; return PADDI_OK;
    case PADDI_DEBUG_LAST_PASSES: *value = ctx->last_passes; return PADDI_OK;
    case PADDI_DEBUG_RECHECK_CAP: *value = ctx->rc_cap; return PADDI_OK;
    case PADDI_DEBUG_WORKERS: *value = (int64_t)ctx->workers.size(); return PADDI_OK;
    case PADDI_DEBUG_WITNESS_STEPS: *value = (int64_t)ctx->wit.steps2; return PADDI_OK;
    default: break;
    }
    return fail(ctx, PADDI_ERR_INVALID_ARG, "paddi_debug_get: unknown key");
}

PADDI_API int64_t paddi_debug_refine_item(int32_t kernel, uint32_t m, uint32_t candidates,
                                          uint32_t windows, uint32_t ctas, int64_t *items)
{
    if (m < 3 || m > 1024 || candidates < 1 || windows < 1 || ctas < 1 || ctas > 1 << 16 ||
        candidates > INT32_MAX - 64 || windows > INT32_MAX - 64)
        return -1;
    const bool fp32 = kernel == PADDI_DIST_FP32 || (int)m > paddi_umma_max_m();
    const paddi::RefineItems I =
        fp32 ? paddi_refine_items_fp32((int32_t)m, (int32_t)candidates, (int32_t)windows,
                                       (int32_t)ctas)
             : paddi_refine_items_umma((int32_t)m, false, (int32_t)candidates, (int32_t)windows,
                                       (int32_t)ctas);
    if (items) *items = I.splits;
    return I.span;
}

// ============================================================ learned r model
PADDI_API paddi_status paddi_r_features(const paddi_discord *out, uint32_t j, uint32_t minL,
                                        float lb, float flat_frac, uint32_t prev_attempts,
                                        float *features)
{
    if (!features || (j > 0 && !out) || minL < 3) return PADDI_ERR_INVALID_ARG;
    r_features_impl(out, (int)j, minL, lb, flat_frac, (int)prev_attempts, features);
    return PADDI_OK;
}

PADDI_API paddi_status paddi_model_set(paddi_ctx *ctx, const float *params, uint32_t count,
                                       float margin)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!params || count != MLP_NPARAM || !(margin > 0.f))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "model parameters: wrong count or margin");
    CK(cudaSetDevice(ctx->device));
    CK(cudaMemcpyAsync(ctx->d_model, params, sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice,
                       ctx->st));
    CK(paddi_launch_mlp_to_bf16(ctx->d_model, ctx->d_model_bf16, ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
    ctx->model_ok = true;
    ctx->model_margin = margin;
    return PADDI_OK;
}

namespace {
struct DevBuf {
    void *p = nullptr;
    ~DevBuf()
    {
        if (p) cudaFree(p);
    }
};
} // namespace

PADDI_API paddi_status paddi_model_grad(paddi_ctx *ctx, const float *X, const float *Y,
                                        uint32_t n, float tau, const float *params, float *grad,
                                        float *loss)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!X || !Y || !params || !grad || !loss || n == 0)
        return fail(ctx, PADDI_ERR_INVALID_ARG, "model_grad: null argument or empty data");
    CK(cudaSetDevice(ctx->device));
    DevBuf dX, dY, dP, dG, dL;
    CK(dmalloc(ctx, &dX.p, sizeof(float) * MLP_NFEAT * n));
    CK(dmalloc(ctx, &dY.p, sizeof(float) * n));
    CK(dmalloc(ctx, &dP.p, sizeof(float) * MLP_NPARAM));
    CK(dmalloc(ctx, &dG.p, sizeof(double) * MLP_NPARAM));
    CK(dmalloc(ctx, &dL.p, sizeof(double)));
    cudaStream_t st = ctx->st;
    CK(cudaMemcpyAsync(dX.p, X, sizeof(float) * MLP_NFEAT * n, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dY.p, Y, sizeof(float) * n, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dP.p, params, sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice, st));
    CK(cudaMemsetAsync(dG.p, 0, sizeof(double) * MLP_NPARAM, st));
    CK(cudaMemsetAsync(dL.p, 0, sizeof(double), st));
    CK(paddi_launch_mlp_grad((float *)dX.p, (float *)dY.p, nullptr, (int)n, tau, (float *)dP.p,
                             (double *)dG.p, (double *)dL.p, ctx->num_sms, st));
    std::vector<double> g(MLP_NPARAM);
    CK(cudaMemcpyAsync(g.data(), dG.p, sizeof(double) * MLP_NPARAM, cudaMemcpyDeviceToHost, st));
    double lsum = 0.0;
    CK(cudaMemcpyAsync(&lsum, dL.p, sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    for (int i = 0; i < MLP_NPARAM; ++i) grad[i] = (float)g[i];
    *loss = (float)lsum;
    return PADDI_OK;
}

PADDI_API paddi_status paddi_model_predict(paddi_ctx *ctx, const float *X, uint32_t n,
                                           const float *params, int32_t bf16, float *Y)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!X || !Y || !params || n == 0)
        return fail(ctx, PADDI_ERR_INVALID_ARG, "model_predict: null argument or empty data");
    CK(cudaSetDevice(ctx->device));
    DevBuf dX, dY, dP, dQ;
    cudaStream_t st = ctx->st;
    CK(dmalloc(ctx, &dX.p, sizeof(float) * MLP_NFEAT * n));
    CK(dmalloc(ctx, &dY.p, sizeof(float) * n));
    CK(dmalloc(ctx, &dP.p, sizeof(float) * MLP_NPARAM));
    CK(dmalloc(ctx, &dQ.p, 2 * MLP_NPARAM));
    CK(cudaMemcpyAsync(dX.p, X, sizeof(float) * MLP_NFEAT * n, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(dP.p, params, sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice, st));
    if (bf16) {
        CK(paddi_launch_mlp_to_bf16((float *)dP.p, dQ.p, st));
        CK(paddi_launch_mlp_forward((float *)dX.p, (int)n, dQ.p, true, (float *)dY.p, st));
    } else {
        CK(paddi_launch_mlp_forward((float *)dX.p, (int)n, dP.p, false, (float *)dY.p, st));
    }
    CK(cudaMemcpyAsync(Y, dY.p, sizeof(float) * n, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    return PADDI_OK;
}

PADDI_API paddi_status paddi_model_train(paddi_ctx *ctx, const float *X, const float *Y,
                                         uint32_t n, float tau, uint32_t epochs, uint32_t batch,
                                         float lr, uint64_t seed, float *params, float *loss)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!X || !Y || !params || n == 0 || batch == 0 || !(tau > 0.f && tau < 1.f) || !(lr > 0.f))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "model_train: bad argument");
    CK(cudaSetDevice(ctx->device));
    cudaStream_t st = ctx->st;
    // one allocation: the samples, an epoch's order, parameters (FP32), gradient, Adam's
    // state and losses (64 bits)
    DevBuf buf;
    size_t bytes = 0;
    auto place = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) & ~(size_t)255;
        return at;
    };
    const size_t np = sizeof(float) * MLP_NPARAM, nl = sizeof(double) * (epochs ? epochs : 1);
    const size_t oX = place(sizeof(float) * MLP_NFEAT * n), oY = place(sizeof(float) * n);
    const size_t oI = place(sizeof(uint32_t) * n), oP = place(np), oG = place(2 * np);
    const size_t oA = place(6 * np), oL = place(nl);
    CK(dmalloc(ctx, &buf.p, bytes));
    auto at = [&](size_t o) { return reinterpret_cast<float *>(static_cast<char *>(buf.p) + o); };
    auto at64 = [&](size_t o) { return reinterpret_cast<double *>(at(o)); };
    uint32_t *dI = reinterpret_cast<uint32_t *>(at(oI));
    CK(cudaMemsetAsync(at(oG), 0, bytes - oG, st));
    CK(cudaMemcpyAsync(at(oP), params, np, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(at(oX), X, sizeof(float) * MLP_NFEAT * n, cudaMemcpyHostToDevice, st));
    CK(cudaMemcpyAsync(at(oY), Y, sizeof(float) * n, cudaMemcpyHostToDevice, st));
    std::vector<uint32_t> perm(n);
    for (uint32_t i = 0; i < n; ++i) perm[i] = i;
    uint64_t rng = seed * 6364136223846793005ull + 1442695040888963407ull;
    int step = 0;
    for (uint32_t e = 0; e < epochs; ++e) {
        // the next order is drawn while the epoch before runs (the copy from
        // pageable memory is done with the host's array when it returns)
        for (uint32_t i = n - 1; i > 0; --i) { // Fisher-Yates with an LCG
            rng = rng * 6364136223846793005ull + 1442695040888963407ull;
            const uint32_t k = (uint32_t)(rng >> 33) % (i + 1);
            std::swap(perm[i], perm[k]);
        }
        CK(cudaMemcpyAsync(dI, perm.data(), sizeof(uint32_t) * n, cudaMemcpyHostToDevice, st));
        for (uint32_t b0 = 0; b0 < n; b0 += batch) {
            const uint32_t bn = std::min(batch, n - b0);
            CK(paddi_launch_mlp_grad(at(oX), at(oY), dI + b0, (int)bn, tau, at(oP), at64(oG),
                                     at64(oL) + e, ctx->num_sms, st));
            CK(paddi_launch_mlp_adam(at(oP), at64(oG), at64(oA), lr, ++step, st));
        }
    }
    CK(cudaMemcpyAsync(params, at(oP), np, cudaMemcpyDeviceToHost, st));
    std::vector<double> lsum(epochs ? epochs : 1);
    CK(cudaMemcpyAsync(lsum.data(), at(oL), nl, cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (loss) {
        const uint32_t nb = (n + batch - 1) / batch;
        for (uint32_t e = 0; e < epochs; ++e) loss[e] = (float)(lsum[e] / (double)nb);
    }
    return PADDI_OK;
}

// ============================================================ batched PALMAD
namespace {
paddi_status add_worker(paddi_ctx *ctx)
{
    paddi_ctx *c = nullptr;
    const paddi_status s = paddi_ctx_create(&c, &ctx->opts);
    if (s == PADDI_OK) ctx->workers.push_back(c);
    return s;
}

// A worker shares the options and the model of its context.
paddi_status set_up_worker(paddi_ctx *ctx, paddi_ctx *c)
{
    c->opts = ctx->opts;
    c->model_ok = ctx->model_ok;
    c->model_margin = ctx->model_margin;
    if (ctx->model_ok) {
        CK(cudaMemcpy(c->d_model, ctx->d_model, sizeof(float) * MLP_NPARAM,
                      cudaMemcpyDeviceToDevice));
        CK(cudaMemcpy(c->d_model_bf16, ctx->d_model_bf16, 2 * MLP_NPARAM,
                      cudaMemcpyDeviceToDevice));
    }
    return PADDI_OK;
}
} // namespace

PADDI_API paddi_status paddi_palmad_batched(paddi_ctx *ctx, const float *const *series,
                                            const size_t *lens, uint32_t count, uint32_t minL,
                                            uint32_t maxL, uint32_t streams, paddi_discord *out,
                                            int32_t *status, uint64_t *attempts)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!series || !lens || !out || count == 0)
        return fail(ctx, PADDI_ERR_INVALID_ARG, "batched: null argument or empty batch");
    for (uint32_t k = 0; k < count; ++k)
        if (!series[k] || !valid_lengths(lens[k], minL, maxL))
            return fail(ctx, PADDI_ERR_INVALID_ARG,
                        "batched: series " + std::to_string(k) + " invalid or shorter than 2*maxL");
    const uint32_t L = maxL - minL + 1;
    int W = streams ? (int)streams : 4;
    if ((uint32_t)W > count) W = (int)count;
    drop_workers(ctx, (size_t)W);
    CK(cudaSetDevice(ctx->device));
    paddi_status ws = PADDI_OK;
    while (ws == PADDI_OK && ctx->workers.size() < (size_t)W) ws = add_worker(ctx);
    for (size_t k = 0; ws == PADDI_OK && k < ctx->workers.size(); ++k)
        ws = set_up_worker(ctx, ctx->workers[k]);
    if (ws != PADDI_OK) return fail(ctx, ws, "batched: cannot create worker contexts");
    // (a test's refused allocation is the first worker's)
    std::swap(ctx->fail_alloc, ctx->workers[0]->fail_alloc);
    CK(cudaDeviceSynchronize()); // the copies precede the workers' (non-blocking) streams
    // longest series first: a worker's buffers are sized by its first one, and the
    // short ones even out the end
    std::vector<uint32_t> order(count);
    for (uint32_t k = 0; k < count; ++k) order[k] = k;
    std::stable_sort(order.begin(), order.end(),
                     [&](uint32_t a, uint32_t b) { return lens[a] > lens[b]; });
    std::atomic<uint32_t> next{0};
    std::vector<int32_t> st(count, (int32_t)PADDI_OK);
    std::vector<std::string> errs(count);
    std::vector<uint64_t> na(count, 0);
    auto run = [&](paddi_ctx *c, std::vector<paddi_attempt_log> &lg, uint32_t k) {
        uint32_t nl = 0;
        st[k] = (int32_t)paddi_palmad(c, series[k], lens[k], minL, maxL, out + (size_t)k * L,
                                      lg.data(), (uint32_t)lg.size(), &nl);
        errs[k] = st[k] != PADDI_OK ? c->err : std::string();
        na[k] = nl;
    };
    std::vector<std::thread> pool;
    for (int w = 0; w < W; ++w) {
        pool.emplace_back([&, w]() {
            paddi_ctx *c = ctx->workers[w];
            cudaSetDevice(c->device);
            std::vector<paddi_attempt_log> lg(4096);
            for (uint32_t q = next++; q < count; q = next++) run(c, lg, order[q]);
        });
    }
    for (auto &t : pool) t.join();
    std::swap(ctx->fail_alloc, ctx->workers[0]->fail_alloc);
    // a worker cannot take the memory of the others, which may have kept theirs from
    // longer series: what did not fit runs again, one by one, on a single worker
    const auto refused = [&](uint32_t k) { return st[k] == (int32_t)PADDI_ERR_OUT_OF_MEMORY; };
    if (std::any_of(order.begin(), order.end(), refused)) {
        drop_workers(ctx);
        std::vector<paddi_attempt_log> lg(4096);
        for (uint32_t k : order) {
            if (!refused(k)) continue;
            if (ctx->workers.empty() &&
                (add_worker(ctx) != PADDI_OK ||
                 set_up_worker(ctx, ctx->workers[0]) != PADDI_OK ||
                 cudaDeviceSynchronize() != cudaSuccess))
                break;
            run(ctx->workers[0], lg, k);
        }
    }
    paddi_status first_err = PADDI_OK;
    std::string msg;
    for (uint32_t k = 0; k < count; ++k) {
        if (status) status[k] = st[k];
        if (attempts) attempts[k] = na[k];
        if (st[k] != PADDI_OK && first_err == PADDI_OK) {
            first_err = (paddi_status)st[k];
            msg = "batched: series " + std::to_string(k) + ": " + errs[k];
        }
    }
    if (first_err != PADDI_OK) {
        drop_workers(ctx);
        return fail(ctx, first_err, msg);
    }
    size_t points = 0, keep = 0;
    while (keep < ctx->workers.size() &&
           (points += ctx->workers[keep]->cap_n) <= kWorkerPoints)
        ++keep;
    drop_workers(ctx, keep);
    return PADDI_OK;
}

// ================================================================ autotuner
PADDI_API paddi_status paddi_autotune(paddi_ctx *ctx, const float *series, size_t n,
                                      uint32_t minL, uint32_t maxL, paddi_opts *chosen,
                                      float *ms)
{
    if (!ctx) return PADDI_ERR_INVALID_ARG;
    if (!series || !valid_lengths(n, minL, maxL))
        return fail(ctx, PADDI_ERR_INVALID_ARG, "autotune: invalid series or lengths");
    CK(cudaSetDevice(ctx->device));
    paddi_status s = ensure_capacity(ctx, n);
    if (s != PADDI_OK) return s;
    CK(cudaMemcpyAsync(ctx->d_x, series, sizeof(float) * n, cudaMemcpyHostToDevice, ctx->st));
    // probe ranges: 3 consecutive lengths at the start, the middle and the end
    std::vector<std::pair<uint32_t, uint32_t>> probes;
    const uint32_t mid = minL + (maxL - minL) / 2;
    for (uint32_t a : {minL, mid, maxL >= minL + 2 ? maxL - 2 : minL}) {
        const uint32_t b = std::min(maxL, a + 2);
        if (probes.empty() || probes.back().first != a) probes.push_back({a, b});
    }
    const uint32_t tiles[2] = {0, 64}, segs[3] = {256, 384, 512}, chunks[3] = {8, 12, 16};
    const paddi_opts saved = ctx->opts;
    std::vector<std::vector<paddi_discord>> ref;
    float best = FLT_MAX;
    paddi_opts best_opts = saved;
    std::vector<paddi_discord> out(3);
    // configurations that are the same program on these lengths (p1_rows_of caps the
    // rows of a segment) are timed once
    std::map<std::vector<int>, float> timed;
    int idx = 0;
    for (uint32_t tr : tiles)
        for (uint32_t sg : segs)
        for (uint32_t ch : chunks) {
            ctx->opts = saved;
            ctx->opts.tile_rows = tr;
            ctx->opts.segment_len = sg;
            ctx->opts.phase1_chunks = ch;
            std::vector<int> program = {(int)tr, (int)ch};
            for (const auto &p : probes)
                for (uint32_t m = p.first; m <= p.second; ++m)
                    program.push_back(p1_rows_of(ctx, (int64_t)(n - m + 1), (int)m));
            const auto same = timed.find(program);
            // one untimed pass (kernel attributes, caches), then the timed one
            float t_total = same == timed.end() ? 0.f : same->second;
            for (int pass = 0; pass < 2 && same == timed.end(); ++pass) {
                t_total = 0.f;
                for (size_t p = 0; p < probes.size(); ++p) {
                    const uint32_t a = probes[p].first, b = probes[p].second;
                    out.assign(b - a + 1, paddi_discord{-1, -FLT_MAX});
                    CK(cudaEventRecord(ctx->ev[2], ctx->st));
                    s = palmad_impl(ctx, ctx->d_x, n, a, b, out.data(), nullptr, 0, nullptr);
                    if (s != PADDI_OK) {
                        ctx->opts = saved;
                        return s;
                    }
                    CK(cudaEventRecord(ctx->ev[3], ctx->st));
                    CK(cudaEventSynchronize(ctx->ev[3]));
                    float t = 0.f;
                    CK(cudaEventElapsedTime(&t, ctx->ev[2], ctx->ev[3]));
                    t_total += t;
                    if (pass == 1) {
                        if (ref.size() <= p) ref.push_back(out);
                        else
                            for (size_t q = 0; q < out.size(); ++q)
                                if (out[q].ind != ref[p][q].ind || out[q].dist != ref[p][q].dist) {
                                    ctx->opts = saved;
                                    return fail(ctx, PADDI_ERR_INTERNAL_LIMIT,
                                                "autotune: configurations disagree");
                                }
                    }
                }
            }
            timed[program] = t_total;
            if (ms) ms[idx] = t_total;
            ++idx;
            if (t_total < best) {
                best = t_total;
                best_opts = ctx->opts;
            }
        }
    ctx->opts = best_opts;
    if (chosen) *chosen = best_opts;
    return PADDI_OK;
}
