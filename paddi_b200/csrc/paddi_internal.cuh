// paddi_internal.cuh -- shared device helpers and launch wrappers of the
// discord-discovery kernels (single GPU, sm_100a).
//
// Per-window data for one subsequence length m, laid out in HBM as arrays
// over the N = n - m + 1 windows (plus PADDI_PAD_WIN zeroed entries so tiles
// may read past the end without bounds checks):
//   wst[i]  float4 {df_i, dg_i, inv_i, n_i}   -- diagonal-update terms
//           df_i = (x[i+m] - x[i]) / 2,  dg_i = (x[i+m] - mu_{i+1}) + (x[i] - mu_i)
//           n_i = |x_i - mu_i| (the window's norm), inv_i = 1 / n_i; both 0 for
//           a flat window (window i is flat iff inv_i == 0)
//   mu[i]   float  window mean
//   ms64[i].x, ms64[i].y  FP64 mean and inverse norm (recheck path)
//   flat[i] uint8
// The correlation of windows i, j is rho = cov(i,j) * inv_i * inv_j with
// cov the centred dot product; the squared z-normalised distance is
// d = 2m (1 - rho) (reference: src/PD3_kernels.cuh:61).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

/* zeroed tail entries after the last window: covers the columns a phase-1
 * task of up to 4096 rows reads past the end (rows + 256) and a tile of the
 * tensor-core refine (2048 windows) */
#define PADDI_PAD_WIN 4608

namespace paddi {

// ---- launches in a chain.  A kernel of an attempt starts while the one
// before it drains (programmatic stream serialization): its first act is to
// wait until that kernel is complete and its writes are visible, its second to
// let the next kernel come in as soon as all of its own blocks run.  Saves the
// launch latency between dependent kernels, about 2 us each; an attempt has a
// dozen of 2 to 60 us.  No parameter that a kernel writes is __restrict__ in such a
// kernel: its life begins while the one before it still writes, and the qualifier
// would allow a load above the wait.
__device__ __forceinline__ void chain_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Time stamps instead of events between the kernels: a stamp costs one store,
// an event a break in the stream.
__device__ __forceinline__ unsigned long long time_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void stamp_begin(unsigned long long *t)
{
    if (t && blockIdx.x == 0 && threadIdx.x == 0) *t = time_ns();
}
// by one thread of every block, when the block is done
__device__ __forceinline__ void stamp_end(unsigned long long *t)
{
    if (t) atomicMax(t, time_ns());
}

// Monotone map float -> uint32 so that unsigned max == float max.
__device__ __forceinline__ uint32_t f2ord(float f)
{
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(uint32_t u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}
// Monotone map double -> uint64 (for FP64 atomic min/max).
__device__ __forceinline__ unsigned long long d2ord(double d)
{
    unsigned long long u = (unsigned long long)__double_as_longlong(d);
    return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord2d(unsigned long long u)
{
    return __longlong_as_double((long long)((u & 0x8000000000000000ull)
                                                ? (u & 0x7fffffffffffffffull)
                                                : ~u));
}

// Rounding bound, in correlation units, of a refine kernel's correlation of
// any candidate with window j whose operand is the series shifted by s:
//     g_j = E * A_j + F * inv_j,   A_j = |x_j - s| / |x_j - mu_j| = sqrt(1 + m b^2),
// b = (mu_j - s) inv_j.  E (per kernel and length) bounds the relative error of
// the dot product with respect to |z| |x_j - s| (|z| = 1), F an absolute error
// term of the operand's representation.  Explicitly rounded operations, so
// every kernel that evaluates it for the same window gets the same value.
__device__ __forceinline__ float window_bound(float inv, float mu, float s, float m, float E,
                                              float F)
{
    const float b = __fmul_rn(__fsub_rn(mu, s), inv);
    const float A = __fsqrt_rn(__fadd_rn(1.f, __fmul_rn(m, __fmul_rn(b, b))));
    return __fadd_rn(__fmul_rn(__fmul_rn(E, A), 1.0001f), __fmul_rn(F, inv));
}

} // namespace paddi

// Bound constants of the refine kernels for length m (see window_bound):
// E covers the 16-bit split operands (FP16: 2^-22 per value and the dropped
// lo*lo term; BF16: 2^-16), one FP32 rounding per tensor-core MMA of the
// accumulator (3 kp/16 MMAs, kp = K padded) and the FP32 arithmetic around it
// (the candidate's z, the sum of its split values, the epilogue); F covers
// FP16 lo halves that fall below the normal range (2^-25 absolute per scaled
// value; F is per unit of the tile's largest |x - s|).  The FP32 CUDA-core
// refine sums in two levels of 32 terms and has F = 0.
struct PaddiBound {
    float E, F;
};
PaddiBound paddi_bound_tc(int m, bool bf16);
PaddiBound paddi_bound_fp32(int m);

// Launches `kern`; chained: as the successor of the stream's previous kernel (see
// paddi::chain_begin, which the kernel must call first).
// carveout >= 0: the percentage of an SM's L1 that the kernel prefers as shared memory.
template <typename... P, typename... A>
cudaError_t paddi_launch_carveout(int carveout, bool chained, void (*kern)(P...), unsigned grid,
                                  unsigned block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at[2] = {};
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = at;
    if (chained) {
        at[c.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[c.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (carveout >= 0) {
        at[c.numAttrs].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
        at[c.numAttrs++].val.sharedMemCarveout = (unsigned)carveout;
    }
    return cudaLaunchKernelEx(&c, kern, P(args)...);
}

template <typename... P, typename... A>
cudaError_t paddi_launch(bool chained, void (*kern)(P...), unsigned grid, unsigned block,
                         size_t smem, cudaStream_t st, A... args)
{
    return paddi_launch_carveout(-1, chained, kern, grid, block, smem, st, args...);
}

// Time stamps (ns, globaltimer) of a length's preparation and of an attempt.
enum { PADDI_T_STATS_B, PADDI_T_STATS_E, PADDI_T_GUIDE_B, PADDI_T_GUIDE_E, PADDI_T_PREP };
enum { PADDI_T_BEGIN, PADDI_T_COMPACT, PADDI_T_REFINE_B, PADDI_T_REFINE_E, PADDI_T_FRAGILE,
       PADDI_T_SELECT, PADDI_T_END, PADDI_T_ATTEMPT };

// Per-attempt device-side state shared by the kernels of one (m, r) attempt.
struct PaddiAttemptDev {
    int32_t n_cand_p1;      // candidates after phase 1 (compacted list length)
    int32_t work_rd[4];     // work-item counters of the refine rounds (one per round)
    int32_t recheck_next;   // work-item counter of the FP64 recheck kernel
    int32_t n_recheck;      // windows queued for the FP64 recheck (at most its capacity)
    int32_t n_recheck_all;  // windows that needed it: above the capacity, the queue overflowed
    int32_t status;         // nonzero: a kernel hit an internal limit
    int32_t task_next;      // task counter of the phase-1 kernel
    int32_t list_count[5];  // candidate-list length entering each refine round (and after
                            // the last); zero when the attempt starts, so the compactions
                            // between rounds need no reset
    int32_t p1_walked;      // phase-1 tasks that walked their rows (instrumentation)
    int32_t n_fail;         // windows whose witness proves nothing (k_witness.cu)
    int32_t n_rescued;      // of those, windows that found a new witness
    int32_t done_rd[4];     // finished work items of the tensor-core refine's rounds
    int32_t round_ready;    // rounds whose survivors are compacted
    int32_t last_rd;        // the round after which no window was left
    unsigned long long n_pairs; // pairs evaluated by the refine (instrumentation)
    unsigned long long n_live;  // of those, pairs of candidates still unpruned at the tile's start
    unsigned long long t[PADDI_T_ATTEMPT]; // time stamps
};
static_assert(sizeof(PaddiAttemptDev) % 4 == 0, "cleared in words");

namespace paddi {

// ---- rounds of a refine launch: the windows in growing ranges (1/16, 1/4,
// 1/2, all of them), the survivors compacted in between.
__host__ __device__ __forceinline__ int refine_rounds(int range) { return range >= (1 << 16) ? 4 : 1; }
// last window + 1 of round rd, on a grid of `tw` windows
__host__ __device__ __forceinline__ int refine_round_end(int rd, int rounds, int lo, int hi, int tw)
{
    return rd == rounds - 1 ? hi : lo + ((hi - lo) >> (rd ? 3 - rd : 4)) / tw * tw;
}

// Work items of a round: `tiles` candidate tiles times `splits` spans of the round's
// windows (spans on a grid of `grid` windows, the last ones may be empty).  `want`
// splits fill the GPU; beyond that an item is at most about `cap` windows, because
// the CTAs that find no item left wait for the others' with a limit: an item has to
// be a small part of that whatever the series' length.  (tiles * splits fits 31 bits.)
struct RefineItems {
    int splits, span;
};
__host__ __device__ __forceinline__ RefineItems refine_items(int range, int tiles, int want,
                                                             int grid, int cap)
{
    RefineItems I;
    const int fill = want < range / grid ? want : range / grid;
    const int need = (int)(((long long)range + cap - 1) / cap), room = (1 << 30) / tiles;
    I.splits = need > fill ? (need < room ? need : room) : fill;
    if (I.splits < 1) I.splits = 1;
    I.span = (int)((((long long)range + I.splits - 1) / I.splits + grid - 1) / grid * grid);
    return I;
}
// Default limit of the refine's waits in clock cycles, about 2 s.
constexpr long long REFINE_WAIT = 4000000000ll;

__device__ __forceinline__ int32_t ld_acquire(const int32_t *p)
{
    int32_t v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int32_t *p, int32_t v)
{
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Unpruned entries of in[0..C) (or of 0..C-1) to out, in order, by one CTA;
// returns their number.  8 entries per thread and step: the survivors are a few
// thousand at most, and 32k entries take about 15 us.
template <int NT>
__device__ int compact_survivors(const int32_t *in, bool identity, int C, const uint8_t *pruned,
                          int32_t *out, int *wsum)
{
    constexpr int PER = 8;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int base = 0;
    for (int b0 = 0; b0 < C; b0 += NT * PER) {
        const int i0 = b0 + threadIdx.x * PER;
        int e[PER];
        unsigned keep = 0;
#pragma unroll
        for (int q = 0; q < PER; ++q)
            e[q] = i0 + q >= C ? -1 : identity ? i0 + q : __ldcg(in + i0 + q);
#pragma unroll
        for (int q = 0; q < PER; ++q)
            if (e[q] >= 0 && !__ldcg(pruned + e[q])) keep |= 1u << q;
        const int cnt = __popc(keep);
        int inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        __syncthreads(); // wsum of the step before is consumed
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        int off = base, all = 0;
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) {
            const int v = wsum[w];
            if (w < warp) off += v;
            all += v;
        }
        int pos = off + inc - cnt;
#pragma unroll
        for (int q = 0; q < PER; ++q)
            if ((keep >> q) & 1u) out[pos++] = e[q];
        base += all;
    }
    __threadfence();
    return base;
}

// The CTA that compacted round rd's survivors (one thread, after a barrier).
__device__ __forceinline__ void publish_round(PaddiAttemptDev *att, int rd, int count)
{
    att->list_count[rd + 1] = count;
    if (count == 0) att->last_rd = rd + 1;
    __threadfence();
    st_release(&att->round_ready, rd + 1);
}

// The others (one thread): survivors of round rd, or -1 when a CTA gave up or
// the wait ran out after `limit` clock cycles (status 3 is then recorded).
__device__ __forceinline__ int wait_round(PaddiAttemptDev *att, int rd, long long limit)
{
    const long long t0 = clock64();
    while (ld_acquire(&att->round_ready) <= rd) {
        if (ld_acquire(&att->status) == 3) return -1;
        if (clock64() - t0 > limit) {
            atomicExch(&att->status, 3);
            return -1;
        }
        __nanosleep(100);
    }
    return __ldcg(&att->list_count[rd + 1]);
}

} // namespace paddi

// Result of one attempt; the selection writes it to device and to pinned host
// memory.
struct PaddiAttemptResult {
    int64_t n_cand;  // windows with nn >= r2 (never pruned)
    int64_t n_disc;  // windows with nn > r2
    int32_t n_sel;   // discords selected (<= top_k)
    int32_t n_recheck;
    int32_t n_p1;    // candidates after phase 1
    int32_t status;
    int32_t sel_ind[16];
    float sel_dist[16];
    unsigned long long n_pairs; // refine pairs evaluated
    unsigned long long n_live;  // of those, pairs of candidates live at the tile's start
    int32_t p1_walked;          // phase-1 tasks that walked their rows
    int32_t n_fragile;          // windows the refine left to the FP64 fragile pass
    int32_t n_flat;             // flat windows of the length
    int32_t n_unproven;         // windows without a proving witness
    unsigned long long t_prep[PADDI_T_PREP], t[PADDI_T_ATTEMPT]; // time stamps
};
static_assert(sizeof(PaddiAttemptResult) % 4 == 0, "copied in words");

// Incremental FP64 nn of the r policy's bound window (k_guide.cu): the state
// of the shifted dot products G (two buffers), the launch's result, and
// kernel counters.  A zeroed record holds no state (no length is 0).
enum { PADDI_GUIDE_SKIPPED = 0, PADDI_GUIDE_REUSED = 1, PADDI_GUIDE_SLID = 2,
       PADDI_GUIDE_BUILT = 3 };
struct PaddiGuide {
    unsigned long long nn_ord; // result: ordered image of the nn (all ones: none)
    double s;                  // state: shift of both operands of G
    int32_t w, m;              // state: window and length G holds
    int32_t cur, age;          // state: buffer holding G, slides since the last build
    int32_t w_used, mode;      // result: window of the launch (-1: skipped), PADDI_GUIDE_*
    int32_t done, item;        // kernel counters (zero between launches)
    int32_t n_flat;            // host copy only: flat windows of the length
    int32_t pad;
};

// Block maxima of the tensor-core refine: for candidate c and half block h
// (windows [1024 h, 1024 h + 1024)) the largest kept correlation, as an ordered
// image, at v[c * halves + h].  Kept while all candidates of the attempt fit
// (every unpruned candidate meets every block exactly once, so no entry needs
// clearing); the FP64 recheck then scans only half blocks that can hold a
// candidate's nearest neighbour.
struct PaddiBlockMax {
    uint32_t *v;
    int64_t cap; // entries
    int32_t halves;
    __device__ __forceinline__ bool kept(int C) const
    {
        return v != nullptr && (int64_t)C * halves <= cap;
    }
};
#define PADDI_HALF 1024

// Witnesses of a PALMAD run (k_witness.cu): per window a known neighbour
// wit[i] (-1: none; WT_HINT: wc[i] holds a code for partners to evaluate), the
// pair's centred dot product wc[i] at the run's current length, and a lower
// bound wrho[i] of its correlation; scal: WT_AMAX the largest |x| (float bits),
// WT_NHINT and WT_DONE counters of a step (zero between steps).
// Codes: kind * WT_CODE + base, one 8-byte store so that two writers cannot
// tear it: WT_ROW the partners base + {0..3} and base + WT_PARTNER + {0..3},
// WT_COL base - {0..3}, WT_ONE base itself.
struct PaddiWitness {
    int32_t *wit;
    double *wc;
    float *wrho;
    uint32_t *scal;
};
enum { WT_AMAX = 0, WT_NHINT = 1, WT_DONE = 2 };
#define WT_HINT (-2)
#define WT_CODE 8589934592.0 /* 2^33 */
#define WT_PARTNER 128       /* phase 1's partner offset */
enum { WT_ROW = 0, WT_COL = 1, WT_ONE = 2 };

// Records a hint for window i (races between writers leave one of them).
__device__ __forceinline__ void wt_hint(const PaddiWitness &W, int i, int kind, int base)
{
    W.wc[i] = (double)kind * WT_CODE + (double)base;
    W.wit[i] = WT_HINT;
}

#define PADDI_MAX_TOPK 16
#define PADDI_MAX_RECHECK 1024 /* initial FP64 recheck capacity (grows on demand) */

// ---------------------------------------------------------------- launches
// All launch wrappers enqueue on `st` and return cudaGetLastError().
// What the statistics kernel also prepares for the kernels after it (all
// optional): alive[0..N) = 1; `next`, the counters of the next length, zeroed
// (4 ints); the guide's result reset; the time stamp of its start.
struct PaddiStatsExtra {
    uint8_t *alive = nullptr;
    int32_t *next = nullptr;
    PaddiGuide *guide = nullptr;
    unsigned long long *t = nullptr;
};
cudaError_t paddi_launch_stats(const float *x, int64_t n, int32_t m, float4 *wst, float *mu,
                               double2 *ms64, uint8_t *flat,
                               int32_t *flat_count, cudaStream_t st,
                               int32_t *flat_span = nullptr, bool chained = false,
                               const PaddiStatsExtra &extra = PaddiStatsExtra());
// flat_span (optional): two zeroed ints that receive {INT_MAX - lowest flat
// window, highest flat window + 1} (both stay 0 without flat windows).

// Empties the witnesses of a run whose shortest length has N windows.
cudaError_t paddi_launch_witness_start(const float *x, int64_t n, int32_t N, const PaddiWitness &W,
                                       int32_t num_sms, cudaStream_t st);
// What the host counts of a run: its shortest length; how often it has stepped back over
// the value that `returns` of the next step is for (this step included); the sum over the
// values of the squared number of steps taken over each.
struct PaddiWitnessRun {
    int32_t m0, returns;
    double steps2;
};

// Advances the witnesses from length `from` (m - 1, m or m + 1) to m, with the
// statistics of m; hint: scratch, N entries.
cudaError_t paddi_launch_witness_step(const float *x, const double2 *ms64,
                                      int32_t N, int32_t m, int32_t from,
                                      const PaddiWitnessRun &R, const PaddiWitness &W,
                                      int32_t *hint, int32_t num_sms, cudaStream_t st,
                                      unsigned long long *t_end = nullptr);
// Writes alive[0..N) from the witnesses at threshold thr and looks for new
// witnesses of the others (listed in fail) while they are at most `limit`.
cudaError_t paddi_launch_witness_check(const double2 *ms64, const float *x,
                                       int32_t N, int32_t m, float thr,
                                       const PaddiWitnessRun &R, const PaddiWitness &W,
                                       uint8_t *alive, int32_t *fail,
                                       PaddiAttemptDev *att, int32_t limit, int32_t num_sms,
                                       cudaStream_t st);

// Phase 1 at threshold thr = 1 - r^2 / (2m): an exact test (the kernel bounds
// its own FP32 rounding, no guard band).
// Only the rows [row_lo, row_hi) are walked (their columns reach anywhere).
// W (optional): alive[] comes from the witnesses; the kernel returns at once
// when at most `enough` candidates are left (att->n_fail - att->n_rescued),
// walks only segments that hold a candidate, and leaves a hint for every
// candidate it prunes.
cudaError_t paddi_launch_phase1_dev(const float *x, const float4 *wst, const float *mu,
                                    const double2 *ms64, uint8_t *alive, int32_t N, int32_t m,
                                    int32_t R, int32_t max_chunks, float thr, int32_t row_lo,
                                    int32_t row_hi, PaddiAttemptDev *att, int32_t num_sms,
                                    cudaStream_t st, const PaddiWitness *W = nullptr,
                                    int32_t enough = 0);

// reset: alive[] is all ones again when the kernel is done.
// prune_flats (r^2 > 0): flat windows with another flat window at least m-1
// away are dropped (distance 0); flat_span as filled by paddi_launch_stats.
// settle_flats (thr >= 0): the others get their value (correlation 0) and
// pruned = PADDI_SETTLED, which the passes over pairs skip and the selection keeps.
constexpr uint8_t PADDI_SETTLED = 2;
cudaError_t paddi_launch_compact(uint8_t *alive, bool reset, int32_t N, int32_t *cand,
                                 uint32_t *rho_max, uint8_t *pruned, int32_t *rc_slot,
                                 PaddiAttemptDev *att, const uint8_t *flat,
                                 const int32_t *flat_span, int32_t m, bool prune_flats,
                                 bool settle_flats, cudaStream_t st);

// FP32 refine of all att->n_cand_p1 candidates over the windows [col_lo, col_hi)
// (col_lo a multiple of 256), all rounds in one launch; list0 / list1 and
// att->list_count as in paddi_launch_refine_umma.  thr is the exact threshold
// 1 - r^2 / (2m): the kernel prunes on lower bounds of the correlations; gcap
// is the guard band.  W (optional): a pruned candidate leaves the window that
// pruned it as a hint.
cudaError_t paddi_launch_refine_fp32(const float *x, const float4 *wst, const float *mu,
                                     const int32_t *cand, int32_t *list0, int32_t *list1,
                                     PaddiAttemptDev *att, uint32_t *rho_max, uint8_t *pruned,
                                     int32_t N, int32_t m, int32_t col_lo, int32_t col_hi,
                                     float thr, float gcap, int32_t num_sms, cudaStream_t st,
                                     long long wait_cycles = 0, const PaddiWitness *W = nullptr);

// Fragile windows of length m in the FP32 refine's geometry, appended to
// frag_list (frag_count zeroed by the caller).
cudaError_t paddi_launch_fragile_scan_fp32(const float *x, const float4 *wst, const float *mu,
                                           int32_t N, int32_t m, float gcap, int32_t *frag_list,
                                           int32_t *frag_count, int32_t num_sms, cudaStream_t st,
                                           unsigned long long *t_end = nullptr);

// Exact FP64 correlations of the refine's unpruned candidates with the fragile
// windows in [col_lo, col_hi) (k_fragile.cu): prunes and raises rho_max.  The
// candidates are those of the refine's last round att->last_rd (list1 if odd,
// else list0, list_count[last_rd] entries; round 0: all candidates).
cudaError_t paddi_launch_fragile(const float *x, const double2 *ms64, const int32_t *cand,
                                 const int32_t *list0, const int32_t *list1,
                                 PaddiAttemptDev *att, uint8_t *pruned, uint32_t *rho_max, const int32_t *frag,
                                 const int32_t *frag_count, int32_t m, float thr, int32_t col_lo,
                                 int32_t col_hi, int32_t num_sms, cudaStream_t st,
                                 const PaddiBlockMax *B = nullptr, float guard = 0.f);

// Tensor-core refine of all att->n_cand_p1 candidates over the windows
// [col_lo, col_hi) (col_lo a multiple of the tile width, col_hi too or N), all
// rounds in one launch; list0 / list1: scratch, one entry per candidate each;
// att->list_count[r] receives the candidates of round r > 0.  bq / wdq: the
// per-length tile data of paddi_launch_prep.  wait_cycles: limit of every
// wait (<= 0: about 2 s); a wait that runs out sets att->status = 3 and the
// kernel returns.  withhold != 0 is a test hook: the CTA holding work item 0
// never fills that item's first stage, so its waits run out.
cudaError_t paddi_launch_refine_umma(bool bf16, const float *x, const float4 *wst,
                                     const float *mu, const int32_t *cand, int32_t *list0,
                                     int32_t *list1, const uint16_t *bq, const float4 *wdq,
                                     PaddiAttemptDev *att, uint32_t *rho_max, uint8_t *pruned,
                                     int32_t N, int32_t m, int32_t col_lo, int32_t col_hi,
                                     float thr_prune, int32_t num_sms, cudaStream_t st,
                                     long long wait_cycles = 0, int32_t withhold = 0,
                                     bool rows64 = false, const PaddiWitness *W = nullptr,
                                     const PaddiBlockMax *B = nullptr, float guard = 1e-3f);

// Per-length tile data of the tensor-core refine: for every block of
// paddi_tile_width() windows, the split 16-bit series slice (bq, at most
// paddi_tile_block_elems_max() elements per block) and the epilogue's window
// data (wdq, paddi_tile_wd_entries() float4 per block).
int32_t paddi_tile_width();
// The work items of a round of `range` windows and C candidates on `ctas` CTAs.
paddi::RefineItems paddi_refine_items_umma(int32_t m, bool rows64, int32_t C, int32_t range,
                                           int32_t ctas);
paddi::RefineItems paddi_refine_items_fp32(int32_t m, int32_t C, int32_t range, int32_t ctas);
int64_t paddi_tile_blocks(int64_t N);
int64_t paddi_tile_block_elems_max();
int64_t paddi_tile_wd_entries();
// Statistics of length m (as paddi_launch_stats) and the tensor-core refine's
// tile data in one kernel.  flat_count: {flat windows, span (2), fragile
// windows}, zeroed; the fragile windows (bound above gcap) go to frag_list.
cudaError_t paddi_launch_prep(bool bf16, const float *x, int64_t n, int32_t m, float4 *wst,
                              float *mu, double2 *ms64, uint8_t *flat, int32_t *flat_count,
                              uint16_t *bq, float4 *wdq, float gcap, int32_t *frag_list,
                              cudaStream_t st, bool chained, const PaddiStatsExtra &extra,
                              unsigned long long *t_end);

cudaError_t paddi_launch_finalize(const int32_t *cand, PaddiAttemptDev *att,
                                  const uint32_t *rho_max, const uint8_t *pruned, int32_t m,
                                  float r2, float thr, float guard, float widen, int32_t top_k,
                                  const uint8_t *flat, int32_t rc_cap, int32_t *recheck,
                                  int32_t *rc_slot, unsigned long long *nn64_ord,
                                  PaddiAttemptResult *res, int32_t known_w,
                                  unsigned long long known_ord, cudaStream_t st);

cudaError_t paddi_launch_recheck(const float *x, const double2 *ms64,
                                 const uint8_t *flat, int32_t N, int32_t m,
                                 const int32_t *cand, const int32_t *recheck,
                                 PaddiAttemptDev *att, unsigned long long *nn64_ord,
                                 int32_t num_sms, int32_t known_w, cudaStream_t st,
                                 const uint32_t *rho_max, const PaddiBlockMax *B, float guard);

// flat_count: {flat windows, span (2), fragile windows}; next: the state of the
// next attempt, cleared here; host: pinned copy of *res.
cudaError_t paddi_launch_select(const int32_t *cand, PaddiAttemptDev *att,
                                const uint32_t *rho_max, const uint8_t *pruned,
                                const int32_t *recheck, const int32_t *rc_slot,
                                const unsigned long long *nn64_ord, int32_t m, float r2,
                                float thr, float guard, int32_t top_k, const uint8_t *flat,
                                const int32_t *flat_count, const unsigned long long *t_prep,
                                PaddiAttemptDev *next, PaddiAttemptResult *res,
                                PaddiAttemptResult *host, cudaStream_t st);

// with_w: room for the flat-window column data (false only when the length is
// known to have no flat window).
size_t paddi_phase1_smem(int R, int m);

// Exact FP64 nn at length m of window w_host (w_host < 0: the top-1 window
// of the attempt result `prev`, skipped when it has none), through the shifted
// dot products (two buffers G of N doubles each, G + g_stride the second) and
// their state in g; result in g->nn_ord (all ones on entry: paddi_launch_stats
// resets it), copied to pinned memory at `host` with the flat-window count.
cudaError_t paddi_launch_guide(const float *x, const double2 *ms64,
                               const uint8_t *flat, int32_t N, int32_t m,
                               const PaddiAttemptResult *prev, int32_t w_host, PaddiGuide *g,
                               double *G, size_t g_stride, int32_t num_sms, cudaStream_t st,
                               PaddiGuide *host, const int32_t *flat_count,
                               unsigned long long *t);

// Mean and population standard deviation of every window of length m.
cudaError_t paddi_launch_mean_std(const float *x, int64_t n, int32_t m, float *mean, float *sd,
                                  cudaStream_t st);
cudaError_t paddi_launch_export_stats(const double2 *ms64, int32_t N,
                                      int32_t m, float *mean, float *sd, cudaStream_t st);

cudaError_t paddi_launch_scatter(const int32_t *cand, const PaddiAttemptDev *att,
                                 const uint32_t *rho_max, const uint8_t *pruned,
                                 const int32_t *rc_slot, const unsigned long long *nn64_ord,
                                 const uint8_t *flat, int32_t N, int32_t m, float r2,
                                 int32_t *is_cand, float *nnd, cudaStream_t st);

// Learned r predictor (k_mlp.cu).
#define MLP_NFEAT 12
#define MLP_HIDDEN 64
#define MLP_NPARAM (MLP_HIDDEN * MLP_NFEAT + MLP_HIDDEN + MLP_HIDDEN * MLP_HIDDEN + MLP_HIDDEN + MLP_HIDDEN + 1)
cudaError_t paddi_launch_mlp_forward(const float *X, int n, const void *P, bool bf16, float *Y,
                                     cudaStream_t st);
// perm (optional): rows of X and Y to take, in order.
cudaError_t paddi_launch_mlp_grad(const float *X, const float *Y, const uint32_t *perm, int n,
                                  float tau, const float *P, double *G, double *loss, int num_sms,
                                  cudaStream_t st);
// A: 3 * MLP_NPARAM values, zero before step 1.
cudaError_t paddi_launch_mlp_adam(float *P, double *G, double *A, float lr, int step,
                                  cudaStream_t st);
cudaError_t paddi_launch_mlp_to_bf16(const float *P, void *Q, cudaStream_t st);

// True when the tcgen05 split refine can run on `device`; longest m it takes.
// Raises a kernel's dynamic shared-memory limit to at least `bytes` on the
// current device.  The limit is a process-wide attribute of the function, so
// host threads that launch the same kernel with different sizes could lower
// it under one another; here it only grows, under a lock.
cudaError_t paddi_raise_smem_limit(const void *func, size_t bytes);

bool paddi_umma_supported(int device);
int paddi_umma_max_m();
