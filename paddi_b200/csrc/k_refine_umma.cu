// k_refine_umma.cu -- dense candidate refine on tcgen05 tensor cores with
// three-term split 16-bit operands (hi*hi + hi*lo + lo*hi, FP32 accumulate).
//
// Reference: gpu_global_discords_refine (src/PD3_kernels.cuh:582-662), a
// 32x32-tiled FP32 SGEMM of a host-gathered candidate matrix against the
// Hankel windows of the series.  Same contraction here, mapped onto UMMA:
//
//   D[(b,c), a] = sum_k' A[(b,c), k'] * B[a, k']       M = 128, N = 256, K' = m+7 rounded to 16
//   A[(b,c), k'] = zhat_c[k' - b]    (8 shifted copies x 16 candidates, zero padded)
//   B[a, k']     = y[8a + k']        (y = scaled series slice minus a shift)
// so D[(b,c), a] = <zhat_c, y[j .. j+m)> for window j = j0 + 8a + b: one tile
// covers 16 candidates x 2048 windows.
//
// The Hankel operand is never expanded: with SWIZZLE_NONE a K-major core
// matrix is 8 rows of 16 bytes, and the rows of B are 8 elements (16 bytes)
// apart in the series, so the descriptor of B is the raw series slice with
// leading-byte offset 16 and stride-byte offset 128.  The 8 shifts live on
// the candidate side instead, where the operand stays resident for a whole
// work item.
//
// Precision: zhat is normalised (|zhat| = 1) and scaled by 2^8, the slice is
// shifted by x[j0] and scaled by a power of two that puts its largest
// magnitude just below 2^14; both are split into hi + lo 16-bit halves.  The
// rounding of the slice is amplified by |x - shift| / sigma_window, which is
// why FP16 (11-bit mantissa, ~2^-22 per split value) is the default element
// type; BF16 (8-bit mantissa, ~2^-17) is available as the alternative.  The
// epilogue removes the shift exactly with the candidate's sum of split
// values: rho = (D 2^-(8+e) - sum(zhat') (mu_j - shift)) inv_j.
//
// Layout of the work.  Tiles sit on a fixed grid of 2048-window blocks.  Once
// per length, k_prep converts every block's slice into its hi / lo
// halves and its per-window epilogue data (inv_j 2^-(8+e), (mu_j - shift)
// inv_j) in global memory (L2-resident).  The refine is then a pipeline of
// roles inside one persistent CTA per SM, coupled only by mbarriers:
//   * loader (one thread): bulk async copies (cp.async.bulk, no multicast)
//     of the next tiles' slices and window data into a ring of shared-memory
//     stages;
//   * MMA issuer (one thread): 3 x K'/16 tcgen05.mma of 128x256x16 per tile
//     into one of two TMEM accumulators (all 512 columns), then commit;
//   * epilogue (8 warps, four per accumulator, one per TMEM lane quarter):
//     double-buffered tcgen05.ld, rho with packed f32x2 FMAs, running maxima,
//     prune flags.
// Screening.  The three products of a tile are needed to 2e-4, but most tiles
// hold nothing that matters: no correlation above what their live candidates are
// known to reach.  hi * hi alone, a third of the MMAs, is within gc (about 5e-3 on
// the headline series) of the exact value; when its maximum plus that bound stays
// below the best value known of every live candidate (this item's tiles, other
// CTAs' through rho_max, the candidate's witness), the three products and the
// full epilogue are skipped.  A candidate whose lower bound is above thr is pruned
// at once.  Nothing kept is computed with less than all three products.  The MMA
// thread issues tile u+1's hi * hi before it takes the verdict on tile u.  From the
// counts of products and pairs: of 166 thousand tiles of 48357 candidates at n =
// 300007, m = 200, 19 % need everything; of the first attempt's 31 thousand at n = 2^21,
// m = 300, 15 %; of the next ones' thousand to three thousand, 1 to 29 %.  (Times at
// UM_SCREEN_K and EPI_WARP0.)
//
// The candidate operand is built by all 384 threads at the start of a work
// item.  When every candidate of the item is pruned the loader stops and
// sends an end token through the pipeline, so all roles consume the same
// barrier phases.  Every mbarrier wait is bounded; on timeout the kernel
// records status 3, waits (bounded) for its own copies and MMAs, releases
// its TMEM and returns.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <float.h>

#include <cmath>

#include "k_stats.cuh"
#include "paddi_internal.cuh"

using paddi::compact_survivors;
using paddi::f2ord;
using paddi::ord2f;

namespace {

constexpr int UM_THREADS = 384;  // 12 warps
constexpr int UM_TCMAX = 16;     // candidates per tile (M = 128); 8 for M = 64
constexpr int UM_N = 256;        // windows at stride 8
constexpr int UM_TW = UM_N * 8;  // windows per tile (one block of the grid)
constexpr int UM_FEW = 4;        // tiles that take all remaining windows after the first round
// A tile is screened by its hi * hi product first (split-FP16, where the work item
// has several tiles and K' is long enough; the comment at the kernel has the
// figures): refine launches at n = 300007 with tens of thousands of candidates, all
// products at once / screened, us: m = 64 (K' 80) 1770 / 1890, m = 100 (112) 2125 /
// 2120, m = 200 (208) 3715 / 3110, m = 500 (512) 18800 / 10810, m = 700 (720) 27500 /
// 14400; PALMAD 64..512 at 2^21 137 ms / 125.  With one to three tiles an item's first
// tile, which nothing is known about yet, is most of it.  BF16 leaves out 2^-8 of the
// slice: its screen rejects little.
constexpr int UM_SCREEN_T = 4;
constexpr int UM_SCREEN_K = 112;
constexpr int UM_WAVES = 1;      // work items per CTA and round when candidate tiles are few
// An item is at most 2048 tiles of at most some 4e4 cycles each (3 K'/16 products of 128
// cycles, twice that for the rest): 8e7 cycles, a fiftieth of the waits' limit.
constexpr int UM_ITEM = 1 << 22; // windows
__host__ __device__ __forceinline__ paddi::RefineItems um_items(int tiles, int range, int ctas)
{
    return paddi::refine_items(range, tiles, UM_WAVES * ctas / tiles, UM_TW, UM_ITEM);
}
constexpr int UM_KMAX128 = 368;  // largest K' with M = 128 (shared-memory bound)
constexpr int UM_KMAX64 = 736;   // largest K' with M = 64
constexpr int UM_STAGES = 4;      // at most
// barriers for the window data of nw stages: an even number of uses around, so that
// each barrier serves one accumulator's epilogue, which sees all of its phases
constexpr int UM_WBARS = 6;
__host__ __device__ constexpr int wd_bars(int nw) { return nw & 1 ? 2 * nw : nw; }
constexpr int ZSCALE = 8;        // zhat scaled by 2^8 before splitting
constexpr int WD_ROW = 129;      // float4 entries per shift row of the window data (128 + pad)
constexpr int WD_ENTRIES = 8 * WD_ROW;
constexpr int WD_BYTES = WD_ENTRIES * 16;
constexpr uint32_t UM_SMEM_MAX = 227 * 1024 - 1920; // dynamic; the rest is UmShared
// limit of the abort path's drain waits (~2 s at 1.9 GHz): copies and MMAs the
// kernel issued complete on their own, so these waits end long before it
constexpr long long kDrainCycles = 4000000000ll;
// Warps 4..11: epilogue, one group of four per accumulator, so that one group's math
// runs under the other's waits (its product, the screen's verdict): with all eight on
// every tile and candidates major in A (below), refine launches at n = 300007 took 2080
// us at m = 64, now 1770; m = 130 2425, now 2245; ECG of 2^23 points 5.0 ms, now 4.5.
// What bounds it: no unit alone.  At n = 300007, m = 200 (48357 candidates) the tensor
// pipe is active 48 % of the time, L1 and shared memory 35 %, issue slots 25 %; at 31
// thousand tiles (n = 2^21, m = 300) 36, 26 and 15 %.  The rest is waiting: a group for its
// next product, the products for an accumulator (the tensor memory holds two).
constexpr int EPI_WARP0 = 4;
constexpr int EPI_GROUP = 4;     // warps per accumulator
constexpr int MMA_WARP = 0, LOAD_WARP = 1;

__host__ __device__ constexpr int kpad_of(int m) { return ((m + 7) + 15) & ~15; }
__host__ __device__ constexpr int slice_cnt(int kp) { return UM_TW + kp + 16; }
// scratch row stride (32-bit words) of the candidate operand build: 4 words of
// front padding + kp/2 words, rounded up to 2 modulo 32
__host__ __device__ constexpr int zrow_words(int kp)
{
    return (4 + kp / 2) + ((2 - (4 + kp / 2) % 32) + 32) % 32;
}

// ------------------------------------------------------------------ PTX helpers
__device__ __forceinline__ uint32_t smem_u32(const void *p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for the completion of the phase with the given parity;
// false when `limit` clock cycles passed first.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, long long limit)
{
    if (mbar_try_wait(bar, parity)) return true; // mostly: no clock is read then
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity))
        if (clock64() - t0 > limit) return false;
    return true;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

// Bulk async copy global -> this CTA's shared memory (no multicast), completing
// `bytes` transaction bytes on bar.  dst, src 16-byte aligned; bytes % 16 == 0.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], "
                 "%2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Shared-memory matrix descriptor, SWIZZLE_NONE, K-major, sm100 version bits.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor: kind::f16, D = F32, A/B = fmt (0 F16, 1 BF16), K-major, M, N.
__host__ __device__ constexpr uint32_t idesc_f16(uint32_t fmt, int M, int N)
{
    return (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
        ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u),
        "r"(0u)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

// tcgen05.ld without the wait, and a wait that is tied to the destination
// registers (so no use of them can be scheduled before it).
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[32])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
                 "[%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                   "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
                   "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
                   "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[32])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                   "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                   "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                   "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                   "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                   "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}

// max(a, b, c) in one instruction (sm_100 three-input form)
__device__ __forceinline__ float fmax3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// ------------------------------------------------------------------ element types
template <bool BF> struct E16;
template <> struct E16<false> {
    using T = __half;
    static constexpr uint32_t fmt = 0;
    static constexpr float uh = 4.8828125e-4f; // 2^-11: relative rounding of a half
    __device__ static __half cvt(float v) { return __float2half_rn(v); }
    __device__ static float back(__half v) { return __half2float(v); }
};
template <> struct E16<true> {
    using T = __nv_bfloat16;
    static constexpr uint32_t fmt = 1;
    static constexpr float uh = 3.90625e-3f; // 2^-8
    __device__ static __nv_bfloat16 cvt(float v) { return __float2bfloat16_rn(v); }
    __device__ static float back(__nv_bfloat16 v) { return __bfloat162float(v); }
};

// ------------------------------------------------------------------ tile prep
// Block b (windows [2048 b, 2048 b + 2048)): slice x[j0 .. j0 + cnt) minus
// its level s, scaled by 2^e (largest magnitude just below 2^14), split
// into hi and lo halves: bq[b * 2cnt ...] = hi, then lo.  Window data for the
// epilogue in its read layout: shift row s = q % 8, column pair k = q / 16,
// slot = (q / 8) % 2: wd[s * 129 + k] = {a(slot 0), a(slot 1), b(slot 0), b(slot 1)}
// with a = inv_j 2^-(8+e) and b = (mu_j - s) inv_j (zero past N).
// Rounding bound: window j's correlations carry at most g_j = window_bound()
// (E A_j + F inv_j); g_j grows with |mu_j - s| / |x_j - mu_j|.  The level s
// is the mean of the block's window means weighted by 1 / |x_j - mu_j|^2 (it
// minimises the sum of (mu_j - s)^2 / |x_j - mu_j|^2, so the low-variance
// windows, where the amplification is large, pull it towards their level);
// the slice's midrange if no window has a norm.  A window with g_j > gcap is
// "fragile": its a is NaN
// (the epilogue's maxima skip it) and it is appended to frag_list, whose
// pairs are evaluated in FP64 later.  The largest g_j of the block's other
// windows, G, is stored in the padding entry wd[128].x: the epilogue
// subtracts it from every correlation of the tile (a lower bound that is safe
// to prune on) and adds it back to the maxima it keeps (the middle of the
// interval, within gcap of every true value).
// The statistics of the length come out of the same kernel: a block's windows
// are a statistics tile, so the staged series and the windows' means and norms
// are used where they are, in shared memory and registers.  As two kernels (the
// second one re-reading 20 B a window) they took 34 us a length at n = 1500007,
// m = 300, as one 25; headline run 168 -> 153 ms.
// Four CTAs per SM (64 registers, 22 bytes of shared memory per staged value: m <= 470):
// a length of 2^21 windows is 1025 blocks, two waves instead of three; 37 us at m = 256
// with three, now 31.
static_assert(ST_TILE == UM_TW, "a statistics tile is a block of the refine's grid");

template <bool BF>
__global__ void __launch_bounds__(ST_THREADS, 4)
k_prep(const float *__restrict__ x, int64_t nser, int32_t cnt, int32_t m, int32_t N, StOut O,
       uint16_t *bq, float4 *wdq, float E, float Fu, float gcap,
       int32_t *frag_list, int32_t *frag_count, unsigned long long *t_end)
{
    using X = E16<BF>;
    extern __shared__ __align__(16) unsigned char st_mem[];
    __shared__ StShared S;
    __shared__ float red[4][ST_THREADS / 32];
    st_begin(O.extra);
    const int b = blockIdx.x;
    const int64_t j0 = (int64_t)b * UM_TW;
    const StTile T = st_prefix(st_mem, S, x, nser, m, j0);
    float iv[ST_WPT], mv[ST_WPT]; // zero past N
    st_write(T, O, j0, m, N, iv, mv);
    if (j0 >= N) { // the zeroed tail holds no tile
        if (threadIdx.x == 0) paddi::stamp_end(t_end);
        return;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // the slice reaches a few values past what is staged
    const int staged = ST_TILE + m + 1;
    auto val = [&](int p) { return p < staged ? T.xs[p] : x[j0 + p]; };
    float sw = 0.f, swm = 0.f; // sums of 1/|x_j - mu_j|^2 and mu_j/|x_j - mu_j|^2
#pragma unroll
    for (int k = 0; k < ST_WPT; ++k)
        if (j0 + threadIdx.x + ST_THREADS * k < N) {
            const float wgt = fminf(iv[k] * iv[k], 1e30f);
            sw += wgt;
            swm = fmaf(wgt, mv[k], swm);
        }
    float lo_v = INFINITY, hi_v = -INFINITY;
    for (int p = threadIdx.x; p < cnt; p += ST_THREADS) {
        if (j0 + p < nser) {
            const float v = val(p);
            lo_v = fminf(lo_v, v);
            hi_v = fmaxf(hi_v, v);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo_v = fminf(lo_v, __shfl_xor_sync(0xffffffffu, lo_v, o));
        hi_v = fmaxf(hi_v, __shfl_xor_sync(0xffffffffu, hi_v, o));
        sw += __shfl_xor_sync(0xffffffffu, sw, o);
        swm += __shfl_xor_sync(0xffffffffu, swm, o);
    }
    if (lane == 0) {
        red[0][w] = lo_v;
        red[1][w] = hi_v;
        red[2][w] = sw;
        red[3][w] = swm;
    }
    __syncthreads();
    lo_v = INFINITY;
    hi_v = -INFINITY;
    sw = 0.f;
    swm = 0.f;
#pragma unroll
    for (int k = 0; k < ST_THREADS / 32; ++k) {
        lo_v = fminf(lo_v, red[0][k]);
        hi_v = fmaxf(hi_v, red[1][k]);
        sw += red[2][k];
        swm += red[3][k];
    }
    __syncthreads();
    float sh = 0.5f * lo_v + 0.5f * hi_v; // midrange (j0 < nser always)
    if (sw > 0.f) {
        const float lv = swm / sw; // the weighted level, kept inside the slice's range
        if (isfinite(lv)) sh = fminf(fmaxf(lv, lo_v), hi_v);
    }
    const float mx = fmaxf(fabsf(hi_v - sh), fabsf(lo_v - sh));
    int e = 0;
    if (mx > 0.f) {
        int ex;
        frexpf(mx, &ex); // mx = f * 2^ex, f in [0.5, 1)
        e = 14 - ex;     // mx * 2^e < 2^14
        e = max(-100, min(100, e));
    }
    const float sc = ldexpf(1.f, e);
    const float dsc = ldexpf(1.f, -(ZSCALE + e));
    uint32_t *hi = reinterpret_cast<uint32_t *>(bq + (size_t)b * 2 * cnt);
    uint32_t *lo = reinterpret_cast<uint32_t *>(bq + (size_t)b * 2 * cnt + cnt);
    for (int p2 = threadIdx.x; p2 < cnt / 2; p2 += ST_THREADS) {
        const int64_t g = j0 + 2 * p2;
        const float u0 = (g < nser ? val(2 * p2) - sh : 0.f) * sc;
        const float u1 = (g + 1 < nser ? val(2 * p2 + 1) - sh : 0.f) * sc;
        const typename X::T h0 = X::cvt(u0), h1 = X::cvt(u1);
        const typename X::T l0 = X::cvt(u0 - X::back(h0)), l1 = X::cvt(u1 - X::back(h1));
        hi[p2] = (uint32_t)reinterpret_cast<const uint16_t &>(h0) |
                 ((uint32_t)reinterpret_cast<const uint16_t &>(h1) << 16);
        lo[p2] = (uint32_t)reinterpret_cast<const uint16_t &>(l0) |
                 ((uint32_t)reinterpret_cast<const uint16_t &>(l1) << 16);
    }
    // built in shared memory (the prefixes are done with), written out in one sweep
    float *wf = reinterpret_cast<float *>(st_mem);
    const float F = Fu * mx, fm = (float)m;
    float gmax = 0.f, amax = 1.f;
#pragma unroll
    for (int kq = 0; kq < ST_WPT; ++kq) {
        const int q = threadIdx.x + ST_THREADS * kq;
        const int64_t j = j0 + q;
        const float g = paddi::window_bound(iv[kq], mv[kq], sh, fm, E, F);
        const bool frag = j < N && g > gcap;
        if (!frag) {
            gmax = fmaxf(gmax, g);
            const float bb = (mv[kq] - sh) * iv[kq];
            amax = fmaxf(amax, sqrtf(fmaf(fm * bb, bb, 1.f)) * 1.0001f);
        }
        const int s = q & 7, i = q >> 3, k = i >> 1, slot = i & 1;
        const float a = frag ? __int_as_float(0x7fffffff) : iv[kq] * dsc;
        wf[(s * WD_ROW + k) * 4 + slot] = a;
        wf[(s * WD_ROW + k) * 4 + 2 + slot] = (mv[kq] - sh) * iv[kq];
        // fragile windows in index order within each warp (runs stay contiguous)
        const unsigned bal = __ballot_sync(0xffffffffu, frag);
        if (bal) {
            int base = 0;
            if (lane == 0) base = atomicAdd(frag_count, __popc(bal));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (frag) frag_list[base + __popc(bal & ((1u << lane) - 1u))] = (int32_t)j;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gmax = fmaxf(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    }
    if (lane == 0) {
        red[0][w] = gmax;
        red[1][w] = amax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float G = 0.f, A = 1.f;
        for (int k = 0; k < ST_THREADS / 32; ++k) {
            G = fmaxf(G, red[0][k]);
            A = fmaxf(A, red[1][k]);
        }
        wf[(0 * WD_ROW + 128) * 4] = G; // padding entry of shift row 0
        wf[(0 * WD_ROW + 128) * 4 + 1] = A;
    }
    __syncthreads();
    const float4 *src = reinterpret_cast<const float4 *>(st_mem);
    for (int k = threadIdx.x; k < WD_ENTRIES; k += ST_THREADS) wdq[(size_t)b * WD_ENTRIES + k] = src[k];
    if (threadIdx.x == 0) paddi::stamp_end(t_end);
}

// ------------------------------------------------------------------ shared memory
struct UmLayout {
    uint32_t a_hi, a_lo, b[UM_STAGES][2], wd[UM_STAGES], bytes;
    int nb, nw; // stages of slices and of window data
};

// As many stages as fit, up to 4, of a slice and its window data each (K' = 208: 4,
// 320: 2), so that a tile's data are requested that many tiles ahead: refine
// launches of an ECG series of 2^23 points 8.2 -> 7.0 ms, m = 64 at n = 300007 2.18 ->
// 2.09 ms.  The largest K' have room for two slices and one set of window data.
__host__ __device__ inline UmLayout um_layout(int MM, int kp)
{
    UmLayout L;
    const uint32_t a_bytes = (uint32_t)MM * kp * 2;
    const uint32_t b_bytes = (uint32_t)slice_cnt(kp) * 2; // multiple of 32
    L.a_hi = 0;
    L.a_lo = a_bytes;
    const int fit = (int)((UM_SMEM_MAX - 2 * a_bytes) / (2 * b_bytes + WD_BYTES));
    L.nb = fit >= UM_STAGES ? UM_STAGES : fit >= 2 ? fit : 2;
    L.nw = fit >= 2 ? L.nb : 1;
    // slice 0, the window data, the other slices: without slice 0, or without the
    // last one, enough contiguous room is left for the operand build's scratch
    uint32_t o = 2 * a_bytes;
    for (int s = 0; s < UM_STAGES; ++s) {
        if (s < L.nb)
            for (int h = 0; h < 2; ++h) {
                L.b[s][h] = o;
                o += b_bytes;
            }
        if (s == 0)
            for (int q = 0; q < UM_STAGES; ++q) {
                L.wd[q] = o;
                if (q < L.nw) o += WD_BYTES;
            }
    }
    L.bytes = o;
    return L;
}

struct UmShared {
    // rings over the stages (full, empty) and over the two accumulators
    uint64_t full_b[UM_STAGES];   // loader -> MMA: the stage holds the tile's slice (or an end token)
    uint64_t wd_full[UM_WBARS];   // loader -> epilogue: and its window data (or an end token)
    uint64_t sl_empty[UM_STAGES]; // epilogue -> loader: done with the slice
    uint64_t wd_empty[UM_STAGES]; // epilogue -> loader: done with the window data
    uint64_t mma_done[2];  // tcgen05.commit: the tile's MMAs are complete
    uint64_t acc_empty[2]; // epilogue -> MMA: accumulator drained
    uint64_t dec[2];       // epilogue -> MMA: hi * hi product screened, need[] decided
    uint64_t rest_done[2]; // tcgen05.commit: a screened tile's three products are complete
    uint64_t put[2];       // epilogue: a fully multiplied tile's block maxima are in bmax
    uint64_t drain;        // final MMA drain on abort
    // phase of the last arrival the loader issued on full_b[s] / wd_full[s] (-1: none
    // yet); the abort path waits only for those
    signed char last_full[UM_STAGES], last_wd[UM_WBARS];
    uint32_t tmem_base;
    int item, abort, tok;
    int built_tile; // candidate tile whose operand sits in A (-1: none)
    int last, next; // round bookkeeping: this CTA finished the round's last item;
                    // candidates of the next round (-1: give up)
    int wsum[UM_THREADS / 32];
    volatile int item_dead;
    volatile uint8_t vb[UM_STAGES], vw[UM_WBARS];
    int cw[UM_TCMAX], cp[UM_TCMAX];
    float cflat[UM_TCMAX], zsum[UM_TCMAX];
    // screening: sum of the hi halves, norm of what they leave out, a correlation
    // the candidate is known to reach; need[s]: tag of the last tile in accumulator
    // s that needs all its products
    float zsumh[UM_TCMAX], zrest[UM_TCMAX];
    volatile uint32_t known[UM_TCMAX]; // (ordered image)
    volatile uint32_t need[2];
    float bmax[2][4][2][UM_TCMAX]; // half-block maxima per accumulator and warp
    uint32_t rmax[UM_TCMAX];
    volatile uint8_t dead[UM_TCMAX];
};

static_assert(sizeof(UmShared) <= 1920, "beside the largest operand and window data");

// The n-th use of a ring of `stages` barriers: its barrier and phase parity.  Every
// tile (and every end token) of a CTA takes one use of every ring, so one count
// over the CTA's work items serves them all.
struct Ring {
    int s;
    uint32_t par;
    __device__ __forceinline__ Ring(uint32_t n, int stages)
        : s((int)(n % (uint32_t)stages)), par((n / (uint32_t)stages) & 1u)
    {
    }
};

// MM = 128: 16 candidates, accumulator row r in TMEM lane r.
// MM = 64:  8 candidates, accumulator row r in TMEM lane (r % 16) + 32 (r / 16)
//           (lanes 16..31 of every subpartition stay unused).
template <bool BF, int MM>
__global__ void __launch_bounds__(UM_THREADS, 1)
k_refine_umma(const float *__restrict__ x, const float4 *wst,
              const float *mu, const int32_t *cand, int32_t *list0,
              int32_t *list1, const uint16_t *bq, const float4 *wdq,
              PaddiAttemptDev *att, uint32_t *rho_max, uint8_t *pruned, int32_t N, int32_t m,
              int32_t col_lo, int32_t col_hi, float thr, int32_t grid_ctas, long long wl,
              int32_t withhold, PaddiWitness W, PaddiBlockMax B, int32_t may_screen, float guard)
{
    using X = E16<BF>;
    constexpr int UM_M = MM;
    constexpr int UM_TC = MM / 8;
    constexpr int RG = MM / 8;          // 8-row core-matrix groups of A
    extern __shared__ __align__(128) unsigned char um_smem[];
    __shared__ UmShared S;
    const int kp = kpad_of(m);
    const int cnt = slice_cnt(kp);
    const UmLayout L = um_layout(MM, kp);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    paddi::chain_begin();
    paddi::stamp_begin(att->t + PADDI_T_REFINE_B);
    int C = att->n_cand_p1;
    if (C <= 0 || col_hi <= col_lo) { // uniform, before any TMEM use
        paddi::stamp_begin(att->t + PADDI_T_REFINE_E);
        return;
    }
    const bool bkeep = B.kept(C);

    if (threadIdx.x == 0) {
        for (int s = 0; s < UM_STAGES; ++s) {
            mbar_init(&S.full_b[s], 1);
            mbar_init(&S.sl_empty[s], EPI_GROUP);
            mbar_init(&S.wd_empty[s], EPI_GROUP);
            S.last_full[s] = -1;
        }
        for (int s = 0; s < UM_WBARS; ++s) {
            mbar_init(&S.wd_full[s], 1);
            S.last_wd[s] = -1;
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&S.mma_done[s], 1);
            mbar_init(&S.acc_empty[s], EPI_GROUP);
            mbar_init(&S.dec[s], EPI_GROUP);
            mbar_init(&S.rest_done[s], 1);
            mbar_init(&S.put[s], EPI_GROUP);
            S.need[s] = 0;
        }
        mbar_init(&S.drain, 1);
        S.abort = 0;
        S.last = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&S.tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    uint32_t G = 0; // tiles and end tokens of this CTA before the current work item
    bool mma_issued = false; // MMA thread: any MMA issued
    uint32_t n_rest = 0u, n_put = 0u; // epilogue: completed phases of its rest_done and put

    const uint32_t idesc = idesc_f16(X::fmt, UM_M, UM_N);
    const uint32_t a_hi_s = smem_u32(um_smem + L.a_hi), a_lo_s = smem_u32(um_smem + L.a_lo);
    const int kblocks = kp / 16;
    // epilogue geometry: lane group g (TMEM lanes 32g..32g+31)
    const int g = warp & 3, grp = (warp - EPI_WARP0) >> 2; // lane quarter, accumulator
    const bool rowok = MM == 128 || lane < 16;
    const int row = MM == 128 ? 32 * g + lane : 16 * g + (lane & 15);
    const int cidx = row % UM_TC, bsh = row / UM_TC; // candidate, shift

    // ---- rounds: the windows [jb, je) of growing ranges (1/16, 1/4, 1/2, all of
    // them), the survivors compacted in between so that every tile is dense.  A
    // round with one tile left takes every remaining window.
    const int nrounds = paddi::refine_rounds(col_hi - col_lo);
    int jb = col_lo;
    for (int rd = 0; rd < nrounds; ++rd) {
        int je = paddi::refine_round_end(rd, nrounds, col_lo, col_hi, UM_TW);
        // one tile left, or a few after the first round: a further round (about 15 us:
        // operand builds, the wait, a last wave) costs more than it could save
        if (C <= (rd == 0 ? 1 : UM_FEW) * UM_TC) je = col_hi;
        int32_t *list = rd & 1 ? list1 : list0; // entries of this round (round 0: all candidates)
        const int range = je - jb;
        const int tiles = (C + UM_TC - 1) / UM_TC;
        // at most UM_WAVES items per CTA when the candidate tiles are few, items of
        // at least one 2048-window block
        const paddi::RefineItems I = um_items(tiles, range, grid_ctas);
        const int splits = I.splits, span = I.span;
        const int total = tiles * splits;
        if (threadIdx.x == 0) S.built_tile = -1;
        bool counted = true; // this CTA's latest item is in done_rd
        for (;;) {
            if (threadIdx.x == 0) {
                // everything this CTA wrote for its item is ordered before the count (the
                // barrier at the item's end, then the fence)
                if (!counted) {
                    __threadfence();
                    S.last = atomicAdd(&att->done_rd[rd], 1) == total - 1;
                }
                S.item = atomicAdd(&att->work_rd[rd], 1);
            }
            counted = false;
            __syncthreads();
            const int item = S.item;
            if (item >= total) break;
            const int tile = item % tiles, split = item / tiles;
            const int j_lo = jb + split * span, j_hi = min(je, j_lo + span);
            if (threadIdx.x < UM_TC) {
                const int li = tile * UM_TC + threadIdx.x;
                const bool v = li < C;
                const int pos = !v ? 0 : rd ? __ldcg(list + li) : li;
                const int w = v ? cand[pos] : -1; // -1: no candidate in this row
                S.cw[threadIdx.x] = w;
                S.cp[threadIdx.x] = pos;
                S.dead[threadIdx.x] = !v || __ldcg(pruned + pos);
                S.cflat[threadIdx.x] = (v && wst[w].z == 0.f) ? 1.f : 0.f; // flat candidate
                S.rmax[threadIdx.x] = f2ord(-INFINITY);
                // a correlation this candidate reaches, from its witness (the kept value
                // of that window is within the guard band of it)
                S.known[threadIdx.x] = f2ord(
                    (v && W.wit) ? fmaxf(W.wrho[w] - guard - 1e-5f, -INFINITY) : -INFINITY);
            }
            if (threadIdx.x == 0) {
                S.item_dead = 0;
                S.tok = -1;
            }
            __syncthreads();
            {
                int a = threadIdx.x < UM_TC ? !S.dead[threadIdx.x] : 0;
                if (!__syncthreads_or(a) || j_lo >= j_hi) continue; // all threads agree
            }
            const int T = (j_hi - j_lo + UM_TW - 1) / UM_TW;
            const bool screen = may_screen && T >= UM_SCREEN_T;
            const int blk0 = j_lo / UM_TW; // j_lo is a multiple of UM_TW
            // the slice of tile u (its stage is free) or an end token
            auto put_slice = [&](int u, bool token) {
                const Ring r(G + (uint32_t)u, L.nb);
                S.last_full[r.s] = (signed char)r.par;
                S.vb[r.s] = !token;
                if (token) {
                    mbar_arrive(&S.full_b[r.s]);
                    return;
                }
                const uint16_t *src = bq + (size_t)(blk0 + u) * 2 * cnt;
                mbar_arrive_expect_tx(&S.full_b[r.s], (uint32_t)(4 * cnt));
                bulk_g2s(um_smem + L.b[r.s][0], src, (uint32_t)(2 * cnt), &S.full_b[r.s]);
                bulk_g2s(um_smem + L.b[r.s][1], src + cnt, (uint32_t)(2 * cnt), &S.full_b[r.s]);
            };
            // the first tile's slice streams in while the operand is built (the build's
            // scratch lies clear of its stage)
            const int stage0 = Ring(G, L.nb).s;
            if (warp == LOAD_WARP && lane == 0) {
                // test hook (withhold != 0): the CTA holding work item 0 never fills
                // its first stage, so the MMA thread's wait runs out; nothing is in flight
                S.vb[stage0] = 1;
                if (!(withhold && rd == 0 && item == 0)) put_slice(0, false);
            }
            // ---- candidate operand: 16 x (hi, lo) rows of scaled zhat, then 8 shifted
            //      copies; kept from the CTA's previous item when that had the same
            //      candidate tile (a candidate pruned since then only costs its rows'
            //      work: its results no longer matter)
            if (S.built_tile != tile) {
                // scratch rows of 32-bit words: 4 zero words (8 elements) of front
                // padding, then zhat[0..kp); stride ksw words with ksw % 32 == 2, so
                // the 16 candidates and two shifts a warp reads sit in different banks
                const int ksw = zrow_words(kp);
                uint32_t *zhw = reinterpret_cast<uint32_t *>(um_smem + (L.nw >= 2 || stage0 == 0 ? L.wd[0] : L.b[0][0]));
                uint32_t *zlw = zhw + UM_TC * ksw;
                typename X::T *zh = reinterpret_cast<typename X::T *>(zhw);
                typename X::T *zl = reinterpret_cast<typename X::T *>(zlw);
                const int c = threadIdx.x >> 4, t16 = threadIdx.x & 15;
                const int w = c < UM_TC ? S.cw[c] : 0;
                const bool live = c < UM_TC && !S.dead[c];
                const float muc = live ? mu[w] : 0.f;
                const float ivc = live ? wst[w].z * 256.f : 0.f; // 2^ZSCALE
                float zs = 0.f, zsh = 0.f, zr = 0.f;
                if (c < UM_TC)
                    for (int q = 4 + (kp >> 1) + t16; q < ksw; q += 16) { // tail words
                        zhw[c * ksw + q] = 0u;
                        zlw[c * ksw + q] = 0u;
                    }
                if (c < UM_TC && t16 < 4) { // front padding
                    zhw[c * ksw + t16] = 0u;
                    zlw[c * ksw + t16] = 0u;
                }
#pragma unroll 4
                for (int k = t16; k < kp; k += 16) {
                    const float v = (live && k < m) ? (x[w + k] - muc) * ivc : 0.f;
                    const typename X::T h = X::cvt(v);
                    const typename X::T l = X::cvt(v - X::back(h));
                    if (c < UM_TC) {
                        zh[c * 2 * ksw + 8 + k] = h;
                        zl[c * 2 * ksw + 8 + k] = l;
                    }
                    const float hb = X::back(h), rs = v - hb;
                    zs += hb + X::back(l);
                    zsh += hb;
                    zr = fmaf(rs, rs, zr);
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) {
                    zs += __shfl_xor_sync(0xffffffffu, zs, o);
                    zsh += __shfl_xor_sync(0xffffffffu, zsh, o);
                    zr += __shfl_xor_sync(0xffffffffu, zr, o);
                }
                if (t16 == 0 && c < UM_TC) {
                    S.zsum[c] = zs * (1.f / 256.f);
                    S.zsumh[c] = zsh * (1.f / 256.f);
                    S.zrest[c] = sqrtf(zr) * (1.01f / 256.f);
                }
                __syncthreads();
                // A[(b,c), k'] = z_c[k' - b] in K-major core matrices, the shift b major: an
                // epilogue warp then works on two shifts, and its reads of the window data go
                // to two addresses (with candidates major, eight: a 16-byte read took 4 cycles
                // of shared memory, now 2):
                // byte offset ((k'/8)*RG + r/8)*128 + (r%8)*16 + (k'%8)*2.
                // Elements k'-b .. k'-b+7 start at padded element p0 = 8 + 8 kc - b:
                // five 32-bit words from word p0/2, funnel-shifted by 16 bits when p0 is odd.
                const int chunks = kp / 8;
                for (int e = threadIdx.x; e < UM_M * chunks; e += UM_THREADS) {
                    const int r = e & (UM_M - 1), kc = e / UM_M;
                    const int cc = r % UM_TC, b = r / UM_TC;
                    const int p0 = 8 + 8 * kc - b;
                    const uint32_t shf = (uint32_t)(p0 & 1) * 16u;
                    const uint32_t *rh = zhw + cc * ksw + (p0 >> 1);
                    const uint32_t *rl = zlw + cc * ksw + (p0 >> 1);
                    uint32_t wh[5], wl[5], ph2[4], pl2[4];
#pragma unroll
                    for (int q = 0; q < 5; ++q) {
                        wh[q] = rh[q];
                        wl[q] = rl[q];
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        ph2[q] = __funnelshift_r(wh[q], wh[q + 1], shf);
                        pl2[q] = __funnelshift_r(wl[q], wl[q + 1], shf);
                    }
                    const uint32_t off = (uint32_t)((kc * RG + (r >> 3)) * 128 + (r & 7) * 16);
                    *reinterpret_cast<uint4 *>(um_smem + L.a_hi + off) =
                        make_uint4(ph2[0], ph2[1], ph2[2], ph2[3]);
                    *reinterpret_cast<uint4 *>(um_smem + L.a_lo + off) =
                        make_uint4(pl2[0], pl2[1], pl2[2], pl2[3]);
                }
                fence_proxy_async_smem(); // A for the tensor core; scratch for the bulk copies
                __syncthreads();
                if (threadIdx.x == 0) S.built_tile = tile; // read after the next item's barrier
            }

            // ================================================================ roles
            if (warp == LOAD_WARP && lane == 0) {
                // the use `before` uses ago of a stage must be consumed (uses of earlier
                // items are)
                auto freed = [&](uint64_t *empty, int u, int stages) -> bool {
                    if (G + (uint32_t)u < (uint32_t)stages) return true;
                    const Ring r(G + (uint32_t)u - (uint32_t)stages, stages);
                    return mbar_wait_bounded(empty + r.s, r.par, wl);
                };
                auto put_wd = [&](int u, bool token) {
                    const uint32_t n = G + (uint32_t)u;
                    const Ring r(n, wd_bars(L.nw));
                    S.last_wd[r.s] = (signed char)r.par;
                    S.vw[r.s] = !token;
                    if (token) {
                        mbar_arrive(&S.wd_full[r.s]);
                        return;
                    }
                    mbar_arrive_expect_tx(&S.wd_full[r.s], (uint32_t)WD_BYTES);
                    bulk_g2s(um_smem + L.wd[Ring(n, L.nw).s], wdq + (size_t)(blk0 + u) * WD_ENTRIES,
                             (uint32_t)WD_BYTES, &S.wd_full[r.s]);
                };
                // once the item is dead, end tokens take the place of the next two tiles (one
                // per accumulator)
                bool ok = freed(S.wd_empty, 0, L.nw);
                if (ok) put_wd(0, false); // slice 0 was issued before the operand build
                int tok = -1;
                for (int u = 1; ok && u < T && (tok < 0 || u == tok + 1); ++u) {
                    ok = freed(S.sl_empty, u, L.nb);
                    if (!ok) break;
                    const bool token = tok >= 0 || S.item_dead;
                    if (token && tok < 0) S.tok = tok = u;
                    put_slice(u, token);
                    ok = freed(S.wd_empty, u, L.nw);
                    if (ok) put_wd(u, token);
                }
                if (!ok) S.abort = 1;
            } else if (warp == MMA_WARP && lane == 0) {
                // products of tile u: hi * hi, or all three
                auto issue = [&](int u, bool all) {
                    const uint32_t n = G + (uint32_t)u;
                    const int st = Ring(n, L.nb).s;
                    tc_fence_after();
                    const uint32_t d = tmem + (n & 1u) * UM_N;
                    const uint32_t bh = smem_u32(um_smem + L.b[st][0]);
                    const uint32_t bl = smem_u32(um_smem + L.b[st][1]);
                    // K-block kb = core-matrix columns 2kb, 2kb+1; LBO = next K column of cores.
                    // The descriptors' address fields (16-byte units) just step along K
                    uint64_t ah = sdesc(a_hi_s, RG * 128, 128), al = sdesc(a_lo_s, RG * 128, 128);
                    uint64_t bhd = sdesc(bh, 16, 128), bld = sdesc(bl, 16, 128);
                    constexpr uint64_t da = 2 * RG * 128 / 16, db = 32 / 16;
                    if (!all) {
#pragma unroll 4
                        for (int kb = 0; kb < kblocks; ++kb, ah += da, bhd += db)
                            umma_f16(d, ah, bhd, idesc, kb > 0 ? 1u : 0u);
                    } else {
                        for (int kb = 0; kb < kblocks; ++kb, ah += da, al += da, bhd += db, bld += db) {
                            umma_f16(d, ah, bhd, idesc, kb > 0 ? 1u : 0u);
                            umma_f16(d, ah, bld, idesc, 1u);
                            umma_f16(d, al, bhd, idesc, 1u);
                        }
                    }
                    mma_issued = true;
                };
                // the screen's verdict on tile u (its own products may still be wanted)
                auto settle = [&](int u) -> bool {
                    const Ring a(G + (uint32_t)u, 2);
                    if (!mbar_wait_bounded(&S.dec[a.s], a.par, wl)) return false;
                    if (S.need[a.s] == G + (uint32_t)u + 1u) {
                        // all three from zero, block by block of K as without the screen: the
                        // two small ones on top of a finished hi * hi would be rounded at the
                        // full sum's size every time (kept correlations at m = 200: 7.9e-7
                        // rms from FP64 instead of 6.2e-7).  The product that is done
                        // twice is 7 % of a refine of many candidates, 1 % of PALMAD
                        issue(u, true);
                        umma_commit(&S.rest_done[a.s]);
                    }
                    return true;
                };
                bool ok = true, ended = false;
                for (int u = 0; ok && u < T; ++u) {
                    const uint32_t n = G + (uint32_t)u;
                    const Ring r(n, L.nb), a(n, 2);
                    if (!mbar_wait_bounded(&S.full_b[r.s], r.par, wl)) {
                        ok = false;
                        break;
                    }
                    // the accumulator's previous tile must be drained first, also before an
                    // end token: its commit completes a phase of mma_done that the epilogue
                    // may still be waiting on for that tile
                    if (n >= 2u && !mbar_wait_bounded(&S.acc_empty[a.s], Ring(n - 2u, 2).par, wl)) {
                        ok = false;
                        break;
                    }
                    if (!S.vb[r.s]) { // end token: pass it on (the commit also covers earlier MMAs)
                        if (screen && u > 0 && !ended) ok = settle(u - 1);
                        umma_commit(&S.mma_done[a.s]);
                        if (ended) break;
                        ended = true;
                        continue;
                    }
                    issue(u, !screen);
                    umma_commit(&S.mma_done[a.s]);
                    // the tile before was screened while this one's product started
                    if (screen && u > 0) ok = settle(u - 1);
                }
                if (ok && screen && !ended) ok = settle(T - 1);
                if (!ok) S.abort = 1;
            } else if (warp >= EPI_WARP0) {
                float rmax = -INFINITY;
                const int wc = S.cw[cidx];
                const float zsc = S.zsum[cidx], fc = S.cflat[cidx];
                const float zsh = S.zsumh[cidx], zrest = S.zrest[cidx];
                const float rsm = rsqrtf((float)m) * 1.001f;
                // tiles of the item and their live candidates (instrumentation)
                int n_tiles = 0, n_alive = 0;
                int alive = __popc(__ballot_sync(0xffffffffu, lane < UM_TC && !S.dead[lane & (UM_TC - 1)]));
                // (the group's first warp asks, for all its candidates)
                const uint8_t *gone_p = pruned + S.cp[cidx];
                const uint32_t *known_p = rho_max + S.cp[cidx];
                const bool asks = g == 0 && lane < UM_TC;
                int gone_next = 0;
                uint32_t kg_next = 0u;
                // Every lane waits (acquire) and the warp then agrees through a vote, so
                // the warp is converged and takes the same branch at every tcgen05.ld.  (One
                // lane polling for the warp was slower: 40 instead of 37 ms per headline run.)
                for (int u = grp ^ (int)(G & 1u); u < T; u += 2) {
                    const uint32_t n = G + (uint32_t)u;
                    const Ring a(n, 2), rw(n, wd_bars(L.nw));
                    const int ws = Ring(n, L.nw).s;
                    const int s = a.s;
                    // what other CTAs have found meanwhile, asked for a tile ahead
                    const int gone = gone_next;
                    const uint32_t kg = kg_next;
                    if (asks) {
                        gone_next = __ldcg(gone_p);
                        if (screen) {
                            kg_next = __ldcg(known_p);
                            if (kg > S.known[cidx])
                                atomicMax(const_cast<uint32_t *>(&S.known[cidx]), kg);
                        }
                    }
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&S.wd_full[rw.s], rw.par, wl) &&
                                                     mbar_wait_bounded(&S.mma_done[s], a.par, wl))) {
                        S.abort = 1;
                        break;
                    }
                    // an end token (its slice twin is committed too) takes its use of every ring
                    const bool token = !__shfl_sync(0xffffffffu, S.vw[rw.s], 0);
                    if (token) {
                        if (lane == 0) {
                            mbar_arrive(&S.dec[s]);
                            mbar_arrive(&S.acc_empty[s]);
                            mbar_arrive(&S.wd_empty[ws]);
                            mbar_arrive(&S.sl_empty[Ring(n, L.nb).s]);
                        }
                        break;
                    }
                    const float4 *wd4 = reinterpret_cast<const float4 *>(um_smem + L.wd[ws]);
                    tc_fence_after();
                    const int j0 = j_lo + u * UM_TW;
                    const uint32_t tag = n + 1u; // the tile's tag in need[s]
                    const bool live = !__shfl_sync(0xffffffffu, S.item_dead, 0);
                    bool full = true;
                    auto keep_block = [&]() {
                        const int c = lane % UM_TC, h = lane / UM_TC;
                        if (g != 0 || h > 1 || S.cw[c] < 0) return;
                        const float v = fmaxf(fmaxf(S.bmax[grp][0][h][c], S.bmax[grp][1][h][c]),
                                              fmaxf(S.bmax[grp][2][h][c], S.bmax[grp][3][h][c]));
                        B.v[(int64_t)S.cp[c] * B.halves + j0 / PADDI_HALF + h] = f2ord(v);
                    };
                    if (live || screen) {
                        const uint32_t tb = tmem + ((uint32_t)(32 * g) << 16) +
                                            (uint32_t)(s * UM_N);
                        const bool masked = (j0 + UM_TW > j_hi) ||
                                            (wc > j0 - m + 1 && wc < j0 + UM_TW + m - 1) || fc != 0.f;
                        const float4 *wrow = wd4 + bsh * WD_ROW;
                        // the tile's rounding bound and largest amplification (k_prep)
                        const float Gt = wd4[128].x, At = wd4[128].y;
                        uint32_t ra[32], rb[32];
                        // f(registers, chunk) over the row's 8 chunks of 32 columns, the load of
                        // a chunk overlapping the math on the one before; half() ends a half block
                        auto columns = [&](auto f, auto half) {
                            tmem_ld32_async(tb, ra);
#pragma unroll 1
                            for (int c2 = 0; c2 < 4; ++c2) {
                                tmem_wait_ld(ra);
                                tmem_ld32_async(tb + 64 * c2 + 32, rb);
                                f(ra, 2 * c2);
                                tmem_wait_ld(rb);
                                if (c2 < 3) tmem_ld32_async(tb + 64 * c2 + 64, ra);
                                f(rb, 2 * c2 + 1);
                                if (c2 & 1) half(c2 >> 1);
                            }
                        };
                        // maxima over the row's two half blocks of D a - z b - sub
                        auto row_max = [&](float z, float sub) -> float2 {
                            const float2 nz2 = make_float2(-z, -z), ns2 = make_float2(-sub, -sub);
                            float tm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                            auto chunk = [&](const uint32_t (&r)[32], int cb) {
                                if (!masked) {
#pragma unroll
                                    for (int i2 = 0; i2 < 16; ++i2) {
                                        const float4 wv = wrow[16 * cb + i2];
                                        const float2 dd = make_float2(__uint_as_float(r[2 * i2]),
                                                                      __uint_as_float(r[2 * i2 + 1]));
                                        const float2 rho = __ffma2_rn(
                                            dd, make_float2(wv.x, wv.y),
                                            __ffma2_rn(nz2, make_float2(wv.z, wv.w), ns2));
                                        tm[i2 & 3] = fmax3(tm[i2 & 3], rho.x, rho.y);
                                    }
                                } else {
#pragma unroll
                                    for (int i = 0; i < 32; ++i) {
                                        const int col = 32 * cb + i;
                                        const int j = j0 + 8 * col + bsh;
                                        const float4 wv = wrow[(32 * cb + i) >> 1];
                                        const float wa = (i & 1) ? wv.y : wv.x;
                                        const float wb = (i & 1) ? wv.w : wv.z;
                                        float rho = fmaf(__uint_as_float(r[i]), wa, fmaf(-z, wb, -sub));
                                        if (fc != 0.f && wa == 0.f) rho += 1.f; // two flat windows
                                        const int dd = wc > j ? wc - j : j - wc;
                                        if (j < j_hi && dd >= m - 1) tm[i & 3] = fmaxf(tm[i & 3], rho);
                                    }
                                }
                            };
                            float2 out = make_float2(-INFINITY, -INFINITY);
                            columns(chunk, [&](int h) {
                                const float v =
                                    rowok ? fmaxf(fmaxf(tm[0], tm[1]), fmaxf(tm[2], tm[3])) : -INFINITY;
                                if (h == 0) out.x = v;
                                else out.y = v;
                                tm[0] = tm[1] = tm[2] = tm[3] = -INFINITY;
                            });
                            return out;
                        };
                        // the same of D a alone
                        auto screen_max = [&]() -> float2 {
                            float tm[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                            auto chunk = [&](const uint32_t (&r)[32], int cb) {
#pragma unroll
                                for (int i2 = 0; i2 < 16; ++i2) {
                                    const float2 wa =
                                        *reinterpret_cast<const float2 *>(&wrow[16 * cb + i2]);
                                    const float2 v = __fmul2_rn(
                                        make_float2(__uint_as_float(r[2 * i2]),
                                                    __uint_as_float(r[2 * i2 + 1])),
                                        wa);
                                    tm[i2 & 3] = fmax3(tm[i2 & 3], v.x, v.y);
                                }
                            };
                            float2 out = make_float2(-INFINITY, -INFINITY);
                            columns(chunk, [&](int h) {
                                const float v =
                                    rowok ? fmaxf(fmaxf(tm[0], tm[1]), fmaxf(tm[2], tm[3])) : -INFINITY;
                                if (h == 0) out.x = v;
                                else out.y = v;
                                tm[0] = tm[1] = tm[2] = tm[3] = -INFINITY;
                            });
                            return out;
                        };
                        // prunes the candidates whose lower bound `low` exceeds thr, and those
                        // pruned elsewhere.  A candidate pruned here leaves the window that did
                        // it as its witness hint: a second pass over the accumulator, at most
                        // once per candidate, finds its column
                        auto prune = [&](float low, float z, float sub) {
                            const unsigned bal = __ballot_sync(0xffffffffu, low > thr);
                            bool hint = false;
                            // (low is -inf in the lanes that hold no row)
                            const unsigned hit = bal | (bal >> UM_TC);
                            if (lane < UM_TC) {
                                const int ci = lane;
                                if (!S.dead[ci]) {
                                    if ((hit >> lane) & 1u) {
                                        S.dead[ci] = 1;
                                        pruned[S.cp[ci]] = 1;
                                        hint = W.wit != nullptr;
                                    } else if (gone) {
                                        S.dead[ci] = 1; // pruned by another CTA's item
                                    }
                                }
                            }
                            const unsigned hints = __ballot_sync(0xffffffffu, hint);
                            if (hints) {
                                int jh = -1;
                                const bool mine = rowok && ((hints >> cidx) & 1u) && low > thr;
                                for (int cb = 0; cb < 8; ++cb) {
                                    tmem_ld32_async(tb + 32 * cb, ra);
                                    tmem_wait_ld(ra);
#pragma unroll
                                    for (int i = 0; i < 32; ++i) {
                                        const int j = j0 + 8 * (32 * cb + i) + bsh;
                                        const float4 wv = wrow[(32 * cb + i) >> 1];
                                        const float rho =
                                            fmaf(__uint_as_float(ra[i]), (i & 1) ? wv.y : wv.x,
                                                 fmaf(-z, (i & 1) ? wv.w : wv.z, -sub));
                                        const int dd = wc > j ? wc - j : j - wc;
                                        if (rho > thr && j < j_hi && dd >= m - 1) jh = j;
                                    }
                                }
                                if (mine && jh >= 0) wt_hint(W, wc, WT_ONE, jh);
                            }
                            __syncwarp();
                        };
                        // the half blocks' maxima (or bounds of them): over the warp's two shifts,
                        // then over the group's warps once all have put theirs
                        auto put_block = [&](float2 bm) {
                            bm.x = fmaxf(bm.x, __shfl_xor_sync(0xffffffffu, bm.x, UM_TC));
                            bm.y = fmaxf(bm.y, __shfl_xor_sync(0xffffffffu, bm.y, UM_TC));
                            if (lane < UM_TC) {
                                S.bmax[grp][g][0][lane] = bm.x;
                                S.bmax[grp][g][1][lane] = bm.y;
                            }
                        };
                        float2 hup = make_float2(-INFINITY, -INFINITY);
                        if (screen && live) {
                            // hi * hi alone is within gc of the exact correlation: the hi halves
                            // leave out zrest of the candidate's unit norm and 2^-11 (BF16: 2^-8)
                            // of the slice, amplified by at most At; Gt covers the arithmetic
                            // and the screen drops the candidate's residual sum (|b| <= At /
                            // sqrt(m))
                            // (a flat row is exact)
                            const bool ex = fc != 0.f;
                            const float g0 =
                                zrest + (X::uh * 1.01f + fabsf(zsh) * rsm) * At + Gt + 1e-6f;
                            float2 h2;
                            // (one choice per warp: both read tensor memory, all lanes together)
                            if (!__any_sync(0xffffffffu, masked)) {
                                h2 = screen_max();
                            } else {
                                h2 = row_max(zsh, 0.f);
                            }
                            const float hh = fmaxf(h2.x, h2.y);
                            const float gc =
                                ex || hh == -INFINITY ? 0.f : g0;
                            prune(hh - gc, zsh, gc);
                            // a value kept after all products is at most this
                            const float up = ex ? 0.f : g0 + Gt;
                            hup = make_float2(h2.x + up, h2.y + up);
                            const bool want = rowok && !S.dead[cidx] &&
                                              f2ord(fmaxf(hup.x, hup.y)) > S.known[cidx];
                            if (bkeep) put_block(hup);
                            if (__any_sync(0xffffffffu, want) && lane == 0) S.need[s] = tag;
                        }
                        if (screen) { // every warp, also one that saw the item dead already
                            tc_fence_before(); // the accumulator has been read
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&S.dec[s]);
                            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&S.dec[s], a.par, wl))) {
                                S.abort = 1;
                                break;
                            }
                            full = __shfl_sync(0xffffffffu, S.need[s], 0) == tag;
                            if (full) {
                                if (!__all_sync(0xffffffffu,
                                                mbar_wait_bounded(&S.rest_done[s], n_rest & 1u, wl))) {
                                    S.abort = 1;
                                    break;
                                }
                                ++n_rest;
                                tc_fence_after();
                            } else if (live && bkeep) {
                                keep_block();
                            }
                        }
                        if (full && live) {
                            // correlations lowered by the tile's bound for the prune test, raised
                            // back for the kept maximum (the interval's middle; -inf stays)
                            const float2 t2 = row_max(zsc, Gt);
                            const float tmax = fmaxf(t2.x, t2.y);
                            rmax = fmaxf(rmax, tmax + Gt);
                            if (bkeep) put_block(make_float2(t2.x + Gt, t2.y + Gt));
                            prune(tmax, zsc, Gt);
                            if (screen) { // for the other CTAs' screens, and this item's next tiles
                                const float v =
                                    fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, UM_TC));
                                if (lane < UM_TC && wc >= 0 && f2ord(v) > S.known[lane] &&
                                    atomicMax(const_cast<uint32_t *>(&S.known[lane]), f2ord(v)) <
                                        f2ord(v))
                                    atomicMax(rho_max + S.cp[lane], f2ord(v));
                            }
                        }
                        if (live && g == 0) {
                            ++n_tiles;
                            n_alive += alive;
                            alive = __popc(__ballot_sync(0xffffffffu, lane < UM_TC && !S.dead[lane & (UM_TC - 1)]));
                            if (!alive) S.item_dead = 1;
                        }
                    }
                    if (full && bkeep) { // the first warp stores what all four have put
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&S.put[s]);
                        if (g == 0) {
                            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&S.put[s], n_put & 1u, wl))) {
                                S.abort = 1;
                                break;
                            }
                            if (live) keep_block();
                        }
                        ++n_put;
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (!screen) mbar_arrive(&S.dec[s]); // no screen: only its use of the ring
                        mbar_arrive(&S.acc_empty[s]);
                        mbar_arrive(&S.wd_empty[ws]);
                        mbar_arrive(&S.sl_empty[Ring(n, L.nb).s]);
                    }
                }
                if (g == 0 && lane == 0) {
                    atomicAdd(&att->n_pairs, (unsigned long long)n_tiles * (UM_TC * UM_TW));
                    atomicAdd(&att->n_live, (unsigned long long)n_alive * UM_TW);
                }
                // fold the running maxima
                const float v = fmaxf(rmax, __shfl_xor_sync(0xffffffffu, rmax, UM_TC));
                if (lane < UM_TC && v > -INFINITY) atomicMax(&S.rmax[lane], f2ord(v));
            }
            __syncthreads();
            G += (uint32_t)(S.tok >= 0 ? min(S.tok + 2, T) : T); // every thread, the same number
            if (threadIdx.x < UM_TC && tile * UM_TC + threadIdx.x < C &&
                S.rmax[threadIdx.x] != f2ord(-INFINITY))
                atomicMax(rho_max + S.cp[threadIdx.x], S.rmax[threadIdx.x]);
            __syncthreads();
            if (S.abort) break;
        }
        if (S.abort) break;
        if (je >= col_hi) {
            if (threadIdx.x == 0) att->last_rd = rd;
            break;
        }
        // ---- between rounds (one launch for all of them: separate launches with a
        // compaction kernel each cost 30 us an attempt, most of it for rounds
        // without work; headline run 249 -> 229 ms).  The CTA that finished the
        // round's last item compacts the survivors; the others wait for it.  A CTA
        // waits only for items that other, running CTAs have taken (it found none
        // left to take), so the wait ends whichever CTAs are resident; it is bounded
        // all the same.
        if (S.last) {
            __threadfence();
            const int nx = compact_survivors<UM_THREADS>(list, rd == 0, C, pruned,
                                                          rd & 1 ? list0 : list1, S.wsum);
            __syncthreads();
            if (threadIdx.x == 0) {
                S.last = 0;
                S.next = nx;
                paddi::publish_round(att, rd, nx);
            }
        } else if (threadIdx.x == 0) {
            S.next = paddi::wait_round(att, rd, wl);
        }
        __syncthreads();
        C = S.next;
        if (C <= 0) break;
        jb = je;
        __syncthreads(); // S.next is read by all before a later round writes it
    }
    if (S.abort) {
        if (threadIdx.x == 0) {
            atomicExch(&att->status, 3); // also ends the other CTAs' waits between rounds
            if (mma_issued) { // let the MMAs in flight finish before TMEM goes away
                umma_commit(&S.drain);
                mbar_wait_bounded(&S.drain, 0u, kDrainCycles);
            }
        }
        // bulk copies in flight complete on their barriers: wait (bounded) for
        // the last phase the loader issued on each before the shared memory goes
        // away (a phase it never issued is not waited for)
        if (threadIdx.x == 32) {
            for (int s = 0; s < UM_STAGES; ++s) {
                if (S.last_full[s] >= 0)
                    mbar_wait_bounded(&S.full_b[s], (uint32_t)S.last_full[s], kDrainCycles);
            }
            for (int s = 0; s < UM_WBARS; ++s) {
                if (S.last_wd[s] >= 0)
                    mbar_wait_bounded(&S.wd_full[s], (uint32_t)S.last_wd[s], kDrainCycles);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) paddi::stamp_end(att->t + PADDI_T_REFINE_E);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u)
                     : "memory");
}

} // namespace

bool paddi_umma_supported(int device)
{
    int major = 0, minor = 0;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, device) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return major == 10 && minor == 0; // sm_100 (B200)
}

int paddi_umma_max_m() { return UM_KMAX64 - 7; } // kpad_of(m) <= UM_KMAX64

int32_t paddi_tile_width() { return UM_TW; }

paddi::RefineItems paddi_refine_items_umma(int32_t m, bool rows64, int32_t C, int32_t range,
                                           int32_t ctas)
{
    const int tc = kpad_of(m) <= UM_KMAX128 && !rows64 ? UM_TCMAX : UM_TCMAX / 2;
    return um_items((C + tc - 1) / tc, range, ctas);
}

int64_t paddi_tile_blocks(int64_t N) { return (N + UM_TW - 1) / UM_TW; }

int64_t paddi_tile_block_elems_max() { return 2 * (int64_t)slice_cnt(UM_KMAX64); }

int64_t paddi_tile_wd_entries() { return WD_ENTRIES; }

PaddiBound paddi_bound_tc(int m, bool bf16)
{
    const double u = std::ldexp(1.0, -24);
    const int kp = kpad_of(m);
    // split representation: z and y each within 2^-22 (FP16) / 2^-16 (BF16) of
    // their value, the dropped lo*lo term as much again; FP16 z halves below the
    // normal range: 2^-25 absolute against |z| = 2^8, i.e. 2^-33 sqrt(m) relative
    const double rep = bf16 ? 3.0 * std::ldexp(1.0, -16)
                            : 3.0 * std::ldexp(1.0, -22) + std::ldexp(1.0, -33) * std::sqrt((double)m);
    // the accumulator: one FP32 rounding (taken as 2^-23, truncation) of at most
    // the sum of |products| per MMA, 3 kp/16 MMAs plus the block sums
    const double acc = std::ldexp(1.0, -23) * (3.0 * kp / 16.0 + 1.0);
    // the candidate's split-value sum (2 kp/16 terms per thread + 4 shuffle
    // levels), its z (two-float centring, scale: 4u), the slice's x - s (u), the
    // epilogue's a, b and FMA (4u), the FP32 rounding of thr (2u)
    const double rest = (2.0 * kp / 16.0 + 4.0 + 4.0 + 1.0 + 4.0 + 2.0) * u; // + thr's rounding
    PaddiBound B;
    B.E = (float)((rep + acc + rest) * 1.01);
    // FP16 y halves below the normal range: 2^-25 per scaled value, 2^-(8+e) <=
    // 2 |x - s|_max 2^-22 of scale, against |z| sqrt(m) 2^8: 2^-38 sqrt(m) |x - s|_max
    B.F = bf16 ? 0.f : (float)(std::ldexp(1.0, -38) * std::sqrt((double)m) * 1.01);
    return B;
}

cudaError_t paddi_launch_prep(bool bf16, const float *x, int64_t n, int32_t m, float4 *wst,
                              float *mu, double2 *ms64, uint8_t *flat, int32_t *flat_count,
                              uint16_t *bq, float4 *wdq, float gcap, int32_t *frag_list,
                              cudaStream_t st, bool chained, const PaddiStatsExtra &extra,
                              unsigned long long *t_end)
{
    const int kp = kpad_of(m);
    if (kp > UM_KMAX64 || m < 3 || n < 2 * (int64_t)m) return cudaErrorInvalidValue;
    const int32_t N = (int32_t)(n - m + 1);
    const unsigned grid = (unsigned)(((int64_t)N + PADDI_PAD_WIN + ST_TILE - 1) / ST_TILE);
    const PaddiBound B = paddi_bound_tc(m, bf16);
    const size_t smem = st_smem(m);
    auto kern = bf16 ? k_prep<true> : k_prep<false>;
    cudaError_t e = paddi_raise_smem_limit((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    const StOut O = {wst, mu, ms64, flat, flat_count, flat_count + 1, extra};
    return paddi_launch(chained, kern, grid, ST_THREADS, smem, st, x, n, slice_cnt(kp), m, N, O, bq,
                        wdq, B.E, B.F, gcap, frag_list, flat_count + 3, t_end);
}

cudaError_t paddi_launch_refine_umma(bool bf16, const float *x, const float4 *wst,
                                     const float *mu, const int32_t *cand, int32_t *list0,
                                     int32_t *list1, const uint16_t *bq, const float4 *wdq,
                                     PaddiAttemptDev *att, uint32_t *rho_max, uint8_t *pruned,
                                     int32_t N, int32_t m, int32_t col_lo, int32_t col_hi,
                                     float thr_prune, int32_t num_sms, cudaStream_t st,
                                     long long wait_cycles, int32_t withhold, bool rows64,
                                     const PaddiWitness *W, const PaddiBlockMax *B, float guard)
{
    const int kp = kpad_of(m);
    if (kp > UM_KMAX64 || m < 3) return cudaErrorInvalidValue;
    if ((col_lo % UM_TW) != 0 || (col_hi % UM_TW != 0 && col_hi != N)) return cudaErrorInvalidValue;
    const int MM = (kp <= UM_KMAX128 && !rows64) ? 128 : 64;
    const UmLayout L = um_layout(MM, kp);
    // request at least half the SM's shared memory so one CTA owns the 512 TMEM columns
    const size_t smem = L.bytes < 120 * 1024 ? 120 * 1024 : L.bytes;
    void (*kern)(const float *, const float4 *, const float *, const int32_t *, int32_t *,
                 int32_t *, const uint16_t *, const float4 *, PaddiAttemptDev *, uint32_t *,
                 uint8_t *, int32_t, int32_t, int32_t, int32_t, float, int32_t, long long, int32_t,
                 PaddiWitness, PaddiBlockMax, int32_t, float);
    if (MM == 128) kern = bf16 ? k_refine_umma<true, 128> : k_refine_umma<false, 128>;
    else kern = bf16 ? k_refine_umma<true, 64> : k_refine_umma<false, 64>;
    cudaError_t e = paddi_raise_smem_limit((const void *)kern, smem);
    if (e != cudaSuccess) return e;
    const int grid = num_sms;
    return paddi_launch(true, kern, grid, UM_THREADS, smem, st, x, wst, mu, cand, list0, list1, bq, wdq, att, rho_max,
                                         pruned, N, m, col_lo, col_hi, thr_prune, grid,
                                         wait_cycles > 0 ? wait_cycles : paddi::REFINE_WAIT, withhold,
                                         W ? *W : PaddiWitness{}, B ? *B : PaddiBlockMax{},
                        !bf16 && kp >= UM_SCREEN_K ? 1 : 0, guard);
}
