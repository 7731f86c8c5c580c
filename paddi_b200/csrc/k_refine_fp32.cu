// k_refine_fp32.cu -- dense candidate refine on CUDA cores (the plain FP32 form).
//
// Reference: gpu_global_discords_refine (src/PD3_kernels.cuh:582-662): a
// 32x32-tiled SGEMM of the candidate matrix C (m x Cc, gathered on the host)
// with the Hankel windows of the series, the distance formula in the
// epilogue, and a CAS-loop float atomicMin per candidate.
//
// Here:
//   * candidates are an index list produced on the device; each work item
//     is (8 candidates) x (a slice of all windows), pulled from a counter by
//     a persistent grid, all rounds in one launch.  8 and not more: after the
//     first round a dozen candidates are left, and with 32 per item most of the
//     arithmetic went to empty rows on a tenth of the SMs (windows of 730..741,
//     n = 131072, 5 to 20 candidates: 1.1 ms an attempt in four launches, now
//     0.28 ms);
//   * the candidate operand is the z-normalised window z_c = (x_c - mu_c) inv_c,
//     staged once per item; the window operand is the raw series shifted by a
//     per-sub-chunk constant (the shift cancels because sum_k z_c[k] = 0, and the
//     rounding residue is removed with the candidate's FP32 sum of z_c);
//   * every thread holds 4 candidates x 8 windows of accumulators; the 8
//     window operands rotate through a register ring (one shared load per k);
//     two warps share a sub-chunk of 256 windows, a chunk is 4 of them;
//   * the epilogue forms rho = <z_c, x_j - mu_j> inv_j, applies the
//     trivial-match exclusion |c - j| >= m-1, keeps the running maximum
//     (maximum rho == minimum distance) and flags a candidate as pruned as
//     soon as its correlation with some window exceeds thr (early abandoning:
//     an item stops when all 8 of its candidates are pruned, and later items
//     of a fully pruned tile are skipped);
//   * one atomicMax per candidate per item on an order-preserving integer
//     image of rho (no CAS loop).
// Rounding: the dot products are summed in two levels (blocks of 64 terms),
// so a correlation with window j is within g_j = window_bound(E, A_j) of the
// exact one, A_j the amplification |x_j - sh| / |x_j - mu_j| of the sub-chunk's
// shift.  Windows with g_j above gcap are fragile: their correlations are
// lowered by their own g_j (a safe lower bound to prune on) and they are
// evaluated in FP64 by the fragile pass.  The sub-chunk's largest other g_j, G,
// is subtracted from the other correlations for the prune test, and added
// back to the kept maxima, so those are the middle of an interval of
// half-width at most gcap (a fragile window's lowered value never exceeds its
// true one).  Sub-chunks start
// at multiples of 256 windows, so the fragile set depends only on the length.
#include <float.h>

#include <cmath>

#include "paddi_internal.cuh"

using paddi::f2ord;

namespace {

constexpr int RF_THREADS = 256; // 8 warps: 2 groups of 4 candidates x 4 sub-chunks
constexpr int RF_TC = 8;        // candidates per item
constexpr int RF_CG = RF_TC / 4;
constexpr int RF_SUB = RF_THREADS / 32 / RF_CG; // sub-chunks in flight
constexpr int RF_TW = 256;      // windows per sub-chunk (32 lanes x 8), one shift each
constexpr int RF_CW = RF_SUB * RF_TW; // windows per chunk
static_assert(RF_TW == RF_THREADS, "one window of each sub-chunk per thread at staging");
constexpr int RF_MAXM = 1024;

__device__ __forceinline__ int xpad(int p) { return p + (p >> 5); }

struct RfSmem {
    float *zT;    // [mpad][RF_TC]
    float *xs;    // xpad(RF_CW + mpad + 8)
    float *cinv;  // [RF_CW]
    float *cmu;   // [RF_CW]
    float *cflt;  // [RF_CW]
    float *cgm;   // [RF_CW]: the bound subtracted from each window's correlations
};

// About two items per CTA; with thousands of candidates one split would do that, and an
// item would be 8 candidates times the whole round.  RF_ITEM bounds its windows times m:
// 8 * 2^30 FMA are some 2.2e8 cycles of a CTA (at 38 a cycle), a twentieth of the
// waits' limit (without it a round of 3.4e7 windows at m = 1000 came to 7e9 cycles).
constexpr int RF_ITEM = 1 << 30;
__host__ __device__ __forceinline__ paddi::RefineItems rf_items(int m, int tiles, int range,
                                                                int ctas)
{
    return paddi::refine_items(range, tiles, (2 * ctas + tiles - 1) / tiles, RF_CW, RF_ITEM / m);
}

constexpr int RF_SUMBLK = 64; // two-level sums: terms per partial sum

__global__ void __launch_bounds__(RF_THREADS)
k_refine_fp32(const float *__restrict__ x, const float4 *wst,
              const float *mu, const int32_t *cand, int32_t *list0,
              int32_t *list1, PaddiAttemptDev *att, uint32_t *rho_max, uint8_t *pruned, int32_t N,
              int32_t m, int32_t col_lo, int32_t col_hi, float thr, float E, float gcap,
              long long wl, PaddiWitness W)
{
    extern __shared__ __align__(16) unsigned char rf_smem[];
    const int mpad = (m + 7) & ~7;
    RfSmem S;
    S.zT = reinterpret_cast<float *>(rf_smem);
    S.xs = S.zT + (size_t)mpad * RF_TC;
    S.cinv = S.xs + xpad(RF_CW + mpad + 8) + 4;
    S.cmu = S.cinv + RF_CW;
    S.cflt = S.cmu + RF_CW;
    S.cgm = S.cflt + RF_CW;
    __shared__ int s_item, s_alive, s_last, s_next;
    __shared__ int s_wsum[RF_THREADS / 32];
    __shared__ float s_gred[RF_SUB][RF_THREADS / 32];
    __shared__ int cw[RF_TC], cp[RF_TC];
    __shared__ float cf[RF_TC], zsum[RF_TC];
    __shared__ uint8_t dead[RF_TC];

    paddi::chain_begin();
    paddi::stamp_begin(att->t + PADDI_T_REFINE_B);
    int C = att->n_cand_p1;
    if (C <= 0 || col_hi <= col_lo) {
        paddi::stamp_begin(att->t + PADDI_T_REFINE_E);
        return;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cg = warp % RF_CG, sub = warp / RF_CG;
    if (threadIdx.x == 0) s_last = 0;
    const int nrounds = paddi::refine_rounds(col_hi - col_lo);
    int jb = col_lo;
    for (int rd = 0; rd < nrounds; ++rd) {
        int je = paddi::refine_round_end(rd, nrounds, col_lo, col_hi, RF_TW);
        if (C <= RF_TC) je = col_hi; // one tile left: later rounds could not shrink it
        int32_t *list = rd & 1 ? list1 : list0; // round 0: all candidates
        const int range = je - jb;
        const int tiles = (C + RF_TC - 1) / RF_TC;
        // about two items per CTA, of at least one chunk
        const paddi::RefineItems I = rf_items(m, tiles, range, (int)gridDim.x);
        const int splits = I.splits, span = I.span;
        const int total = tiles * splits;
        bool counted = true; // this CTA's latest item is in done_rd
        for (;;) {
            if (threadIdx.x == 0) {
                if (!counted) {
                    __threadfence();
                    s_last = atomicAdd(&att->done_rd[rd], 1) == total - 1;
                }
                s_item = atomicAdd(&att->work_rd[rd], 1);
            }
            counted = false;
            __syncthreads();
            const int item = s_item;
            if (item >= total) break;
            const int tile = item % tiles, split = item / tiles;
            // ---- candidates of this item
            if (threadIdx.x < RF_TC) {
                const int li = tile * RF_TC + threadIdx.x;
                const bool v = li < C;
                const int pos = !v ? 0 : rd ? __ldcg(list + li) : li;
                const int w = v ? cand[pos] : 0;
                cw[threadIdx.x] = w;
                cp[threadIdx.x] = pos;
                dead[threadIdx.x] = !v || __ldcg(pruned + pos);
                cf[threadIdx.x] = (v && wst[w].z == 0.f) ? 1.f : 0.f; // flat candidate
            }
            __syncthreads();
            int alive = 0;
            if (threadIdx.x < RF_TC) alive = !dead[threadIdx.x];
            if (!__syncthreads_or(alive)) continue;
            // ---- z-normalised candidate windows, k-major
            for (int e = threadIdx.x; e < mpad * RF_TC; e += RF_THREADS) {
                const int c = e / mpad, k = e - c * mpad;
                float z = 0.f;
                if (k < m && !dead[c]) {
                    const int w = cw[c];
                    z = (x[w + k] - mu[w]) * wst[w].z;
                }
                S.zT[k * RF_TC + c] = z;
            }
            __syncthreads();
            { // two-level sums of the candidates' z: a warp per candidate, a lane per block
                float s = 0.f;
                const int k0 = lane * RF_SUMBLK;
                for (int k = k0; k < min(m, k0 + RF_SUMBLK); ++k) s += S.zT[k * RF_TC + warp];
                float tot = 0.f;
                for (int q = 0; q * RF_SUMBLK < m; ++q) tot += __shfl_sync(0xffffffffu, s, q);
                if (lane == 0) zsum[warp] = tot;
            }
            const int j_lo = jb + split * span, j_hi = min(je, j_lo + span);
            float rmax[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
            for (int j0 = j_lo; j0 < j_hi; j0 += RF_CW) {
                __syncthreads();
                for (int p = threadIdx.x; p < RF_CW + mpad + 8; p += RF_THREADS) {
                    const int g = j0 + p;
                    S.xs[xpad(p)] = g < N + m - 1 ? x[g] : 0.f;
                }
                // one window of each sub-chunk per thread: its bound, fragile or not
                float gt[RF_SUB];
                bool fragt[RF_SUB];
#pragma unroll
                for (int s = 0; s < RF_SUB; ++s) {
                    const int qt = s * RF_TW + threadIdx.x;
                    const bool in = j0 + s * RF_TW < j_hi;
                    const float4 wsq = in ? wst[j0 + qt] : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float mq = in ? mu[j0 + qt] : 0.f;
                    const float sh = in ? x[j0 + s * RF_TW] : 0.f;
                    gt[s] = paddi::window_bound(wsq.z, mq, sh, (float)m, E, 0.f);
                    fragt[s] = j0 + qt < N && gt[s] > gcap;
                    S.cinv[qt] = wsq.z;
                    S.cflt[qt] = wsq.z == 0.f ? 1.f : 0.f; // flat window (or the padded tail)
                    S.cmu[qt] = mq;
                    // the sub-chunk's largest bound over its non-fragile windows
                    float gq = fragt[s] ? 0.f : gt[s];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1)
                        gq = fmaxf(gq, __shfl_xor_sync(0xffffffffu, gq, o));
                    if (lane == 0) s_gred[s][warp] = gq;
                }
                __syncthreads();
#pragma unroll
                for (int s = 0; s < RF_SUB; ++s) {
                    float Gs = 0.f;
#pragma unroll
                    for (int w2 = 0; w2 < RF_THREADS / 32; ++w2) Gs = fmaxf(Gs, s_gred[s][w2]);
                    S.cgm[s * RF_TW + threadIdx.x] = fragt[s] ? gt[s] : Gs;
                }
                float G = 0.f;
#pragma unroll
                for (int w2 = 0; w2 < RF_THREADS / 32; ++w2) G = fmaxf(G, s_gred[sub][w2]);
                __syncthreads();
                int hit[4] = {-1, -1, -1, -1}; // a window that prunes the candidate
                const int q00 = sub * RF_TW; // this warp's sub-chunk
                if (j0 + q00 < j_hi) {
                    const float sh = S.xs[xpad(q00)];
                    float acc[4][8], tot[4][8];
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int jj = 0; jj < 8; ++jj) acc[c][jj] = tot[c][jj] = 0.f;
                    float ring[8];
                    const int p0 = q00 + 8 * lane;
#pragma unroll
                    for (int jj = 0; jj < 8; ++jj) ring[jj] = S.xs[xpad(p0 + jj)] - sh;
                    const float4 *z4 = reinterpret_cast<const float4 *>(S.zT) + cg;
                    for (int k0 = 0; k0 < mpad; k0 += 8) {
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            const float4 z = z4[(k0 + u) * RF_CG];
#pragma unroll
                            for (int jj = 0; jj < 8; ++jj) {
                                const float xv = ring[(u + jj) & 7];
                                acc[0][jj] = fmaf(z.x, xv, acc[0][jj]);
                                acc[1][jj] = fmaf(z.y, xv, acc[1][jj]);
                                acc[2][jj] = fmaf(z.z, xv, acc[2][jj]);
                                acc[3][jj] = fmaf(z.w, xv, acc[3][jj]);
                            }
                            ring[u] = S.xs[xpad(p0 + k0 + u + 8)] - sh;
                        }
                        if (((k0 + 8) & (RF_SUMBLK - 1)) == 0 || k0 + 8 >= mpad) {
#pragma unroll
                            for (int c = 0; c < 4; ++c)
#pragma unroll
                                for (int jj = 0; jj < 8; ++jj) {
                                    tot[c][jj] += acc[c][jj];
                                    acc[c][jj] = 0.f;
                                }
                        }
                    }
                    // ---- epilogue
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int ci = 4 * cg + c;
                        const int w = cw[ci];
                        const float zs = zsum[ci], fc = cf[ci];
                        float cmax = -INFINITY;
#pragma unroll
                        for (int jj = 0; jj < 8; ++jj) {
                            const int q = p0 + jj;
                            const int j = j0 + q;
                            const int dd = w > j ? w - j : j - w;
                            const bool ok = (j < j_hi) && (dd >= m - 1);
                            // lower bound of the correlation (a fragile window: by its own bound)
                            const float rho = fmaf(fmaf(-zs, S.cmu[q] - sh, tot[c][jj]), S.cinv[q],
                                                   fmaf(fc, S.cflt[q], -S.cgm[q]));
                            if (ok) {
                                cmax = fmaxf(cmax, rho);
                                if (rho > thr) hit[c] = j;
                            }
                        }
                        rmax[c] = fmaxf(rmax[c], cmax + G); // the interval's middle
                    }
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int ci = 4 * cg + c;
                    const unsigned any = __ballot_sync(0xffffffffu, hit[c] >= 0);
                    if (any && lane == __ffs(any) - 1 && !dead[ci]) {
                        dead[ci] = 1;
                        pruned[cp[ci]] = 1;
                        if (W.wit) wt_hint(W, cw[ci], WT_ONE, hit[c]);
                    }
                }
                __syncthreads();
                // early abandon: stop once every candidate of the item is pruned
                if (threadIdx.x == 0) s_alive = 0;
                __syncthreads();
                if (threadIdx.x < RF_TC) {
                    if (!dead[threadIdx.x] && __ldcg(pruned + cp[threadIdx.x])) dead[threadIdx.x] = 1;
                    if (!dead[threadIdx.x]) s_alive = 1;
                }
                if (threadIdx.x == 0)
                    atomicAdd(&att->n_pairs, (unsigned long long)RF_TC * min(RF_CW, j_hi - j0));
                __syncthreads();
                if (!s_alive) break;
            }
            // ---- fold the item's maxima into the global ones
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float v = rmax[c];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
                const int ci = 4 * cg + c;
                if (lane == 0 && tile * RF_TC + ci < C && v > -INFINITY)
                    atomicMax(rho_max + cp[ci], f2ord(v));
            }
            __syncthreads();
        }
        if (je >= col_hi) {
            if (threadIdx.x == 0) att->last_rd = rd;
            break;
        }
        // ---- between rounds: as in the tensor-core refine (a CTA waits only for
        // items that running CTAs hold, and the wait is bounded)
        if (s_last) {
            __threadfence();
            const int nx = paddi::compact_survivors<RF_THREADS>(list, rd == 0, C, pruned,
                                                                rd & 1 ? list0 : list1, s_wsum);
            __syncthreads();
            if (threadIdx.x == 0) {
                s_last = 0;
                s_next = nx;
                paddi::publish_round(att, rd, nx);
            }
        } else if (threadIdx.x == 0) {
            s_next = paddi::wait_round(att, rd, wl);
        }
        __syncthreads();
        C = s_next;
        if (C <= 0) break;
        jb = je;
        __syncthreads(); // s_next is read by all before a later round writes it
    }
    if (threadIdx.x == 0) paddi::stamp_end(att->t + PADDI_T_REFINE_E);
}

} // namespace

cudaError_t paddi_launch_refine_fp32(const float *x, const float4 *wst, const float *mu,
                                     const int32_t *cand, int32_t *list0, int32_t *list1,
                                     PaddiAttemptDev *att, uint32_t *rho_max, uint8_t *pruned,
                                     int32_t N, int32_t m, int32_t col_lo, int32_t col_hi,
                                     float thr, float gcap, int32_t num_sms, cudaStream_t st,
                                     long long wait_cycles, const PaddiWitness *W)
{
    if (m > RF_MAXM) return cudaErrorInvalidValue;
    if ((col_lo % RF_TW) != 0) return cudaErrorInvalidValue; // sub-chunks on the 256-window grid
    const int mpad = (m + 7) & ~7;
    const size_t smem = sizeof(float) * ((size_t)mpad * RF_TC + (RF_CW + mpad + 8) +
                                         ((RF_CW + mpad + 8) >> 5) + 4 + 4 * RF_CW) + 16;
    cudaError_t e = paddi_raise_smem_limit((const void *)k_refine_fp32, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_refine_fp32, RF_THREADS, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int grid = num_sms * per_sm;
    return paddi_launch(true, k_refine_fp32, grid, RF_THREADS, smem, st, x, wst, mu, cand, list0, list1, att, rho_max, pruned, N, m, col_lo, col_hi, thr,
        paddi_bound_fp32(m).E, gcap, wait_cycles > 0 ? wait_cycles : paddi::REFINE_WAIT,
        W ? *W : PaddiWitness{});
}

paddi::RefineItems paddi_refine_items_fp32(int32_t m, int32_t C, int32_t range, int32_t ctas)
{
    return rf_items(m, (C + RF_TC - 1) / RF_TC, range, ctas);
}

PaddiBound paddi_bound_fp32(int m)
{
    const double u = std::ldexp(1.0, -24);
    const int mpad = (m + 7) & ~7;
    // the dot product in two levels (64 terms, then mpad/64 partials), the z
    // sum likewise, z's own rounding (x - mu, times inv: 3u), the shifted slice
    // (u), the epilogue (4u), the FP32 rounding of thr (2u)
    const double dot = (double)RF_SUMBLK + std::ceil(mpad / (double)RF_SUMBLK) + 1.0;
    PaddiBound B;
    B.E = (float)((2.0 * dot + 10.0) * u * 1.01);
    B.F = 0.f;
    return B;
}

// Fragile windows of length m for the FP32 refine's geometry (chunks of 256
// windows shifted by their first value): the same test as the refine applies.
__global__ void k_fragile_scan_fp32(const float *__restrict__ x, const float4 *wst,
                                    const float *mu, int32_t N, int32_t m, float E,
                                    float gcap, int32_t *frag_list, int32_t *frag_count,
                                    unsigned long long *t_end)
{
    paddi::chain_begin();
    const int lane = threadIdx.x & 31;
    for (int j0 = blockIdx.x * blockDim.x; j0 < N; j0 += gridDim.x * blockDim.x) {
        const int j = j0 + threadIdx.x;
        bool frag = false;
        if (j < N) {
            const float sh = x[j & ~(RF_TW - 1)];
            frag = paddi::window_bound(wst[j].z, mu[j], sh, (float)m, E, 0.f) > gcap;
        }
        const unsigned bal = __ballot_sync(0xffffffffu, frag);
        if (bal) {
            int base = 0;
            if (lane == 0) base = atomicAdd(frag_count, __popc(bal));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (frag) frag_list[base + __popc(bal & ((1u << lane) - 1u))] = j;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) paddi::stamp_end(t_end);
}

cudaError_t paddi_launch_fragile_scan_fp32(const float *x, const float4 *wst, const float *mu,
                                           int32_t N, int32_t m, float gcap, int32_t *frag_list,
                                           int32_t *frag_count, int32_t num_sms, cudaStream_t st,
                                           unsigned long long *t_end)
{
    return paddi_launch(true, k_fragile_scan_fp32, num_sms * 4, 256, 0, st, x, wst, mu, N, m,
                        paddi_bound_fp32(m).E, gcap, frag_list, frag_count, t_end);
}
