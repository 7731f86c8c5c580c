// k_fragile.cu -- exact correlations of the surviving candidates with the
// fragile windows of a length.
//
// No counterpart in the reference, whose FP32 refine (gpu_global_discords_refine,
// src/PD3_kernels.cuh:582-662) evaluates every pair the same way.  Here the
// refine kernels evaluate a pair (candidate c, window j) with an error bound
// g_j that grows with |x_j - s| / |x_j - mu_j| for the shift s of j's tile
// (window_bound in paddi_internal.cuh).  Windows whose bound exceeds the
// guard band -- near-flat windows far from their tile's level, series with a
// large offset and small local variance -- are "fragile": the tensor-core
// refine skips them (the FP32 refine uses them lowered by their own bound, to
// prune), and this kernel, run after the refine's last round, evaluates them
// in FP64 against every candidate still unpruned:
//     rho = sum_k (x_c+k - mu_c)(x_f+k - mu_f) inv_c inv_f,
// both windows centred on their own FP64 means, so the error is ~1e-14 of
// the result whatever the offset.  A correlation above thr + 1e-7 prunes the
// candidate (the margin covers the FP32 rounding of thr); every value enters
// the candidate's kept maximum.
//
// Work items: (a group of 8 entries of the candidate list, 64, 32 or 16 consecutive
// entries of the fragile list).  The group's centred candidate values sit in
// shared memory (read as broadcasts, two terms per load); a fragile window is
// shared by 4, 8 or 16 threads, two halves of the group times 2, 4 or 8 parts of the
// length, each with 4 FP64 accumulators and reading the window's values straight
// from the series (consecutive addresses per part, so most loads hit L1).
// What bounds it is the serial chain of one thread, not FP64 issue: a headline
// attempt has about 3000 fragile windows and a handful of candidates, 50 to 100 items
// of 64 windows for 592 resident CTAs, so the windows per item shrink (and the parts
// grow) while the items still fit the CTAs.  All fragile passes of a headline run: with
// one split of 4 threads a window 10.9 ms, now 6.0 (run 137.7 -> 132.5).  Halves whose
// candidates are all pruned, and items with no live candidate, are skipped.
#include <float.h>

#include "paddi_internal.cuh"

using paddi::f2ord;
using paddi::ord2f;

namespace {

constexpr int FG_THREADS = 256;
constexpr int FG_WIN = 64;      // fragile windows per item, at most
constexpr int FG_SPLIT = 2;     // halvings of it, at most
constexpr int FG_CAND = 8;      // candidate-list entries per item
constexpr int FG_HALF = 4;      // accumulators per thread
constexpr int FG_MAXM = 1024;
static_assert(FG_THREADS / 32 == FG_CAND, "a warp stages a candidate");

__global__ void __launch_bounds__(FG_THREADS)
k_fragile(const float *__restrict__ x, const double2 *ms64,
          const int32_t *cand,
          const int32_t *list0, const int32_t *list1,
          PaddiAttemptDev *att, uint8_t *pruned, uint32_t *rho_max,
          const int32_t *frag,
          const int32_t *frag_count, int32_t m, float thr, int32_t col_lo,
          int32_t col_hi, PaddiBlockMax B, float guard)
{
    // [FG_CAND][mp] centred candidate values, mp = m rounded up to even
    extern __shared__ __align__(16) double fg_a[];
    __shared__ int cw[FG_CAND], cp[FG_CAND], live[FG_CAND];
    __shared__ double civ[FG_CAND], cmu[FG_CAND];
    __shared__ double best_s[FG_CAND][4];
    __shared__ int s_any;
    paddi::chain_begin();
    paddi::stamp_begin(att->t + PADDI_T_FRAGILE);
    // the candidates of the refine's last round (round 0: all of them)
    const int rd = att->last_rd;
    const int32_t *list = rd & 1 ? list1 : list0;
    const int C = rd ? att->list_count[rd] : att->n_cand_p1, F = __ldcg(frag_count);
    if (C <= 0 || F <= 0) return;
    const bool bkeep = B.kept(att->n_cand_p1);
    const int mp = (m + 1) & ~1;
    const int groups = (C + FG_CAND - 1) / FG_CAND;
    int sh = 0; // FG_WIN >> sh windows per item
    while (sh < FG_SPLIT &&
           (long long)groups * ((F + (FG_WIN >> sh) / 2 - 1) / ((FG_WIN >> sh) / 2)) <= gridDim.x)
        ++sh;
    const int win = FG_WIN >> sh;
    const int chunks = (F + win - 1) / win;
    const long long total = (long long)groups * chunks;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (long long item = blockIdx.x; item < total; item += gridDim.x) {
        const int grp = (int)(item % groups), chunk = (int)(item / groups);
        __syncthreads(); // the previous item's shared data is consumed
        if (t == 0) s_any = 0;
        __syncthreads();
        if (t < FG_CAND) {
            const int li = grp * FG_CAND + t;
            const int pos = li >= C ? -1 : rd ? list[li] : li;
            const int w = pos >= 0 ? cand[pos] : 0;
            cp[t] = pos;
            cw[t] = w;
            live[t] = pos >= 0 && !__ldcg(pruned + pos);
            const double2 s2 = ms64[w];
            cmu[t] = s2.x;
            civ[t] = s2.y;
            if (live[t]) atomicOr(&s_any, 1);
        }
        __syncthreads();
        if (!s_any) continue;
        { // a warp per candidate
            const bool lv = live[warp] != 0;
            const float *xc = x + cw[warp];
            const double mc = cmu[warp];
#pragma unroll 4
            for (int k = lane; k < mp; k += 32)
                fg_a[warp * mp + k] = (lv && k < m) ? (double)__ldg(xc + k) - mc : 0.0;
        }
        __syncthreads();
        // warp: half of the group (h), 16 >> sh windows; lane: window, part of the length (s)
        const int lw = 4 - sh; // log2 of the warp's windows
        const int h = warp & 1, wsub = warp >> 1, s = lane >> lw;
        const int fi = chunk * win + (wsub << lw) + (lane & ((1 << lw) - 1));
        const int f = fi < F ? frag[fi] : -1;
        const bool fok = f >= col_lo && f < col_hi;
        const int c0 = h * FG_HALF;
        double b[FG_HALF];
#pragma unroll
        for (int c = 0; c < FG_HALF; ++c) b[c] = -INFINITY;
        bool any = false; // uniform over the warp
#pragma unroll
        for (int c = 0; c < FG_HALF; ++c) any |= live[c0 + c] != 0;
        if (any) {
            double acc[FG_HALF];
#pragma unroll
            for (int c = 0; c < FG_HALF; ++c) acc[c] = 0.0;
            const double2 sf = fok ? ms64[f] : make_double2(0.0, 0.0);
            const double2 *a2 = reinterpret_cast<const double2 *>(fg_a + c0 * mp);
            const int mh = mp >> 1, q0 = (mh * s) >> (sh + 1), q1 = (mh * (s + 1)) >> (sh + 1);
            if (fok) {
                const float *y = x + f;
#pragma unroll 4
                for (int q = q0; q < q1; ++q) {
                    // terms 2q, 2q+1 (the even padding term has zero candidate values)
                    const double v0 = (double)__ldg(y + 2 * q) - sf.x;
                    const double v1 = 2 * q + 1 < m ? (double)__ldg(y + 2 * q + 1) - sf.x : 0.0;
#pragma unroll
                    for (int c = 0; c < FG_HALF; ++c) {
                        const double2 av = a2[c * mh + q];
                        acc[c] = fma(av.y, v1, fma(av.x, v0, acc[c]));
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < FG_HALF; ++c) {
                for (int o = 16; o >> lw; o >>= 1)
                    acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
                const int ci = c0 + c;
                const int d = cw[ci] > f ? cw[ci] - f : f - cw[ci];
                if (fok && live[ci] && d >= m - 1) {
                    b[c] = acc[c] * civ[ci] * sf.y;
                    // may be the nearest neighbour: the recheck has to look here
                    if (s == 0 && bkeep &&
                        b[c] >= (double)ord2f(__ldcg(rho_max + cp[ci])) - 2.0 * guard)
                        atomicMax(B.v + (int64_t)cp[ci] * B.halves + f / PADDI_HALF,
                                  f2ord((float)b[c]));
                }
            }
        }
        // maxima over the item's windows, per candidate
#pragma unroll
        for (int c = 0; c < FG_HALF; ++c) {
            double v = b[c];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
            if (lane == 0) best_s[c0 + c][wsub] = v;
        }
        __syncthreads();
        if (t < FG_CAND && live[t]) {
            double v = -INFINITY;
#pragma unroll
            for (int q = 0; q < 4; ++q) v = fmax(v, best_s[t][q]);
            if (v > -INFINITY) {
                atomicMax(rho_max + cp[t], f2ord((float)v));
                if (v > (double)thr + 1e-7) pruned[cp[t]] = 1;
            }
        }
    }
}

} // namespace

cudaError_t paddi_launch_fragile(const float *x, const double2 *ms64,
                                 const int32_t *cand, const int32_t *list0,
                                 const int32_t *list1, PaddiAttemptDev *att,
                                 uint8_t *pruned, uint32_t *rho_max,
                                 const int32_t *frag, const int32_t *frag_count, int32_t m,
                                 float thr, int32_t col_lo, int32_t col_hi, int32_t num_sms,
                                 cudaStream_t st, const PaddiBlockMax *B, float guard)
{
    if (m > FG_MAXM || m < 3) return cudaErrorInvalidValue;
    const size_t smem = sizeof(double) * (size_t)FG_CAND * (size_t)((m + 1) & ~1);
    cudaError_t e = paddi_raise_smem_limit((const void *)k_fragile, smem);
    if (e != cudaSuccess) return e;
    return paddi_launch(true, k_fragile, num_sms * 4, FG_THREADS, smem, st, x, ms64, cand, list0, list1, att,
                                                    pruned, rho_max, frag, frag_count, m, thr,
                                                    col_lo, col_hi, B ? *B : PaddiBlockMax{}, guard);
}
