// k_witness.cu -- a known close neighbour ("witness") per window, carried from
// one length of a PALMAD run to the next.
//
// (No counterpart in the reference, which starts every attempt's candidate
// selection from nothing: gpu_local_candidate_select, src/PD3_kernels.cuh:9-259.)
// A window is no candidate as soon as one admissible neighbour is closer than
// r, and a neighbour that proves this at length m mostly still does at m + 1,
// where r is nearly the same.  So PALMAD keeps, per window i, one neighbour
// wit[i] and the pair's centred dot product wc[i] in FP64.  One more value per
// window extends it exactly (Welford's update in the length):
//     cov_{m+1} = cov_m + (m+1)/m (x[i+m] - mu_i)(x[w+m] - mu_w),  means at m+1,
// which turns candidate selection of the next length from 256 or more pairs
// per window (k_phase1) into one:
//   k_witness_step    advances all pairs to the new length and leaves a lower
//                     bound wrho[i] of their correlations;
//   k_witness_check   (per attempt) windows with wrho[i] > thr are no candidates;
//                     lists the others;
//   k_witness_rescue  (per attempt) looks for a new witness of each listed
//                     window: one warp ranks up to 32 neighbours in FP32 -- the
//                     diagonals of the witnesses of nearby windows, those
//                     neighbours' own witnesses, and a few pseudo-random ones --
//                     and evaluates the best one in FP64.
// Measured (n = 2^21, lengths 64..512, learned r, per run): without witnesses
// phase 1 160 ms and the refine of its survivors 165 ms, the run 442 ms; with
// them step 13, hints 4, check 2, rescue 15, phase 1 4, refine 87 ms, the run
// 249 ms (120 to 135 ms with what was made faster since).  A step at n = 2^21 takes 28 us (bound by memory: 56 B per window, 4.2
// TB/s); one window per thread, the mean and the norm in two arrays, took 50.
// Phase 1 runs only when more windows are left than the refine should take
// (the first attempts of a run, where no window has a witness yet).  Phase 1
// and the refine record which pairs pruned a window; the next step evaluates
// those afresh (state WT_HINT).
//
// Soundness.  Every prune compares a lower bound of the exact correlation with
// thr.  The FP64 means carry an error of at most delta = 5e5 u A / m0 (prefix
// sums over a tile of at most 3074 values, <= 36 additions deep; u = 2^-53, A the
// largest |x|, m0 the shortest length of the run).  A step's term is off by
// |a| delta + |b| delta; a pair that has taken c_l steps over the value l (one, and
// two more per step back) is off by sum c_l (|a_l| + |b_l|) delta, at most
// s delta (n_i + n_w) with s^2 = sum c_l^2, by Cauchy-Schwarz (norms grow with the
// length), so the correlation is within t + t^2 with t = (s + 1) delta (inv_i +
// inv_w), the 1 for the pair's first dot product.  The host counts s^2 of the run
// (at least 1089: the at most 1021 lengths of a run without steps back all take
// s + 1 = 34).  2 t is subtracted, and 1e-7 for the FP32 rounding of thr.  A pair
// with t of the order of 1 proves nothing and prunes nothing.
// A step back (a missed attempt whose next length was already queued) takes one
// term away again: the norms shrink, and what the two steps over that term
// rounded may be large beside the shorter windows (a window of small values just
// before a spike).  With a, b the term's centred values at the shorter length, a
// step over it rounds by at most delta (|a| + |b| + delta) and 5 u |a b| (beside
// u |cov|, which the 1e-7 covers 1e8 times over), so 2.1 delta (|a| + |b| + 2
// delta) + 16 u (|a| + delta)(|b| + delta) per return, times inv_i inv_w, are
// subtracted as well.  At the longer length a and b are below the norms again.
#include <float.h>

#include <algorithm>
#include <cmath>

#include "paddi_internal.cuh"

namespace {

constexpr int WT_THREADS = 256;
constexpr int WT_SWIN = 4;      // windows per thread of the step
constexpr int WT_CWIN = 8;      // windows per thread of the check
constexpr int WT_MANY = 32768;  // hints from which on a thread takes one (below: a warp)
constexpr int WT_SOON = 64;     // lengths within which a partner counts as soon excluded
constexpr int WT_RWARPS = 4;    // warps per CTA of the rescue
constexpr int WT_MAXM = 1024;
constexpr int WT_BATCH = 8;     // partners ranked together
constexpr float WT_EASY = 0.1f; // a correlation this far above thr ends the search
constexpr double kU64 = 1.1102230246251565e-16;

// lower bound of a pair's correlation from its centred dot product
__device__ __forceinline__ float wt_bound(double c, double inv_i, double inv_w, double t1)
{
    if (inv_i == 0.0 || inv_w == 0.0) return -INFINITY; // flat windows: left to the selection
    return __double2float_rd(c * inv_i * inv_w - (1e-7 + 2.0 * t1 * (inv_i + inv_w)));
}

__device__ __forceinline__ bool wt_admissible(int i, int j, int N, int m)
{
    const int d = i > j ? i - j : j - i;
    return j >= 0 && j < N && d >= m - 1;
}

// A hint's partner windows: one or two groups of 4 consecutive windows
// starting at g0 (and g1); mask: the group's windows that are meant.
struct WtGroups {
    int g0, g1, n;
    unsigned mask;
};
__device__ __forceinline__ WtGroups wt_decode(double code)
{
    const int kind = (int)(code * (1.0 / WT_CODE));
    const int base = (int)(code - (double)kind * WT_CODE);
    WtGroups G;
    G.n = kind == WT_ROW ? 2 : 1;
    G.g0 = kind == WT_COL ? base - 3 : base;
    G.g1 = base + WT_PARTNER;
    G.mask = kind == WT_ONE ? 1u : 15u;
    return G;
}

// ------------------------------------------------------------------ step
// Bound by memory: 56 B read or written per window, the partner's mean and
// norm (one 16-byte entry) and its new value as gathers; neighbouring windows
// mostly have neighbouring witnesses.  WT_SWIN windows per thread keep that
// many chains wit -> partner in flight.  Hinted windows are listed for
// k_witness_hints.
// BACK: a step from m + 1, its rounding bounded as above (its own kernel: in one with
// the forward step the run of 449 lengths took 1.5 % longer).
template <bool BACK>
__global__ void __launch_bounds__(WT_THREADS)
k_witness_step(const float *__restrict__ x, const double2 *ms64, int32_t N,
               int32_t m, int32_t from, int32_t *wit, double *wc,
               float *wrho, int32_t *hint, uint32_t *scal,
               double dscale, double delta1, int32_t returns)
{
    paddi::chain_begin();
    const int i0 = blockIdx.x * (WT_THREADS * WT_SWIN) + threadIdx.x;
    const double t1 = dscale * (double)__uint_as_float(scal[WT_AMAX]);
    // the window's new value: the last one of length m, or (back to the length
    // before, for a repeated attempt) the one that length m does not have
    const int off = from == m + 1 ? m : m - 1;
    const double f = from == m - 1   ? (double)m / (double)(m - 1)
                     : from == m + 1 ? -(double)m / (double)(m + 1)
                                     : 0.0;
    const double delta = delta1 * (double)__uint_as_float(scal[WT_AMAX]);
    int w[WT_SWIN];
#pragma unroll
    for (int q = 0; q < WT_SWIN; ++q) {
        const int i = i0 + q * WT_THREADS;
        w[q] = i < N ? wit[i] : -1;
        if (i == N) wit[i] = -1; // a window of length m - 1 that this length does not have
    }
    double2 si[WT_SWIN], sw[WT_SWIN];
    float xi[WT_SWIN], xw[WT_SWIN];
    double c[WT_SWIN];
    bool ok[WT_SWIN];
#pragma unroll
    for (int q = 0; q < WT_SWIN; ++q) {
        const int i = i0 + q * WT_THREADS;
        ok[q] = w[q] >= 0 && wt_admissible(i, w[q], N, m);
        if (ok[q]) {
            si[q] = ms64[i];
            sw[q] = ms64[w[q]];
            c[q] = wc[i];
            xi[q] = f != 0.0 ? x[i + off] : 0.f;
            xw[q] = f != 0.0 ? x[w[q] + off] : 0.f;
        }
    }
#pragma unroll
    for (int q = 0; q < WT_SWIN; ++q) {
        const int i = i0 + q * WT_THREADS;
        float out = -INFINITY;
        if (ok[q]) {
            double ret = 0.0; // rounding of the returns over the term taken away
            if (f != 0.0) {
                const double a = (double)xi[q] - si[q].x, b = (double)xw[q] - sw[q].x;
                c[q] = fma(f * a, b, c[q]);
                wc[i] = c[q];
                if (BACK)
                    ret = (double)returns * (2.1 * delta * (fabs(a) + fabs(b) + 2.0 * delta) +
                                             16.0 * kU64 * (fabs(a) + delta) * (fabs(b) + delta));
            }
            out = wt_bound(BACK ? c[q] - ret : c[q], si[q].y, sw[q].y, t1);
        } else if (w[q] >= 0) {
            wit[i] = -1;
        }
        if (i < N) wrho[i] = out;
        const unsigned h = __ballot_sync(0xffffffffu, w[q] == WT_HINT);
        if (h) {
            const int lane = threadIdx.x & 31;
            int base = 0;
            if (lane == 0) base = (int)atomicAdd(scal + WT_NHINT, (uint32_t)__popc(h));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (w[q] == WT_HINT) hint[base + __popc(h & ((1u << lane) - 1u))] = i;
        }
    }
}

// ------------------------------------------------------------------ hints
// Direct FP64 dot products of the listed windows with the up to 8 partners of
// their hints; the best one becomes the witness (partners that the growing
// exclusion zone soon reaches come last).  Many hints (after phase 1): one
// thread per window, a register ring over the partners' common stretch; few
// (after a refine): the warp along one window.
struct WtBest {
    double rank, c;
    int j;
};
__device__ __forceinline__ void wt_settle(WtBest &B, int i, int j, double c, const double2 &sj,
                                          double ii, int N, int m)
{
    if (!wt_admissible(i, j, N, m)) return;
    const double rank = c * ii * sj.y - (abs(i - j) < m + WT_SOON ? 1.0 : 0.0);
    if (rank > B.rank) {
        B.rank = rank;
        B.c = c;
        B.j = j;
    }
}

__global__ void __launch_bounds__(WT_THREADS)
k_witness_hints(const float *__restrict__ x, const double2 *ms64, int32_t N,
                int32_t m, int32_t *wit, double *wc,
                float *wrho, const int32_t *hint, uint32_t *scal,
                double dscale, unsigned long long *t_end)
{
    paddi::chain_begin();
    const int nh = (int)scal[WT_NHINT];
    const int lane = threadIdx.x & 31;
    const int nser = N + m - 1;
    const double t1 = dscale * (double)__uint_as_float(scal[WT_AMAX]);
    auto at = [&](int k) { return (double)x[min(max(k, 0), nser - 1)]; };
    auto store = [&](int i, const WtBest &B, double ii) {
        wit[i] = B.j;
        wc[i] = B.c;
        wrho[i] = B.j >= 0 ? wt_bound(B.c, ii, ms64[B.j].y, t1) : -INFINITY;
    };
    if (nh >= WT_MANY) {
        // ranked in FP32, the best partner then evaluated in FP64
        for (int e = blockIdx.x * WT_THREADS + threadIdx.x; e < nh; e += gridDim.x * WT_THREADS) {
            const int i = hint[e];
            const WtGroups G = wt_decode(wc[i]);
            const double2 si = ms64[i];
            WtBest B = {-INFINITY, 0.0, -1};
            const float mf = (float)si.x;
            for (int q = 0; q < G.n; ++q) {
                const int g = q ? G.g1 : G.g0;
                const float sh = (float)at(g);
                float acc[4] = {0.f, 0.f, 0.f, 0.f}, y[4], as = 0.f;
                auto atf = [&](int k) { return x[min(max(k, 0), nser - 1)] - sh; };
#pragma unroll
                for (int c = 0; c < 3; ++c) y[c] = atf(g + c);
                for (int k = 0; k < m; ++k) {
                    const float a = x[i + k] - mf;
                    y[3] = atf(g + k + 3);
                    as += a;
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c] = fmaf(a, y[c], acc[c]);
                    y[0] = y[1];
                    y[1] = y[2];
                    y[2] = y[3];
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if ((G.mask >> c) & 1u && g + c >= 0 && g + c < N) {
                        const double2 sj = ms64[g + c];
                        wt_settle(B, i, g + c,
                                  (double)acc[c] - (sj.x - (double)sh) * (double)as, sj, si.y, N, m);
                    }
            }
            if (B.j >= 0) {
                const double mj = ms64[B.j].x;
                double c0 = 0.0, c1 = 0.0;
                int k = 0;
                for (; k + 2 <= m; k += 2) {
                    c0 = fma((double)x[i + k] - si.x, (double)x[B.j + k] - mj, c0);
                    c1 = fma((double)x[i + k + 1] - si.x, (double)x[B.j + k + 1] - mj, c1);
                }
                if (k < m) c0 = fma((double)x[i + k] - si.x, (double)x[B.j + k] - mj, c0);
                B.c = c0 + c1;
            }
            store(i, B, si.y);
        }
    } else {
        const int nw = gridDim.x * (WT_THREADS / 32);
        for (int e = (blockIdx.x * WT_THREADS + threadIdx.x) >> 5; e < nh; e += nw) {
            const int i = hint[e];
            const WtGroups G = wt_decode(wc[i]);
            const double2 si = ms64[i];
            WtBest B = {-INFINITY, 0.0, -1};
            for (int q = 0; q < G.n; ++q) {
                const int g = q ? G.g1 : G.g0;
                const double sh = at(g);
                double acc[4] = {0.0, 0.0, 0.0, 0.0}, as = 0.0;
                for (int k = lane; k < m; k += 32) {
                    const double a = (double)x[i + k] - si.x;
                    as += a;
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c] = fma(a, at(g + k + c) - sh, acc[c]);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    as += __shfl_xor_sync(0xffffffffu, as, o);
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if ((G.mask >> c) & 1u && g + c >= 0 && g + c < N) {
                        const double2 sj = ms64[g + c];
                        wt_settle(B, i, g + c, acc[c] - (sj.x - sh) * as, sj, si.y, N, m);
                    }
            }
            __syncwarp(); // every lane has read wc[i]
            if (lane == 0) store(i, B, si.y);
        }
    }
    // the last CTA clears the list for the next step
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(scal + WT_DONE, 1u) == gridDim.x - 1) {
            scal[WT_NHINT] = 0;
            scal[WT_DONE] = 0;
        }
        paddi::stamp_end(t_end);
    }
}

// Largest |x| as the bits of a non-negative float (zeroed by the caller; a NaN
// sorts above everything and disables the prunes).
__global__ void __launch_bounds__(WT_THREADS)
k_absmax(const float *__restrict__ x, int64_t n, uint32_t *amax)
{
    uint32_t v = 0;
    for (int64_t i = blockIdx.x * (int64_t)WT_THREADS + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * WT_THREADS)
        v = max(v, __float_as_uint(x[i]) & 0x7fffffffu);
    v = __reduce_max_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) atomicMax(amax, v);
}

// ------------------------------------------------------------------ check
// alive[i] = 0 where the witness proves it; the others are listed (order
// within a CTA kept).  5 B per window.
__global__ void __launch_bounds__(WT_THREADS)
k_witness_check(const float *wrho, int32_t N, float thr, uint8_t *alive,
                int32_t *fail, PaddiAttemptDev *att)
{
    paddi::chain_begin();
    paddi::stamp_begin(att->t + PADDI_T_BEGIN);
    __shared__ int wcnt[WT_THREADS / 32];
    __shared__ int base;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int i0 = (blockIdx.x * WT_THREADS + threadIdx.x) * WT_CWIN;
    unsigned mask = 0;
    if (i0 + WT_CWIN <= N) {
        const float4 a = *reinterpret_cast<const float4 *>(wrho + i0);
        const float4 b = *reinterpret_cast<const float4 *>(wrho + i0 + 4);
        const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t lo = 0, hi = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const unsigned f0 = !(v[q] > thr), f1 = !(v[q + 4] > thr); // NaN: still a candidate
            mask |= f0 << q | f1 << (q + 4);
            lo |= f0 << (8 * q);
            hi |= f1 << (8 * q);
        }
        *reinterpret_cast<uint2 *>(alive + i0) = make_uint2(lo, hi);
    } else {
        for (int q = 0; q < WT_CWIN && i0 + q < N; ++q) {
            const unsigned f = !(wrho[i0 + q] > thr);
            mask |= f << q;
            alive[i0 + q] = (uint8_t)f;
        }
    }
    const int cnt = __popc(mask);
    int inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wcnt[wp] = inc;
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int q = 0; q < WT_THREADS / 32; ++q) {
            const int t = wcnt[q];
            wcnt[q] = s;
            s += t;
        }
        base = s ? atomicAdd(&att->n_fail, s) : 0;
    }
    __syncthreads();
    int pos = base + wcnt[wp] + inc - cnt;
    while (mask) {
        fail[pos++] = i0 + __ffs(mask) - 1;
        mask &= mask - 1;
    }
}

// ------------------------------------------------------------------ rescue
// 32-bit integer hash "lowbias32" (C. Wellons, hash-prospector)
__device__ __forceinline__ uint32_t wt_hash(uint32_t a)
{
    a ^= a >> 16;
    a *= 0x7feb352du;
    a ^= a >> 15;
    a *= 0x846ca68bu;
    return a ^ (a >> 16);
}

__global__ void __launch_bounds__(32 * WT_RWARPS)
k_witness_rescue(const float *__restrict__ x, const double2 *ms64, int32_t N, int32_t m, float thr,
                 const int32_t *fail, const int32_t *n_fail,
                 int32_t limit, int32_t *wit, double *wc, float *wrho,
                 uint8_t *alive, int32_t *n_rescued,
                 const uint32_t *scal, double dscale)
{
    extern __shared__ float wt_a[]; // per warp: the centred window
    paddi::chain_begin();
    const int nf = __ldcg(n_fail);
    if (nf > limit) return;
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    float *a = wt_a + (size_t)wp * m;
    const double t1 = dscale * (double)__uint_as_float(scal[WT_AMAX]);
    for (int f = blockIdx.x * WT_RWARPS + wp; f < nf; f += gridDim.x * WT_RWARPS) {
        const int i = fail[f];
        const double2 si = ms64[i];
        const double mi = si.x, ii = si.y;
        if (ii == 0.0) continue; // flat
        __syncwarp();
        for (int k = lane; k < m; k += 32) a[k] = (float)((double)x[i + k] - mi);
        // lanes 0..3 pseudo-random partners; 4..17: the witnesses of the partners that
        // nearby windows' diagonals give; 18..31: those partners themselves
        int j = -1;
        if (lane < 4) {
            j = (int)(wt_hash((uint32_t)i * 4u + (uint32_t)lane + (uint32_t)m * 0x9e3779b9u) %
                      (uint32_t)N);
        } else {
            const int q = lane < 18 ? lane - 4 : lane - 18;
            const int step = (q >> 1) < 4 ? (q >> 1) + 1 : 1 << ((q >> 1) - 1); // 1 2 3 4 8 16 32
            const int o = (q & 1) ? -step : step;
            const int s = i + o;
            if (s >= 0 && s < N) {
                const int ws = __ldcg(wit + s);
                if (ws >= 0) j = ws - o;
            }
            if (lane < 18 && j >= 0 && j < N) {
                const int v = __ldcg(wit + j);
                j = v >= 0 ? v : -1;
            }
        }
        if (!wt_admissible(i, j, N, m)) j = -1;
        const double2 sj = j >= 0 ? ms64[j] : make_double2(0.0, 0.0);
        const float ij = (float)sj.y * (float)ii;
        const float muj = (float)sj.x;
        const unsigned have = __ballot_sync(0xffffffffu, j >= 0);
        __syncwarp();
        // FP32 correlations of 8 partners at a time, the lanes along the window;
        // a batch that holds a promising one ends the search
        float rb = -INFINITY;
        int jb = -1;
        for (int b0 = 0; b0 < 32; b0 += WT_BATCH) {
            if (!((have >> b0) & 0xffu)) continue;
            float acc[WT_BATCH], mq[WT_BATCH];
            const float *y[WT_BATCH];
#pragma unroll
            for (int q = 0; q < WT_BATCH; ++q) {
                const int jq = __shfl_sync(0xffffffffu, j, b0 + q);
                mq[q] = __shfl_sync(0xffffffffu, muj, b0 + q);
                y[q] = x + max(jq, 0);
                acc[q] = 0.f;
            }
            for (int k = lane; k < m; k += 32) {
                const float ak = a[k];
#pragma unroll
                for (int q = 0; q < WT_BATCH; ++q) acc[q] = fmaf(ak, y[q][k] - mq[q], acc[q]);
            }
            // transposing reduction: lane l ends with the sum of partner l / 4
#pragma unroll
            for (int h = WT_BATCH / 2, o = 16; h >= 1; h >>= 1, o >>= 1) {
                const bool up = lane & o;
#pragma unroll
                for (int q = 0; q < WT_BATCH / 2; ++q)
                    if (q < h) {
                        const float mine = up ? acc[q + h] : acc[q];
                        acc[q] = mine + __shfl_xor_sync(0xffffffffu, up ? acc[q] : acc[q + h], o);
                    }
            }
            float v = acc[0];
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            const int src = b0 + (lane >> 2);
            const float iq = __shfl_sync(0xffffffffu, ij, src);
            const int jq = __shfl_sync(0xffffffffu, j, src);
            float r = jq >= 0 ? v * iq : -INFINITY;
            if (!(r > -2.f)) r = -INFINITY; // no partner, or NaN
            else if (abs(jq - i) < m + WT_SOON) r -= 0.5f; // soon excluded: comes last
            float best = r;
#pragma unroll
            for (int o = 16; o >= 4; o >>= 1)
                best = fmaxf(best, __shfl_xor_sync(0xffffffffu, best, o));
            if (best > rb) {
                rb = best;
                jb = __shfl_sync(0xffffffffu, jq, __ffs(__ballot_sync(0xffffffffu, r == best)) - 1);
            }
            if (rb > thr + WT_EASY) break;
        }
        if (jb < 0) continue;
        j = jb;
        const double2 sb = ms64[j];
        double c = 0.0;
        for (int k = lane; k < m; k += 32)
            c = fma((double)x[i + k] - mi, (double)x[j + k] - sb.x, c);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
        if (lane == 0) {
            const float b = wt_bound(c, ii, sb.y, t1);
            const bool ok = b > thr;
            if (ok || b > wrho[i]) {
                wit[i] = j;
                wc[i] = c;
                wrho[i] = b;
            }
            if (ok) {
                alive[i] = 0;
                atomicAdd(n_rescued, 1);
            }
        }
    }
}

// delta over the largest |x|, and t over that and the inverse norms
double wt_delta(int32_t m0) { return 5e5 / (double)m0 * kU64; }
double wt_dscale(const PaddiWitnessRun &R)
{
    return (std::sqrt(std::max(1089.0, R.steps2)) + 1.0) * wt_delta(R.m0);
}

} // namespace

cudaError_t paddi_launch_witness_start(const float *x, int64_t n, int32_t N, const PaddiWitness &W,
                                       int32_t num_sms, cudaStream_t st)
{
    cudaError_t e = cudaMemsetAsync(W.wit, 0xff, sizeof(int32_t) * (size_t)N, st); // -1
    if (e == cudaSuccess) // NaN: proves nothing
        e = cudaMemsetAsync(W.wrho, 0xff, sizeof(float) * (size_t)N, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(W.scal, 0, sizeof(uint32_t) * 4, st);
    if (e != cudaSuccess) return e;
    k_absmax<<<num_sms * 4, WT_THREADS, 0, st>>>(x, n, W.scal + WT_AMAX);
    return cudaGetLastError();
}

cudaError_t paddi_launch_witness_step(const float *x, const double2 *ms64,
                                      int32_t N, int32_t m, int32_t from,
                                      const PaddiWitnessRun &R, const PaddiWitness &W,
                                      int32_t *hint, int32_t num_sms, cudaStream_t st,
                                      unsigned long long *t_end)
{
    if (m < 3 || m > WT_MAXM || N < 1 || from < m - 1 || from > m + 1) return cudaErrorInvalidValue;
    const int per = WT_THREADS * WT_SWIN;
    // the partner gathers live off L1, and the kernel before (k_prep) leaves the SM with
    // nearly all of it as shared memory: without a preference of its own the step ran
    // under that split (headline run, statistics and step of a length: 104 us behind
    // four k_prep CTAs per SM, 79 behind three, 66 with the preference and four)
    auto kern = from == m + 1 ? k_witness_step<true> : k_witness_step<false>;
    cudaError_t e = paddi_launch_carveout(0, true, kern, (unsigned)(N / per + 1), WT_THREADS, 0, st, x,
                                 ms64, N, m, from, W.wit, W.wc, W.wrho, hint, W.scal,
                                 wt_dscale(R), wt_delta(R.m0), R.returns);
    if (e != cudaSuccess) return e;
    return paddi_launch(true, k_witness_hints, num_sms * 4, WT_THREADS, 0, st, x, ms64, N, m, W.wit,
                        W.wc, W.wrho, hint, W.scal, wt_dscale(R), t_end);
}

cudaError_t paddi_launch_witness_check(const double2 *ms64, const float *x,
                                       int32_t N, int32_t m, float thr,
                                       const PaddiWitnessRun &R, const PaddiWitness &W, uint8_t *alive, int32_t *fail,
                                       PaddiAttemptDev *att, int32_t limit, int32_t num_sms,
                                       cudaStream_t st)
{
    const int per = WT_THREADS * WT_CWIN;
    cudaError_t e = paddi_launch(true, k_witness_check, (unsigned)((N + per - 1) / per), WT_THREADS,
                                 0, st, W.wrho, N, thr, alive, fail, att);
    if (e != cudaSuccess) return e;
    const size_t smem = sizeof(float) * (size_t)WT_RWARPS * (size_t)m;
    return paddi_launch(true, k_witness_rescue, num_sms * 8, 32 * WT_RWARPS, smem, st, x, ms64, N, m,
                        thr, fail, &att->n_fail, limit, W.wit, W.wc, W.wrho, alive,
                        &att->n_rescued, W.scal, wt_dscale(R));
}
