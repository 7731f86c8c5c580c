// k_stats.cuh -- window statistics of one 2048-window tile from FP64 prefix
// sums, shared by k_window_stats (k_stats.cu) and the tensor-core refine's
// preparation (k_prep in k_refine_umma.cu).
//
// A CTA stages a tile of the series, shifts it by the tile's first value c and
// builds exclusive FP64 prefix sums of (x-c) and (x-c)^2 in shared memory;
// window sums are differences of two prefix entries, so the variance never
// subtracts two numbers of the size of the raw values; flatness (all m values
// equal) is an exact integer test on a prefix count of equal neighbours.
#pragma once
#include <limits.h>

#include "paddi_internal.cuh"

constexpr int ST_THREADS = 256;
constexpr int ST_TILE = 2048; // windows per CTA (the staged halo of m values is amortised over them)
constexpr int ST_WPT = ST_TILE / ST_THREADS; // windows per thread
constexpr int ST_MAXM = 1024; // longest supported window

// dynamic shared memory of one CTA for length m: P1, P2 (FP64 prefixes), E
// (prefix of equal neighbours, at most ST_TILE + m) and the staged values, ST_TILE + m + 2
// each
__host__ __device__ inline size_t st_smem(int m)
{
    const size_t L = (size_t)ST_TILE + (size_t)m + 2;
    return L * (2 * sizeof(double) + sizeof(float) + sizeof(uint16_t));
}

struct StTile {
    double *P1, *P2;
    float *xs;
    uint16_t *E;
    float c;
};

// Warp totals of the block scan.
struct StShared {
    double s1[ST_THREADS / 32], s2[ST_THREADS / 32];
    int se[ST_THREADS / 32];
};

// Stages x[t0 .. t0 + ST_TILE + m] and builds the prefixes.  The three sums are
// scanned together with one barrier between the warps' scans and the block's
// (three scans with three barriers each took a third of the kernel); an odd
// number of values per thread keeps the strided 8-byte accesses conflict-free.
__device__ __forceinline__ StTile st_prefix(unsigned char *mem, StShared &S, const float *x,
                                            int64_t n, int32_t m, int64_t t0)
{
    const int LS = ST_TILE + m + 2;
    StTile T;
    T.P1 = reinterpret_cast<double *>(mem);
    T.P2 = T.P1 + LS;
    T.xs = reinterpret_cast<float *>(T.P2 + LS);
    T.E = reinterpret_cast<uint16_t *>(T.xs + LS);
    const int len = ST_TILE + m + 1; // values staged
    T.c = x[t0 < n ? t0 : n - 1];
    for (int k = threadIdx.x; k < len; k += ST_THREADS) {
        const int64_t g = t0 + k;
        T.xs[k] = g < n ? x[g] : T.c;
    }
    __syncthreads();
    // per-thread serial chunk, then a scan of the chunk totals
    const int per = ((len + ST_THREADS - 1) / ST_THREADS) | 1;
    const int k0 = threadIdx.x * per, k1 = min(len, k0 + per);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double c = (double)T.c;
    double s1 = 0.0, s2 = 0.0;
    int se = 0;
    for (int k = k0; k < k1; ++k) {
        const double d = (double)T.xs[k] - c;
        s1 += d;
        s2 = fma(d, d, s2);
        se += k + 1 < len ? T.xs[k] == T.xs[k + 1] : 0;
    }
    double i1 = s1, i2 = s2;
    int ie = se;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double a = __shfl_up_sync(0xffffffffu, i1, o), b = __shfl_up_sync(0xffffffffu, i2, o);
        const int e = __shfl_up_sync(0xffffffffu, ie, o);
        if (lane >= o) {
            i1 += a;
            i2 += b;
            ie += e;
        }
    }
    if (lane == 31) {
        S.s1[w] = i1;
        S.s2[w] = i2;
        S.se[w] = ie;
    }
    // exclusive within the warp
    double b1 = __shfl_up_sync(0xffffffffu, i1, 1), b2 = __shfl_up_sync(0xffffffffu, i2, 1);
    int be = __shfl_up_sync(0xffffffffu, ie, 1);
    if (lane == 0) {
        b1 = b2 = 0.0;
        be = 0;
    }
    __syncthreads();
    double w1 = 0.0, w2 = 0.0;
    int we = 0;
#pragma unroll
    for (int q = 0; q < ST_THREADS / 32; ++q)
        if (q < w) {
            w1 += S.s1[q];
            w2 += S.s2[q];
            we += S.se[q];
        }
    b1 += w1;
    b2 += w2;
    be += we;
    // exclusive prefixes: P[k] = sum over staged values < k
    for (int k = k0; k < k1; ++k) {
        T.P1[k] = b1;
        T.P2[k] = b2;
        T.E[k] = (uint16_t)be;
        const double d = (double)T.xs[k] - c;
        b1 += d;
        b2 = fma(d, d, b2);
        be += k + 1 < len ? T.xs[k] == T.xs[k + 1] : 0;
    }
    if (k0 < len && k1 == len) {
        T.P1[len] = b1;
        T.P2[len] = b2;
        T.E[len] = (uint16_t)be;
    }
    __syncthreads();
    return T;
}

// Window l of the tile: FP64 mean, norm |x - mu| and its inverse (both 0 when
// flat).
struct StWindow {
    double mu, nrm, inv;
    bool flat;
};
__device__ __forceinline__ StWindow st_window(const StTile &T, int l, int m, double invm)
{
    StWindow W;
    const double a1 = T.P1[l + m] - T.P1[l], a2 = T.P2[l + m] - T.P2[l];
    const bool fe = (T.E[l + m - 1] - T.E[l]) == (m - 1);
    const double um = a1 * invm;
    const double q = a2 - a1 * um;
    W.flat = fe || !(q > 0.0);
    W.inv = W.flat ? 0.0 : rsqrt(q); // one rsqrt for the square root and the division
    W.nrm = W.flat ? 0.0 : q * W.inv;
    W.mu = fe ? (double)T.xs[l] : (double)T.c + um;
    return W;
}

// Mean of window l alone (the next window's, for its neighbour's dg).
__device__ __forceinline__ double st_mean(const StTile &T, int l, int m, double invm)
{
    const bool fe = (T.E[l + m - 1] - T.E[l]) == (m - 1);
    return fe ? (double)T.xs[l] : (double)T.c + (T.P1[l + m] - T.P1[l]) * invm;
}

struct StOut {
    float4 *wst;
    float *mu;
    double2 *ms64;
    uint8_t *flat;
    int32_t *flat_count, *flat_span;
    PaddiStatsExtra extra;
};

// Start of a statistics kernel: what it prepares for the kernels after it.
__device__ __forceinline__ void st_begin(const PaddiStatsExtra &extra)
{
    paddi::chain_begin();
    paddi::stamp_begin(extra.t);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (extra.next)
            for (int k = 0; k < 4; ++k) extra.next[k] = 0;
        if (extra.guide) extra.guide->nn_ord = ~0ull;
    }
}

// The tile's windows to global memory (zeroed past N, so tiles can over-read);
// iv / mv: the FP32 inverse norms and means of this thread's windows l =
// threadIdx.x + ST_THREADS k.
__device__ __forceinline__ void st_write(const StTile &T, const StOut &O, int64_t t0, int32_t m,
                                         int32_t N, float (&iv)[ST_WPT], float (&mv)[ST_WPT])
{
    const double invm = 1.0 / (double)m;
    int nflat = 0;
#pragma unroll
    for (int k = 0; k < ST_WPT; ++k) {
        const int l = threadIdx.x + ST_THREADS * k;
        const int64_t i = t0 + l;
        iv[k] = mv[k] = 0.f;
        if (i >= (int64_t)N + PADDI_PAD_WIN) continue;
        if (i >= N) {
            O.wst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            O.mu[i] = 0.f;
            O.ms64[i] = make_double2(0.0, 0.0);
            O.flat[i] = 0;
            continue;
        }
        const StWindow W = st_window(T, l, m, invm);
        float df = 0.f, dg = 0.f;
        if (i + 1 < N) {
            const double xe = (double)T.xs[l + m], xb = (double)T.xs[l];
            df = (float)((xe - xb) * 0.5);
            dg = (float)((xe - st_mean(T, l + 1, m, invm)) + (xb - W.mu));
        }
        iv[k] = (float)W.inv;
        mv[k] = (float)W.mu;
        O.wst[i] = make_float4(df, dg, iv[k], (float)W.nrm);
        O.mu[i] = mv[k];
        O.ms64[i] = make_double2(W.mu, W.inv);
        O.flat[i] = (uint8_t)W.flat;
        if (O.extra.alive) O.extra.alive[i] = 1;
        nflat += W.flat;
        // lowest and highest flat window, both kept as maxima over a zeroed
        // pair: {INT_MAX - lowest, highest + 1} (flat windows are rare)
        if (W.flat && O.flat_span) {
            atomicMax(O.flat_span, INT_MAX - (int)i);
            atomicMax(O.flat_span + 1, (int)i + 1);
        }
    }
    if (nflat) atomicAdd(O.flat_count, nflat);
}
