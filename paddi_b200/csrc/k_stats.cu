// k_stats.cu -- per-length window statistics from FP64 prefix sums.
//
// Replaces the reference's gpu_compute_statistics / gpu_update_statistics
// (src/preprocessing.cuh:12-65: FP32, one-pass E[x^2]-mu^2, chained updates
// from length m-1 to m).  Here every length is computed afresh, tile by tile
// (k_stats.cuh).  k_window_stats serves the FP32 refine's lengths and the
// allocation-free entry point; the tensor-core lengths get their statistics
// from k_prep (k_refine_umma.cu) together with the refine's tiles.
// k_mean_std writes only the mean and the standard deviation (the reference's
// compute_statistics): 12 B of HBM traffic per window instead of 53 with an
// export pass after k_window_stats (n = 2^21, m = 256: 30.4 us a call, now 11.4).  What bounds all of them is FP64 issue and the latency of a tile's
// phases, not memory.
#include "k_stats.cuh"

namespace {

__global__ void __launch_bounds__(ST_THREADS)
k_window_stats(const float *__restrict__ x, int64_t n, int32_t m, int32_t N, StOut O)
{
    extern __shared__ __align__(16) unsigned char st_mem[];
    __shared__ StShared S;
    st_begin(O.extra);
    const int64_t t0 = (int64_t)blockIdx.x * ST_TILE;
    const StTile T = st_prefix(st_mem, S, x, n, m, t0);
    float iv[ST_WPT], mv[ST_WPT];
    st_write(T, O, t0, m, N, iv, mv);
}

// mean / population std in the reference's FP32 layout (src/preprocessing.cuh:31-34)
__global__ void __launch_bounds__(ST_THREADS)
k_mean_std(const float *__restrict__ x, int64_t n, int32_t m, int32_t N, float *__restrict__ mean,
           float *__restrict__ sd)
{
    extern __shared__ __align__(16) unsigned char st_mem[];
    __shared__ StShared S;
    const int64_t t0 = (int64_t)blockIdx.x * ST_TILE;
    const StTile T = st_prefix(st_mem, S, x, n, m, t0);
    const double invm = 1.0 / (double)m, rsm = 1.0 / sqrt((double)m);
    for (int l = threadIdx.x; l < ST_TILE && t0 + l < N; l += ST_THREADS) {
        const StWindow W = st_window(T, l, m, invm);
        mean[t0 + l] = (float)W.mu;
        sd[t0 + l] = (float)(W.nrm * rsm);
    }
}

__global__ void k_export_stats(const double2 *__restrict__ ms64, int32_t N, int32_t m, float *mean,
                               float *sd)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    mean[i] = (float)ms64[i].x;
    const double iv = ms64[i].y;
    sd[i] = iv > 0.0 ? (float)(1.0 / (iv * sqrt((double)m))) : 0.f;
}

} // namespace

cudaError_t paddi_launch_export_stats(const double2 *ms64, int32_t N, int32_t m, float *mean,
                                      float *sd, cudaStream_t st)
{
    k_export_stats<<<(N + 255) / 256, 256, 0, st>>>(ms64, N, m, mean, sd);
    return cudaGetLastError();
}

cudaError_t paddi_launch_mean_std(const float *x, int64_t n, int32_t m, float *mean, float *sd,
                                  cudaStream_t st)
{
    if (m < 2 || m > ST_MAXM || n < 2 * (int64_t)m) return cudaErrorInvalidValue;
    const int32_t N = (int32_t)(n - m + 1);
    const size_t smem = st_smem(m);
    cudaError_t e = paddi_raise_smem_limit((const void *)k_mean_std, smem);
    if (e != cudaSuccess) return e;
    k_mean_std<<<(unsigned)((N + ST_TILE - 1) / ST_TILE), ST_THREADS, smem, st>>>(x, n, m, N, mean,
                                                                                 sd);
    return cudaGetLastError();
}

cudaError_t paddi_launch_stats(const float *x, int64_t n, int32_t m, float4 *wst, float *mu,
                               double2 *ms64, uint8_t *flat, int32_t *flat_count, cudaStream_t st,
                               int32_t *flat_span, bool chained, const PaddiStatsExtra &extra)
{
    if (m < 2 || m > ST_MAXM || n < 2 * (int64_t)m) return cudaErrorInvalidValue;
    const int32_t N = (int32_t)(n - m + 1);
    const int64_t total = (int64_t)N + PADDI_PAD_WIN;
    const unsigned grid = (unsigned)((total + ST_TILE - 1) / ST_TILE);
    const size_t smem = st_smem(m);
    cudaError_t e = paddi_raise_smem_limit((const void *)k_window_stats, smem);
    if (e != cudaSuccess) return e;
    const StOut O = {wst, mu, ms64, flat, flat_count, flat_span, extra};
    return paddi_launch(chained, k_window_stats, grid, ST_THREADS, smem, st, x, n, m, N, O);
}
