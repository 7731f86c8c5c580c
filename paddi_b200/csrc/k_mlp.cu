// k_mlp.cu -- the learned r predictor: a 12 -> 64 -> 64 -> 1 MLP with GELU,
// trained and evaluated by these kernels (no framework).
//
// It predicts y = log(d_m / d_{m-1}), the growth of the top-1 squared
// discord distance from one length to the next, from features of the
// previous lengths (see paddi_r_features).  Training minimises the pinball
// (quantile) loss at quantile tau, so the prediction is a low quantile of
// the growth: r^2 = d_{m-1} * exp(y_hat) then usually lies just below the
// true top-1 distance.  A guess above it only costs a retry: PALMAD lowers r
// the way MERLIN does and the discords do not depend on r.
//
// Parameter vector (FP32, MLP_NPARAM values):
//   W1[64][12]  b1[64]  W2[64][64]  b2[64]  W3[64]  b3
// Inference uses a BF16 copy of the weights with FP32 accumulation.
//
// Inference: one warp evaluates one sample; lane l owns hidden units l and l + 32.
// Training: a CTA takes tiles of 32 samples through forward and backward as
// small matrix products in shared memory (8 outputs per thread and step), keeps
// its share of the gradient in registers over all its tiles and adds it to the
// global gradient once; an Adam kernel applies the step.  With one warp per
// sample and a gradient per warp in shared memory, a batch of 4096 spent its
// time on 2368 warps loading the parameters and adding 5057 values each to the
// same addresses; now 128 CTAs do: 70 us a batch, 24 with FP32 sums and 28 with the
// FP64 sums of k_mlp_adam's gradient (staging the parameters, a chain of five small
// products, and the atomics, in about equal parts).
#include <cuda_bf16.h>

#include <cmath>

#include "paddi_internal.cuh"

namespace {

constexpr int F = MLP_NFEAT, H = MLP_HIDDEN;
constexpr int OW1 = 0, OB1 = OW1 + H * F, OW2 = OB1 + H, OB2 = OW2 + H * H, OW3 = OB2 + H,
              OB3 = OW3 + H;
static_assert(OB3 + 1 == MLP_NPARAM, "parameter layout");

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678f)); }
// GELU and its derivative Phi(z) + z phi(z) together.
__device__ __forceinline__ void gelu2(float z, float &g, float &d)
{
    const float phi = 0.5f * (1.f + erff(z * 0.70710678f));
    g = z * phi;
    d = phi + z * 0.39894228f * expf(-0.5f * z * z);
}

template <typename W>
__device__ __forceinline__ float ld(const W *p, int i);
template <>
__device__ __forceinline__ float ld<float>(const float *p, int i) { return p[i]; }
template <>
__device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16 *p, int i)
{
    return __bfloat162float(p[i]);
}

// Parameters of one model.  (This struct and what mlp_forward returns beside y served
// the earlier training kernel too; a forward pass without them let the compiler
// contract the output sum the other way, which moved predictions in the last place.)
template <typename W>
struct MlpView {
    const W *w1, *b1, *w2, *b2, *w3, *b3;
    int w2s; // row stride of W2
};

template <typename W>
__device__ __forceinline__ MlpView<W> packed_view(const W *P)
{
    return MlpView<W>{P + OW1, P + OB1, P + OW2, P + OB2, P + OW3, P + OB3, H};
}

// Forward pass of one sample by one warp; returns y_hat on every lane and the
// pre-activations / activations of the lane's two units per layer.
template <typename W>
__device__ float mlp_forward(const MlpView<W> &P, const float *x, int lane, float (&z1)[2],
                             float (&h1)[2], float (&z2)[2], float (&h2)[2])
{
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int u = lane + 32 * q;
        float a = ld(P.b1, u);
#pragma unroll
        for (int k = 0; k < F; ++k) a = fmaf(ld(P.w1, u * F + k), x[k], a);
        z1[q] = a;
        h1[q] = gelu(a);
    }
    float a0 = ld(P.b2, lane), a1 = ld(P.b2, lane + 32);
#pragma unroll 4
    for (int v = 0; v < H; ++v) {
        const float hv = __shfl_sync(0xffffffffu, v < 32 ? h1[0] : h1[1], v & 31);
        a0 = fmaf(ld(P.w2, lane * P.w2s + v), hv, a0);
        a1 = fmaf(ld(P.w2, (lane + 32) * P.w2s + v), hv, a1);
    }
    z2[0] = a0;
    z2[1] = a1;
    h2[0] = gelu(a0);
    h2[1] = gelu(a1);
    float y = ld(P.w3, lane) * h2[0] + ld(P.w3, lane + 32) * h2[1];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    return y + ld(P.b3, 0);
}

template <typename W>
__global__ void k_mlp_forward(const float *__restrict__ X, int n, const W *__restrict__ Pg,
                              float *Y)
{
    const int lane = threadIdx.x & 31;
    const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const MlpView<W> P = packed_view(Pg);
    for (int s = wid; s < n; s += nw) {
        float x[F];
#pragma unroll
        for (int k = 0; k < F; ++k) x[k] = X[(size_t)s * F + k];
        float z1[2], h1[2], z2[2], h2[2];
        const float y = mlp_forward(P, x, lane, z1, h1, z2, h2);
        if (lane == 0) Y[s] = y;
    }
}

// Gradient of the mean pinball loss over n samples (rows perm[0..n) of X and
// Yt, or 0..n-1; added into G; the mean loss into *loss).
constexpr int GT = 256;    // threads
constexpr int GS = 32;     // samples per tile
constexpr int LD = H + 4;  // row stride of the tile's arrays (16-byte rows, banks spread)
struct GradSmem {
    float w1t[F][H];          // W1 transposed
    float w2[H][H], w2t[H][H];
    float b1[H], b2[H], w3[H];
    float x[GS][F];
    float h1[GS][LD], d1[GS][LD], dz1[GS][LD]; // activations, GELU', deltas
    float h2[GS][LD], dz2[GS][LD];
    float dy[GS];
};

__global__ void __launch_bounds__(GT)
k_mlp_grad(const float *__restrict__ X, const float *__restrict__ Yt,
           const uint32_t *__restrict__ perm, int n, float tau, const float *P, double *G,
           double *loss)
{
    extern __shared__ __align__(16) unsigned char g_mem[];
    GradSmem &S = *reinterpret_cast<GradSmem *>(g_mem);
    paddi::chain_begin();
    const int t = threadIdx.x;
    for (int i = t; i < H * F; i += GT) S.w1t[i % F][i / F] = __ldcg(P + OW1 + i);
    for (int i = t; i < H * H; i += GT) {
        const float v = __ldcg(P + OW2 + i);
        S.w2[i / H][i % H] = v;
        S.w2t[i % H][i / H] = v;
    }
    if (t < H) {
        S.b1[t] = __ldcg(P + OB1 + t);
        S.b2[t] = __ldcg(P + OB2 + t);
        S.w3[t] = __ldcg(P + OW3 + t);
    }
    const float b3 = __ldcg(P + OB3);
    const float inv_n = 1.f / (float)n;
    // row-wise products: sample s, units u0..u0+7; dW2: rows r0..r0+3, columns c0..c0+3
    const int s = t >> 3, u0 = (t & 7) * 8;
    const int r0 = (t >> 4) * 4, c0 = (t & 15) * 4;
    float gw2[4][4] = {}, gw1[3] = {}, gv[3] = {}, gb3 = 0.f; // gv: b1, b2, W3
    double lsum = 0.0; // an epoch adds up some 16k of these
    auto axpy8 = [](float (&acc)[8], float a, const float *w) {
        const float4 p = *reinterpret_cast<const float4 *>(w);
        const float4 q = *reinterpret_cast<const float4 *>(w + 4);
        acc[0] = fmaf(a, p.x, acc[0]);
        acc[1] = fmaf(a, p.y, acc[1]);
        acc[2] = fmaf(a, p.z, acc[2]);
        acc[3] = fmaf(a, p.w, acc[3]);
        acc[4] = fmaf(a, q.x, acc[4]);
        acc[5] = fmaf(a, q.y, acc[5]);
        acc[6] = fmaf(a, q.z, acc[6]);
        acc[7] = fmaf(a, q.w, acc[7]);
    };
    for (int base = blockIdx.x * GS; base < n; base += gridDim.x * GS) {
        __syncthreads(); // the parameters are staged; the tile before is consumed
        for (int i = t; i < GS * F; i += GT) {
            const int q = base + i / F;
            S.x[i / F][i % F] =
                q < n ? X[(size_t)(perm ? perm[q] : (uint32_t)q) * F + i % F] : 0.f;
        }
        __syncthreads();
        float acc[8], h[8], d[8];
        // ---- layer 1
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = S.b1[u0 + j];
#pragma unroll
        for (int k = 0; k < F; ++k) axpy8(acc, S.x[s][k], &S.w1t[k][u0]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            gelu2(acc[j], h[j], d[j]);
            S.h1[s][u0 + j] = h[j];
            S.d1[s][u0 + j] = d[j];
        }
        __syncwarp(); // the 8 threads of a sample are in one warp
        // ---- layer 2 and the output
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = S.b2[u0 + j];
#pragma unroll 8
        for (int v = 0; v < H; ++v) axpy8(acc, S.h1[s][v], &S.w2t[v][u0]);
        float y = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            gelu2(acc[j], h[j], d[j]);
            y = fmaf(S.w3[u0 + j], h[j], y);
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
        y += b3;
        const bool in = base + s < n;
        const float e = in ? Yt[perm ? perm[base + s] : (uint32_t)(base + s)] - y : 0.f;
        const float dy = in ? (e > 0.f ? -tau : 1.f - tau) * inv_n : 0.f;
        if ((t & 7) == 0) {
            lsum += (double)(e > 0.f ? tau * e : (tau - 1.f) * e);
            gb3 += dy;
            S.dy[s] = dy;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            S.h2[s][u0 + j] = h[j];
            S.dz2[s][u0 + j] = dy * S.w3[u0 + j] * d[j];
        }
        __syncwarp();
        // ---- back through layer 2
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll 8
        for (int u = 0; u < H; ++u) axpy8(acc, S.dz2[s][u], &S.w2[u][u0]);
#pragma unroll
        for (int j = 0; j < 8; ++j) S.dz1[s][u0 + j] = acc[j] * S.d1[s][u0 + j];
        __syncthreads();
        // ---- the tile's share of the gradient
#pragma unroll 4
        for (int q = 0; q < GS; ++q) {
            const float4 a = *reinterpret_cast<const float4 *>(&S.dz2[q][r0]);
            const float4 b = *reinterpret_cast<const float4 *>(&S.h1[q][c0]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) gw2[i][j] = fmaf(av[i], bv[j], gw2[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int o = t + GT * i, u = o / F, k = o % F;
            for (int q = 0; q < GS; ++q) gw1[i] = fmaf(S.dz1[q][u], S.x[q][k], gw1[i]);
        }
        if (t < H)
            for (int q = 0; q < GS; ++q) {
                gv[0] += S.dz1[q][t];
                gv[1] += S.dz2[q][t];
                gv[2] = fmaf(S.dy[q], S.h2[q][t], gv[2]);
            }
    }
    static_assert(GT * 3 == H * F, "three entries of W1 per thread");
#pragma unroll
    for (int i = 0; i < 3; ++i) atomicAdd(G + OW1 + t + GT * i, (double)gw1[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) atomicAdd(G + OW2 + (r0 + i) * H + c0 + j, (double)gw2[i][j]);
    if (t < H) {
        atomicAdd(G + OB1 + t, (double)gv[0]);
        atomicAdd(G + OB2 + t, (double)gv[1]);
        atomicAdd(G + OW3 + t, (double)gv[2]);
    }
    // the samples' losses and output deltas, one per 8 threads
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, o);
        lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    }
    if ((t & 31) == 0) {
        atomicAdd(G + OB3, (double)gb3);
        atomicAdd(loss, lsum / (double)n);
    }
}

// Adam step with bias correction on 64-bit parameters and moments (A: parameters,
// first, second moments), P their FP32 image; clears the gradient for the next
// batch.  In FP32 the parameters rounded at each step and the batch gradient's atomics
// at each addition: distance of the trained parameters from 64 bits (two epochs of
// 65536 and 20011 samples, 12 seeds) 1.6e-7 to 2.4e-6 and two runs 1e-4, now 4e-8 to
// 2.4e-6, smaller on each seed.  A step takes 33 us at 4096 samples (gradient 28, this
// kernel 3.4), beside some 1.2 ms a call for the copies and the first shuffle.
__global__ void k_mlp_adam(float *P, double *G, double *A, int np, double lr, double b1,
                           double b2, double eps, double bc1, double bc2, bool first)
{
    paddi::chain_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= np) return;
    const double g = G[i];
    const double m = b1 * A[np + i] + (1.0 - b1) * g;
    const double v = b2 * A[2 * np + i] + (1.0 - b2) * g * g;
    const double p = (first ? (double)P[i] : A[i]) - lr * (m / bc1) / (sqrt(v / bc2) + eps);
    A[i] = p;
    A[np + i] = m;
    A[2 * np + i] = v;
    P[i] = (float)p;
    G[i] = 0.0;
}

__global__ void k_to_bf16(const float *P, __nv_bfloat16 *Q, int np)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < np) Q[i] = __float2bfloat16_rn(P[i]);
}

} // namespace

cudaError_t paddi_launch_mlp_forward(const float *X, int n, const void *P, bool bf16, float *Y,
                                     cudaStream_t st)
{
    const int warps = n < 4096 ? n : 4096;
    const int threads = 128;
    const int grid = (warps * 32 + threads - 1) / threads;
    if (bf16)
        k_mlp_forward<__nv_bfloat16><<<grid > 0 ? grid : 1, threads, 0, st>>>(
            X, n, static_cast<const __nv_bfloat16 *>(P), Y);
    else
        k_mlp_forward<float><<<grid > 0 ? grid : 1, threads, 0, st>>>(
            X, n, static_cast<const float *>(P), Y);
    return cudaGetLastError();
}

cudaError_t paddi_launch_mlp_grad(const float *X, const float *Y, const uint32_t *perm, int n,
                                  float tau, const float *P, double *G, double *loss, int num_sms,
                                  cudaStream_t st)
{
    cudaError_t e = paddi_raise_smem_limit((const void *)k_mlp_grad, sizeof(GradSmem));
    if (e != cudaSuccess) return e;
    const int tiles = (n + GS - 1) / GS;
    return paddi_launch(true, k_mlp_grad, tiles < num_sms ? tiles : num_sms, GT, sizeof(GradSmem),
                        st, X, Y, perm, n, tau, P, G, loss);
}

cudaError_t paddi_launch_mlp_adam(float *P, double *G, double *A, float lr, int step,
                                  cudaStream_t st)
{
    const double b1 = 0.9, b2 = 0.999;
    return paddi_launch(true, k_mlp_adam, (MLP_NPARAM + 127) / 128, 128, 0, st, P, G, A, MLP_NPARAM,
                        (double)lr, b1, b2, 1e-8, 1.0 - std::pow(b1, step),
                        1.0 - std::pow(b2, step), step == 1);
}

cudaError_t paddi_launch_mlp_to_bf16(const float *P, void *Q, cudaStream_t st)
{
    k_to_bf16<<<(MLP_NPARAM + 255) / 256, 256, 0, st>>>(P, static_cast<__nv_bfloat16 *>(Q),
                                                        MLP_NPARAM);
    return cudaGetLastError();
}
