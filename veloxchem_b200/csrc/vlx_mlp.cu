// Kernels of the learned initial-guess network: a multilayer perceptron over
// atom-pair descriptors whose outputs are density-matrix blocks.  Training
// runs in FP32 (forward with the pre-activations kept, backward, masked mean
// squared error, Adam); inference reads BF16 weights and BF16-rounded inputs
// on the tensor cores (mma.sync, FP32 accumulation).  The layer shapes are
// small (inputs of about a hundred features, width 128, outputs up to 196),
// so each layer is one tiled GEMM launch with bias and SiLU fused into its
// epilogue; the FP32 kernel serves the forward pass of training and the three
// products of the backward pass through operand strides.
// No counterpart in the reference (its initial guesses are SAD / core / read).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "../../include/vlx_b200.h"

namespace {

constexpr int kTile = 64;  // output tile (rows and columns)
constexpr int kTileK = 16; // reduction slice staged in shared memory

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }

// C(m, n) = sum_k A(m, k) B(k, n) (+ bias[n]) in FP32; A(m, k) = A[m lda + k]
// (AK) or A[k lda + m], B(k, n) = B[n ldb + k] (BK) or B[k ldb + n], so the
// staging loads run along the contiguous index of either operand.  Z (optional)
// gets the value, Y SiLU of it (act) or the value itself.  SUM (optional):
// sum_k A(m, k).
//
// 64 x 64 outputs per block of 256 threads, 4 x 4 per thread, slices of 16 in k
// with the next slice's loads in flight during the products.  The weight
// gradients reduce over the samples into only 4 to 8 output tiles, so there
// the blocks of a cluster (grid z) share a tile's k range and add their partial
// tiles through distributed shared memory in rank order (the same sums on every
// run).  Latency bound: a training step at 4096 samples (134 - 128 - 128 - 196,
// 8 products) takes 0.38 ms, of which host calls are most; with one block per
// tile for the gradients and the bias sums by one block per 32 columns it took
// 1.67 ms.
constexpr int kSplitMax = 8;      // portable cluster size
constexpr int kSplitRows = 128;   // least samples of a split

template <bool AK, bool BK>
__global__ void __launch_bounds__(256) gemm_kernel(const float* __restrict__ A, const int lda,
                                                   const float* __restrict__ B, const int ldb,
                                                   const float* __restrict__ bias,
                                                   float* __restrict__ Z, float* __restrict__ Y,
                                                   float* __restrict__ SUM, const int M, const int N, const int K,
                                                   const int act)
{
    constexpr int kLoads = kTile * kTileK / 256;
    __shared__ __align__(16) float As[kTileK][kTile + 4];
    __shared__ __align__(16) float Bs[kTileK][kTile + 4];
    __shared__ float part[kTile][kTile];
    __shared__ float psum[kTile];
    const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    const int split = gridDim.z, rank = blockIdx.z;
    const int per = ((K + split - 1) / split + kTileK - 1) / kTileK * kTileK;
    const int kend = min(K, (rank + 1) * per);
    const bool sums = SUM != nullptr && blockIdx.x == 0;
    float acc[4][4], ra[kLoads], rb[kLoads], s = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
    const auto fetch = [&](const int k0) {
#pragma unroll
        for (int x = 0; x < kLoads; x++) {
            const int e = t + 256 * x;
            const int mr = AK ? e / kTileK : e % kTile, mk = AK ? e % kTileK : e / kTile;
            const int nr = BK ? e / kTileK : e % kTile, nk = BK ? e % kTileK : e / kTile;
            const int m = m0 + mr, n = n0 + nr, ka = k0 + mk, kb = k0 + nk;
            const size_t ia = AK ? (size_t)m * lda + ka : (size_t)ka * lda + m;
            const size_t ib = BK ? (size_t)n * ldb + kb : (size_t)kb * ldb + n;
            ra[x] = (m < M && ka < kend) ? __ldg(A + ia) : 0.0f;
            rb[x] = (n < N && kb < kend) ? __ldg(B + ib) : 0.0f;
        }
    };
    fetch(rank * per);
    for (int k0 = rank * per; k0 < kend; k0 += kTileK) {
#pragma unroll
        for (int x = 0; x < kLoads; x++) {
            const int e = t + 256 * x;
            As[AK ? e % kTileK : e / kTile][AK ? e / kTileK : e % kTile] = ra[x];
            Bs[BK ? e % kTileK : e / kTile][BK ? e / kTileK : e % kTile] = rb[x];
        }
        __syncthreads();
        fetch(k0 + kTileK);
        if (sums && t < kTile) {
#pragma unroll
            for (int kk = 0; kk < kTileK; kk++) s += As[kk][t];
        }
#pragma unroll
        for (int kk = 0; kk < kTileK; kk++) {
            const float4 a = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4*>(&Bs[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    const auto write = [&](const int m, const int n, const float v) {
        if (m >= M || n >= N) return;
        const float z = v + (bias ? __ldg(bias + n) : 0.0f);
        if (Z) Z[(size_t)m * N + n] = z;
        Y[(size_t)m * N + n] = act ? silu(z) : z;
    };
    if (split == 1) {
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) write(m0 + ty * 4 + i, n0 + tx * 4 + j, acc[i][j]);
        if (sums && t < kTile && m0 + t < M) SUM[m0 + t] = s;
        return;
    }
    cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) part[ty * 4 + i][tx * 4 + j] = acc[i][j];
    if (t < kTile) psum[t] = s;
    cluster.sync();
    for (int e = rank * 256 + t; e < kTile * kTile; e += split * 256) {
        float v = 0.0f;
        for (int r = 0; r < split; r++) v += cluster.map_shared_rank(&part[0][0], r)[e];
        write(m0 + e / kTile, n0 + e % kTile, v);
    }
    if (sums && rank == 0 && t < kTile && m0 + t < M) {
        float v = 0.0f;
        for (int r = 0; r < split; r++) v += cluster.map_shared_rank(&psum[0], r)[t];
        SUM[m0 + t] = v;
    }
    cluster.sync();  // the partial tiles stay until every block has read them
}

// Inference layer on the tensor cores: Y[M, N] = act(X[M, K] W[N, K]^T + b)
// with X rounded to BF16 as it is staged, W in BF16, FP32 accumulation
// (mma.sync m16n8k16 BF16, operand fragments read straight from shared
// memory).  Block: 4 warps on a 64 x 64 output tile, each warp 32 x 32
// (2 x 4 MMA tiles); K in steps of 16, zero-padded at the edges.
constexpr int kMmaTile = 64;
constexpr int kMmaK = 16;
constexpr int kMmaPad = kMmaK + 8;  // row stride 48 B: the fragment loads of a warp hit 32 distinct banks

__device__ __forceinline__ void mma_bf16_16816(float* c, const uint32_t* a, const uint32_t* b)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__global__ void __launch_bounds__(128) gemm_bf16_mma_kernel(const float* __restrict__ X,
                                                            const __nv_bfloat16* __restrict__ W,
                                                            const float* __restrict__ bias, float* __restrict__ Y,
                                                            const int M, const int N, const int K, const int act)
{
    __shared__ __align__(16) __nv_bfloat16 As[kMmaTile][kMmaPad];
    __shared__ __align__(16) __nv_bfloat16 Bs[kMmaTile][kMmaPad];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, tq = lane & 3;
    const int m0 = blockIdx.y * kMmaTile, n0 = blockIdx.x * kMmaTile;
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) acc[i][j][e] = 0.0f;
    const __nv_bfloat16 zero = __float2bfloat16_rn(0.0f);
    for (int k0 = 0; k0 < K; k0 += kMmaK) {
        for (int t = threadIdx.x; t < kMmaTile * kMmaK; t += blockDim.x) {
            const int r = t / kMmaK, kk = t % kMmaK, k = k0 + kk;
            const int m = m0 + r, n = n0 + r;
            As[r][kk] = (m < M && k < K) ? __float2bfloat16_rn(__ldg(X + (size_t)m * K + k)) : zero;
            Bs[r][kk] = (n < N && k < K) ? W[(size_t)n * K + k] : zero;
        }
        __syncthreads();
        uint32_t a[2][4], b[4][2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = wm + i * 16 + g;
            a[i][0] = *reinterpret_cast<const uint32_t*>(&As[r][2 * tq]);
            a[i][1] = *reinterpret_cast<const uint32_t*>(&As[r + 8][2 * tq]);
            a[i][2] = *reinterpret_cast<const uint32_t*>(&As[r][2 * tq + 8]);
            a[i][3] = *reinterpret_cast<const uint32_t*>(&As[r + 8][2 * tq + 8]);
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = wn + j * 8 + g;
            b[j][0] = *reinterpret_cast<const uint32_t*>(&Bs[c][2 * tq]);
            b[j][1] = *reinterpret_cast<const uint32_t*>(&Bs[c][2 * tq + 8]);
        }
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) mma_bf16_16816(acc[i][j], a[i], b[j]);
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int m = m0 + wm + i * 16 + g + ((e & 2) ? 8 : 0);
                const int n = n0 + wn + j * 8 + 2 * tq + (e & 1);
                if (m < M && n < N) {
                    const float z = acc[i][j][e] + (bias ? __ldg(bias + n) : 0.0f);
                    Y[(size_t)m * N + n] = act ? silu(z) : z;
                }
            }
}

// dZ = dY SiLU'(Z), SiLU'(z) = s (1 + z (1 - s)), s = 1 / (1 + e^-z); dZ may be dY
// or Z.  A pass of its own: as a factor of the products' staging loads it was
// evaluated again for every 64 columns of the output, in their critical path (dW
// and dX of 64 / 4096 / 30000 samples with 128 inputs and outputs 31 / 84 / 521 us
// against 24 / 55 / 285 with this pass), and the products read what they write when
// dX is dY's buffer.
__global__ void silu_backward_kernel(const float* dY, const float* Z, float* dZ, const size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float z = Z[i], s = 1.0f / (1.0f + expf(-z));
        dZ[i] = dY[i] * s * (1.0f + z * (1.0f - s));
    }
}

// masked squared error: dY = 2 w (Y - T) / count, loss += sum w (Y - T)^2
__global__ void mse_kernel(const float* __restrict__ Y, const float* __restrict__ T, const float* __restrict__ W,
                           float* __restrict__ dY, double* __restrict__ loss, const size_t n, const float inv_count)
{
    __shared__ double part[256];
    double acc = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float w = W[i];
        const float r = Y[i] - T[i];
        dY[i] = 2.0f * w * r * inv_count;
        acc += (double)(w * r * r);
    }
    part[threadIdx.x] = acc;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) part[threadIdx.x] += part[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) atomicAdd(loss, part[0]);
}

// Adam with bias-corrected moments (Kingma & Ba 2015); c1 = 1 - beta1^t, c2 = 1 - beta2^t
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, const size_t n, const float lr, const float b1, const float b2,
                            const float eps, const float c1, const float c2)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

__global__ void to_bf16_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, const size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        y[i] = __float2bfloat16_rn(x[i]);
}

int grid_1d(size_t n) { return (int)std::min<size_t>((n + 255) / 256, 148 * 8); }

}  // namespace

extern "C" int vlx_b200_set_error_internal(int code, const char* msg);

#define MLP_CHECK()                                                                       \
    do {                                                                                  \
        cudaError_t e_ = cudaGetLastError();                                              \
        if (e_ != cudaSuccess) return vlx_b200_set_error_internal(VLX_B200_ERR_CUDA, cudaGetErrorString(e_)); \
    } while (0)

extern "C" {

int vlx_b200_mlp_linear(const float* X, const float* W, const float* b, float* Z, float* Y, int M, int K, int N,
                        int silu_act, void* stream)
{
    if (!X || !W || !Y || M < 0 || K < 1 || N < 1)
        return vlx_b200_set_error_internal(VLX_B200_ERR_ARGUMENT, "mlp_linear: bad arguments");
    if (M == 0) return VLX_B200_OK;
    const dim3 grid((N + kTile - 1) / kTile, (M + kTile - 1) / kTile);
    gemm_kernel<true, true><<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(X, K, W, K, b, Z, Y, nullptr, M, N, K,
                                                                                 silu_act);
    MLP_CHECK();
    return VLX_B200_OK;
}

int vlx_b200_mlp_linear_bf16(const float* X, const void* W_bf16, const float* b, float* Y, int M, int K, int N,
                             int silu_act, void* stream)
{
    if (!X || !W_bf16 || !Y || M < 0 || K < 1 || N < 1)
        return vlx_b200_set_error_internal(VLX_B200_ERR_ARGUMENT, "mlp_linear_bf16: bad arguments");
    if (M == 0) return VLX_B200_OK;
    const dim3 grid((N + kMmaTile - 1) / kMmaTile, (M + kMmaTile - 1) / kMmaTile);
    gemm_bf16_mma_kernel<<<grid, 128, 0, static_cast<cudaStream_t>(stream)>>>(
        X, static_cast<const __nv_bfloat16*>(W_bf16), b, Y, M, N, K, silu_act);
    MLP_CHECK();
    return VLX_B200_OK;
}

int vlx_b200_mlp_linear_backward(const float* X, const float* W, const float* Z, const float* dY, float* dZ,
                                 float* dX, float* dW, float* db, int M, int K, int N, int silu_act, void* stream)
{
    if (!X || !W || !dY || !dW || !db || (silu_act && (!Z || !dZ)) || M < 1 || K < 1 || N < 1)
        return vlx_b200_set_error_internal(VLX_B200_ERR_ARGUMENT, "mlp_linear_backward: bad arguments");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float* g = dY;
    if (silu_act) {
        const size_t n = (size_t)M * N;
        silu_backward_kernel<<<grid_1d(n), 256, 0, st>>>(dY, Z, dZ, n);
        g = dZ;
    }
    // dW[N, K] = g^T X and db = column sums of g: rows n, reduction over the
    // samples, split over a cluster
    int split = 1;
    while (split < kSplitMax && M >= 2 * split * kSplitRows) split *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((K + kTile - 1) / kTile, (N + kTile - 1) / kTile, split);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {1, 1, (unsigned)split};
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_kernel<false, false>, g, N, X, K,
                                             static_cast<const float*>(nullptr), static_cast<float*>(nullptr), dW, db,
                                             N, K, M, 0);
    if (e != cudaSuccess) return vlx_b200_set_error_internal(VLX_B200_ERR_CUDA, cudaGetErrorString(e));
    // dX[M, K] = g W
    if (dX)
        gemm_kernel<true, false><<<dim3((K + kTile - 1) / kTile, (M + kTile - 1) / kTile), 256, 0, st>>>(
            g, N, W, K, nullptr, nullptr, dX, nullptr, M, K, N, 0);
    MLP_CHECK();
    return VLX_B200_OK;
}

int vlx_b200_mlp_mse(const float* Y, const float* T, const float* mask, float* dY, double* d_loss_sum, long long n,
                     double count, void* stream)
{
    if (!Y || !T || !mask || !dY || !d_loss_sum || n < 0 || !(count > 0.0))
        return vlx_b200_set_error_internal(VLX_B200_ERR_ARGUMENT, "mlp_mse: bad arguments");
    if (n == 0) return VLX_B200_OK;
    mse_kernel<<<grid_1d(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(Y, T, mask, dY, d_loss_sum, (size_t)n,
                                                                         (float)(1.0 / count));
    MLP_CHECK();
    return VLX_B200_OK;
}

int vlx_b200_adam_step(float* params, const float* grads, float* m, float* v, long long n, float lr, float beta1,
                       float beta2, float eps, int step, void* stream)
{
    if (!params || !grads || !m || !v || n < 0 || step < 1)
        return vlx_b200_set_error_internal(VLX_B200_ERR_ARGUMENT, "adam_step: bad arguments");
    if (n == 0) return VLX_B200_OK;
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<grid_1d(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(params, grads, m, v, (size_t)n, lr, beta1,
                                                                          beta2, eps, c1, c2);
    MLP_CHECK();
    return VLX_B200_OK;
}

int vlx_b200_to_bf16(const float* x, void* y, long long n, void* stream)
{
    if (!x || !y || n < 0) return vlx_b200_set_error_internal(VLX_B200_ERR_ARGUMENT, "to_bf16: bad arguments");
    if (n == 0) return VLX_B200_OK;
    to_bf16_kernel<<<grid_1d(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, static_cast<__nv_bfloat16*>(y),
                                                                             (size_t)n);
    MLP_CHECK();
    return VLX_B200_OK;
}

}  // extern "C"
