// Training and batch inference of the selector's cost model: a perceptron
// 16 -> 64 (ReLU) -> 64 (ReLU) -> 3 predicting log-microseconds of the LOP3,
// M4R and tensor-core variants of a product term from its features.
//
// Loss over the logged samples (x_n, y_n, m_n), m_nj = 1 where variant j was
// timed:  L = sum_n sum_j m_nj (f(x_n)_j - y_nj)^2 / (2 sum m).
//
// k_mlp_fb: forward and backward, 64 samples at a time per block of 256 threads,
// blocks resident (2 per SM) and walking the samples.  Every layer is a small
// matrix product out of shared memory with a 4 x 4 register tile per thread (8
// FMAs per 4-word load; one thread per sample read two words per FMA and left
// 128 threads per SM).  Activations are kept transposed ([feature][sample], 68
// samples apart: 16-byte loads along the samples are free of bank conflicts).
// Weight gradients stay in registers over all samples of the block and go to
// memory with one atomicAdd per weight and block.  Bound: shared-memory loads
// and FMA issue, 1.26 GFLOP for 39,685 samples; 204 -> 65 us (ncu).
// k_adam: Adam step with decoupled weight decay, zeroing the gradient.
// k_mlp_predict: one warp per sample (the same warp routine the selector runs
// inside the closure).
#include <algorithm>

#include "launch.h"
#include "select_device.cuh"

namespace cfpq {

namespace {

constexpr int F = kSelFeatures, H = kSelHidden, O = kSelOutputs;
constexpr int kSamples = 64;        // samples per block step
constexpr int kFbThreads = 256;     // 16 x 16 threads, 4 x 4 outputs each
constexpr int kRow = kSamples + 4;  // transposed activation rows
static_assert(F == 16 && H == 64 && O == 3, "the thread tiles are laid out for 16-64-64-3");

struct MlpSmem {
    alignas(16) float w1[F * H];
    alignas(16) float w2[H * H];
    alignas(16) float w2t[H * H];
    float w3[H * O], b1[H], b2[H], b3[O];
    // [feature][sample], read 16 bytes at a time; h2 later holds d1
    alignas(16) float x[F * kRow];
    alignas(16) float h1[H * kRow];
    alignas(16) float h2[H * kRow];
    alignas(16) float d2[H * kRow];
    alignas(16) float dout[O * kRow];
    float loss[kFbThreads / 32];
};

__device__ __forceinline__ float4 lds4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// acc[i][j] += sum over k of a[k][4 ty + i] * b[k][4 tx + j] (rows kA, kB words apart), k ascending
template <int kK, int kA, int kB>
__device__ __forceinline__ void tile_product(const float *a, const float *b, uint32_t ty, uint32_t tx,
                                             float (&acc)[4][4]) {
#pragma unroll 8
    for (int k = 0; k < kK; ++k) {
        const float4 av = lds4(a + k * kA + 4 * ty), bv = lds4(b + k * kB + 4 * tx);
        const float ar[4] = {av.x, av.y, av.z, av.w}, br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(br[j], ar[i], acc[i][j]);
    }
}

// out[4 tx + j][4 ty + i] = acc[i][j] (transposed store)
__device__ __forceinline__ void store_tile(float *out, uint32_t ty, uint32_t tx, const float (&acc)[4][4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(out + (4 * tx + j) * kRow + 4 * ty) =
            make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
}

__global__ void __launch_bounds__(kFbThreads, 2) k_mlp_fb(const float *__restrict__ W, const float *__restrict__ X,
                                                          const float *__restrict__ Y, const float *__restrict__ M,
                                                          uint32_t N, float inv_msum, float *grad, float *loss) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MlpSmem &S = *reinterpret_cast<MlpSmem *>(smem_raw);
    const uint32_t t = threadIdx.x, tx = t & 15, ty = t >> 4;
    const float *W1 = W, *b1 = W1 + F * H, *W2 = b1 + H, *b2 = W2 + H * H, *W3 = b2 + H, *b3 = W3 + H * O;
    for (int i = t; i < F * H; i += kFbThreads) S.w1[i] = W1[i];
    for (int i = t; i < H * H; i += kFbThreads) {
        const float w = W2[i];
        S.w2[i] = w;
        S.w2t[(i % H) * H + i / H] = w;
    }
    if (t < H * O) S.w3[t] = W3[t];
    if (t < H) {
        S.b1[t] = b1[t];
        S.b2[t] = b2[t];
    }
    if (t < O) S.b3[t] = b3[t];
    // gradients of this thread's weights: g2[i][j] of W2[ty + 16 i][tx + 16 j],
    // g1[j] of W1[ty][tx + 16 j], g3 of W3 (t < 192), gb of b1 / b2 / b3
    float g2[4][4] = {}, g1[4] = {}, g3 = 0.f, gb1 = 0.f, gb2 = 0.f, gb3 = 0.f, l = 0.f;
    const uint32_t steps = (N + kSamples - 1) / kSamples;
    for (uint32_t step = blockIdx.x; step < steps; step += gridDim.x) {
        const uint32_t s0 = step * kSamples;
        __syncthreads();  // the last step's readers of x, h1, h2, d2 are done (first step: the weights are there)
        for (int i = t; i < F * kSamples; i += kFbThreads) {
            const uint32_t s = i / F, f = i % F;
            S.x[f * kRow + s] = s0 + s < N ? X[(size_t)s0 * F + i] : 0.f;
        }
        __syncthreads();
        {
            float a[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) a[i][j] = S.b1[4 * tx + j];
            tile_product<F, kRow, H>(S.x, S.w1, ty, tx, a);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) a[i][j] = fmaxf(a[i][j], 0.f);
            store_tile(S.h1, ty, tx, a);
        }
        __syncthreads();
        {
            float a[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) a[i][j] = S.b2[4 * tx + j];
            tile_product<H, kRow, H>(S.h1, S.w2, ty, tx, a);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) a[i][j] = fmaxf(a[i][j], 0.f);
            store_tile(S.h2, ty, tx, a);
        }
        __syncthreads();
        if (t < kSamples * O) {
            const uint32_t j = t / kSamples, s = t % kSamples;
            const bool valid = s0 + s < N;
            float a = S.b3[j];
#pragma unroll 16
            for (int u = 0; u < H; ++u) a = fmaf(S.w3[u * O + j], S.h2[u * kRow + s], a);
            const float m = valid ? M[(size_t)(s0 + s) * O + j] : 0.f;
            const float e = valid ? a - Y[(size_t)(s0 + s) * O + j] : 0.f;
            S.dout[j * kRow + s] = m * e * inv_msum;
            l += 0.5f * m * e * e * inv_msum;
        }
        __syncthreads();
        {  // d2 = (h2 > 0) * (W3 dout)
            float a[4][4] = {};
#pragma unroll
            for (int o = 0; o < O; ++o) {
                const float4 dv = lds4(S.dout + o * kRow + 4 * ty);
                const float dr[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float w = S.w3[(4 * tx + j) * O + o];
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[i][j] = fmaf(w, dr[i], a[i][j]);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 h = lds4(S.h2 + (4 * tx + j) * kRow + 4 * ty);
                const float hr[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i][j] = hr[i] > 0.f ? a[i][j] : 0.f;
            }
            store_tile(S.d2, ty, tx, a);
        }
        if (t < H * O) {
            const uint32_t u = t / O, j = t % O;
#pragma unroll 4
            for (int s = 0; s < kSamples; s += 4) {
                const float4 h = lds4(S.h2 + u * kRow + s), d = lds4(S.dout + j * kRow + s);
                g3 = fmaf(h.x, d.x, g3);
                g3 = fmaf(h.y, d.y, g3);
                g3 = fmaf(h.z, d.z, g3);
                g3 = fmaf(h.w, d.w, g3);
            }
        } else if (t < H * O + O) {
            for (int s = 0; s < kSamples; ++s) gb3 += S.dout[(t - H * O) * kRow + s];
        }
        __syncthreads();  // d2 is complete; h2 has been read
        {  // d1 = (h1 > 0) * (W2 d2), into h2
            float a[4][4] = {};
            tile_product<H, kRow, H>(S.d2, S.w2t, ty, tx, a);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 h = lds4(S.h1 + (4 * tx + j) * kRow + 4 * ty);
                const float hr[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i][j] = hr[i] > 0.f ? a[i][j] : 0.f;
            }
            store_tile(S.h2, ty, tx, a);
        }
#pragma unroll 4
        for (int s = 0; s < kSamples; s += 4) {  // W2: sum over the samples of h1[k] d2[u]
            float4 hv[4], dv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                hv[i] = lds4(S.h1 + (ty + 16 * i) * kRow + s);
                dv[i] = lds4(S.d2 + (tx + 16 * i) * kRow + s);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    g2[i][j] = fmaf(hv[i].x, dv[j].x, g2[i][j]);
                    g2[i][j] = fmaf(hv[i].y, dv[j].y, g2[i][j]);
                    g2[i][j] = fmaf(hv[i].z, dv[j].z, g2[i][j]);
                    g2[i][j] = fmaf(hv[i].w, dv[j].w, g2[i][j]);
                }
        }
        __syncthreads();  // d1 is complete
#pragma unroll 4
        for (int s = 0; s < kSamples; s += 4) {  // W1: sum over the samples of x[f] d1[u]
            const float4 xv = lds4(S.x + ty * kRow + s);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float4 dv = lds4(S.h2 + (tx + 16 * j) * kRow + s);
                g1[j] = fmaf(xv.x, dv.x, g1[j]);
                g1[j] = fmaf(xv.y, dv.y, g1[j]);
                g1[j] = fmaf(xv.z, dv.z, g1[j]);
                g1[j] = fmaf(xv.w, dv.w, g1[j]);
            }
        }
        if (t < 2 * H) {  // biases: sums of d1 (t < H) and d2
            const float *row = t < H ? S.h2 + t * kRow : S.d2 + (t - H) * kRow;
            float &g = t < H ? gb1 : gb2;
            for (int s = 0; s < kSamples; s += 4) {
                const float4 v = lds4(row + s);
                g += v.x;
                g += v.y;
                g += v.z;
                g += v.w;
            }
        }
    }
    for (int d = 16; d > 0; d >>= 1) l += __shfl_xor_sync(0xffffffffu, l, d);
    if ((t & 31) == 0) S.loss[t >> 5] = l;
    __syncthreads();
    if (t == 0) {
        float bl = 0.f;
        for (int w = 0; w < kFbThreads / 32; ++w) bl += S.loss[w];
        if (bl != 0.f) atomicAdd(loss, bl);
    }
    auto add = [&](int w, float g) {
        if (g != 0.f) atomicAdd(grad + w, g);
    };
    constexpr int oB1 = F * H, oW2 = oB1 + H, oB2 = oW2 + H * H, oW3 = oB2 + H, oB3 = oW3 + H * O;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        add(ty * H + tx + 16 * j, g1[j]);
#pragma unroll
        for (int i = 0; i < 4; ++i) add(oW2 + (ty + 16 * i) * H + tx + 16 * j, g2[i][j]);
    }
    if (t < H) add(oB1 + t, gb1);
    else if (t < 2 * H) add(oB2 + t - H, gb2);
    if (t < H * O) add(oW3 + t, g3);
    else if (t < H * O + O) add(oB3 + t - H * O, gb3);
}

__global__ void k_adam(float *W, float *grad, float *m, float *v, uint32_t n, float lr, float beta1, float beta2,
                       float eps, float wd, float c1, float c2) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = grad[i];
    const float mi = beta1 * m[i] + (1.f - beta1) * g;
    const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
    m[i] = mi;
    v[i] = vi;
    W[i] -= lr * ((mi / c1) / (sqrtf(vi / c2) + eps) + wd * W[i]);
    grad[i] = 0.f;
}

__global__ void k_mlp_predict(const float *__restrict__ W, const float *__restrict__ X, uint32_t N, float *out) {
    const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (s >= N) return;
    float x[F], p[O];
#pragma unroll
    for (int i = 0; i < F; ++i) x[i] = X[(size_t)s * F + i];
    sel::selector_mlp_warp(W, x, p);
    if ((threadIdx.x & 31) == 0)
        for (int j = 0; j < O; ++j) out[(size_t)s * O + j] = p[j];
}

}  // namespace

cudaError_t mlp_loss_grad(const float *d_w, const float *d_x, const float *d_y, const float *d_m, uint32_t n,
                          float inv_msum, float *d_grad, float *d_loss, cudaStream_t s) {
    cudaError_t e = cudaFuncSetAttribute(k_mlp_fb, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MlpSmem));
    if (e != cudaSuccess) return e;
    if (n == 0) return cudaSuccess;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    const uint32_t steps = (n + kSamples - 1) / kSamples;
    k_mlp_fb<<<std::min(steps, 2u * (uint32_t)sms), kFbThreads, sizeof(MlpSmem), s>>>(d_w, d_x, d_y, d_m, n, inv_msum,
                                                                                     d_grad, d_loss);
    return cudaGetLastError();
}

cudaError_t mlp_adam_step(float *d_w, float *d_grad, float *d_m, float *d_v, float lr, float wd, uint32_t step,
                          cudaStream_t s) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<(kSelWeights + 255) / 256, 256, 0, s>>>(d_w, d_grad, d_m, d_v, kSelWeights, lr, b1, b2, 1e-8f, wd, c1,
                                                     c2);
    return cudaGetLastError();
}

cudaError_t mlp_predict(const float *d_w, const float *d_x, uint32_t n, float *d_out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    k_mlp_predict<<<(unsigned)(((size_t)n * 32 + 127) / 128), 128, 0, s>>>(d_w, d_x, n, d_out);
    return cudaGetLastError();
}

}  // namespace cfpq
