// mgbvh_mlp.cu — training and batch inference of the learned split proposer.
//
// The network (layout in mgbvh_mlp.cuh) is trained on node samples whose
// label is the exact full-sweep SAH optimum (axis and position bucket) and
// whether it beats the plain binned split. Parameters are BF16 in the
// forward and backward passes, with FP32 accumulation; the optimizer keeps
// FP32 master weights (Adam) and rewrites the BF16 copy after each step.
//
// One CTA handles 32 samples: weights (as FP32) and activations in shared
// memory, forward through both hidden layers, softmax cross-entropy over the
// 48 position logits plus binary cross-entropy of the refine logit, then the
// backward pass; each CTA adds its parameter gradients to the global FP32
// gradient with one atomic per parameter.
//
// The products are small (32 samples, 64 units) and stay in FP32 on the CUDA
// cores: what bounds a CTA is shared-memory wavefronts and the chain of its
// eight products, so every thread holds a register tile (2 samples x 4 units,
// or 4 x 4 weights) and reads float4s along the rows. Rows are padded to an
// odd number of 16-byte words, which keeps eight neighbouring rows on distinct
// banks. Every sum is one fused multiply-add per term, in the terms' order.
// A CTA of 32 samples gives 128 CTAs at a batch of 4,096, one per SM; half the
// samples would double the gradient's atomics and the weights' loads.
// A step of 4,096 samples (two clears, this kernel, Adam) took 73.8 us with
// one output a thread, scalar reads and one warp of softmaxes; now 28.7 us.

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/mgbvh.h"
#include "mgbvh_mlp.cuh"

namespace mgbvh_mlp {

constexpr int kSB = 32;  // samples per CTA
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kOutPad = 52;  // outputs rounded up to whole float4s; the padding is zero
constexpr int kLdX = 28, kLdH = 68, kLdO = 52;  // row strides: odd counts of 16-byte words

struct TrainSmem {
    float w1[kH][kLdX];
    float b1[kH];
    float w2[kH][kLdH];
    float b2[kH];
    float w3[kOutPad][kLdH];
    float b3[kOutPad];
    float x[kSB][kLdX];
    float a1[kSB][kLdH], g1[kSB][kLdH];  // activation and GELU derivative; then d1
    float a2[kSB][kLdH], g2[kSB][kLdH];  // the same, then d2
    float d3[kSB][kLdO];                 // logits, then their gradients
    float loss[2][kWarps];
};

// Where element i of the flat parameter vector lies.
__device__ __forceinline__ float* param_slot(TrainSmem& S, int i) {
    if (i < kOB1) return &S.w1[i / kIn][i % kIn];
    if (i < kOW2) return &S.b1[i - kOB1];
    if (i < kOB2) return &S.w2[(i - kOW2) / kH][(i - kOW2) % kH];
    if (i < kOW3) return &S.b2[i - kOB2];
    if (i < kOB3) return &S.w3[(i - kOW3) / kH][(i - kOW3) % kH];
    return &S.b3[i - kOB3];
}

// acc[a][b] += sum over k < K of x[s0 + 16 a][k] * w[row[b]][k]
template <int K, int LDX, int LDW>
__device__ __forceinline__ void mul_rows(const float (*x)[LDX], const float (*w)[LDW], int s0, const int (&row)[4],
                                         float (&acc)[2][4]) {
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        float4 xv[2], wv4[4];
#pragma unroll
        for (int a = 0; a < 2; ++a) xv[a] = *reinterpret_cast<const float4*>(&x[s0 + 16 * a][k]);
#pragma unroll
        for (int b = 0; b < 4; ++b) wv4[b] = *reinterpret_cast<const float4*>(&w[row[b]][k]);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                float v = acc[a][b];
                v = fmaf(wv4[b].x, xv[a].x, v);
                v = fmaf(wv4[b].y, xv[a].y, v);
                v = fmaf(wv4[b].z, xv[a].z, v);
                acc[a][b] = fmaf(wv4[b].w, xv[a].w, v);
            }
    }
}

// One hidden layer: a = gelu(x W^T + b), and for training g = gelu'(.).
template <bool kTrain, int K, int LD>
__device__ __forceinline__ void hidden_layer(const float (*x)[LD], const float (*w)[LD], const float* bias,
                                             float (*act)[kLdH], float (*der)[kLdH]) {
    const int j0 = threadIdx.x % 16, s0 = threadIdx.x / 16;
    const int row[4] = {j0, j0 + 16, j0 + 32, j0 + 48};
    float acc[2][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[0][b] = acc[1][b] = bias[row[b]];
    mul_rows<K>(x, w, s0, row, acc);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const float z = acc[a][b];
            act[s0 + 16 * a][row[b]] = gelu(z);
            if (kTrain) der[s0 + 16 * a][row[b]] = gelu_grad(z);
        }
}

// d[s][j] = (sum over o < K of w[o][j] * up[s][o]) * der[s][j], in der's place.
template <int K, int LDU>
__device__ __forceinline__ void back_layer(const float (*up)[LDU], const float (*w)[kLdH], float (*der)[kLdH]) {
    const int j0 = 4 * (threadIdx.x % 16), s0 = threadIdx.x / 16;
    float acc[2][4] = {};
#pragma unroll 4
    for (int o = 0; o < K; o += 4) {
        float u[2][4];
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const float4 v = *reinterpret_cast<const float4*>(&up[s0 + 16 * a][o]);
            u[a][0] = v.x;
            u[a][1] = v.y;
            u[a][2] = v.z;
            u[a][3] = v.w;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float4 v = *reinterpret_cast<const float4*>(&w[o + c][j0]);
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                acc[a][0] = fmaf(v.x, u[a][c], acc[a][0]);
                acc[a][1] = fmaf(v.y, u[a][c], acc[a][1]);
                acc[a][2] = fmaf(v.z, u[a][c], acc[a][2]);
                acc[a][3] = fmaf(v.w, u[a][c], acc[a][3]);
            }
        }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        float4* p = reinterpret_cast<float4*>(&der[s0 + 16 * a][j0]);
        const float4 g = *p;
        *p = make_float4(acc[a][0] * g.x, acc[a][1] * g.y, acc[a][2] * g.z, acc[a][3] * g.w);
    }
}

// gw[o][i] += sum over the CTA's samples of d[s][o] * in[s][i] for o < M,
// i < N, and gb[o] += sum of d[s][o]. A half-warp's 16 threads hold 16
// neighbouring columns, so their atomics fill whole sectors.
template <int M, int N, int LDD, int LDI>
__device__ __forceinline__ void weight_grad(const float (*d)[LDD], const float (*in)[LDI], float* __restrict__ gw,
                                            float* __restrict__ gb) {
    constexpr int kCols = (N + 15) / 16;
    const int i0 = threadIdx.x % 16, o0 = 4 * (threadIdx.x / 16);
    if (o0 >= M) return;
    float acc[4][kCols] = {}, sum[4] = {};
#pragma unroll 4
    for (int s = 0; s < kSB; ++s) {
        const float4 v = *reinterpret_cast<const float4*>(&d[s][o0]);
        const float dv[4] = {v.x, v.y, v.z, v.w};
        float iv[kCols];
#pragma unroll
        for (int b = 0; b < kCols; ++b) iv[b] = (N % 16 == 0 || i0 + 16 * b < N) ? in[s][i0 + 16 * b] : 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            sum[c] += dv[c];
#pragma unroll
            for (int b = 0; b < kCols; ++b) acc[c][b] = fmaf(dv[c], iv[b], acc[c][b]);
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (o0 + c >= M) break;
#pragma unroll
        for (int b = 0; b < kCols; ++b)
            if (i0 + 16 * b < N) atomicAdd(&gw[(o0 + c) * N + i0 + 16 * b], acc[c][b]);
        if (i0 == 0) atomicAdd(&gb[o0 + c], sum[c]);
    }
}

__device__ __forceinline__ void load_block(TrainSmem& S, const float* __restrict__ x,
                                           const __nv_bfloat16* __restrict__ w, uint32_t base, int ns) {
    const int tid = threadIdx.x;
    for (int i = tid; i < kSB * kIn; i += kThreads) {
        const int s = i / kIn;
        S.x[s][i % kIn] = s < ns ? x[(size_t)(base + s) * kIn + (i % kIn)] : 0.0f;
    }
    // every matrix's rows and offsets are multiples of 8, so 8 parameters
    // read at once stay within one row; an unaligned vector takes single loads
    int done = 0;
    if ((reinterpret_cast<uintptr_t>(w) & 15u) == 0) {
        constexpr int kVecs = kParams / 8;
        const uint4* wv8 = reinterpret_cast<const uint4*>(w);
#pragma unroll
        for (int r = 0; r < (kVecs + kThreads - 1) / kThreads; ++r) {
            const int i = tid + r * kThreads;
            if (i < kVecs) {
                const uint4 q = wv8[i];
                float4* p = reinterpret_cast<float4*>(param_slot(S, 8 * i));
                p[0] = make_float4(__uint_as_float(q.x << 16), __uint_as_float(q.x & 0xFFFF0000u),
                                   __uint_as_float(q.y << 16), __uint_as_float(q.y & 0xFFFF0000u));
                p[1] = make_float4(__uint_as_float(q.z << 16), __uint_as_float(q.z & 0xFFFF0000u),
                                   __uint_as_float(q.w << 16), __uint_as_float(q.w & 0xFFFF0000u));
            }
        }
        done = 8 * kVecs;
    }
    for (int i = done + tid; i < kParams; i += kThreads) *param_slot(S, i) = __bfloat162float(w[i]);
    if (tid < kOutPad - kOut) S.b3[kOut + tid] = 0.0f;
    for (int i = tid; i < (kOutPad - kOut) * kH; i += kThreads) S.w3[kOut + i / kH][i % kH] = 0.0f;
    __syncthreads();
}

template <bool kTrain>
__device__ __forceinline__ void forward_block(TrainSmem& S) {
    hidden_layer<kTrain, kIn>(S.x, S.w1, S.b1, S.a1, S.g1);
    __syncthreads();
    hidden_layer<kTrain, kH>(S.a1, S.w2, S.b2, S.a2, S.g2);
    __syncthreads();
    const int o0 = threadIdx.x % 16, s0 = threadIdx.x / 16;
    const int row[4] = {o0, o0 + 16, o0 + 32, min(o0 + 48, kOutPad - 1)};
    float acc[2][4];
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[0][b] = acc[1][b] = S.b3[row[b]];
    mul_rows<kH>(S.a2, S.w3, s0, row, acc);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (o0 + 16 * b < kOutPad) S.d3[s0 + 16 * a][o0 + 16 * b] = acc[a][b];
    __syncthreads();
}

// Losses of the CTA's samples and the logits' gradients (mean over the batch:
// scale 1/B), a warp per sample: lane l has position logits l and 32 + l.
__device__ __forceinline__ void output_grad(TrainSmem& S, const uint32_t* __restrict__ label,
                                            const float* __restrict__ gain, uint32_t base, int ns, float invB) {
    const uint32_t full = 0xFFFFFFFFu;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const bool hi = lane < kPos - 32;  // this lane's second position logit exists
    float ce = 0.0f, bce = 0.0f;
#pragma unroll
    for (int s = warp; s < kSB; s += kWarps) {
        float* d = S.d3[s];
        float g0 = 0.0f, g1 = 0.0f;  // of outputs l and 32 + l; zero for no sample or label and for the padding
        if (s < ns) {
            const uint32_t lab = label[base + s];
            const float g = gain[base + s], l = d[kPos];
            const float l0 = d[lane], l1 = hi ? d[32 + lane] : -INFINITY;
            if (lab < (uint32_t)kPos) {  // kNoLabel and anything out of range: no position loss
                float m = fmaxf(l0, l1);
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(full, m, off));
                const float e0 = expf(l0 - m), e1 = hi ? expf(l1 - m) : 0.0f;
                float sum = e0 + e1;
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(full, sum, off);
                ce += logf(sum) + m - d[lab];
                g0 = (e0 / sum - (lane == (int)lab ? 1.0f : 0.0f)) * invB;
                if (hi) g1 = (e1 / sum - (32 + lane == (int)lab ? 1.0f : 0.0f)) * invB;
            }
            bce += fmaxf(l, 0.0f) + log1pf(expf(-fabsf(l))) - g * l;
            if (lane == kPos - 32) g1 = (1.0f / (1.0f + expf(-l)) - g) * invB;
        }
        __syncwarp();  // the logits are read before their gradients replace them
        d[lane] = g0;
        if (32 + lane < kOutPad) d[32 + lane] = g1;
    }
    if (lane == 0) {
        S.loss[0][warp] = ce;
        S.loss[1][warp] = bce;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads) train_kernel(const float* __restrict__ x,
                                                        const uint32_t* __restrict__ label,
                                                        const float* __restrict__ gain, uint32_t B,
                                                        const __nv_bfloat16* __restrict__ w,
                                                        float* __restrict__ grad, float* loss) {
    extern __shared__ __align__(16) unsigned char raw[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(raw);
    const uint32_t base = blockIdx.x * kSB;
    const int ns = (int)min((uint32_t)kSB, B - base);
    load_block(S, x, w, base, ns);
    forward_block<true>(S);
    output_grad(S, label, gain, base, ns, 1.0f / (float)B);
    if (threadIdx.x < 2) {
        float sum = 0.0f;
        for (int k = 0; k < kWarps; ++k) sum += S.loss[threadIdx.x][k];
        atomicAdd(&loss[threadIdx.x], sum);
    }
    weight_grad<kOut, kH>(S.d3, S.a2, grad + kOW3, grad + kOB3);
    back_layer<kOutPad>(S.d3, S.w3, S.g2);
    __syncthreads();
    weight_grad<kH, kH>(S.g2, S.a1, grad + kOW2, grad + kOB2);
    back_layer<kH>(S.g2, S.w2, S.g1);
    __syncthreads();
    weight_grad<kH, kIn>(S.g1, S.x, grad + kOW1, grad + kOB1);
}

__global__ void __launch_bounds__(kThreads) forward_kernel(const float* __restrict__ x, uint32_t B,
                                                          const __nv_bfloat16* __restrict__ w,
                                                          float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char raw[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(raw);
    const uint32_t base = blockIdx.x * kSB;
    const int ns = (int)min((uint32_t)kSB, B - base);
    load_block(S, x, w, base, ns);
    forward_block<false>(S);
    for (int idx = threadIdx.x; idx < ns * kOut; idx += kThreads)
        out[(size_t)(base + idx / kOut) * kOut + idx % kOut] = S.d3[idx / kOut][idx % kOut];
}

// Adam on FP32 master weights; writes the BF16 copy used by the passes.
__global__ void adam_kernel(float* __restrict__ master, __nv_bfloat16* __restrict__ w,
                            const float* __restrict__ grad, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps,
                            float bc1, float bc2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kParams) return;
    const float g = grad[i];
    const float mi = b1 * m[i] + (1.0f - b1) * g;
    const float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float p = master[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    master[i] = p;
    w[i] = __float2bfloat16_rn(p);
}

}  // namespace mgbvh_mlp

using namespace mgbvh_mlp;

extern "C" {

int mgbvh_mlp_train_step_dev(const float* d_features, const uint32_t* d_labels, const float* d_gains,
                             uint32_t batch, const void* d_weights_bf16, float* d_grad,
                             float* d_loss, void* stream) {
    if (!d_features || !d_labels || !d_gains || !d_weights_bf16 || !d_grad || !d_loss || batch == 0)
        return MGBVH_ERR_INVALID_ARG;
    // (a limit of the current device and context, so set on every call)
    if (cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(TrainSmem)) != cudaSuccess)
        return MGBVH_ERR_CUDA;
    train_kernel<<<(batch + kSB - 1) / kSB, kThreads, sizeof(TrainSmem),
                   reinterpret_cast<cudaStream_t>(stream)>>>(
        d_features, d_labels, d_gains, batch, static_cast<const __nv_bfloat16*>(d_weights_bf16), d_grad,
        d_loss);
    return cudaGetLastError() == cudaSuccess ? MGBVH_OK : MGBVH_ERR_CUDA;
}

int mgbvh_mlp_forward_dev(const float* d_features, uint32_t batch, const void* d_weights_bf16,
                          float* d_out, void* stream) {
    if (!d_features || !d_weights_bf16 || !d_out) return MGBVH_ERR_INVALID_ARG;
    if (batch == 0) return MGBVH_OK;
    if (cudaFuncSetAttribute(forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(TrainSmem)) != cudaSuccess)
        return MGBVH_ERR_CUDA;
    forward_kernel<<<(batch + kSB - 1) / kSB, kThreads, sizeof(TrainSmem),
                     reinterpret_cast<cudaStream_t>(stream)>>>(
        d_features, batch, static_cast<const __nv_bfloat16*>(d_weights_bf16), d_out);
    return cudaGetLastError() == cudaSuccess ? MGBVH_OK : MGBVH_ERR_CUDA;
}

int mgbvh_mlp_adam_dev(float* d_master, void* d_weights_bf16, const float* d_grad, float* d_m,
                       float* d_v, uint32_t step, float lr, float beta1, float beta2, float eps,
                       void* stream) {
    if (!d_master || !d_weights_bf16 || !d_grad || !d_m || !d_v || step == 0) return MGBVH_ERR_INVALID_ARG;
    const float bc1 = 1.0f - powf(beta1, (float)step);
    const float bc2 = 1.0f - powf(beta2, (float)step);
    adam_kernel<<<(kParams + 255) / 256, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        d_master, static_cast<__nv_bfloat16*>(d_weights_bf16), d_grad, d_m, d_v, lr, beta1, beta2, eps,
        bc1, bc2);
    return cudaGetLastError() == cudaSuccess ? MGBVH_OK : MGBVH_ERR_CUDA;
}

}  // extern "C"
