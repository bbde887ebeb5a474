// mlp.cu -- the learned step-size proposer: an 8 -> 64 -> 64 -> 1 perceptron with SiLU
// activations, BF16 weights and FP32 accumulation, trained on the GPU by the kernels below
// (forward, backward, AdamW) from the attempt logs the ensemble integrator writes.
//
// Not in the reference (the reference has no learned component).  Inputs are standardised
// features of a disk at the start of a step; the output is log(ideal step / last ideal step).
//
// Parameter vector (FP32 master copy; the forward passes read its BF16 image):
//   W1[64][8] b1[64] W2[64][64] b2[64] w3[64] b3
// Training: CTAs walk tiles of MLP_TB samples with the activations in shared memory; the
// matrix products are register-tiled FP32 FMA loops (the activations and their gradients stay
// FP32, which the tensor cores do not take), the weight gradients stay in registers from tile
// to tile, and each CTA adds its sums to a global FP32 buffer once, with atomics.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <random>
#include <string>
#include <vector>

#include "../../include/redgb.h"
#include "abi_guard.h"
#include "common.cuh"
#include "mlp.h"

namespace redgb {
int set_error(int code, const std::string& msg);

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z)
{
    const float s = 1.0f / (1.0f + __expf(-z));
    return s * (1.0f + z * (1.0f - s));
}

// FP32 master -> BF16 image
__global__ void mlp_to_bf16(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) wb[i] = __float2bfloat16_rn(w[i]);
}

__device__ __forceinline__ float bf(const __nv_bfloat16* w, int i) { return __bfloat162float(w[i]); }

struct MlpNorm {
    float mean[MLP_IN], std[MLP_IN];
};

// Shared-memory matrices are H rows of MLP_TB or H columns, padded so that a row starts four
// banks after the one before it: the float4 stores of 8 neighbouring lanes to 8 neighbouring
// rows touch every bank once.  A thread's four units are u = (t & 15) + 16 j; in rows over
// units they stand together (position 4 (u & 15) + (u >> 4)), one float4.
constexpr int MLP_PITCH = MLP_TB + 4;
constexpr int MLP_MAT = MLP_HIDDEN * MLP_PITCH;
static_assert(MLP_TB == MLP_HIDDEN && MLP_TB == 64, "256 threads hold a tile as 4 x 4 blocks");
__device__ __forceinline__ int mlp_pos(int u) { return ((u & 15) << 2) | (u >> 4); }

struct MlpSmem {
    float W1t[MLP_IN][MLP_HIDDEN];  // [f][position of u]
    float X[MLP_TB][MLP_IN];        // standardised inputs
    float b1[MLP_HIDDEN], b2[MLP_HIDDEN], w3[MLP_HIDDEN];
    float D[MLP_TB];  // dL/dy per sample
    float W2t[MLP_MAT];  // [v][position of u]
    float A1t[MLP_MAT];  // silu(Z1), [v][s]
    float A2t[MLP_MAT];  // silu(Z2), [u][s]; then dL/dZ2, [u][s]
};
struct MlpTrainSmem : MlpSmem {
    float W2p[MLP_MAT];  // [u][position of v]
    float A1p[MLP_MAT];  // silu(Z1), [s][position of v]
    float G2p[MLP_MAT];  // dL/dZ2, [s][position of u]
};
constexpr int MLP_FORWARD_CTAS = 3;  // per SM (training: 2)
constexpr int MLP_GROUP = MLP_HIDDEN * (MLP_IN + 1);  // dW1 and db1 of one sample group
static_assert(16 * MLP_GROUP <= 3 * MLP_MAT, "the groups' sums fit over the last three matrices");
static_assert(sizeof(MlpSmem) % 16 == 0, "float4 rows");

// acc[i][j] += sum over k of A[k][4 a + i] B[k][4 b + j], k ascending
__device__ __forceinline__ void mlp_mma(float (&acc)[4][4], const float* A, const float* B)
{
#pragma unroll 8
    for (int k = 0; k < 64; k++) {
        const float4 a = *reinterpret_cast<const float4*>(A + k * MLP_PITCH);
        const float4 b = *reinterpret_cast<const float4*>(B + k * MLP_PITCH);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
}

// Forward (and optionally backward) of the samples.  x: n x 8; y: targets (training); index:
// the samples' rows or null; out: predictions; grad: += dL/dw and, behind it, += the loss (FP32).
// Thread t holds samples 4 (t / 16) .. + 3 and units (t & 15) + 16 j of a tile of 64.
// Bound: the FP32 pipe (three 64 x 64 x 64 products a tile in training, one in the forward
// pass) behind the SiLUs and the barriers between the phases; 16 warps an SM in training, limited
// by the matrices' shared memory, 24 in the forward pass (16: 55 us, 32: as 24).  A thread's 4 x 4
// block reads two float4 for 16 FMAs, each SiLU is taken once, and the weights' gradients go to
// global memory once a CTA; one output per thread with its operands and SiLUs from shared memory
// and a CTA's atomics per 32 samples took 280 us (forward) and 617 us (training) for 100 000
// samples, this 46 and 112 us.  The loss is summed like the gradient of b3, a thread's tiles first
// (1e-6 of it off up to a million samples; half of the samples one by one in one FP32 sum: 114 us,
// and 1e-5 off at 100 000, 3e-4 at a million).
template <bool TRAIN>
__global__ void __launch_bounds__(256, TRAIN ? 2 : MLP_FORWARD_CTAS)
    mlp_tile_kernel(const __nv_bfloat16* __restrict__ wb, const MlpNorm norm, const float* __restrict__ x,
                    const float* __restrict__ y, const int* __restrict__ index, int n, float inv_batch,
                    float* __restrict__ out, float* __restrict__ grad)
{
    constexpr int H = MLP_HIDDEN, I = MLP_IN, TB = MLP_TB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MlpTrainSmem& S = *reinterpret_cast<MlpTrainSmem*>(smem_raw);  // the forward pass stops at MlpSmem's end
    const int t = threadIdx.x, ug = t & 15, sg = t >> 4, s0 = 4 * sg;
    for (int k = t; k < H * I; k += 256) S.W1t[k % I][mlp_pos(k / I)] = bf(wb, MLP_OFF_W1 + k);
    for (int k = t; k < H * H; k += 256) {
        const float w = bf(wb, MLP_OFF_W2 + k);
        S.W2t[(k % H) * MLP_PITCH + mlp_pos(k / H)] = w;
        if (TRAIN) S.W2p[(k / H) * MLP_PITCH + mlp_pos(k % H)] = w;
    }
    if (t < H) {
        S.b1[t] = bf(wb, MLP_OFF_B1 + t);
        S.b2[t] = bf(wb, MLP_OFF_B2 + t);
        S.w3[t] = bf(wb, MLP_OFF_W3 + t);
    }
    const float b3 = bf(wb, MLP_OFF_B3);
    [[maybe_unused]] float gw2[4][4], gw1[4][I], gb1[4], gw3 = 0.0f, gb2 = 0.0f, gb3 = 0.0f, loss = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        gb1[j] = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; i++) gw2[i][j] = 0.0f;
#pragma unroll
        for (int f = 0; f < I; f++) gw1[j][f] = 0.0f;
    }
    const int tiles = n / TB + (n % TB != 0);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int first = tile * TB, ns = min(TB, n - first);
        if (t < 2 * TB) {  // four inputs of sample t / 2
            const int s = t >> 1, f = 4 * (t & 1);
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (s < ns) {
                v = *reinterpret_cast<const float4*>(x + (size_t)(index ? index[first + s] : first + s) * I + f);
                v.x = __fdiv_rn(v.x - norm.mean[f], norm.std[f]);
                v.y = __fdiv_rn(v.y - norm.mean[f + 1], norm.std[f + 1]);
                v.z = __fdiv_rn(v.z - norm.mean[f + 2], norm.std[f + 2]);
                v.w = __fdiv_rn(v.w - norm.mean[f + 3], norm.std[f + 3]);
            }
            *reinterpret_cast<float4*>(&S.X[s][f]) = v;
        }
        __syncthreads();
        [[maybe_unused]] float ds1[4][4];
        float acc[4][4];
        // layer 1: Z1 = X W1^T + b1
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float b = S.b1[ug + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i][j] = b;
        }
#pragma unroll
        for (int f = 0; f < I; f++) {
            const float4 w = *reinterpret_cast<const float4*>(&S.W1t[f][4 * ug]);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float v = S.X[s0 + i][f];
                acc[i][0] = fmaf(w.x, v, acc[i][0]);
                acc[i][1] = fmaf(w.y, v, acc[i][1]);
                acc[i][2] = fmaf(w.z, v, acc[i][2]);
                acc[i][3] = fmaf(w.w, v, acc[i][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                if (TRAIN) ds1[i][j] = dsilu(acc[i][j]);
                acc[i][j] = silu(acc[i][j]);
            }
#pragma unroll
        for (int j = 0; j < 4; j++)
            *reinterpret_cast<float4*>(&S.A1t[(ug + 16 * j) * MLP_PITCH + s0]) =
                make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
        if constexpr (TRAIN)
#pragma unroll
            for (int i = 0; i < 4; i++)
                *reinterpret_cast<float4*>(&S.A1p[(s0 + i) * MLP_PITCH + 4 * ug]) =
                    make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        __syncthreads();
        // layer 2: Z2 = silu(Z1) W2^T + b2
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float b = S.b2[ug + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; i++) acc[i][j] = b;
        }
        mlp_mma(acc, S.A1t + s0, S.W2t + 4 * ug);
#pragma unroll
        for (int j = 0; j < 4; j++)
            *reinterpret_cast<float4*>(&S.A2t[(ug + 16 * j) * MLP_PITCH + s0]) =
                make_float4(silu(acc[0][j]), silu(acc[1][j]), silu(acc[2][j]), silu(acc[3][j]));
        __syncthreads();
        // output: y = w3 . silu(Z2) + b3
        if (t < TB) {
            float o = b3;
#pragma unroll 16
            for (int u = 0; u < H; u++) o = fmaf(S.w3[u], S.A2t[u * MLP_PITCH + t], o);
            [[maybe_unused]] float d = 0.0f, e = 0.0f;
            if (t < ns) {
                if (out) out[first + t] = o;
                if (TRAIN) {
                    const float r = o - y[index ? index[first + t] : first + t];
                    d = 2.0f * r * inv_batch;
                    e = r * r * inv_batch;
                }
            }
            if constexpr (TRAIN) {
                S.D[t] = d;
                gb3 += d;
                loss += e;
            }
        }
        __syncthreads();
        if constexpr (TRAIN) {
            // backward.  dw3 = sum_s D_s silu(Z2_s): unit t / 4, a quarter of the samples
            {
                const float* a = &S.A2t[(t >> 2) * MLP_PITCH + 16 * (t & 3)];
#pragma unroll
                for (int q = 0; q < 16; q++) gw3 = fmaf(S.D[16 * (t & 3) + q], a[q], gw3);
            }
            __syncthreads();
            // dZ2 = D w3 silu'(Z2)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float w = S.w3[ug + 16 * j];
#pragma unroll
                for (int i = 0; i < 4; i++) acc[i][j] = S.D[s0 + i] * w * dsilu(acc[i][j]);
                *reinterpret_cast<float4*>(&S.A2t[(ug + 16 * j) * MLP_PITCH + s0]) =
                    make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
                *reinterpret_cast<float4*>(&S.G2p[(s0 + i) * MLP_PITCH + 4 * ug]) =
                    make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
            __syncthreads();
            // db2[u] = sum_s dZ2[s][u]
            {
                const float* a = &S.A2t[(t >> 2) * MLP_PITCH + 16 * (t & 3)];
#pragma unroll
                for (int q = 0; q < 16; q++) gb2 += a[q];
            }
            // dW2[u][v] = sum_s dZ2[s][u] silu(Z1[s][v]): units sg + 16 i
            mlp_mma(gw2, S.G2p + 4 * sg, S.A1p + 4 * ug);
            // dZ1[s][v] = (sum_u dZ2[s][u] W2[u][v]) silu'(Z1[s][v])
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
            mlp_mma(acc, S.A2t + s0, S.W2p + 4 * ug);
            // dW1[v][f] = sum_s dZ1[s][v] X[s][f]; db1[v] = sum_s dZ1[s][v]
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 xa = *reinterpret_cast<const float4*>(&S.X[s0 + i][0]);
                const float4 xb = *reinterpret_cast<const float4*>(&S.X[s0 + i][4]);
                const float xv[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float d = acc[i][j] * ds1[i][j];
                    gb1[j] += d;
#pragma unroll
                    for (int f = 0; f < I; f++) gw1[j][f] = fmaf(d, xv[f], gw1[j][f]);
                }
            }
            __syncthreads();  // the next tile overwrites X and the matrices
        }
    }
    if constexpr (!TRAIN) return;
    // the CTA's sums, once
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) atomicAdd(&grad[MLP_OFF_W2 + (sg + 16 * i) * H + ug + 16 * j], gw2[i][j]);
    float* const g = S.W2p + sg * MLP_GROUP;
#pragma unroll
    for (int j = 0; j < 4; j++) {
#pragma unroll
        for (int f = 0; f < I; f++) g[(ug + 16 * j) * (I + 1) + f] = gw1[j][f];
        g[(ug + 16 * j) * (I + 1) + I] = gb1[j];
    }
    for (int d = 1; d < 4; d <<= 1) {
        gw3 += __shfl_xor_sync(0xffffffffu, gw3, d);
        gb2 += __shfl_xor_sync(0xffffffffu, gb2, d);
    }
    if ((t & 3) == 0) {
        atomicAdd(&grad[MLP_OFF_W3 + (t >> 2)], gw3);
        atomicAdd(&grad[MLP_OFF_B2 + (t >> 2)], gb2);
    }
    if (t < TB) {
        for (int d = 1; d < 32; d <<= 1) {
            gb3 += __shfl_xor_sync(0xffffffffu, gb3, d);
            loss += __shfl_xor_sync(0xffffffffu, loss, d);
        }
        if ((t & 31) == 0) {
            atomicAdd(&grad[MLP_OFF_B3], gb3);
            atomicAdd(&grad[MLP_NPARAM], loss);
        }
    }
    __syncthreads();
    for (int k = t; k < MLP_GROUP; k += 256) {
        float v = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; q++) v += S.W2p[q * MLP_GROUP + k];
        const int u = k / (I + 1), f = k % (I + 1);
        atomicAdd(&grad[f < I ? MLP_OFF_W1 + u * I + f : MLP_OFF_B1 + u], v);
    }
}

// AdamW on the FP32 master weights (decoupled weight decay on the matrices only)
__global__ void mlp_adamw_kernel(float* w, float* m, float* v, const float* g, int n, float lr, float b1, float b2,
                                 float eps, float wd, float bc1, float bc2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bool matrix = (i >= MLP_OFF_W1 && i < MLP_OFF_B1) || (i >= MLP_OFF_W2 && i < MLP_OFF_B2) ||
                        (i >= MLP_OFF_W3 && i < MLP_OFF_B3);
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float wi = w[i];
    if (matrix) wi -= lr * wd * wi;
    wi -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    w[i] = wi;
}

}  // namespace redgb

using namespace redgb;

struct rg_mlp {
    std::vector<float> w;  // FP32 master (host copy kept in sync on demand)
    float norm_mean[MLP_IN], norm_std[MLP_IN];
    float* d_w = nullptr;
    float* d_m = nullptr;
    float* d_v = nullptr;
    float* d_g = nullptr;  // gradient and, behind it, the loss
    __nv_bfloat16* d_wb = nullptr;
    float* h_g = nullptr;  // pinned copy of d_g
    // samples of the last calls (grown, freed with the network): a call holds `lock` while it
    // uses them and the gradient buffer
    float *d_x = nullptr, *d_y = nullptr;
    int* d_idx = nullptr;
    size_t cap_x = 0, cap_y = 0, cap_idx = 0;
    int n_sm = 0;
    std::mutex lock;
    int64_t step = 0;
    cudaStream_t st = nullptr;
};

namespace {

int sync_bf16(rg_mlp* m)
{
    mlp_to_bf16<<<(MLP_NPARAM + 255) / 256, 256, 0, m->st>>>(m->d_w, m->d_wb, MLP_NPARAM);
    RG_CUDA_CHECK(cudaGetLastError());
    return RG_OK;
}

template <class T>
int dalloc(T** p, size_t n)
{
    if (cudaMalloc((void**)p, (n ? n : 1) * sizeof(T)) != cudaSuccess) {
        *p = nullptr;
        return set_error(RG_ERR_NOMEM, "cudaMalloc (mlp)");
    }
    return RG_OK;
}

int create_impl(uint64_t seed, rg_mlp** out)
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n <= 0) {
        cudaGetLastError();
        return set_error(RG_ERR_NO_DEVICE, "no CUDA device");
    }
    rg_mlp* m = new rg_mlp();
    m->w.assign(MLP_NPARAM, 0.0f);
    std::mt19937_64 rng(seed);
    auto init = [&](int off, int fan_out, int fan_in) {
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / (float)(fan_in + fan_out)));
        for (int k = 0; k < fan_out * fan_in; k++) m->w[off + k] = nd(rng);
    };
    init(MLP_OFF_W1, MLP_HIDDEN, MLP_IN);
    init(MLP_OFF_W2, MLP_HIDDEN, MLP_HIDDEN);
    init(MLP_OFF_W3, 1, MLP_HIDDEN);
    for (int f = 0; f < MLP_IN; f++) {
        m->norm_mean[f] = 0.0f;
        m->norm_std[f] = 1.0f;
    }
    int rc = RG_OK;
    if (cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking) != cudaSuccess) rc = set_error(RG_ERR_CUDA, "stream");
    if (!rc) rc = dalloc(&m->d_w, MLP_NPARAM);
    if (!rc) rc = dalloc(&m->d_m, MLP_NPARAM);
    if (!rc) rc = dalloc(&m->d_v, MLP_NPARAM);
    if (!rc) rc = dalloc(&m->d_g, MLP_NPARAM + 1);
    if (!rc) rc = dalloc(&m->d_wb, MLP_NPARAM);
    if (!rc && cudaMallocHost((void**)&m->h_g, (MLP_NPARAM + 1) * sizeof(float)) != cudaSuccess) {
        m->h_g = nullptr;
        cudaGetLastError();
        rc = set_error(RG_ERR_NOMEM, "cudaMallocHost (mlp)");
    }
    int dev = 0;
    if (!rc && (cudaGetDevice(&dev) != cudaSuccess ||
                cudaDeviceGetAttribute(&m->n_sm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess))
        rc = set_error(RG_ERR_CUDA, "device attributes");
    if (!rc && (cudaFuncSetAttribute(mlp_tile_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(MlpSmem)) != cudaSuccess ||
                cudaFuncSetAttribute(mlp_tile_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(MlpTrainSmem)) != cudaSuccess))
        rc = set_error(RG_ERR_CUDA, "shared memory of the proposer's kernels");
    if (!rc && cudaMemcpy(m->d_w, m->w.data(), MLP_NPARAM * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess)
        rc = set_error(RG_ERR_CUDA, "upload");
    if (!rc && cudaMemset(m->d_m, 0, MLP_NPARAM * sizeof(float)) != cudaSuccess) rc = RG_ERR_CUDA;
    if (!rc && cudaMemset(m->d_v, 0, MLP_NPARAM * sizeof(float)) != cudaSuccess) rc = RG_ERR_CUDA;
    if (!rc) rc = sync_bf16(m);
    if (!rc && cudaStreamSynchronize(m->st) != cudaSuccess) rc = set_error(RG_ERR_CUDA, "init");
    if (rc) {
        rg_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return RG_OK;
}

template <class T>
int reserve(T** p, size_t* cap, size_t n)
{
    if (n <= *cap) return RG_OK;
    cudaFree(*p);
    *p = nullptr;
    *cap = 0;
    const int rc = dalloc(p, n);
    if (!rc) *cap = n;
    return rc;
}

// the inputs (and targets) in the network's device buffers
int upload(rg_mlp* m, const float* x, const float* y, int n)
{
    int rc = reserve(&m->d_x, &m->cap_x, (size_t)n * MLP_IN);
    if (!rc) rc = reserve(&m->d_y, &m->cap_y, (size_t)n);
    if (!rc)
        RG_CUDA_CHECK(cudaMemcpyAsync(m->d_x, x, (size_t)n * MLP_IN * sizeof(float), cudaMemcpyHostToDevice, m->st));
    if (!rc && y) RG_CUDA_CHECK(cudaMemcpyAsync(m->d_y, y, n * sizeof(float), cudaMemcpyHostToDevice, m->st));
    return rc;
}

int run_tiles(rg_mlp* m, bool train, const float* d_x, const float* d_y, const int* d_idx, int n, float* d_out,
              float inv_batch)
{
    if (n <= 0) return RG_OK;
    const int grid = std::min(n / MLP_TB + (n % MLP_TB != 0), (train ? 2 : MLP_FORWARD_CTAS) * m->n_sm);
    MlpNorm norm;
    for (int f = 0; f < MLP_IN; f++) {
        norm.mean[f] = m->norm_mean[f];
        norm.std[f] = m->norm_std[f];
    }
    if (train)
        mlp_tile_kernel<true><<<grid, 256, sizeof(MlpTrainSmem), m->st>>>(m->d_wb, norm, d_x, d_y, d_idx, n, inv_batch,
                                                                          d_out, m->d_g);
    else
        mlp_tile_kernel<false><<<grid, 256, sizeof(MlpSmem), m->st>>>(m->d_wb, norm, d_x, d_y, d_idx, n, inv_batch,
                                                                      d_out, nullptr);
    RG_CUDA_CHECK(cudaGetLastError());
    return RG_OK;
}

int zero_gradient(rg_mlp* m)
{
    RG_CUDA_CHECK(cudaMemsetAsync(m->d_g, 0, (MLP_NPARAM + 1) * sizeof(float), m->st));
    return RG_OK;
}

int forward_impl(rg_mlp* m, const float* x, int n, float* y)
{
    std::lock_guard<std::mutex> hold(m->lock);
    int rc = upload(m, x, nullptr, n);
    if (!rc) rc = run_tiles(m, false, m->d_x, nullptr, nullptr, n, m->d_y, 0.0f);
    if (!rc) RG_CUDA_CHECK(cudaMemcpyAsync(y, m->d_y, n * sizeof(float), cudaMemcpyDeviceToHost, m->st));
    if (!rc) RG_CUDA_CHECK(cudaStreamSynchronize(m->st));
    return rc;
}

int gradient_impl(rg_mlp* m, const float* x, const float* y, int n, float* grads, float* loss)
{
    std::lock_guard<std::mutex> hold(m->lock);
    int rc = upload(m, x, y, n);
    if (!rc) rc = zero_gradient(m);
    if (!rc) rc = run_tiles(m, true, m->d_x, m->d_y, nullptr, n, nullptr, 1.0f / (float)n);
    if (!rc)
        RG_CUDA_CHECK(cudaMemcpyAsync(m->h_g, m->d_g, (MLP_NPARAM + 1) * sizeof(float), cudaMemcpyDeviceToHost, m->st));
    if (!rc) RG_CUDA_CHECK(cudaStreamSynchronize(m->st));
    if (rc) return rc;
    std::memcpy(grads, m->h_g, MLP_NPARAM * sizeof(float));
    if (loss) *loss = m->h_g[MLP_NPARAM];
    return RG_OK;
}

int train_impl(rg_mlp* m, const float* x, const float* y, int n, int epochs, int batch, float lr, float weight_decay,
               uint64_t seed, float* final_loss)
{
    std::lock_guard<std::mutex> hold(m->lock);
    int rc = upload(m, x, y, n);
    if (!rc) rc = reserve(&m->d_idx, &m->cap_idx, (size_t)n);
    if (rc) return rc;
    std::vector<int> idx(n);
    for (int i = 0; i < n; i++) idx[i] = i;
    std::mt19937_64 rng(seed);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    for (int ep = 0; ep < epochs && !rc; ep++) {
        std::shuffle(idx.begin(), idx.end(), rng);
        RG_CUDA_CHECK(cudaMemcpyAsync(m->d_idx, idx.data(), n * sizeof(int), cudaMemcpyHostToDevice, m->st));
        for (int b0 = 0; b0 < n && !rc; b0 += batch) {
            const int nb = std::min(batch, n - b0);
            rc = zero_gradient(m);
            if (!rc) rc = run_tiles(m, true, m->d_x, m->d_y, m->d_idx + b0, nb, nullptr, 1.0f / (float)nb);
            if (rc) break;
            m->step++;
            const float bc1 = 1.0f - std::pow(b1, (float)m->step), bc2 = 1.0f - std::pow(b2, (float)m->step);
            mlp_adamw_kernel<<<(MLP_NPARAM + 255) / 256, 256, 0, m->st>>>(m->d_w, m->d_m, m->d_v, m->d_g, MLP_NPARAM, lr,
                                                                        b1, b2, eps, weight_decay, bc1, bc2);
            RG_CUDA_CHECK(cudaGetLastError());
            rc = sync_bf16(m);
        }
    }
    if (!rc)
        RG_CUDA_CHECK(cudaMemcpyAsync(m->h_g, m->d_g + MLP_NPARAM, sizeof(float), cudaMemcpyDeviceToHost, m->st));
    if (!rc) RG_CUDA_CHECK(cudaStreamSynchronize(m->st));
    if (!rc && final_loss) *final_loss = m->h_g[0];
    return rc;
}

}  // namespace

extern "C" {

int rg_mlp_create(uint64_t seed, rg_mlp** out)
{
    if (!out) return set_error(RG_ERR_ARG, "null output");
    try {
        return create_impl(seed, out);
    } catch (const std::bad_alloc&) {
        return set_error(RG_ERR_NOMEM, "host allocation failed");
    }
}

int rg_mlp_destroy(rg_mlp* m)
{
    if (!m) return set_error(RG_ERR_ARG, "null network");
    if (m->st) cudaStreamSynchronize(m->st);
    cudaFree(m->d_w);
    cudaFree(m->d_m);
    cudaFree(m->d_v);
    cudaFree(m->d_g);
    cudaFree(m->d_wb);
    cudaFree(m->d_x);
    cudaFree(m->d_y);
    cudaFree(m->d_idx);
    cudaFreeHost(m->h_g);
    if (m->st) cudaStreamDestroy(m->st);
    delete m;
    return RG_OK;
}

int rg_mlp_set_normalisation(rg_mlp* m, const float mean[MLP_IN], const float stdev[MLP_IN])
{
    if (!m || !mean || !stdev) return set_error(RG_ERR_ARG, "bad argument");
    for (int f = 0; f < MLP_IN; f++) {
        if (!(stdev[f] > 0.0f)) return set_error(RG_ERR_ARG, "standard deviation must be positive");
        m->norm_mean[f] = mean[f];
        m->norm_std[f] = stdev[f];
    }
    return RG_OK;
}

int rg_mlp_get_normalisation(rg_mlp* m, float mean[MLP_IN], float stdev[MLP_IN])
{
    if (!m || !mean || !stdev) return set_error(RG_ERR_ARG, "bad argument");
    for (int f = 0; f < MLP_IN; f++) {
        mean[f] = m->norm_mean[f];
        stdev[f] = m->norm_std[f];
    }
    return RG_OK;
}

int rg_mlp_get_params(rg_mlp* m, float* w, int n)
{
    if (!m || !w || n != MLP_NPARAM) return set_error(RG_ERR_ARG, "bad argument");
    RG_CUDA_CHECK(cudaMemcpy(w, m->d_w, MLP_NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    return RG_OK;
}

int rg_mlp_set_params(rg_mlp* m, const float* w, int n)
{
    if (!m || !w || n != MLP_NPARAM) return set_error(RG_ERR_ARG, "bad argument");
    RG_CUDA_CHECK(cudaMemcpy(m->d_w, w, MLP_NPARAM * sizeof(float), cudaMemcpyHostToDevice));
    int rc = sync_bf16(m);
    if (!rc) RG_CUDA_CHECK(cudaStreamSynchronize(m->st));
    return rc;
}

int rg_mlp_forward(rg_mlp* m, const float* x, int n, float* y)
{
    if (!m || n < 0 || (n > 0 && (!x || !y))) return set_error(RG_ERR_ARG, "bad argument");
    if (n == 0) return RG_OK;
    RG_GUARD(forward_impl(m, x, n, y));
}

// mean-squared-error gradient of one batch (no update): grads[MLP_NPARAM], loss
int rg_mlp_gradient(rg_mlp* m, const float* x, const float* y, int n, float* grads, float* loss)
{
    if (!m || n <= 0 || !x || !y || !grads) return set_error(RG_ERR_ARG, "bad argument");
    RG_GUARD(gradient_impl(m, x, y, n, grads, loss));
}

// AdamW training: `epochs` passes over the n samples in shuffled minibatches.
int rg_mlp_train(rg_mlp* m, const float* x, const float* y, int n, int epochs, int batch, float lr, float weight_decay,
                 uint64_t seed, float* final_loss)
{
    if (!m || !x || !y || n <= 0 || epochs <= 0 || batch <= 0 || !(lr > 0.0f))
        return set_error(RG_ERR_ARG, "bad argument");
    RG_GUARD(train_impl(m, x, y, n, epochs, batch, lr, weight_decay, seed, final_loss));
}

}  // extern "C"

// access for the ensemble's proposer kernel
namespace redgb {
const void* mlp_device_weights(const rg_mlp* m) { return m ? (const void*)m->d_wb : nullptr; }
void mlp_normalisation(const rg_mlp* m, float* mean, float* stdev)
{
    for (int f = 0; f < MLP_IN; f++) {
        mean[f] = m->norm_mean[f];
        stdev[f] = m->norm_std[f];
    }
}
}  // namespace redgb
