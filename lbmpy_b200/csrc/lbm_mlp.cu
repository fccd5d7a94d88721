// Training and evaluation kernels of the learned eddy-viscosity closure (lbm_closure.cuh).
//
// The network is tiny (1441 trained parameters) and the samples many, so training is a stream
// over samples: each block keeps the parameters in shared memory, runs forward and backward for
// one sample per thread with the activations in registers, parks the vectors that the weight
// gradient needs in shared memory, and then accumulates the outer products of a chunk of samples
// in register tiles.  Block partial gradients are summed in a fixed order by a second kernel
// (FP64), so the gradient is deterministic.  Adam updates the parameters in place.
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>

#include "../../include/lbm_b200.h"
#include "lbm_closure.cuh"
#include "lbm_dispatch.h"

using namespace lbm;

struct LbmMlp {
    int device;
    int max_blocks;
    float* partial;      // [max_blocks][MLP_TRAINED]
    double* loss_part;   // [max_blocks]
};

namespace {

constexpr int CHUNK = 64;                               // samples per block iteration (= threads)
// Record of one sample: h1, dz2, dz1, h2 (32 each), x (10) with a 1 behind it for the bias row, dy.
// Rows of 140 words: 16-byte accesses of neighbouring samples fall into different banks.
constexpr int REC_H1 = 0, REC_DZ2 = MLP_H, REC_DZ1 = 2 * MLP_H, REC_H2 = 3 * MLP_H, REC_X = 4 * MLP_H;
constexpr int REC_DY = REC_X + MLP_IN + 1;
constexpr int REC = 140;
static_assert(REC_DY < REC && REC % 4 == 0 && REC % 32 == 12 && MLP_IN == 10 && MLP_H == 32, "record layout");
constexpr int GRAD_SMEM = (MLP_PARAMS + 2 + CHUNK * REC) * int(sizeof(float));
static_assert(MLP_B1 % 4 == 0 && MLP_W2 % 4 == 0 && MLP_B2 % 4 == 0 && MLP_W3 % 4 == 0 && (MLP_PARAMS + 2) % 4 == 0,
              "16-byte loads of the staged parameters");

// Features from the per-sample state (SoA [10][n]: Pxx Pyy Pzz Pxy Pxz Pyz rho ux uy uz).
__global__ void __launch_bounds__(256) k_closure_features(const float* __restrict__ state, long long n,
                                                         float* __restrict__ feats) {
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        float v[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) v[k] = state[k * n + s];
        float x[MLP_IN];
        closure_features<float>(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], x);
#pragma unroll
        for (int k = 0; k < MLP_IN; ++k) feats[k * n + s] = x[k];
    }
}

// Evaluation: one sample per thread, first-layer activations parked in shared memory (the same
// summation order as closure_nu_t).
__global__ void __launch_bounds__(128) k_mlp_forward(const float* __restrict__ params, const float* __restrict__ feats,
                                                    long long n, float* __restrict__ nu) {
    __shared__ float w[MLP_PARAMS];
    __shared__ float hs[MLP_H][128 + 1];
    for (int i = threadIdx.x; i < MLP_PARAMS; i += blockDim.x) w[i] = params[i];
    __syncthreads();
    for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < n; s += (long long)gridDim.x * blockDim.x) {
        float x[MLP_IN];
#pragma unroll
        for (int k = 0; k < MLP_IN; ++k) x[k] = feats[k * n + s];
#pragma unroll 1
        for (int k = 0; k < MLP_H; ++k) {
            float z = w[MLP_B1 + k];
#pragma unroll
            for (int i = 0; i < MLP_IN; ++i) z += x[i] * w[MLP_W1 + i * MLP_H + k];
            hs[k][threadIdx.x] = mlp_silu<float>(z);
        }
        float y = w[MLP_B3];
#pragma unroll 1
        for (int k = 0; k < MLP_H; ++k) {
            float z = w[MLP_B2 + k];
#pragma unroll 8
            for (int j = 0; j < MLP_H; ++j) z += hs[j][threadIdx.x] * w[MLP_W2 + j * MLP_H + k];
            y += mlp_silu<float>(z) * w[MLP_W3 + k];
        }
        nu[s] = w[MLP_SCALE] * mlp_softplus<float>(y);
    }
}

// z[k] += a * w[k] for the 32 units of a layer: w in shared memory, the same address for every
// lane, two units per packed FP32 instruction.
__device__ __forceinline__ void axpy_row(float2 (&z)[MLP_H / 2], float a, const float* w) {
    const float2 aa = make_float2(a, a);
#pragma unroll
    for (int q = 0; q < MLP_H / 4; ++q) {
        const float4 v = reinterpret_cast<const float4*>(w)[q];
        z[2 * q] = __ffma2_rn(aa, make_float2(v.x, v.y), z[2 * q]);
        z[2 * q + 1] = __ffma2_rn(aa, make_float2(v.z, v.w), z[2 * q + 1]);
    }
}

__device__ __forceinline__ void load_row(float2 (&z)[MLP_H / 2], const float* w) {
#pragma unroll
    for (int q = 0; q < MLP_H / 4; ++q) {
        const float4 v = reinterpret_cast<const float4*>(w)[q];
        z[2 * q] = make_float2(v.x, v.y);
        z[2 * q + 1] = make_float2(v.z, v.w);
    }
}

// SiLU of the pre-activations z (into h) and its derivative (into z).
__device__ __forceinline__ void activate(float2 (&z)[MLP_H / 2], float2 (&h)[MLP_H / 2]) {
    auto one = [](float& v, float& o) {
        const float sg = mlp_sigmoid<float>(v);
        o = v * sg;
        v = sg * (1.f + v * (1.f - sg));
    };
#pragma unroll
    for (int q = 0; q < MLP_H / 2; ++q) {
        one(z[q].x, h[q].x);
        one(z[q].y, h[q].y);
    }
}

__device__ __forceinline__ void store_row(float* r, const float2 (&v)[MLP_H / 2]) {
#pragma unroll
    for (int q = 0; q < MLP_H / 4; ++q)
        reinterpret_cast<float4*>(r)[q] = make_float4(v[2 * q].x, v[2 * q].y, v[2 * q + 1].x, v[2 * q + 1].y);
}

// Forward + backward of one chunk of samples per iteration, then that chunk's part of the weight
// gradient, accumulated per block over its chunks.
// Bound by instruction issue.  A sample's 2400 multiply-adds of forward and backward run on packed
// FP32 pairs against parameters that one 16-byte shared load brings to the whole warp, and each thread
// keeps a 4 x 4 tile of the second layer's gradient, so that a sample costs it two 16-byte loads for 16
// products.  (One gradient entry at a time, with two shared loads per product and the activations in
// shared memory, took 72 us for 65536 samples.)  Chunks of 64 samples and 4 blocks per SM (as many as the
// default trainer launches).  Every second chunk the tiles are added to totals of their own, so that a
// chain of FP32 additions is 128 samples, or the number of such groups, long: one tile over all samples of a
// block loses digits as they grow in number (3e-3 relative at 2^19 samples a block, 5e-5 so).
__global__ void __launch_bounds__(CHUNK, 4) k_mlp_grad_partial(const float* __restrict__ params,
                                                           const float* __restrict__ feats,
                                                           const float* __restrict__ target,
                                                           const float* __restrict__ weight, long long n,
                                                           float inv_wsum, float* __restrict__ partial,
                                                           double* __restrict__ loss_part) {
    extern __shared__ __align__(16) float sm[];
    float* w = sm;                         // MLP_PARAMS
    float* rec = sm + MLP_PARAMS + 2;      // CHUNK * REC (offset keeps 16-byte alignment)
    const int tid = threadIdx.x, lane = tid & 31;
    for (int i = tid; i < MLP_PARAMS; i += CHUNK) w[i] = params[i];
    // second layer: rows 4 jt .. + 3, columns 4 kt .. + 3; first warp: the first layer's 10 rows and
    // its bias, column `lane`; second warp: output weights and the other biases, column `lane`
    const int jt = tid >> 3, kt = tid & 7;
    float g2[4][4], g1[MLP_IN + 1];
    float sum2[4][4], sum1[MLP_IN + 1];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) g2[a][b] = sum2[a][b] = 0.f;
#pragma unroll
    for (int a = 0; a <= MLP_IN; ++a) g1[a] = sum1[a] = 0.f;
    auto close_group = [&] {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                sum2[a][b] += g2[a][b];
                g2[a][b] = 0.f;
            }
#pragma unroll
        for (int a = 0; a <= MLP_IN; ++a) {
            sum1[a] += g1[a];
            g1[a] = 0.f;
        }
    };
    bool second = false;
    double loss = 0.0;
    const float scale = params[MLP_SCALE];
    __syncthreads();
    const long long nchunks = (n + CHUNK - 1) / CHUNK;
    for (long long c = blockIdx.x; c < nchunks; c += gridDim.x) {
        const long long s = c * CHUNK + tid;
        float* r = rec + tid * REC;
        if (s < n) {
            float2 z1[MLP_H / 2], h[MLP_H / 2];
            load_row(z1, w + MLP_B1);
            float x[MLP_IN];
#pragma unroll
            for (int i = 0; i < MLP_IN; ++i) x[i] = r[REC_X + i] = feats[i * n + s];
#pragma unroll
            for (int i = 0; i < MLP_IN; ++i) axpy_row(z1, x[i], w + MLP_W1 + i * MLP_H);
            r[REC_X + MLP_IN] = 1.f;
            activate(z1, h);
            store_row(r + REC_H1, h);
            store_row(r + REC_DZ1, z1);                        // derivative, turned into dz1 below
            float2 z2[MLP_H / 2];
            load_row(z2, w + MLP_B2);
#pragma unroll 1
            for (int j = 0; j < MLP_H; j += 4) {               // rolled: unrolled it keeps 1024 weights in flight
                const float4 hj = *reinterpret_cast<const float4*>(r + REC_H1 + j);
                axpy_row(z2, hj.x, w + MLP_W2 + j * MLP_H);
                axpy_row(z2, hj.y, w + MLP_W2 + (j + 1) * MLP_H);
                axpy_row(z2, hj.z, w + MLP_W2 + (j + 2) * MLP_H);
                axpy_row(z2, hj.w, w + MLP_W2 + (j + 3) * MLP_H);
            }
            activate(z2, h);
            store_row(r + REC_H2, h);
            float2 w3[MLP_H / 2], yy = make_float2(w[MLP_B3], 0.f);
            load_row(w3, w + MLP_W3);
#pragma unroll
            for (int q = 0; q < MLP_H / 2; ++q) yy = __ffma2_rn(h[q], w3[q], yy);
            const float y = yy.x + yy.y;
            const float nu = scale * mlp_softplus<float>(y);
            const float wt = weight ? weight[s] : 1.f;
            const float res = nu - target[s];
            loss += (double)wt * res * res * inv_wsum;
            const float dy = 2.f * wt * res * inv_wsum * scale * (y > 20.f ? 1.f : mlp_sigmoid<float>(y));
            r[REC_DY] = dy;
            const float2 dd = make_float2(dy, dy);
#pragma unroll
            for (int q = 0; q < MLP_H / 2; ++q) z2[q] = __fmul2_rn(z2[q], __fmul2_rn(dd, w3[q]));   // dz2
            store_row(r + REC_DZ2, z2);
            auto dot = [&](int j) {
                float2 d = make_float2(0.f, 0.f);
#pragma unroll
                for (int q = 0; q < MLP_H / 4; ++q) {
                    const float4 v = reinterpret_cast<const float4*>(w + MLP_W2 + j * MLP_H)[q];
                    d = __ffma2_rn(z2[2 * q], make_float2(v.x, v.y), d);
                    d = __ffma2_rn(z2[2 * q + 1], make_float2(v.z, v.w), d);
                }
                return d.x + d.y;
            };
#pragma unroll 1
            for (int j = 0; j < MLP_H; j += 4) {
                float4* dz1 = reinterpret_cast<float4*>(r + REC_DZ1 + j);
                const float4 v = *dz1;
                *dz1 = make_float4(v.x * dot(j), v.y * dot(j + 1), v.z * dot(j + 2), v.w * dot(j + 3));
            }
        } else {
            for (int k = 0; k < REC; ++k) r[k] = 0.f;
        }
        __syncthreads();
#pragma unroll 4
        for (int t = 0; t < CHUNK; ++t) {
            const float* q = rec + t * REC;
            const float4 a = reinterpret_cast<const float4*>(q + REC_H1)[jt];
            const float4 b = reinterpret_cast<const float4*>(q + REC_DZ2)[kt];
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int k = 0; k < 4; ++k) g2[i][k] += av[i] * bv[k];
            if (tid < 32) {
                const float d = q[REC_DZ1 + lane];
                const float4 x0 = reinterpret_cast<const float4*>(q + REC_X)[0];
                const float4 x1 = reinterpret_cast<const float4*>(q + REC_X)[1];
                const float4 x2 = reinterpret_cast<const float4*>(q + REC_X)[2];   // x8, x9, 1, dy
                const float xv[MLP_IN + 1] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w, x2.x, x2.y, x2.z};
#pragma unroll
                for (int i = 0; i <= MLP_IN; ++i) g1[i] += xv[i] * d;
            } else {
                const float dy = q[REC_DY];
                g1[0] += q[REC_H2 + lane] * dy;     // output weights
                g1[1] += q[REC_DZ2 + lane];         // second bias
                g1[2] += dy;                        // output bias
            }
        }
        __syncthreads();
        if (second) close_group();
        second = !second;
    }
    close_group();
    float* out = partial + (long long)blockIdx.x * MLP_TRAINED;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) out[MLP_W2 + (4 * jt + i) * MLP_H + 4 * kt + k] = sum2[i][k];
    if (tid < 32) {
#pragma unroll
        for (int i = 0; i < MLP_IN; ++i) out[MLP_W1 + i * MLP_H + lane] = sum1[i];
        out[MLP_B1 + lane] = sum1[MLP_IN];
    } else {
        out[MLP_W3 + lane] = sum1[0];
        out[MLP_B2 + lane] = sum1[1];
        if (lane == 0) out[MLP_B3] = sum1[2];
    }
    // block loss: fixed-order tree in shared memory
    __shared__ double red[CHUNK];
    red[tid] = loss;
    __syncthreads();
    for (int h = CHUNK / 2; h > 0; h >>= 1) {
        if (tid < h) red[tid] += red[tid + h];
        __syncthreads();
    }
    if (tid == 0) loss_part[blockIdx.x] = red[0];
}

// Sum of the block partials, FP64.  Bound by the latency of the loads: a warp takes 32 neighbouring
// entries, FINISH_WARPS warps share the blocks between them (block b goes to warp b % FINISH_WARPS)
// and their sums are added in order, so the result does not depend on timing.  One thread per entry
// running over all blocks took 27 us for 592 blocks.
constexpr int FINISH_WARPS = 16;
__global__ void __launch_bounds__(32 * FINISH_WARPS) k_mlp_grad_finish(const float* __restrict__ partial,
                                                                       const double* __restrict__ loss_part, int blocks,
                                                                       float* __restrict__ grad,
                                                                       double* __restrict__ loss) {
    __shared__ double part[FINISH_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane;
    double s = 0.0;
    if (e < MLP_TRAINED) {
#pragma unroll 4
        for (int b = warp; b < blocks; b += FINISH_WARPS) s += partial[(long long)b * MLP_TRAINED + e];
    } else if (e == MLP_TRAINED && loss) {
#pragma unroll 4
        for (int b = warp; b < blocks; b += FINISH_WARPS) s += loss_part[b];
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp != 0 || e > MLP_TRAINED) return;
    s = 0.0;
#pragma unroll
    for (int k = 0; k < FINISH_WARPS; ++k) s += part[k][lane];
    if (e < MLP_TRAINED) {
        grad[e] = (float)s;
    } else {
        grad[e] = 0.f;                    // the output scale is not trained
        if (loss) *loss = s;
    }
}

__global__ void k_mlp_adam(const float* __restrict__ grad, float* __restrict__ params, float* __restrict__ m,
                           float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= MLP_TRAINED) return;
    const float g = grad[e];
    const float mm = b1 * m[e] + (1.f - b1) * g;
    const float vv = b2 * v[e] + (1.f - b2) * g * g;
    m[e] = mm;
    v[e] = vv;
    params[e] -= lr * (mm / c1) / (sqrtf(vv / c2) + eps);
}

int device_ptr_ok(const void* p, bool nullable) {
    if (p == nullptr) return nullable ? 0 : 1;
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return 1;
    }
    return (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged) ? 0 : 1;
}

int grid_for(long long n, int threads) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    long long b = (n + threads - 1) / threads;
    const long long cap = (long long)sms * 8;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace

extern "C" {

int lbm_closure_features(const float* state, int64_t n, float* feats, void* stream) {
    if (n < 1) return abi_fail(LBM_E_INVALID, "n must be positive");
    if (device_ptr_ok(state, false) || device_ptr_ok(feats, false))
        return abi_fail(LBM_E_INVALID, "state and feats must be device pointers");
    k_closure_features<<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(state, n, feats);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? LBM_OK : abi_fail(LBM_E_CUDA, "closure features: %s", cudaGetErrorString(e));
}

int lbm_mlp_forward(const float* params, const float* feats, int64_t n, float* nu, void* stream) {
    if (n < 1) return abi_fail(LBM_E_INVALID, "n must be positive");
    if (device_ptr_ok(params, false) || device_ptr_ok(feats, false) || device_ptr_ok(nu, false))
        return abi_fail(LBM_E_INVALID, "params, feats and nu must be device pointers");
    k_mlp_forward<<<grid_for(n, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(params, feats, n, nu);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? LBM_OK : abi_fail(LBM_E_CUDA, "mlp forward: %s", cudaGetErrorString(e));
}

int lbm_mlp_create(int max_blocks, LbmMlp** out) {
    if (out == nullptr || max_blocks < 1) return abi_fail(LBM_E_INVALID, "out must not be NULL, max_blocks >= 1");
    *out = nullptr;
    LbmMlp* m = new LbmMlp();
    cudaGetDevice(&m->device);
    m->max_blocks = max_blocks;
    m->partial = nullptr;
    m->loss_part = nullptr;
    cudaError_t e = cudaMalloc(&m->partial, sizeof(float) * MLP_TRAINED * (size_t)max_blocks);
    if (e == cudaSuccess) e = cudaMalloc(&m->loss_part, sizeof(double) * (size_t)max_blocks);
    if (e == cudaSuccess) {
        e = cudaFuncSetAttribute(k_mlp_grad_partial, cudaFuncAttributeMaxDynamicSharedMemorySize, GRAD_SMEM);
    }
    if (e != cudaSuccess) {
        cudaFree(m->partial);
        cudaFree(m->loss_part);
        delete m;
        return abi_fail(LBM_E_CUDA, "lbm_mlp_create: %s", cudaGetErrorString(e));
    }
    *out = m;
    return LBM_OK;
}

int lbm_mlp_destroy(LbmMlp* m) {
    if (m == nullptr) return LBM_OK;
    cudaFree(m->partial);
    cudaFree(m->loss_part);
    delete m;
    return LBM_OK;
}

int lbm_mlp_loss_grad(LbmMlp* m, const float* params, const float* feats, const float* target, const float* weight,
                      int64_t n, double inv_wsum, float* grad, double* loss, void* stream) {
    if (m == nullptr) return abi_fail(LBM_E_INVALID, "trainer is NULL");
    if (n < 1) return abi_fail(LBM_E_INVALID, "n must be positive");
    if (device_ptr_ok(params, false) || device_ptr_ok(feats, false) || device_ptr_ok(target, false) ||
        device_ptr_ok(weight, true) || device_ptr_ok(grad, false) || device_ptr_ok(loss, true))
        return abi_fail(LBM_E_INVALID, "params, feats, target, weight, grad and loss must be device pointers");
    const long long chunks = (n + CHUNK - 1) / CHUNK;
    const int blocks = (int)(chunks < m->max_blocks ? chunks : m->max_blocks);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_mlp_grad_partial<<<blocks, CHUNK, GRAD_SMEM, s>>>(params, feats, target, weight, n, (float)inv_wsum, m->partial,
                                                   m->loss_part);
    k_mlp_grad_finish<<<(MLP_PARAMS + 31) / 32, 32 * FINISH_WARPS, 0, s>>>(m->partial, m->loss_part, blocks, grad, loss);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? LBM_OK : abi_fail(LBM_E_CUDA, "mlp loss/grad: %s", cudaGetErrorString(e));
}

int lbm_mlp_adam(const float* grad, float* params, float* m1, float* m2, double lr, double beta1, double beta2,
                 double eps, int step, void* stream) {
    if (step < 1) return abi_fail(LBM_E_INVALID, "Adam steps count from 1");
    if (device_ptr_ok(grad, false) || device_ptr_ok(params, false) || device_ptr_ok(m1, false) ||
        device_ptr_ok(m2, false))
        return abi_fail(LBM_E_INVALID, "grad, params and the moment buffers must be device pointers");
    const float c1 = (float)(1.0 - pow(beta1, step)), c2 = (float)(1.0 - pow(beta2, step));
    k_mlp_adam<<<(MLP_TRAINED + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(
        grad, params, m1, m2, (float)lr, (float)beta1, (float)beta2, (float)eps, c1, c2);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? LBM_OK : abi_fail(LBM_E_CUDA, "mlp adam: %s", cudaGetErrorString(e));
}

}  // extern "C"
