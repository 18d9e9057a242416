// Training and inference kernels of the learned block order's scorer: a multilayer perceptron
// 32 -> 64 -> 64 -> 1 with ReLU, BF16 operands (inputs, weights, activations and the
// backward products' gradient operands rounded to BF16) and FP32 products and sums.  The
// gradient is that of the mean weighted binary cross-entropy with logits.  Every unit sums
// its inputs in index order, as the planner's scorer does (mlp_score_warp in score.cuh).
//
// The reference has no learned component; these kernels back the block ordering only.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include "ltl_kernels.cuh"
#include "ltlgpu.h"

namespace ltlg {
namespace {

constexpr int NF = ORDER_NF, H = ORDER_H;
constexpr int REC = 16;       // records a CTA of the gradient kernel works on at a time
constexpr int THREADS = 512;  // threads per CTA of the gradient kernel
constexpr int GRAD_CTAS = 296;  // CTAs at most (each then takes several groups of records)
constexpr int PER = (MLP_PARAMS + THREADS - 1) / THREADS;  // parameters per thread

__device__ __forceinline__ float bf(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ float wf(__nv_bfloat16 w) { return __bfloat162float(w); }

// Forward pass of one record (x already rounded to BF16): the logit; h1, h2 receive the
// BF16-rounded activations.
__device__ float forward_record(const MlpDev &M, const float *x, float *h1, float *h2) {
    for (int j = 0; j < H; ++j) {
        float acc = 0.0f;
        for (int i = 0; i < NF; ++i) acc += wf(M.w1[j * NF + i]) * x[i];
        h1[j] = bf(fmaxf(acc + M.b1[j], 0.0f));
    }
    for (int j = 0; j < H; ++j) {
        float acc = 0.0f;
        for (int k = 0; k < H; ++k) acc += wf(M.w2[j * H + k]) * h1[k];
        h2[j] = bf(fmaxf(acc + M.b2[j], 0.0f));
    }
    float z = 0.0f;
    for (int k = 0; k < H; ++k) z += wf(M.w3[k]) * h2[k];
    return z + M.b3;
}

__global__ void forward_kernel(const MlpDev *__restrict__ M, const float *__restrict__ X, int count,
                               float *__restrict__ logits) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= count) return;
    float x[NF], h1[H], h2[H];
    for (int i = 0; i < NF; ++i) x[i] = bf(X[(size_t)r * NF + i]);
    logits[r] = forward_record(*M, x, h1, h2);
}

// Gradient of inv_norm * sum_r w_r * BCE(z_r, y_r) over the records idx[first .. first + n)
// (or first .. first + n when idx is null): each CTA's part into part[CTA][MLP_PARAMS], its loss into
// *loss.  A CTA takes REC records at a time: a layer's units of all of them are spread over the threads
// (thread = unit of some records), then the parameters, each thread keeping the sums of its own over
// the CTA's records in registers.
//
// A batch of 1,024 records is 10 million multiply-adds, nothing for the chip; what it took was one
// thread's chain through a whole record (weights read by each thread, activations in local memory) and
// the atomic adds of 6,337 sums per CTA: 194 us a training step with the update, 16,384 records.
__global__ void __launch_bounds__(THREADS) grad_kernel(const MlpDev *__restrict__ M, const float *__restrict__ X,
                                                       const float *__restrict__ Y, const int *__restrict__ idx,
                                                       long long first, int n, float pos_weight, float inv_norm,
                                                       float *__restrict__ part, float *__restrict__ loss) {
    __shared__ __align__(16) __nv_bfloat16 w1t[NF * H], w2[H * H], w2t[H * H];  // filled 16 bytes at a time
    __shared__ __nv_bfloat16 w3[H];
    static_assert(__alignof__(w1t) >= 16 && __alignof__(w2) >= 16 && __alignof__(w2t) >= 16, "16-byte stores");
    __shared__ float b1[H], b2[H], x[REC][NF], h1[REC][H], h2[REC][H], d1[REC][H], d2[REC][H], dz[REC], dzb[REC];
    const int t = threadIdx.x;
    for (int i = t; i < NF * H / 8; i += THREADS) reinterpret_cast<uint4 *>(w1t)[i] = reinterpret_cast<const uint4 *>(M->w1t)[i];
    for (int i = t; i < H * H / 8; i += THREADS) {
        reinterpret_cast<uint4 *>(w2)[i] = reinterpret_cast<const uint4 *>(M->w2)[i];
        reinterpret_cast<uint4 *>(w2t)[i] = reinterpret_cast<const uint4 *>(M->w2t)[i];
    }
    if (t < H) {
        w3[t] = M->w3[t];
        b1[t] = M->b1[t];
        b2[t] = M->b2[t];
    }
    float g[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) g[q] = 0.0f;
    float my_loss = 0.0f;
    const int j = t & (H - 1), r0 = t / H;
    constexpr int RS = THREADS / H;
    for (int base = blockIdx.x * REC; base < n; base += gridDim.x * REC) {
        __syncthreads();
        for (int i = t; i < REC * NF; i += THREADS) {
            const int q = base + i / NF;
            const long long r = q < n ? (idx ? (long long)idx[first + q] : first + q) : 0;
            x[i / NF][i % NF] = q < n ? bf(X[r * NF + i % NF]) : 0.0f;
        }
        __syncthreads();
        for (int r = r0; r < REC; r += RS) {
            float acc = 0.0f;
#pragma unroll 8
            for (int i = 0; i < NF; ++i) acc += wf(w1t[i * H + j]) * x[r][i];
            h1[r][j] = bf(fmaxf(acc + b1[j], 0.0f));
        }
        __syncthreads();
        for (int r = r0; r < REC; r += RS) {
            float acc = 0.0f;
#pragma unroll 8
            for (int k = 0; k < H; ++k) acc += wf(w2t[k * H + j]) * h1[r][k];
            h2[r][j] = bf(fmaxf(acc + b2[j], 0.0f));
        }
        __syncthreads();
        if (t < REC) {
            const int q = base + t;
            float v = 0.0f;
            if (q < n) {
                float z = 0.0f;
#pragma unroll 8
                for (int k = 0; k < H; ++k) z += wf(w3[k]) * h2[t][k];
                z += M->b3;
                const float y = Y[idx ? (long long)idx[first + q] : first + q];
                const float w = y > 0.5f ? pos_weight : 1.0f;
                const float p = 1.0f / (1.0f + expf(-z));
                my_loss += w * (fmaxf(z, 0.0f) - z * y + log1pf(expf(-fabsf(z))));
                v = w * (p - y) * inv_norm;
            }
            dz[t] = v;
            dzb[t] = bf(v);
        }
        __syncthreads();
        for (int r = r0; r < REC; r += RS) d2[r][j] = h2[r][j] > 0.0f ? bf(dz[r] * wf(w3[j])) : 0.0f;
        __syncthreads();
        for (int r = r0; r < REC; r += RS) {
            float acc = 0.0f;
#pragma unroll 8
            for (int k = 0; k < H; ++k) acc += wf(w2[k * H + j]) * d2[r][k];
            d1[r][j] = h1[r][j] > 0.0f ? bf(acc) : 0.0f;
        }
        __syncthreads();
        const int m = min(REC, n - base);
#pragma unroll
        for (int q = 0; q < PER; ++q) {
            const int p = t + q * THREADS;
            float s = g[q];
            if (p < MLP_B1) {
                const int a = p / NF, i = p % NF;
                for (int r = 0; r < m; ++r) s += d1[r][a] * x[r][i];
            } else if (p < MLP_W2) {
                for (int r = 0; r < m; ++r) s += d1[r][p - MLP_B1];
            } else if (p < MLP_B2) {
                const int k = (p - MLP_W2) / H, a = (p - MLP_W2) % H;
                for (int r = 0; r < m; ++r) s += d2[r][k] * h1[r][a];
            } else if (p < MLP_W3) {
                for (int r = 0; r < m; ++r) s += d2[r][p - MLP_B2];
            } else if (p < MLP_B3) {
                for (int r = 0; r < m; ++r) s += dzb[r] * h2[r][p - MLP_W3];
            } else if (p < MLP_PARAMS) {
                for (int r = 0; r < m; ++r) s += dz[r];
            }
            g[q] = s;
        }
    }
#pragma unroll
    for (int q = 0; q < PER; ++q)
        if (t + q * THREADS < MLP_PARAMS) part[(size_t)blockIdx.x * MLP_PARAMS + t + q * THREADS] = g[q];
    if (t < 32) {
        for (int o = 16; o > 0; o >>= 1) my_loss += __shfl_xor_sync(0xFFFFFFFFu, my_loss, o);
        if (t == 0 && my_loss != 0.0f) atomicAdd(loss, my_loss);
    }
}
int grad_ctas(int n) { return std::min(GRAD_CTAS, (n + REC - 1) / REC); }

// Parameter i's gradient: the CTAs' parts in order.
__device__ __forceinline__ float sum_parts(const float *__restrict__ part, int ctas, int i) {
    float g = 0.0f;
#pragma unroll 8
    for (int c = 0; c < ctas; ++c) g += part[(size_t)c * MLP_PARAMS + i];
    return g;
}
__global__ void sum_kernel(const float *__restrict__ part, int ctas, float *__restrict__ grad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < MLP_PARAMS) grad[i] = sum_parts(part, ctas, i);
}

// Parameter i of the packed FP32 vector into the scorer's device form: weights rounded to BF16.
__device__ __forceinline__ void pack_param(MlpDev *m, int i, float v) {
    if (i < MLP_B1) {
        m->w1[i] = __float2bfloat16(v);
        m->w1t[(i % NF) * H + i / NF] = __float2bfloat16(v);
    } else if (i < MLP_W2) {
        m->b1[i - MLP_B1] = v;
    } else if (i < MLP_B2) {
        const int q = i - MLP_W2;
        m->w2[q] = __float2bfloat16(v);
        m->w2t[(q % H) * H + q / H] = __float2bfloat16(v);
    } else if (i < MLP_W3) {
        m->b2[i - MLP_B2] = v;
    } else if (i < MLP_B3) {
        m->w3[i - MLP_W3] = __float2bfloat16(v);
    } else {
        m->b3 = v;
    }
}
__global__ void scorer_pack_kernel(const float *__restrict__ p, MlpDev *__restrict__ m) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < MLP_PARAMS) pack_param(m, i, p[i]);
}

// AdamW step on the FP32 master parameters (weight decay on weights only) from the gradient's parts,
// and the device form refreshed.
__global__ void adam_kernel(float *__restrict__ p, const float *__restrict__ part, int ctas, float *__restrict__ m,
                            float *__restrict__ v, MlpDev *__restrict__ dev, float lr, float b1, float b2, float eps, float wd,
                            float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= MLP_PARAMS) return;
    const float gi = sum_parts(part, ctas, i);
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const bool weight = i < MLP_B1 || (i >= MLP_W2 && i < MLP_B2) || (i >= MLP_W3 && i < MLP_B3);
    float pi = p[i];
    if (weight) pi -= lr * wd * pi;
    pi -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    pack_param(dev, i, pi);
}

// Device buffers of one scorer call (default stream), freed on scope exit.
struct Bufs {
    std::vector<void *> ptrs;
    ~Bufs() {
        for (void *p : ptrs) cudaFreeAsync(p, 0);
    }
    template <class T>
    T *alloc(size_t n, cudaError_t &err) {
        void *p = nullptr;
        if (err == cudaSuccess) err = cudaMallocAsync(&p, std::max<size_t>(n, 1) * sizeof(T), 0);
        if (err == cudaSuccess) ptrs.push_back(p);
        return (T *)p;
    }
};

int status_of(cudaError_t e) {
    return e == cudaSuccess ? 0 : e == cudaErrorMemoryAllocation ? LTLG_NO_MEMORY : LTLG_CUDA_ERROR;
}

bool has_device() {
    int n = 0;
    return cudaGetDeviceCount(&n) == cudaSuccess && n > 0;
}

}  // namespace

cudaError_t launch_scorer_pack(const float *params, MlpDev *out, cudaStream_t s) {
    scorer_pack_kernel<<<(MLP_PARAMS + 255) / 256, 256, 0, s>>>(params, out);
    return cudaGetLastError();
}

}  // namespace ltlg

using namespace ltlg;

extern "C" LTLG_API int ltlg_scorer_forward(const float *params, const float *features, int32_t count, float *logits) {
    if (!params || count < 0 || (count > 0 && (!features || !logits))) return LTLG_BAD_ARGS;
    if (!has_device()) return LTLG_NO_DEVICE;
    if (count == 0) return 0;
    cudaError_t err = cudaSuccess;
    Bufs b;
    float *dp = b.alloc<float>(MLP_PARAMS, err);
    MlpDev *dm = b.alloc<MlpDev>(1, err);
    float *dx = b.alloc<float>((size_t)count * NF, err);
    float *dz = b.alloc<float>(count, err);
    if (err == cudaSuccess) err = cudaMemcpy(dp, params, MLP_PARAMS * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = cudaMemcpy(dx, features, (size_t)count * NF * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = launch_scorer_pack(dp, dm, 0);
    if (err == cudaSuccess) {
        forward_kernel<<<(count + 127) / 128, 128>>>(dm, dx, count, dz);
        err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaMemcpy(logits, dz, (size_t)count * sizeof(float), cudaMemcpyDeviceToHost);
    return status_of(err);
}

extern "C" LTLG_API int ltlg_scorer_grad(const float *params, const float *features, const float *labels, int32_t count,
                                         float pos_weight, float *grad, float *loss) {
    if (!params || !grad || count <= 0 || !features || !labels) return LTLG_BAD_ARGS;
    if (!has_device()) return LTLG_NO_DEVICE;
    cudaError_t err = cudaSuccess;
    Bufs b;
    float *dp = b.alloc<float>(MLP_PARAMS, err);
    MlpDev *dm = b.alloc<MlpDev>(1, err);
    float *dx = b.alloc<float>((size_t)count * NF, err);
    float *dy = b.alloc<float>(count, err);
    float *dg = b.alloc<float>(MLP_PARAMS + 1, err);
    float *dpart = b.alloc<float>((size_t)grad_ctas(count) * MLP_PARAMS, err);
    if (err == cudaSuccess) err = cudaMemcpy(dp, params, MLP_PARAMS * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = cudaMemcpy(dx, features, (size_t)count * NF * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = cudaMemcpy(dy, labels, (size_t)count * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = cudaMemset(dg, 0, (MLP_PARAMS + 1) * sizeof(float));
    if (err == cudaSuccess) err = launch_scorer_pack(dp, dm, 0);
    if (err == cudaSuccess) {
        grad_kernel<<<grad_ctas(count), THREADS>>>(dm, dx, dy, nullptr, 0, count, pos_weight, 1.0f / (float)count, dpart,
                                                   dg + MLP_PARAMS);
        sum_kernel<<<(MLP_PARAMS + 255) / 256, 256>>>(dpart, grad_ctas(count), dg);
        err = cudaGetLastError();
    }
    std::vector<float> h(MLP_PARAMS + 1);
    if (err == cudaSuccess) err = cudaMemcpy(h.data(), dg, h.size() * sizeof(float), cudaMemcpyDeviceToHost);
    if (err != cudaSuccess) return status_of(err);
    memcpy(grad, h.data(), MLP_PARAMS * sizeof(float));
    if (loss) *loss = h[MLP_PARAMS] / (float)count;
    return 0;
}

extern "C" LTLG_API int ltlg_scorer_train(float *params, const float *features, const float *labels, int32_t count,
                                          const ltlg_train_config *cfg, float *epoch_loss) {
    if (!params || !cfg || count <= 0 || !features || !labels || cfg->epochs < 0 || cfg->batch <= 0)
        return LTLG_BAD_ARGS;
    if (!has_device()) return LTLG_NO_DEVICE;
    cudaError_t err = cudaSuccess;
    Bufs b;
    float *dp = b.alloc<float>(MLP_PARAMS, err);
    float *dm1 = b.alloc<float>(MLP_PARAMS, err);
    float *dv = b.alloc<float>(MLP_PARAMS, err);
    float *dloss = b.alloc<float>(1, err);
    float *dpart = b.alloc<float>((size_t)grad_ctas(std::min(cfg->batch, count)) * MLP_PARAMS, err);
    MlpDev *dm = b.alloc<MlpDev>(1, err);
    float *dx = b.alloc<float>((size_t)count * NF, err);
    float *dy = b.alloc<float>(count, err);
    int *didx = b.alloc<int>(count, err);
    if (err == cudaSuccess) err = cudaMemcpy(dp, params, MLP_PARAMS * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = cudaMemset(dm1, 0, MLP_PARAMS * sizeof(float));
    if (err == cudaSuccess) err = cudaMemset(dv, 0, MLP_PARAMS * sizeof(float));
    if (err == cudaSuccess) err = cudaMemcpy(dx, features, (size_t)count * NF * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = cudaMemcpy(dy, labels, (size_t)count * sizeof(float), cudaMemcpyHostToDevice);
    if (err == cudaSuccess) err = launch_scorer_pack(dp, dm, 0);
    std::vector<int> perm(count);
    for (int i = 0; i < count; ++i) perm[i] = i;
    uint64_t s = cfg->seed;
    auto next = [&]() {  // splitmix64
        s += 0x9E3779B97F4A7C15ull;
        uint64_t z = s;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    long long step = 0;
    for (int ep = 0; ep < cfg->epochs && err == cudaSuccess; ++ep) {
        for (int i = count - 1; i > 0; --i) std::swap(perm[i], perm[(int)(next() % (uint64_t)(i + 1))]);
        err = cudaMemcpy(didx, perm.data(), (size_t)count * sizeof(int), cudaMemcpyHostToDevice);
        if (err == cudaSuccess) err = cudaMemset(dloss, 0, sizeof(float));
        for (long long first = 0; first < count && err == cudaSuccess; first += cfg->batch) {
            const int nb = (int)std::min<long long>(cfg->batch, count - first);
            ++step;
            const int ctas = grad_ctas(nb);
            grad_kernel<<<ctas, THREADS>>>(dm, dx, dy, didx, first, nb, cfg->pos_weight, 1.0f / (float)nb, dpart, dloss);
            const float c1 = 1.0f - std::pow(cfg->beta1, (float)step), c2 = 1.0f - std::pow(cfg->beta2, (float)step);
            adam_kernel<<<(MLP_PARAMS + 63) / 64, 64>>>(dp, dpart, ctas, dm1, dv, dm, cfg->lr, cfg->beta1, cfg->beta2,
                                                        cfg->eps, cfg->weight_decay, c1, c2);
            err = cudaGetLastError();
        }
        float lsum = 0.0f;
        if (err == cudaSuccess) err = cudaMemcpy(&lsum, dloss, sizeof(float), cudaMemcpyDeviceToHost);
        if (epoch_loss) epoch_loss[ep] = lsum / (float)count;
    }
    if (err == cudaSuccess) err = cudaMemcpy(params, dp, MLP_PARAMS * sizeof(float), cudaMemcpyDeviceToHost);
    return status_of(err);
}
