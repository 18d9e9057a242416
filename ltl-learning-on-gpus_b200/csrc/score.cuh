// The learned block order's scorer on the device, one warp per feature vector.  Shared by
// the planner (the level kernel's planning warp) and nothing else on the device; the training
// kernels (mlp.cu) compute the same function one record per thread.
#pragma once

#include <cuda_bf16.h>

#include "ops.cuh"

namespace ltlg {

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16(x)); }

// The scorer on up to SCORE_N feature vectors at once, one warp: lane l computes hidden units l and
// l + 32 of each layer for all of them.  Vector q is f of lane src[q]; the logits go to z (the same
// in every lane).  Operands are rounded to BF16, products and sums are FP32, and every unit sums its
// inputs in index order (the same order as forward_record in mlp.cu).
//
// Bound by the loads of the weights: read [in][out], a warp's loads are two cache lines a layer input,
// and one load serves all the vectors.  One vector at a time from [out][in] weights (a line per lane)
// took about 11 us each, 115 us of planning for a level's ten blocks.
constexpr int SCORE_N = 4;
__device__ __noinline__ void mlp_score_warp(const MlpDev &M, const float *f, const int (&src)[SCORE_N], int lane,
                                            float (&z)[SCORE_N]) {
    float acc[SCORE_N][2], h[SCORE_N][2];
#pragma unroll
    for (int q = 0; q < SCORE_N; ++q) acc[q][0] = acc[q][1] = 0.0f;
#pragma unroll 8
    for (int i = 0; i < ORDER_NF; ++i) {
        const float w0 = __bfloat162float(M.w1t[i * ORDER_H + lane]), w1 = __bfloat162float(M.w1t[i * ORDER_H + lane + 32]);
        const float fi = bf16r(f[i]);
#pragma unroll
        for (int q = 0; q < SCORE_N; ++q) {
            const float x = __shfl_sync(FULL, fi, src[q]);
            acc[q][0] += w0 * x;
            acc[q][1] += w1 * x;
        }
    }
#pragma unroll
    for (int q = 0; q < SCORE_N; ++q)
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            h[q][u] = bf16r(fmaxf(acc[q][u] + M.b1[lane + 32 * u], 0.0f));
            acc[q][u] = 0.0f;
        }
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
            const int in = (k + 32 * v) * ORDER_H + lane;
            const float w0 = __bfloat162float(M.w2t[in]), w1 = __bfloat162float(M.w2t[in + 32]);
#pragma unroll
            for (int q = 0; q < SCORE_N; ++q) {
                const float x = __shfl_sync(FULL, h[q][v], k);
                acc[q][0] += w0 * x;
                acc[q][1] += w1 * x;
            }
        }
#pragma unroll
    for (int q = 0; q < SCORE_N; ++q) {
#pragma unroll
        for (int u = 0; u < 2; ++u) h[q][u] = bf16r(fmaxf(acc[q][u] + M.b2[lane + 32 * u], 0.0f));
        z[q] = 0.0f;
    }
#pragma unroll
    for (int v = 0; v < 2; ++v)
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
            const float w = __bfloat162float(M.w3[k + 32 * v]);
#pragma unroll
            for (int q = 0; q < SCORE_N; ++q) z[q] += w * __shfl_sync(FULL, h[q][v], k);
        }
#pragma unroll
    for (int q = 0; q < SCORE_N; ++q) z[q] += M.b3;
}

}  // namespace ltlg
