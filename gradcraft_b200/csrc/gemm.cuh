// Shared argument block and engine entry points of the two GEMM engines.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace gcb {

struct GemmArgs {
    int64_t M, N, K;
    float alpha, beta;
    const float *A, *B, *bias;
    float* C;
    int64_t lda, ldb, ldc;
    int64_t a_so, a_si, b_so, b_si, c_so, c_si;  // batch strides (outer, inner) in elements
    int64_t batch_outer, batch_inner;
    int causal = 0;  // 0 none; 1 output needed on/below the diagonal only; 2 op(A)[m,k] = 0 for k > m; 3 op(A)[m,k] = 0 for k < m
    // softmax-backward epilogue (needs causal == 1): C[m,n] = sm_scale * sm_probs[m,n] * (alpha * (op(A) op(B))[m,n] - sm_rowdot[m]) for n <= m, 0 for n > m.
    // sm_probs is laid out like C; sm_rowdot holds M values per batch item, batch items in (outer, inner) order.
    // GELU-backward epilogue (needs beta == 0): C[m,n] = (alpha * (op(A) op(B))[m,n] + bias[n]) * gelu'(gelu_pre[m,n]); gelu_pre is laid out like C
    const float* gelu_pre = nullptr;
    // GELU-forward epilogue: besides C, gelu(C[m,n]) is written to gelu_act, laid out like C
    float* gelu_act = nullptr;
    // residual epilogue (needs beta == 0, no GELU epilogue, unbatched): C[m,n] = alpha * (op(A) op(B))[m,n] + bias[n] + residual[m,n]; residual is laid out
    // like C and must not alias it
    const float* residual = nullptr;
    const float* sm_probs = nullptr;
    const float* sm_rowdot = nullptr;
    float sm_scale = 1.0f;
    // column sums of op(B) as a by-product (the bias gradient next to dW = X^T dY: op(B) = dY): colsum[n] = sum_k op(B)[k, n]
    // (+ colsum[n] when colsum_accumulate).  Unbatched problems only.
    float* colsum = nullptr;
    int colsum_accumulate = 0;
    // Several linear layers of one shape over the same input (inner batch items; batch_outer == 1, causal == 0).  grouped: bias and column
    // sums move with the item by bias_si / colsum_si, and a_si == 0 means that A is shared.  k_groups > 1 (one item, C = sum over g):
    // K is walked once per group, A and B moving by a_si / b_si.
    bool grouped = false;
    int64_t bias_si = 0, colsum_si = 0;
    int k_groups = 1;
};

// fp32 FMA engine: any shape, any leading dimension, every epilogue.
int gemm_simt_launch(gcb_ctx* ctx, bool ta, bool tb, const GemmArgs& g);
// A linear layer's two gradients in one launch of the FMA engine: dx = dY W^T (op N, T), dw = X^T dY (op T, N).
bool gemm_simt_backward_fits(const GemmArgs& dx, const GemmArgs& dw);
int gemm_simt_backward_launch(gcb_ctx* ctx, const GemmArgs& dx, const GemmArgs& dw);
// tcgen05 3xTF32 engine.  Returns GCB_UNSUPPORTED (without touching C) when the operands cannot be described
// to TMA: bases must be 16-byte aligned and every leading dimension / batch stride a multiple of 4 floats.
int gemm_tc_launch(gcb_ctx* ctx, bool ta, bool tb, const GemmArgs& g);
bool gemm_tc_eligible(const GemmArgs& g);
// cuTensorMapEncodeTiled, looked up once per context (NULL: not there).
typedef CUresult (*TmaEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
TmaEncodeFn tma_encode(gcb_ctx* ctx);

}  // namespace gcb
