// GEMM entry points: argument validation and engine choice.
// Reference counterparts: CUDAMath::apply_normal_gemm / apply_batched_gemm (backend/cuda/kernels_math.cu:725-779),
// whose NMMMeta / BMMMeta fields (core/types.hpp:118-158) map one to one onto the arguments here.
#include <algorithm>

#include "gemm.cuh"

using namespace gcb;

// Products of fewer multiply-adds run on the FMA engine, fused epilogues included: it takes 3 - 8 us for them, while no tensor-core
// kernel returns in less than 12.
static constexpr int64_t kSmallWork = int64_t(1) << 26;

namespace gcb {

// out[b][r][c] = in[b][r][c] for c < cols, rows `pitch` floats apart (a multiple of four; what lies beyond cols is never read as
// an operand: the tensor maps end at cols).  Bound by memory; a block copies 1024 columns of one row per step, neighbouring
// threads neighbouring elements, because neither side's rows need start on a 16-byte boundary.
__global__ void __launch_bounds__(256) pack_rows_kernel(float* __restrict__ out, const float* __restrict__ in, int64_t rows, int64_t cols, int64_t ld, int64_t so, int64_t si, int64_t n_inner,
                                                        int64_t total_rows, int64_t pitch) {
    pdl_trigger();
    pdl_wait();
    const int64_t c0 = (int64_t)blockIdx.x * 1024 + threadIdx.x;
    for (int64_t r = blockIdx.y; r < total_rows; r += gridDim.y) {
        const int64_t item = r / rows, row = r - item * rows, bo = item / n_inner, bi = item - bo * n_inner;
        const float* src = in + bo * so + bi * si + row * ld;
        float* dst = out + r * pitch;
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = c0 + 256 * u < cols ? __ldcs(src + c0 + 256 * u) : 0.0f;
#pragma unroll
        for (int u = 0; u < 4; ++u) if (c0 + 256 * u < cols) dst[c0 + 256 * u] = v[u];
    }
}

// An operand TMA cannot address (base off a 16-byte boundary, row or batch strides no multiple of four floats) is copied into
// rows that it can address.  rows x cols as stored.
struct PackedOperand {
    Scratch sc;
    explicit PackedOperand(gcb_ctx* ctx) : sc(ctx) {}
    int pack(gcb_ctx* ctx, const float** p, int64_t* ld, int64_t* so, int64_t* si, int64_t rows, int64_t cols, int64_t n_outer, int64_t n_inner) {
        auto ok4 = [](int64_t v) { return v % 4 == 0; };
        if (aligned16(*p) && ok4(*ld) && (n_inner == 1 || ok4(*si)) && (n_outer == 1 || ok4(*so))) return GCB_OK;
        const int64_t pitch = (cols + 3) / 4 * 4, total_rows = rows * n_outer * n_inner;
        int rc = sc.get(sizeof(float) * (size_t)(total_rows * pitch));
        if (rc) return rc;
        dim3 grid((unsigned)((cols + 1023) / 1024), (unsigned)std::min<int64_t>(total_rows, 65535), 1);
        GCB_CHECK_CUDA(launch_chained(ctx->stream, grid, 256, 0, pack_rows_kernel, sc.as<float>(), *p, rows, cols, *ld, *so, *si, n_inner, total_rows, pitch));
        *p = sc.as<float>();
        *ld = pitch;
        *si = rows * pitch;
        *so = n_inner * rows * pitch;
        return after_launch(ctx, "gemm_pack");
    }
};

}  // namespace gcb

// Engine choice for one validated problem; no timing here, so the GELU fallback below may call it again freely.
static int dispatch_gemm(gcb_ctx* ctx, bool ta, bool tb, const GemmArgs& g, const char* who) {
    const int64_t work = g.M * g.N * g.K * g.batch_outer * g.batch_inner * g.k_groups;
    if (ctx->gemm_engine == 1 || (ctx->gemm_engine == 0 && work < kSmallWork)) return gemm_simt_launch(ctx, ta, tb, g);
    int rc = GCB_UNSUPPORTED;
    if (gemm_tc_eligible(g)) rc = gemm_tc_launch(ctx, ta, tb, g);
    if (rc == GCB_UNSUPPORTED && g.grouped) return rc;  // the caller takes the layers one by one
    // operands that only their addresses keep from the tensor cores are copied into rows that suit them (~3 us each)
    if (rc == GCB_UNSUPPORTED && ctx->gemm_engine == 0 && g.batch_outer * g.batch_inner <= 65535) {
        GemmArgs packed = g;
        PackedOperand pa(ctx), pb(ctx);
        rc = pa.pack(ctx, &packed.A, &packed.lda, &packed.a_so, &packed.a_si, ta ? g.K : g.M, ta ? g.M : g.K, g.batch_outer, g.batch_inner);
        if (rc == GCB_OK) rc = pb.pack(ctx, &packed.B, &packed.ldb, &packed.b_so, &packed.b_si, tb ? g.N : g.K, tb ? g.K : g.N, g.batch_outer, g.batch_inner);
        if (rc) return rc;
        rc = GCB_UNSUPPORTED;
        if (packed.A != g.A || packed.B != g.B) {
            if (gemm_tc_eligible(packed)) rc = gemm_tc_launch(ctx, ta, tb, packed);
            if (rc == GCB_UNSUPPORTED && gemm_tc_eligible(packed)) {  // an epilogue that this kernel lacks runs as a second pass, the product on the packed operands
                packed.colsum = nullptr;  // of the operand as it was: packed rows lie further apart
                rc = dispatch_gemm(ctx, ta, tb, packed, who);
                if (rc == GCB_OK && g.colsum) rc = gcb_reduce_rows_f32(ctx, g.colsum, g.B, g.K, g.N, g.colsum_accumulate);
                return rc;
            }
        }
    }
    if (rc == GCB_UNSUPPORTED && (g.gelu_pre || g.gelu_act)) {
        // no kernel with the fused GELU epilogues takes this problem: the same product, then the elementwise pass over C
        GemmArgs plain = g;
        plain.gelu_pre = nullptr;
        plain.gelu_act = nullptr;
        rc = dispatch_gemm(ctx, ta, tb, plain, who);
        if (rc == GCB_OK && g.gelu_pre) rc = gcb_gelu_bwd_f32(ctx, g.C, g.C, g.gelu_pre, g.M * g.N, 0);
        if (rc == GCB_OK && g.gelu_act) rc = gcb_gelu_fwd_f32(ctx, g.gelu_act, g.C, g.M * g.N);
        return rc;
    }
    if (rc == GCB_UNSUPPORTED && g.residual) {
        // no kernel with the residual epilogue takes this problem: the same product, then the addition as a pass of its own (same order of operations)
        GemmArgs plain = g;
        plain.residual = nullptr;
        rc = dispatch_gemm(ctx, ta, tb, plain, who);
        if (rc == GCB_OK) rc = gcb_binary_f32(ctx, GCB_B_ADD, g.C, g.C, g.residual, g.M * g.N);
        return rc;
    }
    if (rc == GCB_UNSUPPORTED && g.colsum) {
        // no kernel gathers the column sums of op(B) for this problem: the same product, then the row reduction as a pass of its own
        GemmArgs plain = g;
        plain.colsum = nullptr;
        rc = dispatch_gemm(ctx, ta, tb, plain, who);
        if (rc != GCB_OK) return rc;
        if (!tb && g.ldb == g.N) return gcb_reduce_rows_f32(ctx, g.colsum, g.B, g.K, g.N, g.colsum_accumulate);
        set_error("%s: column sums need op(B) stored K x N with ldb == N", who);
        return GCB_UNSUPPORTED;
    }
    if (rc == GCB_UNSUPPORTED) {
        if (ctx->gemm_engine == 2) {
            set_error("%s: the tcgen05 engine was forced but cannot take these operands (alignment / leading dimensions)", who);
            return GCB_UNSUPPORTED;
        }
        rc = gemm_simt_launch(ctx, ta, tb, g);
    }
    return rc;
}

// A dispatch bracketed by one pair of timing events when profiling is on: it is counted once whatever path it takes, and the closing
// event is recorded on every exit so that gcb_profile_gemm_end never meets an unrecorded event.
template <class F>
static int profiled(gcb_ctx* ctx, double flops, F&& dispatch) {
    if (!ctx->prof_on) return dispatch();
    if (ctx->prof_used + 2 > ctx->prof_events.size()) {
        for (int i = 0; i < 512; ++i) { cudaEvent_t e; GCB_CHECK_CUDA(cudaEventCreate(&e)); ctx->prof_events.push_back(e); }
    }
    cudaEvent_t e0 = ctx->prof_events[ctx->prof_used], e1 = ctx->prof_events[ctx->prof_used + 1];
    GCB_CHECK_CUDA(cudaEventRecord(e0, ctx->stream));
    const int rc = dispatch();
    GCB_CHECK_CUDA(cudaEventRecord(e1, ctx->stream));
    if (rc == GCB_OK) {  // a refused problem leaves no trace in the tally
        ctx->prof_used += 2;
        ctx->prof_flops += flops;
    }
    return rc;
}

static int run_gemm(gcb_ctx* ctx, int op_a, int op_b, const GemmArgs& g, const char* who) {
    GCB_REQUIRE((op_a == GCB_OP_N || op_a == GCB_OP_T) && (op_b == GCB_OP_N || op_b == GCB_OP_T), "%s: op must be GCB_OP_N or GCB_OP_T", who);
    GCB_REQUIRE(g.M >= 0 && g.N >= 0 && g.K >= 0, "%s: negative dimension", who);
    if (g.M == 0 || g.N == 0 || g.batch_outer * g.batch_inner == 0) return GCB_OK;
    GCB_REQUIRE(g.C && (g.K == 0 || (g.A && g.B)), "%s: NULL operand", who);
    const bool ta = op_a == GCB_OP_T, tb = op_b == GCB_OP_T;
    GCB_REQUIRE(g.lda >= (ta ? g.M : g.K) && g.ldb >= (tb ? g.K : g.N) && g.ldc >= g.N, "%s: leading dimension smaller than the row length (lda %lld ldb %lld ldc %lld)", who,
                (long long)g.lda, (long long)g.ldb, (long long)g.ldc);
    return profiled(ctx, 2.0 * (double)g.M * (double)g.N * (double)g.K * (double)(g.batch_outer * g.batch_inner * g.k_groups), [&] { return dispatch_gemm(ctx, ta, tb, g, who); });
}

extern "C" {

int gcb_gemm_f32(gcb_ctx* ctx, int op_a, int op_b, int64_t M, int64_t N, int64_t K, float alpha, const float* A, int64_t lda, const float* B, int64_t ldb, float beta, float* C,
                 int64_t ldc, const float* bias) {
    GCB_REQUIRE(ctx, "gcb_gemm_f32: ctx is NULL");
    GemmArgs g{M, N, K, alpha, beta, A, B, bias, C, lda, ldb, ldc, 0, 0, 0, 0, 0, 0, 1, 1};
    return run_gemm(ctx, op_a, op_b, g, "gcb_gemm_f32");
}

int gcb_gemm_colsum_f32(gcb_ctx* ctx, int op_a, int64_t M, int64_t N, int64_t K, float alpha, const float* A, int64_t lda, const float* B, float beta, float* C, int64_t ldc, float* colsum,
                        int colsum_accumulate) {
    GCB_REQUIRE(ctx, "gcb_gemm_colsum_f32: ctx is NULL");
    GCB_REQUIRE(N == 0 || colsum, "gcb_gemm_colsum_f32: colsum is NULL");
    if (K == 0 && N > 0 && !colsum_accumulate) { int rc = gcb_fill_f32(ctx, colsum, 0.0f, N); if (rc) return rc; }
    GemmArgs g{M, N, K, alpha, beta, A, B, nullptr, C, lda, N, ldc, 0, 0, 0, 0, 0, 0, 1, 1};
    g.colsum = colsum;
    g.colsum_accumulate = colsum_accumulate;
    if (M == 0 && N > 0 && K > 0) return gcb_reduce_rows_f32(ctx, colsum, B, K, N, colsum_accumulate);  // no product, but the sums are still owed
    return run_gemm(ctx, op_a, GCB_OP_N, g, "gcb_gemm_colsum_f32");
}

int gcb_gemm_batched_f32(gcb_ctx* ctx, int op_a, int op_b, int64_t M, int64_t N, int64_t K, float alpha, const float* A, int64_t lda, int64_t a_so, int64_t a_si, const float* B,
                         int64_t ldb, int64_t b_so, int64_t b_si, float beta, float* C, int64_t ldc, int64_t c_so, int64_t c_si, int64_t batch_outer, int64_t batch_inner) {
    GCB_REQUIRE(ctx, "gcb_gemm_batched_f32: ctx is NULL");
    GCB_REQUIRE(batch_outer >= 0 && batch_inner >= 0, "gcb_gemm_batched_f32: negative batch count");
    GemmArgs g{M, N, K, alpha, beta, A, B, nullptr, C, lda, ldb, ldc, a_so, a_si, b_so, b_si, c_so, c_si, batch_outer, batch_inner};
    return run_gemm(ctx, op_a, op_b, g, "gcb_gemm_batched_f32");
}

int gcb_gemm_batched_causal_f32(gcb_ctx* ctx, int op_a, int op_b, int64_t M, int64_t N, int64_t K, float alpha, const float* A, int64_t lda, int64_t a_so, int64_t a_si, const float* B,
                                int64_t ldb, int64_t b_so, int64_t b_si, float beta, float* C, int64_t ldc, int64_t c_so, int64_t c_si, int64_t batch_outer, int64_t batch_inner, int causal) {
    GCB_REQUIRE(ctx, "gcb_gemm_batched_causal_f32: ctx is NULL");
    GCB_REQUIRE(batch_outer >= 0 && batch_inner >= 0, "gcb_gemm_batched_causal_f32: negative batch count");
    GCB_REQUIRE(causal >= 0 && causal <= 3, "gcb_gemm_batched_causal_f32: causal must be 0..3");
    GCB_REQUIRE(causal != 1 || M == N, "gcb_gemm_batched_causal_f32: a triangular output needs M == N");
    GCB_REQUIRE(causal < 2 || M == K, "gcb_gemm_batched_causal_f32: a triangular op(A) needs M == K");
    GemmArgs g{M, N, K, alpha, beta, A, B, nullptr, C, lda, ldb, ldc, a_so, a_si, b_so, b_si, c_so, c_si, batch_outer, batch_inner};
    g.causal = causal;
    return run_gemm(ctx, op_a, op_b, g, "gcb_gemm_batched_causal_f32");
}

int gcb_gemm_batched_softmax_bwd_f32(gcb_ctx* ctx, int op_a, int op_b, int64_t M, int64_t K, float alpha, const float* A, int64_t lda, int64_t a_so, int64_t a_si, const float* B, int64_t ldb,
                                     int64_t b_so, int64_t b_si, float* dscores, int64_t ldc, int64_t c_so, int64_t c_si, int64_t batch_outer, int64_t batch_inner, const float* probs,
                                     const float* row_dot, float scale) {
    GCB_REQUIRE(ctx, "gcb_gemm_batched_softmax_bwd_f32: ctx is NULL");
    GCB_REQUIRE(batch_outer >= 0 && batch_inner >= 0, "gcb_gemm_batched_softmax_bwd_f32: negative batch count");
    GCB_REQUIRE(M == 0 || batch_outer * batch_inner == 0 || (probs && row_dot), "gcb_gemm_batched_softmax_bwd_f32: NULL probs / row_dot");
    GCB_REQUIRE(probs != dscores, "gcb_gemm_batched_softmax_bwd_f32: dscores must not alias probs");
    GemmArgs g{M, M, K, alpha, 0.0f, A, B, nullptr, dscores, lda, ldb, ldc, a_so, a_si, b_so, b_si, c_so, c_si, batch_outer, batch_inner};
    g.causal = 1;
    g.sm_probs = probs; g.sm_rowdot = row_dot; g.sm_scale = scale;
    return run_gemm(ctx, op_a, op_b, g, "gcb_gemm_batched_softmax_bwd_f32");
}

int gcb_gemm_gelu_bwd_f32(gcb_ctx* ctx, int op_a, int op_b, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda, const float* B, int64_t ldb, const float* pre, float* dpre) {
    GCB_REQUIRE(ctx, "gcb_gemm_gelu_bwd_f32: ctx is NULL");
    GCB_REQUIRE(M == 0 || N == 0 || (pre && dpre), "gcb_gemm_gelu_bwd_f32: NULL pre / dpre");
    GCB_REQUIRE(pre != dpre, "gcb_gemm_gelu_bwd_f32: dpre must not alias pre");
    GemmArgs g{M, N, K, 1.0f, 0.0f, A, B, nullptr, dpre, lda, ldb, N, 0, 0, 0, 0, 0, 0, 1, 1};
    g.gelu_pre = pre;
    return run_gemm(ctx, op_a, op_b, g, "gcb_gemm_gelu_bwd_f32");
}

int gcb_linear_gelu_fwd_f32(gcb_ctx* ctx, int op_b, int64_t M, int64_t N, int64_t K, const float* x, int64_t lda, const float* W, int64_t ldb, const float* bias, float* pre, float* act) {
    GCB_REQUIRE(ctx, "gcb_linear_gelu_fwd_f32: ctx is NULL");
    GCB_REQUIRE(M == 0 || N == 0 || (pre && act), "gcb_linear_gelu_fwd_f32: NULL pre / act");
    GCB_REQUIRE(pre != act, "gcb_linear_gelu_fwd_f32: act must not alias pre");
    GemmArgs g{M, N, K, 1.0f, 0.0f, x, W, bias, pre, lda, ldb, N, 0, 0, 0, 0, 0, 0, 1, 1};
    g.gelu_act = act;
    return run_gemm(ctx, GCB_OP_N, op_b, g, "gcb_linear_gelu_fwd_f32");
}

int gcb_linear_residual_f32(gcb_ctx* ctx, int op_b, int64_t M, int64_t N, int64_t K, const float* x, int64_t lda, const float* W, int64_t ldb, const float* bias, const float* residual, float* out) {
    GCB_REQUIRE(ctx, "gcb_linear_residual_f32: ctx is NULL");
    GCB_REQUIRE(M == 0 || N == 0 || (residual && out), "gcb_linear_residual_f32: NULL residual / out");
    GCB_REQUIRE(residual != out, "gcb_linear_residual_f32: out must not alias residual");
    GemmArgs g{M, N, K, 1.0f, 0.0f, x, W, bias, out, lda, ldb, N, 0, 0, 0, 0, 0, 0, 1, 1};
    g.residual = residual;
    return run_gemm(ctx, GCB_OP_N, op_b, g, "gcb_linear_residual_f32");
}

// Linear layers of one shape over one input in one launch each way (q, k and v; the two halves of a SwiGLU).  A layer by itself leaves
// the last round of tiles nearly empty and small ones are bound by launches: 4096 x 768 x 768 is 48 pair tiles on 74 pairs, three
// layers are 144 on two full rounds.
int gcb_linear_group_f32(gcb_ctx* ctx, int64_t groups, int64_t M, int64_t N, int64_t K, const float* x, const float* W, int64_t w_stride, const float* bias, int64_t bias_stride, float* y, int64_t y_stride) {
    GCB_REQUIRE(ctx && groups >= 1 && groups <= 64, "gcb_linear_group_f32: bad arguments");
    GemmArgs g{M, N, K, 1.0f, 0.0f, x, W, bias, y, K, N, N, 0, 0, 0, w_stride, 0, y_stride, 1, groups};
    g.grouped = true;
    g.bias_si = bias_stride;
    int rc = run_gemm(ctx, GCB_OP_N, GCB_OP_N, g, "gcb_linear_group_f32");
    if (rc == GCB_UNSUPPORTED)
        for (int64_t i = 0; i < groups; ++i) {
            rc = gcb_gemm_f32(ctx, GCB_OP_N, GCB_OP_N, M, N, K, 1.0f, x, K, W + i * w_stride, N, 0.0f, y + i * y_stride, N, bias ? bias + i * bias_stride : nullptr);
            if (rc) return rc;
        }
    return rc;
}

int gcb_linear_group_dx_f32(gcb_ctx* ctx, int64_t groups, int64_t M, int64_t N, int64_t K, const float* dy, int64_t dy_stride, const float* W, int64_t w_stride, float beta, float* dx) {
    GCB_REQUIRE(ctx && groups >= 1 && groups <= 64, "gcb_linear_group_dx_f32: bad arguments");
    GemmArgs g{M, K, N, 1.0f, beta, dy, W, nullptr, dx, N, N, K, 0, dy_stride, 0, w_stride, 0, 0, 1, 1};
    g.grouped = true;
    g.k_groups = (int)groups;
    int rc = dy_stride > 0 && dy_stride % 4 == 0 && w_stride > 0 && w_stride % 4 == 0 ? run_gemm(ctx, GCB_OP_N, GCB_OP_T, g, "gcb_linear_group_dx_f32") : GCB_UNSUPPORTED;
    if (rc == GCB_UNSUPPORTED)
        for (int64_t i = 0; i < groups; ++i) {
            rc = gcb_gemm_f32(ctx, GCB_OP_N, GCB_OP_T, M, K, N, 1.0f, dy + i * dy_stride, N, W + i * w_stride, N, i ? 1.0f : beta, dx, K, nullptr);
            if (rc) return rc;
        }
    return rc;
}

int gcb_linear_group_dw_f32(gcb_ctx* ctx, int64_t groups, int64_t M, int64_t N, int64_t K, const float* x, const float* dy, int64_t dy_stride, float beta, float* dW, int64_t w_stride, float* dbias,
                            int64_t bias_stride, int bias_accumulate) {
    GCB_REQUIRE(ctx && groups >= 1 && groups <= 64 && (N == 0 || dbias), "gcb_linear_group_dw_f32: bad arguments");
    GemmArgs g{K, N, M, 1.0f, beta, x, dy, nullptr, dW, K, N, N, 0, 0, 0, dy_stride, 0, w_stride, 1, groups};
    g.grouped = true;
    g.colsum = dbias;
    g.colsum_si = bias_stride;
    g.colsum_accumulate = bias_accumulate;
    int rc = M > 0 && K > 0 ? run_gemm(ctx, GCB_OP_T, GCB_OP_N, g, "gcb_linear_group_dw_f32") : GCB_UNSUPPORTED;
    if (rc == GCB_UNSUPPORTED)
        for (int64_t i = 0; i < groups; ++i) {
            rc = gcb_gemm_colsum_f32(ctx, GCB_OP_T, K, N, M, 1.0f, x, K, dy + i * dy_stride, beta, dW + i * w_stride, N, dbias + i * bias_stride, bias_accumulate);
            if (rc) return rc;
        }
    return rc;
}

int gcb_linear_group_bwd_f32(gcb_ctx* ctx, int64_t groups, int64_t M, int64_t N, int64_t K, const float* x, const float* dy, int64_t dy_stride, const float* W, int64_t w_stride, const float* gelu_pre, float dx_beta,
                             float* dx, float dw_beta, float* dW, int64_t dw_stride, float* dbias, int64_t bias_stride, int bias_accumulate) {
    GCB_REQUIRE(ctx && groups >= 1 && groups <= 64 && (M == 0 || K == 0 || dx) && (N == 0 || dbias), "gcb_linear_group_bwd_f32: bad arguments");
    GCB_REQUIRE(gelu_pre == nullptr || (groups == 1 && dx_beta == 0.0f && gelu_pre != dx), "gcb_linear_group_bwd_f32: a GELU behind the input takes one layer and overwrites its gradient");
    const int64_t work = M * N * K * groups;
    if (work > 0 && (ctx->gemm_engine == 1 || (ctx->gemm_engine == 0 && work < kSmallWork)) && x && dy && W && dW && (groups == 1 || (dy_stride >= M * N && w_stride > 0))) {
        GemmArgs gx{M, K, N, 1.0f, dx_beta, dy, W, nullptr, dx, N, N, K, 0, dy_stride, 0, w_stride, 0, 0, 1, 1};
        gx.gelu_pre = gelu_pre;
        gx.k_groups = (int)groups;
        GemmArgs gw{K, N, M, 1.0f, dw_beta, x, dy, nullptr, dW, K, N, N, 0, 0, 0, dy_stride, 0, dw_stride, 1, groups};
        gw.grouped = gx.grouped = true;
        gw.colsum = dbias; gw.colsum_si = bias_stride; gw.colsum_accumulate = bias_accumulate;
        if (gemm_simt_backward_fits(gx, gw)) return profiled(ctx, 4.0 * (double)work, [&] { return gemm_simt_backward_launch(ctx, gx, gw); });
    }
    int rc = gelu_pre ? gcb_gemm_gelu_bwd_f32(ctx, GCB_OP_N, GCB_OP_T, M, K, N, dy, N, W, N, gelu_pre, dx)
             : groups == 1 ? gcb_gemm_f32(ctx, GCB_OP_N, GCB_OP_T, M, K, N, 1.0f, dy, N, W, N, dx_beta, dx, K, nullptr)
                           : gcb_linear_group_dx_f32(ctx, groups, M, N, K, dy, dy_stride, W, w_stride, dx_beta, dx);
    if (rc) return rc;
    return groups == 1 ? gcb_gemm_colsum_f32(ctx, GCB_OP_T, K, N, M, 1.0f, x, K, dy, dw_beta, dW, N, dbias, bias_accumulate)
                       : gcb_linear_group_dw_f32(ctx, groups, M, N, K, x, dy, dy_stride, dw_beta, dW, dw_stride, dbias, bias_stride, bias_accumulate);
}

int gcb_profile_gemm_begin(gcb_ctx* ctx) {
    GCB_REQUIRE(ctx, "gcb_profile_gemm_begin: ctx is NULL");
    ctx->prof_on = true;
    ctx->prof_used = 0;
    ctx->prof_flops = 0.0;
    return GCB_OK;
}

int gcb_profile_gemm_end(gcb_ctx* ctx, int64_t* launches, double* total_ms, double* total_flops) {
    GCB_REQUIRE(ctx, "gcb_profile_gemm_end: ctx is NULL");
    ctx->prof_on = false;
    GCB_CHECK_CUDA(cudaStreamSynchronize(ctx->stream));
    double ms = 0.0;
    for (size_t i = 0; i + 1 < ctx->prof_used; i += 2) {
        float t = 0.0f;
        GCB_CHECK_CUDA(cudaEventElapsedTime(&t, ctx->prof_events[i], ctx->prof_events[i + 1]));
        ms += t;
    }
    if (launches) *launches = (int64_t)(ctx->prof_used / 2);
    if (total_ms) *total_ms = ms;
    if (total_flops) *total_flops = ctx->prof_flops;
    return GCB_OK;
}

}  // extern "C"
