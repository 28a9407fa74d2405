// Causal attention of short sequences in fp32 FMA arithmetic, one launch each way.  A head of 64 x 64 takes 3 + 6 launches through the
// product and softmax kernels, each bound by launch and latency (4 - 5 us); here a CTA owns 32 rows of a head and walks over the other
// side in tiles of 64 kept in shared memory.  Forward: 32 queries, the key tiles up to the diagonal (running maximum and sum).
// Backward: one CTA for the dQ of 32 queries and one for the dK and dV of 32 keys, each working out its blocks of P and dS itself, so
// that nothing is shared between CTAs.  16 heads of 64 x 32: 6 + 13 us, with one CTA for 64 rows of everything 7 + 17.
// Bound by latency: eight warps an SM, a shared-memory load for every four to eight FMAs.
#pragma once
#include "gemm.cuh"

namespace gcb {

constexpr int AS_OWN = 32, AS_T = 64;

struct SmallAttn {
    const float *q, *k, *v, *g, *o;
    float *out, *dq, *dk, *dv, *row_max, *row_inv;
    int64_t q_ld, q_so, q_si, k_ld, k_so, k_si, v_ld, v_so, v_si, g_ld, g_so, g_si, o_ld, o_so, o_si, d_ld, d_so, d_si, Tp;
    int T, D, H;
    float scale;
};

// ROWS rows of D columns from row r0 into [row][D + 4], asynchronously; rows beyond T are zero
template <int ROWS>
__device__ __forceinline__ void as_load(float* sm, const float* p, int64_t ld, int r0, int T, int D) {
    const int d4 = D >> 2;
    for (int i = threadIdx.x; i < ROWS * d4; i += 256) {
        const int r = i / d4, c = (i - r * d4) * 4;
        const bool live = r0 + r < T;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(sm + r * (D + 4) + c)), "l"(live ? p + (r0 + r) * ld + c : p), "r"(live ? 16 : 0) : "memory");
    }
}
__device__ __forceinline__ void as_landed() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}
// c[i][j] = a[ty + 16 i] . b[tx + 16 j]
template <int R, int C>
__device__ __forceinline__ void as_abt(float (&c)[R][C], const float* a, const float* b, int D, int ty, int tx) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) c[i][j] = 0.0f;
    const int P = D + 4;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
        float4 x[R], y[C];
#pragma unroll
        for (int i = 0; i < R; ++i) x[i] = ld4(a + (ty + 16 * i) * P + d);
#pragma unroll
        for (int j = 0; j < C; ++j) y[j] = ld4(b + (tx + 16 * j) * P + d);
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
            for (int j = 0; j < C; ++j) c[i][j] = fmaf(x[i].x, y[j].x, fmaf(x[i].y, y[j].y, fmaf(x[i].z, y[j].z, fmaf(x[i].w, y[j].w, c[i][j]))));
    }
}
// acc[i][4 n + e] += sum_k p[ty + 16 i][k] b[k][64 n + 4 tx + e], k < 64
template <int NC>
__device__ __forceinline__ void as_ab(float (&acc)[2][4 * NC], const float* p, const float* b, int D, int ty, int tx) {
    const int P = D + 4;
#pragma unroll 4
    for (int k = 0; k < AS_T; k += 4) {
        float a[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) { const float4 x = ld4(p + (ty + 16 * i) * (AS_T + 4) + k); a[i][0] = x.x; a[i][1] = x.y; a[i][2] = x.z; a[i][3] = x.w; }
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int c = 64 * n + 4 * tx;
            if (c >= D) break;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 y = ld4(b + (k + q) * P + c);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    acc[i][4 * n] = fmaf(a[i][q], y.x, acc[i][4 * n]); acc[i][4 * n + 1] = fmaf(a[i][q], y.y, acc[i][4 * n + 1]);
                    acc[i][4 * n + 2] = fmaf(a[i][q], y.z, acc[i][4 * n + 2]); acc[i][4 * n + 3] = fmaf(a[i][q], y.w, acc[i][4 * n + 3]);
                }
            }
        }
    }
}
// acc[i][4 n + e] += sum_r p[r][2 ty + i] b[r][64 n + 4 tx + e], r < 64
template <int NC>
__device__ __forceinline__ void as_atb(float (&acc)[2][4 * NC], const float* p, const float* b, int D, int ty, int tx) {
    const int P = D + 4;
#pragma unroll 8
    for (int r = 0; r < AS_T; ++r) {
        const float2 a = *reinterpret_cast<const float2*>(p + r * (AS_OWN + 4) + 2 * ty);
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int c = 64 * n + 4 * tx;
            if (c >= D) break;
            const float4 y = ld4(b + r * P + c);
            acc[0][4 * n] = fmaf(a.x, y.x, acc[0][4 * n]); acc[0][4 * n + 1] = fmaf(a.x, y.y, acc[0][4 * n + 1]);
            acc[0][4 * n + 2] = fmaf(a.x, y.z, acc[0][4 * n + 2]); acc[0][4 * n + 3] = fmaf(a.x, y.w, acc[0][4 * n + 3]);
            acc[1][4 * n] = fmaf(a.y, y.x, acc[1][4 * n]); acc[1][4 * n + 1] = fmaf(a.y, y.y, acc[1][4 * n + 1]);
            acc[1][4 * n + 2] = fmaf(a.y, y.z, acc[1][4 * n + 2]); acc[1][4 * n + 3] = fmaf(a.y, y.w, acc[1][4 * n + 3]);
        }
    }
}
__device__ __forceinline__ float as_row(float v, bool is_max) {  // over the 16 threads of a row
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) { const float w = __shfl_xor_sync(0xffffffffu, v, o); v = is_max ? fmaxf(v, w) : v + w; }
    return v;
}

// floats of shared memory: the 32-row tiles, the 64-row tiles and `blocks` blocks of scores
static size_t as_floats(int own, int other, int blocks, int64_t D) { return (size_t)(own * AS_OWN + other * AS_T) * (D + 4) + (size_t)blocks * AS_T * (AS_OWN + 4); }

template <int NC>
__global__ void __launch_bounds__(256) attention_small_fwd_kernel(const SmallAttn p) {
    extern __shared__ __align__(16) float as_sm[];
    pdl_trigger();
    pdl_wait();
    const int D = p.D, tx = threadIdx.x & 15, ty = threadIdx.x >> 4, q0 = blockIdx.y * AS_OWN, last = min(q0 + AS_OWN, p.T);
    const int64_t b = blockIdx.x / p.H, h = blockIdx.x - b * p.H;
    float *sq = as_sm, *sk = sq + AS_OWN * (D + 4), *sv = sk + AS_T * (D + 4), *sp = sv + AS_T * (D + 4);
    const float *k = p.k + b * p.k_so + h * p.k_si, *v = p.v + b * p.v_so + h * p.v_si;
    as_load<AS_OWN>(sq, p.q + b * p.q_so + h * p.q_si, p.q_ld, q0, p.T, D);
    float acc[2][4 * NC] = {}, m[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
    for (int k0 = 0; k0 < last; k0 += AS_T) {
        __syncthreads();
        as_load<AS_T>(sk, k, p.k_ld, k0, p.T, D);
        as_load<AS_T>(sv, v, p.v_ld, k0, p.T, D);
        as_landed();
        float s[2][4];
        as_abt(s, sq, sk, D, ty, tx);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int row = q0 + ty + 16 * i;
            float mx = m[i];
#pragma unroll
            for (int j = 0; j < 4; ++j) { s[i][j] = k0 + tx + 16 * j <= row ? s[i][j] * p.scale : -INFINITY; mx = fmaxf(mx, s[i][j]); }
            mx = as_row(mx, true);
            const float f = __expf(m[i] - mx);
            m[i] = mx;
            float part = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) { const float e = __expf(s[i][j] - mx); part += e; sp[(ty + 16 * i) * (AS_T + 4) + tx + 16 * j] = e; }
            sum[i] = sum[i] * f + as_row(part, false);
#pragma unroll
            for (int e = 0; e < 4 * NC; ++e) acc[i][e] *= f;
        }
        __syncthreads();
        as_ab<NC>(acc, sp, sv, D, ty, tx);
    }
    float* out = p.out + b * p.o_so + h * p.o_si;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = q0 + ty + 16 * i;
        if (row >= p.T) continue;
        const float inv = 1.0f / sum[i];
#pragma unroll
        for (int n = 0; n < NC; ++n)
            if (64 * n + 4 * tx < D) st4(out + row * p.o_ld + 64 * n + 4 * tx, make_float4(acc[i][4 * n] * inv, acc[i][4 * n + 1] * inv, acc[i][4 * n + 2] * inv, acc[i][4 * n + 3] * inv));
        if (tx == 0) { p.row_max[blockIdx.x * p.Tp + row] = m[i]; p.row_inv[blockIdx.x * p.Tp + row] = inv; }
    }
}

// dO . O and the statistics of this thread's rows ty + 16 i of a query tile (dO in shared memory, O requested before it has landed)
template <int R, int NC>
struct AsRows {
    float delta[R], m[R], inv[R];
    float4 y[R][NC];
    __device__ __forceinline__ void request(const SmallAttn& p, const float* o, int r0, int ty, int tx) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int row = r0 + ty + 16 * i;
            const bool live = row < p.T;
            m[i] = live ? p.row_max[blockIdx.x * p.Tp + row] : 0.0f;
            inv[i] = live ? p.row_inv[blockIdx.x * p.Tp + row] : 0.0f;
#pragma unroll
            for (int n = 0; n < NC; ++n) y[i][n] = live && 64 * n + 4 * tx < p.D ? ld4(o + row * p.o_ld + 64 * n + 4 * tx) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    __device__ __forceinline__ void finish(const float* sg, int D, int ty, int tx) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float d = 0.0f;
#pragma unroll
            for (int n = 0; n < NC; ++n)
                if (64 * n + 4 * tx < D) {
                    const float4 x = ld4(sg + (ty + 16 * i) * (D + 4) + 64 * n + 4 * tx);
                    d = fmaf(x.x, y[i][n].x, fmaf(x.y, y[i][n].y, fmaf(x.z, y[i][n].z, fmaf(x.w, y[i][n].w, d))));
                }
            delta[i] = as_row(d, false);
        }
    }
};

template <int NC>
__global__ void __launch_bounds__(256) attention_small_bwd_kernel(const SmallAttn p) {
    extern __shared__ __align__(16) float as_sm[];
    pdl_trigger();
    pdl_wait();
    const int D = p.D, tx = threadIdx.x & 15, ty = threadIdx.x >> 4, t0 = (blockIdx.y >> 1) * AS_OWN;
    const int64_t b = blockIdx.x / p.H, h = blockIdx.x - b * p.H, at = b * p.d_so + h * p.d_si;
    float *s0 = as_sm, *s1 = s0 + AS_OWN * (D + 4), *s2 = s1 + AS_OWN * (D + 4), *s3 = s2 + AS_T * (D + 4), *sp = s3 + AS_T * (D + 4), *ss = sp + AS_T * (AS_OWN + 4);
    const float *q = p.q + b * p.q_so + h * p.q_si, *k = p.k + b * p.k_so + h * p.k_si, *v = p.v + b * p.v_so + h * p.v_si, *g = p.g + b * p.g_so + h * p.g_si, *o = p.o + b * p.o_so + h * p.o_si;
    if (blockIdx.y & 1) {  // dQ of 32 queries: s0 = q, s1 = dO, s2 = k, s3 = v
        float dq[2][4 * NC] = {};
        AsRows<2, NC> rows;
        as_load<AS_OWN>(s0, q, p.q_ld, t0, p.T, D);
        as_load<AS_OWN>(s1, g, p.g_ld, t0, p.T, D);
        rows.request(p, o, t0, ty, tx);
        for (int k0 = 0; k0 < min(t0 + AS_OWN, p.T); k0 += AS_T) {
            __syncthreads();
            as_load<AS_T>(s2, k, p.k_ld, k0, p.T, D);
            as_load<AS_T>(s3, v, p.v_ld, k0, p.T, D);
            as_landed();
            if (k0 == 0) rows.finish(s1, D, ty, tx);
            float s[2][4], dp[2][4];
            as_abt(s, s0, s2, D, ty, tx);
            as_abt(dp, s1, s3, D, ty, tx);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float pr = k0 + tx + 16 * j <= t0 + ty + 16 * i ? __expf(s[i][j] * p.scale - rows.m[i]) * rows.inv[i] : 0.0f;
                    ss[(ty + 16 * i) * (AS_T + 4) + tx + 16 * j] = p.scale * pr * (dp[i][j] - rows.delta[i]);
                }
            __syncthreads();
            as_ab<NC>(dq, ss, s2, D, ty, tx);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                const int c = 64 * n + 4 * tx, r = t0 + ty + 16 * i;
                if (c < D && r < p.T) st4(p.dq + at + r * p.d_ld + c, make_float4(dq[i][4 * n], dq[i][4 * n + 1], dq[i][4 * n + 2], dq[i][4 * n + 3]));
            }
        return;
    }
    // dK and dV of 32 keys: s0 = k, s1 = v, s2 = q, s3 = dO
    float dk[2][4 * NC] = {}, dv[2][4 * NC] = {};
    as_load<AS_OWN>(s0, k, p.k_ld, t0, p.T, D);
    as_load<AS_OWN>(s1, v, p.v_ld, t0, p.T, D);
    for (int r0 = t0 / AS_T * AS_T; r0 < p.T; r0 += AS_T) {
        __syncthreads();
        AsRows<4, NC> rows;
        as_load<AS_T>(s2, q, p.q_ld, r0, p.T, D);
        as_load<AS_T>(s3, g, p.g_ld, r0, p.T, D);
        rows.request(p, o, r0, ty, tx);
        as_landed();
        rows.finish(s3, D, ty, tx);
        float s[4][2], dp[4][2];
        as_abt(s, s2, s0, D, ty, tx);
        as_abt(dp, s3, s1, D, ty, tx);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float pr = t0 + tx + 16 * j <= r0 + ty + 16 * i ? __expf(s[i][j] * p.scale - rows.m[i]) * rows.inv[i] : 0.0f;
                sp[(ty + 16 * i) * (AS_OWN + 4) + tx + 16 * j] = pr;
                ss[(ty + 16 * i) * (AS_OWN + 4) + tx + 16 * j] = p.scale * pr * (dp[i][j] - rows.delta[i]);
            }
        __syncthreads();
        as_atb<NC>(dv, sp, s3, D, ty, tx);
        as_atb<NC>(dk, ss, s2, D, ty, tx);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int c = 64 * n + 4 * tx, r = t0 + 2 * ty + i;
            if (c >= D || r >= p.T) continue;
            st4(p.dk + at + r * p.d_ld + c, make_float4(dk[i][4 * n], dk[i][4 * n + 1], dk[i][4 * n + 2], dk[i][4 * n + 3]));
            st4(p.dv + at + r * p.d_ld + c, make_float4(dv[i][4 * n], dv[i][4 * n + 1], dv[i][4 * n + 2], dv[i][4 * n + 3]));
        }
}

static int small_launch(gcb_ctx* ctx, void (*kernel)(const SmallAttn), bool* done, int64_t heads, int ctas, size_t floats, const SmallAttn& p) {
    if (!done[ctx->device]) { GCB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448 - 1024)); done[ctx->device] = true; }
    GCB_CHECK_CUDA(launch_next(ctx->stream, dim3((unsigned)heads, (unsigned)ctas), 256, sizeof(float) * floats, kernel, p));
    return GCB_OK;
}

}  // namespace gcb
