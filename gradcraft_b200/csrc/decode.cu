// Incremental decoding of a GPT: one persistent kernel takes a few sequences through any number of positions, keeping the keys
// and values of earlier positions in a cache.
// Reference counterpart: GPTGenerator::run_inference (nn/generators/gpt_generator.hpp:12-132), which forwards the whole context
// again for every new token.
//
// What bounds a position is reading the weights once (743 MB for the 180M-parameter model: 0.11 ms at the copy rate); the
// arithmetic is a matrix-vector product per weight.  As separate launches a position is ~85 dependent kernels of 2 - 4 us each,
// so the whole model runs inside one cooperative kernel, one CTA per SM: five phases per layer (q/k/v, attention, output
// projection, first and second half of the MLP), a grid barrier after each (~1.3 us), then the tied head with its arg-max, whose
// result is the next position's input without a trip to the host.
//   * Products: a CTA owns tiles of eight output columns, i.e. one 32-byte sector of every weight row.  Two lanes take a row's
//     sector, sixteen rows per warp load, 256 rows per CTA; lane and warp sums are combined by shuffles and shared memory in a
//     fixed order.  N = 1024 columns give 128 tiles for 148 SMs, which wider tiles would not.
//   * Such reads gather from DRAM pages in an order that suits nobody, so every phase first asks for the NEXT phase's weights
//     with bulk L2 prefetches, each CTA a contiguous stretch: DRAM streams without a break across the barriers and the tiles
//     are read from L2.
//   * Attention: a unit is one head of one sequence and a stretch of at least 64 positions, so that few heads still fill the
//     chip; the output projection merges the stretches while it loads them.
// Everything is fp32 FMA.  Waits at the grid barrier are bounded: one that runs out reports through the status word and the
// kernel returns.
#include <algorithm>

#include "common.cuh"

namespace gcb {

constexpr int kDecThreads = 512, kDecWarps = kDecThreads / 32;
constexpr int kDecMaxLayers = 48, kDecMaxHead = 128;
constexpr int kDecSplit = 64;  // positions from which a second unit pays for one head: four per warp

struct DecodeParams {
    gcb_gpt_layer layers[kDecMaxLayers];
    const float *token_embed, *pos_embed, *final_gamma, *final_beta;
    float* cache;      // [layer][key, value][sequence][position][C]
    int64_t seq_stride, kv_stride, layer_stride;  // of the cache, in elements
    int64_t* tokens;   // [sequence][tokens_ld]
    int64_t tokens_ld;
    float *x, *q, *part, *h;  // exchange between CTAs: residual stream, queries, attention stretches, hidden activations
    float2* cand;             // [CTA][S]: best logit and its token
    float* logits;            // [sequence][V] or NULL
    unsigned* barrier;
    int* status;
    float eps, scale;
    int n_seq, pos0, n_pos, n_known;
    int V, C, H, D, L, F, gated, vec;
};

__device__ __forceinline__ void l2_prefetch(const float* p, int64_t n) {  // this CTA's stretch of p[0 .. n)
    const int64_t bytes = n * 4, share = ((bytes + gridDim.x - 1) / gridDim.x + 4095) & ~int64_t(4095);
    const int64_t b0 = share * blockIdx.x, b1 = min(bytes & ~int64_t(15), b0 + share);
    for (int64_t b = b0 + 4096 * (int64_t)threadIdx.x; b < b1; b += 4096 * (int64_t)kDecThreads)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const char*>(p) + b), "r"((uint32_t)min((int64_t)4096, b1 - b)));
}

// All CTAs of the grid meet; false when the wait ran out (every thread of the CTA gets the same answer).
__device__ __forceinline__ bool grid_barrier(unsigned* counter, unsigned target, int* status, int* flag) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
        int ok = 0;
        for (unsigned i = 0; i < (1u << 22); ++i) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            if ((int)(v - target) >= 0) { ok = 1; break; }
        }
        if (!ok) { atomicExch(&status[0], 1); atomicExch(&status[1], 120); }
        *flag = ok;
    }
    __syncthreads();
    return *flag != 0;
}

// acc[w][s][e] = this thread's share of sum_k act[k][s] * W_w[k][n + e], e = 0..3, n = n0 + 4 * (lane & 1)
template <int S, int NW>
__device__ __forceinline__ void tile_dot(const float* const (&W)[NW], int n0, int N, int K, int vec, const float* act, float (&acc)[NW][S][4]) {
    constexpr int U = NW == 2 ? 2 : 4;  // weight loads in flight per thread and matrix
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = n0 + 4 * (lane & 1);
#pragma unroll
    for (int w = 0; w < NW; ++w)
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[w][s][e] = 0.0f;
    for (int k0 = warp * 16 + (lane >> 1); k0 < K; k0 += 16 * kDecWarps * U) {
        float4 v[U][NW];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + 16 * kDecWarps * u;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                v[u][w] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (k >= K) continue;
                const float* src = W[w] + (int64_t)k * N + n;
                if (vec && n + 4 <= N) v[u][w] = __ldg(reinterpret_cast<const float4*>(src));
                else {
                    if (n + 0 < N) v[u][w].x = __ldg(src);
                    if (n + 1 < N) v[u][w].y = __ldg(src + 1);
                    if (n + 2 < N) v[u][w].z = __ldg(src + 2);
                    if (n + 3 < N) v[u][w].w = __ldg(src + 3);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = min(k0 + 16 * kDecWarps * u, K - 1);  // beyond K the weights read as zero
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float a = act[k * S + s];
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    acc[w][s][0] = fmaf(a, v[u][w].x, acc[w][s][0]); acc[w][s][1] = fmaf(a, v[u][w].y, acc[w][s][1]);
                    acc[w][s][2] = fmaf(a, v[u][w].z, acc[w][s][2]); acc[w][s][3] = fmaf(a, v[u][w].w, acc[w][s][3]);
                }
            }
        }
    }
}

template <int S>
struct DecSmem {
    // floats: x [S][C], activations [max(C, F)][S] (the head: [S][C]), then the fixed part
    static constexpr int RED = 2 * kDecWarps * 2 * S * 8;                      // two buffers of warp sums, up to two matrices
    static constexpr int ATT = kDecWarps * (kDecMaxHead + 2);                  // a warp's stretch: sum of values, maximum, sum of weights
    static constexpr int FIXED = RED + ATT + 2 * S + 2 * kDecWarps * S + S + 4;  // + statistics, head candidates, tokens, flag
    static size_t bytes(int64_t C, int64_t F) { return sizeof(float) * (size_t)((S * C + 3) / 4 * 4 + (S * std::max(C, F) + 3) / 4 * 4 + FIXED); }
};

template <int S>
__global__ void __launch_bounds__(kDecThreads, 1) gpt_decode_kernel(const __grid_constant__ DecodeParams p) {
    extern __shared__ __align__(16) float dsm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = p.C, D = p.D, F = p.F, H = p.H;
    float* xs = dsm;
    float* act = xs + (S * C + 3) / 4 * 4;
    float* red = act + (S * max(C, F) + 3) / 4 * 4;
    float* att = red + DecSmem<S>::RED;
    float* stat = att + DecSmem<S>::ATT;
    float2* best = reinterpret_cast<float2*>(stat + 2 * S);
    int* tok = reinterpret_cast<int*>(best + kDecWarps * S);
    int* flag = tok + S;
    unsigned target = 0;
    int buf = 0;
    const float inv_c = 1.0f / (float)C;

    // act <- the normalised rows of xs: [k][s] for the products, [s][k] for the head
    auto normalise = [&](const float* gamma, const float* beta, bool by_row) {
        if (warp < S) {
            const float* r = xs + warp * C;
            float s = 0.0f;
            for (int c = lane; c < C; c += 32) s += beta ? r[c] : r[c] * r[c];
            s = warp_sum(s);
            float mu = 0.0f, rs;
            if (beta) {
                mu = s * inv_c;
                float q = 0.0f;
                for (int c = lane; c < C; c += 32) { const float d = r[c] - mu; q = fmaf(d, d, q); }
                q = warp_sum(q);
                rs = 1.0f / sqrtf(q * inv_c + p.eps);
            } else {
                rs = 1.0f / sqrtf(s * inv_c + p.eps);
            }
            if (lane == 0) { stat[2 * warp] = mu; stat[2 * warp + 1] = rs; }
        }
        __syncthreads();
        for (int c = tid; c < C; c += kDecThreads) {
            const float g = __ldg(gamma + c), b = beta ? __ldg(beta + c) : 0.0f;
#pragma unroll
            for (int s = 0; s < S; ++s) act[by_row ? s * C + c : c * S + s] = (xs[s * C + c] - stat[2 * s]) * stat[2 * s + 1] * g + b;
        }
        __syncthreads();
    };
    auto load_x = [&] {  // the residual stream as the other CTAs left it
        for (int i = tid; i < S * C; i += kDecThreads) xs[i] = __ldcg(p.x + i);
        __syncthreads();
    };
    // adds up a tile's warp sums; f(s, column, sum of the first matrix, of the second) on one thread per result
    auto finish_tile = [&](auto& acc, int n0, int N, auto&& f) {
        constexpr int NW = sizeof(acc) / sizeof(acc[0]);
        float* rb = red + (buf & 1) * (kDecWarps * 2 * S * 8);
        ++buf;
#pragma unroll
        for (int w = 0; w < NW; ++w)
#pragma unroll
            for (int s = 0; s < S; ++s)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float v = acc[w][s][e];
#pragma unroll
                    for (int o = 2; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                    if (lane < 2) rb[(warp * NW + w) * S * 8 + s * 8 + 4 * lane + e] = v;
                }
        __syncthreads();
        if (tid < S * 8) {
            float v[2] = {0.0f, 0.0f};
#pragma unroll
            for (int w = 0; w < NW; ++w)
#pragma unroll
                for (int j = 0; j < kDecWarps; ++j) v[w] += rb[(j * NW + w) * S * 8 + tid];
            const int s = tid >> 3, n = n0 + (tid & 7);
            if (n < N && s < p.n_seq) f(s, n, v[0], v[1]);
        }
    };

    auto given_token = [&](int pos) {  // an id outside the vocabulary is reported, not dereferenced
        if (tid < S) {
            int64_t t = tid < p.n_seq ? p.tokens[tid * p.tokens_ld + pos] : 0;
            if (t < 0 || t >= p.V) { atomicExch(&p.status[0], 2); atomicExch(&p.status[1], pos); t = 0; }
            tok[tid] = (int)t;
        }
        __syncthreads();
    };
    given_token(p.pos0);
    const int tiles_c = (C + 7) / 8, tiles_f = (F + 7) / 8;

    for (int pos = p.pos0; pos < p.pos0 + p.n_pos; ++pos) {
        for (int l = 0; l < p.L; ++l) {
            const gcb_gpt_layer& w = p.layers[l];
            float* kc = p.cache + l * p.layer_stride;
            float* vc = kc + p.kv_stride;
            // ---- q, k, v of this position; keys and values go into the cache
            if (p.vec) {
                l2_prefetch(w.wo, (int64_t)C * C);
                for (int s = 0; s < p.n_seq; ++s) { l2_prefetch(kc + s * p.seq_stride, (int64_t)pos * C); l2_prefetch(vc + s * p.seq_stride, (int64_t)pos * C); }
            }
            if (l == 0) {
                for (int i = tid; i < S * C; i += kDecThreads) { const int s = i / C, c = i - s * C; xs[i] = __ldg(p.token_embed + (int64_t)tok[s] * C + c) + __ldg(p.pos_embed + (int64_t)pos * C + c); }
                __syncthreads();
            } else {
                load_x();
            }
            normalise(w.norm1_gamma, w.norm1_beta, false);
            for (int t = blockIdx.x; t < 3 * tiles_c; t += gridDim.x) {
                const int which = t / tiles_c, n0 = (t - which * tiles_c) * 8;
                const float* const W[1] = {which == 0 ? w.wq : which == 1 ? w.wk : w.wv};
                const float* bias = which == 0 ? w.bq : which == 1 ? w.bk : w.bv;
                float acc[1][S][4];
                tile_dot<S, 1>(W, n0, C, C, p.vec, act, acc);
                finish_tile(acc, n0, C, [&](int s, int n, float v, float) {
                    v += bias[n];
                    if (which == 0) __stcg(p.q + s * C + n, v);
                    else __stcg((which == 1 ? kc : vc) + s * p.seq_stride + (int64_t)pos * C + n, v);
                });
            }
            if (!grid_barrier(p.barrier, target += gridDim.x, p.status, flag)) return;
            // ---- attention over the positions so far, in stretches
            if (p.vec) {
                l2_prefetch(w.w1, (int64_t)C * F);
                if (p.gated) l2_prefetch(w.w2, (int64_t)C * F);
            }
            const int len = pos + 1, heads = p.n_seq * H;
            const int most = max(1, (int)gridDim.x / heads), per = max(kDecSplit, (len + most - 1) / most), nsplit = (len + per - 1) / per;
            for (int u = blockIdx.x; u < heads * nsplit; u += gridDim.x) {
                const int sh = u / nsplit, s = sh / H, h = sh - s * H, j0 = (u - sh * nsplit) * per, j1 = min(len, j0 + per);
                const float* kb = kc + s * p.seq_stride + h * D;
                const float* vb = vc + s * p.seq_stride + h * D;
                constexpr int DI = kDecMaxHead / 32;
                float q[DI], o[DI], m = -INFINITY, sum = 0.0f;
#pragma unroll
                for (int i = 0; i < DI; ++i) { q[i] = lane + 32 * i < D ? __ldcg(p.q + s * C + h * D + lane + 32 * i) * p.scale : 0.0f; o[i] = 0.0f; }
                for (int j = j0 + warp; j < j1; j += 4 * kDecWarps) {
                    float kk[4][DI], vv[4][DI], z[4];
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const int64_t row = (int64_t)(j + g * kDecWarps) * C;
                        const bool live = j + g * kDecWarps < j1;
#pragma unroll
                        for (int i = 0; i < DI; ++i) {
                            const bool in = live && lane + 32 * i < D;
                            kk[g][i] = in ? __ldcg(kb + row + lane + 32 * i) : 0.0f;
                            vv[g][i] = in ? __ldcg(vb + row + lane + 32 * i) : 0.0f;
                        }
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        float d = 0.0f;
#pragma unroll
                        for (int i = 0; i < DI; ++i) d = fmaf(q[i], kk[g][i], d);
                        d = warp_sum(d);
                        z[g] = j + g * kDecWarps < j1 ? d : -INFINITY;
                    }
                    const float mn = fmaxf(fmaxf(m, fmaxf(z[0], z[1])), fmaxf(z[2], z[3])), r = __expf(m - mn);
                    m = mn;
                    sum *= r;
#pragma unroll
                    for (int i = 0; i < DI; ++i) o[i] *= r;
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        const float e = __expf(z[g] - m);
                        sum += e;
#pragma unroll
                        for (int i = 0; i < DI; ++i) o[i] = fmaf(e, vv[g][i], o[i]);
                    }
                }
                float* mine = att + warp * (kDecMaxHead + 2);
#pragma unroll
                for (int i = 0; i < DI; ++i) if (lane + 32 * i < D) mine[lane + 32 * i] = o[i];
                if (lane == 0) { mine[kDecMaxHead] = m; mine[kDecMaxHead + 1] = sum; }
                __syncthreads();
                if (tid < D + 2) {
                    float M = -INFINITY;
#pragma unroll
                    for (int j = 0; j < kDecWarps; ++j) M = fmaxf(M, att[j * (kDecMaxHead + 2) + kDecMaxHead]);
                    float r = 0.0f;
                    const int at = tid < D ? tid : kDecMaxHead + 1;
#pragma unroll
                    for (int j = 0; j < kDecWarps; ++j) {
                        const float mj = att[j * (kDecMaxHead + 2) + kDecMaxHead];
                        if (mj > -INFINITY) r += __expf(mj - M) * att[j * (kDecMaxHead + 2) + at];
                    }
                    __stcg(p.part + (int64_t)u * (D + 2) + tid, tid == D ? M : r);  // values, maximum, sum of weights
                }
                __syncthreads();
            }
            if (!grid_barrier(p.barrier, target += gridDim.x, p.status, flag)) return;
            // ---- output projection on top of the residual stream
            if (p.vec) l2_prefetch(p.gated ? w.w3 : w.w2, (int64_t)C * F);
            for (int i = tid; i < p.n_seq * C; i += kDecThreads) {
                const int s = i / C, c = i - s * C, h = c / D;
                const float* pp = p.part + (int64_t)(s * H + h) * nsplit * (D + 2);
                float M = -INFINITY;
                for (int j = 0; j < nsplit; ++j) M = fmaxf(M, __ldcg(pp + j * (D + 2) + D));
                float o = 0.0f, sum = 0.0f;
                for (int j = 0; j < nsplit; ++j) {
                    const float e = __expf(__ldcg(pp + j * (D + 2) + D) - M);
                    sum = fmaf(e, __ldcg(pp + j * (D + 2) + D + 1), sum);
                    o = fmaf(e, __ldcg(pp + j * (D + 2) + c - h * D), o);
                }
                act[c * S + s] = o / sum;
            }
            for (int i = p.n_seq * C + tid; i < S * C; i += kDecThreads) act[(i % C) * S + i / C] = 0.0f;
            __syncthreads();
            for (int t = blockIdx.x; t < tiles_c; t += gridDim.x) {
                const float* const W[1] = {w.wo};
                float acc[1][S][4];
                tile_dot<S, 1>(W, t * 8, C, C, p.vec, act, acc);
                finish_tile(acc, t * 8, C, [&](int s, int n, float v, float) { __stcg(p.x + s * C + n, xs[s * C + n] + v + w.bo[n]); });
            }
            if (!grid_barrier(p.barrier, target += gridDim.x, p.status, flag)) return;
            // ---- MLP, first half
            if (p.vec && l + 1 < p.L) {
                const gcb_gpt_layer& nx = p.layers[l + 1];
                l2_prefetch(nx.wq, (int64_t)C * C); l2_prefetch(nx.wk, (int64_t)C * C); l2_prefetch(nx.wv, (int64_t)C * C);
            }
            load_x();
            normalise(w.norm2_gamma, w.norm2_beta, false);
            for (int t = blockIdx.x; t < tiles_f; t += gridDim.x) {
                if (p.gated) {
                    const float* const W[2] = {w.w1, w.w2};
                    float acc[2][S][4];
                    tile_dot<S, 2>(W, t * 8, F, C, p.vec, act, acc);
                    finish_tile(acc, t * 8, F, [&](int s, int n, float a, float b) {
                        a += w.b1[n];
                        __stcg(p.h + s * F + n, a * __fdividef(1.0f, 1.0f + __expf(-a)) * (b + w.b2[n]));
                    });
                } else {
                    const float* const W[1] = {w.w1};
                    float acc[1][S][4];
                    tile_dot<S, 1>(W, t * 8, F, C, p.vec, act, acc);
                    finish_tile(acc, t * 8, F, [&](int s, int n, float a, float) { __stcg(p.h + s * F + n, gelu_f(a + w.b1[n])); });
                }
            }
            if (!grid_barrier(p.barrier, target += gridDim.x, p.status, flag)) return;
            // ---- MLP, second half, on top of the residual stream
            for (int i = tid; i < S * F; i += kDecThreads) { const int s = i / F, f = i - s * F; act[f * S + s] = s < p.n_seq ? __ldcg(p.h + i) : 0.0f; }
            __syncthreads();
            {
                const float* const W[1] = {p.gated ? w.w3 : w.w2};
                const float* bias = p.gated ? w.b3 : w.b2;
                for (int t = blockIdx.x; t < tiles_c; t += gridDim.x) {
                    float acc[1][S][4];
                    tile_dot<S, 1>(W, t * 8, C, F, p.vec, act, acc);
                    finish_tile(acc, t * 8, C, [&](int s, int n, float v, float) { __stcg(p.x + s * C + n, xs[s * C + n] + v + bias[n]); });
                }
            }
            if (!grid_barrier(p.barrier, target += gridDim.x, p.status, flag)) return;
        }
        // ---- the next token
        if (pos + 1 < p.n_known) {  // already given
            given_token(pos + 1);
            continue;
        }
        load_x();
        normalise(p.final_gamma, p.final_beta, true);
        float top[S];
        int arg[S];
#pragma unroll
        for (int s = 0; s < S; ++s) { top[s] = -INFINITY; arg[s] = 0x7fffffff; }
        const int stride = gridDim.x * kDecWarps;
        for (int r0 = blockIdx.x * kDecWarps + warp; r0 < p.V; r0 += 2 * stride) {  // two rows of the embedding at a time
            float acc[2][S];
#pragma unroll
            for (int s = 0; s < S; ++s) acc[0][s] = acc[1][s] = 0.0f;
            const bool two = r0 + stride < p.V;
            const float* e0 = p.token_embed + (int64_t)r0 * C;
            const float* e1 = two ? e0 + (int64_t)stride * C : e0;
            if (p.vec) {
#pragma unroll 4
                for (int c = lane * 4; c < C; c += 128) {
                    const float4 a = __ldg(reinterpret_cast<const float4*>(e0 + c)), b = __ldg(reinterpret_cast<const float4*>(e1 + c));
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        const float4 y = ld4(act + s * C + c);
                        acc[0][s] = fmaf(a.x, y.x, fmaf(a.y, y.y, fmaf(a.z, y.z, fmaf(a.w, y.w, acc[0][s]))));
                        acc[1][s] = fmaf(b.x, y.x, fmaf(b.y, y.y, fmaf(b.z, y.z, fmaf(b.w, y.w, acc[1][s]))));
                    }
                }
            } else {
                for (int c = lane; c < C; c += 32) {
                    const float a = __ldg(e0 + c), b = __ldg(e1 + c);
#pragma unroll
                    for (int s = 0; s < S; ++s) { acc[0][s] = fmaf(a, act[s * C + c], acc[0][s]); acc[1][s] = fmaf(b, act[s * C + c], acc[1][s]); }
                }
            }
#pragma unroll
            for (int g = 0; g < 2; ++g)
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float v = warp_sum(acc[g][s]);
                    const int r = r0 + g * stride;
                    if (g == 1 && !two) continue;
                    if (p.logits != nullptr && lane == 0 && s < p.n_seq) p.logits[(int64_t)s * p.V + r] = v;
                    if (v > top[s]) { top[s] = v; arg[s] = r; }  // rows ascend: the first of equal logits stays
                }
        }
        if (p.logits != nullptr) continue;  // the caller picks the token (one position per call)
        if (p.vec) { l2_prefetch(p.layers[0].wq, (int64_t)C * C); l2_prefetch(p.layers[0].wk, (int64_t)C * C); l2_prefetch(p.layers[0].wv, (int64_t)C * C); }
        if (lane == 0) {
#pragma unroll
            for (int s = 0; s < S; ++s) best[warp * S + s] = make_float2(top[s], __int_as_float(arg[s]));
        }
        __syncthreads();
        auto better = [](float2& a, float2 b) { if (b.x > a.x || (b.x == a.x && __float_as_int(b.y) < __float_as_int(a.y))) a = b; };
        if (tid < S) {
            float2 b = best[tid];
            for (int j = 1; j < kDecWarps; ++j) better(b, best[j * S + tid]);
            __stcg(p.cand + blockIdx.x * S + tid, b);
        }
        if (!grid_barrier(p.barrier, target += gridDim.x, p.status, flag)) return;
        if (warp < S) {
            float2 b = make_float2(-INFINITY, __int_as_float(0x7fffffff));
            for (int j = lane; j < gridDim.x; j += 32) better(b, __ldcg(p.cand + j * S + warp));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) better(b, make_float2(__shfl_xor_sync(0xffffffffu, b.x, o), __shfl_xor_sync(0xffffffffu, b.y, o)));
            const int t = min(__float_as_int(b.y), p.V - 1);
            if (lane == 0) {
                tok[warp] = t;
                if (blockIdx.x == 0 && warp < p.n_seq) p.tokens[warp * p.tokens_ld + pos + 1] = t;
            }
        }
        __syncthreads();
    }
}

template <int S>
static int launch_decode(gcb_ctx* ctx, DecodeParams& p) {
    auto kfn = gpt_decode_kernel<S>;
    const size_t smem = DecSmem<S>::bytes(p.C, p.F);
    static bool attr_done[kMaxDevices] = {};
    if (!attr_done[ctx->device]) { GCB_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024)); attr_done[ctx->device] = true; }
    // small models have no work for every SM, and fewer CTAs meet faster: as many as the widest phase has tiles (or warps' worth of head rows)
    const int64_t tiles = std::max<int64_t>({(3 * (int64_t)p.C + 7) / 8, ((int64_t)p.F + 7) / 8, ((int64_t)p.V + 2 * kDecWarps - 1) / (2 * kDecWarps), (int64_t)p.n_seq * p.H});
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, kSMs);
    Scratch sc(ctx);
    const int64_t parts = (int64_t)p.n_seq * p.H * std::max<int64_t>(1, grid / ((int64_t)p.n_seq * p.H));
    auto up = [](int64_t n) { return (n + 127) / 128 * 128; };
    const int64_t n_x = up((int64_t)S * p.C), n_h = up((int64_t)S * p.F), n_part = up(parts * (p.D + 2)), n_cand = up(2 * (int64_t)kSMs * S);
    int rc = sc.get(sizeof(float) * (size_t)(2 * n_x + n_h + n_part + n_cand + 32));
    if (rc) return rc;
    float* b = sc.as<float>();
    p.barrier = reinterpret_cast<unsigned*>(b); b += 32;
    p.x = b; b += n_x;
    p.q = b; b += n_x;
    p.h = b; b += n_h;
    p.part = b; b += n_part;
    p.cand = reinterpret_cast<float2*>(b);
    GCB_CHECK_CUDA(cudaMemsetAsync(p.barrier, 0, sizeof(float) * (size_t)(32 + n_x), ctx->stream));  // the barrier; and rows of x beyond the last sequence stay finite
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kDecThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GCB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kfn, p));
    return after_launch(ctx, "gpt_decode");
}

// Sequences one launch takes: as many as fit beside the activations in shared memory (0: not even one does).
static int decode_group(int64_t C, int64_t F) {
    const size_t limit = 220 * 1024;
    if (DecSmem<8>::bytes(C, F) <= limit) return 8;
    if (DecSmem<4>::bytes(C, F) <= limit) return 4;
    if (DecSmem<2>::bytes(C, F) <= limit) return 2;
    return DecSmem<1>::bytes(C, F) <= limit ? 1 : 0;
}

}  // namespace gcb

using namespace gcb;

extern "C" {

int gcb_gpt_decode_supported(gcb_ctx* ctx, const gcb_gpt_model* m) {
    if (!ctx || !m || m->L < 1 || m->L > kDecMaxLayers || m->H < 1 || m->C < 1 || m->F < 1 || m->V < 1 || m->C % m->H != 0 || m->C / m->H > kDecMaxHead) return 0;
    if (m->V >= (int64_t(1) << 30) || m->C > 65536 || m->F > 65536) return 0;
    return decode_group(m->C, m->F) > 0 ? 1 : 0;
}

int gcb_gpt_decode_f32(gcb_ctx* ctx, const gcb_gpt_model* m, int64_t n_seq, float* cache, int64_t cache_len, int64_t* tokens, int64_t tokens_ld, int64_t pos0, int64_t n_pos, int64_t n_known, float* logits) {
    GCB_REQUIRE(ctx && m && cache && tokens && m->layers && m->token_embed && m->pos_embed && m->final_gamma, "gcb_gpt_decode_f32: NULL argument");
    if (!gcb_gpt_decode_supported(ctx, m)) {
        set_error("gcb_gpt_decode_f32: at most %d layers, heads of at most %d columns and activations that fit into shared memory", kDecMaxLayers, kDecMaxHead);
        return GCB_UNSUPPORTED;
    }
    GCB_REQUIRE(n_seq >= 0 && pos0 >= 0 && n_pos >= 0 && pos0 + n_pos <= cache_len && pos0 + n_pos <= m->T && tokens_ld >= pos0 + n_pos && n_known > pos0, "gcb_gpt_decode_f32: positions beyond the cache, the position table or the token rows");
    GCB_REQUIRE(logits == nullptr || n_known >= pos0 + n_pos, "gcb_gpt_decode_f32: with logits wanted every token of the call must be given");
    GCB_REQUIRE(logits != nullptr || n_known >= pos0 + n_pos + 1 || tokens_ld >= pos0 + n_pos + 1, "gcb_gpt_decode_f32: no room for the token that follows the last position");
    if (n_seq == 0 || n_pos == 0) return GCB_OK;
    cudaSetDevice(ctx->device);
    static_assert(sizeof(DecodeParams) < 32000, "kernel parameters");
    DecodeParams p;
    memset(&p, 0, sizeof(p));
    p.gated = m->layers[0].w3 != nullptr;
    bool vec = m->C % 4 == 0 && m->F % 4 == 0 && aligned16(m->token_embed) && aligned16(cache);
    for (int64_t l = 0; l < m->L; ++l) {
        const gcb_gpt_layer& w = m->layers[l];
        GCB_REQUIRE(w.norm1_gamma && w.wq && w.bq && w.wk && w.bk && w.wv && w.bv && w.wo && w.bo && w.norm2_gamma && w.w1 && w.b1 && w.w2 && w.b2 && (!p.gated || (w.w3 && w.b3)), "gcb_gpt_decode_f32: layer %lld has a NULL weight", (long long)l);
        p.layers[l] = w;
        vec = vec && aligned16(w.wq) && aligned16(w.wk) && aligned16(w.wv) && aligned16(w.wo) && aligned16(w.w1) && aligned16(w.w2) && aligned16(w.w3);
    }
    p.vec = vec;
    p.token_embed = m->token_embed; p.pos_embed = m->pos_embed; p.final_gamma = m->final_gamma; p.final_beta = m->final_beta;
    p.seq_stride = cache_len * m->C;
    p.kv_stride = n_seq * p.seq_stride;
    p.layer_stride = 2 * p.kv_stride;
    p.tokens_ld = tokens_ld;
    p.status = ctx->d_status;
    p.eps = m->eps;
    p.V = (int)m->V; p.C = (int)m->C; p.H = (int)m->H; p.D = (int)(m->C / m->H); p.L = (int)m->L; p.F = (int)m->F;
    p.scale = 1.0f / sqrtf((float)p.D);
    p.pos0 = (int)pos0; p.n_pos = (int)n_pos; p.n_known = (int)std::min<int64_t>(n_known, logits ? pos0 + n_pos : int64_t(1) << 30);
    const int64_t group = decode_group(m->C, m->F);
    for (int64_t s = 0; s < n_seq; s += group) {
        p.n_seq = (int)std::min(group, n_seq - s);
        p.cache = cache + s * p.seq_stride;
        p.tokens = tokens + s * tokens_ld;
        p.logits = logits ? logits + s * m->V : nullptr;
        const int rc = p.n_seq > 4 ? launch_decode<8>(ctx, p) : p.n_seq > 2 ? launch_decode<4>(ctx, p) : p.n_seq > 1 ? launch_decode<2>(ctx, p) : launch_decode<1>(ctx, p);
        if (rc) return rc;
    }
    return GCB_OK;
}

}  // extern "C"
