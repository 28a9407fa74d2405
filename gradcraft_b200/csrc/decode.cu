// Incremental decoding of a GPT: one persistent kernel takes a few sequences through any number of positions, keeping the keys
// and values of earlier positions in a cache.
// Reference counterpart: GPTGenerator::run_inference (nn/generators/gpt_generator.hpp:12-132), which forwards the whole context
// again for every new token.
//
// What bounds a position is reading the weights once (743 MB for the 180M-parameter model: 0.11 ms at the copy rate); the
// arithmetic is a matrix-vector product per weight.  As separate launches a position is ~85 dependent kernels of 2 - 4 us each,
// so the whole model runs inside one cooperative kernel, one CTA per SM: five phases per layer (q/k/v, attention, output
// projection, first and second half of the MLP), then the tied head with its arg-max, whose result is the next position's input
// without a trip to the host.
//   * Exchange: a phase needs what all CTAs computed in the one before.  Every exchanged value is an 8-byte word, the float beside
//     the number of the layer it belongs to; the reader polls the words themselves.  That is one store and one load latency per
//     phase and no fence (a fence also waits for the weights in flight); only keys and values, read a position later, are fenced,
//     once a position.  Each buffer is written again only after its readers have contributed to something the writer needs, so
//     one copy of each is enough (candidates of the arg-max: two).
//   * Products: a CTA owns tiles of eight output columns, i.e. one 32-byte sector of every weight row: N = 1024 columns give 128
//     tiles for 148 SMs, which wider tiles would not.  Two lanes take a row's sector, sixteen rows per warp load; lane and warp
//     sums are combined by shuffles and shared memory in a fixed order.
//   * Weights depend on nothing, so one thread runs ahead of the others: it has TMA copy the tiles, 256 rows at a time, into a ring
//     in shared memory in the order of use, across phases, layers and positions.  Up to 190 KB per SM in flight keep DRAM
//     streaming while the CTAs wait for one another, and the eight computing warps spend no instruction on addresses: with four
//     of them per scheduler a phase of the first version (every thread copying its own weights) was bound by issue slots.
//   * Attention: a unit is one head of one sequence and a stretch of at least kDecSplit positions, so that few heads still fill
//     the chip; the output projection merges the stretches while it loads them.
// Everything is fp32 FMA.  Every wait is bounded: one that runs out reports through the status word and the kernel returns.
#include <algorithm>

#include "gemm.cuh"

namespace gcb {

constexpr int kDecWarps = 8, kDecThreads = 32 * kDecWarps;  // computing threads; one more warp feeds the ring
constexpr int kDecMaxLayers = 48, kDecMaxHead = 128;
constexpr size_t kDecSmemLimit = 226 * 1024;
constexpr int kDecBox = 256;                              // weight rows one copy brings (the largest box)
constexpr int kDecRows = 1024, kDecStage = kDecRows * 8;  // weight rows and floats of a ring stage: waiting for a stage and handing it back costs ~200 cycles however many rows it has
constexpr int kDecMaxStages = 6, kDecMinStages = 2;
constexpr int kDecSplit = 128;  // positions from which a second unit pays for one head
constexpr int kDecMeet = 4;    // tiles whose sums are finished together (even: a gated tile has two)
constexpr int kDecMaps = 7;    // tensor maps per layer: wq, wk, wv, wo, w1, w2, w3

struct DecodeParams {
    gcb_gpt_layer layers[kDecMaxLayers];
    const CUtensorMap* maps;  // [layer][kDecMaps]
    const float *token_embed, *pos_embed, *final_gamma, *final_beta;
    float* cache;      // [layer][key, value][sequence][position][C]
    int64_t seq_stride, kv_stride, layer_stride;  // of the cache, in elements
    int64_t* tokens;   // [sequence][tokens_ld]
    int64_t tokens_ld;
    // exchange between CTAs: residual stream after the attention and after the MLP, q / k / v, attention stretches, hidden
    // activations, [2][CTA][S] best logits and their tokens
    unsigned long long *xa, *xb, *qkv, *part, *h, *cand;
    float* logits;  // [sequence][V] or NULL
    int* status;
    float eps, scale;
    int n_seq, pos0, n_pos, n_known, stages;
    int V, C, H, D, L, F, gated;
};

__device__ __forceinline__ uint32_t dec_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void l2_prefetch(const float* p, int64_t n) {  // this CTA's stretch of p[0 .. n)
    const int64_t bytes = n * 4, share = ((bytes + gridDim.x - 1) / gridDim.x + 4095) & ~int64_t(4095);
    const int64_t b0 = share * blockIdx.x, b1 = min(bytes & ~int64_t(15), b0 + share);
    for (int64_t b = b0 + 4096 * (int64_t)threadIdx.x; b < b1; b += 4096 * (int64_t)kDecThreads)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(reinterpret_cast<const char*>(p) + b), "r"((uint32_t)min((int64_t)4096, b1 - b)));
}

// Barriers among the computing warps.
__device__ __forceinline__ void dec_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kDecThreads) : "memory"); }
__device__ __forceinline__ bool dec_sync_and(bool v) {  // the same answer for every thread
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.and.pred q, 1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"((int)v), "n"(kDecThreads) : "memory");
    return r != 0;
}

// Exchanged words: a float and the number of the layer (counted over all positions of the call) it belongs to.
__device__ __forceinline__ void put_word(unsigned long long* w, float v, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"(((unsigned long long)epoch << 32) | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ unsigned long long look_word(const unsigned long long* w) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(w) : "memory");
    return v;
}
// Keys and values travel through the cache with plain stores and loads; the words say when they are there.  Between such a store and the
// word that announces it, and between the word as seen and the load, stands a fence: of the thread that does both, or of the one that
// deals with the word where a barrier of the CTA lies between (the fence is cumulative).
__device__ __forceinline__ void dec_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
constexpr unsigned kDecPolls = 1u << 21;  // of ~1 us: seconds
// out[u] = the float of w[index(u)] (index < 0: none, 0) as soon as all of them belong to `epoch`; false when they do not in time
template <int B, class Index>
__device__ __forceinline__ bool get_words(const unsigned long long* w, Index&& index, unsigned epoch, float (&out)[B], int* status) {
    for (unsigned t = 0; t < kDecPolls; ++t) {
        unsigned long long v[B];
        bool all = true;
#pragma unroll
        for (int u = 0; u < B; ++u) v[u] = index(u) >= 0 ? look_word(w + index(u)) : (unsigned long long)epoch << 32;
#pragma unroll
        for (int u = 0; u < B; ++u) { all = all && (unsigned)(v[u] >> 32) == epoch; out[u] = __uint_as_float((unsigned)v[u]); }
        if (__all_sync(__activemask(), all)) return true;  // together, or what follows would be run once per straggler
    }
    atomicExch(&status[0], 1);
    atomicExch(&status[1], 120);
    return false;
}
__device__ __forceinline__ bool dec_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}

// The feeding thread: the tiles of this CTA, in the order in which the computing warps take them.
__device__ void feed_weights(const DecodeParams& p, float* ring, uint32_t full, uint32_t empty, volatile int* abort_flag) {
    const int tiles_c = (p.C + 7) / 8, tiles_f = (p.F + 7) / 8;
    uint32_t it = 0;
    bool ok = true;
    auto rows = [&](const CUtensorMap* map, int n0, int k0, int K) {
        const int boxes = (min(kDecRows, K - k0) + kDecBox - 1) / kDecBox;
        const int s = (int)(it % (uint32_t)p.stages);
        const uint32_t ph = (it / (uint32_t)p.stages) & 1u;
        bool free_now = false;
        for (unsigned t = 0; t < (1u << 18) && !*abort_flag; ++t)
            if (dec_try_wait(empty + 8 * s, ph ^ 1u)) { free_now = true; break; }
        if (!free_now) { ok = false; return; }
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + 8 * s), "r"((uint32_t)(boxes * kDecBox * 8 * sizeof(float))) : "memory");
        for (int i = 0; i < boxes; ++i)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dec_smem(ring + s * kDecStage + i * kDecBox * 8)), "l"(map), "r"(full + 8 * s),
                         "r"(n0), "r"(k0 + i * kDecBox) : "memory");
        ++it;
    };
    for (int pos = 0; pos < p.n_pos && ok; ++pos)
        for (int l = 0; l < p.L && ok; ++l) {
            const CUtensorMap* m = p.maps + l * kDecMaps;
            for (int t = blockIdx.x; t < 3 * tiles_c && ok; t += gridDim.x) {
                const int which = t / tiles_c;
                for (int k0 = 0; k0 < p.C && ok; k0 += kDecRows) rows(m + which, (t - which * tiles_c) * 8, k0, p.C);
            }
            for (int t = blockIdx.x; t < tiles_c && ok; t += gridDim.x)
                for (int k0 = 0; k0 < p.C && ok; k0 += kDecRows) rows(m + 3, t * 8, k0, p.C);
            for (int t = blockIdx.x; t < tiles_f && ok; t += gridDim.x)
                for (int i = 4; i < (p.gated ? 6 : 5); ++i)
                    for (int k0 = 0; k0 < p.C && ok; k0 += kDecRows) rows(m + i, t * 8, k0, p.C);
            for (int t = blockIdx.x; t < tiles_c && ok; t += gridDim.x)
                for (int k0 = 0; k0 < p.F && ok; k0 += kDecRows) rows(m + (p.gated ? 6 : 5), t * 8, k0, p.F);
        }
    if (!ok)  // given up: the copies in flight still have to land before the CTA may go
        for (uint32_t j = it > (uint32_t)p.stages ? it - (uint32_t)p.stages : 0; j < it; ++j)
            for (unsigned t = 0; t < (1u << 18); ++t)
                if (dec_try_wait(full + 8 * (j % (uint32_t)p.stages), (j / (uint32_t)p.stages) & 1u)) break;
}

// Sums NV values over the sixteen lanes of the same parity, halving what a lane holds at every step.  Returns the index of the
// first of the max(1, NV / 16) values that lane ends up with, or -1 where another lane has the same ones.
template <int NV>
__device__ __forceinline__ int sum_rows(float (&v)[NV]) {
    const int lane = threadIdx.x & 31;
    int n = NV, first = 0;
    bool dup = false;
#pragma unroll
    for (int o = 16; o >= 2; o >>= 1) {
        const bool up = (lane & o) != 0;
        if (n > 1) {
            const int h = n / 2;
#pragma unroll
            for (int i = 0; i < NV / 2; ++i)
                if (i < h) {
                    const float send = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            first += up ? h : 0;
            n = h;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
            dup = dup || up;
        }
    }
    return dup ? -1 : first;
}

template <int S>
struct DecSmem {
    // floats: ring [stages][kDecStage], x [S][C], activations [max(C, F)][S] (the head: [S][C]), then the fixed part
    static constexpr int RED = 2 * kDecMeet * kDecWarps * S * 8;                              // two buffers of warp sums
    static constexpr int ATT = kDecWarps * (kDecMaxHead + 4) + 3 * kDecMaxHead;               // a warp's stretch: sum of values, maximum, sum of weights; q, k, v of this position
    static constexpr int FIXED = RED + ATT + 2 * kDecWarps * S + 2 * kDecWarps * S + 8 + 4 + 4 * kDecMaxStages;  // + two sets of warp sums, best logits, tokens, flag, barriers
    static size_t bytes(int stages, int64_t C, int64_t F) { return 128 + sizeof(float) * (size_t)(stages * kDecStage + (S * C + 3) / 4 * 4 + (S * std::max(C, F) + 3) / 4 * 4 + FIXED); }
    static int stages(int64_t C, int64_t F) {  // what fits, 0 when less than kDecMinStages does
        int n = kDecMaxStages;
        while (n >= kDecMinStages && bytes(n, C, F) > kDecSmemLimit) --n;
        return n >= kDecMinStages ? n : 0;
    }
};

template <int S>
__global__ void __launch_bounds__(kDecThreads + 32, 1) gpt_decode_kernel(const __grid_constant__ DecodeParams p) {
    using Smem = DecSmem<S>;
    extern __shared__ uint8_t dec_raw[];
    float* ring = reinterpret_cast<float*>(dec_raw + ((128u - (dec_smem(dec_raw) & 127u)) & 127u));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = p.C, D = p.D, F = p.F, H = p.H;
    float* xs = ring + p.stages * kDecStage;
    float* act = xs + (S * C + 3) / 4 * 4;
    float* red = act + (S * max(C, F) + 3) / 4 * 4;
    float* att = red + Smem::RED;
    float* stat = att + Smem::ATT;  // [2][S][warps]
    float2* best = reinterpret_cast<float2*>(stat + 2 * kDecWarps * S);
    int* tok = reinterpret_cast<int*>(best + kDecWarps * S);
    int* abort_flag = tok + 8;
    uint64_t* bars = reinterpret_cast<uint64_t*>(abort_flag + 4);
    const uint32_t full = dec_smem(bars), empty = full + 8 * kDecMaxStages;
    if (tid == 0) {
        for (int s = 0; s < p.stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + 8 * s));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty + 8 * s), "r"(kDecWarps));
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (warp == kDecWarps) {
        if (lane == 0) feed_weights(p, ring, full, empty, abort_flag);
        return;
    }

    unsigned epoch = 1;
    int buf = 0, stage = 0;
    uint32_t stage_ph = 0;
    bool ok = true;  // no wait of this thread has run out; loops are left on it only after dec_sync_and has made it the same for all
    const float inv_c = 1.0f / (float)C;
    const int kt = warp * 16 + (lane >> 1);  // this thread's weight rows: kt + 128 u

    constexpr int NV = 4;  // columns of a row per thread that are kept in registers (C <= 1024: all of them)
    float gm[NV], bt[NV];  // the coming normalisation's gamma and beta, requested before its input arrives
    auto fetch_norm = [&](const float* gamma, const float* beta) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = tid + i * kDecThreads;
            gm[i] = c < C ? __ldg(gamma + c) : 0.0f;
            bt[i] = c < C && beta ? __ldg(beta + c) : 0.0f;
        }
    };
    // xs and xr <- the residual stream as the other CTAs left it; thread t takes the columns t, t + 256, ... (xr: the first NV of them)
    float xr[S][NV];
    auto load_x = [&](const unsigned long long* x, unsigned epoch) {
        for (int c0 = tid; c0 < C; c0 += NV * kDecThreads)
#pragma unroll
            for (int s0 = 0; s0 < S; s0 += 2) {
                constexpr int SB = S < 2 ? 1 : 2;
                float v[NV * SB];
                ok = get_words<NV * SB>(x, [&](int u) { const int c = c0 + (u % NV) * kDecThreads, s = s0 + u / NV; return c < C && s < p.n_seq ? s * C + c : -1; }, epoch, v, p.status) && ok;
#pragma unroll
                for (int u = 0; u < NV * SB; ++u) {
                    const int c = c0 + (u % NV) * kDecThreads;
                    if (c < C) xs[(s0 + u / NV) * C + c] = v[u];
                    if (c0 == tid) xr[s0 + u / NV][u % NV] = v[u];
                }
            }
    };
    auto all_warps = [&](const float* w) {  // the sum of the warps' sums, in warp order
        float r = 0.0f;
#pragma unroll
        for (int j = 0; j < kDecWarps; j += 4) { const float4 v = ld4(w + j); r += v.x; r += v.y; r += v.z; r += v.w; }
        return r;
    };
    // act <- the normalised rows: [k][s] for the products, [s][k] for the head.  Two passes over what every thread itself loaded.
    // False when an exchange ran out of polls.
    auto normalise = [&](const float* gamma, const float* beta, bool by_row) {
        float mu[S], rs[S];
#pragma unroll
        for (int s = 0; s < S; ++s) {
            float sum = 0.0f;
#pragma unroll
            for (int i = 0; i < NV; ++i) if (tid + i * kDecThreads < C) sum += beta ? xr[s][i] : xr[s][i] * xr[s][i];
            for (int c = tid + NV * kDecThreads; c < C; c += kDecThreads) { const float v = xs[s * C + c]; sum += beta ? v : v * v; }
            sum = warp_sum(sum);
            if (lane == 0) stat[s * kDecWarps + warp] = sum;
        }
        __syncwarp();
        if (!(ok = dec_sync_and(ok))) return false;
#pragma unroll
        for (int s = 0; s < S; ++s) mu[s] = all_warps(stat + s * kDecWarps) * inv_c;
        if (beta) {
#pragma unroll
            for (int s = 0; s < S; ++s) {
                float q = 0.0f;
#pragma unroll
                for (int i = 0; i < NV; ++i) if (tid + i * kDecThreads < C) { const float d = xr[s][i] - mu[s]; q = fmaf(d, d, q); }
                for (int c = tid + NV * kDecThreads; c < C; c += kDecThreads) { const float d = xs[s * C + c] - mu[s]; q = fmaf(d, d, q); }
                q = warp_sum(q);
                if (lane == 0) stat[(S + s) * kDecWarps + warp] = q;
            }
            __syncwarp();
            dec_sync();
#pragma unroll
            for (int s = 0; s < S; ++s) rs[s] = __frsqrt_rn(all_warps(stat + (S + s) * kDecWarps) * inv_c + p.eps);
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) { rs[s] = __frsqrt_rn(mu[s] + p.eps); mu[s] = 0.0f; }
        }
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = tid + i * kDecThreads;
            if (c < C) {
#pragma unroll
                for (int s = 0; s < S; ++s) act[by_row ? s * C + c : c * S + s] = (xr[s][i] - mu[s]) * rs[s] * gm[i] + bt[i];
            }
        }
        for (int c = tid + NV * kDecThreads; c < C; c += kDecThreads) {
            const float g = __ldg(gamma + c), b = beta ? __ldg(beta + c) : 0.0f;
#pragma unroll
            for (int s = 0; s < S; ++s) act[by_row ? s * C + c : c * S + s] = (xs[s * C + c] - mu[s]) * rs[s] * g + b;
        }
        __syncwarp();
        dec_sync();
        return true;
    };
    // The next tile of the ring times act: this warp's share of sum_k act[k][s] * W[k][column j of the tile] goes to out[s * 8 + j].
    auto tile_dot = [&](int K, float* out) {
        float acc[S * 4];
#pragma unroll
        for (int i = 0; i < S * 4; ++i) acc[i] = 0.0f;
#pragma unroll 1
        for (int k0 = 0; k0 < K; k0 += kDecRows) {
            bool landed = false;
            for (unsigned t = 0; t < (1u << 18) && ok; ++t) if (dec_try_wait(full + 8 * stage, stage_ph)) { landed = true; break; }
            if (!landed && ok) { atomicExch(&p.status[0], 1); atomicExch(&p.status[1], 121); ok = false; }
            const float* st = ring + stage * kDecStage + kt * 8 + 4 * (lane & 1);
            const float* x = act + (k0 + kt) * S;
            auto row = [&](int u) {
                const float4 v = ld4(st + u * 1024);
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float y = x[u * 128 * S + s];
                    float* c = acc + s * 4;
                    c[0] = fmaf(y, v.x, c[0]); c[1] = fmaf(y, v.y, c[1]); c[2] = fmaf(y, v.z, c[2]); c[3] = fmaf(y, v.w, c[3]);
                }
            };
            if (K - k0 >= kDecRows) {
#pragma unroll
                for (int u = 0; u < kDecRows / 128; ++u) row(u);
            } else {
#pragma unroll 2
                for (int u = 0; k0 + kt + 128 * u < K; ++u) row(u);
            }
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty + 8 * stage) : "memory");
            if (++stage == p.stages) { stage = 0; stage_ph ^= 1u; }
        }
        constexpr int HELD = S * 4 / 16 > 1 ? S * 4 / 16 : 1;
        const int first = sum_rows(acc);
        if (first >= 0) {
#pragma unroll
            for (int i = 0; i < HELD; ++i) { const int q = first + i; out[(q >> 2) * 8 + 4 * (lane & 1) + (q & 3)] = acc[i]; }
        }
    };
    auto given_token = [&](int pos) {  // an id outside the vocabulary is reported, not dereferenced
        if (tid < S) {
            int64_t t = tid < p.n_seq ? p.tokens[tid * p.tokens_ld + pos] : 0;
            if (t < 0 || t >= p.V) { atomicExch(&p.status[0], 2); atomicExch(&p.status[1], pos); t = 0; }
            tok[tid] = (int)t;
        }
        dec_sync();
    };
    given_token(p.pos0);
    const int tiles_c = (C + 7) / 8, tiles_f = (F + 7) / 8, cta = blockIdx.x;
    const int heads = p.n_seq * H, most = max(1, (int)gridDim.x / heads);

    // One pass through the loop body per phase, all products through the same code: what runs once per phase is bound by fetching
    // its instructions, so there should be few of them.
    enum { QKV, ATTENTION, OUT, MLP1, MLP2, HEAD };
    for (int pos = p.pos0; pos < p.pos0 + p.n_pos && ok; ++pos) {
        const int len = pos + 1, per = max(kDecSplit, (len + most - 1) / most), nsplit = (len + per - 1) / per;
        const bool head = pos + 1 >= p.n_known;
        for (int l = 0; l < p.L && ok; ++l, ++epoch) {  // epoch: number of this layer in the call, from 1
            const gcb_gpt_layer& w = p.layers[l];
            float* kc = p.cache + l * p.layer_stride;
            float* vc = kc + p.kv_stride;
#pragma unroll 1
            for (int ph = QKV; ph <= (head && l + 1 == p.L ? HEAD : MLP2) && ok; ++ph) {
                if (ph == ATTENTION) {  // over the positions so far, in stretches
                    for (int u = cta; u < heads * nsplit; u += gridDim.x) {
                        const int sh = u / nsplit, s = sh / H, h = sh - s * H, j0 = (u - sh * nsplit) * per, j1 = min(len, j0 + per);
                        const float* kb = kc + s * p.seq_stride + h * D;
                        const float* vb = vc + s * p.seq_stride + h * D;
                        float* now = att + kDecWarps * (kDecMaxHead + 4);  // [q, k, v][D] of this position
                        // four columns per lane; a warp load takes 32 / lpr rows, four of them are in flight
                        const int lpr = D <= 32 ? 8 : D <= 64 ? 16 : 32, rpw = 32 / lpr, col = 4 * (lane % lpr), step = kDecWarps * rpw, j_first = j0 + warp * rpw + lane / lpr;
                        const bool in = col < D;
                        float4 kk[4], vv[4], kn[4], vn[4];  // rows in hand, and the next ones
                        auto rows = [&](int j, float4 (&kk)[4], float4 (&vv)[4]) {
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                const int jj = j + g * step;
                                const bool live = in && jj < min(j1, pos);
                                kk[g] = live ? __ldcg(reinterpret_cast<const float4*>(kb + (int64_t)jj * C + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
                                vv[g] = live ? __ldcg(reinterpret_cast<const float4*>(vb + (int64_t)jj * C + col)) : make_float4(0.f, 0.f, 0.f, 0.f);
                            }
                        };
                        // Earlier rows are requested before this position's q arrives, where all of them are known to be there: written
                        // before this call, or before the arg-max exchange that gave this position its token.  Otherwise this position's
                        // k and v say so: the thread that wrote a column of the earlier rows has fenced them and writes the word now.
                        const bool early = pos == p.pos0 || pos >= p.n_known;
                        if (early) rows(j_first, kk, vv);
                        if (tid < D) {
                            float v[3];
                            ok = get_words<3>(p.qkv + s * C + h * D + tid, [&](int which) { return which * S * C; }, epoch, v, p.status) && ok;
                            if (!early) dec_fence();
#pragma unroll
                            for (int i = 0; i < 3; ++i) now[i * kDecMaxHead + tid] = v[i];
                        }
                        if (!(ok = dec_sync_and(ok))) break;
                        float4 q = make_float4(0.f, 0.f, 0.f, 0.f), o = q;
                        float m = -INFINITY, sum = 0.0f;
                        if (in) { q = ld4(now + col); q.x *= p.scale; q.y *= p.scale; q.z *= p.scale; q.w *= p.scale; }
                        for (int j = j_first; j - lane / lpr < j1; j += 4 * step) {  // the same trips for every lane of a warp
                            if (j == j_first && !early) rows(j, kk, vv);
                            rows(j + 4 * step, kn, vn);
                            float z[4];
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                const int jj = j + g * step;
                                if (jj == pos && in) { kk[g] = ld4(now + kDecMaxHead + col); vv[g] = ld4(now + 2 * kDecMaxHead + col); }
                                z[g] = fmaf(q.x, kk[g].x, fmaf(q.y, kk[g].y, fmaf(q.z, kk[g].z, q.w * kk[g].w)));
                            }
                            for (int b = lpr / 2; b > 0; b >>= 1) {
#pragma unroll
                                for (int g = 0; g < 4; ++g) z[g] += __shfl_xor_sync(0xffffffffu, z[g], b);
                            }
#pragma unroll
                            for (int g = 0; g < 4; ++g) if (j + g * step >= j1) z[g] = -INFINITY;
                            const float mn = fmaxf(fmaxf(m, fmaxf(z[0], z[1])), fmaxf(z[2], z[3]));
                            if (mn > -INFINITY) {
                                const float r = __expf(m - mn);
                                m = mn;
                                sum *= r;
                                o.x *= r; o.y *= r; o.z *= r; o.w *= r;
#pragma unroll
                                for (int g = 0; g < 4; ++g) {
                                    const float e = __expf(z[g] - m);
                                    sum += e;
                                    o.x = fmaf(e, vv[g].x, o.x); o.y = fmaf(e, vv[g].y, o.y); o.z = fmaf(e, vv[g].z, o.z); o.w = fmaf(e, vv[g].w, o.w);
                                }
                            }
#pragma unroll
                            for (int g = 0; g < 4; ++g) { kk[g] = kn[g]; vv[g] = vn[g]; }
                        }
                        for (int b = lpr; b < 32; b <<= 1) {  // the warp's rows of the same columns
                            const float m2 = __shfl_xor_sync(0xffffffffu, m, b), s2 = __shfl_xor_sync(0xffffffffu, sum, b), M = fmaxf(m, m2);
                            const float x = __shfl_xor_sync(0xffffffffu, o.x, b), y = __shfl_xor_sync(0xffffffffu, o.y, b), zz = __shfl_xor_sync(0xffffffffu, o.z, b), w4 = __shfl_xor_sync(0xffffffffu, o.w, b);
                            const float e1 = m > -INFINITY ? __expf(m - M) : 0.0f, e2 = m2 > -INFINITY ? __expf(m2 - M) : 0.0f;
                            sum = e1 * sum + e2 * s2;
                            o.x = e1 * o.x + e2 * x; o.y = e1 * o.y + e2 * y; o.z = e1 * o.z + e2 * zz; o.w = e1 * o.w + e2 * w4;
                            m = M;
                        }
                        float* mine = att + warp * (kDecMaxHead + 4);
                        if (lane < lpr && in) st4(mine + col, o);
                        if (lane == 0) { mine[kDecMaxHead] = m; mine[kDecMaxHead + 1] = sum; }
                        dec_sync();
                        if (tid < D + 2) {
                            float M = -INFINITY;
#pragma unroll
                            for (int j = 0; j < kDecWarps; ++j) M = fmaxf(M, att[j * (kDecMaxHead + 4) + kDecMaxHead]);
                            float r = 0.0f, sums = 0.0f;
                            const int at = tid < D ? tid : kDecMaxHead + 1;
#pragma unroll
                            for (int j = 0; j < kDecWarps; ++j) {
                                const float mj = att[j * (kDecMaxHead + 4) + kDecMaxHead], e = mj > -INFINITY ? __expf(mj - M) : 0.0f;
                                if (e != 0.0f) {
                                    r = fmaf(e, att[j * (kDecMaxHead + 4) + at], r);
                                    sums = fmaf(e, att[j * (kDecMaxHead + 4) + kDecMaxHead + 1], sums);
                                }
                            }
                            if (nsplit > 1) put_word(p.part + (int64_t)u * (D + 2) + tid, tid == D ? M : r, epoch);  // values, maximum, sum of weights
                            else if (tid < D) put_word(p.part + s * C + h * D + tid, r / sums, epoch);               // the whole head: its output
                        }
                        dec_sync();
                    }
                    continue;
                }
                const int tiles = ph == QKV ? 3 * tiles_c : ph == MLP1 ? tiles_f : ph == HEAD ? 0 : tiles_c;
                if (cta >= tiles && ph != HEAD && !(ph == MLP1 && cta < tiles_c)) continue;
                // ---- what the phase multiplies by its weights
                if (ph == QKV || ph == MLP1 || ph == HEAD) {
                    const float* gamma = ph == QKV ? w.norm1_gamma : ph == MLP1 ? w.norm2_gamma : p.final_gamma;
                    const float* beta = ph == QKV ? w.norm1_beta : ph == MLP1 ? w.norm2_beta : p.final_beta;
                    fetch_norm(gamma, beta);
                    // A given token holds no CTA back, and one with tiles of q, k and v alone (hidden widths below three widths) waits for nobody
                    // after them: it would write a position's words over the last ones while somebody still looks for those.  The
                    // stream after the last layer says that nobody does.
                    if (ph != QKV || l > 0 || (pos > p.pos0 && pos < p.n_known)) load_x(ph == MLP1 ? p.xa : p.xb, ph == QKV ? epoch - 1 : epoch);
                    if (ph == QKV && l == 0) {
                        for (int c0 = tid; c0 < C; c0 += NV * kDecThreads)
#pragma unroll
                            for (int i = 0; i < NV; ++i) {
                                const int c = c0 + i * kDecThreads;
                                if (c >= C) continue;
                                const float at = __ldg(p.pos_embed + (int64_t)pos * C + c);
#pragma unroll
                                for (int s = 0; s < S; ++s) {
                                    const float v = __ldg(p.token_embed + (int64_t)tok[s] * C + c) + at;
                                    xs[s * C + c] = v;
                                    if (c0 == tid) xr[s][i] = v;
                                }
                            }
                    }
                    if (ph == QKV) for (int s = 0; s < p.n_seq; ++s) { l2_prefetch(kc + s * p.seq_stride, (int64_t)pos * C); l2_prefetch(vc + s * p.seq_stride, (int64_t)pos * C); }
                    if (cta < tiles || ph == HEAD) {
                        if (!normalise(gamma, beta, ph == HEAD)) break;
                    } else {  // the stream alone, for the residual of MLP2
                        __syncwarp();
                        if (!(ok = dec_sync_and(ok))) break;
                    }
                } else if (ph == OUT && nsplit > 1) {
                    // weights of the stretches of every head, then their weighted sum: at most 148 stretches in all
                    for (int i = tid; i < heads * nsplit; i += kDecThreads) {
                        float v[2];
                        ok = get_words<2>(p.part + (int64_t)i * (D + 2) + D, [](int u) { return u; }, epoch, v, p.status) && ok;
                        att[2 * i] = v[0];
                        att[2 * i + 1] = v[1];
                    }
                    dec_sync();
                    for (int i = tid; i < heads; i += kDecThreads) {
                        float* mine = att + 2 * i * nsplit;
                        float M = -INFINITY, sum = 0.0f;
                        for (int j = 0; j < nsplit; ++j) M = fmaxf(M, mine[2 * j]);
                        for (int j = 0; j < nsplit; ++j) { mine[2 * j] = __expf(mine[2 * j] - M); sum = fmaf(mine[2 * j], mine[2 * j + 1], sum); }
                        for (int j = 0; j < nsplit; ++j) mine[2 * j] /= sum;
                    }
                    dec_sync();
                    for (int i = tid; i < p.n_seq * C; i += 4 * kDecThreads) {
                        float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                        int head_of[4], at[4];  // (sequence, head) and first word of four columns (C is a multiple of D)
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const int e = i + g * kDecThreads;
                            head_of[g] = e < p.n_seq * C ? e / D : -1;
                            at[g] = head_of[g] * nsplit * (D + 2) + e - head_of[g] * D;
                        }
                        for (int j0 = 0; j0 < nsplit; j0 += 4) {
                            float v[16];
                            ok = get_words<16>(p.part, [&](int u) { const int g = u >> 2, j = j0 + (u & 3); return head_of[g] >= 0 && j < nsplit ? at[g] + j * (D + 2) : -1; }, epoch, v, p.status) && ok;
#pragma unroll
                            for (int u = 0; u < 16; ++u) if (head_of[u >> 2] >= 0 && j0 + (u & 3) < nsplit) o[u >> 2] = fmaf(att[2 * (head_of[u >> 2] * nsplit + j0 + (u & 3))], v[u], o[u >> 2]);
                        }
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            const int e = i + g * kDecThreads, s = S == 1 ? 0 : e / C;
                            if (head_of[g] >= 0) act[(e - s * C) * S + s] = o[g];
                        }
                    }
                } else {
                    const int n = ph == OUT ? C : F, total = p.n_seq * n;
                    for (int i = tid; i < total; i += 16 * kDecThreads) {
                        float v[16];
                        ok = get_words<16>(ph == OUT ? p.part : p.h, [&](int u) { const int e = i + u * kDecThreads; return e < total ? e : -1; }, epoch, v, p.status) && ok;
#pragma unroll
                        for (int u = 0; u < 16; ++u) {
                            const int e = i + u * kDecThreads, s = S == 1 ? 0 : e / n;
                            if (e < total) act[(e - s * n) * S + s] = v[u];
                        }
                    }
                }
                if (ph == OUT || ph == MLP2) {
                    const int n = ph == OUT ? C : F;
                    for (int i = p.n_seq * n + tid; i < S * n; i += kDecThreads) act[(i % n) * S + i / n] = 0.0f;  // no further sequence
                    if (!(ok = dec_sync_and(ok))) break;
                }
                // ---- the products: up to kDecMeet tiles of this CTA, then one meeting of its warps for all of them
                const int K = ph == MLP2 ? F : C, N = ph == MLP1 ? F : C, each = ph == MLP1 && p.gated ? 2 : 1;  // matrices per tile
#pragma unroll 1
                for (int t0 = cta; t0 < tiles; t0 += kDecMeet / each * gridDim.x) {
                    // what this thread finishes: sequence s, column n of the group's g-th tile
                    const int g = tid / (S * 8), s = (tid >> 3) % S, t = t0 + g * gridDim.x, which = ph == QKV ? t / tiles_c : 0, n = (t - which * tiles_c) * 8 + (tid & 7);
                    const bool mine = g < kDecMeet / each && t < tiles && n < N && s < p.n_seq;
                    float b = 0.0f, b2 = 0.0f;
                    if (mine) {
                        b = __ldg((ph == QKV ? (which == 0 ? w.bq : which == 1 ? w.bk : w.bv) : ph == OUT ? w.bo : ph == MLP1 ? w.b1 : p.gated ? w.b3 : w.b2) + n);
                        if (each == 2) b2 = __ldg(w.b2 + n);
                    }
                    float* rb = red + (buf & 1) * (kDecMeet * kDecWarps * S * 8);
                    ++buf;
#pragma unroll 1
                    for (int e = 0; e < kDecMeet && t0 + e / each * (int)gridDim.x < tiles; ++e) tile_dot(K, rb + (e * kDecWarps + warp) * (S * 8));
                    __syncwarp();
                    if (!(ok = dec_sync_and(ok))) break;
                    if (mine) {
                        const float* r = rb + g * each * (kDecWarps * S * 8) + (tid & 7) + 8 * s;
                        float v = 0.0f, v2 = 0.0f;
#pragma unroll
                        for (int j = 0; j < kDecWarps; ++j) v += r[j * (S * 8)];
                        if (ph == QKV) {
                            v += b;
                            put_word(p.qkv + (which * S + s) * C + n, v, epoch);
                            if (which > 0) __stcg((which == 1 ? kc : vc) + s * p.seq_stride + (int64_t)pos * C + n, v);
                        } else if (ph == MLP1) {
                            v += b;
                            if (each == 2) {
#pragma unroll
                                for (int j = 0; j < kDecWarps; ++j) v2 += r[(kDecWarps + j) * (S * 8)];
                                v = v * __fdividef(1.0f, 1.0f + __expf(-v)) * (v2 + b2);
                            } else {
                                v = gelu_f(v);
                            }
                            put_word(p.h + s * F + n, v, epoch);
                        } else {
                            put_word((ph == OUT ? p.xa : p.xb) + s * C + n, xs[s * C + n] + v + b, epoch);
                        }
                    }
                    __syncwarp();
                }
            }
        }
        if (!ok) break;
        if (!head) {  // the next token is given: who wrote keys and values (the threads that finish a group's tiles) writes q, k and v next
            if (tid < kDecMeet * S * 8 && cta < 3 * tiles_c) dec_fence();
            given_token(pos + 1);
            continue;
        }
        float top[S];
        int arg[S];
#pragma unroll
        for (int s = 0; s < S; ++s) { top[s] = -INFINITY; arg[s] = 0x7fffffff; }
        const int stride = gridDim.x * kDecWarps;
        for (int r0 = cta * kDecWarps + warp; r0 < p.V; r0 += 2 * stride) {  // two rows of the embedding at a time
            float acc[2][S];
#pragma unroll
            for (int s = 0; s < S; ++s) acc[0][s] = acc[1][s] = 0.0f;
            const bool two = r0 + stride < p.V;
            const float* e0 = p.token_embed + (int64_t)r0 * C;
            const float* e1 = two ? e0 + (int64_t)stride * C : e0;
#pragma unroll 8
            for (int c = lane * 4; c < C; c += 128) {
                const float4 a = __ldg(reinterpret_cast<const float4*>(e0 + c)), b = __ldg(reinterpret_cast<const float4*>(e1 + c));
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float4 y = ld4(act + s * C + c);
                    acc[0][s] = fmaf(a.x, y.x, fmaf(a.y, y.y, fmaf(a.z, y.z, fmaf(a.w, y.w, acc[0][s]))));
                    acc[1][s] = fmaf(b.x, y.x, fmaf(b.y, y.y, fmaf(b.z, y.z, fmaf(b.w, y.w, acc[1][s]))));
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
        if (lane == 0) {
#pragma unroll
            for (int s = 0; s < S; ++s) best[warp * S + s] = make_float2(top[s], __int_as_float(arg[s]));
        }
        dec_sync();
        auto better = [](float2& a, float2 b) { if (b.x > a.x || (b.x == a.x && __float_as_int(b.y) < __float_as_int(a.y))) a = b; };
        unsigned long long* cand = p.cand + (pos & 1) * (int)gridDim.x * S * 2;
        if (tid < S) {
            float2 b = best[tid];
#pragma unroll
            for (int j = 1; j < kDecWarps; ++j) better(b, best[j * S + tid]);
            dec_fence();  // for the keys and values of all of this CTA's threads, which the barrier above has gathered
            put_word(cand + 2 * (cta * S + tid), b.x, epoch);
            put_word(cand + 2 * (cta * S + tid) + 1, b.y, epoch);
        }
        if (warp < S) {
            float2 b = make_float2(-INFINITY, __int_as_float(0x7fffffff));
            constexpr int B = (kSMs + 31) / 32;
            float v[2 * B];
            ok = get_words<2 * B>(cand, [&](int u) { const int j = lane + 32 * (u >> 1); return j < (int)gridDim.x ? 2 * (j * S + warp) + (u & 1) : -1; }, epoch, v, p.status) && ok;
            dec_fence();
#pragma unroll
            for (int u = 0; u < B; ++u) if (lane + 32 * u < (int)gridDim.x) better(b, make_float2(v[2 * u], v[2 * u + 1]));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) better(b, make_float2(__shfl_xor_sync(0xffffffffu, b.x, o), __shfl_xor_sync(0xffffffffu, b.y, o)));
            const int t = min(__float_as_int(b.y), p.V - 1);
            if (lane == 0) {
                tok[warp] = t;
                if (cta == 0 && warp < p.n_seq) p.tokens[warp * p.tokens_ld + pos + 1] = t;
            }
        }
        if (!(ok = dec_sync_and(ok))) break;
    }
    if (!ok && tid == 0) *reinterpret_cast<volatile int*>(abort_flag) = 1;
}

template <int S>
static int launch_decode(gcb_ctx* ctx, DecodeParams& p) {
    auto kfn = gpt_decode_kernel<S>;
    p.stages = DecSmem<S>::stages(p.C, p.F);
    const size_t smem = DecSmem<S>::bytes(p.stages, p.C, p.F);
    static bool attr_done[kMaxDevices] = {};
    if (!attr_done[ctx->device]) { GCB_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDecSmemLimit)); attr_done[ctx->device] = true; }
    // small models have no work for every SM, and fewer CTAs meet faster: as many as the widest phase has tiles (or warps' worth of head rows)
    const int64_t tiles = std::max<int64_t>({(3 * (int64_t)p.C + 7) / 8, ((int64_t)p.F + 7) / 8, ((int64_t)p.V + 2 * kDecWarps - 1) / (2 * kDecWarps), (int64_t)p.n_seq * p.H});
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, kSMs);
    Scratch sc(ctx);
    const int64_t parts = (int64_t)p.n_seq * p.H * std::max<int64_t>(1, grid / ((int64_t)p.n_seq * p.H));
    auto up = [](int64_t n) { return (n + 63) / 64 * 64; };
    const int64_t n_x = up((int64_t)p.n_seq * p.C), n_qkv = up(3 * (int64_t)S * p.C), n_h = up((int64_t)p.n_seq * p.F), n_part = up(parts * (p.D + 2)), n_cand = up(4 * (int64_t)kSMs * S);
    const size_t bytes = sizeof(unsigned long long) * (size_t)(2 * n_x + n_qkv + n_h + n_part + n_cand);
    int rc = sc.get(bytes);
    if (rc) return rc;
    unsigned long long* b = sc.as<unsigned long long>();
    p.xa = b; b += n_x;
    p.xb = b; b += n_x;
    p.qkv = b; b += n_qkv;
    p.h = b; b += n_h;
    p.part = b; b += n_part;
    p.cand = b;
    GCB_CHECK_CUDA(cudaMemsetAsync(p.xa, 0, bytes, ctx->stream));  // no word belongs to a layer yet
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(kDecThreads + 32, 1, 1);
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

// Sequences the next launch takes, of n: as many as fit beside the activations in shared memory (0: not even one does).
static int64_t decode_group(int64_t n, int64_t C, int64_t F) {
    if (n > 4 && DecSmem<8>::stages(C, F)) return 8;
    if (n > 2 && DecSmem<4>::stages(C, F)) return 4;
    if (n > 1 && DecSmem<2>::stages(C, F)) return 2;
    return DecSmem<1>::stages(C, F) ? 1 : 0;
}

}  // namespace gcb

using namespace gcb;

struct gcb_gpt_decoder {
    gcb_ctx* ctx;
    DecodeParams p;
    int64_t T;
    void* maps;  // arena block: the tensor maps of the weights
};

extern "C" {

int gcb_gpt_decode_supported(gcb_ctx* ctx, const gcb_gpt_model* m) {
    if (!ctx || !m || !m->layers || m->L < 1 || m->L > kDecMaxLayers || m->H < 1 || m->C < 1 || m->F < 1 || m->V < 1 || m->C % m->H != 0 || m->C / m->H > kDecMaxHead || m->C / m->H % 4 != 0) return 0;
    if (m->V >= (int64_t(1) << 30) || m->C > 65536 || m->F > 65536 || m->C % 4 != 0 || m->F % 4 != 0 || !aligned16(m->token_embed)) return 0;
    for (int64_t l = 0; l < m->L; ++l) {
        const gcb_gpt_layer& w = m->layers[l];
        for (const float* q : {w.wq, w.wk, w.wv, w.wo, w.w1, w.w2, w.w3}) if (!aligned16(q)) return 0;
    }
    return decode_group(1, m->C, m->F) > 0 ? 1 : 0;
}

int gcb_gpt_decoder_create(gcb_ctx* ctx, const gcb_gpt_model* m, gcb_gpt_decoder** out) {
    GCB_REQUIRE(ctx && m && out && m->layers && m->token_embed && m->pos_embed && m->final_gamma, "gcb_gpt_decoder_create: NULL argument");
    *out = nullptr;
    for (int64_t l = 0; l < m->L; ++l) {
        const gcb_gpt_layer& w = m->layers[l];
        GCB_REQUIRE(w.norm1_gamma && w.wq && w.bq && w.wk && w.bk && w.wv && w.bv && w.wo && w.bo && w.norm2_gamma && w.w1 && w.b1 && w.w2 && w.b2 && (w.w3 != nullptr) == (m->layers[0].w3 != nullptr) &&
                        (w.w3 == nullptr || w.b3), "gcb_gpt_decoder_create: layer %lld has a NULL weight", (long long)l);
    }
    TmaEncodeFn enc = tma_encode(ctx);
    if (!enc || !gcb_gpt_decode_supported(ctx, m)) {
        set_error("gcb_gpt_decoder_create: at most %d layers, heads of at most %d columns, widths (of heads too) that are multiples of four and activations that fit into shared memory", kDecMaxLayers, kDecMaxHead);
        return GCB_UNSUPPORTED;
    }
    static_assert(sizeof(DecodeParams) < 32000, "kernel parameters");
    auto* d = new gcb_gpt_decoder();
    d->ctx = ctx;
    d->T = m->T;
    d->maps = nullptr;
    DecodeParams& p = d->p;
    memset(&p, 0, sizeof(p));
    p.gated = m->layers[0].w3 != nullptr;
    std::vector<CUtensorMap> maps((size_t)(m->L * kDecMaps));
    int rc = GCB_OK;
    for (int64_t l = 0; l < m->L && rc == GCB_OK; ++l) {
        const gcb_gpt_layer& w = m->layers[l];
        p.layers[l] = w;
        struct { const float* w; int64_t K, N; } mat[kDecMaps] = {{w.wq, m->C, m->C}, {w.wk, m->C, m->C}, {w.wv, m->C, m->C}, {w.wo, m->C, m->C}, {w.w1, m->C, m->F},
                                                                  {w.w2, p.gated ? m->C : m->F, p.gated ? m->F : m->C}, {w.w3, m->F, m->C}};
        for (int i = 0; i < (p.gated ? kDecMaps : kDecMaps - 1); ++i) {
            cuuint64_t dims[2] = {(cuuint64_t)mat[i].N, (cuuint64_t)mat[i].K}, strides[1] = {(cuuint64_t)mat[i].N * 4};
            cuuint32_t box[2] = {8u, (cuuint32_t)kDecBox}, estr[2] = {1u, 1u};
            if (enc(&maps[(size_t)(l * kDecMaps + i)], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(mat[i].w), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS) {
                set_error("gcb_gpt_decoder_create: a weight of layer %lld cannot be described to TMA", (long long)l);
                rc = GCB_UNSUPPORTED;
                break;
            }
        }
    }
    const size_t bytes = sizeof(CUtensorMap) * maps.size();
    if (rc == GCB_OK) {
        cudaSetDevice(ctx->device);
        std::lock_guard<std::mutex> g(ctx->mu);
        rc = ctx->arena.alloc(bytes, &d->maps);
    }
    if (rc == GCB_OK) rc = gcb_copy_h2d(ctx, d->maps, maps.data(), bytes);
    if (rc != GCB_OK) { gcb_gpt_decoder_destroy(d); return rc; }
    p.maps = static_cast<const CUtensorMap*>(d->maps);
    p.token_embed = m->token_embed; p.pos_embed = m->pos_embed; p.final_gamma = m->final_gamma; p.final_beta = m->final_beta;
    p.status = ctx->d_status;
    p.eps = m->eps;
    p.V = (int)m->V; p.C = (int)m->C; p.H = (int)m->H; p.D = (int)(m->C / m->H); p.L = (int)m->L; p.F = (int)m->F;
    p.scale = 1.0f / sqrtf((float)p.D);
    *out = d;
    return GCB_OK;
}

int gcb_gpt_decoder_destroy(gcb_gpt_decoder* d) {
    if (!d) return GCB_OK;
    int rc = GCB_OK;
    if (d->maps) {
        std::lock_guard<std::mutex> g(d->ctx->mu);
        rc = d->ctx->arena.free(d->maps);
    }
    delete d;
    return rc;
}

int gcb_gpt_decode_f32(gcb_gpt_decoder* d, int64_t n_seq, float* cache, int64_t cache_len, int64_t* tokens, int64_t tokens_ld, int64_t pos0, int64_t n_pos, int64_t n_known, float* logits) {
    GCB_REQUIRE(d && cache && tokens && aligned16(cache), "gcb_gpt_decode_f32: NULL argument, or a cache off a 16-byte boundary");
    GCB_REQUIRE(n_seq >= 0 && pos0 >= 0 && n_pos >= 0 && pos0 + n_pos <= cache_len && pos0 + n_pos <= d->T && tokens_ld >= pos0 + n_pos && n_known > pos0, "gcb_gpt_decode_f32: positions beyond the cache, the position table or the token rows");
    GCB_REQUIRE(logits == nullptr || n_known >= pos0 + n_pos, "gcb_gpt_decode_f32: with logits wanted every token of the call must be given");
    GCB_REQUIRE(logits != nullptr || n_known >= pos0 + n_pos + 1 || tokens_ld >= pos0 + n_pos + 1, "gcb_gpt_decode_f32: no room for the token that follows the last position");
    if (n_seq == 0 || n_pos == 0) return GCB_OK;
    gcb_ctx* ctx = d->ctx;
    cudaSetDevice(ctx->device);
    DecodeParams p = d->p;
    p.seq_stride = cache_len * p.C;
    p.kv_stride = n_seq * p.seq_stride;
    p.layer_stride = 2 * p.kv_stride;
    p.tokens_ld = tokens_ld;
    p.pos0 = (int)pos0; p.n_pos = (int)n_pos; p.n_known = (int)std::min<int64_t>(n_known, logits ? pos0 + n_pos : int64_t(1) << 30);
    for (int64_t s = 0; s < n_seq; s += p.n_seq) {
        const int64_t group = decode_group(n_seq - s, p.C, p.F);
        p.n_seq = (int)std::min(group, n_seq - s);
        p.cache = cache + s * p.seq_stride;
        p.tokens = tokens + s * tokens_ld;
        p.logits = logits ? logits + s * p.V : nullptr;
        const int rc = group == 8 ? launch_decode<8>(ctx, p) : group == 4 ? launch_decode<4>(ctx, p) : group == 2 ? launch_decode<2>(ctx, p) : launch_decode<1>(ctx, p);
        if (rc) return rc;
    }
    return GCB_OK;
}

}  // extern "C"
