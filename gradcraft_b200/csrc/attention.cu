// Causal attention, softmax(scale q k^T) v, in one kernel and its backward in one kernel and a GEMM, on tcgen05 / TMEM with the
// split-fp32 arithmetic of the GEMMs (one TF32 product of truncated operands + two BF16 cross products, tcgen05.cuh).
// Reference counterpart: matmul, causal_softmax and their backward nodes as composed by frontend/tensor_other.hpp:53-93.
//
// Why: through memory, scores and probabilities of 32 x 16 heads of 1024 x 1024 are written and read eight times forward and
// backward (10 GB a layer), and the kernels between them are bound by that and by splitting what they have just loaded.  Here a
// 128 x 64 block of scores lives in tensor memory from the product that makes it to the product that uses it: a thread owns one
// row, turns it into probabilities in registers and writes back the three parts (t, bf16(p), bf16(p - t)) as the A operand of the
// next product, in the place of the scores.
//
// Forward: a CTA takes two 128-query tiles that share every key block, so one tile's softmax passes behind the other's products.
//   warp 0       TMA producer: rings of two 64-key blocks of k and of v
//   warp 1       MMA issuer: S = q k^T (q: t from tensor memory, companions from shared memory), O += P v
//   warps 4..7   splitter: BF16 companions of the landed blocks (those of v transposed to K-major)
//   warps 8..15, 16..23   two threads per query of tile 0 / tile 1, 32 of a block's keys each: the query's operands, its softmax, the
//                         output row; registers move to them from the other warps (setmaxnreg)
// The running maximum is followed lazily: O and the sum are rescaled only when it has grown by 2^8, so almost never after the
// first block; the quotient is exact either way.
// Backward: a CTA takes 128 keys and walks over the queries from the diagonal on, with everything transposed (a thread owns a
// key): S^T = k q^T, dP^T = v dO^T, dV += P^T dO, dK += dS^T q.  P comes from the row maximum and reciprocal sum the forward kept.
// dS^T leaves through TMA for dQ = dS k, which is a GEMM: the one T x T matrix that goes through memory.  Products are ordered so that the tensor core has dV(i), S(i+1) to do
// while dS(i) is made and dK(i), dP(i+1) while P(i+1) is.  Four threads per key, 16 of a block's queries each; one splitter group per
// layout (one for both: 10 % slower).
// Measured, 32 x 16 heads of 1024 x 64: forward 391 us, forward + backward 1812 us (through memory: 2373 - 2480); 8 x 12 heads of 512:
// 173 (188).  2800 cycles a block forward, 7000 backward, the tensor pipe active in 37 % / 29 % of them, memory under a third of the
// copy rate; the threads between the products, which split what they have made and store it to tensor memory, were timed at 1400 and
// 3000, so that the rest of the time has no name yet.
// The tiling with a running maximum, P formed again from row statistics, and two query tiles in alternation are steps of the
// FlashAttention publications (Dao et al. 2022, Dao 2023, Shah et al. 2024).
// Every wait is bounded, as in the GEMM kernels.
#include <algorithm>

#include "tcgen05.cuh"
#include "attention_small.cuh"
#include "gemm.cuh"

namespace gcb {

constexpr int AT_ROWS = 128, AT_KEYS = 64;  // rows of tensor memory; the other side's block
constexpr int AT_FWD_THREADS = 768, AT_BWD_THREADS = 896;  // six / seven groups of four warps

struct AttnParams {
    int64_t T, D, q_ld, q_so, q_si, k_ld, k_so, k_si, v_ld, v_so, v_si, o_ld, o_so, o_si;  // backward: o_* addresses dV and dK
    const float *q, *k, *v;
    float *out, *dk, *dv;
    float *row_max, *row_inv;  // per query: maximum in log2 units, 1 / sum; pitch Tp a head, zero beyond T
    const float* delta;        // backward: dO . O per query, same pitch
    int64_t Tp;
    float scale, c;  // c = scale * log2(e)
    int H, heads, units, group, tiles_per_unit;
    int64_t items, loop_end;
    int* status;
};

struct AttnItem {
    int b, h, unit;
    bool skip;
};
// Items run from the heaviest unit of a group of heads to its lightest, dealt out in snake order (left to right, right to left), so
// that CTAs end together and a group's k and v stay in the L2 cache.  `ascending`: unit 0 is the heaviest (backward).
__device__ __forceinline__ AttnItem attn_item(const AttnParams& p, int64_t w, bool ascending) {
    AttnItem it;
    const int64_t G = gridDim.x, round = w / G, c = w - round * G, x = round * G + ((round & 1) ? G - 1 - c : c);
    it.skip = x >= p.items;
    const int64_t per_group = (int64_t)p.group * p.units;
    const int g = (int)(x / per_group), r = (int)(x - g * per_group), gh = min(p.group, p.heads - g * p.group);
    const int cls = gh > 0 ? r / gh : 0, head = g * p.group + (gh > 0 ? r - cls * gh : 0);
    it.unit = ascending ? cls : p.units - 1 - cls;
    it.b = head / p.H;
    it.h = head - it.b * p.H;
    return it;
}

template <int DP>
struct AttnSmem {
    static constexpr int TWIN = AT_ROWS * DP * 4;          // BF16 companions of a 128-row operand
    static constexpr int RAW = AT_KEYS * DP * 4;           // a landed 64-row block; its companions take as much again
    static constexpr int BLOCK = 2 * RAW;
    static constexpr int BLOCKS_OFF = 2 * TWIN;            // four blocks: forward k0 k1 v0 v1, backward q, dO (K-major), dO, q (MN-major)
    static constexpr int STAGE_OFF = BLOCKS_OFF + 4 * BLOCK;  // backward: 4 KB a warp on the way out; forward: words two threads of a row exchange
    static constexpr int BAR_OFF = STAGE_OFF + 8 * 4096;
    static constexpr int STATS_OFF = BAR_OFF + 256;        // backward: row maximum, 1 / sum and dO . O of a block's queries, two blocks
    static constexpr int TOTAL = STATS_OFF + 2 * 3 * AT_KEYS * 4 + 1024;
    static_assert(TOTAL <= 232448, "shared memory");
};

// D[128 x 64] = A[128 x DP] B[64 x DP]^T.  A: t in tensor memory, companions in shared memory; B: K-major block and companions (addresses in 16-byte units).
template <int DP>
__device__ __forceinline__ void issue_scores(uint32_t d, uint32_t a_t, uint32_t a_twin, uint32_t b_raw) {
    constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(AT_KEYS >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
    constexpr uint32_t idesc_bf = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(AT_KEYS >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
    constexpr uint32_t twin = AT_KEYS * DP * 4 / 16;
    asm volatile("" : "+r"(a_t), "+r"(a_twin), "+r"(b_raw));  // descriptors are made here, one addition each: kept across the loop they are spilled
#pragma unroll
    for (int kb = 0; kb < DP / 16; ++kb) {
        const uint32_t b = b_raw + kb * 256, a = a_twin + kb * 512;
        umma_tf32_ts(d, a_t + 16 * kb, tile_desc<16, 512, 4>(b), idesc, kb > 0 ? 1u : 0u);
        umma_tf32_ts(d, a_t + 16 * kb + 8, tile_desc<16, 512, 4>(b + 2), idesc, 1u);
        umma_bf16(d, tile_desc<128, 256, 0>(a + 256), tile_desc<128, 256, 0>(b + twin), idesc_bf, 1u);
        umma_bf16(d, tile_desc<128, 256, 0>(a), tile_desc<128, 256, 0>(b + twin + 128), idesc_bf, 1u);
    }
}
// D[128 x DP] (+)= A[128 x 64] B[64 x DP].  A: its three parts in tensor memory; B: MN-major block and K-major companions.
template <int DP>
__device__ __forceinline__ void issue_values(uint32_t d, uint32_t a_t, uint32_t a_big, uint32_t a_sml, uint32_t b_raw, bool accumulate) {
    constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (1u << 16) | ((uint32_t)(DP >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
    constexpr uint32_t idesc_bf = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(DP >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
    constexpr uint32_t twin = AT_KEYS * DP * 4 / 16;
    asm volatile("" : "+r"(a_t), "+r"(a_big), "+r"(a_sml), "+r"(b_raw));
#pragma unroll
    for (int kb = 0; kb < AT_KEYS / 16; ++kb) {
        const uint32_t b = b_raw + kb * 128, tw = b_raw + twin + kb * DP * 4;
        umma_tf32_ts(d, a_t + 16 * kb, tile_desc<8192, 512, 1>(b), idesc, (kb > 0 || accumulate) ? 1u : 0u);
        umma_tf32_ts(d, a_t + 16 * kb + 8, tile_desc<8192, 512, 1>(b + 64), idesc, 1u);
        umma_bf16_ts(d, a_sml + 8 * kb, tile_desc<128, 256, 0>(tw), idesc_bf, 1u);
        umma_bf16_ts(d, a_big + 8 * kb, tile_desc<128, 256, 0>(tw + DP * 2), idesc_bf, 1u);
    }
}
// Copies of a 64-row block starting at row r0: 16-wide slabs of 64-byte rows (K-major), or 32-wide chunks (MN-major).
template <int DP>
__device__ __forceinline__ void load_k_major(uint32_t dst, const CUtensorMap* map, uint32_t bar, int r0, int h, int b) {
    mbar_expect_tx(bar, AttnSmem<DP>::RAW);
#pragma unroll
    for (int kb = 0; kb < DP / 16; ++kb) tma_load_4d(dst + kb * 4096, map, bar, 16 * kb, r0, h, b);
}
template <int DP>
__device__ __forceinline__ void load_mn_major(uint32_t dst, const CUtensorMap* map, uint32_t bar, int r0, int h, int b) {
    mbar_expect_tx(bar, AttnSmem<DP>::RAW);
#pragma unroll
    for (int c = 0; c < DP / 32; ++c) tma_load_4d(dst + c * 8192, map, bar, 32 * c, r0, h, b);
}
template <int DP>
__device__ __forceinline__ void split_k_major(uint8_t* raw, int t) {  // a thread: one half row (8 columns) of every slab, as in split_hybrid; all loads first
    const int q = t >> 3, h = q & 1, row = (q >> 1) * 8 + (t & 7), sw = (row >> 1) & 3;
    float4 x[DP / 8];
#pragma unroll
    for (int kb = 0; kb < DP / 16; ++kb)
#pragma unroll
        for (int e = 0; e < 2; ++e) x[2 * kb + e] = *reinterpret_cast<const float4*>(raw + kb * 4096 + row * 64 + (((2 * h + e) ^ sw) << 4));
    uint8_t* big = raw + AttnSmem<DP>::RAW + (row >> 3) * 256 + h * 128 + (row & 7) * 16;
#pragma unroll
    for (int kb = 0; kb < DP / 16; ++kb) {
        const float4 a = x[2 * kb], b = x[2 * kb + 1];
        *reinterpret_cast<uint4*>(big + kb * 4096) = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
        *reinterpret_cast<uint4*>(big + kb * 4096 + 2048) = make_uint4(pack_bf16(a.x - trunc_tf32(a.x), a.y - trunc_tf32(a.y)), pack_bf16(a.z - trunc_tf32(a.z), a.w - trunc_tf32(a.w)),
                                                                       pack_bf16(b.x - trunc_tf32(b.x), b.y - trunc_tf32(b.y)), pack_bf16(b.z - trunc_tf32(b.z), b.w - trunc_tf32(b.w)));
    }
}
template <int DP>
__device__ __forceinline__ void split_mn_major(const uint8_t* raw, uint8_t* twin, int t) {  // a thread: one column, 16 rows at a time
    const int n = t % DP, j = n & 31;
#pragma unroll
    for (int kb = t / DP; kb < AT_KEYS / 16; kb += 128 / DP) {
        const uint8_t* box = raw + (n >> 5) * 8192 + kb * 2048;
        float x[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) x[k] = *reinterpret_cast<const float*>(box + k * 128 + ((((j >> 3) ^ (k & 3)) << 5) | ((j & 7) << 2)));
        uint8_t* big = twin + kb * DP * 64 + (n >> 3) * 256 + (n & 7) * 16;
#pragma unroll
        for (int kc = 0; kc < 2; ++kc) {
            const float* y = x + 8 * kc;
            *reinterpret_cast<uint4*>(big + kc * 128) = make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
            float s[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) s[e] = y[e] - trunc_tf32(y[e]);
            *reinterpret_cast<uint4*>(big + DP * 32 + kc * 128) = make_uint4(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]), pack_bf16(s[4], s[5]), pack_bf16(s[6], s[7]));
        }
    }
}
// KBS 16-column slabs of this thread's row of a 128-row A operand: from global memory, then t to tensor memory and the companions to shared memory.
template <int KBS>
__device__ __forceinline__ void load_row(float (&x)[16 * KBS], const float* src, bool live, int cols) {
#pragma unroll
    for (int e = 0; e < 4 * KBS; ++e) {
        const float4 f = live && 4 * e < cols ? ld4(src + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[4 * e] = f.x; x[4 * e + 1] = f.y; x[4 * e + 2] = f.z; x[4 * e + 3] = f.w;
    }
}
template <int KBS>
__device__ __forceinline__ void place_row(const float (&row_x)[16 * KBS], uint32_t t_addr, uint8_t* twin, int row) {
#pragma unroll
    for (int kb = 0; kb < KBS; ++kb) {
        const float* x = row_x + 16 * kb;
        uint32_t t[16];
        float s[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) { t[k] = __float_as_uint(x[k]) & 0xffffe000u; s[k] = x[k] - __uint_as_float(t[k]); }
        tmem_st16(t_addr + 16 * kb, t);
        uint8_t* big = twin + kb * 8192 + (row >> 3) * 256 + (row & 7) * 16;
#pragma unroll
        for (int kc = 0; kc < 2; ++kc) {
            const float *y = x + 8 * kc, *z = s + 8 * kc;
            *reinterpret_cast<uint4*>(big + kc * 128) = make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
            *reinterpret_cast<uint4*>(big + 4096 + kc * 128) = make_uint4(pack_bf16(z[0], z[1]), pack_bf16(z[2], z[3]), pack_bf16(z[4], z[5]), pack_bf16(z[6], z[7]));
        }
    }
}
__device__ __forceinline__ void place_parts16(const float* x, uint32_t t_addr, uint32_t big, uint32_t sml) {  // 16 columns of an A operand in tensor memory
    uint32_t t[16], b[8], s[8];
#pragma unroll
    for (int k = 0; k < 16; ++k) t[k] = __float_as_uint(x[k]) & 0xffffe000u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        b[i] = pack_bf16(x[2 * i], x[2 * i + 1]);
        s[i] = pack_bf16(x[2 * i] - __uint_as_float(t[2 * i]), x[2 * i + 1] - __uint_as_float(t[2 * i + 1]));
    }
    tmem_st16(t_addr, t);
    tmem_st8(big, b);
    tmem_st8(sml, s);
}
__device__ __forceinline__ void place_parts(const float (&x)[32], uint32_t t_addr, uint32_t big, uint32_t sml) {
    place_parts16(x, t_addr, big, sml);
    place_parts16(x + 16, t_addr + 16, big + 8, sml + 8);
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void tmem_stores_done() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int* status, int where) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, status, where)) != 0; }

template <int R>
__device__ __forceinline__ void regs_give() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void regs_take() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
__device__ __forceinline__ void pair_sync(int id) { asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory"); }
__device__ __forceinline__ bool pair_any(int id, bool x) {  // barrier of the 256 threads of a query tile, with the or of their x
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, %2, 256, p;\n\tselp.b32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"((uint32_t)x), "r"(id) : "memory");
    return r != 0;
}
__device__ __forceinline__ float max32(const float (&v)[32]) {
    float m[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) m[e] = v[e];
#pragma unroll
    for (int e = 4; e < 32; ++e) m[e & 3] = fmaxf(m[e & 3], v[e]);
    return fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]));
}

// Tensor memory, shared by both kernels: all 512 columns, taken by warp 1, given back at the end.
__device__ __forceinline__ uint32_t tmem_take(uint32_t slot, volatile uint32_t* slot_gen, int warp) {
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    after_sync();
    return *slot_gen;
}
__device__ __forceinline__ void tmem_give(uint32_t tmem, int warp) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        after_sync();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// ---- forward ------------------------------------------------------------------------------------------------------------------
// Tensor memory of query tile q, from column 256 q: scores / t of P [0, 64), bf16(P) [64, 96), bf16(P - t) [96, 128), O [128, 192), t of q [192, 256).
template <int DP>
__global__ void __launch_bounds__(AT_FWD_THREADS, 1) attention_fwd_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ AttnParams p) {
    using S = AttnSmem<DP>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + S::BAR_OFF;
    auto full = [&](int b) { return bars + 8u * b; };        // blocks k0 k1 v0 v1: landed
    auto conv = [&](int b) { return bars + 8u * (4 + b); };  // companions written
    auto empty = [&](int b) { return bars + 8u * (8 + b); }; // products have read it
    auto s_full = [&](int q) { return bars + 8u * (12 + q); };
    auto p_ready = [&](int q) { return bars + 8u * (14 + q); };
    auto o_full = [&](int q) { return bars + 8u * (16 + q); };
    auto q_ready = [&](int q) { return bars + 8u * (18 + q); };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 4; ++b) { mbar_init(full(b), 1); mbar_init(conv(b), 4); mbar_init(empty(b), 1); }
        for (int q = 0; q < 2; ++q) { mbar_init(s_full(q), 1); mbar_init(p_ready(q), 8); mbar_init(o_full(q), 1); mbar_init(q_ready(q), 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_take(bars + 8u * 20, reinterpret_cast<volatile uint32_t*>(gen + S::BAR_OFF + 8 * 20), warp);
    pdl_trigger();
    pdl_wait();
    // 64-key blocks that query tile q of an item looks at
    auto steps = [&](const AttnItem& it, int q) -> int {
        const int64_t r0 = ((int64_t)it.unit * p.tiles_per_unit + q) * AT_ROWS;
        return q < p.tiles_per_unit && r0 < p.T ? (int)((min(p.T, r0 + AT_ROWS) + AT_KEYS - 1) / AT_KEYS) : 0;
    };
    auto block_at = [&](int kind, uint32_t n) { return (int)(2 * kind + (n & 1u)); };  // kind 0: k, 1: v; n: running block number

    if (warp < 4) regs_give<56>();
    if (warp == 0) {
        if (lane == 0) {
            uint32_t n = 0;
            bool ok = true;
            for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x) {
                const AttnItem it = attn_item(p, w, false);
                if (it.skip) continue;
                const int blocks = max(steps(it, 0), steps(it, 1));
                for (int j = 0; j < blocks && ok; ++j, ++n) {
                    const uint32_t ph = ((n >> 1) & 1u) ^ 1u;
                    const int kb = block_at(0, n), vb = block_at(1, n);
                    ok = mbar_wait(empty(kb), ph, p.status, 21);
                    if (!ok) break;
                    load_k_major<DP>(base + S::BLOCKS_OFF + kb * S::BLOCK, &map_k, full(kb), j * AT_KEYS, it.h, it.b);
                    ok = mbar_wait(empty(vb), ph, p.status, 21);
                    if (!ok) break;
                    load_mn_major<DP>(base + S::BLOCKS_OFF + vb * S::BLOCK, &map_v, full(vb), j * AT_KEYS, it.h, it.b);
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t base16 = base >> 4;
            uint32_t n = 0, q_phase[2] = {0, 0}, p_phase[2] = {0, 0};
            bool ok = true;
            for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x) {
                const AttnItem it = attn_item(p, w, false);
                if (it.skip) continue;
                const int cnt[2] = {steps(it, 0), steps(it, 1)};
                const int blocks = max(cnt[0], cnt[1]);
                auto scores = [&](int q, int j) {
                    const int kb = block_at(0, n + j);
                    issue_scores<DP>(tmem + 256 * q, tmem + 256 * q + 192, base16 + q * (S::TWIN / 16), base16 + S::BLOCKS_OFF / 16 + kb * (S::BLOCK / 16));
                    umma_commit(s_full(q));
                };
                auto k_landed = [&](int j) {
                    const int kb = block_at(0, n + j);
                    const bool r = mbar_wait(conv(kb), ((n + j) >> 1) & 1u, p.status, 22);
                    after_sync();
                    return r;
                };
                for (int q = 0; q < 2 && ok; ++q)
                    if (cnt[q]) { ok = mbar_wait(q_ready(q), q_phase[q] & 1u, p.status, 23); ++q_phase[q]; }
                if (ok) ok = k_landed(0);
                if (!ok) break;
                for (int q = 0; q < 2; ++q)
                    if (cnt[q]) scores(q, 0);
                umma_commit(empty(block_at(0, n)));
                for (int j = 0; j < blocks && ok; ++j) {
                    const int vb = block_at(1, n + j);
                    const uint32_t v_raw = base16 + S::BLOCKS_OFF / 16 + vb * (S::BLOCK / 16);
                    ok = mbar_wait(conv(vb), ((n + j) >> 1) & 1u, p.status, 24);
                    bool k_here = false;
                    for (int q = 0; q < 2 && ok; ++q) {
                        if (j >= cnt[q]) continue;
                        ok = mbar_wait(p_ready(q), p_phase[q] & 1u, p.status, 25);
                        ++p_phase[q];
                        if (!ok) break;
                        after_sync();
                        const uint32_t t0 = tmem + 256 * q;
                        issue_values<DP>(t0 + 128, t0, t0 + 64, t0 + 96, v_raw, j > 0);
                        if (j + 1 < cnt[q]) {
                            if (!k_here) { ok = k_landed(j + 1); k_here = true; }
                            if (!ok) break;
                            scores(q, j + 1);
                        } else {
                            umma_commit(o_full(q));
                        }
                    }
                    umma_commit(empty(vb));
                    if (j + 1 < blocks) umma_commit(empty(block_at(0, n + j + 1)));
                }
                n += blocks;
            }
        }
    } else if (warp >= 4 && warp < 8) {
        regs_give<72>();
        const int t = threadIdx.x - 128;
        uint32_t n = 0;
        bool ok = true;
        for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x) {
            const AttnItem it = attn_item(p, w, false);
            if (it.skip) continue;
            const int blocks = max(steps(it, 0), steps(it, 1));
            for (int j = 0; j < blocks && ok; ++j, ++n) {
#pragma unroll
                for (int kind = 0; kind < 2; ++kind) {
                    const int b = block_at(kind, n);
                    ok = warp_wait(full(b), (n >> 1) & 1u, p.status, 26);
                    if (!ok) break;
                    uint8_t* raw = gen + S::BLOCKS_OFF + b * S::BLOCK;
                    if (kind == 0) split_k_major<DP>(raw, t);
                    else split_mn_major<DP>(raw, raw + S::RAW, t);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(conv(b));
                }
            }
        }
    } else if (warp >= 8) {
        regs_take<88>();
        // two threads a query: each has 32 of a block's 64 keys, and half of the columns of q and O
        const int q = (warp - 8) >> 3, half = ((warp - 8) >> 2) & 1, row = 32 * (warp & 3) + lane, bar = 1 + q;
        const uint32_t t0 = tmem + 256 * q + ((uint32_t)(32 * (warp & 3)) << 16);
        float* xch = reinterpret_cast<float*>(gen + S::STAGE_OFF) + q * 256;  // [half][row]
        constexpr int OC = DP / 2;
        uint32_t s_phase = 0, o_phase = 0;
        bool ok = true;
        for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x) {
            const AttnItem it = attn_item(p, w, false);
            if (it.skip) continue;
            const int blocks = steps(it, q);
            if (!blocks) continue;
            const int64_t r = ((int64_t)it.unit * p.tiles_per_unit + q) * AT_ROWS + row;
            const bool live = r < p.T;
            {
                float x[OC];
                load_row<DP / 32>(x, p.q + it.b * p.q_so + it.h * p.q_si + r * p.q_ld + half * OC, live, (int)p.D - half * OC);
                place_row<DP / 32>(x, t0 + 192 + half * OC, gen + q * S::TWIN + half * (OC / 16) * 8192, row);
            }
            tmem_stores_done();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(q_ready(q));
            float m = 0.0f, sum = 0.0f;  // m: the maximum the probabilities are relative to
            bool good = true;
            for (int j = 0; j < blocks; ++j) {
                good = good && warp_wait(s_full(q), s_phase & 1u, p.status, 27);  // every thread keeps step with the barriers below, whatever a wait says
                ++s_phase;
                after_sync();
                float v[32];
                tmem_ld32(t0 + 32 * half, v);
                const int64_t room = r - (int64_t)j * AT_KEYS - 32 * half;  // columns up to here are at or left of the diagonal
                if (room - lane < 31) {                                     // warp-uniform: the warp's first row
#pragma unroll
                    for (int e = 0; e < 32; ++e) v[e] = e <= room ? v[e] : -INFINITY;
                }
                float mx = max32(v);
                if (pair_any(bar, j == 0 || (mx - m) * p.c > 8.0f)) {  // almost only in the first block
                    xch[half * 128 + row] = mx;
                    pair_sync(bar);
                    mx = fmaxf(mx, xch[(half ^ 1) * 128 + row]);
                    if (j == 0) {
                        m = mx;
                    } else {  // O holds the previous blocks' sums: their products came before these scores
                        const float f = mx > m ? ex2((m - mx) * p.c) : 1.0f;
                        m = fmaxf(m, mx);
                        sum *= f;
#pragma unroll
                        for (int g = 0; g < OC / 16; ++g) {
                            uint32_t u[16];
                            tmem_ld16(t0 + 128 + half * OC + 16 * g, u);
#pragma unroll
                            for (int e = 0; e < 16; ++e) u[e] = __float_as_uint(__uint_as_float(u[e]) * f);
                            tmem_st16(t0 + 128 + half * OC + 16 * g, u);
                        }
                    }
                    pair_sync(bar);  // both have read before either writes again
                }
                const float m2 = m * p.c;
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    v[e] = ex2(fmaf(v[e], p.c, -m2));
                    acc[e & 3] += v[e];
                }
                sum += (acc[0] + acc[1]) + (acc[2] + acc[3]);
                place_parts(v, t0 + 32 * half, t0 + 64 + 16 * half, t0 + 96 + 16 * half);
                tmem_stores_done();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready(q));
            }
            good = good && warp_wait(o_full(q), o_phase & 1u, p.status, 28);
            ++o_phase;
            after_sync();
            xch[half * 128 + row] = sum;
            ok = !pair_any(bar, !good);  // all of a tile's threads leave together
            const float inv = 1.0f / (sum + xch[(half ^ 1) * 128 + row]);
            pair_sync(bar);
            if (!ok) break;
            float* dst = p.out + it.b * p.o_so + it.h * p.o_si + r * p.o_ld;
#pragma unroll
            for (int g = 0; g < OC / 16; ++g) {
                uint32_t u[16];
                tmem_ld16(t0 + 128 + half * OC + 16 * g, u);
                if (live)
#pragma unroll
                    for (int e = 0; e < 16; e += 4)
                        if (half * OC + 16 * g + e < p.D)
                            st4(dst + half * OC + 16 * g + e, make_float4(__uint_as_float(u[e]) * inv, __uint_as_float(u[e + 1]) * inv, __uint_as_float(u[e + 2]) * inv, __uint_as_float(u[e + 3]) * inv));
            }
            if (half == 0) {
                const int64_t at = ((int64_t)it.b * p.H + it.h) * p.Tp + r;
                p.row_max[at] = live ? m * p.c : 0.0f;
                p.row_inv[at] = live ? inv : 0.0f;
            }
        }
    }
    tmem_give(tmem, warp);
}

// ---- backward -----------------------------------------------------------------------------------------------------------------
// Tensor memory: S^T / t of P^T [0, 64), dP^T / t of dS^T [64, 128), P^T companions [128, 192), dS^T companions [192, 256), dV [256, 320), dK [320, 384),
// t of k [384, 448), t of v [448, 512).
template <int DP>
__global__ void __launch_bounds__(AT_BWD_THREADS, 1) attention_bwd_kernel(const __grid_constant__ CUtensorMap map_qk, const __grid_constant__ CUtensorMap map_qn, const __grid_constant__ CUtensorMap map_ok,
                                                                      const __grid_constant__ CUtensorMap map_on, const __grid_constant__ CUtensorMap map_ds, const __grid_constant__ AttnParams p) {
    using S = AttnSmem<DP>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + S::BAR_OFF;
    enum { QK = 0, OK = 1, ON = 2, QN = 3 };  // blocks: q and dO K-major for the scores and dP, dO and q MN-major for dV and dK
    auto full = [&](int b) { return bars + 8u * b; };
    auto conv = [&](int b) { return bars + 8u * (4 + b); };
    auto empty = [&](int b) { return bars + 8u * (8 + b); };
    const uint32_t s_full = bars + 8u * 12, dp_full = bars + 8u * 13, p_ready = bars + 8u * 14, ds_ready = bars + 8u * 15, acc_full = bars + 8u * 16, kv_ready = bars + 8u * 17;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int b = 0; b < 4; ++b) { mbar_init(full(b), 1); mbar_init(conv(b), 4); mbar_init(empty(b), 1); }
        mbar_init(s_full, 1); mbar_init(dp_full, 1); mbar_init(acc_full, 1);
        mbar_init(p_ready, 16); mbar_init(ds_ready, 16); mbar_init(kv_ready, 16);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t tmem = tmem_take(bars + 8u * 20, reinterpret_cast<volatile uint32_t*>(gen + S::BAR_OFF + 8 * 20), warp);
    pdl_trigger();
    pdl_wait();
    auto steps = [&](const AttnItem& it) { return (int)((p.T - (int64_t)it.unit * AT_ROWS + AT_KEYS - 1) / AT_KEYS); };
    // the order in which blocks are loaded, split and used within an item of n steps
    auto sequence = [&](int n, auto&& f) -> bool {
        if (!f((int)QK, 0) || !f((int)OK, 0)) return false;
        for (int i = 0; i < n; ++i) {
            if (!f((int)ON, i)) return false;
            if (i + 1 < n && !f((int)QK, i + 1)) return false;
            if (!f((int)QN, i)) return false;
            if (i + 1 < n && !f((int)OK, i + 1)) return false;
        }
        return true;
    };

    if (warp < 4) regs_give<64>();
    if (warp == 0) {
        if (lane == 0) {
            uint32_t n0 = 0;
            bool ok = true;
            for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x) {
                const AttnItem it = attn_item(p, w, true);
                if (it.skip) continue;
                const int n = steps(it);
                ok = sequence(n, [&](int b, int i) {
                    if (!mbar_wait(empty(b), ((n0 + i) & 1u) ^ 1u, p.status, 31)) return false;
                    const uint32_t dst = base + S::BLOCKS_OFF + b * S::BLOCK;
                    const int r0 = it.unit * AT_ROWS + i * AT_KEYS;
                    if (b == QK) load_k_major<DP>(dst, &map_qk, full(b), r0, it.h, it.b);
                    else if (b == OK) load_k_major<DP>(dst, &map_ok, full(b), r0, it.h, it.b);
                    else load_mn_major<DP>(dst, b == ON ? &map_on : &map_qn, full(b), r0, it.h, it.b);
                    return true;
                });
                n0 += n;
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t base16 = base >> 4;
            uint32_t n0 = 0, items = 0;
            bool ok = true;
            for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x, ++items) {
                const AttnItem it = attn_item(p, w, true);
                if (it.skip) break;  // only the last round has items left out
                const int n = steps(it);
                auto landed = [&](int b, int i) {
                    const bool r = mbar_wait(conv(b), (n0 + i) & 1u, p.status, 32);
                    after_sync();
                    return r;
                };
                ok = mbar_wait(kv_ready, items & 1u, p.status, 33);
                if (!ok) break;
                ok = sequence(n, [&](int b, int i) {
                    const uint32_t blk = base16 + S::BLOCKS_OFF / 16 + b * (S::BLOCK / 16), ph = (n0 + i) & 1u;
                    if (b == ON && !mbar_wait(p_ready, ph, p.status, 34)) return false;
                    if (b == QN && !mbar_wait(ds_ready, ph, p.status, 35)) return false;
                    if (!landed(b, i)) return false;
                    if (b == QK) issue_scores<DP>(tmem, tmem + 384, base16, blk);
                    else if (b == OK) issue_scores<DP>(tmem + 64, tmem + 448, base16 + S::TWIN / 16, blk);
                    else if (b == ON) issue_values<DP>(tmem + 256, tmem, tmem + 128, tmem + 160, blk, i > 0);
                    else issue_values<DP>(tmem + 320, tmem + 64, tmem + 192, tmem + 224, blk, i > 0);
                    umma_commit(empty(b));
                    if (b == QK) umma_commit(s_full);
                    else if (b == OK) umma_commit(dp_full);
                    return true;
                });
                if (!ok) break;
                umma_commit(acc_full);
                n0 += n;
            }
        }
    } else if (warp >= 4 && warp < 12) {
        regs_give<56>();
        // warps 4..7: the K-major blocks and the query statistics; warps 8..11: the MN-major blocks
        const int t = threadIdx.x & 127;
        const bool k_major = warp < 8;
        float* stats_sm = reinterpret_cast<float*>(gen + S::STATS_OFF);
        uint32_t n0 = 0;
        bool ok = true;
        for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x) {
            const AttnItem it = attn_item(p, w, true);
            if (it.skip) continue;
            const int n = steps(it);
            const int64_t at = ((int64_t)it.b * p.H + it.h) * p.Tp + (int64_t)it.unit * AT_ROWS + t;
            float nm = 0.f, ni = 0.f, nd = 0.f;  // the next block's, loaded a block ahead
            const bool keeps = k_major && t < AT_KEYS;
            if (keeps) { nm = __ldg(p.row_max + at); ni = __ldg(p.row_inv + at); nd = __ldg(p.delta + at); }
            ok = sequence(n, [&](int b, int i) {
                if (k_major != (b <= OK)) return true;
                if (!warp_wait(full(b), (n0 + i) & 1u, p.status, 36)) return false;
                uint8_t* raw = gen + S::BLOCKS_OFF + b * S::BLOCK;
                // Two slots, by the running number of the block: the one before last has been used (its products preceded the last one's, which
                // this block's copy waited for), also where the last one belongs to the item before.
                if (keeps) {
                    float* slot = stats_sm + ((n0 + i) & 1u) * 3 * AT_KEYS + t;
                    const int64_t next = at + (int64_t)(i + 1) * AT_KEYS;
                    if (b == QK) {
                        slot[0] = nm; slot[AT_KEYS] = ni;
                        if (i + 1 < n) { nm = __ldg(p.row_max + next); ni = __ldg(p.row_inv + next); }
                    } else {
                        slot[2 * AT_KEYS] = nd;
                        if (i + 1 < n) nd = __ldg(p.delta + next);
                    }
                }
                if (k_major) split_k_major<DP>(raw, t);
                else split_mn_major<DP>(raw, raw + S::RAW, t);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(conv(b));
                return true;
            });
            n0 += n;
        }
    } else if (warp >= 12) {
        regs_take<80>();
        const int part = (warp - 12) >> 2, row = 32 * (warp & 3) + lane;  // this warp: 32 keys x 16 of the block's 64 queries
        constexpr int OC = DP / 2;                                       // and half of the columns of k (parts 0, 1) or v (2, 3)
        const int half = part & 1;
        const uint32_t lanes = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
        const uint32_t stage = base + S::STAGE_OFF + (warp - 12) * 2048;
        uint8_t* stage_row = gen + S::STAGE_OFF + (warp - 12) * 2048 + lane * 64;
        uint32_t n = 0, items = 0;
        bool ok = true;
        for (int64_t w = blockIdx.x; w < p.loop_end && ok; w += gridDim.x, ++items) {
            const AttnItem it = attn_item(p, w, true);
            if (it.skip) break;
            const int64_t key = (int64_t)it.unit * AT_ROWS + row;
            const int key_warp = it.unit * AT_ROWS + 32 * (warp & 3);
            const bool live = key < p.T;
            {
                float x[OC];
                load_row<DP / 32>(x, (part < 2 ? p.k + it.b * p.k_so + it.h * p.k_si + key * p.k_ld : p.v + it.b * p.v_so + it.h * p.v_si + key * p.v_ld) + half * OC, live, (int)p.D - half * OC);
                place_row<DP / 32>(x, lanes + (part < 2 ? 384 : 448) + half * OC, gen + (part >> 1) * S::TWIN + half * (OC / 16) * 8192, row);
            }
            tmem_stores_done();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(kv_ready);
            const int cnt = steps(it);
#pragma unroll 1
            for (int i = 0; i < cnt; ++i, ++n) {
                const float4* mp = reinterpret_cast<const float4*>(gen + S::STATS_OFF + (n & 1u) * 3 * AT_KEYS * 4) + 4 * part;
                const float4 *ip = mp + AT_KEYS / 4, *dp = ip + AT_KEYS / 4;
                ok = warp_wait(s_full, n & 1u, p.status, 37);
                if (!ok) break;
                after_sync();
                uint32_t u[16];
                float pr[16];
                tmem_ld16(lanes + 16 * part, u);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float4 m = mp[e], iv = ip[e];
                    const float mm[4] = {m.x, m.y, m.z, m.w}, ii[4] = {iv.x, iv.y, iv.z, iv.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) pr[4 * e + c] = ex2(fmaf(__uint_as_float(u[4 * e + c]), p.c, -mm[c])) * ii[c];
                }
                if (i < 2) {  // the diagonal block
                    const int first = row - i * AT_KEYS - 16 * part;  // queries from here on look at this key
#pragma unroll
                    for (int e = 0; e < 16; ++e) pr[e] = e >= first ? pr[e] : 0.0f;
                }
                place_parts16(pr, lanes + 16 * part, lanes + 128 + 8 * part, lanes + 160 + 8 * part);
                tmem_stores_done();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(p_ready);
                    tma_store_wait_read<0>();  // the previous block's dS has left the staging block
                }
                ok = warp_wait(dp_full, n & 1u, p.status, 38);
                if (!ok) break;
                after_sync();
                tmem_ld16(lanes + 64 + 16 * part, u);
#pragma unroll
                for (int e = 0; e < 4; ++e) {  // dS = scale P (dP - dO . O); a masked P is zero whatever dP holds
                    const float4 d = dp[e];
                    const float dd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) pr[4 * e + c] = pr[4 * e + c] * p.scale * (__uint_as_float(u[4 * e + c]) - dd[c]);
                }
                place_parts16(pr, lanes + 64 + 16 * part, lanes + 192 + 8 * part, lanes + 224 + 8 * part);
                tmem_stores_done();
                __syncwarp();
                if (lane == 0) mbar_arrive(ds_ready);
#pragma unroll
                for (int e = 0; e < 4; ++e) *reinterpret_cast<float4*>(stage_row + ((e ^ ((lane >> 1) & 3)) << 4)) = make_float4(pr[4 * e], pr[4 * e + 1], pr[4 * e + 2], pr[4 * e + 3]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                const int q0 = it.unit * AT_ROWS + i * AT_KEYS + 16 * part;
                if (lane == 0 && q0 < p.T && key_warp < p.T) {
                    tma_store_4d(&map_ds, stage, q0, key_warp, it.h, it.b);
                    tma_store_commit();
                }
            }
            if (!ok) break;
            ok = warp_wait(acc_full, items & 1u, p.status, 39);
            if (!ok) break;
            after_sync();
            float* dst = (part < 2 ? p.dk : p.dv) + it.b * p.o_so + it.h * p.o_si + key * p.o_ld + half * OC;
#pragma unroll
            for (int g = 0; g < OC / 16; ++g) {
                uint32_t u[16];
                tmem_ld16(lanes + (part < 2 ? 320 : 256) + half * OC + 16 * g, u);
                if (live)
#pragma unroll
                    for (int e = 0; e < 16; e += 4)
                        if (half * OC + 16 * g + e < p.D) st4(dst + 16 * g + e, make_float4(__uint_as_float(u[e]), __uint_as_float(u[e + 1]), __uint_as_float(u[e + 2]), __uint_as_float(u[e + 3])));
            }
        }
        if (lane == 0) tma_store_wait_all();
    }
    tmem_give(tmem, warp);
}

// delta = dO . O per query: 16 threads a row; rows of the padding are zero.
__global__ void __launch_bounds__(256) attention_delta_kernel(float* __restrict__ delta, const float* __restrict__ g, int64_t g_ld, int64_t g_so, int64_t g_si, const float* __restrict__ o, int64_t o_ld, int64_t o_so,
                                                              int64_t o_si, int64_t T, int64_t Tp, int H, int64_t rows, int D) {
    pdl_trigger();
    pdl_wait();
    const int sub = threadIdx.x & 15;
    for (int64_t r0 = (int64_t)blockIdx.x * 16; r0 < rows; r0 += (int64_t)gridDim.x * 16) {  // rows is a multiple of 16
        const int64_t r = r0 + (threadIdx.x >> 4), head = r / Tp, row = r - head * Tp, b = head / H, h = head - b * H;
        float acc = 0.0f;
        if (row < T)
            for (int c = 4 * sub; c < D; c += 64) {
                const float4 x = ld4(g + b * g_so + h * g_si + row * g_ld + c), y = ld4(o + b * o_so + h * o_si + row * o_ld + c);
                acc = fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, fmaf(x.w, y.w, acc))));
            }
#pragma unroll
        for (int s = 8; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
        if (sub == 0) delta[r] = acc;
    }
}

// ---- host side ----------------------------------------------------------------------------------------------------------------
// (column, row, head, sequence) view of one operand in boxes of `cols` x 64.
static bool encode_rows(TmaEncodeFn enc, CUtensorMap* map, const float* ptr, int64_t cols, int64_t T, int64_t ld, int64_t si, int64_t so, int64_t H, int64_t B, int box_cols, int box_rows, CUtensorMapSwizzle swizzle) {
    const cuuint64_t row_bytes = (cuuint64_t)ld * 4;
    cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)T, (cuuint64_t)H, (cuuint64_t)B};
    cuuint64_t strides[3] = {row_bytes, H > 1 ? (cuuint64_t)si * 4 : row_bytes * (cuuint64_t)T, B > 1 ? (cuuint64_t)so * 4 : row_bytes * (cuuint64_t)T};
    cuuint32_t box[4] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1u, 1u}, estr[4] = {1, 1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
static bool rows_ok(const float* p, int64_t ld, int64_t so, int64_t si, int64_t B, int64_t H) {
    return p && aligned16(p) && ld > 0 && ld % 4 == 0 && (H == 1 || (si > 0 && si % 4 == 0)) && (B == 1 || (so > 0 && so % 4 == 0));
}
static size_t span_bytes(int64_t B, int64_t H, int64_t T, int64_t D, int64_t ld, int64_t so, int64_t si) { return sizeof(float) * (size_t)((B - 1) * so + (H - 1) * si + (T - 1) * ld + D); }
static int64_t padded(int64_t T) { return (T + AT_ROWS - 1) / AT_ROWS * AT_ROWS; }

static void plan(AttnParams& p, int64_t B, int64_t H, int64_t T, int tiles_per_unit) {
    p.H = (int)H; p.heads = (int)(B * H); p.Tp = padded(T);
    p.tiles_per_unit = tiles_per_unit;
    p.units = (int)((p.Tp / AT_ROWS + tiles_per_unit - 1) / tiles_per_unit);
    p.items = (int64_t)p.units * p.heads;
    const int64_t grid = std::min<int64_t>(p.items, kSMs);
    p.loop_end = (p.items + grid - 1) / grid * grid;
    p.group = (int)std::max<int64_t>(1, std::min<int64_t>(p.heads, 2 * grid / p.units));
}

}  // namespace gcb

using namespace gcb;

extern "C" {

int64_t gcb_attention_stats_floats(int64_t batch, int64_t heads, int64_t seq_len) { return 2 * batch * heads * padded(seq_len); }

}  // extern "C"

// Short sequences, in any split mode, while a CTA per 32 rows leaves SMs over.
constexpr int64_t kSmallT = 128;
static int64_t small_ctas(int64_t B, int64_t H, int64_t T) { return B * H * ((T + AS_OWN - 1) / AS_OWN); }
static bool takes_small(gcb_ctx* ctx, int64_t B, int64_t H, int64_t T, int64_t D) { return T <= kSmallT && T > 0 && D > 0 && D <= 128 && D % 4 == 0 && ctx->gemm_engine != 2 && small_ctas(B, H, T) <= kSMs; }

extern "C" {

// Long sequences: heads of up to 64 columns (tensor memory holds two query tiles of that width) and the split arithmetic of mode 2; TMA wants
// every stride in whole 16 bytes.  From 129 positions on this is the faster way whatever the number of heads (8 heads of 180 x 64: 94 ->
// 55 us, 768 of 130 x 48: 329 -> 303, 1024 of 192 x 64: 456 -> 393, 80 of 256 x 64:
// 99 -> 77, 512 of 256 x 64: 306 -> 283).
int gcb_attention_supported(gcb_ctx* ctx, int64_t B, int64_t H, int64_t T, int64_t D, const float* q, int64_t q_ld, int64_t q_so, int64_t q_si, const float* k, int64_t k_ld, int64_t k_so, int64_t k_si, const float* v,
                            int64_t v_ld, int64_t v_so, int64_t v_si, float scale) {
    if (!ctx || B <= 0 || H <= 0 || !rows_ok(q, q_ld, q_so, q_si, B, H) || !rows_ok(k, k_ld, k_so, k_si, B, H) || !rows_ok(v, v_ld, v_so, v_si, B, H)) return 0;
    if (takes_small(ctx, B, H, T, D)) return 1;
    return ctx->gemm_engine != 1 && ctx->gemm_split_mode == 2 && T > kSmallT && T < (int64_t(1) << 24) && D > 0 && D <= 64 && D % 4 == 0 && B * H * ((T + 127) / 128) < (int64_t(1) << 30) && scale > 0.0f && tma_encode(ctx) != nullptr;
}

// Where the short kernels pay.  A CTA's chain is as long as its tiles of 64 on the other side times their columns, and the nine launches
// that it replaces spread theirs over more CTAs.  Forward + backward in a stream of launches, separate -> fused: a chain of 64 columns
// wins at any number of heads (16 heads of 64 x 32 30 -> 20 us, 96 of 32 x 32 31 -> 20, 36 of 128 x 32 46 -> 44); one of 128 from about 60
// CTAs on (32 CTAs of 128 x 64 37 -> 40, 48 of 96 x 64 40 -> 41, 96 of 128 x 64 48 -> 42, 144 53 -> 50, 144 of 64 x 128 57 -> 48; a
// two-layer step with 12 CTAs of 96 x 64 413 -> 434 us, with 60 of 128 x 64 691 -> 685); a longer one does not (64 CTAs of 128 x 96
// 51 -> 75, 144 of 100 x 68 55 -> 79), but where a product in between meets an unlucky tile (147 CTAs of 96 x 72: 94 -> 71).
int gcb_attention_preferred(gcb_ctx* ctx, int64_t B, int64_t H, int64_t T, int64_t D) {
    if (!ctx || !ctx->fused_attention || B <= 0 || H <= 0) return 0;
    if (!takes_small(ctx, B, H, T, D)) return 1;  // whatever gcb_attention_supported takes
    const int64_t chain = (T + AS_T - 1) / AS_T * D;
    return chain <= 64 || (chain <= 128 && 5 * small_ctas(B, H, T) >= 2 * kSMs);
}

int gcb_attention_fwd_f32(gcb_ctx* ctx, int64_t B, int64_t H, int64_t T, int64_t D, float* out, int64_t o_ld, int64_t o_so, int64_t o_si, float* stats, const float* q, int64_t q_ld, int64_t q_so, int64_t q_si,
                          const float* k, int64_t k_ld, int64_t k_so, int64_t k_si, const float* v, int64_t v_ld, int64_t v_so, int64_t v_si, float scale) {
    if (!gcb_attention_supported(ctx, B, H, T, D, q, q_ld, q_so, q_si, k, k_ld, k_so, k_si, v, v_ld, v_so, v_si, scale)) return GCB_UNSUPPORTED;
    GCB_REQUIRE(rows_ok(out, o_ld, o_so, o_si, B, H) && stats && aligned16(stats), "gcb_attention_fwd_f32: output or row statistics missing or off 16-byte boundaries");
    cudaSetDevice(ctx->device);
    if (takes_small(ctx, B, H, T, D)) {
        SmallAttn a = {};
        a.q = q; a.q_ld = q_ld; a.q_so = q_so; a.q_si = q_si;
        a.k = k; a.k_ld = k_ld; a.k_so = k_so; a.k_si = k_si;
        a.v = v; a.v_ld = v_ld; a.v_so = v_so; a.v_si = v_si;
        a.out = out; a.o_ld = o_ld; a.o_so = o_so; a.o_si = o_si;
        a.Tp = padded(T); a.T = (int)T; a.D = (int)D; a.H = (int)H; a.scale = scale;
        a.row_max = stats; a.row_inv = stats + B * H * a.Tp;
        const size_t floats = as_floats(1, 2, 1, D);
        const int ctas = (int)((T + AS_OWN - 1) / AS_OWN);
        static bool one[kMaxDevices] = {}, two[kMaxDevices] = {};
        const int rc = D <= 64 ? small_launch(ctx, attention_small_fwd_kernel<1>, one, B * H, ctas, floats, a) : small_launch(ctx, attention_small_fwd_kernel<2>, two, B * H, ctas, floats, a);
        if (rc) return rc;
        note_write(ctx, out, span_bytes(B, H, T, D, o_ld, o_so, o_si));
        return after_launch(ctx, "attention_small_fwd");
    }
    TmaEncodeFn enc = tma_encode(ctx);
    AttnParams p = {};
    p.T = T; p.D = D; p.q = q; p.q_ld = q_ld; p.q_so = q_so; p.q_si = q_si;
    p.out = out; p.o_ld = o_ld; p.o_so = o_so; p.o_si = o_si;
    p.scale = scale; p.c = scale * 1.4426950408889634f; p.status = ctx->d_status;
    // two query tiles share each key block; one tile a CTA where pairs would leave SMs idle
    plan(p, B, H, T, B * H * ((T + 255) / 256) < kSMs ? 1 : 2);
    p.row_max = stats; p.row_inv = stats + B * H * p.Tp;
    CUtensorMap mk, mv;
    if (!encode_rows(enc, &mk, k, D, T, k_ld, k_si, k_so, H, B, 16, AT_KEYS, CU_TENSOR_MAP_SWIZZLE_64B) || !encode_rows(enc, &mv, v, D, T, v_ld, v_si, v_so, H, B, 32, AT_KEYS, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B))
        return GCB_UNSUPPORTED;
    const unsigned grid = (unsigned)std::min<int64_t>(p.items, kSMs);
    auto run = [&](auto kfn, size_t smem, bool* done) -> int {
        if (!done[ctx->device]) { GCB_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); done[ctx->device] = true; }
        GCB_CHECK_CUDA(launch_chained(ctx->stream, dim3(grid), AT_FWD_THREADS, smem, kfn, mk, mv, p));
        return GCB_OK;
    };
    static bool done32[kMaxDevices] = {}, done64[kMaxDevices] = {};
    const int rc = D <= 32 ? run(attention_fwd_kernel<32>, AttnSmem<32>::TOTAL, done32) : run(attention_fwd_kernel<64>, AttnSmem<64>::TOTAL, done64);
    if (rc) return rc;
    note_write(ctx, out, span_bytes(B, H, T, D, o_ld, o_so, o_si));
    return after_launch(ctx, "attention_fwd");
}

int gcb_attention_bwd_f32(gcb_ctx* ctx, int64_t B, int64_t H, int64_t T, int64_t D, float* dq, float* dk, float* dv, int64_t d_ld, int64_t d_so, int64_t d_si, const float* dout, int64_t g_ld, int64_t g_so, int64_t g_si,
                          const float* out, int64_t o_ld, int64_t o_so, int64_t o_si, const float* stats, const float* q, int64_t q_ld, int64_t q_so, int64_t q_si, const float* k, int64_t k_ld, int64_t k_so,
                          int64_t k_si, const float* v, int64_t v_ld, int64_t v_so, int64_t v_si, float scale) {
    if (!gcb_attention_supported(ctx, B, H, T, D, q, q_ld, q_so, q_si, k, k_ld, k_so, k_si, v, v_ld, v_so, v_si, scale)) return GCB_UNSUPPORTED;
    GCB_REQUIRE(rows_ok(dq, d_ld, d_so, d_si, B, H) && rows_ok(dk, d_ld, d_so, d_si, B, H) && rows_ok(dv, d_ld, d_so, d_si, B, H) && rows_ok(dout, g_ld, g_so, g_si, B, H) && rows_ok(out, o_ld, o_so, o_si, B, H) &&
                    stats && aligned16(stats), "gcb_attention_bwd_f32: operand missing or off 16-byte boundaries");
    cudaSetDevice(ctx->device);
    if (takes_small(ctx, B, H, T, D)) {
        SmallAttn a = {};
        a.q = q; a.q_ld = q_ld; a.q_so = q_so; a.q_si = q_si;
        a.k = k; a.k_ld = k_ld; a.k_so = k_so; a.k_si = k_si;
        a.v = v; a.v_ld = v_ld; a.v_so = v_so; a.v_si = v_si;
        a.g = dout; a.g_ld = g_ld; a.g_so = g_so; a.g_si = g_si;
        a.o = out; a.o_ld = o_ld; a.o_so = o_so; a.o_si = o_si;
        a.dq = dq; a.dk = dk; a.dv = dv; a.d_ld = d_ld; a.d_so = d_so; a.d_si = d_si;
        a.Tp = padded(T); a.T = (int)T; a.D = (int)D; a.H = (int)H; a.scale = scale;
        a.row_max = const_cast<float*>(stats); a.row_inv = a.row_max + B * H * a.Tp;
        const size_t floats = as_floats(2, 2, 2, D);
        const int ctas = 2 * (int)((T + AS_OWN - 1) / AS_OWN);
        static bool one[kMaxDevices] = {}, two[kMaxDevices] = {};
        const int rc = D <= 64 ? small_launch(ctx, attention_small_bwd_kernel<1>, one, B * H, ctas, floats, a) : small_launch(ctx, attention_small_bwd_kernel<2>, two, B * H, ctas, floats, a);
        if (rc) return rc;
        for (float* d : {dq, dk, dv}) note_write(ctx, d, span_bytes(B, H, T, D, d_ld, d_so, d_si));
        return after_launch(ctx, "attention_small_bwd");
    }
    TmaEncodeFn enc = tma_encode(ctx);
    AttnParams p = {};
    p.T = T; p.D = D;
    p.k = k; p.k_ld = k_ld; p.k_so = k_so; p.k_si = k_si;
    p.v = v; p.v_ld = v_ld; p.v_so = v_so; p.v_si = v_si;
    p.dk = dk; p.dv = dv; p.o_ld = d_ld; p.o_so = d_so; p.o_si = d_si;
    p.scale = scale; p.c = scale * 1.4426950408889634f; p.status = ctx->d_status;
    plan(p, B, H, T, 1);
    p.row_max = const_cast<float*>(stats); p.row_inv = p.row_max + B * H * p.Tp;
    const int64_t ld = (T + 3) / 4 * 4, rows = B * H * p.Tp;
    Scratch delta(ctx), ds(ctx);
    int rc = delta.get(sizeof(float) * (size_t)rows);
    if (!rc) rc = ds.get(sizeof(float) * (size_t)(B * H * T * ld));
    if (rc) return rc;
    p.delta = delta.as<float>();
    CUtensorMap mqk, mqn, mok, mon, mds;
    if (!encode_rows(enc, &mqk, q, D, T, q_ld, q_si, q_so, H, B, 16, AT_KEYS, CU_TENSOR_MAP_SWIZZLE_64B) || !encode_rows(enc, &mqn, q, D, T, q_ld, q_si, q_so, H, B, 32, AT_KEYS, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B) ||
        !encode_rows(enc, &mok, dout, D, T, g_ld, g_si, g_so, H, B, 16, AT_KEYS, CU_TENSOR_MAP_SWIZZLE_64B) || !encode_rows(enc, &mon, dout, D, T, g_ld, g_si, g_so, H, B, 32, AT_KEYS, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B) ||
        !encode_rows(enc, &mds, ds.as<float>(), T, T, ld, T * ld, H * T * ld, H, B, 16, 32, CU_TENSOR_MAP_SWIZZLE_64B))
        return GCB_UNSUPPORTED;
    GCB_CHECK_CUDA(launch_next(ctx->stream, dim3((unsigned)std::min<int64_t>(rows / 16, (int64_t)kSMs * 16)), 256, 0, attention_delta_kernel, delta.as<float>(), dout, g_ld, g_so, g_si, out, o_ld, o_so, o_si, T,
                               p.Tp, (int)H, rows, (int)D));
    rc = after_launch(ctx, "attention_delta");
    if (rc) return rc;
    const unsigned grid = (unsigned)std::min<int64_t>(p.items, kSMs);
    auto run = [&](auto kfn, size_t smem, bool* done) -> int {
        if (!done[ctx->device]) { GCB_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); done[ctx->device] = true; }
        GCB_CHECK_CUDA(launch_chained(ctx->stream, dim3(grid), AT_BWD_THREADS, smem, kfn, mqk, mqn, mok, mon, mds, p));
        return GCB_OK;
    };
    static bool done32[kMaxDevices] = {}, done64[kMaxDevices] = {};
    rc = D <= 32 ? run(attention_bwd_kernel<32>, AttnSmem<32>::TOTAL, done32) : run(attention_bwd_kernel<64>, AttnSmem<64>::TOTAL, done64);
    if (rc) return rc;
    note_write(ctx, dk, span_bytes(B, H, T, D, d_ld, d_so, d_si));
    note_write(ctx, dv, span_bytes(B, H, T, D, d_ld, d_so, d_si));
    rc = after_launch(ctx, "attention_bwd");
    if (rc) return rc;
    return gcb_gemm_batched_causal_f32(ctx, GCB_OP_T, GCB_OP_N, T, D, T, 1.0f, ds.as<float>(), ld, H * T * ld, T * ld, k, k_ld, k_so, k_si, 0.0f, dq, d_ld, d_so, d_si, B, H, 2);  // dQ = dS k
}

}  // extern "C"
