// fp32 FMA GEMM: the engine for small products, and for operands TMA cannot address.  True fp32 arithmetic, so it also serves as
// the on-device yardstick the tensor-core engine is checked against.  Reference counterpart: cublasSgemm /
// cublasSgemmStridedBatched behind CUDAMath::apply_normal_gemm / apply_batched_gemm (backend/cuda/kernels_math.cu:725-779).
//
// What bounds a small product is latency: one trip to memory, the K loop, one trip back.  The tensor-core kernels take 12 - 13 us
// for 256 x 128 x 128 (tensor memory, descriptors and barriers are set up, each operand is split into three, and two CTAs work on
// it); here the tiles are small so that many SMs share the work, and what is still short of CTAs is cut along K as well:
//   * 32 x 32 tiles, four groups of 64 threads taking a quarter of every K block each, while 64 x 64 tiles would leave SMs idle;
//   * up to eight CTAs of a cluster take a slice of K each and add their tiles through distributed shared memory, in rank order
//     (deterministic, no scratch memory and no second launch);
//   * three K blocks of 32 in flight with cp.async; operands off 16-byte boundaries are copied in 4-byte pieces.
// An operand contiguous along K stays [row][k] in shared memory and is read four k at a time, one contiguous along M / N stays
// [k][column] and is read four columns at a time: 8 vector loads per 64 FMAs either way, without bank conflicts.
#include <algorithm>

#include "gemm.cuh"

namespace gcb {

constexpr int SG_BK = 32, SG_THREADS = 256, SG_KP = SG_BK + 4;

template <int BM>
struct SgSmem {
    static constexpr int STAGES = 3;                                  // K blocks in shared memory (six of them: 0.1 us slower)
    static constexpr int KG = BM == 32 ? 4 : 1;                       // groups of threads sharing a K block
    static constexpr int OP = BM * SG_KP > SG_BK * (BM + 4) ? BM * SG_KP : SG_BK * (BM + 4);  // floats of one operand's block
    static constexpr int LOOP = STAGES * 2 * OP, OUT = KG * BM * BM;
    static constexpr int FLOATS = (LOOP > OUT ? LOOP : OUT) + BM;     // + column sums
};

__device__ __forceinline__ void sg_copy(float* dst, const float* src, int n, bool vec, const float* safe) {  // n of four floats, the rest zero
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if (vec) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(n > 0 ? src : safe), "r"(4 * n) : "memory");
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * e), "l"(e < n ? src + e : safe), "r"(e < n ? 4 : 0) : "memory");
    }
}
// One K block of an operand: KC: stored rows x K (contiguous along k), otherwise K x rows.
template <int BM, bool KC>
__device__ __forceinline__ void sg_load(float* sm, const float* p, int64_t ld, int64_t r0, int64_t rows, int64_t k0, int64_t k_end, bool vec) {
#pragma unroll
    for (int i = 0; i < BM * SG_BK / 4 / SG_THREADS; ++i) {
        const int c = threadIdx.x + i * SG_THREADS;
        if (KC) {
            const int r = c >> 3, k = (c & 7) * 4;
            const int n = r0 + r < rows ? (int)max((int64_t)0, min((int64_t)4, k_end - k0 - k)) : 0;
            sg_copy(sm + r * SG_KP + k, p + (r0 + r) * ld + k0 + k, n, vec, p);
        } else {
            const int k = c / (BM / 4), r = (c % (BM / 4)) * 4;
            const int n = k0 + k < k_end ? (int)max((int64_t)0, min((int64_t)4, rows - r0 - r)) : 0;
            sg_copy(sm + k * (BM + 4) + r, p + (k0 + k) * ld + r0 + r, n, vec, p);
        }
    }
}
// f[i][q] = element (row i of this thread, k + q): rows t + (BM / 4) i where the block is [row][k], 4 t + i where it is [k][row]
template <int BM, bool KC>
__device__ __forceinline__ void sg_fragment(const float* sm, int t, int k, float (&f)[4][4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 v = KC ? ld4(sm + (t + (BM / 4) * i) * SG_KP + k) : ld4(sm + (k + i) * (BM + 4) + 4 * t);
        if (KC) { f[i][0] = v.x; f[i][1] = v.y; f[i][2] = v.z; f[i][3] = v.w; }
        else { f[0][i] = v.x; f[1][i] = v.y; f[2][i] = v.z; f[3][i] = v.w; }
    }
}

// Row-major C[M,N] = alpha * op(A) * op(B) + beta * C (+ bias[n]) and the epilogues of GemmArgs.  TA: A is stored K x M; TB: B is
// stored N x K.  A cluster of `slices` CTAs takes one tile.
struct SgShape {
    int tiles_m, tiles_n;
    bool a_vec, b_vec, c_vec;  // 16-byte accesses
};
template <int BM, bool TA, bool TB>
__device__ __forceinline__ void sg_tile(const GemmArgs& g, const SgShape& sh, int slices, unsigned block) {
    using S = SgSmem<BM>;
    constexpr int KG = S::KG, TPR = BM / 4, GT = TPR * TPR;  // threads along an edge of the tile, threads of a K group
    extern __shared__ __align__(16) float sg[];
    const int tiles_m = sh.tiles_m, tiles_n = sh.tiles_n;
    const bool a_vec = sh.a_vec, b_vec = sh.b_vec, c_vec = sh.c_vec;
    const int t = threadIdx.x, rank = (int)(block % (unsigned)slices);
    int64_t w = block / (unsigned)slices;
    const int64_t bz = w / ((int64_t)tiles_m * tiles_n);
    w -= bz * tiles_m * tiles_n;
    const int64_t m0 = (w / tiles_n) * BM, n0 = (w % tiles_n) * BM;
    const int64_t bo = bz / g.batch_inner, bi = bz % g.batch_inner;
    const float* A = g.A + bo * g.a_so + bi * g.a_si;
    const float* B = g.B + bo * g.b_so + bi * g.b_si;
    // a triangular output is read in 128-wide diagonal blocks and, as scores, at or below the diagonal only; the softmax backward
    // writes the zeros of those blocks, which take no product
    const bool above = g.causal == 1 && n0 > m0 + BM - 1;
    if (above && (g.sm_probs == nullptr || n0 >= (m0 / 128 + 1) * 128)) return;  // the whole cluster
    // K over several operand pairs: walked as if every group's K were whole blocks
    const int64_t per_group = (g.K + SG_BK - 1) / SG_BK * SG_BK;
    int64_t k_begin = 0, k_end = above ? 0 : g.k_groups > 1 ? per_group * g.k_groups : g.K;
    if (g.causal == 2) k_end = min(g.K, m0 + BM);
    else if (g.causal == 3) k_begin = min(g.K, m0);
    {
        const int64_t blocks = (k_end - k_begin + SG_BK - 1) / SG_BK, each = (blocks + slices - 1) / slices * SG_BK;
        const int64_t b0 = k_begin + rank * each;
        k_end = min(k_end, b0 + each);
        k_begin = b0;
    }
    const int nblk = k_end > k_begin ? (int)((k_end - k_begin + SG_BK - 1) / SG_BK) : 0;
    auto load = [&](int i) {
        if (i < nblk) {
            float* st = sg + (i % S::STAGES) * 2 * S::OP;
            int64_t k0 = k_begin + (int64_t)i * SG_BK, last = k_end;
            const float *pa = A, *pb = B;
            if (g.k_groups > 1) {
                const int64_t q = k0 / per_group;
                k0 -= q * per_group;
                last = g.K;
                pa += q * g.a_si; pb += q * g.b_si;
            }
            sg_load<BM, !TA>(st, pa, g.lda, m0, g.M, k0, last, a_vec);
            sg_load<BM, TB>(st + S::OP, pb, g.ldb, n0, g.N, k0, last, b_vec);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int grp = t / GT, tt = t % GT, tx = tt % TPR, ty = tt / TPR;
    const bool sum_cols = g.colsum != nullptr && m0 == 0;
    float acc[4][4], csum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll
    for (int i = 0; i < S::STAGES - 1; ++i) load(i);
    for (int i = 0; i < nblk; ++i) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S::STAGES - 2) : "memory");
        __syncthreads();  // block i has landed for everybody, and everybody is done with block i - 1
        load(i + S::STAGES - 1);
        const float* as = sg + (i % S::STAGES) * 2 * S::OP;
        const float* bs = as + S::OP;
#pragma unroll
        for (int k = 0; k < SG_BK / KG; k += 4) {
            float a[4][4], b[4][4];
            sg_fragment<BM, !TA>(as, ty, grp * (SG_BK / KG) + k, a);
            sg_fragment<BM, TB>(bs, tx, grp * (SG_BK / KG) + k, b);
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(a[r][q], b[c][q], acc[r][c]);
        }
        if (sum_cols && t < BM) {
#pragma unroll 8
            for (int k = 0; k < SG_BK; ++k) csum += bs[k * (BM + 4) + t];  // op(B) is stored K x N here
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // the tile, K groups side by side, in row-major order
    float* out = sg;
    float* cols = sg + (S::LOOP > S::OUT ? S::LOOP : S::OUT);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int row = TA ? 4 * ty + r : ty + TPR * r;
        float* o = out + grp * BM * BM + row * BM;
        if (!TB) st4(o + 4 * tx, make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]));
        else
#pragma unroll
            for (int c = 0; c < 4; ++c) o[tx + TPR * c] = acc[r][c];
    }
    if (sum_cols && t < BM) cols[t] = csum;
    __syncthreads();
    constexpr int VECS = BM * BM / 4;
    if (KG > 1) {
#pragma unroll
        for (int v = t; v < VECS; v += SG_THREADS) {
            float4 s = ld4(out + 4 * v);
#pragma unroll
            for (int q = 1; q < KG; ++q) { const float4 x = ld4(out + q * BM * BM + 4 * v); s.x += x.x; s.y += x.y; s.z += x.z; s.w += x.w; }
            st4(out + 4 * v, s);
        }
    }
    if (slices > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    auto remote = [&](const float* p, int r) {  // the same place in rank r's shared memory
        uint32_t a;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(r));
        return a;
    };
    float* C = g.C + bo * g.c_so + bi * g.c_si;
    const int64_t side_off = bo * g.c_so + bi * g.c_si;
    const int share = VECS / slices;  // of the tile's vectors, per rank
    for (int v = rank * share + t; v < (rank + 1) * share; v += SG_THREADS) {
        const int row = v / (BM / 4), col = (v % (BM / 4)) * 4;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        if (slices == 1) {
            s = ld4(out + 4 * v);  // KG > 1: this thread's own sum
        } else {
            float4 x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (r < slices) asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[r].x), "=f"(x[r].y), "=f"(x[r].z), "=f"(x[r].w) : "r"(remote(out + 4 * v, r)) : "memory");
#pragma unroll
            for (int r = 0; r < 8; ++r) if (r < slices) { s.x += x[r].x; s.y += x[r].y; s.z += x[r].z; s.w += x[r].w; }
        }
        const int64_t m = m0 + row, n = n0 + col;
        if (m >= g.M || n >= g.N) continue;
        float o[4] = {g.alpha * s.x, g.alpha * s.y, g.alpha * s.z, g.alpha * s.w};
        const int64_t at = m * g.ldc + n;
        const int live = (int)min((int64_t)4, g.N - n);
        const bool whole = c_vec && live == 4;
        float old[4] = {0.f, 0.f, 0.f, 0.f}, side[4] = {0.f, 0.f, 0.f, 0.f};
        const float* sp = g.residual ? g.residual : g.gelu_pre ? g.gelu_pre : g.sm_probs;
        if (whole) {
            if (g.beta != 0.0f) { const float4 x = ld4(C + at); old[0] = x.x; old[1] = x.y; old[2] = x.z; old[3] = x.w; }
            if (sp) { const float4 x = ld4(sp + side_off + at); side[0] = x.x; side[1] = x.y; side[2] = x.z; side[3] = x.w; }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) if (e < live) { if (g.beta != 0.0f) old[e] = C[at + e]; if (sp) side[e] = sp[side_off + at + e]; }
        }
        const float rd = g.sm_probs ? g.sm_rowdot[bz * g.M + m] : 0.0f;
        float act[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (g.bias && e < live) o[e] += g.bias[bi * g.bias_si + n + e];
            if (g.beta != 0.0f) o[e] += g.beta * old[e];
            if (g.residual) o[e] += side[e];
            else if (g.gelu_pre) o[e] *= gelu_grad_f(side[e]);
            else if (g.sm_probs) o[e] = n + e <= m ? g.sm_scale * side[e] * (o[e] - rd) : 0.0f;
            act[e] = g.gelu_act ? gelu_f(o[e]) : 0.0f;
        }
        if (whole) {
            st4(C + at, make_float4(o[0], o[1], o[2], o[3]));
            if (g.gelu_act) st4(g.gelu_act + side_off + at, make_float4(act[0], act[1], act[2], act[3]));
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) if (e < live) { C[at + e] = o[e]; if (g.gelu_act) g.gelu_act[side_off + at + e] = act[e]; }
        }
    }
    if (sum_cols && rank == 0 && t < BM && n0 + t < g.N) {
        float s = 0.0f;
        for (int r = 0; r < slices; ++r) {
            float x;
            if (slices == 1) x = cols[t];
            else asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x) : "r"(remote(cols + t, r)) : "memory");
            s += x;
        }
        float* d = g.colsum + bi * g.colsum_si + n0 + t;
        *d = g.colsum_accumulate ? *d + s : s;
    }
    if (slices > 1) {  // nobody leaves while its shared memory is still read
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

template <int BM, bool TA, bool TB>
__global__ void __launch_bounds__(SG_THREADS) gemm_simt_kernel(const GemmArgs g, const SgShape sh, int slices) {
    pdl_trigger();
    pdl_wait();
    sg_tile<BM, TA, TB>(g, sh, slices, blockIdx.x);
}
// A linear layer's dX = dY W^T and dW = X^T dY side by side: neither waits for the other, and in a small model each is a launch of
// 5 - 6 us that leaves most SMs idle (two-layer step: 13 launches less).
template <int BM>
__global__ void __launch_bounds__(SG_THREADS) gemm_simt_backward_kernel(const GemmArgs dx, const SgShape dx_sh, const GemmArgs dw, const SgShape dw_sh, int slices, unsigned dx_blocks) {
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x < dx_blocks) sg_tile<BM, false, true>(dx, dx_sh, slices, blockIdx.x);
    else sg_tile<BM, true, false>(dw, dw_sh, slices, blockIdx.x - dx_blocks);
}

static SgShape sg_shape(const GemmArgs& g, int bm) {
    auto ok4 = [](int64_t v) { return v % 4 == 0; };
    auto vec = [&](const float* p, int64_t ld, int64_t so, int64_t si) { return aligned16(p) && ok4(ld) && ((g.batch_inner == 1 && g.k_groups == 1) || ok4(si)) && (g.batch_outer == 1 || ok4(so)); };
    const bool c_vec = vec(g.C, g.ldc, g.c_so, g.c_si) && aligned16(g.residual) && aligned16(g.gelu_pre) && aligned16(g.gelu_act) && aligned16(g.sm_probs);
    return {(int)((g.M + bm - 1) / bm), (int)((g.N + bm - 1) / bm), vec(g.A, g.lda, g.a_so, g.a_si), vec(g.B, g.ldb, g.b_so, g.b_si), c_vec};
}
static int64_t sg_tiles(const GemmArgs& g, int64_t bm) { return ((g.M + bm - 1) / bm) * ((g.N + bm - 1) / bm) * g.batch_outer * g.batch_inner; }
// K is cut while SMs are left over and every slice keeps two K blocks; beyond one CTA per SM only for slices of 96 and more
// (256 x 512 x 128: one slice 5.5 us, two 6.4; 256 x 256 x 512: one 10.8, two 8.3, four 7.7, eight 12.9)
static int sg_slices(int64_t tiles, int64_t K) {
    int slices = 1;
    while (slices < 8 && K >= (int64_t)slices * 2 * 2 * SG_BK && tiles * slices * 2 <= (K >= (int64_t)slices * 2 * 96 ? 2 * kSMs : kSMs)) slices *= 2;
    return slices;
}
template <int BM, class... P, class... Args>
static int sg_launch(gcb_ctx* ctx, bool* attr_done, void (*kfn)(P...), int64_t tiles, int slices, Args... args) {
    constexpr size_t smem = sizeof(float) * SgSmem<BM>::FLOATS;
    // attr_done: function attributes belong to a device
    if (smem > 48 * 1024 && !attr_done[ctx->device]) { GCB_CHECK_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)); attr_done[ctx->device] = true; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * slices), 1, 1);
    cfg.blockDim = dim3(SG_THREADS, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)slices;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = slices > 1 ? 2 : 1;
    GCB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kfn, args...));
    return GCB_OK;
}
template <int BM, bool TA, bool TB>
static int sg_run(gcb_ctx* ctx, const GemmArgs& g, int64_t tiles, int slices) {
    static bool done[kMaxDevices] = {};
    return sg_launch<BM>(ctx, done, gemm_simt_kernel<BM, TA, TB>, tiles, slices, g, sg_shape(g, BM), slices);
}

int gemm_simt_launch(gcb_ctx* ctx, bool ta, bool tb, const GemmArgs& g) {
    const int64_t batches = g.batch_outer * g.batch_inner;
    if (g.M == 0 || g.N == 0 || batches == 0) return GCB_OK;
    if (g.colsum && tb) { set_error("gemm (FMA): column sums need op(B) stored K x N"); return GCB_UNSUPPORTED; }
    // 64-wide tiles read shared memory and L2 half as often per FMA: they are taken once they fill the chip by themselves
    const int bm = sg_tiles(g, 64) >= kSMs ? 64 : 32;
    const int64_t tiles = sg_tiles(g, bm);
    GCB_REQUIRE(tiles <= 0x7fffffff / 8, "gemm (FMA): grid too large");
    const int slices = sg_slices(tiles, g.K * g.k_groups);
    cudaSetDevice(ctx->device);
    int rc;
#define GCB_SG(BMV) (!ta && !tb ? sg_run<BMV, false, false>(ctx, g, tiles, slices) : !ta ? sg_run<BMV, false, true>(ctx, g, tiles, slices) \
                     : !tb ? sg_run<BMV, true, false>(ctx, g, tiles, slices) : sg_run<BMV, true, true>(ctx, g, tiles, slices))
    rc = bm == 64 ? GCB_SG(64) : GCB_SG(32);
#undef GCB_SG
    if (rc) return rc;
    ctx->last_gemm_engine = 1;
    return after_launch(ctx, "gemm_simt");
}

// dX (op N, T) and dW (op T, N) in one launch; both with the 32-wide tiles.  False: too large for that.
bool gemm_simt_backward_fits(const GemmArgs& dx, const GemmArgs& dw) { return sg_tiles(dx, 64) + sg_tiles(dw, 64) < kSMs; }
int gemm_simt_backward_launch(gcb_ctx* ctx, const GemmArgs& dx, const GemmArgs& dw) {
    const int64_t t0 = sg_tiles(dx, 32), t1 = sg_tiles(dw, 32);
    const int slices = sg_slices(t0 + t1, std::min(dx.K * dx.k_groups, dw.K));
    cudaSetDevice(ctx->device);
    static bool done[kMaxDevices] = {};
    const int rc = sg_launch<32>(ctx, done, gemm_simt_backward_kernel<32>, t0 + t1, slices, dx, sg_shape(dx, 32), dw, sg_shape(dw, 32), slices, (unsigned)(t0 * slices));
    if (rc) return rc;
    ctx->last_gemm_engine = 1;
    return after_launch(ctx, "gemm_simt_backward");
}

}  // namespace gcb
