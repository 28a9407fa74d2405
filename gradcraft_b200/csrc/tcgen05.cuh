// Building blocks of the tensor-core kernels: mbarriers with bounded waits, TMA copies, tcgen05 instructions, tensor-memory access
// and the split of an fp32 operand into a TF32 part and two BF16 companions.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace gcb {

constexpr uint32_t kSpinLimit = 1u << 18;  // polls of up to ~20 us each: seconds in total, far beyond any legitimate wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// try_wait with a suspend-time hint: the thread is parked by the hardware until the phase completes or ~20 us pass, so a
// waiting role does not burn issue slots that the working roles of the same scheduler need.
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when it gave up (and records where).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status, int where) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
    }
    atomicExch(&status[0], 1);
    atomicExch(&status[1], where);
    return false;
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
                 : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1, int c2, int c3, int c4) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
                 "r"(c4)
                 : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2, int c3) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }  // the sources of all but the last N groups have been read
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Shared-memory descriptor of an operand tile whose address is given in 16-byte units.  Everything but the address is a constant, so one
// addition makes the next descriptor: the issuing thread's own instructions otherwise cost more than a narrow product (128 x 64 x 32 B: 32
// cycles in the tensor core).  LAYOUT: 0 none, 1 128-byte swizzle in 32-byte units, 2 128-byte swizzle, 4 64-byte swizzle.
template <uint32_t LBO_BYTES, uint32_t SBO_BYTES, uint32_t LAYOUT>
__device__ __forceinline__ uint64_t tile_desc(uint32_t addr16) {
    constexpr uint32_t hi = (SBO_BYTES >> 4) | (1u << 14) /* descriptor version of this architecture */ | (LAYOUT << 29);
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(addr16 + ((LBO_BYTES >> 4) << 16)), "r"(hi));
    return d;
}
// One lane of a converged warp, in a form the compiler knows to be one: tcgen05 instructions issued under it need no loop over active
// lanes (a narrow product every 32 cycles instead of every 46).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) { asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
          "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
          "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ float round_tf32(float x) {  // nearest TF32 value, returned as an fp32 with 13 zero low bits
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return __uint_as_float(r);
}

__device__ __forceinline__ float trunc_tf32(float x) { return __uint_as_float(__float_as_uint(x) & 0xffffe000u); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {  // two round-to-nearest bf16 values, `lo` at the lower address
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void umma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {  // A from tensor memory
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]),
                 "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// Split mode 2 ("TF32 + 2 x BF16"): x = t + s with t = x truncated to TF32 (what the tensor core reads from the raw tile) and
// s = x - t (exact).  a b ~ t_a t_b (one TF32 product) + bf16(s_a) bf16(b) + bf16(a) bf16(s_b) (two BF16 products at twice
// the TF32 rate): two thirds of the tensor time of three TF32 products, error ~ 2^-19 of a product instead of 2^-22,
// full fp32 exponent range.  The BF16 operands go to the twin tile of each operand (same bytes as an fp32 `small` tile):
// bf16(x) in its first half, bf16(s) in the second, both K-major without swizzle — 8-row x 16-byte core matrices,
// 128 B apart along K (LBO), 256 B apart along M / N (SBO) — whatever the raw tile's orientation.
// ROWS = rows of the operand tile (its M or N extent).  t = thread index among the 128 splitter threads.
template <bool MN, int ROWS>
__device__ __forceinline__ void split_hybrid(const uint8_t* raw, uint8_t* twin, int t, float* colsum = nullptr) {
    uint8_t* big = twin;
    uint8_t* sml = twin + ROWS * 32;
    if (!MN) {
        // raw: ROWS rows of 64 B (16 k), 16-byte chunk index XOR ((row >> 1) & 3)  [64-byte swizzle]
        // A thread takes one half row (8 k = two chunks) and writes it as one 16-byte core-matrix row of each companion.  Eight
        // consecutive lanes take eight consecutive rows of the same half: their loads fall into the eight different 16-byte
        // slots of a 128-byte bank line (that is what the swizzle is for) and so do their stores: no bank conflicts either way.
#pragma unroll
        for (int v = 0; v < ROWS / 64; ++v) {
            const int u = t + 128 * v, q = u >> 3, h = q & 1, row = (q >> 1) * 8 + (u & 7), sw = (row >> 1) & 3;
            const uint8_t* r = raw + row * 64;
            const float4 a = *reinterpret_cast<const float4*>(r + (((2 * h) ^ sw) << 4)), b = *reinterpret_cast<const float4*>(r + (((2 * h + 1) ^ sw) << 4));
            const uint32_t off = (uint32_t)(row >> 3) * 256u + (uint32_t)h * 128u + (uint32_t)(row & 7) * 16u;
            *reinterpret_cast<uint4*>(big + off) = make_uint4(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w), pack_bf16(b.x, b.y), pack_bf16(b.z, b.w));
            *reinterpret_cast<uint4*>(sml + off) = make_uint4(pack_bf16(a.x - trunc_tf32(a.x), a.y - trunc_tf32(a.y)), pack_bf16(a.z - trunc_tf32(a.z), a.w - trunc_tf32(a.w)),
                                                              pack_bf16(b.x - trunc_tf32(b.x), b.y - trunc_tf32(b.y)), pack_bf16(b.z - trunc_tf32(b.z), b.w - trunc_tf32(b.w)));
        }
    } else {
        // raw: ROWS / 32 boxes of 16 k-rows x 32 floats (128 B rows), 32-byte unit index XOR (k & 3)  [128-byte swizzle in 32-byte units]
#pragma unroll
        for (int mn = t; mn < ROWS; mn += 128) {
            const uint8_t* box = raw + (mn >> 5) * 2048;
            const int j = mn & 31;
            float x[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) x[k] = *reinterpret_cast<const float*>(box + k * 128 + ((((j >> 3) ^ (k & 3)) << 5) | ((j & 7) << 2)));
            if (colsum != nullptr)  // this thread's column over the 16 rows of the K block, pairwise, then onto the running sum (fixed order: deterministic)
                *colsum += (((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]))) + (((x[8] + x[9]) + (x[10] + x[11])) + ((x[12] + x[13]) + (x[14] + x[15])));
            const uint32_t off = (uint32_t)(mn >> 3) * 256u + (uint32_t)(mn & 7) * 16u;
#pragma unroll
            for (int kc = 0; kc < 2; ++kc) {
                const float* y = x + 8 * kc;
                float s[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) s[e] = y[e] - trunc_tf32(y[e]);
                *reinterpret_cast<uint4*>(big + off + kc * 128) = make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
                *reinterpret_cast<uint4*>(sml + off + kc * 128) = make_uint4(pack_bf16(s[0], s[1]), pack_bf16(s[2], s[3]), pack_bf16(s[4], s[5]), pack_bf16(s[6], s[7]));
            }
        }
    }
}

}  // namespace gcb
