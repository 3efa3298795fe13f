// Products of activations with weights that stay quantised in memory, on the fifth-generation tensor cores:
//   y[m][n] = sum over scale groups g of scale[n][g] * sum over k in g of w[n][k] * x[m][k]   (+ bias[n])
// for QuantizedLinear's packed codes (2, 4 and 8 bits), the codes a decoded EOQWeight leaves, and PolarLinear's byte codes
// with a centroid table.
//
// A CTA takes 128 weight rows and up to 256 activation rows (tokens).  The weight is the A operand and lives in tensor
// memory: a thread owns one weight row, turns 64 of its codes at a time into exact 16-bit floats in registers and stores
// them to TMEM (32 columns), so that dequantised weights touch neither global nor shared memory.  The activations are the
// B operand, brought by TMA (128-byte swizzle) from the caller's matrix.  Packed codes come by TMA as well, 128 rows x
// 128 bytes at a time.
//
// Two ways to apply the scales:
//   fold    the codes are multiplied as they are (exact in fp16 and bf16); the accumulator of a scale group is read back
//           and added to the row's fp32 totals times the scale, two accumulators in turn.  No rounding of the weight at
//           all.  Activations of 32 bits go in as two fp16 halves each (twice the products), polar centroids likewise.
//   scaled  code x scale is rounded once to the activations' type, as dequantise-then-matmul does, and one accumulator
//           runs over all of K: for many tokens (up to 256 a CTA), where reading accumulators back would cost more.
//
// Warp roles: producers (four warps per set, one per TMEM lane quadrant; the sets take blocks of columns in turn), readers
// (fold and epilogue, the same quadrants), and one warp each to issue the MMAs, the weight copies and the activation
// copies and to fetch the scales.  Few row tiles: the columns are split over the CTAs of a cluster, which add their
// totals up through distributed shared memory, so there is no scratch in global memory and the order of the additions
// is fixed.
#include "eoq_internal.h"

#include <algorithm>
#include <atomic>
#include <cooperative_groups.h>
#include <cstdio>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <mutex>
#include <vector>

namespace cg = cooperative_groups;

namespace eoq {

__device__ uint32_t g_qmm_status = 0;      // set when a bounded wait ran out (a copy or a product that never completed)

namespace {

constexpr uint32_t kRows = 128;
constexpr int kPolar = 5;                  // "BITS" of the byte codes that go through a centroid table
constexpr int kBlocked4 = 6;               // "BITS" of 4-bit codes in [K / 16][rows] words of sixteen

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory"); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory"); }
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded: after about two seconds of polling the status word is set, and nobody waits for long any more.
__device__ __forceinline__ void bar_wait(uint32_t bar, uint32_t parity)
{
    if (bar_try(bar, parity)) return;
    const long long t0 = clock64();
    while (!bar_try(bar, parity))
        if (clock64() - t0 > 4000000000ll || *(volatile uint32_t *)&g_qmm_status) { g_qmm_status = 1u; return; }
}
__device__ __forceinline__ void tma_2d(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar) : "memory");
}
// One lane of the warp, the same in every call.  The loops that issue copies and products run on all lanes and elect one
// for these instructions only: their operands then stay in the warp's uniform registers (from a branch that one lane had
// taken alone, four products and two commits took 1900 cycles).
__device__ __forceinline__ bool elect()
{
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred e, p;\n\telect.sync _|e, 0xffffffff;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
                 "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// K-major tile with the 128-byte swizzle: rows of 128 bytes, groups of eight rows 1024 bytes apart
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
__device__ __forceinline__ uint32_t hsub2(uint32_t a, uint32_t b) { uint32_t r; asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) { uint32_t r; asm("mul.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t bfma2(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
__device__ __forceinline__ uint32_t bsub2(uint32_t a, uint32_t b) { uint32_t r; asm("sub.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) { uint32_t r; asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo)); return r; }
__device__ __forceinline__ uint32_t dup_byte(uint32_t w, uint32_t j) { return __byte_perm(w, 0u, 0x1111u * j); }

// Code pairs in their natural order, exact, from one word (4 bits: eight codes; 2 bits: sixteen; 8 bits: four).  A byte is
// put into both halves of a register; each half keeps its own bits under the exponent of 1024 (bf16: 128), which
// makes it 1024 + 2^s code, and one fused multiply-add with a constant pair takes the shift and the offset out: three
// instructions for two codes.  A bf16 has no mantissa bit for the upper nibble, so that one comes from the word shifted
// right by four.
template <int BITS, bool BF16>
__device__ __forceinline__ void codes_exact(uint32_t w, uint32_t *h)
{
    if (BITS == 4) {
        const uint32_t u = w >> 4;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++)
            if (BF16) h[j] = bsub2((__byte_perm(w, u, 0x4400u + 0x1111u * j) & 0x000F000Fu) | 0x43004300u, 0x43074307u);
            else h[j] = hfma2((dup_byte(w, j) & 0x00F0000Fu) | 0x64006400u, 0x2C003C00u, 0xD470E407u);
    } else if (BITS == 2) {
        const uint32_t u = w >> 4;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            if (BF16) {
                h[2 * j] = bfma2((dup_byte(w, j) & 0x000C0003u) | 0x43004300u, 0x3E803F80u, 0xC204C301u);
                h[2 * j + 1] = bfma2((dup_byte(u, j) & 0x000C0003u) | 0x43004300u, 0x3E803F80u, 0xC204C301u);
            } else {
                const uint32_t b = dup_byte(w, j);
                h[2 * j] = hfma2((b & 0x000C0003u) | 0x64006400u, 0x34003C00u, 0xDC04E401u);
                h[2 * j + 1] = hfma2((b & 0x00C00030u) | 0x64006400u, 0x24002C00u, 0xCC40D410u);
            }
        }
    } else {
        const uint32_t u = w ^ 0x80808080u;          // code + 128
#pragma unroll
        for (uint32_t j = 0; j < 2; j++) {
            if (BF16) {
                // 128 + u needs nine significant bits, a bf16 has eight: through fp32 (2^23 + u), exact
                const float f0 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7540u | (2 * j))) - 8388736.0f;
                const float f1 = __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7540u | (2 * j + 1))) - 8388736.0f;
                h[j] = pack_bf16(f0, f1);
            } else {
                h[j] = hsub2(__byte_perm(u, 0x64646464u, j ? 0x4342u : 0x4140u), 0x64806480u);
            }
        }
    }
}

// The same times the scale, rounded once: fp16 by one multiplication of the exact code; bf16 in fp32, where
// (128 + 2^s code) (scale / 2^s) - offset scale is exact in one fused multiply-add, then one rounding to the pair.
template <int BITS, bool BF16>
__device__ __forceinline__ void codes_scaled(uint32_t w, uint32_t *h, uint16_t sbits)
{
    if (!BF16) {
        codes_exact<BITS, false>(w, h);
        const uint32_t s2 = sbits | ((uint32_t)sbits << 16);
#pragma unroll
        for (int i = 0; i < 16 / BITS; i++) h[i] = hmul2(h[i], s2);
        return;
    }
    const float s = __half2float(__ushort_as_half(sbits));
    auto pair = [](uint32_t t, float m0, float c0, float m1, float c1) {
        return pack_bf16(fmaf(__uint_as_float(t << 16), m0, c0), fmaf(__uint_as_float(t & 0xFFFF0000u), m1, c1));
    };
    const uint32_t u = w >> 4;
    if (BITS == 4) {
        const float c = -135.0f * s;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) h[j] = pair((__byte_perm(w, u, 0x4400u + 0x1111u * j) & 0x000F000Fu) | 0x43004300u, s, c, s, c);
    } else if (BITS == 2) {
        const float q = 0.25f * s, c0 = -129.0f * s, c1 = -33.0f * s;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            h[2 * j] = pair((dup_byte(w, j) & 0x000C0003u) | 0x43004300u, s, c0, q, c1);
            h[2 * j + 1] = pair((dup_byte(u, j) & 0x000C0003u) | 0x43004300u, s, c0, q, c1);
        }
    } else {
        const uint32_t v = w ^ 0x80808080u;
#pragma unroll
        for (uint32_t j = 0; j < 2; j++) {
            const float f0 = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540u | (2 * j))) - 8388736.0f;
            const float f1 = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7540u | (2 * j + 1))) - 8388736.0f;
            h[j] = pack_bf16(f0 * s, f1 * s);
        }
    }
}

__device__ __forceinline__ void tmem_st32(uint32_t addr, const uint32_t (&r)[32])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
                 "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
                 ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
                   "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
                   "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
                   "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr) : "memory");
}
// The values of a load exist after this only: they go through it, so that no use can be scheduled in front of it.
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                   "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]) :: "memory");
}
