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
// (fold, the same quadrants; at the end of `scaled` both take the accumulator to shared memory: 200 bf16 rows in groups of 128
// against 11008 x 4096 34.3 us with the readers alone, 31.6), and one warp each to issue the MMAs, the weight copies and the activation
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

// Set when a bounded wait ran out (a copy or a product that never completed), unless the call has a status word of its own.
__device__ uint32_t g_qmm_status = 0;

namespace {

constexpr uint32_t kRows = 128;
constexpr int kPolar = 5;                  // "BITS" of the byte codes that go through a centroid table
constexpr int kPolarRot = 7;               // the same in blocks of 64, rotated here: every 64 values of a row times the Hadamard matrix
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
struct QmmArgs {
    const uint16_t *scales;      // [N][K / group] fp16 (polar: norms)
    const float *centroids;      // polar: `entries` of them
    const void *bias;            // [N] fp32 (bias_half: fp16), or null
    const float *tok_scale;      // [M] factor of every activation row, or null
    void *y;                     // [M][N]
    uint32_t N, K, M, T, group, sgroups, seg, units, split, planes, entries;
    uint32_t nw, ns, nd, a_base; // stages of packed weights and of operands (A in TMEM, activations in shared memory); accumulators; first A column
    uint32_t at_x, at_bar;       // shared-memory offsets
    int y_dtype, bias_half, late;   // late: the packed codes are the previous kernel's to write
    long long limit;             // clock ticks a wait may take
    uint32_t *status;            // word to set when one runs out, or null: g_qmm_status
};

// Waits are bounded.  One that runs out marks the CTA, which ends the waits of all its warps, and sets the status word; the
// warps run on with whatever is there, only that nobody requests copies any more, nor tells the barriers that count a copy's
// bytes (an arrival beyond their count while a copy is under way would break them).  The CTA's results become NaN.  Nothing
// of that outlives the launch but the word: later launches wait as ever, only an eighth as long (a grid of many rounds would
// otherwise take the full limit in each).
//   The time of a kernel before this one, which programmatic launch may leave running for as long as it likes, does not
// count.  (A limit of 0 has no patience with them either.)
//   The outcome of a wait is not returned for every warp to leave its loop by: that alone costs the products' warp some
// eighty cycles a block (24 rows against 11008 x 4096: 17.9 instead of 17.0 us).  What follows a first failed attempt is a
// function of its own, out of the loops' way: 16.2 us (inline 17.0); four rows against a polar 14336 x 4096 36.0 (37.5).  Not so
// in loops that keep more in registers than a call leaves alone (`near`: the readers, and the polar producers of the variants
// with 20 warps), which cost up to 40 % by the call (100 rows in groups of 32: 88.5 us, now 56.9).
struct Waits {
    uint32_t mark;               // shared address of two words: the CTA has given up; the kernels before this one have ended
    const QmmArgs &a;            // (read where it is needed: the readers have no registers to spare)
    __device__ __forceinline__ uint32_t *status() const { return a.status ? a.status : &g_qmm_status; }
    __device__ __forceinline__ bool stopped() const
    {
        uint32_t v;
        asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(mark) : "memory");
        return v != 0;
    }
    __device__ __forceinline__ void operator()(uint32_t bar, uint32_t parity) const
    {
        if (!bar_try(bar, parity)) slow(bar, parity, mark, a.limit, status());
    }
    // The same, and whether the CTA has not given up: asked for together, in one latency.
    template <bool NEAR = false>
    __device__ __forceinline__ bool go(uint32_t bar, uint32_t parity) const
    {
        uint32_t ok, stop;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%2], %3;\n\tld.volatile.shared.u32 %1, [%4];\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok), "=r"(stop) : "r"(bar), "r"(parity), "r"(mark) : "memory");
        if (ok) return stop == 0;
        if (NEAR) poll(bar, parity, mark, a.limit, status());
        else slow(bar, parity, mark, a.limit, status());
        return !stopped();
    }
    // The same with what follows a failed attempt in its place.
    __device__ __forceinline__ void near(uint32_t bar, uint32_t parity) const
    {
        if (!bar_try(bar, parity)) poll(bar, parity, mark, a.limit, status());
    }
    static __device__ __noinline__ void slow(uint32_t bar, uint32_t parity, uint32_t mark, long long limit, uint32_t *status)
    {
        poll(bar, parity, mark, limit, status);
    }
    static __device__ __forceinline__ void poll(uint32_t bar, uint32_t parity, uint32_t mark, long long limit, uint32_t *status)
    {
        long long t0 = clock64();
        while (!bar_try(bar, parity)) {
            const long long now = clock64();
            uint32_t stop, alone;
            asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(stop), "=r"(alone) : "r"(mark) : "memory");
            if (!alone && limit) t0 = now;
            if (!stop && now - t0 <= limit && !(now - t0 > limit / 8 && *reinterpret_cast<volatile uint32_t *>(status))) continue;
            asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(mark), "r"(1u) : "memory");
            *reinterpret_cast<volatile uint32_t *>(status) = 1u;
            return;
        }
    }
};
// The last uses of a ring of n barriers, of which `used` have been made: what the copy engine still has to bring is
// there (or does not come for some ten milliseconds) before the CTA may leave its shared memory.
__device__ __forceinline__ void drain(uint32_t bar, uint32_t used, uint32_t n)
{
    const long long t0 = clock64();
    for (uint32_t u = used > n ? used - n : 0u; u < used; u++)
        while (!bar_try(bar + 8u * (u % n), (u / n) & 1u))
            if (clock64() - t0 > 20000000ll) return;
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
// (a & b) | c in one instruction (from two immediate operands the compiler makes two, of the half-rate pipe that bounds the conversions)
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
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
            if (BF16) h[j] = bsub2(and_or(__byte_perm(w, u, 0x4400u + 0x1111u * j), 0x000F000Fu, 0x43004300u), 0x43074307u);
            else h[j] = hfma2(and_or(dup_byte(w, j), 0x00F0000Fu, 0x64006400u), 0x2C003C00u, 0xD470E407u);
    } else if (BITS == 2) {
        const uint32_t u = w >> 4;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            if (BF16) {
                h[2 * j] = bfma2(and_or(dup_byte(w, j), 0x000C0003u, 0x43004300u), 0x3E803F80u, 0xC204C301u);
                h[2 * j + 1] = bfma2(and_or(dup_byte(u, j), 0x000C0003u, 0x43004300u), 0x3E803F80u, 0xC204C301u);
            } else {
                const uint32_t b = dup_byte(w, j);
                h[2 * j] = hfma2(and_or(b, 0x000C0003u, 0x64006400u), 0x34003C00u, 0xDC04E401u);
                h[2 * j + 1] = hfma2(and_or(b, 0x00C00030u, 0x64006400u), 0x24002C00u, 0xCC40D410u);
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
        for (uint32_t j = 0; j < 4; j++) h[j] = pair(and_or(__byte_perm(w, u, 0x4400u + 0x1111u * j), 0x000F000Fu, 0x43004300u), s, c, s, c);
    } else if (BITS == 2) {
        const float q = 0.25f * s, c0 = -129.0f * s, c1 = -33.0f * s;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) {
            h[2 * j] = pair(and_or(dup_byte(w, j), 0x000C0003u, 0x43004300u), s, c0, q, c1);
            h[2 * j + 1] = pair(and_or(dup_byte(u, j), 0x000C0003u, 0x43004300u), s, c0, q, c1);
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

// two fp32 in a register pair
__device__ __forceinline__ uint64_t pack2(float a, float b) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float low2(uint64_t v) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return a; }
__device__ __forceinline__ float high2(uint64_t v) { float a, b; asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); return b; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) { uint64_t r; asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }

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

template <int BITS, int KB>
struct Unit {                    // what one weight copy brings: 128 rows of kBytes, in blocks of KB columns (a stage of operands)
    static constexpr uint32_t kBytes = BITS == 2 ? 64u : 128u;
    static constexpr uint32_t kCols = BITS == 2 || BITS == 4 || BITS == kBlocked4 ? 256u : 128u;
    static constexpr uint32_t kBlocks = kCols / KB;
    static constexpr uint32_t kStage = kRows * kBytes;
    static constexpr int kWords = BITS == 4 || BITS == kBlocked4 ? 8 : BITS == 2 ? 4 : 16;       // words of one row and 64 columns
};

// Position in a ring of n stages and the parity of its current lap.
struct Ring {
    uint32_t at = 0, lap = 0;
    __device__ __forceinline__ void next(uint32_t n) { if (++at == n) { at = 0; lap ^= 1u; } }
};

// barriers, in this order, eight bytes each
enum { kWFull = 0, kWEmpty = 8, kFull = 16, kEmpty = 24, kDFull = 32, kDEmpty = 36, kSFull = 40, kSEmpty = 44, kTmemSlot = 48, kDrain = 49, kMark = 50, kUsedW = 51, kUsedX = 52 };
constexpr uint32_t kScaleRing = 4, kScaleGroups = 8, kScaleEntry = kScaleGroups * kRows * 2u;      // scales of 8 groups x 128 rows an entry

// The scales of one weight row in the order of the groups, out of the ring that a warp of the CTA keeps filled.
template <bool NEAR>
struct ScaleReader {
    uint32_t full, empty, at, row, entry = 0;      // barrier addresses, ring address
    Ring ring;
    bool here = false;                             // this entry has been waited for
    const Waits &wait;
    __device__ __forceinline__ ScaleReader(const Waits &w, uint32_t f, uint32_t e, uint32_t a, uint32_t r) : full(f), empty(e), at(a), row(r), wait(w) {}
    __device__ __forceinline__ uint16_t get(uint32_t g, uint32_t lane)      // g: group, counted from the CTA's first
    {
        while ((g >> 3) > entry) {
            __syncwarp();
            if (lane == 0) bar_arrive(empty + 8u * ring.at);
            ring.next(kScaleRing);
            entry++;
            here = false;
        }
        if (!here) {
            if (NEAR) wait.near(full + 8u * ring.at, ring.lap);
            else wait(full + 8u * ring.at, ring.lap);
            here = true;
        }
        uint16_t v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(at + ring.at * kScaleEntry + (g & 7u) * (kRows * 2u) + row * 2u));
        return v;
    }
};

template <int BITS, bool BF16, bool FOLD, int NP, int NF, int TC, int KB>
__global__ void __launch_bounds__((4 * NP + 4 * NF + 4) * 32, 1)
qmm_kernel(const QmmArgs a, const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap)
{
    using U = Unit<BITS, KB>;
    constexpr bool kRot = BITS == kPolarRot, kPol = BITS == kPolar || kRot;
    static_assert(!kRot || (!FOLD && KB == 64), "a thread rotates one block of 64 columns");
    constexpr int kCode = kPol ? 8 : BITS == kBlocked4 ? 4 : BITS;
    constexpr uint32_t kHalves = KB / 64;                         // 64-column parts of a block
    constexpr uint32_t kACols = (kPol ? 64u : 32u) * kHalves;     // TMEM columns of a block (polar: high and low halves)
    constexpr uint32_t kB16 = KB / 16;                            // products (K = 16) of a block
    constexpr uint32_t kTmem = 512u;
    extern __shared__ uint8_t raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(raw) + 1023u) & ~(uintptr_t)1023u);
    const uint32_t base = saddr(smem), bars = base + a.at_bar;
    auto bar = [&](uint32_t i) { return bars + 8u * i; };
    const Waits wait{bars + 8u * kMark, a};
    auto word = [&](uint32_t i) { return reinterpret_cast<volatile uint32_t *>(smem + a.at_bar + 8u * i); };
    const uint32_t scale_ring = bars + 512u;
    uint32_t *table = reinterpret_cast<uint32_t *>(smem + a.at_bar + 512 + kScaleRing * kScaleEntry);      // polar: centroids, as {high half, low half} (fold) or fp32
    uint32_t *largest = table + 256;              // polar, scaled: the largest norm of each row (bits of a float), then the largest centroid
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31u;       // the same in all lanes, and known to be
    const uint32_t rank = blockIdx.x % a.split, row0 = blockIdx.x / a.split * kRows, tok0 = blockIdx.y * a.T;
    const uint32_t u0 = (uint32_t)((uint64_t)a.units * rank / a.split), u1 = (uint32_t)((uint64_t)a.units * (rank + 1) / a.split);
    const uint32_t kb0 = u0 * U::kBlocks, nkb = min(u1 * U::kBlocks, (a.K + KB - 1) / KB) - kb0;
    const uint32_t k16_0 = kb0 * kB16, k16_n = min((kb0 + nkb) * kB16, a.K / 16u), g16 = a.group / 16u;
    const uint32_t grp0 = k16_0 / g16, ngroups = (k16_n - 1u) / g16 - grp0 + 1u;
    // fold: an accumulator runs over `seg` columns, a group or an equal part of a long one (of 128 at most: the tensor cores
    // round each addition towards zero, which 1024 columns of byte codes show: 2e-6 against 3e-7)
    const uint32_t f16 = a.seg / 16u, seg0 = k16_0 / f16, nseg = (k16_n - 1u) / f16 - seg0 + 1u;
    const uint32_t plane = a.T * 128u * kHalves, xstage = plane * a.planes;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < 8; i++) {
            bar_init(bar(kWFull + i), 1); bar_init(bar(kWEmpty + i), 4 * U::kBlocks);
            bar_init(bar(kFull + i), 5); bar_init(bar(kEmpty + i), 1);          // four producer warps and the activation copy
        }
        for (uint32_t i = 0; i < kScaleRing; i++) { bar_init(bar(kSFull + i), 1); bar_init(bar(kSEmpty + i), 4 * (FOLD ? NF : NP)); }
        for (uint32_t i = 0; i < 4; i++) { bar_init(bar(kDFull + i), 1); bar_init(bar(kDEmpty + i), 4 * NF); }
        bar_init(bar(kDrain), 1);
        word(kMark)[0] = word(kMark)[1] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (kPol) {
        for (uint32_t i = threadIdx.x; i < 256u; i += blockDim.x) {
            const float c = __ldg(a.centroids + (i & (a.entries - 1u)));
            const __half hi = __float2half_rn(c), lo = __float2half_rn(c - __half2float(hi));
            table[i] = FOLD ? __half_as_ushort(hi) | ((uint32_t)__half_as_ushort(lo) << 16) : __float_as_uint(c);
        }
        if (!FOLD) for (uint32_t i = threadIdx.x; i < kRows + 1u; i += blockDim.x) largest[i] = 0u;
    }
    __syncwarp();
    if (warp == 4 * NP + 4 * NF) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bar(kTmemSlot)), "n"(kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    // all 512 columns are this CTA's, so they start at column 0: addresses below are constants plus offsets
    constexpr uint32_t tmem = 0;

    // polar, scaled: what a row's values are multiplied by, a power of two that brings the largest of centroid x norm to
    // 2^14 .. 2^15, so that their two fp16 halves hold 22 bits of it and nothing of it is below what fp16 holds
    float up = 1.0f, down = 1.0f;
    if (kPol && !FOLD && warp < 4 * NP + 4 * NF) {
        const uint32_t r = (warp & 3u) * 32u + lane;
        if (warp < 4 * NP) {
            const uint16_t *norms = a.scales + (size_t)min(row0 + r, a.N - 1u) * a.sgroups + grp0;
            float most = 0.0f;
            auto larger = [&](uint32_t bits) { most = fmaxf(most, fabsf(__half2float(__ushort_as_half((uint16_t)bits)))); };
            if (((reinterpret_cast<uintptr_t>(a.scales) | a.sgroups * 2u | grp0 * 2u | ngroups * 2u) & 15u) == 0) {
                // eight a load (64 norms a row one at a time: 7 of the 187 us of 512 rows against 14336 x 4096)
#pragma unroll 4
                for (uint32_t g = (warp >> 2) * 8u; g < ngroups; g += NP * 8u) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(norms + g));
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) { larger(w[i] & 0xFFFFu); larger(w[i] >> 16); }
                }
            } else {
#pragma unroll 16
                for (uint32_t g = warp >> 2; g < ngroups; g += NP) larger(__ldg(norms + g));
            }
            atomicMax(largest + r, __float_as_uint(most));
            if (threadIdx.x < 256u) atomicMax(largest + kRows, table[threadIdx.x] & 0x7fffffffu);
        }
        asm volatile("bar.sync 1, %0;" ::"n"((4 * NP + 4 * NF) * 32) : "memory");
        const float most = __uint_as_float(largest[r]) * __uint_as_float(largest[kRows]);
        int e = 0;
        if (most > 0.0f && most < __int_as_float(0x7f800000)) e = min(120, 141 - (int)(__float_as_uint(most) >> 23));
        up = __uint_as_float((uint32_t)(127 + e) << 23);
        down = __uint_as_float((uint32_t)(127 - e) << 23);
    }

    if (warp < 4 * NP) {
        // ---- producers: packed codes of one row, a block of columns at a time, to the A operand in tensor memory
        const uint32_t set = warp >> 2, r = (warp & 3u) * 32u + lane;
        const uint32_t lane_base = tmem + (((warp & 3u) * 32u) << 16) + a.a_base;
        uint32_t four;
        asm volatile("mov.b32 %0, 4;" : "=r"(four));
        // a code to its table entry in one instruction: the dot product of the word's four codes with 4 at the code's place, on
        // top of the table's address (4 rows against 14336 x 4096 36.0 -> 32.0 us with the four accumulators of few tokens; with
        // two reader sets, where the readers bound it, 1 % slower than a byte permute and a multiply-add: 108 rows against
        // 13338 x 896 19.5 / 19.3); the table repeats up to 256 entries
        const uint32_t tab_addr = saddr(table);
        auto entry = [&](uint32_t word, uint32_t b) {
            uint32_t off;
            if (NF == 1) asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(off) : "r"(word), "r"(4u << (8 * b)), "r"(tab_addr));
            else asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(off) : "r"(__byte_perm(word, 0u, 0x4440u + b)), "r"(four), "r"(tab_addr));
            return off;
        };
        // scaled: the groups of 32-column parts, counted along
        ScaleReader<false> sr(wait, bar(kSFull), bar(kSEmpty), scale_ring, r);
        uint32_t gi = 0, pos = 0;
        if (!FOLD) {
            const uint32_t c = (kb0 + set) * KB;
            gi = c / a.group; pos = c - gi * a.group; gi -= grp0;
        }
        Ring wr, ar;
        uint32_t unit = 0;
        for (uint32_t j = 0; j < set; j++) ar.next(a.ns);
        for (uint32_t i = set; i < nkb; i += NP) {
            const uint32_t q = i % U::kBlocks, st = ar.at;
            for (; unit < i / U::kBlocks; unit++) wr.next(a.nw);
            const uint32_t ws = wr.at, row_at = base + ws * U::kStage + r * U::kBytes;
            const uint32_t sw = BITS == 2 ? (r >> 1) & 3u : r & 7u;
            wait(bar(kWFull + ws), wr.lap);
            bool go = true;
#pragma unroll
            for (uint32_t part = 0; part < kHalves; part++) {
                uint32_t w[U::kWords];
                if (BITS == kBlocked4) {
#pragma unroll
                    for (uint32_t c = 0; c < U::kWords / 2; c++)
                        asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];" : "=r"(w[2 * c]), "=r"(w[2 * c + 1])
                                     : "r"(base + ws * U::kStage + ((q * kHalves + part) * 4u + c) * (kRows * 8u) + r * 8u));
                }
#pragma unroll
                for (uint32_t c = 0; c < (BITS == kBlocked4 ? 0u : U::kWords / 4); c++) {
                    const uint32_t at = row_at + ((((q * kHalves + part) * (U::kWords / 4) + c) ^ sw) << 4);
                    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[4 * c]), "=r"(w[4 * c + 1]), "=r"(w[4 * c + 2]), "=r"(w[4 * c + 3]) : "r"(at));
                }
                uint32_t h[32], lo[kPol ? 32 : 1];
                if constexpr (kRot) {
                    // the block's values, a fast Walsh-Hadamard transform of them in registers (pairs of neighbours a register
                    // pair), times norm / 64, as two fp16 halves
                    const float sc = __half2float(__ushort_as_half(sr.get(gi, lane))) * up * (1.0f / 64.0f);
                    gi += NP;
                    uint64_t e[32];
#pragma unroll
                    for (int c = 0; c < 16; c++) {
                        float f[4];
#pragma unroll
                        for (int b = 0; b < 4; b++) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f[b]) : "r"(entry(w[c % U::kWords], b)));
                        e[2 * c] = pack2(f[0] + f[1], f[0] - f[1]);
                        e[2 * c + 1] = pack2(f[2] + f[3], f[2] - f[3]);
                    }
#pragma unroll
                    for (int d = 1; d < 32; d <<= 1)
#pragma unroll
                        for (int c = 0; c < 32; c++)
                            if (!(c & d)) { const uint64_t s = e[c], t = e[c | d]; e[c] = add2(s, t); e[c | d] = sub2(s, t); }
                    const uint64_t sc2 = pack2(sc, sc);
#pragma unroll
                    for (int c = 0; c < 32; c++) {
                        const uint64_t v = mul2(e[c], sc2);
                        const __half2 hi = __floats2half2_rn(low2(v), high2(v));
                        h[c] = *reinterpret_cast<const uint32_t *>(&hi);
                        // what the halves left, each in one multiply-add of an fp16 with an fp32 (-1 x half + value)
                        float l0, l1;
                        asm("{.reg .b16 a, b, m;\n\tmov.b32 {a, b}, %2;\n\tmov.b16 m, 0xBC00;\n\tfma.rn.f32.f16 %0, a, m, %3;\n\tfma.rn.f32.f16 %1, b, m, %4;}"
                            : "=f"(l0), "=f"(l1) : "r"(h[c]), "f"(low2(v)), "f"(high2(v)));
                        const __half2 rest = __floats2half2_rn(l0, l1);
                        lo[c] = *reinterpret_cast<const uint32_t *>(&rest);
                    }
                } else if (kPol && !FOLD) {
                    const float sc = __half2float(__ushort_as_half(sr.get(gi, lane))) * up;
                    for (pos += part + 1 == kHalves ? 64u + KB * (NP - 1) : 64u; pos >= a.group; pos -= a.group) gi++;
#pragma unroll
                    for (int c = 0; c < 16; c++) {
                        float e[4];
#pragma unroll
                        for (int b = 0; b < 4; b++) {
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(e[b]) : "r"(entry(w[c % U::kWords], b)));
                        }
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            const __half2 hi = __floats2half2_rn(e[2 * b] * sc, e[2 * b + 1] * sc);
                            const float2 back = __half22float2(hi);
                            const __half2 rest = __floats2half2_rn(fmaf(e[2 * b], sc, -back.x), fmaf(e[2 * b + 1], sc, -back.y));
                            h[2 * c + b] = *reinterpret_cast<const uint32_t *>(&hi);
                            lo[kPol ? 2 * c + b : 0] = *reinterpret_cast<const uint32_t *>(&rest);
                        }
                    }
                } else if (kPol) {
#pragma unroll
                    for (int c = 0; c < 16; c++) {
                        uint32_t e[4];
#pragma unroll
                        for (int b = 0; b < 4; b++) {
                            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(e[b]) : "r"(entry(w[c % U::kWords], b)));
                        }
#pragma unroll
                        for (int b = 0; b < 2; b++) {
                            h[2 * c + b] = __byte_perm(e[2 * b], e[2 * b + 1], 0x5410u);
                            lo[kPol ? 2 * c + b : 0] = __byte_perm(e[2 * b], e[2 * b + 1], 0x7632u);
                        }
                    }
                } else if (FOLD) {
#pragma unroll
                    for (int c = 0; c < U::kWords; c++) codes_exact<kCode, BF16>(w[c], h + c * (32 / U::kWords));
                } else {
                    const uint16_t s0 = sr.get(gi, lane);
                    const bool other = pos + 32u >= a.group && (kb0 + i) * KB + part * 64u + 32u < a.K;
                    const uint16_t s1 = other ? sr.get(gi + 1u, lane) : s0;
                    for (pos += part + 1 == kHalves ? 64u + KB * (NP - 1) : 64u; pos >= a.group; pos -= a.group) gi++;
#pragma unroll
                    for (int c = 0; c < U::kWords; c++) codes_scaled<kCode, BF16>(w[c], h + c * (32 / U::kWords), c < U::kWords / 2 ? s0 : s1);
                }
                if (part == 0) {
                    go = wait.template go<(kPol && NF > 1)>(bar(kEmpty + st), ar.lap ^ 1u);
                    fence_after();
                }
                __syncwarp();
                tmem_st32(lane_base + st * kACols + part * 32u, h);
                if constexpr (kPol) tmem_st32(lane_base + st * kACols + (kHalves + part) * 32u, lo);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            fence_before();
            __syncwarp();
            // every lane's codes are in its registers, converted and stored: only now may the copy engine have the stage
            // (an arrival straight behind the shared-memory loads let it overwrite rows that were still on their way)
            if (lane == 0 && go) { bar_arrive(bar(kFull + st)); bar_arrive(bar(kWEmpty + ws)); }
#pragma unroll
            for (int j = 0; j < NP; j++) ar.next(a.ns);
        }
    } else if (warp < 4 * NP + 4 * NF) {
        // ---- readers: accumulators to fp32 totals (fold) and totals to shared memory, [token][row]
        const uint32_t set = (warp - 4 * NP) >> 2, r = (warp & 3u) * 32u + lane, cols = a.T / NF;
        const uint32_t lane_base = tmem + (((warp & 3u) * 32u) << 16) + set * cols;
        float *stage = reinterpret_cast<float *>(smem) + (size_t)set * cols * kRows + r;
        if (FOLD) {
            ScaleReader<true> sr(wait, bar(kSFull), bar(kSEmpty), scale_ring, r);
            float tot[TC];
#pragma unroll
            for (int c = 0; c < TC; c++) tot[c] = 0.0f;
            uint32_t g = 0, in_group = seg0 - grp0 * (g16 / f16);           // segments of group g that are behind
            Ring dr;
            for (uint32_t s = 0; s < nseg; s++, dr.next(a.nd)) {
                const float sc = __half2float(__ushort_as_half(sr.get(g, lane)));
                if (++in_group == g16 / f16) { in_group = 0; g++; }
                wait.near(bar(kDFull + dr.at), dr.lap);
                __syncwarp();
                fence_after();
                // 64 totals a lane and 96 registers: sixteen columns at a time.  With 32 under way the variant spilled in this loop,
                // or did not, as the compiler happened to choose (100 rows in groups of 32: 64.2 to 75 us, now 56.9).
                if constexpr (TC == 64) {
#pragma unroll
                    for (int c = 0; c < TC; c += 16) {
                        if ((uint32_t)c >= cols) break;
                        uint32_t v[16];
                        tmem_ld16(lane_base + dr.at * a.T + c, v);
                        tmem_ld_wait(v);
                        if (c + 16u >= cols) {
                            fence_before();
                            __syncwarp();
                            if (lane == 0) bar_arrive(bar(kDEmpty + dr.at));
                        }
#pragma unroll
                        for (int j = 0; j < 16; j++) tot[c + j] = fmaf(sc, __uint_as_float(v[j]), tot[c + j]);
                    }
                } else {
#pragma unroll
                for (int c = 0; c < TC; c += 32) {
                    if ((uint32_t)c >= cols) break;
                    uint32_t v[2][16];
                    tmem_ld16(lane_base + dr.at * a.T + c, v[0]);
                    if (c + 16u < cols) tmem_ld16(lane_base + dr.at * a.T + c + 16, v[1]);
                    tmem_ld_wait(v[0]);
                    tmem_ld_wait(v[1]);
                    if (c + 32u >= cols) {              // the last read of this accumulator: the next segment may have it
                        fence_before();
                        __syncwarp();
                        if (lane == 0) bar_arrive(bar(kDEmpty + dr.at));
                    }
#pragma unroll
                    for (int j = 0; j < 16; j++) tot[c + j] = fmaf(sc, __uint_as_float(v[0][j]), tot[c + j]);
                    if (c + 16u < cols) {
#pragma unroll
                        for (int j = 0; j < 16; j++) tot[c + 16 + j] = fmaf(sc, __uint_as_float(v[1][j]), tot[c + 16 + j]);
                    }
                }
                }
            }
#pragma unroll
            for (int c = 0; c < TC; c++)
                if ((uint32_t)c < cols) stage[c * kRows] = tot[c];
        }
    } else if (warp == 4 * NP + 4 * NF) {
        // ---- products.  This warp's instructions are what a block costs when tokens are few: one barrier and one commit a
        // block, and where segments are whole blocks, no tests between the products
        const uint32_t idesc = (1u << 4) | (BF16 ? (1u << 7) | (1u << 10) : 0u) | ((a.T >> 3) << 17) | ((kRows >> 4) << 24);
        const uint64_t desc0 = sw128_desc(base + a.at_x);
        const bool whole = !FOLD || f16 % kB16 == 0;
        const bool two = a.planes == 2;
        const uint32_t half16 = (a.T * 128u) >> 4;                 // the second 64 columns of a plane, in descriptor units
        uint32_t in_seg = k16_0 - seg0 * f16, acc = 0, d = tmem;
        Ring ar, dr;
        for (uint32_t i = 0; i < nkb; i++) {
            wait(bar(kFull + ar.at), ar.lap);
            fence_after();
            const uint32_t at = tmem + a.a_base + ar.at * kACols, left = k16_n - (kb0 + i) * kB16;
            const uint64_t desc = desc0 + ((ar.at * xstage) >> 4);
            auto product = [&](uint32_t j) {
                const uint64_t b = desc + (j / 4u) * half16 + (j & 3u) * 2u;
                mma_ts(d, at + j * 8u, b, idesc, acc);
                acc = 1;
                if (two) mma_ts(d, at + j * 8u, b + (plane >> 4), idesc, 1u);
                if (kPol) mma_ts(d, at + kHalves * 32u + j * 8u, b, idesc, 1u);
            };
            auto open = [&]() {
                d = tmem + dr.at * a.T;
                wait(bar(kDEmpty + dr.at), dr.lap ^ 1u);
                fence_after();
            };
            auto close = [&]() {
                mma_commit(bar(kDFull + dr.at));
                dr.next(a.nd);
                in_seg = 0; acc = 0;
            };
            if (whole && left >= kB16) {
                if (FOLD && acc == 0) open();
#pragma unroll
                for (uint32_t j = 0; j < kB16; j++) product(j);
                in_seg += kB16;
                if (FOLD && (in_seg == f16 || left == kB16)) close();
            } else {
                // segments are multiples of 32 columns: their ends fall between pairs of products
#pragma unroll
                for (uint32_t j = 0; j < kB16; j += 2) {
                    if (j >= left) break;
                    if (FOLD && acc == 0) open();
                    product(j);
                    product(j + 1);
                    in_seg += 2;
                    if (FOLD && (in_seg == f16 || j + 2 >= left)) close();
                }
            }
            mma_commit(bar(kEmpty + ar.at));
            ar.next(a.ns);
        }
        if (!FOLD) mma_commit(bar(kDFull));
    } else if (warp == 4 * NP + 4 * NF + 1) {
        // ---- weight copies: a resident weight depends on nothing that came before in the stream
        const bool leader = elect();
        if (a.late) asm volatile("griddepcontrol.wait;" ::: "memory");
        Ring wr;
        uint32_t used = 0;
        for (uint32_t u = u0; u < u1; u++) {
            const bool go = wait.go(bar(kWEmpty + wr.at), wr.lap ^ 1u);
            if (leader && go) {
                used++;
                bar_expect(bar(kWFull + wr.at), U::kStage);
                if (BITS == kBlocked4) tma_2d(base + wr.at * U::kStage, &wmap, row0, u * (U::kCols / 16), bar(kWFull + wr.at));
                else tma_2d(base + wr.at * U::kStage, &wmap, u * U::kBytes, row0, bar(kWFull + wr.at));
            }
            __syncwarp();
            wr.next(a.nw);
        }
        if (leader) *word(kUsedW) = used;
    } else if (warp == 4 * NP + 4 * NF + 2) {
        // ---- activation copies
        const bool leader = elect();
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (leader) word(kMark)[1] = 1u;
        Ring xr;
        uint32_t used = 0;
        for (uint32_t i = 0; i < nkb; i++) {
            const bool go = wait.go(bar(kEmpty + xr.at), xr.lap ^ 1u);
            if (leader && go) {
                used++;
                bar_expect(bar(kFull + xr.at), xstage);
                for (uint32_t p = 0; p < a.planes; p++)
#pragma unroll
                    for (uint32_t q = 0; q < kHalves; q++)
                        tma_2d(base + a.at_x + xr.at * xstage + p * plane + q * a.T * 128u, &xmap, (kb0 + i) * KB + q * 64u, p * a.M + tok0, bar(kFull + xr.at));
            }
            __syncwarp();
            xr.next(a.ns);
        }
        if (leader) *word(kUsedX) = used;
    } else {
        // ---- scales: eight groups of 128 rows at a time, transposed on the way ([group][row])
        Ring sr;
        for (uint32_t g0 = 0; g0 < ngroups; g0 += kScaleGroups) {
            uint16_t v[4][kScaleGroups];
#pragma unroll
            for (uint32_t j = 0; j < 4; j++) {
                const uint16_t *srow = a.scales + (size_t)min(row0 + lane + 32u * j, a.N - 1u) * a.sgroups;
#pragma unroll
                for (uint32_t g = 0; g < kScaleGroups; g++) v[j][g] = __ldg(srow + min(grp0 + g0 + g, a.sgroups - 1u));
            }
            wait(bar(kSEmpty + sr.at), sr.lap ^ 1u);
            const uint32_t to = scale_ring + sr.at * kScaleEntry + lane * 2u;
#pragma unroll
            for (uint32_t j = 0; j < 4; j++)
#pragma unroll
                for (uint32_t g = 0; g < kScaleGroups; g++)
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(to + g * (kRows * 2u) + j * 64u), "h"(v[j][g]) : "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(bar(kSFull + sr.at));
            sr.next(kScaleRing);
        }
    }
    __syncwarp();
    if (!FOLD && warp < 4 * NP + 4 * NF) {
        // totals to shared memory, [token][row]: sixteen tokens at a time, the producers' warps among the takers
        const uint32_t r = (warp & 3u) * 32u + lane;
        wait(bar(kDFull), 0u);
        __syncwarp();
        fence_after();
        for (uint32_t c = (warp >> 2) * 16u; c < a.T; c += (NP + NF) * 16u) {
            uint32_t v[16];
            tmem_ld16(tmem + (((warp & 3u) * 32u) << 16) + c, v);
            tmem_ld_wait(v);
#pragma unroll
            for (int j = 0; j < 16; j++) reinterpret_cast<float *>(smem)[(size_t)(c + j) * kRows + r] = kPol ? __uint_as_float(v[j]) * down : __uint_as_float(v[j]);
        }
        fence_before();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __syncthreads();
    if (wait.stopped()) {                          // the same for all threads: whoever sets the mark does so before the barrier above
        // nothing may be under way any more when tensor and shared memory are given back
        if (warp == 4 * NP + 4 * NF) { mma_commit(bar(kDrain)); drain(bar(kDrain), 1u, 1u); }
        if (warp == 4 * NP + 4 * NF + 1) drain(bar(kWFull), *word(kUsedW), a.nw);
        if (warp == 4 * NP + 4 * NF + 2) drain(bar(kFull), *word(kUsedX), a.ns);
        __syncthreads();
        for (uint32_t e = threadIdx.x; e < a.T * kRows; e += blockDim.x) reinterpret_cast<uint32_t *>(smem)[e] = 0x7fffffffu;
        __syncthreads();
    }
    if (warp == 4 * NP + 4 * NF) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmem) : "memory");
    }
    cg::cluster_group cluster = cg::this_cluster();
    if (a.split > 1) cluster.sync();
    // totals of all the cluster's CTAs, four rows of a token at a time, this CTA's share of them
    const float *mine = reinterpret_cast<const float *>(smem);
    const bool vec = (a.N & 3u) == 0;
    for (uint32_t e = rank * blockDim.x + threadIdx.x; e < a.T * 32u; e += blockDim.x * a.split) {
        const uint32_t t = e >> 5, r = (e & 31u) * 4u, m = tok0 + t, n = row0 + r;
        if (m >= a.M || n >= a.N) continue;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (a.split == 1) {
            v = *reinterpret_cast<const float4 *>(mine + t * kRows + r);
        } else {
            // all of them requested before the first is added: a load from another SM takes some seven hundred cycles
            float4 o[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; k++)
                o[k] = k < a.split ? *reinterpret_cast<const float4 *>(cluster.map_shared_rank(mine, k) + t * kRows + r) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) { v.x += o[k].x; v.y += o[k].y; v.z += o[k].z; v.w += o[k].w; }
        }
        float o[4] = {v.x, v.y, v.z, v.w};
        const float ts = a.tok_scale ? __ldg(a.tok_scale + m) : 1.0f;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float b = !a.bias || n + j >= a.N ? 0.0f
                          : a.bias_half ? __half2float(reinterpret_cast<const __half *>(a.bias)[n + j]) : reinterpret_cast<const float *>(a.bias)[n + j];
            o[j] = o[j] * ts + b;
        }
        const size_t at = (size_t)m * a.N + n;
        if (a.y_dtype == EOQ_B200_F32) {
            float *y = reinterpret_cast<float *>(a.y) + at;
            if (vec) *reinterpret_cast<float4 *>(y) = make_float4(o[0], o[1], o[2], o[3]);
            else for (int j = 0; j < 4; j++) if (n + j < a.N) y[j] = o[j];
        } else {
            uint32_t p[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                if (a.y_dtype == EOQ_B200_F16) { const __half2 q = __floats2half2_rn(o[2 * j], o[2 * j + 1]); p[j] = *reinterpret_cast<const uint32_t *>(&q); }
                else p[j] = pack_bf16(o[2 * j], o[2 * j + 1]);
            }
            uint16_t *y = reinterpret_cast<uint16_t *>(a.y) + at;
            if (vec) *reinterpret_cast<uint2 *>(y) = make_uint2(p[0], p[1]);
            else for (int j = 0; j < 4; j++) if (n + j < a.N) y[j] = (uint16_t)(p[j >> 1] >> (16 * (j & 1)));
        }
    }
    if (a.split > 1) cluster.sync();               // nobody leaves while its totals are being read
}

}  // namespace

// ---------------------------------------------------------------------------
// Activations as two fp16 planes (the nearest fp16, then the nearest to the remainder: 22 bits), rotated first where the
// weight is PolarLinear's: every block of 32 V columns times the normalised Hadamard matrix of that order (Sylvester
// construction, core/polar_quant.py:104-120) over sqrt(block), a fast Walsh-Hadamard transform inside a warp.  A row is
// brought to a largest magnitude of 2^14 .. 2^15 by a power of two, which goes to tok_scale inverted: the planes then hold
// any fp32 row, large or small, with the same relative precision.  One CTA per row, the row in shared memory between
// finding the largest value and writing the planes.
// ---------------------------------------------------------------------------
template <int V>
__global__ void __launch_bounds__(512) split_rows_kernel(const void *__restrict__ x, int x_dtype, uint32_t K, uint32_t M, __half *__restrict__ planes,
                                                         float *__restrict__ tok_scale)
{
    extern __shared__ float row[];
    __shared__ float part[16];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, nwarps = blockDim.x >> 5, m = blockIdx.x;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    auto load = [&](uint32_t k) -> float {
        const size_t i = (size_t)m * K + k;
        if (x_dtype == EOQ_B200_F32) return __ldg(reinterpret_cast<const float *>(x) + i);
        const uint16_t b = __ldg(reinterpret_cast<const uint16_t *>(x) + i);
        return x_dtype == EOQ_B200_F16 ? __half2float(__ushort_as_half(b)) : __uint_as_float((uint32_t)b << 16);
    };
    auto finite = [](float v) { return fabsf(v) < __int_as_float(0x7f800000) ? fabsf(v) : 0.0f; };
    float most = 0.0f;
    if (V == 0) {
        for (uint32_t k = threadIdx.x; k < K; k += blockDim.x) {
            const float v = load(k);
            row[k] = v;
            most = fmaxf(most, finite(v));
        }
    } else {
        constexpr int kV = V ? V : 1;
        for (uint32_t b = warp * 32u * kV; b < K; b += nwarps * 32u * kV) {
            float v[kV];
#pragma unroll
            for (int j = 0; j < kV; j++) v[j] = load(b + 32u * j + lane);
#pragma unroll
            for (int h = 1; h < kV; h <<= 1)
#pragma unroll
                for (int j = 0; j < kV; j++)
                    if (!(j & h)) { const float p = v[j], q = v[j | h]; v[j] = p + q; v[j | h] = p - q; }
#pragma unroll
            for (uint32_t h = 1; h < 32; h <<= 1)
#pragma unroll
                for (int j = 0; j < kV; j++) {
                    const float o = __shfl_xor_sync(0xffffffffu, v[j], h);
                    v[j] = lane & h ? o - v[j] : v[j] + o;
                }
#pragma unroll
            for (int j = 0; j < kV; j++) {
                v[j] *= 1.0f / (32.0f * kV);
                row[b + 32u * j + lane] = v[j];
                most = fmaxf(most, finite(v[j]));
            }
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, d));
    if (lane == 0) part[warp] = most;
    __syncthreads();
    most = 0.0f;
    for (uint32_t w = 0; w < nwarps; w++) most = fmaxf(most, part[w]);
    // 2^e with 2^14 <= most 2^e < 2^15, e within what a float holds, for the largest finite value; rows without one stay as they are
    int e = 0;
    if (most > 0.0f) e = min(120, 141 - (int)(__float_as_uint(most) >> 23));
    const float up = __uint_as_float((uint32_t)(127 + e) << 23);
    if (threadIdx.x == 0) tok_scale[m] = __uint_as_float((uint32_t)(127 - e) << 23);
    for (uint32_t k = threadIdx.x * 2u; k < K; k += blockDim.x * 2u) {
        const float a = row[k] * up, b = row[k + 1] * up;
        const __half ha = __float2half_rn(a), hb = __float2half_rn(b);
        // an infinity has no remainder (and infinity less itself would make the row's results NaN)
        const __half la = __hisinf(ha) ? __half(0) : __float2half_rn(a - __half2float(ha)), lb = __hisinf(hb) ? __half(0) : __float2half_rn(b - __half2float(hb));
        *reinterpret_cast<__half2 *>(planes + (size_t)m * K + k) = __halves2half2(ha, hb);
        *reinterpret_cast<__half2 *>(planes + (size_t)(M + m) * K + k) = __halves2half2(la, lb);
    }
}

static std::atomic<long long> g_qmm_limit{4000000000ll};         // about two seconds
void set_qmm_wait_us(int v) { g_qmm_limit.store(std::min(std::max(v, 0), 60000000) * 2000ll); }

namespace {

typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                             const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn()
{
    static EncodeFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}

bool map_2d(CUtensorMap &m, CUtensorMapDataType type, const void *p, uint64_t inner, uint64_t rows, uint64_t row_bytes, uint32_t box_inner,
            uint32_t box_rows, CUtensorMapSwizzle sw)
{
    const cuuint64_t dims[2] = {inner, rows}, strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_inner, box_rows}, step[2] = {1, 1};
    EncodeFn fn = encode_fn();
    return fn && fn(&m, type, 2, const_cast<void *>(p), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// CTAs of a kernel in clusters of `split` that fit on the device at once, asked once per kernel, size and shared memory.
uint32_t resident_ctas(const void *kern, uint32_t threads, size_t smem, uint32_t split)
{
    struct Known { const void *k; size_t smem; uint32_t split; int dev; uint32_t n; };
    static std::mutex mu;
    static std::vector<Known> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mu);
    for (const Known &k : known) if (k.k == kern && k.smem == smem && k.split == split && k.dev == dev) return k.n;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(split);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = split; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
    known.push_back(Known{kern, smem, split, dev, (uint32_t)std::max(n, 0) * split});
    return known.back().n;
}

struct Shape { uint32_t T, nw, ns, nd, a_base; size_t smem; uint32_t at_x, at_bar; };

// Stages and shared memory of a kernel variant for a token tile T.  A producer set has to come by every stage on every lap
// (its parity waits look one lap back): operand stages in multiples of the sets, weight stages in multiples of the copies
// that a set steps over.  Four accumulators where tokens are few: the way from a product's commit over a reader and back takes
// longer than two segments of products (24 rows against 11008 x 4096 in groups of 64 columns 22.1 -> 20.5 us, of 128 15.95 ->
// 14.9, with the shorter conversions).
void place(Shape &s, uint32_t stage_w, uint32_t unit_blocks, uint32_t sets, uint32_t planes, uint32_t a_cols, uint32_t kb, bool fold)
{
    const size_t fixed = 512 + 1024 + 1024 + (kRows + 4) * 4 + kScaleRing * kScaleEntry, room = 226u * 1024u - fixed;
    const uint32_t xstage = s.T * 2u * kb * planes, step = std::max(1u, sets / unit_blocks);
    s.nd = !fold ? 1u : s.T <= 32u ? 4u : 2u;
    s.a_base = s.nd * s.T;
    s.ns = std::min(8u, (512u - s.a_base) / a_cols) / sets * sets;
    while (s.ns > sets && room < (size_t)s.ns * xstage + std::max(4u, step) * stage_w) s.ns -= sets;
    s.nw = (uint32_t)std::min<size_t>(8, (room - (size_t)s.ns * xstage) / stage_w) / step * step;      // the rest of the room hides DRAM
    s.at_x = s.nw * stage_w;
    s.at_bar = std::max(s.at_x + s.ns * xstage, s.T * kRows * 4u);
    s.smem = s.at_bar + fixed;
}

// How a call is cut: token tiles of at most `most` tokens (multiples of `step`) and the columns over the CTAs of a cluster.
// The cut with the least rounds of resident CTAs x what a CTA takes: its blocks of 64 columns, each the longer of its
// products (two cycles a token) and its producers' work, and some four thousand cycles to start, fill and store (half as
// many more to meet in a cluster).  The constants are measured (1024 x 4096 to 11008 x 4096, 8 to 2048 tokens).
struct Plan { uint32_t T, tok_tiles, split; double cycles; };
struct PlanKey {
    uint32_t rows, K, M, planes;
    int dev;
    bool operator==(const PlanKey &o) const { return rows == o.rows && K == o.K && M == o.M && planes == o.planes && dev == o.dev; }
};

// With `cycles`: what the call would take by the plan's own estimate, nothing launched.
template <int BITS, bool BF16, bool FOLD, int NP, int NF, int TC, int KB>
int run_variant(QmmArgs a, uint32_t most, uint32_t step, const void *packed, uint64_t row_bytes, const void *x, cudaStream_t st, double *cycles)
{
    using U = Unit<BITS, KB>;
    auto kern = qmm_kernel<BITS, BF16, FOLD, NP, NF, TC, KB>;
    constexpr uint32_t threads = (4 * NP + 4 * NF + 4) * 32, a_cols = (BITS == kPolar || BITS == kPolarRot ? 64u : 32u) * (KB / 64);
    constexpr bool kPol = BITS == kPolar || BITS == kPolarRot;
    const uint32_t rows = (a.N + kRows - 1) / kRows;
    a.units = (a.K + U::kCols - 1) / U::kCols;
    auto placed = [&](uint32_t T) {
        Shape s = {};
        s.T = T;
        place(s, U::kStage, U::kBlocks, NP, a.planes, a_cols, KB, FOLD);
        return s;
    };
    // the plans of the last shapes this kernel was called with (a model has a handful)
    static std::mutex mu;
    static PlanKey keys[32];
    static Plan plans[32];
    static uint32_t used = 0;
    PlanKey key{rows, a.K, a.M, a.planes, 0};
    if (cudaGetDevice(&key.dev) != cudaSuccess) return (int)cudaErrorInvalidDevice;
    Plan plan = {};
    {
        std::lock_guard<std::mutex> lock(mu);
        for (uint32_t i = 0; i < std::min(used, 32u); i++) if (keys[i] == key) plan = plans[i];
    }
    if (!plan.T) {
        const double producers = BITS == kPolarRot ? 1250.0 : kPol ? FOLD ? 700.0 : 1100.0 : FOLD ? 450.0 : !BF16 ? 400.0 : BITS == 8 ? 600.0 : 660.0, products = BITS == kPolar ? 3.0 : kPol ? 2.0 : a.planes;
        const double fixed = kPol && !FOLD ? 8000.0 : 4000.0;       // (a row's norms are read first, and tiles are large)
        double best = 1e30;
        const uint32_t least = (a.M + most - 1) / most;
        for (uint32_t n = least; n < least + 4; n++) {
            const uint32_t T = ((a.M + n - 1) / n + step - 1) / step * step;
            if (T > most || (n > least && (T >= plan.T || (a.M + T - 1) / T < n))) continue;
            const Shape s = placed(T);
            const double block = std::max(producers, 2.0 * T * products + 150.0);
            for (uint32_t split = 1; split <= 8 && split <= a.units; split++) {
                const uint32_t room = resident_ctas(reinterpret_cast<const void *>(kern), threads, s.smem, split);
                if (room == 0) continue;
                const double cost = (double)((rows * n * split + room - 1) / room) *
                                    ((double)((a.units + split - 1) / split) * (U::kCols / 64) * block + fixed * (split > 1 ? 1.5 : 1.0));
                // a cut into more token tiles repeats the producers' work: only for a clear gain
                if (cost < best * (n > plan.tok_tiles && plan.T ? 0.95 : 0.999)) { best = cost; plan = Plan{T, n, split, cost}; }
            }
        }
        if (!plan.T) return (int)cudaErrorNotSupported;
        std::lock_guard<std::mutex> lock(mu);
        keys[used % 32] = key;
        plans[used % 32] = plan;
        used = used + 1 >= 64 ? 32 : used + 1;
    }
    if (cycles) { *cycles = plan.cycles; return 0; }
    const Shape s = placed(plan.T);
    a.T = s.T; a.nw = s.nw; a.ns = s.ns; a.nd = s.nd; a.a_base = s.a_base; a.at_x = s.at_x; a.at_bar = s.at_bar; a.split = plan.split;
    CUtensorMap wmap, xmap;
    const bool mapped = BITS == kBlocked4
        ? map_2d(wmap, CU_TENSOR_MAP_DATA_TYPE_INT64, packed, row_bytes / 8, a.K / 16, row_bytes, kRows, U::kCols / 16, CU_TENSOR_MAP_SWIZZLE_NONE)
        : map_2d(wmap, CU_TENSOR_MAP_DATA_TYPE_UINT8, packed, row_bytes, a.N, row_bytes, U::kBytes, kRows,
                 BITS == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B);
    if (!mapped ||
        !map_2d(xmap, BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, x, a.K, (uint64_t)a.M * a.planes, (uint64_t)a.K * 2,
                64, s.T, CU_TENSOR_MAP_SWIZZLE_128B))
        return (int)cudaErrorNotSupported;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(rows * a.split, plan.tok_tiles);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = programmatic_launches();
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = a.split; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, a, wmap, xmap);
    count_launch();
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

template <int BITS, bool BF16>
int run_fold(const QmmArgs &a, const void *packed, uint64_t row_bytes, const void *x, cudaStream_t st, double *cycles)
{
    // few tokens: long blocks (polar centroids take two operand planes, which leaves room for short ones), and as few
    // warps as keep up: 4096 x 4096, 24 tokens takes 9.1 us with two producer sets and one reader set, 9.8 with four sets
    constexpr int kLong = BITS == kPolar ? 64 : 128;
    if (a.M <= 32) return run_variant<BITS, BF16, true, 2, 1, 32, kLong>(a, 32, 16, packed, row_bytes, x, st, cycles);
    if (a.M <= 64) return run_variant<BITS, BF16, true, 2, 2, 32, kLong>(a, 64, 32, packed, row_bytes, x, st, cycles);
    return run_variant<BITS, BF16, true, 2, 2, 64, 64>(a, 128, 32, packed, row_bytes, x, st, cycles);
}

template <int BITS, bool BF16>
int run_scaled(const QmmArgs &a, const void *packed, uint64_t row_bytes, const void *x, cudaStream_t st, double *cycles)
{
    return run_variant<BITS, BF16, false, 4, 1, 32, 64>(a, 256, 16, packed, row_bytes, x, st, cycles);
}

// Byte codes: up to this many tokens the centroids are multiplied and each block's sum scaled in fp32 (every 64 columns a
// reader's pass over the accumulator, 128 tokens at most); beyond, centroid x norm goes in as two fp16 halves, a row at a
// time brought to their range, and a CTA takes 256 tokens: a block costs 1100 cycles whatever the tokens up to some 160, so
// fewer, larger tiles pay.  14336 x 4096, 64 columns a block, 128 tokens 55 us / 52, 256 tokens 100 / 82.  Both leave 22
// bits of each factor.
//   Blocks of 64 columns against 16-bit activations (c.rotate): the producers rotate the weight's blocks in registers, where
// the other two want rotated activations of two halves each.  The activations are exact then, and a pair takes two
// products, not three.  What bounds it, 512 tokens against 14336 x 4096: the tensor pipe, busy 66 % of an SM's active
// cycles, beside the producers (instruction slots 49 %, multiply-add pipe 41 %); SMs are active 68 % of the time, for 224 CTAs are a round and a half.  512 tokens against 14336 x 4096 187 -> 139 us, 11008 x 4096 127 -> 94.8 (97.8 before
// the remainders came from one mixed multiply-add each; look-ups by byte permutes instead of dot products 103), with a third
// less error (4096 columns, fp32 results: 1.88e-6 -> 1.27e-6).
constexpr uint32_t kPolarFold = 112;

int qmm(const QmmCall &c, void *stream, double *cycles)
{
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    QmmArgs a = {};
    a.scales = c.scales; a.centroids = c.centroids; a.bias = c.bias; a.tok_scale = c.tok_scale; a.y = c.y;
    a.N = c.N; a.K = c.K; a.M = c.M; a.group = c.group; a.sgroups = c.K / c.group; a.y_dtype = c.y_dtype;
    a.bias_half = c.bias_half;
    a.late = c.late;
    a.limit = g_qmm_limit.load(std::memory_order_relaxed);
    a.status = c.status;
    for (uint32_t parts = 1; a.seg == 0; parts++)              // the fewest equal parts of a group, of 32-column multiples, that are short enough
        if (c.group % (32u * parts) == 0 && c.group / parts <= 128u) a.seg = c.group / parts;
    a.planes = c.split_x ? 2u : 1u;
    a.entries = c.centroids ? 1u << c.bits : 1u;
    const bool bf = c.bf16 && !c.split_x;
    const uint64_t row_bytes = c.blocked_rows ? (uint64_t)c.blocked_rows * 8 : c.centroids ? c.K : c.bits == 4 ? c.K / 2 : c.bits == 2 ? c.K / 4 : c.K;
    if (c.rotate) return run_variant<kPolarRot, false, false, 2, 1, 32, 64>(a, 256, 16, c.packed, row_bytes, c.x, st, cycles);
    if (c.centroids && c.M > kPolarFold) return run_variant<kPolar, false, false, 2, 1, 32, 64>(a, 256, 16, c.packed, row_bytes, c.x, st, cycles);
    if (c.centroids) return run_fold<kPolar, false>(a, c.packed, row_bytes, c.x, st, cycles);
    const bool fold = c.split_x || c.M <= 128u;
#define EOQ_QMM(B)                                                                                                                      \
    (fold ? (bf ? run_fold<B, true>(a, c.packed, row_bytes, c.x, st, cycles) : run_fold<B, false>(a, c.packed, row_bytes, c.x, st, cycles)) \
          : (bf ? run_scaled<B, true>(a, c.packed, row_bytes, c.x, st, cycles) : run_scaled<B, false>(a, c.packed, row_bytes, c.x, st, cycles)))
    if (c.blocked_rows) return EOQ_QMM(kBlocked4);
    if (c.bits == 4) return EOQ_QMM(4);
    if (c.bits == 2) return EOQ_QMM(2);
    return EOQ_QMM(8);
#undef EOQ_QMM
}

}  // namespace

// Whether the kernels above take a packed weight of this shape: whole groups per row, copies aligned.
bool qmm_takes(uint32_t K, uint32_t bits, uint32_t group, const void *packed, const void *x)
{
    const uint32_t per16 = bits == 4 ? 32u : bits == 2 ? 64u : 16u;
    return K % per16 == 0 && group % 32u == 0 && K % group == 0 && ((reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(x)) & 15u) == 0;
}

int launch_qmm(const QmmCall &c, void *stream) { return qmm(c, stream, nullptr); }

// Whether the call is to be preferred to a dequantised copy of the weight and a library GEMM, given the microseconds that
// the copy takes longer than what this kernel reads takes to make, and `least_us`, which the two launches of that route take
// at any size.  fp32 activations: always (the library multiplies them on the CUDA cores: 13 x slower at 512 rows).  16-bit
// ones: up to 32 rows, or where the plan's estimate, at the 1.5 cycles a nanosecond that long products run at (with a tenth
// more where scales are applied before the product, and another for bf16, whose codes take a rounding more), is not above the
// GEMM's (1.45 PFLOP/s, 7 us at least; where rows of y are not 16-byte multiples, cutting them out of padded ones besides)
// less 4 us.  Fitted over thirteen shapes from 512 x 512 to 28672 x 8192, 40 to 2048 rows, fp16 and bf16, both ways timed:
// the choice costs 0.8 % (from decoded codes) and 1.1 % (from packed ones) of device time on the mean against the better of
// the two.
bool qmm_preferred(const QmmCall &c, double copy_us, double least_us)
{
    if (c.split_x || c.M <= 32u) return true;
    if (c.N % 8u) copy_us += 4.0 + (double)c.M * c.N / 1e6;
    double cycles = 0;
    if (qmm(c, nullptr, &cycles) != 0) return false;
    if (c.M > 128u) cycles *= c.bf16 ? 1.21 : 1.1;
    return cycles / 1500.0 <= std::max(least_us, std::max(7.0, 2.0 * c.M * (double)c.N * c.K / 1.45e9) + copy_us - 4.0);
}

bool split_rows_takes(uint32_t K, uint32_t block) { return K % 16u == 0 && K <= 48u * 1024u && (block == 1 || block == 64 || block == 128 || block == 256); }

// x [M][K] to two fp16 planes [2][M][K] and M factors; block 1: no rotation.
int launch_split_rows(const void *x, int x_dtype, uint32_t K, uint32_t M, uint32_t block, void *planes, float *tok_scale, void *stream)
{
    auto kern = block == 1 ? split_rows_kernel<0> : block == 64 ? split_rows_kernel<2> : block == 128 ? split_rows_kernel<4> : split_rows_kernel<8>;
    static std::atomic<uint64_t> asked{0};                  // kernels whose shared-memory limit has been raised, per device
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    const uint64_t mark = dev < 16 ? 1ull << (dev * 4 + (block == 1 ? 0 : block == 64 ? 1 : block == 128 ? 2 : 3)) : 0u;
    if (!mark || !(asked.load() & mark)) {
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 48 * 1024 * 4);
        if (e != cudaSuccess) return (int)e;
        asked.fetch_or(mark);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(M);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = (size_t)K * 4;
    cfg.stream = reinterpret_cast<cudaStream_t>(stream);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = programmatic_launches();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, x, x_dtype, K, M, reinterpret_cast<__half *>(planes), tok_scale);
    count_launch();
    return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

uint32_t qmm_status()
{
    uint32_t v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_qmm_status, 4) != cudaSuccess) return ~0u;
    if (v && cudaMemcpyToSymbol(g_qmm_status, &zero, 4) != cudaSuccess) return ~0u;
    return v;
}

}  // namespace eoq
