// The wire format's encoder on the device: counts of symbols, one rANS chain per block and lane, and the blocks' bytes put
// one behind the other (core/rans.py:210-276, core/rans_blocked.py:88-114).
//
// What bounds it is the chain (two dependent multiplications, a compare and a shift; 0.073 us a symbol), of which
// thousands run side by side where the host's sixteen cores run sixty-four (few, long blocks are the host's: eoq_b200_symbols_preferred); the copies
// to and from the host take longer than the kernels: 4 Mi codes in blocks of 256 60 us (move 6.6, count 6.2, encode 25.8, scan 11.2, gather 9.9) of a
// call of 0.85 ms.
#include "eoq_internal.h"

namespace eoq {

namespace {

__device__ __forceinline__ uint32_t bswap16(uint32_t v) { return ((v & 0xFFu) << 8) | (v >> 8); }

// Bytes as the caller has them to symbols, in place: value + shift, clamped to the alphabet; how many had to be.
__global__ void __launch_bounds__(256) wire_move_kernel(uint8_t *__restrict__ sym, int is_signed, int shift, uint32_t n, int top, unsigned long long *__restrict__ outside)
{
    uint32_t out = 0;
    auto symbol = [&](uint32_t byte) -> uint32_t {
        const int v = (is_signed ? (int)(int8_t)byte : (int)byte) + shift, c = min(max(v, 0), top);
        out += c != v;
        return (uint32_t)c;
    };
    const uint32_t whole = n / 16u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < whole; i += gridDim.x * blockDim.x) {
        uint4 v = reinterpret_cast<uint4 *>(sym)[i];
        uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (uint32_t j = 0; j < 4; j++)
            w[j] = symbol(w[j] & 0xFFu) | symbol((w[j] >> 8) & 0xFFu) << 8 | symbol((w[j] >> 16) & 0xFFu) << 16 | symbol(w[j] >> 24) << 24;
        reinterpret_cast<uint4 *>(sym)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (blockIdx.x == 0) for (uint32_t i = whole * 16u + threadIdx.x; i < n; i += blockDim.x) sym[i] = (uint8_t)symbol(sym[i]);
    out = __reduce_add_sync(0xffffffffu, out);
    if (out && (threadIdx.x & 31u) == 0) atomicAdd(outside, (unsigned long long)out);
}

template <typename T>
__global__ void __launch_bounds__(256) wire_count_kernel(const T *__restrict__ sym, uint32_t n, uint32_t alphabet, unsigned long long *__restrict__ counts)
{
    extern __shared__ uint32_t part[];               // one table a warp
    const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (uint32_t i = threadIdx.x; i < alphabet * warps; i += blockDim.x) part[i] = 0u;
    __syncthreads();
    uint32_t *mine = part + warp * alphabet;
    constexpr uint32_t kPer = 16u / sizeof(T);
    const uint32_t whole = n / kPer;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < whole; i += gridDim.x * blockDim.x) {
        const uint4 v = reinterpret_cast<const uint4 *>(sym)[i];
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (uint32_t j = 0; j < kPer; j++) atomicAdd(mine + (sizeof(T) == 1 ? (w[j / 4] >> (8 * (j & 3u))) & 0xFFu : (w[j / 2] >> (16 * (j & 1u))) & 0xFFFFu), 1u);
    }
    if (blockIdx.x == 0) for (uint32_t i = whole * kPer + threadIdx.x; i < n; i += blockDim.x) atomicAdd(mine + sym[i], 1u);
    __syncthreads();
    for (uint32_t s = threadIdx.x; s < alphabet; s += blockDim.x) {
        uint32_t sum = 0;
        for (uint32_t w = 0; w < warps; w++) sum += part[w * alphabet + s];
        if (sum) atomicAdd(counts + s, (unsigned long long)sum);
    }
}

// One block a lane, last symbol first.  The bytes that leave the state go out as words, [word][lane] of the warp's part of
// the scratch (a word holds four bytes in their final order, words are in reverse); the last zero to three bytes and the state
// stay with the block's record.  A division is a multiplication by the reciprocal, as on the host (wire_host.cpp, EncSym).
template <typename T, bool VEC>
__global__ void __launch_bounds__(128) wire_encode_kernel(const WireEncodeArgs a)
{
    extern __shared__ uint4 table[];                 // {reciprocal, low and high word; frequency; cumulative}
    for (uint32_t i = threadIdx.x; i < a.alphabet; i += blockDim.x) table[i] = a.table[i];
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= a.nblocks) return;
    const uint32_t first = b * a.block, len = min(a.block, a.n - first), M = 1u << a.p;
    const T *src = reinterpret_cast<const T *>(a.sym) + first;
    uint32_t *out = a.scratch + (size_t)(b >> 5) * 32u * a.words + lane;
    uint32_t x = 1u << (a.p + 8u), held = 0, words = 0;
    uint64_t acc = 0;
    auto put = [&](uint32_t s) {
        const uint4 e = table[s];
        const uint32_t hi = x >> 16, k = (hi >= e.z) + ((hi >> 8) >= e.z);
        const uint32_t low = k == 2 ? bswap16(x & 0xFFFFu) : x & 0xFFu;
        acc = k ? (acc << (8u * k)) | low : acc;
        held += k;
        if (held >= 4u) {
            held -= 4u;
            out[(size_t)words * 32u] = (uint32_t)(acc >> (8u * held));
            words++;
        }
        x = k == 2 ? hi : k ? x >> 8 : x;
        const uint64_t lo = (uint64_t)x * e.x, up = (uint64_t)x * e.y;
        const uint32_t q = (uint32_t)((up + (lo >> 32)) >> 16);
        x += q * (M - e.z) + e.w;
    };
    constexpr uint32_t kPer = 16u / sizeof(T);
    uint32_t i = len;
    if (VEC) {
        while (i % kPer) put(src[--i]);
        for (; i > 0; i -= kPer) {
            const uint4 v = *reinterpret_cast<const uint4 *>(src + i - kPer);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (uint32_t j = kPer; j-- > 0;) put(sizeof(T) == 1 ? (w[j / 4] >> (8 * (j & 3u))) & 0xFFu : (w[j / 2] >> (16 * (j & 1u))) & 0xFFFFu);
        }
    } else {
        while (i > 0) put(src[--i]);
    }
    const uint32_t state_len = x >> 24 ? 4u : x >> 16 ? 3u : x >> 8 ? 2u : 1u;
    a.record[b] = make_uint4(x, words, (uint32_t)acc, held);
    a.sizes[b] = 1u + state_len + held + 4u * words;
}

// Exclusive sums of the blocks' sizes; the total goes behind them.  One CTA: a few microseconds for tens of thousands.
__global__ void __launch_bounds__(1024) wire_scan_kernel(const uint32_t *__restrict__ sizes, uint32_t n, uint32_t *__restrict__ offsets, unsigned long long *__restrict__ total)
{
    __shared__ uint32_t sums[32];
    __shared__ unsigned long long base;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (uint32_t at = 0; at < n; at += 4096u) {
        const uint32_t i = at + threadIdx.x * 4u;
        uint32_t v[4], s = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) { v[j] = i + j < n ? sizes[i + j] : 0u; s += v[j]; }
        uint32_t inc = s;
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) { const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d); if (lane >= d) inc += o; }
        if (lane == 31) sums[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            uint32_t t = sums[lane];
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) { const uint32_t o = __shfl_up_sync(0xffffffffu, t, d); if (lane >= d) t += o; }
            sums[lane] = t;
        }
        __syncthreads();
        unsigned long long o = base + (warp ? sums[warp - 1] : 0u) + inc - s;
#pragma unroll
        for (uint32_t j = 0; j < 4; j++) { if (i + j < n) offsets[i + j] = (uint32_t)o; o += v[j]; }
        __syncthreads();
        if (threadIdx.x == 0) base += sums[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = base;
}

// [1 B state length][state, big-endian][bytes] of every block to its place, a warp a block.
__global__ void __launch_bounds__(256) wire_gather_kernel(const WireEncodeArgs a, const uint32_t *__restrict__ offsets, uint8_t *__restrict__ out)
{
    const uint32_t b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;      // (threads of all blocks can be more than 2^32)
    if (b >= a.nblocks) return;
    const uint4 r = a.record[b];
    const uint32_t *words = a.scratch + (size_t)(b >> 5) * 32u * a.words + (b & 31u);
    uint8_t *to = out + offsets[b];
    const uint32_t state_len = r.x >> 24 ? 4u : r.x >> 16 ? 3u : r.x >> 8 ? 2u : 1u;
    if (lane == 0) to[0] = (uint8_t)state_len;
    if (lane < state_len) to[1u + lane] = (uint8_t)(r.x >> (8u * (state_len - 1u - lane)));
    if (lane < r.w) to[1u + state_len + lane] = (uint8_t)(r.z >> (8u * lane));
    to += 1u + state_len + r.w;
    for (uint32_t e = lane; e < r.y * 4u; e += 32u) to[e] = (uint8_t)(words[(size_t)(r.y - 1u - e / 4u) * 32u] >> (8u * (e & 3u)));
}

}  // namespace

int launch_wire_move(uint8_t *sym, int is_signed, int shift, uint32_t n, uint32_t alphabet, unsigned long long *outside, void *stream)
{
    wire_move_kernel<<<std::min(592u, n / 4096u + 1u), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(sym, is_signed, shift, n, (int)alphabet - 1, outside);
    count_launch();
    return (int)cudaGetLastError();
}

int launch_wire_count(const void *sym, int wide, uint32_t n, uint32_t alphabet, unsigned long long *counts, void *stream)
{
    const uint32_t warps = alphabet <= 1024u ? 8u : 1u, grid = std::min(512u, n / 4096u + 1u);
    const size_t smem = (size_t)alphabet * warps * 4u;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (wide) wire_count_kernel<uint16_t><<<grid, warps * 32u, smem, st>>>(static_cast<const uint16_t *>(sym), n, alphabet, counts);
    else wire_count_kernel<uint8_t><<<grid, warps * 32u, smem, st>>>(static_cast<const uint8_t *>(sym), n, alphabet, counts);
    count_launch();
    return (int)cudaGetLastError();
}

int launch_wire_encode(const WireEncodeArgs &a, int wide, uint32_t *offsets, unsigned long long *total, uint8_t *out, void *stream)
{
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uint32_t grid = (a.nblocks + 127u) / 128u;
    const size_t smem = (size_t)a.alphabet * 16u;
    // sixteen bytes of symbols a load where every block starts on such a boundary (the array does)
    const bool vec = (uint64_t)a.block * (wide ? 2u : 1u) % 16u == 0;
    void (*kern)(WireEncodeArgs) = wide ? (vec ? wire_encode_kernel<uint16_t, true> : wire_encode_kernel<uint16_t, false>)
                                        : (vec ? wire_encode_kernel<uint8_t, true> : wire_encode_kernel<uint8_t, false>);
    if (smem > 48u * 1024u) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    kern<<<grid, 128, smem, st>>>(a);
    wire_scan_kernel<<<1, 1024, 0, st>>>(a.sizes, a.nblocks, offsets, total);
    wire_gather_kernel<<<(a.nblocks + 7u) / 8u, 256, 0, st>>>(a, offsets, out);
    count_launch(); count_launch(); count_launch();
    return (int)cudaGetLastError();
}

}  // namespace eoq
