// Wire-format encoder on the host's cores: symbols in whatever integer type the caller has them, counted and encoded
// without an intermediate copy of the array.
//
// What bounds it is one serial chain per block (compare, shift, multiply, multiply, add: some fifteen cycles a symbol).
// Four blocks are encoded side by side on a core so that their chains fill each other's latencies, a division is one
// 64-bit multiplication by a reciprocal that is exact over the range a state can have, and renormalisation is
// branch-free (zero, one or two bytes).
#include "eoq_internal.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <memory>
#include <thread>

namespace eoq {

namespace {

// x / f for x < f << 16, f <= 65536, as (x * m) >> 48 with m = floor(2^48 / f) + 1.  Error: x m / 2^48 exceeds x / f by
// less than x / 2^48 < f / 2^32 <= 1 / f (as f <= 2^16), so the floor is exact; and x m <= (f 2^16 - 1)(2^48 / f + 1)
// < 2^64 because f 2^16 <= 2^48 / f.
struct EncSym {
    uint64_t m;
    uint32_t f, c;
};

template <typename T>
struct Source {
    const T *p;
    int64_t shift, top;      // symbol = value + shift, clamped to [0, top]
    bool clamp;
    uint32_t operator[](size_t i) const
    {
        int64_t v = (int64_t)p[i] + shift;
        if (clamp) v = v < 0 ? 0 : v > top ? top : v;
        return (uint32_t)v;
    }
};

// one step of the encoder (core/rans.py:229-262): up to two bytes of the state leave below `at`, then the symbol goes in
static inline void put(uint32_t &x, uint8_t *&at, const EncSym &s, uint32_t M)
{
    const uint32_t hi = x >> 16;
    const uint32_t k = (hi >= s.f) + ((hi >> 8) >= s.f);
    at[-1] = (uint8_t)x;
    at[-2] = (uint8_t)(x >> 8);
    at -= k;
    x = (uint32_t)((uint64_t)x >> (8 * k));
    const uint32_t q = (uint32_t)(((uint64_t)x * s.m) >> 48);
    x += q * (M - s.f) + s.c;
}

// [1 B state_len][state, big-endian] in front of the bytes that start at `at`
static inline uint8_t *finish(uint32_t x, uint8_t *at)
{
    uint32_t len = 0;
    for (uint32_t v = x; v; v >>= 8) { *--at = (uint8_t)v; len++; }
    *--at = (uint8_t)len;
    return at;
}

}  // namespace

// Ranges of blocks, each encoded into a buffer of its own.
struct WireEncoded {
    std::vector<std::unique_ptr<uint8_t[]>> buf;
    std::vector<size_t> bytes, first_block;
    std::vector<uint32_t> sizes;
};

// Threads worth starting for n symbols: one costs some twenty microseconds to start, about 10 K symbols of encoding.
static size_t threads_for(size_t n)
{
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    return std::max<size_t>(1, std::min<size_t>({hw, 32, n >> 15}));
}

template <typename T>
static bool encode_ranges(Source<T> src, size_t n, const std::vector<EncSym> &tab, uint32_t p, uint32_t block, WireEncoded &out)
{
    const bool check = !src.clamp;
    std::atomic<bool> bad{false};
    src.clamp = true;                  // whatever the array holds, no look-up leaves the table
    const uint32_t M = 1u << p;
    const size_t nb = (n + block - 1) / block, nt = threads_for(n);
    const size_t nranges = nt == 1 ? 1 : std::min<size_t>(nb, nt * 4);
    out.buf.resize(nranges);
    out.bytes.assign(nranges, 0);
    out.first_block.resize(nranges + 1);
    out.sizes.resize(nb);
    for (size_t r = 0; r <= nranges; r++) out.first_block[r] = nb * r / nranges;
    const size_t slot = 2 * (size_t)block + 16;
    parallel_for(nranges, [&](size_t r) {
        const size_t lo = out.first_block[r], hi = out.first_block[r + 1];
        if (check) {
            const size_t b = lo * block, e = std::min<size_t>(n, hi * block);
            bool out_of_range = false;
            for (size_t i = b; i < e; i++) out_of_range |= (uint64_t)((int64_t)src.p[i] + src.shift) > (uint64_t)src.top;
            if (out_of_range) { bad.store(true); return; }
        }
        std::unique_ptr<uint8_t[]> scratch(new uint8_t[4 * slot]);
        size_t cap = 0, used = 0;
        std::unique_ptr<uint8_t[]> buf;
        auto append = [&](const uint8_t *b, const uint8_t *e, size_t blk) {
            const size_t len = (size_t)(e - b);
            if (used + len > cap) {
                // as long as the rest of the range gets at this block's rate and a little more
                const size_t want = used + len + std::max<size_t>(len, 64) * (hi - blk) * 17 / 16 + 4096;
                std::unique_ptr<uint8_t[]> bigger(new uint8_t[want]);
                if (used) std::memcpy(bigger.get(), buf.get(), used);
                buf = std::move(bigger);
                cap = want;
            }
            std::memcpy(buf.get() + used, b, len);
            used += len;
            out.sizes[blk] = (uint32_t)len;
        };
        size_t b = lo;
        const EncSym *t = tab.data();
        for (; b + 4 <= hi && (b + 4) * block <= n; b += 4) {
            uint32_t x0 = 1u << (p + 8), x1 = x0, x2 = x0, x3 = x0;
            uint8_t *e0 = scratch.get() + slot, *e1 = e0 + slot, *e2 = e1 + slot, *e3 = e2 + slot;
            uint8_t *a0 = e0, *a1 = e1, *a2 = e2, *a3 = e3;
            const size_t i0 = b * block, i1 = i0 + block, i2 = i1 + block, i3 = i2 + block;
            for (size_t i = block; i-- > 0;) {
                put(x0, a0, t[src[i0 + i]], M);
                put(x1, a1, t[src[i1 + i]], M);
                put(x2, a2, t[src[i2 + i]], M);
                put(x3, a3, t[src[i3 + i]], M);
            }
            append(finish(x0, a0), e0, b);
            append(finish(x1, a1), e1, b + 1);
            append(finish(x2, a2), e2, b + 2);
            append(finish(x3, a3), e3, b + 3);
        }
        for (; b < hi; b++) {
            uint32_t x = 1u << (p + 8);
            uint8_t *e = scratch.get() + slot, *a = e;
            const size_t first = b * block, len = std::min<size_t>(block, n - first);
            for (size_t i = len; i-- > 0;) put(x, a, t[src[first + i]], M);
            append(finish(x, a), e, b);
        }
        out.buf[r] = std::move(buf);
        out.bytes[r] = used;
    }, nt);
    return !bad.load();
}

template <typename T>
static void count_range(const Source<T> &src, size_t n, uint32_t alphabet, uint64_t *counts, int64_t &lo, int64_t &hi)
{
    const size_t nt = threads_for(n), nr = nt == 1 ? 1 : nt * 2;
    std::vector<std::vector<uint32_t>> part(nr);
    std::vector<int64_t> los(nr, INT64_MAX), his(nr, INT64_MIN);
    parallel_for(nr, [&](size_t r) {
        const size_t b = n * r / nr, e = n * (r + 1) / nr;
        // four tables for small alphabets: equal neighbours do not wait for each other's increments
        const size_t stride = alphabet <= 1024 ? ((size_t)alphabet + 15) & ~(size_t)15 : 0, copies = stride ? 4 : 1;
        std::vector<uint32_t> &c = part[r];
        c.assign(std::max<size_t>(stride * copies, alphabet), 0u);
        int64_t mn = INT64_MAX, mx = INT64_MIN;
        if (src.clamp) {
            for (size_t i = b; i < e; i++) c[(i & (copies - 1)) * stride + src[i]]++;
            mn = 0; mx = 0;
        } else {
            for (size_t i = b; i < e; i++) {
                const int64_t v = (int64_t)src.p[i] + src.shift;
                mn = std::min(mn, v); mx = std::max(mx, v);
                if ((uint64_t)v < alphabet) c[(i & (copies - 1)) * stride + (size_t)v]++;
            }
        }
        los[r] = mn; his[r] = mx;
        if (copies > 1)
            for (size_t s = 0; s < alphabet; s++) c[s] += c[stride + s] + c[2 * stride + s] + c[3 * stride + s];
    }, nt);
    lo = INT64_MAX; hi = INT64_MIN;
    for (uint32_t s = 0; s < alphabet; s++) counts[s] = 0;
    for (size_t r = 0; r < nr; r++) {
        for (uint32_t s = 0; s < alphabet; s++) counts[s] += part[r][s];
        if (n * r / nr < n * (r + 1) / nr) { lo = std::min(lo, los[r]); hi = std::max(hi, his[r]); }
    }
}

template <typename F>
static bool by_type(const void *sym, int elem, int64_t shift, bool clamp, uint32_t alphabet, F &&f)
{
    const int64_t top = (int64_t)alphabet - 1;
    switch (elem) {
        case EOQ_B200_SYM_I8: f(Source<int8_t>{static_cast<const int8_t *>(sym), shift, top, clamp}); return true;
        case EOQ_B200_SYM_U8: f(Source<uint8_t>{static_cast<const uint8_t *>(sym), shift, top, clamp}); return true;
        case EOQ_B200_SYM_I16: f(Source<int16_t>{static_cast<const int16_t *>(sym), shift, top, clamp}); return true;
        case EOQ_B200_SYM_U16: f(Source<uint16_t>{static_cast<const uint16_t *>(sym), shift, top, clamp}); return true;
        case EOQ_B200_SYM_I32: f(Source<int32_t>{static_cast<const int32_t *>(sym), shift, top, clamp}); return true;
        case EOQ_B200_SYM_U32: f(Source<uint32_t>{static_cast<const uint32_t *>(sym), shift, top, clamp}); return true;
        case EOQ_B200_SYM_I64: f(Source<int64_t>{static_cast<const int64_t *>(sym), shift, top, clamp}); return true;
    }
    return false;
}

template <typename T, typename D>
static bool narrow(const T *p, size_t n, int64_t shift, bool clamp, int64_t top, D *out)
{
    bool outside = false;
    if (sizeof(T) <= 2 && shift > -(1 << 24) && shift < (1 << 24)) {
        const int32_t s = (int32_t)shift, t = (int32_t)top;
        for (size_t i = 0; i < n; i++) {
            const int32_t v = (int32_t)p[i] + s, c = v < 0 ? 0 : v > t ? t : v;
            outside |= c != v;
            out[i] = (D)c;
        }
    } else if (!clamp) {
        // (no compare in the loop, which the compiler then vectorises: bits above the result's, and a second look at the results)
        uint64_t high = 0;
        D most = 0;
        for (size_t i = 0; i < n; i++) {
            const uint64_t v = (uint64_t)((int64_t)p[i] + shift);
            high |= v;
            out[i] = (D)v;
        }
        for (size_t i = 0; i < n; i++) most = std::max(most, out[i]);
        return (high >> (8 * sizeof(D))) == 0 && (int64_t)most <= top;
    } else {
        for (size_t i = 0; i < n; i++) {
            const int64_t v = (int64_t)p[i] + shift, c = v < 0 ? 0 : v > top ? top : v;
            outside |= c != v;
            out[i] = (D)c;
        }
    }
    return clamp || !outside;
}

bool wire_narrow(const void *symbols, int elem, size_t lo, size_t n, int64_t shift, bool clamp, uint32_t alphabet, void *out)
{
    bool fine = false;
    by_type(symbols, elem, shift, clamp, alphabet, [&](auto src) {
        fine = alphabet <= 256 ? narrow(src.p + lo, n, shift, clamp, src.top, static_cast<uint8_t *>(out))
                               : narrow(src.p + lo, n, shift, clamp, src.top, static_cast<uint16_t *>(out));
    });
    return fine;
}

bool wire_table(const uint32_t *freq, uint32_t alphabet, uint32_t p, std::vector<uint32_t> &words)
{
    words.resize((size_t)alphabet * 4);
    uint64_t sum = 0;
    for (uint32_t s = 0; s < alphabet; s++) {
        if (freq[s] == 0 || freq[s] > 1u << p) return false;
        const uint64_t m = (1ull << 48) / freq[s] + 1;
        words[4 * s] = (uint32_t)m; words[4 * s + 1] = (uint32_t)(m >> 32); words[4 * s + 2] = freq[s]; words[4 * s + 3] = (uint32_t)sum;
        sum += freq[s];
    }
    return sum == 1ull << p;
}

}  // namespace eoq

using namespace eoq;

struct eoq_b200_wire { WireEncoded enc; };

extern "C" eoq_error_t eoq_b200_count_symbols(const void *symbols, int elem, size_t n, int64_t shift, int clamp, uint32_t alphabet,
                                              uint64_t *counts, int64_t *range)
{
    if (!counts || !range || (n && !symbols)) return EOQ_ERR_NULL_PTR;
    if (alphabet == 0) return EOQ_ERR_INVALID_HEADER;
    range[0] = range[1] = 0;
    if (!by_type(symbols, elem, shift, clamp != 0, alphabet,
                 [&](auto src) { count_range(src, n, alphabet, counts, range[0], range[1]); })) return EOQ_ERR_UNSUPPORTED;
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_wire_encode(const void *symbols, int elem, uint32_t n, int64_t shift, int clamp, const uint32_t *freq,
                                            uint32_t alphabet, uint32_t precision_bits, uint32_t block_size, eoq_b200_wire_t **out, size_t *bytes)
{
    if (!symbols || !freq || !out || !bytes) return EOQ_ERR_NULL_PTR;
    if (n == 0 || alphabet == 0 || block_size == 0 || precision_bits < 1) return EOQ_ERR_INVALID_HEADER;
    if (precision_bits > 16) return EOQ_ERR_UNSUPPORTED;            // the state must fit 32 bits
    const uint32_t M = 1u << precision_bits;
    std::vector<EncSym> tab(alphabet);
    uint64_t sum = 0;
    for (uint32_t s = 0; s < alphabet; s++) {
        if (freq[s] == 0 || freq[s] > M) return EOQ_ERR_INVALID_HEADER;
        tab[s] = EncSym{(1ull << 48) / freq[s] + 1, freq[s], (uint32_t)sum};
        sum += freq[s];
    }
    if (sum != M) return EOQ_ERR_INVALID_HEADER;
    std::unique_ptr<eoq_b200_wire> w(new eoq_b200_wire());
    bool fine = true;
    if (!by_type(symbols, elem, shift, clamp != 0, alphabet,
                 [&](auto src) { fine = encode_ranges(src, n, tab, precision_bits, block_size, w->enc); })) return EOQ_ERR_UNSUPPORTED;
    if (!fine) return EOQ_ERR_CORRUPT_STREAM;
    size_t total = 0;
    for (size_t b : w->enc.bytes) total += b;
    if (total > 0xFFFFFFFFull) return EOQ_ERR_OVERFLOW;
    *bytes = total;
    *out = w.release();
    return EOQ_OK;
}

extern "C" void eoq_b200_wire_take(eoq_b200_wire_t *w, uint8_t *data, uint32_t *offsets)
{
    if (!w) return;
    WireEncoded &e = w->enc;
    const size_t nr = e.buf.size();
    if (data && offsets) {
        std::vector<size_t> at(nr + 1, 0);
        for (size_t r = 0; r < nr; r++) at[r + 1] = at[r] + e.bytes[r];
        parallel_for(nr, [&](size_t r) {
            if (e.bytes[r]) std::memcpy(data + at[r], e.buf[r].get(), e.bytes[r]);
            size_t off = at[r];
            for (size_t b = e.first_block[r]; b < e.first_block[r + 1]; b++) { offsets[b] = (uint32_t)off; off += e.sizes[b]; }
        }, std::min<size_t>(threads_for(e.sizes.size() * 256), 8));
    }
    delete w;
}
