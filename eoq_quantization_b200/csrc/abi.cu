// C ABI of libeoq_b200.so (declarations and reference citations: include/eoq_b200.h).
// Host-side validation mirrors the reference's checks and error codes; all
// decoding runs on the GPU.
#include "eoq_internal.h"

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cuda.h>
#include <cuda_runtime.h>
#include <exception>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <unistd.h>

using namespace eoq;

namespace {

#define CU_TRY(call)                                                                          \
    do {                                                                                      \
        cudaError_t e__ = (call);                                                             \
        if (e__ != cudaSuccess) {                                                             \
            std::fprintf(stderr, "eoq_b200: %s failed: %s\n", #call, cudaGetErrorString(e__)); \
            return EOQ_ERR_CUDA;                                                              \
        }                                                                                     \
    } while (0)

bool have_device()
{
    int n = 0;
    return cudaGetDeviceCount(&n) == cudaSuccess && n > 0;
}

// Owns a set of device allocations; frees them when it goes out of scope.
struct DeviceBuf {
    void *p = nullptr;
    DeviceBuf() = default;
    DeviceBuf(const DeviceBuf &) = delete;
    DeviceBuf &operator=(const DeviceBuf &) = delete;
    ~DeviceBuf() { release(); }
    // A refused allocation is the caller's to report: left set as the runtime's last error it would fail the next launch too.
    cudaError_t alloc(size_t n)
    {
        const cudaError_t e = cudaMalloc(&p, n ? n : 1);
        if (e != cudaSuccess) { p = nullptr; (void)cudaGetLastError(); }
        return e;
    }
    // Out of this library's own memory pool: a model load allocates and a replaced layer releases without the driver mapping
    // and unmapping memory each time (cudaMalloc and cudaFree of the 24 MB of a layer: 0.5 to 10 ms).  The pool keeps at
    // most 256 MB that nobody uses; what is beyond goes back to the driver.
    cudaError_t alloc_pooled(size_t n)
    {
        cudaMemPool_t pool;
        cudaError_t e = cudaGetDevice(&device);
        if (e == cudaSuccess) e = weight_pool(device, pool);
        if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&p, n ? n : 1, pool, nullptr);
        pooled = e == cudaSuccess;
        if (!pooled) { p = nullptr; (void)cudaGetLastError(); }
        return e;
    }
    void take(DeviceBuf &o)
    {
        p = o.p; pooled = o.pooled; device = o.device;
        o.p = nullptr;
    }
    void release()
    {
        if (!p) return;
        if (pooled) {
            int cur = device;
            cudaGetDevice(&cur);
            if (cur != device) cudaSetDevice(device);
            cudaDeviceSynchronize();                 // as cudaFree does: whatever stream still reads it
            cudaFreeAsync(p, nullptr);
            if (cur != device) cudaSetDevice(cur);
        } else {
            cudaFree(p);
        }
        p = nullptr;
    }

  private:
    bool pooled = false;
    int device = 0;
    static cudaError_t weight_pool(int dev, cudaMemPool_t &out)
    {
        static std::mutex *mu = new std::mutex();
        static cudaMemPool_t pools[64] = {};
        if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
        std::lock_guard<std::mutex> lock(*mu);
        if (!pools[dev]) {
            cudaMemPoolProps props = {};
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            cudaError_t e = cudaMemPoolCreate(&pools[dev], &props);
            uint64_t keep = 256ull << 20;
            if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
            if (e != cudaSuccess) { pools[dev] = nullptr; return e; }
        }
        out = pools[dev];
        return cudaSuccess;
    }

  public:
    template <typename T> T *as() const { return reinterpret_cast<T *>(p); }
};

// A part of somebody else's allocation.
struct DeviceView {
    void *p = nullptr;
    template <typename T> T *as() const { return reinterpret_cast<T *>(p); }
};

// Pieces of a validated tensor payload `[u16 freq x A][u32 offsets x B][blocks]`.
struct Payload {
    uint32_t alphabet = 0, p = 0, block = 0, total = 0, nblocks = 0;
    const uint16_t *freq = nullptr;
    const uint8_t *offsets_raw = nullptr;   // may be unaligned
    const uint8_t *stream = nullptr;
    uint32_t stream_bytes = 0;
    std::vector<uint32_t> offsets, sizes;
};

// Checks of eoq_decode_tensor_v2 (eoq_rans_v2.c:586-619), then the per-block
// checks its workers make while decoding (:542-545 offsets, :392 state length),
// done here on the host so nothing corrupt is ever launched.
eoq_error_t parse_payload(const eoq_tensor_header_t *h, const uint8_t *comp, size_t comp_size, size_t out_cap, Payload &pl)
{
    eoq_error_t rc = eoq_validate_header(h);
    if (rc != EOQ_OK) return rc;
    if (out_cap < h->uncompressed_size) return EOQ_ERR_BUFFER_TOO_SMALL;
    if (comp_size < h->compressed_size) return EOQ_ERR_CORRUPT_STREAM;
    pl.alphabet = h->freq_table_size; pl.p = h->precision_bits; pl.block = h->rans_block_size;
    pl.total = h->uncompressed_size;
    pl.nblocks = (uint32_t)(((uint64_t)pl.total + pl.block - 1) / pl.block);
    const uint64_t meta = (uint64_t)pl.alphabet * 2 + (uint64_t)pl.nblocks * 4;
    if (meta > h->compressed_size) return EOQ_ERR_CORRUPT_STREAM;
    pl.freq = reinterpret_cast<const uint16_t *>(comp);
    pl.offsets_raw = comp + (size_t)pl.alphabet * 2;
    pl.stream = comp + meta;
    pl.stream_bytes = h->compressed_size - (uint32_t)meta;
    pl.offsets.resize(pl.nblocks);
    pl.sizes.resize(pl.nblocks);
    std::memcpy(pl.offsets.data(), pl.offsets_raw, (size_t)pl.nblocks * 4);
    for (uint32_t b = 0; b < pl.nblocks; b++) {
        const uint32_t lo = pl.offsets[b];
        const uint32_t hi = b + 1 < pl.nblocks ? pl.offsets[b + 1] : pl.stream_bytes;
        if (hi < lo || hi > pl.stream_bytes) return EOQ_ERR_CORRUPT_STREAM;
        pl.sizes[b] = hi - lo;
        if (pl.sizes[b] && 1u + pl.stream[lo] > pl.sizes[b]) return EOQ_ERR_CORRUPT_STREAM;
    }
    return EOQ_OK;
}

void make_v1_table(const std::vector<uint32_t> &freq, const std::vector<uint32_t> &cdf, uint32_t p, std::vector<V1Table> &t)
{
    t.assign((size_t)1 << p, V1Table{1, 0});
    for (uint32_t s = 0; s + 1 < cdf.size(); s++)
        for (uint32_t k = cdf[s]; k < cdf[s + 1]; k++) t[k] = V1Table{freq[s], (s << 16) | (k - cdf[s])};
}

eoq_error_t table_from_u16(const uint16_t *raw16, uint32_t alphabet, uint32_t p, std::vector<V1Table> &t)
{
    std::vector<uint32_t> raw(alphabet), freq, cdf;
    for (uint32_t s = 0; s < alphabet; s++) { uint16_t v; std::memcpy(&v, raw16 + s, 2); raw[s] = v; }
    eoq_error_t rc = normalize_reference(raw.data(), alphabet, p, freq, cdf);
    if (rc != EOQ_OK) return rc;
    make_v1_table(freq, cdf, p, t);
    return EOQ_OK;
}

// One device allocation that serves a whole decode call (streams, block tables, frequencies, task descriptors,
// outputs): the decode entry points make no allocation per tensor.  Allocations are kept in a small process-wide cache
// between calls (grow-only, at most four, freed at exit), so a loader that decodes tensor after tensor allocates once.
class DeviceArena {
  public:
    DeviceArena() = default;
    DeviceArena(const DeviceArena &) = delete;
    DeviceArena &operator=(const DeviceArena &) = delete;
    ~DeviceArena() { release(); }
    cudaError_t acquire(size_t bytes)
    {
        release();
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        {
            std::lock_guard<std::mutex> lock(cache().mu);
            auto &v = cache().free_list;
            int best = -1;
            for (int i = 0; i < (int)v.size(); i++)
                if (v[i].dev == dev && v[i].cap >= bytes && (best < 0 || v[i].cap < v[best].cap)) best = i;
            if (best < 0)                         // none large enough: recycle the largest of this device rather than keep both
                for (int i = 0; i < (int)v.size(); i++)
                    if (v[i].dev == dev && (best < 0 || v[i].cap > v[best].cap)) best = i;
            if (best >= 0) { cur_ = v[best]; v.erase(v.begin() + best); }
        }
        if (cur_.p && cur_.cap < bytes) { cudaFree(cur_.p); cur_ = Block(); }
        if (!cur_.p) {
            const size_t cap = std::max<size_t>((bytes + (1u << 20)) & ~(size_t)((1u << 20) - 1), 4u << 20);
            e = cudaMalloc(&cur_.p, cap);
            if (e != cudaSuccess) { cur_ = Block(); return e; }
            cur_.cap = cap; cur_.dev = dev;
        }
        return cudaSuccess;
    }
    void release()
    {
        if (!cur_.p) return;
        std::lock_guard<std::mutex> lock(cache().mu);
        if (cache().free_list.size() < 4) cache().free_list.push_back(cur_);
        else cudaFree(cur_.p);
        cur_ = Block();
    }
    // gives the memory back to the device where it is more than `keep`
    void release_beyond(size_t keep)
    {
        if (!cur_.p || cur_.cap <= keep) return;
        cudaFree(cur_.p);
        cur_ = Block();
    }
    // what is kept between calls, back to the device
    static void trim()
    {
        std::lock_guard<std::mutex> lock(cache().mu);
        for (const Block &b : cache().free_list) cudaFree(b.p);
        cache().free_list.clear();
    }
    uint8_t *base() const { return static_cast<uint8_t *>(cur_.p); }

  private:
    struct Block { void *p = nullptr; size_t cap = 0; int dev = 0; };
    struct Cache { std::mutex mu; std::vector<Block> free_list; };
    static Cache &cache() { static Cache *c = new Cache(); return *c; }      // never destroyed: no CUDA call after main
    Block cur_;
};

constexpr size_t kPinnedChunk = 256u << 10, kPinnedThreads = 16, kPinnedBytes = 2 * kPinnedChunk * kPinnedThreads;

std::atomic<int> g_pinned_refused{0};                    // "pinned_refused" in eoq_b200_tune: requests for staging memory are too large to be met

// Page-locked staging memory (8 MB a block), kept between calls: at most two blocks, the rest is given back at once.
class PinnedBlock {
  public:
    PinnedBlock() = default;
    PinnedBlock(const PinnedBlock &) = delete;
    PinnedBlock &operator=(const PinnedBlock &) = delete;
    // False where the system has no such memory to give: the caller copies without it, and the refusal is nobody's error
    // (left set, it would be what the next launch reports).
    bool acquire()
    {
        const bool refused = g_pinned_refused.load() != 0;
        if (!refused) {
            std::lock_guard<std::mutex> lock(cache().mu);
            if (!cache().free_list.empty()) { p_ = cache().free_list.back(); cache().free_list.pop_back(); return true; }
        }
        if (cudaHostAlloc(reinterpret_cast<void **>(&p_), refused ? (size_t)1 << 60 : kPinnedBytes, cudaHostAllocPortable) == cudaSuccess) return true;
        p_ = nullptr;
        (void)cudaGetLastError();
        return false;
    }
    ~PinnedBlock()
    {
        if (!p_) return;
        std::lock_guard<std::mutex> lock(cache().mu);
        if (cache().free_list.size() < 2) cache().free_list.push_back(p_);
        else cudaFreeHost(p_);
    }
    static void trim()
    {
        std::lock_guard<std::mutex> lock(cache().mu);
        for (uint8_t *p : cache().free_list) cudaFreeHost(p);
        cache().free_list.clear();
    }
    uint8_t *chunk(size_t i) const { return p_ + i * kPinnedChunk; }

  private:
    struct Cache { std::mutex mu; std::vector<uint8_t *> free_list; };
    static Cache &cache() { static Cache *c = new Cache(); return *c; }      // never destroyed: no CUDA call after main
    uint8_t *p_ = nullptr;
};

// `bytes` that have to be made on the way to the device, through page-locked memory: `fill(lo, cnt, chunk)` puts bytes
// [lo, lo + cnt) into a chunk of it.  A few threads fill, this one hands the chunks to the copy engine in order and frees their
// slots.  Complete when this returns.  False from a fill: its error, cudaErrorInvalidValue.
template <typename Fill>
cudaError_t upload_filled(PinnedBlock &pinned, void *dst, size_t bytes, cudaStream_t st, size_t threads, Fill &&fill)
{
    constexpr size_t kSlots = kPinnedBytes / kPinnedChunk, kAhead = kSlots / 2;
    const size_t chunks = (bytes + kPinnedChunk - 1) / kPinnedChunk;
    auto size_of = [&](size_t c) { return std::min(kPinnedChunk, bytes - c * kPinnedChunk); };
    auto copy = [&](size_t c) {
        return cudaMemcpyAsync(static_cast<uint8_t *>(dst) + c * kPinnedChunk, pinned.chunk(c % kSlots), size_of(c), cudaMemcpyHostToDevice, st);
    };
    cudaError_t e = cudaSuccess;
    cudaEvent_t done[2] = {nullptr, nullptr};            // behind every kAhead chunks, in turn
    for (cudaEvent_t &ev : done) if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    std::atomic<size_t> next{0}, freed{kSlots};          // chunk to fill next; chunks below this have a slot
    std::unique_ptr<std::atomic<int>[]> filled(new std::atomic<int>[chunks]);
    for (size_t c = 0; c < chunks; c++) filled[c].store(0, std::memory_order_relaxed);
    std::atomic<bool> stop{false};
    auto work = [&] {
        for (size_t c; !stop.load(std::memory_order_relaxed) && (c = next.fetch_add(1)) < chunks;) {
            while (c >= freed.load(std::memory_order_acquire)) { if (stop.load(std::memory_order_relaxed)) return; std::this_thread::yield(); }
            filled[c].store(fill(c * kPinnedChunk, size_of(c), pinned.chunk(c % kSlots)) ? 1 : -1, std::memory_order_release);
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(threads);
    if (threads > 1 && e == cudaSuccess) {
        // (where the system gives no more threads, those that there are fill, or this one)
        try { for (size_t t = 0; t < threads; t++) pool.emplace_back(work); } catch (const std::system_error &) {}
    }
    for (size_t c = 0; e == cudaSuccess && c < chunks; c++) {
        if (pool.empty()) filled[c].store(fill(c * kPinnedChunk, size_of(c), pinned.chunk(c % kSlots)) ? 1 : -1, std::memory_order_relaxed);
        int f;
        while (!(f = filled[c].load(std::memory_order_acquire))) std::this_thread::yield();
        if (f < 0) { e = cudaErrorInvalidValue; break; }
        e = copy(c);
        if (e == cudaSuccess && (c + 1) % kAhead == 0) {
            // the half of the slots that was handed over before this one
            const size_t half = (c + 1) / kAhead;
            e = cudaEventRecord(done[half & 1], st);
            if (e == cudaSuccess && half > 1) { e = cudaEventSynchronize(done[(half - 1) & 1]); freed.store(kSlots + (half - 1) * kAhead, std::memory_order_release); }
        }
    }
    stop.store(true);
    for (std::thread &t : pool) t.join();
    cudaError_t last = cudaEventRecord(done[0], st);     // the staging memory is another call's from here on
    if (last == cudaSuccess) last = cudaEventSynchronize(done[0]);
    for (cudaEvent_t ev : done) if (ev) cudaEventDestroy(ev);
    return e != cudaSuccess ? e : last;
}

// `bytes` of pageable host memory to the device by several threads, each through two chunks of its own.  The source has been
// read when this returns.  For decodes whose symbols threads deliver to the host afterwards (a 7 MB container: 0.1 to 0.2 ms less
// in all than behind one copy by the driver); streams that stay on the device go by the driver's.
cudaError_t upload(void *dst, const void *src, size_t bytes, cudaStream_t st)
{
    const size_t chunks = (bytes + kPinnedChunk - 1) / kPinnedChunk, hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t threads = std::min<size_t>({kPinnedThreads / 2, hw, chunks / 4});
    PinnedBlock pinned;
    if (threads < 2 || !pinned.acquire()) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    std::atomic<int> failed{(int)cudaSuccess};
    parallel_for(threads, [&](size_t t) {
        cudaEvent_t free_again[2] = {nullptr, nullptr};
        cudaError_t r = cudaSetDevice(device);
        for (cudaEvent_t &ev : free_again) if (r == cudaSuccess) r = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        int slot = 0;
        for (size_t c = t; r == cudaSuccess && c < chunks; c += threads, slot ^= 1) {
            const size_t lo = c * kPinnedChunk, cnt = std::min(kPinnedChunk, bytes - lo);
            r = cudaEventSynchronize(free_again[slot]);              // never recorded: complete
            if (r != cudaSuccess) break;
            std::memcpy(pinned.chunk(2 * t + slot), static_cast<const uint8_t *>(src) + lo, cnt);
            r = cudaMemcpyAsync(static_cast<uint8_t *>(dst) + lo, pinned.chunk(2 * t + slot), cnt, cudaMemcpyHostToDevice, st);
            if (r == cudaSuccess) r = cudaEventRecord(free_again[slot], st);
        }
        for (cudaEvent_t ev : free_again)
            if (ev) { cudaEventSynchronize(ev); cudaEventDestroy(ev); }      // the staging memory is another call's from here on
        if (r != cudaSuccess) failed.store((int)r);
    }, threads);
    return (cudaError_t)failed.load();
}

// Status words (of resident weights, of a decode's checks): 64 bytes each of page-locked memory that the device can address, dealt out of
// pages (a page-locked allocation per weight, and its release, took 1.5 ms each).  A page whose words have all come
// back is given back unless it is the only one.
class StatusWords {
  public:
    static cudaError_t take(uint32_t **host, uint32_t **dev)
    {
        std::lock_guard<std::mutex> lock(mu());
        Page *page = nullptr;
        for (Page &p : pages()) if (p.used != ~0ull) { page = &p; break; }
        if (!page) {
            Page fresh;
            cudaError_t e = cudaHostAlloc(reinterpret_cast<void **>(&fresh.host), 64 * 64, cudaHostAllocPortable | cudaHostAllocMapped);
            if (e == cudaSuccess) e = cudaHostGetDevicePointer(reinterpret_cast<void **>(&fresh.dev), fresh.host, 0);
            if (e != cudaSuccess) return e;
            pages().push_back(fresh);
            page = &pages().back();
        }
        int slot = 0;
        while ((page->used >> slot) & 1) slot++;
        page->used |= 1ull << slot;
        *host = reinterpret_cast<uint32_t *>(page->host + 64 * slot);
        *dev = reinterpret_cast<uint32_t *>(page->dev + 64 * slot);
        std::memset(*host, 0, 64);
        return cudaSuccess;
    }
    static void give(uint32_t *word)
    {
        if (!word) return;
        std::lock_guard<std::mutex> lock(mu());
        uint8_t *at = reinterpret_cast<uint8_t *>(word);
        for (size_t i = 0; i < pages().size(); i++) {
            Page &p = pages()[i];
            if (at < p.host || at >= p.host + 64 * 64) continue;
            p.used &= ~(1ull << ((at - p.host) / 64));
            if (p.used == 0 && pages().size() > 1) { cudaFreeHost(p.host); pages().erase(pages().begin() + i); }
            return;
        }
    }

  private:
    struct Page { uint8_t *host = nullptr, *dev = nullptr; uint64_t used = 0; };
    static std::mutex &mu() { static std::mutex *m = new std::mutex(); return *m; }
    static std::vector<Page> &pages() { static std::vector<Page> *v = new std::vector<Page>(); return *v; }
};

// One tensor of a decode call.
struct V1Job {
    Payload pl;                         // validated host views of the payload
    std::vector<uint32_t> freq, cdf;    // normalised table
    uint32_t out_elem_bytes = 1;
    void *host_out = nullptr;           // where the symbols go on the host, or
    void *dev_out = nullptr;            // the caller's device buffer
    std::vector<uint8_t> own_payload;   // batch context: the caller's host bytes, kept until launch
    // placement inside the arena
    size_t at_stream = 0, at_offsets = 0, at_sizes = 0, at_freq = 0, at_table = 0, at_out = 0;
    bool lanes = false;
    // blocks checked on the device (`job_verdict` has the outcome): the offsets as they lie in the caller's memory, whatever their alignment
    const uint8_t *raw_offsets = nullptr;
    size_t at_raw = 0, at_verdict = 0;
    uint32_t *verdict = nullptr;        // page-locked, complete once `checked` is; without such memory null both
    cudaEvent_t checked = nullptr;
    V1Job() = default;
    V1Job(const V1Job &) = delete;
    V1Job &operator=(const V1Job &) = delete;
    ~V1Job()
    {
        if (checked) cudaEventDestroy(checked);
        StatusWords::give(verdict);
    }
};

eoq_error_t job_from_payload(const eoq_tensor_header_t *h, const uint8_t *comp, size_t comp_size, size_t out_cap, V1Job &j)
{
    eoq_error_t rc = parse_payload(h, comp, comp_size, out_cap, j.pl);
    if (rc != EOQ_OK) return rc;
    std::vector<uint32_t> raw(j.pl.alphabet);
    for (uint32_t s = 0; s < j.pl.alphabet; s++) { uint16_t v; std::memcpy(&v, j.pl.freq + s, 2); raw[s] = v; }
    return normalize_reference(raw.data(), j.pl.alphabet, j.pl.p, j.freq, j.cdf);
}

// Decode `n` validated jobs: one arena, one upload of all metadata, the streams copied in, ONE launch of the lane kernel
// over every job it serves (others run the one-thread-per-block kernel), results copied to the host buffers that ask
// for it (with copy_out false they stay in the arena, at at_out, for the caller to fetch).  Asynchronous on `st`; the arena must stay acquired until the stream has been synchronised.
eoq_error_t decode_jobs(V1Job **jobs, size_t n, cudaStream_t st, DeviceArena &arena, bool copy_out = true)
{
    if (n == 0) return EOQ_OK;
    if (!have_device()) return EOQ_ERR_CUDA;
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    // layout: [metadata blob: per job offsets, sizes, freq (or slot table); task descriptors; CTA map][streams][outputs]
    std::vector<V1Task> tasks;
    std::vector<size_t> task_job;
    size_t meta = 0;
    for (size_t i = 0; i < n; i++) {
        V1Job &j = *jobs[i];
        if (j.raw_offsets) { j.at_verdict = meta; meta = up(meta + 4); }
        else {
            j.at_offsets = meta; meta = up(meta + (size_t)j.pl.nblocks * 4);
            j.at_sizes = meta;   meta = up(meta + (size_t)j.pl.nblocks * 4);
        }
        j.at_freq = meta;    meta = up(meta + (size_t)j.pl.alphabet * 4);
        V1Task t = {};
        t.nblocks = j.pl.nblocks; t.block_size = j.pl.block; t.total = j.pl.total; t.p = j.pl.p; t.alphabet = j.pl.alphabet;
        t.out_elem_bytes = j.out_elem_bytes;
        t.stream = reinterpret_cast<const uint8_t *>((uintptr_t)0);       // alignment is that of the arena slice: always 256
        j.lanes = v1_lanes_enabled() && v1_task_prepare(t);
        if (j.lanes) { tasks.push_back(t); task_job.push_back(i); }
        else { j.at_table = meta; meta = up(meta + ((size_t)8 << j.pl.p)); }
    }
    uint32_t warps_per_cta = 1, grid = 0;
    size_t smem = 0;
    if (!tasks.empty()) grid = v1_plan_ctas(tasks.data(), (uint32_t)tasks.size(), warps_per_cta, smem);
    const size_t at_tasks = meta; meta = up(meta + tasks.size() * sizeof(V1Task));
    const size_t at_cta = meta;   meta = up(meta + (size_t)grid * 4);
    size_t total = meta;
    for (size_t i = 0; i < n; i++) {
        V1Job &j = *jobs[i];
        j.at_stream = total; total = up(total + j.pl.stream_bytes + 16);
        if (j.raw_offsets) {
            j.at_raw = total;     total = up(total + (size_t)j.pl.nblocks * 4);
            j.at_offsets = total; total = up(total + (size_t)j.pl.nblocks * 4);
            j.at_sizes = total;   total = up(total + (size_t)j.pl.nblocks * 4);
        }
        if (!j.dev_out) { j.at_out = total; total = up(total + (size_t)j.pl.total * j.out_elem_bytes + 32); }
    }
    if (arena.acquire(total) != cudaSuccess) return EOQ_ERR_ALLOC;
    uint8_t *d = arena.base();
    std::vector<uint8_t> blob(meta, 0);
    for (size_t i = 0; i < n; i++) {
        V1Job &j = *jobs[i];
        if (j.raw_offsets) std::memset(blob.data() + j.at_verdict, 0xFF, 4);
        else {
            std::memcpy(blob.data() + j.at_offsets, j.pl.offsets.data(), (size_t)j.pl.nblocks * 4);
            std::memcpy(blob.data() + j.at_sizes, j.pl.sizes.data(), (size_t)j.pl.nblocks * 4);
        }
        std::memcpy(blob.data() + j.at_freq, j.freq.data(), (size_t)j.pl.alphabet * 4);
        if (!j.lanes) {
            std::vector<V1Table> table;
            make_v1_table(j.freq, j.cdf, j.pl.p, table);
            std::memcpy(blob.data() + j.at_table, table.data(), table.size() * sizeof(V1Table));
        }
    }
    std::vector<uint32_t> cta_task(grid);
    for (size_t k = 0; k < tasks.size(); k++) {
        V1Job &j = *jobs[task_job[k]];
        V1Task &t = tasks[k];
        t.stream = d + j.at_stream; t.offsets = reinterpret_cast<const uint32_t *>(d + j.at_offsets);
        t.sizes = reinterpret_cast<const uint32_t *>(d + j.at_sizes); t.freq = reinterpret_cast<const uint32_t *>(d + j.at_freq);
        t.table = nullptr; t.out = j.dev_out ? j.dev_out : d + j.at_out;
        const uint32_t last = k + 1 < tasks.size() ? tasks[k + 1].first_cta : grid;
        for (uint32_t c = t.first_cta; c < last; c++) cta_task[c] = (uint32_t)k;
    }
    if (!tasks.empty()) {
        std::memcpy(blob.data() + at_tasks, tasks.data(), tasks.size() * sizeof(V1Task));
        std::memcpy(blob.data() + at_cta, cta_task.data(), (size_t)grid * 4);
    }
    // pageable sources are consumed before cudaMemcpyAsync returns (the driver stages them at some 27 GB/s; several threads that
    // staged them through page-locked memory of this library's took 1.2 to 1.6 ms for 19 MB, this way takes 0.75)
    CU_TRY(cudaMemcpyAsync(d, blob.data(), meta, cudaMemcpyHostToDevice, st));
    for (size_t i = 0; i < n; i++) {
        V1Job &j = *jobs[i];
        if (j.pl.stream_bytes) CU_TRY(j.dev_out ? cudaMemcpyAsync(d + j.at_stream, j.pl.stream, j.pl.stream_bytes, cudaMemcpyHostToDevice, st) : upload(d + j.at_stream, j.pl.stream, j.pl.stream_bytes, st));
        if (j.raw_offsets) {
            CU_TRY(cudaMemcpyAsync(d + j.at_raw, j.raw_offsets, (size_t)j.pl.nblocks * 4, cudaMemcpyHostToDevice, st));
            if (launch_v1_check(d + j.at_stream, j.pl.stream_bytes, reinterpret_cast<const uint32_t *>(d + j.at_raw), j.pl.nblocks,
                                reinterpret_cast<uint32_t *>(d + j.at_offsets), reinterpret_cast<uint32_t *>(d + j.at_sizes),
                                reinterpret_cast<uint32_t *>(d + j.at_verdict), st) != 0)
                return EOQ_ERR_CUDA;
            uint32_t *unused;
            if (g_pinned_refused.load() == 0 && StatusWords::take(&j.verdict, &unused) == cudaSuccess &&
                cudaEventCreateWithFlags(&j.checked, cudaEventDisableTiming) == cudaSuccess) {
                CU_TRY(cudaMemcpyAsync(j.verdict, d + j.at_verdict, 4, cudaMemcpyDeviceToHost, st));
                CU_TRY(cudaEventRecord(j.checked, st));
            } else {
                j.checked = nullptr;
                (void)cudaGetLastError();
            }
        }
    }
    if (!tasks.empty()) {
        int e = launch_decode_v1_lanes(reinterpret_cast<const V1Task *>(d + at_tasks), reinterpret_cast<const uint32_t *>(d + at_cta), grid,
                                       warps_per_cta, smem, st);
        if (e != 0) { std::fprintf(stderr, "eoq_b200: decode launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    }
    for (size_t i = 0; i < n; i++) {
        V1Job &j = *jobs[i];
        void *out = j.dev_out ? j.dev_out : d + j.at_out;
        if (!j.lanes) {
            int e = launch_decode_v1(d + j.at_stream, reinterpret_cast<const uint32_t *>(d + j.at_offsets),
                                     reinterpret_cast<const uint32_t *>(d + j.at_sizes), reinterpret_cast<const V1Table *>(d + j.at_table), out,
                                     (int)j.out_elem_bytes, j.pl.nblocks, j.pl.block, j.pl.total, j.pl.p, j.pl.alphabet, st);
            if (e != 0) { std::fprintf(stderr, "eoq_b200: decode launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
        }
        if (j.host_out && copy_out) CU_TRY(cudaMemcpyAsync(j.host_out, out, (size_t)j.pl.total * j.out_elem_bytes, cudaMemcpyDeviceToHost, st));
    }
    return EOQ_OK;
}

// What the checks on the device found, in the order in which the host's would have: waits for them, and not for the decoder behind
// them (but where there is no page-locked memory).
eoq_error_t job_verdict(const V1Job &j, const DeviceArena &arena, cudaStream_t st)
{
    uint32_t v = 0;
    if (j.checked) {
        CU_TRY(cudaEventSynchronize(j.checked));
        v = *static_cast<volatile uint32_t *>(j.verdict);
    } else {
        CU_TRY(cudaMemcpyAsync(&v, arena.base() + j.at_verdict, 4, cudaMemcpyDeviceToHost, st));
        CU_TRY(cudaStreamSynchronize(st));
    }
    return v == ~0u ? EOQ_OK : v & 1u ? EOQ_ERR_UNSUPPORTED : EOQ_ERR_CORRUPT_STREAM;
}

eoq_error_t decode_host_to_host(const eoq_tensor_header_t *h, const uint8_t *comp, size_t comp_size, void *output,
                                size_t out_cap, cudaStream_t st)
{
    V1Job job;
    eoq_error_t rc = job_from_payload(h, comp, comp_size, out_cap, job);
    if (rc != EOQ_OK) return rc;
    job.host_out = output;
    V1Job *one = &job;
    DeviceArena arena;
    rc = decode_jobs(&one, 1, st, arena);
    if (rc != EOQ_OK) return rc;
    CU_TRY(cudaStreamSynchronize(st));
    return EOQ_OK;
}

}  // namespace

// =========================================================================
// Part 1: the reference's C interface
// =========================================================================

extern "C" const char *eoq_error_string(eoq_error_t err)
{
    switch (err) {
        case EOQ_OK: return "success";
        case EOQ_ERR_NULL_PTR: return "null pointer argument";
        case EOQ_ERR_BUFFER_TOO_SMALL: return "output buffer too small";
        case EOQ_ERR_CORRUPT_STREAM: return "corrupt compressed stream";
        case EOQ_ERR_INVALID_HEADER: return "invalid tensor header";
        case EOQ_ERR_ALLOC: return "memory allocation failed";
        case EOQ_ERR_THREAD: return "threading error";
        case EOQ_ERR_OVERFLOW: return "integer overflow";
        case EOQ_ERR_CUDA: return "CUDA device unavailable or CUDA call failed";
        case EOQ_ERR_UNSUPPORTED: return "input not supported by this build";
    }
    return "unknown error";
}

extern "C" eoq_error_t eoq_validate_header(const eoq_tensor_header_t *h)
{
    if (!h) return EOQ_ERR_NULL_PTR;
    if (h->freq_table_size == 0 || h->freq_table_size > 4096) return EOQ_ERR_INVALID_HEADER;
    if (h->precision_bits == 0 || h->precision_bits > 16) return EOQ_ERR_INVALID_HEADER;
    if (h->rans_block_size == 0) return EOQ_ERR_INVALID_HEADER;
    if ((uint64_t)h->compressed_size < (uint64_t)h->freq_table_size * 2 + 4) return EOQ_ERR_INVALID_HEADER;
    return EOQ_OK;
}

extern "C" int eoq_detect_num_threads(void)
{
    long n = sysconf(_SC_NPROCESSORS_ONLN);
    if (n > 0) return (int)n;
    n = sysconf(_SC_NPROCESSORS_CONF);
    return n > 0 ? (int)n : 4;
}

extern "C" eoq_error_t eoq_decode_tensor_v2(const eoq_tensor_header_t *header, const uint8_t *compressed, size_t comp_size,
                                            void *output, size_t out_cap, const eoq_decode_opts_t *opts)
{
    if (!header || !compressed || !output) return EOQ_ERR_NULL_PTR;
    if (header->uncompressed_size == 0) return EOQ_OK;
    eoq_error_t rc = decode_host_to_host(header, compressed, comp_size, output, out_cap, nullptr);
    // the whole tensor is one launch, so progress is reported once, complete (eoq_rans_v2.c:757-762)
    if (rc == EOQ_OK && opts && opts->progress_cb)
        opts->progress_cb(header->uncompressed_size, header->uncompressed_size, opts->progress_ud);
    return rc;
}

extern "C" int eoq_decode_tensor(const eoq_tensor_header_t *header, const uint8_t *compressed, void *output)
{
    if (!header) return (int)EOQ_ERR_NULL_PTR;
    return (int)eoq_decode_tensor_v2(header, compressed, header->compressed_size, output, header->uncompressed_size, nullptr);
}

// Tensors are decoded in groups: the tasks of a group are validated on the host, uploaded together and decoded by ONE
// kernel launch (every rANS block of every tensor of the group is a lane of that launch).  A group is as many tasks as
// fit 256 tasks and 256 MB of symbols, whatever opts->num_threads says: the launch is only efficient when it is wide.
// Results are then delivered in task order, opts->num_threads tasks at a time (the number of tasks the reference would
// have in flight; 64 when it is 0): their symbols are copied to the callers' buffers, then the progress callback runs
// on the calling thread for each, so calls are serialised and count up by one.  After a cancel request the tasks being
// delivered complete; the rest get EOQ_ERR_THREAD and their buffers are not written, decoded on the device or not.
extern "C" eoq_error_t eoq_parallel_decode(eoq_decode_task_t *tasks, int num_tasks, const eoq_parallel_opts_t *opts)
{
    if (!tasks && num_tasks > 0) return EOQ_ERR_NULL_PTR;
    if (num_tasks <= 0) return EOQ_OK;
    int deliver = opts ? opts->num_threads : 0;
    deliver = deliver <= 0 ? 64 : std::min(deliver, 256);
    constexpr int kGroupTasks = 256;
    constexpr uint64_t kGroupSymbols = 256ull << 20;
    eoq_parallel_progress_fn cb = opts ? opts->progress_cb : nullptr;
    void *ud = opts ? opts->progress_ud : nullptr;
    cudaStream_t st = nullptr;
    const bool device_ok = have_device() && cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess;

    int done = 0;
    bool cancelled = false;
    DeviceArena arena;
    for (int g0 = 0; g0 < num_tasks;) {
        int g1 = g0;
        uint64_t symbols = 0;
        while (g1 < num_tasks && g1 - g0 < kGroupTasks) {
            const uint64_t add = tasks[g1].header ? tasks[g1].header->uncompressed_size : 0;
            if (g1 > g0 && symbols + add > kGroupSymbols) break;
            symbols += add;
            g1++;
        }
        if (cancelled) {
            for (int i = g0; i < g1; i++) tasks[i].result = EOQ_ERR_THREAD;          // eoq_parallel_decode.c:72-82
            g0 = g1;
            continue;
        }
        std::vector<std::unique_ptr<V1Job>> jobs;
        std::vector<V1Job *> live;
        std::vector<V1Job *> job_of(g1 - g0, nullptr);
        for (int i = g0; i < g1; i++) {
            eoq_decode_task_t &t = tasks[i];
            t.task_index = i;
            if (!t.header || !t.compressed_data || !t.output) { t.result = EOQ_ERR_NULL_PTR; continue; }
            if (t.header->uncompressed_size == 0) { t.result = EOQ_OK; continue; }
            std::unique_ptr<V1Job> j(new V1Job());
            t.result = job_from_payload(t.header, t.compressed_data, t.compressed_size, t.output_capacity, *j);
            if (t.result == EOQ_OK && !device_ok) t.result = EOQ_ERR_CUDA;
            if (t.result != EOQ_OK) continue;
            j->host_out = t.output;
            live.push_back(j.get());
            job_of[i - g0] = j.get();
            jobs.push_back(std::move(j));
        }
        eoq_error_t rc = live.empty() ? EOQ_OK : decode_jobs(live.data(), live.size(), st, arena, /*copy_out=*/false);
        for (int d0 = g0; d0 < g1; d0 += deliver) {
            const int d1 = std::min(g1, d0 + deliver);
            if (cancelled) {
                for (int i = d0; i < d1; i++) tasks[i].result = EOQ_ERR_THREAD;
                continue;
            }
            eoq_error_t drc = rc;
            bool any = false;
            for (int i = d0; i < d1 && drc == EOQ_OK; i++) {
                const V1Job *j = job_of[i - g0];
                if (!j) continue;
                any = true;
                if (cudaMemcpyAsync(j->host_out, arena.base() + j->at_out, (size_t)j->pl.total * j->out_elem_bytes, cudaMemcpyDeviceToHost, st) != cudaSuccess)
                    drc = EOQ_ERR_CUDA;
            }
            if (drc == EOQ_OK && any && cudaStreamSynchronize(st) != cudaSuccess) drc = EOQ_ERR_CUDA;
            for (int i = d0; i < d1; i++) {
                if (job_of[i - g0] && drc != EOQ_OK) tasks[i].result = drc;
                done++;
                if (cb && !cancelled && cb(done, num_tasks, ud)) cancelled = true;
            }
        }
        if (!live.empty()) cudaStreamSynchronize(st);            // the arena is reused by the next group
        g0 = g1;
    }
    arena.release();
    if (st) cudaStreamDestroy(st);

    for (int i = 0; i < num_tasks; i++)
        if (tasks[i].result != EOQ_OK) return tasks[i].result;        // eoq_parallel_decode.c:290-300
    return EOQ_OK;
}

// -- incremental single-block decoder --------------------------------------
namespace {
struct DecoderDev {
    DeviceBuf table, block, state_pos, out;
    size_t out_cap = 0;
    uint32_t stream_off = 0;
};
}

extern "C" eoq_error_t eoq_decoder_init(eoq_decoder_t *dec, const uint16_t *freq_table, uint32_t alphabet_size,
                                        uint32_t precision_bits, const uint8_t *block_data, size_t block_size)
{
    if (!dec || !freq_table || !block_data) return EOQ_ERR_NULL_PTR;
    if (alphabet_size == 0 || alphabet_size > 4096) return EOQ_ERR_INVALID_HEADER;
    if (precision_bits == 0 || precision_bits > 16) return EOQ_ERR_INVALID_HEADER;
    dec->precision_bits = precision_bits;
    dec->precision_mask = (1u << precision_bits) - 1;
    dec->sym_info = nullptr;
    dec->state = 0; dec->stream = block_data; dec->stream_pos = 0; dec->stream_end = 0;
    std::vector<V1Table> table;
    eoq_error_t rc = table_from_u16(freq_table, alphabet_size, precision_bits, table);
    if (rc != EOQ_OK) return rc;
    uint32_t state = 0, off = 0;
    if (block_size > 0) {
        const uint32_t sl = block_data[0];
        if ((size_t)1 + sl > block_size) return EOQ_ERR_CORRUPT_STREAM;
        for (uint32_t i = 0; i < sl; i++) state = (state << 8) | block_data[1 + i];
        off = 1 + sl;
        dec->stream = block_data + off;
        dec->stream_end = block_size - off;
    }
    dec->state = state;
    if (!have_device()) return EOQ_ERR_CUDA;
    std::unique_ptr<DecoderDev> d(new DecoderDev());
    d->stream_off = off;
    if (d->table.alloc(table.size() * sizeof(V1Table)) != cudaSuccess || d->block.alloc(block_size) != cudaSuccess ||
        d->state_pos.alloc(8) != cudaSuccess)
        return EOQ_ERR_ALLOC;
    const uint32_t sp[2] = {state, 0};
    CU_TRY(cudaMemcpy(d->table.p, table.data(), table.size() * sizeof(V1Table), cudaMemcpyHostToDevice));
    if (block_size) CU_TRY(cudaMemcpy(d->block.p, block_data, block_size, cudaMemcpyHostToDevice));
    CU_TRY(cudaMemcpy(d->state_pos.p, sp, 8, cudaMemcpyHostToDevice));
    dec->sym_info = reinterpret_cast<struct eoq_sym_info *>(d.release());
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_decoder_decode(eoq_decoder_t *dec, uint8_t *out, uint32_t count)
{
    if (!dec || !out) return EOQ_ERR_NULL_PTR;
    if (!dec->sym_info) return EOQ_ERR_NULL_PTR;
    if (count == 0) return EOQ_OK;
    DecoderDev *d = reinterpret_cast<DecoderDev *>(dec->sym_info);
    if (d->out_cap < count) {
        if (d->out.p) { cudaFree(d->out.p); d->out.p = nullptr; }
        if (d->out.alloc(count) != cudaSuccess) return EOQ_ERR_ALLOC;
        d->out_cap = count;
    }
    int e = launch_decode_v1_resume(d->block.as<uint8_t>() + d->stream_off, (uint32_t)dec->stream_end, d->table.as<V1Table>(),
                                    d->state_pos.as<uint32_t>(), d->out.as<uint8_t>(), count, dec->precision_bits, nullptr);
    if (e != 0) return EOQ_ERR_CUDA;
    uint32_t sp[2];
    CU_TRY(cudaMemcpy(out, d->out.p, count, cudaMemcpyDeviceToHost));
    CU_TRY(cudaMemcpy(sp, d->state_pos.p, 8, cudaMemcpyDeviceToHost));
    dec->state = sp[0];
    dec->stream_pos = sp[1];
    return EOQ_OK;
}

extern "C" void eoq_decoder_free(eoq_decoder_t *dec)
{
    if (dec && dec->sym_info) {
        delete reinterpret_cast<DecoderDev *>(dec->sym_info);
        dec->sym_info = nullptr;
    }
}

// -- eoq_cuda_* family -------------------------------------------------------

extern "C" int eoq_cuda_decode_tensor(const eoq_tensor_header_t *header, const uint8_t *compressed, uint8_t *output, void *stream)
{
    if (!header || !compressed || !output) return -1;
    if (header->uncompressed_size == 0) return 0;
    return decode_host_to_host(header, compressed, header->compressed_size, output, header->uncompressed_size,
                               reinterpret_cast<cudaStream_t>(stream)) == EOQ_OK ? 0 : -1;
}

extern "C" int eoq_cuda_decode_tensor_device(const uint8_t *d_compressed_stream, const uint32_t *d_block_offsets,
                                             const uint32_t *d_block_sizes, const eoq_sym_info_packed *d_sym_info,
                                             uint8_t *d_output, uint32_t num_rans_blocks, uint32_t rans_block_size,
                                             uint32_t total_symbols, uint32_t precision_bits, void *cuda_stream)
{
    if (total_symbols == 0) return 0;
    if (!d_compressed_stream || !d_block_offsets || !d_block_sizes || !d_sym_info || !d_output) return -1;
    if (precision_bits == 0 || precision_bits > 16 || rans_block_size == 0) return -1;
    if (!have_device()) return -1;
    int e = launch_decode_v1_syminfo(d_compressed_stream, d_block_offsets, d_block_sizes, d_sym_info, d_output,
                                     num_rans_blocks, rans_block_size, total_symbols, precision_bits, cuda_stream);
    if (e != 0) { std::fprintf(stderr, "eoq_cuda_decode_tensor_device: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return -1; }
    return 0;
}

namespace {
struct BatchImpl {
    std::vector<std::unique_ptr<V1Job>> tensors;
    DeviceArena arena;
    bool launched = false;
};
BatchImpl *batch_impl(eoq_cuda_batch_ctx_t *ctx, bool make)
{
    if (!ctx->impl && make) ctx->impl = new (std::nothrow) BatchImpl();
    return static_cast<BatchImpl *>(ctx->impl);
}
}  // namespace

extern "C" void eoq_cuda_batch_init(eoq_cuda_batch_ctx_t *ctx, void *stream)
{
    if (!ctx) return;
    std::memset(ctx, 0, sizeof(*ctx));
    ctx->stream = stream;
}

extern "C" eoq_cuda_batch_ctx_t *eoq_cuda_batch_create(void *stream)
{
    eoq_cuda_batch_ctx_t *c = new (std::nothrow) eoq_cuda_batch_ctx_t();
    if (c) eoq_cuda_batch_init(c, stream);
    return c;
}

extern "C" int eoq_cuda_batch_prepare_tensor(eoq_cuda_batch_ctx_t *ctx, const eoq_tensor_header_t *header,
                                             const uint8_t *compressed_host, uint8_t *d_output)
{
    if (!ctx || !header || !compressed_host || !d_output) return -1;
    if (ctx->n_tensors >= EOQ_CUDA_MAX_BATCH_TENSORS) {                  // eoq_cuda_decompress.cu:906-910
        std::fprintf(stderr, "eoq_cuda_batch_prepare_tensor: batch full (%d tensors)\n", EOQ_CUDA_MAX_BATCH_TENSORS);
        return -1;
    }
    if (header->uncompressed_size == 0) return 0;
    BatchImpl *impl = batch_impl(ctx, true);
    if (!impl) return -1;
    // the caller may release its host buffer after this call (the reference uploads here): keep a copy until launch
    std::unique_ptr<V1Job> j(new V1Job());
    j->own_payload.assign(compressed_host, compressed_host + header->compressed_size);
    if (job_from_payload(header, j->own_payload.data(), header->compressed_size, header->uncompressed_size, *j) != EOQ_OK) return -1;
    j->dev_out = d_output;
    impl->tensors.push_back(std::move(j));
    ctx->n_tensors = (uint32_t)impl->tensors.size();
    return 0;
}

// One kernel launch decodes every prepared tensor (eoq_cuda_decompress.cu:985-1003 launches one kernel per tensor).
extern "C" int eoq_cuda_batch_launch(eoq_cuda_batch_ctx_t *ctx)
{
    if (!ctx) return -1;
    BatchImpl *impl = batch_impl(ctx, false);
    if (!impl || impl->tensors.empty() || impl->launched) return 0;
    std::vector<V1Job *> live;
    for (auto &t : impl->tensors) live.push_back(t.get());
    if (decode_jobs(live.data(), live.size(), reinterpret_cast<cudaStream_t>(ctx->stream), impl->arena) != EOQ_OK) return -1;
    impl->launched = true;
    return 0;
}

extern "C" int eoq_cuda_batch_sync_and_free(eoq_cuda_batch_ctx_t *ctx)
{
    if (!ctx) return -1;
    int rc = 0;
    BatchImpl *impl = batch_impl(ctx, false);
    if (impl && impl->launched && cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(ctx->stream)) != cudaSuccess) rc = -1;
    delete impl;                   // releases the staging arena; outputs belong to the caller
    ctx->impl = nullptr;
    ctx->n_tensors = 0;
    return rc;
}

extern "C" void eoq_cuda_batch_destroy(eoq_cuda_batch_ctx_t *ctx)
{
    if (!ctx) return;
    delete batch_impl(ctx, false);
    delete ctx;
}

// =========================================================================
// Part 2: Python-facing codec entry points and the fused path
// =========================================================================

// Blocks up to which the checks stay on the host: some 5 ns a block, against one more copy, launch and wait, some 14 us. Decodes
// to int8 of blocks of 256, host's checks and device's: 2048 blocks 180 and 192 us, 5154 347 and 314, 65536 2111 and 1806.
// (And from 2^30 blocks on, where a verdict would not hold the block's number.)
constexpr uint32_t kHostChecks = 4096;
static bool checks_on_device(uint32_t num_blocks) { return num_blocks > kHostChecks && num_blocks < (1u << 30); }

// Validates a blocked stream, as the reference's decoders do block by block, and makes it a job: on the host, but for the blocks where
// `check_on_device` and there are many.
static eoq_error_t blocked_job(const uint32_t *freq, uint32_t alphabet, uint32_t precision_bits, const uint8_t *data, size_t data_len,
                               const uint32_t *offsets, uint32_t num_blocks, uint32_t block_size, uint32_t num_symbols,
                               int out_elem_bytes, V1Job &job, bool check_on_device = false)
{
    if (!freq || !data || !offsets) return EOQ_ERR_NULL_PTR;
    if (alphabet == 0 || block_size == 0) return EOQ_ERR_INVALID_HEADER;
    if (precision_bits < 1 || precision_bits > 16) return EOQ_ERR_UNSUPPORTED;   // 32-bit device state
    if (out_elem_bytes != 1 && out_elem_bytes != 2) return EOQ_ERR_UNSUPPORTED;
    if (alphabet > (out_elem_bytes == 1 ? 256u : 65536u)) return EOQ_ERR_UNSUPPORTED;
    if (data_len > 0xFFFFFFFFull) return EOQ_ERR_OVERFLOW;
    if (num_blocks != (uint32_t)(((uint64_t)num_symbols + block_size - 1) / block_size)) return EOQ_ERR_INVALID_HEADER;
    uint64_t sum = 0;
    std::vector<uint32_t> f(freq, freq + alphabet), cdf(alphabet + 1, 0);
    for (uint32_t s = 0; s < alphabet; s++) { sum += f[s]; cdf[s + 1] = cdf[s] + f[s]; }
    if (sum != (1ull << precision_bits)) return EOQ_ERR_INVALID_HEADER;
    // (a look at the first byte of each of 176 K blocks of a cold 19 MB stream takes 1.5 ms here, a few microseconds on the device)
    check_on_device = check_on_device && checks_on_device(num_blocks);
    std::vector<uint32_t> sizes(check_on_device ? 0 : num_blocks);
    for (uint32_t b = 0; b < (uint32_t)sizes.size(); b++) {
        const uint64_t lo = offsets[b], hi = b + 1 < num_blocks ? offsets[b + 1] : data_len;
        if (hi < lo || hi > data_len) return EOQ_ERR_CORRUPT_STREAM;
        sizes[b] = (uint32_t)(hi - lo);
        if (sizes[b] && 1u + data[lo] > sizes[b]) return EOQ_ERR_CORRUPT_STREAM;
        if (sizes[b] && data[lo] > 4) return EOQ_ERR_UNSUPPORTED;                  // state wider than 32 bits
    }
    job.pl.alphabet = alphabet; job.pl.p = precision_bits; job.pl.block = block_size; job.pl.total = num_symbols;
    job.pl.nblocks = num_blocks; job.pl.stream = data; job.pl.stream_bytes = (uint32_t)data_len;
    if (check_on_device) job.raw_offsets = reinterpret_cast<const uint8_t *>(offsets);
    else job.pl.offsets.assign(offsets, offsets + num_blocks);
    job.pl.sizes = std::move(sizes);
    job.freq = std::move(f);
    job.cdf = std::move(cdf);
    job.out_elem_bytes = (uint32_t)out_elem_bytes;
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_decode_blocked(const uint32_t *freq, uint32_t alphabet, uint32_t precision_bits,
                                               const uint8_t *data, size_t data_len, const uint32_t *offsets,
                                               uint32_t num_blocks, uint32_t block_size, uint32_t num_symbols,
                                               void *out, int out_elem_bytes, int out_on_device, void *stream)
{
    if (num_symbols == 0) return EOQ_OK;
    if (!out) return EOQ_ERR_NULL_PTR;
    V1Job job;
    eoq_error_t rc = blocked_job(freq, alphabet, precision_bits, data, data_len, offsets, num_blocks, block_size, num_symbols, out_elem_bytes, job);
    if (rc != EOQ_OK) return rc;
    if (!have_device()) return EOQ_ERR_CUDA;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (out_on_device) job.dev_out = out; else job.host_out = out;
    V1Job *one = &job;
    DeviceArena arena;
    rc = decode_jobs(&one, 1, st, arena);
    if (rc != EOQ_OK) return rc;
    CU_TRY(cudaStreamSynchronize(st));   // the staging arena goes back to the cache on return
    return EOQ_OK;
}

// -- symbols from the device to a host array of another integer type ------------
//
// The decoder leaves one or two bytes per symbol; the Python interface wants int64 (or int8 codes).  Copying the bytes to
// pageable memory and converting them on one core took 22 of the 24 ms of a 4096 x 4096 container: here a few threads
// each move chunks through page-locked memory of their own (two chunks each: one on the bus while the other is
// converted) and write the caller's array, page faults of a fresh array included, side by side: 5 ms.
namespace {

template <typename S, typename D>
void convert(const void *src, void *dst, size_t n, int64_t shift)
{
    const S *s = static_cast<const S *>(src);
    D *d = static_cast<D *>(dst);
    for (size_t i = 0; i < n; i++) d[i] = (D)((int64_t)s[i] + shift);
}

typedef void (*ConvertFn)(const void *, void *, size_t, int64_t);

// This thread's rule for calls beside a stream that is recording (relaxed: allocations and waits are allowed although a stream may be,
// since they have no part in the recording), as long as this lives.
struct CaptureMode {
    cudaStreamCaptureMode mode;
    explicit CaptureMode(cudaStreamCaptureMode m = cudaStreamCaptureModeRelaxed) : mode(m) { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~CaptureMode() { cudaThreadExchangeStreamCaptureMode(&mode); }
    CaptureMode(const CaptureMode &) = delete;
    CaptureMode &operator=(const CaptureMode &) = delete;
    static cudaStreamCaptureMode current() { return CaptureMode().mode; }
};

// Symbols (1 or 2 bytes each on the device, complete on `st`) to `out`, of the type EOQ_B200_SYM_* names.
eoq_error_t deliver(const uint8_t *dev, uint32_t elem, size_t n, void *out, int out_type, int64_t shift, cudaStream_t st)
{
    static const size_t width[7] = {1, 1, 2, 2, 4, 4, 8};
    ConvertFn fn = nullptr;
    switch (out_type) {
        case EOQ_B200_SYM_I8: fn = elem == 1 ? convert<uint8_t, int8_t> : convert<uint16_t, int8_t>; break;
        case EOQ_B200_SYM_U8: fn = elem == 1 ? convert<uint8_t, uint8_t> : convert<uint16_t, uint8_t>; break;
        case EOQ_B200_SYM_I16: fn = elem == 1 ? convert<uint8_t, int16_t> : convert<uint16_t, int16_t>; break;
        case EOQ_B200_SYM_U16: fn = elem == 1 ? convert<uint8_t, uint16_t> : convert<uint16_t, uint16_t>; break;
        case EOQ_B200_SYM_I32: fn = elem == 1 ? convert<uint8_t, int32_t> : convert<uint16_t, int32_t>; break;
        case EOQ_B200_SYM_I64: fn = elem == 1 ? convert<uint8_t, int64_t> : convert<uint16_t, int64_t>; break;
        default: return EOQ_ERR_UNSUPPORTED;
    }
    const size_t per = kPinnedChunk / elem, chunks = (n + per - 1) / per;
    PinnedBlock pinned;
    if (!pinned.acquire()) {
        // through pageable memory, a chunk at a time (such a copy has ended when the call returns)
        std::vector<uint8_t> chunk(std::min(n, per) * elem);
        for (size_t lo = 0; lo < n; lo += per) {
            const size_t cnt = std::min(per, n - lo);
            CU_TRY(cudaMemcpyAsync(chunk.data(), dev + lo * elem, cnt * elem, cudaMemcpyDeviceToHost, st));
            CU_TRY(cudaStreamSynchronize(st));
            fn(chunk.data(), static_cast<uint8_t *>(out) + lo * width[out_type], cnt, shift);
        }
        return EOQ_OK;
    }
    int device = 0;
    CU_TRY(cudaGetDevice(&device));
    // a thread costs some tens of microseconds to start, a chunk of 256 Ki symbols about a hundred to convert to int64
    const size_t hw = std::max(1u, std::thread::hardware_concurrency());
    const size_t threads = std::max<size_t>(1, std::min<size_t>({kPinnedThreads, hw, (chunks + 1) / 2}));
    std::atomic<int> failed{0};
    const cudaStreamCaptureMode mode = CaptureMode::current();              // a thread starts with one of its own
    parallel_for(threads, [&](size_t t) {
        const CaptureMode as_the_caller(mode);
        cudaEvent_t done[2] = {nullptr, nullptr};
        bool ok = cudaSetDevice(device) == cudaSuccess && cudaEventCreateWithFlags(&done[0], cudaEventDisableTiming) == cudaSuccess &&
                  cudaEventCreateWithFlags(&done[1], cudaEventDisableTiming) == cudaSuccess;
        auto request = [&](size_t c, int slot) {
            const size_t lo = c * per, cnt = std::min(per, n - lo);
            ok = ok && cudaMemcpyAsync(pinned.chunk(2 * t + slot), dev + lo * elem, cnt * elem, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
                 cudaEventRecord(done[slot], st) == cudaSuccess;
        };
        if (ok && t < chunks) request(t, 0);
        int slot = 0;
        for (size_t c = t; ok && c < chunks; c += threads, slot ^= 1) {
            if (c + threads < chunks) request(c + threads, slot ^ 1);
            ok = ok && cudaEventSynchronize(done[slot]) == cudaSuccess;
            const size_t lo = c * per, cnt = std::min(per, n - lo);
            if (ok) fn(pinned.chunk(2 * t + slot), static_cast<uint8_t *>(out) + lo * width[out_type], cnt, shift);
        }
        if (!ok) failed.store(1);
        for (cudaEvent_t e : done) if (e) cudaEventDestroy(e);
    }, threads);
    if (failed.load()) { cudaStreamSynchronize(st); return EOQ_ERR_CUDA; }      // nothing may still be on its way into the staging memory
    return EOQ_OK;
}

}  // namespace

extern "C" eoq_error_t eoq_b200_decode_blocked_as(const uint32_t *freq, uint32_t alphabet, uint32_t precision_bits, const uint8_t *data,
                                                  size_t data_len, const uint32_t *offsets, uint32_t num_blocks, uint32_t block_size,
                                                  uint32_t num_symbols, void *out, int out_type, int64_t shift, void *stream)
{
    if (num_symbols == 0) return EOQ_OK;
    if (!out) return EOQ_ERR_NULL_PTR;
    if (out_type < EOQ_B200_SYM_I8 || out_type > EOQ_B200_SYM_I64 || out_type == EOQ_B200_SYM_U32) return EOQ_ERR_UNSUPPORTED;
    V1Job job;
    eoq_error_t rc = blocked_job(freq, alphabet, precision_bits, data, data_len, offsets, num_blocks, block_size, num_symbols,
                                 alphabet <= 256 ? 1 : 2, job, have_device());
    if (rc != EOQ_OK) return rc;
    if (!have_device()) return EOQ_ERR_CUDA;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    V1Job *one = &job;
    DeviceArena arena;
    rc = decode_jobs(&one, 1, st, arena, false);
    if (rc == EOQ_OK && job.raw_offsets) rc = job_verdict(job, arena, st);      // a stream that is refused leaves `out` alone
    if (rc == EOQ_OK) rc = deliver(arena.base() + job.at_out, job.out_elem_bytes, num_symbols, out, out_type, shift, st);
    const cudaError_t e = cudaStreamSynchronize(st);                  // the arena is another call's from here on
    if (rc != EOQ_OK) return rc;
    CU_TRY(e);
    return EOQ_OK;
}

// -- symbols of a host array staged on the device, counted and encoded there (for the torch-facing front; not in the public header) --
//
// Used where the process has a context on the device already (encoding alone makes none), the array is long enough for the
// copies to be worth it (64 Ki symbols in blocks of 256, the whole call: 0.22 ms on the host's sixteen cores, 0.16 here), its blocks are short
// enough (eoq_b200_symbols_preferred) and the alphabet fits shared memory.  On a
// stream of its own: whatever else is under way on the device is not waited for, but where scratch is allocated or given back (a larger
// array than before, one that wants more than 256 MB: cudaMalloc and cudaFree wait for the device).  Nothing is accepted or refused here that
// the host encoder does not accept or refuse: what this one does not take, an array with symbols outside the alphabet among it,
// goes there, and so does an array with which any call to the device fails.
namespace {

constexpr size_t kStageSymbols = 1u << 16;

// "symbols_refused" in eoq_b200_tune: the step of a device encode that fails as if the device had nothing to give.
enum { kRefuseStage = 1, kRefuseCount, kRefuseScratch, kRefuseEncode, kRefuseFetch };
std::atomic<int> g_symbols_refused{0};
bool refused(int step) { return g_symbols_refused.load(std::memory_order_relaxed) == step; }

// A block is one chain, 0.073 us a symbol, while what the device saves with short chains grows as about n^(2/3): 0.03 ms x
// (n / 32 Ki)^(2/3).  Whole calls, device / host's sixteen cores, us, fifteen symbols: 64 Ki symbols in blocks of 512 199 / 221, 1024
// 235 / 220, in one 4820 / 390; 256 Ki in blocks of 1024 222 / 390, 4096 470 / 430; 1 Mi in blocks of 4096 546 / 789, 16384 1540 / 900, in one
// 75600 / 5240; 4 Mi in blocks of 4096 895 / 1650, 16384 2110 / 1740; 16 Mi in blocks of 16384 3280 / 4750, 65536 7090 / 6300.
bool chains_are_short(double n, double block) { const double b = std::min(n, block); return 16.0 * b * b * b <= n * n; }

bool context_is_active(int dev)
{
    typedef CUresult (*StateFn)(CUdevice, unsigned int *, int *);
    static StateFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuDevicePrimaryCtxGetState", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
        (void)cudaGetLastError();
        return reinterpret_cast<StateFn>(p);
    }();
    unsigned int flags = 0;
    int active = 0;
    return fn && fn(dev, &flags, &active) == CUDA_SUCCESS && active;
}

// Streams kept between calls, a few a device; the others are destroyed.
class SideStream {
  public:
    SideStream() = default;
    SideStream(const SideStream &) = delete;
    SideStream &operator=(const SideStream &) = delete;
    bool acquire(int dev)
    {
        dev_ = dev;
        {
            std::lock_guard<std::mutex> lock(cache().mu);
            auto &v = cache().free_list;
            for (size_t i = 0; i < v.size(); i++)
                if (v[i].first == dev) { st_ = v[i].second; v.erase(v.begin() + i); return true; }
        }
        if (cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking) == cudaSuccess) return true;
        st_ = nullptr;
        return false;
    }
    ~SideStream()
    {
        if (!st_) return;
        std::lock_guard<std::mutex> lock(cache().mu);
        if (cache().free_list.size() < 4) cache().free_list.emplace_back(dev_, st_);
        else cudaStreamDestroy(st_);
    }
    cudaStream_t get() const { return st_; }

  private:
    struct Cache { std::mutex mu; std::vector<std::pair<int, cudaStream_t>> free_list; };
    static Cache &cache() { static Cache *c = new Cache(); return *c; }      // never destroyed: no CUDA call after main
    cudaStream_t st_ = nullptr;
    int dev_ = 0;
};

struct OnDevice {
    int was = -1;
    explicit OnDevice(int dev) { if (cudaGetDevice(&was) != cudaSuccess || (was != dev && cudaSetDevice(dev) != cudaSuccess)) was = -1; else if (was == dev) was = -1; }
    ~OnDevice() { if (was >= 0) cudaSetDevice(was); }
};

}  // namespace

struct eoq_b200_symbols {
    SideStream stream;               // given back last
    DeviceArena sym, work;
    int dev = 0, wide = 0, shift = 0;
    bool moved = false, is_signed = false, clamp = false;        // the bytes are the caller's: value + shift, clamped or not, is the symbol
    uint32_t n = 0, alphabet = 0, nblocks = 0;
    size_t at_counts = 0, at_table = 0, at_offsets = 0, at_out = 0, bytes = 0;
    ~eoq_b200_symbols()
    {
        const CaptureMode beside;
        if (stream.get()) cudaStreamSynchronize(stream.get());      // the arenas are another call's from here on
        sym.release_beyond(256u << 20);                             // a process that encoded a large array once does not keep its scratch
        work.release_beyond(256u << 20);
        (void)cudaGetLastError();
    }
};

extern "C" void eoq_b200_symbols_free(eoq_b200_symbols *s) { delete s; }

extern "C" size_t eoq_b200_symbols_size(const eoq_b200_symbols *s) { return s ? s->n : 0; }

// Whether n symbols in blocks of `block` are encoded sooner on the device than on the host's cores.
extern "C" int eoq_b200_symbols_preferred(size_t n, uint64_t block) { return n >= kStageSymbols && chains_are_short((double)n, (double)block) ? 1 : 0; }

// The staged array, or null: the host encodes.
extern "C" eoq_b200_symbols *eoq_b200_symbols_stage(const void *symbols, int elem, size_t n, int64_t shift, int clamp, uint32_t alphabet)
try {
    if (!symbols || n < kStageSymbols || n > (1u << 28) || alphabet == 0 || alphabet > 4096u || elem < EOQ_B200_SYM_I8 || elem > EOQ_B200_SYM_I64) return nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || !context_is_active(dev)) { (void)cudaGetLastError(); return nullptr; }
    const CaptureMode beside;
    std::unique_ptr<eoq_b200_symbols> s(new eoq_b200_symbols());
    s->dev = dev; s->n = (uint32_t)n; s->alphabet = alphabet; s->wide = alphabet > 256u;
    const size_t width = s->wide ? 2 : 1;
    s->at_counts = (n * width + 255) & ~(size_t)255;
    s->at_table = s->at_counts + (((size_t)alphabet * 8 + 8 + 255) & ~(size_t)255);
    PinnedBlock pinned;
    if (refused(kRefuseStage) || !s->stream.acquire(dev) || s->sym.acquire(s->at_table + (size_t)alphabet * 16) != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
    cudaStream_t st = s->stream.get();
    uint8_t *to = s->sym.base();
    // Bytes that hold a symbol as it will be kept go up as they are, and the device moves and clamps them; other types are
    // narrowed on the way into the staging memory (a core reads some 1 G of them a second).
    const bool as_is = !s->wide && (elem == EOQ_B200_SYM_I8 || elem == EOQ_B200_SYM_U8) && shift > -(1 << 24) && shift < (1 << 24);
    cudaError_t e = cudaSuccess;
    if (as_is) {
        e = cudaMemcpyAsync(to, symbols, n, cudaMemcpyHostToDevice, st);
    } else if (!pinned.acquire()) {
        return nullptr;
    } else {
        const size_t bytes = n * width, hw = std::max(1u, std::thread::hardware_concurrency());
        const size_t threads = std::min<size_t>({kPinnedThreads / 2, hw, (bytes + kPinnedChunk - 1) / kPinnedChunk});
        e = upload_filled(pinned, to, bytes, st, threads, [&](size_t lo, size_t cnt, uint8_t *chunk) {
            return wire_narrow(symbols, elem, lo / width, cnt / width, shift, clamp != 0, alphabet, chunk);
        });
    }
    if (e != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
    if (as_is) { s->moved = true; s->is_signed = elem == EOQ_B200_SYM_I8; s->shift = (int)shift; s->clamp = clamp != 0; }
    return s.release();
} catch (const std::exception &) { return nullptr; }

// Counts of the symbols; EOQ_ERR_UNSUPPORTED where one is outside the alphabet (and not to be clamped).
extern "C" eoq_error_t eoq_b200_symbols_count(eoq_b200_symbols *s, uint64_t *counts)
try {
    const CaptureMode beside;
    OnDevice on(s->dev);
    cudaStream_t st = s->stream.get();
    unsigned long long *d = reinterpret_cast<unsigned long long *>(s->sym.base() + s->at_counts);
    if (refused(kRefuseCount)) return EOQ_ERR_CUDA;
    CU_TRY(cudaMemsetAsync(d, 0, (size_t)s->alphabet * 8 + 8, st));
    unsigned long long *outside = d + s->alphabet;
    if (s->moved && launch_wire_move(s->sym.base(), s->is_signed, s->shift, s->n, s->alphabet, outside, st) != 0) return EOQ_ERR_CUDA;
    s->moved = false;
    std::vector<uint64_t> got((size_t)s->alphabet + 1);
    if (launch_wire_count(s->sym.base(), s->wide, s->n, s->alphabet, d, st) != 0) return EOQ_ERR_CUDA;
    CU_TRY(cudaMemcpyAsync(got.data(), d, got.size() * 8, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    std::memcpy(counts, got.data(), (size_t)s->alphabet * 8);
    return got.back() && !s->clamp ? EOQ_ERR_UNSUPPORTED : EOQ_OK;
} catch (const std::exception &) { return EOQ_ERR_ALLOC; }

extern "C" eoq_error_t eoq_b200_symbols_encode(eoq_b200_symbols *s, const uint32_t *freq, uint32_t alphabet, uint32_t p, uint32_t block, size_t *bytes)
try {
    if (!s || !freq || !bytes) return EOQ_ERR_NULL_PTR;
    if (p < 1 || block == 0) return EOQ_ERR_INVALID_HEADER;
    if (p > 16 || alphabet != s->alphabet) return EOQ_ERR_UNSUPPORTED;
    std::vector<uint32_t> table;
    if (!wire_table(freq, alphabet, p, table)) return EOQ_ERR_INVALID_HEADER;
    const CaptureMode beside;
    OnDevice on(s->dev);
    cudaStream_t st = s->stream.get();
    WireEncodeArgs a = {};
    a.sym = s->sym.base(); a.n = s->n; a.alphabet = alphabet; a.p = p; a.block = std::min(block, s->n);
    a.nblocks = s->nblocks = (uint32_t)(((uint64_t)s->n + block - 1) / block);
    a.words = a.block / 2u + 1u;                       // two bytes a symbol at most
    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t scratch = (size_t)((a.nblocks + 31u) / 32u) * 128u * a.words, most = (size_t)s->n * 2 + (size_t)a.nblocks * 8;
    if (scratch > (2ull << 30)) return EOQ_ERR_UNSUPPORTED;         // few, long blocks: the host's
    const size_t at_record = up(scratch), at_sizes = up(at_record + (size_t)a.nblocks * 16);
    s->at_offsets = up(at_sizes + (size_t)a.nblocks * 4);
    const size_t at_total = up(s->at_offsets + (size_t)a.nblocks * 4);
    s->at_out = at_total + 256;
    if (refused(kRefuseScratch) || s->work.acquire(s->at_out + most) != cudaSuccess) { (void)cudaGetLastError(); return EOQ_ERR_UNSUPPORTED; }
    uint8_t *d = s->work.base();
    a.table = reinterpret_cast<const uint4 *>(s->sym.base() + s->at_table);
    a.scratch = reinterpret_cast<uint32_t *>(d); a.record = reinterpret_cast<uint4 *>(d + at_record); a.sizes = reinterpret_cast<uint32_t *>(d + at_sizes);
    unsigned long long *total = reinterpret_cast<unsigned long long *>(d + at_total), sum = 0;
    CU_TRY(cudaMemcpyAsync(s->sym.base() + s->at_table, table.data(), table.size() * 4, cudaMemcpyHostToDevice, st));
    if (refused(kRefuseEncode) || launch_wire_encode(a, s->wide, reinterpret_cast<uint32_t *>(d + s->at_offsets), total, d + s->at_out, st) != 0) return EOQ_ERR_CUDA;
    CU_TRY(cudaMemcpyAsync(&sum, total, 8, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    if (sum > 0xFFFFFFFFull) return EOQ_ERR_OVERFLOW;
    *bytes = s->bytes = (size_t)sum;
    return EOQ_OK;
} catch (const std::exception &) { return EOQ_ERR_ALLOC; }

// The encoded bytes (as many as eoq_b200_symbols_encode said) and the blocks' offsets.
extern "C" eoq_error_t eoq_b200_symbols_fetch(eoq_b200_symbols *s, uint8_t *data, uint32_t *offsets)
try {
    if (!s || !data || !offsets || !s->work.base()) return EOQ_ERR_NULL_PTR;
    if (refused(kRefuseFetch)) return EOQ_ERR_CUDA;
    const CaptureMode beside;
    OnDevice on(s->dev);
    cudaStream_t st = s->stream.get();
    const eoq_error_t rc = deliver(s->work.base() + s->at_out, 1, s->bytes, data, EOQ_B200_SYM_U8, 0, st);
    if (rc != EOQ_OK) return rc;
    CU_TRY(cudaMemcpyAsync(offsets, s->work.base() + s->at_offsets, (size_t)s->nblocks * 4, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    return EOQ_OK;
} catch (const std::exception &) { return EOQ_ERR_ALLOC; }

extern "C" eoq_error_t eoq_b200_encode_blocked(const uint32_t *freq, uint32_t alphabet, uint32_t precision_bits,
                                               const uint32_t *symbols, uint32_t num_symbols, uint32_t block_size,
                                               uint8_t *out, size_t *out_len, uint32_t *offsets)
{
    if (!out_len) return EOQ_ERR_NULL_PTR;
    if (num_symbols == 0) { *out_len = 0; return EOQ_OK; }
    if (!freq || !symbols || !out || !offsets) return EOQ_ERR_NULL_PTR;
    if (alphabet == 0 || block_size == 0 || precision_bits < 1 || precision_bits > 20) return EOQ_ERR_INVALID_HEADER;
    std::vector<uint32_t> cdf(alphabet + 1, 0);
    uint64_t sum = 0;
    for (uint32_t s = 0; s < alphabet; s++) { if (!freq[s]) return EOQ_ERR_INVALID_HEADER; sum += freq[s]; cdf[s + 1] = cdf[s] + freq[s]; }
    if (sum != (1ull << precision_bits)) return EOQ_ERR_INVALID_HEADER;
    for (uint32_t i = 0; i < num_symbols; i++) if (symbols[i] >= alphabet) return EOQ_ERR_CORRUPT_STREAM;
    if (precision_bits <= 16) {
        eoq_b200_wire_t *w = nullptr;
        size_t total = 0;
        eoq_error_t rc = eoq_b200_wire_encode(symbols, EOQ_B200_SYM_U32, num_symbols, 0, 0, freq, alphabet, precision_bits, block_size, &w, &total);
        if (rc != EOQ_OK) return rc;
        const bool fits = total <= *out_len;
        eoq_b200_wire_take(w, fits ? out : nullptr, fits ? offsets : nullptr);
        if (!fits) return EOQ_ERR_BUFFER_TOO_SMALL;
        *out_len = total;
        return EOQ_OK;
    }
    // states wider than 32 bits: one division per symbol
    const uint32_t nb = (uint32_t)(((uint64_t)num_symbols + block_size - 1) / block_size);
    // blocks are independent streams: ranges of blocks are encoded on the host's cores (one range, on the calling thread,
    // for small inputs), then laid out back to back in block order
    const size_t nranges = num_symbols < (1u << 18) ? 1 : std::min<size_t>(nb, 256);
    std::vector<std::vector<uint8_t>> bytes(nranges);
    std::vector<uint32_t> sizes(nb);
    auto encode_range = [&](size_t r) {
        const uint32_t lo = (uint32_t)((uint64_t)nb * r / nranges), hi = (uint32_t)((uint64_t)nb * (r + 1) / nranges);
        std::vector<uint8_t> blk;
        for (uint32_t b = lo; b < hi; b++) {
            const uint32_t first = b * block_size, n = std::min(block_size, num_symbols - first);
            encode_block_v1(freq, cdf.data(), precision_bits, symbols + first, n, blk);
            sizes[b] = (uint32_t)blk.size();
            bytes[r].insert(bytes[r].end(), blk.begin(), blk.end());
        }
    };
    if (nranges == 1) encode_range(0); else parallel_for(nranges, encode_range);
    size_t at = 0;
    for (size_t r = 0; r < nranges; r++) {
        const uint32_t lo = (uint32_t)((uint64_t)nb * r / nranges), hi = (uint32_t)((uint64_t)nb * (r + 1) / nranges);
        if (at + bytes[r].size() > *out_len) return EOQ_ERR_BUFFER_TOO_SMALL;
        size_t off = at;
        for (uint32_t b = lo; b < hi; b++) {
            if (off > 0xFFFFFFFFull) return EOQ_ERR_OVERFLOW;
            offsets[b] = (uint32_t)off;
            off += sizes[b];
        }
        if (!bytes[r].empty()) std::memcpy(out + at, bytes[r].data(), bytes[r].size());
        at += bytes[r].size();
    }
    *out_len = at;
    return EOQ_OK;
}

// -- resident weights ---------------------------------------------------------

struct eoq_b200_weight {
    int device = 0;
    uint32_t N = 0, K = 0, Npad = 0, G = 0, bits = 0, p = 0, group = 0, kind = 0, alphabet = 0;
    uint32_t ntiles = 0, nseg = 0, nrb = 0;
    uint32_t stage_bytes = 0, max_ncols = 0;          // geometry of the pair kernel's staging buffers (see GemvArgs)
    uint32_t head_bytes = 0;                          // TiledWeights::head_bytes
    // scales_t: transposed copy of the scales for the pair kernel (INT4 x 3 only); pair_partials: partial rows of the pair
    // kernel, every word 0xFFFFFFFF between launches
    size_t pair_partial_bytes = 0;
    DeviceBuf slab, stream;                           // everything but the stream in one allocation, the parts below point into it
    DeviceView table, tiles, scales, scales_t, centroids, counters, pair_partials;
    DeviceView xbuf, ybuf, biasbuf;                   // staging of the host-buffer calls: eight rows of fp32 each, one bias
    DeviceBuf partials;                               // the ring kernel's scratch
    DeviceBuf gemm_x, gemm_partials, gemm_counters;   // scratch of the tensor-core path, allocated by its first call
    uint32_t gemm_rows = 0;                           // activation rows per pass that scratch was sized for
    // The status word the kernels set when a bounded wait expires lives in pinned host memory that the device writes
    // directly (pinned allocations are device-addressable): a healthy launch never touches it, and reading it after a
    // stream synchronise needs no copy.
    uint32_t *status_host = nullptr, *status_dev = nullptr;
    uint32_t *status_word()
    {
        return status_dev;
    }
    ~eoq_b200_weight()
    {
        slab.release();       // waits for the device: no launch can write the word below any more
        StatusWords::give(status_host);
    }
    size_t stream_bytes = 0, scale_bytes = 0, partial_bytes = 0;
    std::mutex mu;   // one call at a time may use the scratch of a weight
    std::mutex scratch_mu;   // guards the late allocation of `partials`
};

namespace {

uint32_t public_kind(uint32_t family, uint32_t bits)
{
    if (family != EOQ_B200_KIND_INT4_ABSMAX) return family;
    return bits == 2 ? EOQ_B200_KIND_INT2_ABSMAX : bits == 3 ? EOQ_B200_KIND_INT3_ABSMAX : bits == 8 ? EOQ_B200_KIND_INT8_ABSMAX : EOQ_B200_KIND_INT4_ABSMAX;
}

eoq_error_t resolve_opts(const eoq_b200_weight_opts_t *o, uint32_t &bits, uint32_t &G, uint32_t &p, uint32_t &target, uint8_t &pad)
{
    if (!o) return EOQ_ERR_NULL_PTR;
    if (o->kind == EOQ_B200_KIND_INT4_ABSMAX) { bits = 4; G = o->symbols_per_step ? o->symbols_per_step : 3; pad = 7; }
    else if (o->kind == EOQ_B200_KIND_Q5_POLAR) { bits = 5; G = o->symbols_per_step ? o->symbols_per_step : 2; pad = 16; if (!o->centroids) return EOQ_ERR_NULL_PTR; }
    else if (o->kind == EOQ_B200_KIND_INT2_ABSMAX || o->kind == EOQ_B200_KIND_INT3_ABSMAX || o->kind == EOQ_B200_KIND_INT8_ABSMAX) {
        // the other widths the reference's packers know (core/weight_packing.py:35-51): one layout each
        bits = o->kind == EOQ_B200_KIND_INT2_ABSMAX ? 2 : o->kind == EOQ_B200_KIND_INT3_ABSMAX ? 3 : 8;
        const uint32_t g = bits == 8 ? 1 : 3;
        if (o->symbols_per_step && o->symbols_per_step != g) return EOQ_ERR_UNSUPPORTED;
        G = g; pad = (uint8_t)((1u << (bits - 1)) - 1u);
    }
    else return EOQ_ERR_UNSUPPORTED;
    if (G < 1 || G > (bits <= 4 ? 3u : bits == 8 ? 1u : 2u)) return EOQ_ERR_UNSUPPORTED;
    // INT4 x 3: 13 bits, a 32 KB table; 8-bit codes: 255 symbols want the finest table shared memory holds (at 12 bits the
    // rare symbols would all be rounded up to a frequency of 1 and the stream would be larger than the codes)
    p = o->precision_bits ? o->precision_bits : bits * G == 8 ? 14u : std::min(16u, std::max(12u, bits * G + 1));
    if (p > 14 || p < bits * G) return EOQ_ERR_UNSUPPORTED;        // table must fit shared memory beside x
    target = o->target_tiles;
    return EOQ_OK;
}

// `built` (optional): the stream already on the device, `built_bytes` long (tw.stream is then empty); it is taken over.
eoq_error_t upload_weight(const TiledWeights &tw, const uint16_t *scales, const float *centroids, eoq_b200_weight_t **out,
                          DeviceBuf *built = nullptr, size_t built_bytes = 0)
{
    std::unique_ptr<eoq_b200_weight> w(new eoq_b200_weight());
    CU_TRY(cudaGetDevice(&w->device));
    w->N = tw.N; w->K = tw.K; w->Npad = tw.Npad; w->G = tw.G; w->bits = tw.bits; w->p = tw.p; w->group = tw.group;
    w->kind = tw.kind; w->alphabet = tw.alphabet; w->ntiles = (uint32_t)tw.tiles.size(); w->nseg = tw.nseg; w->nrb = tw.nrb;
    w->head_bytes = tw.head_bytes;
    for (const TileDesc &d : tw.tiles) {
        w->stage_bytes = std::max(w->stage_bytes, ((d.len64 << 6) + 64u + 127u) & ~127u);
        w->max_ncols = std::max(w->max_ncols, d.ncols);
    }
    w->stream_bytes = built ? built_bytes : tw.stream.size();
    w->scale_bytes = (size_t)tw.N * (tw.K / tw.group) * 2;
    w->partial_bytes = tw.nseg > 1 ? (size_t)tw.nseg * tw.Npad * 8 * sizeof(float) : 0;
    // INT4 x 3 weights run through the pair kernel, which meets in a few partial rows; the ring kernel's scratch (one
    // row per column segment) is allocated by the first call that needs it (see ring_scratch)
    const bool pairs_layout = tw.kind == EOQ_B200_KIND_INT4_ABSMAX && tw.bits == 4 && tw.G == 3;
    // The pair kernel reuses a warp's two tile buffers after its column loop: the warp's sums (2 tiles x 3 rows x 4
    // activation rows x 32 lanes of fp32 = 3 KB) go into the first, its share of a cooperative meeting into the second.
    // Tiles shorter than that (32-column tiles, low-entropy weights) get buffers of that size all the same.
    if (pairs_layout) w->stage_bytes = std::max(w->stage_bytes, 3072u);
    // one allocation for all the small parts (ten of them, and their release, took 2 ms of a 7 ms load)
    w->pair_partial_bytes = pairs_layout ? (size_t)pair_partial_slots(tw.nrb, tw.nseg) * tw.Npad * 4 * sizeof(float) : 0;
    const uint32_t sg = tw.K / tw.group, triples = tw.Npad / 3;
    size_t used = 0;
    auto part = [&](size_t bytes) { const size_t at = used; used += (bytes + 255) & ~(size_t)255; return at; };
    const size_t at_table = part(tw.table.size() * 4), at_tiles = part(tw.tiles.size() * sizeof(TileDesc)), at_scales = part(w->scale_bytes),
                 at_scales_t = part(pairs_layout ? (size_t)sg * triples * 8 : 0), at_cent = part(32 * 4), at_counters = part((size_t)tw.nrb * 4),
                 at_partials = part(w->pair_partial_bytes), at_x = part((size_t)8 * tw.K * 4), at_y = part((size_t)8 * tw.N * 4),
                 at_bias = part((size_t)tw.N * 4);
    if (w->slab.alloc_pooled(used) != cudaSuccess || (!built && w->stream.alloc_pooled(tw.stream.size()) != cudaSuccess) ||
        (!pairs_layout && w->partials.alloc(w->partial_bytes) != cudaSuccess))
        return EOQ_ERR_ALLOC;
    uint8_t *base = w->slab.as<uint8_t>();
    w->table.p = base + at_table; w->tiles.p = base + at_tiles; w->scales.p = base + at_scales; w->counters.p = base + at_counters;
    w->xbuf.p = base + at_x; w->ybuf.p = base + at_y; w->biasbuf.p = base + at_bias;
    if (built) w->stream.take(*built);
    else CU_TRY(cudaMemcpyAsync(w->stream.p, tw.stream.data(), tw.stream.size(), cudaMemcpyHostToDevice, nullptr));
    if (centroids) {
        w->centroids.p = base + at_cent;
        CU_TRY(cudaMemcpyAsync(w->centroids.p, centroids, 32 * 4, cudaMemcpyHostToDevice, nullptr));
    }
    CU_TRY(cudaMemcpyAsync(w->table.p, tw.table.data(), tw.table.size() * 4, cudaMemcpyHostToDevice, nullptr));
    CU_TRY(cudaMemcpyAsync(w->tiles.p, tw.tiles.data(), tw.tiles.size() * sizeof(TileDesc), cudaMemcpyHostToDevice, nullptr));
    CU_TRY(cudaMemcpyAsync(w->scales.p, scales, w->scale_bytes, cudaMemcpyHostToDevice, nullptr));
    if (pairs_layout) {
        w->scales_t.p = base + at_scales_t;
        w->pair_partials.p = base + at_partials;
        CU_TRY(cudaMemsetAsync(w->pair_partials.p, 0xFF, w->pair_partial_bytes, nullptr));
        if (launch_transpose_scales(w->scales.as<uint16_t>(), w->scales_t.as<uint2>(), tw.N, sg, triples, nullptr) != 0) return EOQ_ERR_CUDA;
    }
    CU_TRY(cudaMemsetAsync(w->counters.p, 0, (size_t)tw.nrb * 4, nullptr));
    CU_TRY(StatusWords::take(&w->status_host, &w->status_dev));
    CU_TRY(cudaStreamSynchronize(nullptr));            // what the weight holds is there for every stream
    *out = w.release();
    return EOQ_OK;
}

}  // namespace

struct eoq_b200_tiles { TiledWeights tw; };
extern "C" eoq_error_t eoq_b200_tiles_build(const uint8_t *symbols, const eoq_b200_weight_opts_t *opts, eoq_b200_tiles_t **out);
extern "C" void eoq_b200_tiles_free(eoq_b200_tiles_t *t);

// How many tiles a weight is cut into when the caller does not say.
static uint32_t default_target_tiles(const eoq_b200_weight_opts_t *opts, uint32_t bits, uint32_t G)
{
    const int sms = have_device() ? device_sm_count() : 0;
    const uint32_t warps = (uint32_t)(sms > 0 ? sms : 148) * 16;      // one wave of 16-warp CTAs
    uint32_t target = warps;
    if (opts->kind == EOQ_B200_KIND_INT4_ABSMAX && bits == 4 && G == 3) {
        // The pair kernel gives every warp two vertically adjacent tiles and stages them whole in shared memory,
        // which holds tiles of up to 7 x 16 columns: take the fewest waves of pairs whose column segments are
        // that narrow, and as many segments as fill those waves.
        const uint32_t nrb = (opts->rows + 32 * G - 1) / (32 * G), nrbp = (nrb + 1) / 2;
        const uint32_t units = opts->cols / 16, need = (units + 6) / 7;
        uint32_t nseg = 1;
        for (uint32_t waves = 1; waves <= 64; waves++) {
            nseg = std::max(1u, waves * warps / nrbp);
            if (nseg >= need) break;
        }
        target = nseg * nrb;
    }
    // by default no tile is narrower than 64 columns (an explicit target_tiles may go down to 32) ...
    const uint32_t nrb = (opts->rows + 32 * G - 1) / (32 * G);
    target = std::min<uint32_t>(target, std::max(1u, opts->cols / 64) * nrb);
    // ... except small matrices in the pair layout (row shards of a layer, narrow projections): while tile pairs of 32
    // columns still fit one wave they are taken, twice as many warps share the columns and a launch is 6-16 % shorter
    // (1376 x 4096: 9.8 -> 9.2 us, 512 x 4096: 11.0 -> 9.2 us) for 4-5 % more bytes
    if (opts->kind == EOQ_B200_KIND_INT4_ABSMAX && bits == 4 && G == 3 && opts->cols % 32u == 0 && opts->cols >= 64u &&
        (uint64_t)((nrb + 1) / 2) * (opts->cols / 32u) <= warps)
        target = (opts->cols / 32u) * nrb;
    return target;
}

// The tiled layout built on the device from symbols that are already there (one per byte, row-major [rows, cols], in
// memory this library allocated: 256-byte aligned): joint-symbol counts by a kernel, frequencies and table on the host
// (a few thousand numbers), every tile encoded by one warp, the stream laid out on the host from the tiles' sizes and
// filled by a scatter kernel.  Byte-identical to build_tiled.  EOQ_ERR_UNSUPPORTED (nothing launched) when a tile has
// 65536 columns or more or the scratch would pass 4 GB: the caller then encodes on the host.
static eoq_error_t build_tiled_device(const uint8_t *d_sym, const eoq_b200_weight_opts_t *opts, TiledWeights &tw, DeviceBuf &stream,
                                      size_t &stream_bytes, cudaStream_t st)
{
    uint32_t bits, G, p, target; uint8_t pad;
    eoq_error_t rc = resolve_opts(opts, bits, G, p, target, pad);
    if (rc != EOQ_OK) return rc;
    if (opts->rows == 0 || opts->cols == 0 || opts->group == 0) return EOQ_ERR_INVALID_HEADER;
    if (target == 0) target = default_target_tiles(opts, bits, G);
    const uint32_t family = opts->kind == EOQ_B200_KIND_Q5_POLAR ? EOQ_B200_KIND_Q5_POLAR : EOQ_B200_KIND_INT4_ABSMAX;
    rc = tiled_geometry(opts->rows, opts->cols, bits, G, p, opts->group, family, target, tw);
    if (rc != EOQ_OK) return rc;
    const size_t ntiles = tw.tiles.size();
    uint32_t max_ncols = 0;
    for (const TileDesc &d : tw.tiles) max_ncols = std::max(max_ncols, d.ncols);
    const size_t scratch_bytes = ntiles * (size_t)max_ncols * 128u;
    if (max_ncols >= 65536u || scratch_bytes > (4ull << 30)) return EOQ_ERR_UNSUPPORTED;

    auto up = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t at_counts = 0, at_fc = up(at_counts + (size_t)tw.alphabet * 8), at_tiles = up(at_fc + (size_t)tw.alphabet * 8),
                 at_state = up(at_tiles + ntiles * sizeof(TileDesc)), at_count = up(at_state + ntiles * 128), at_info = up(at_count + ntiles * 128),
                 at_scratch = up(at_info + ntiles * 8), total_tmp = at_scratch + scratch_bytes;
    DeviceArena tmp;
    if (tmp.acquire(total_tmp) != cudaSuccess) return EOQ_ERR_ALLOC;
    uint8_t *d = tmp.base();

    CU_TRY(cudaMemsetAsync(d + at_counts, 0, (size_t)tw.alphabet * 8, st));
    if (launch_tile_hist(d_sym, tw.N, tw.K, tw.Npad, G, bits, reinterpret_cast<unsigned long long *>(d + at_counts), st) != 0) return EOQ_ERR_CUDA;
    std::vector<uint64_t> count(tw.alphabet);
    CU_TRY(cudaMemcpyAsync(count.data(), d + at_counts, (size_t)tw.alphabet * 8, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    std::vector<uint32_t> freq, cum;
    rc = tiled_table(count, tw, freq, cum);
    if (rc != EOQ_OK) return rc;
    std::vector<uint32_t> fc((size_t)tw.alphabet * 2);
    for (uint32_t s = 0; s < tw.alphabet; s++) { fc[2 * s] = freq[s] ? freq[s] : 1u; fc[2 * s + 1] = cum[s]; }   // absent symbols never occur
    CU_TRY(cudaMemcpyAsync(d + at_fc, fc.data(), fc.size() * 4, cudaMemcpyHostToDevice, st));
    CU_TRY(cudaMemcpyAsync(d + at_tiles, tw.tiles.data(), ntiles * sizeof(TileDesc), cudaMemcpyHostToDevice, st));
    TileEncodeArgs ea = {};
    ea.sym = d_sym; ea.tiles = reinterpret_cast<const TileDesc *>(d + at_tiles); ea.freq_cum = reinterpret_cast<const uint2 *>(d + at_fc);
    ea.scratch = reinterpret_cast<uint32_t *>(d + at_scratch); ea.state = reinterpret_cast<uint32_t *>(d + at_state);
    ea.count = reinterpret_cast<uint32_t *>(d + at_count); ea.info = reinterpret_cast<uint2 *>(d + at_info);
    ea.N = tw.N; ea.K = tw.K; ea.G = G; ea.bits = bits; ea.p = p; ea.ntiles = (uint32_t)ntiles; ea.max_ncols = max_ncols;
    if (launch_tile_encode(ea, st) != 0) return EOQ_ERR_CUDA;
    std::vector<uint32_t> info(ntiles * 2);
    CU_TRY(cudaMemcpyAsync(info.data(), d + at_info, ntiles * 8, cudaMemcpyDeviceToHost, st));
    CU_TRY(cudaStreamSynchronize(st));
    for (size_t t = 0; t < ntiles; t++) {
        const uint32_t rows = info[2 * t], drift = info[2 * t + 1];
        tw.tiles[t].len64 = (128u + rows * 64u) >> 6;
        if (drift > kMaxRingDrift) tw.tiles[t].seg |= kTileDirectFlag;
        tw.max_drift = std::max(tw.max_drift, drift);
    }
    rc = tiled_layout(tw, stream_bytes);
    if (rc != EOQ_OK) return rc;
    if (stream.alloc_pooled(stream_bytes) != cudaSuccess) return EOQ_ERR_ALLOC;
    CU_TRY(cudaMemsetAsync(stream.p, 0, stream_bytes, st));
    CU_TRY(cudaMemcpyAsync(d + at_tiles, tw.tiles.data(), ntiles * sizeof(TileDesc), cudaMemcpyHostToDevice, st));
    TileScatterArgs sa = {};
    sa.tiles = reinterpret_cast<const TileDesc *>(d + at_tiles); sa.scratch = ea.scratch; sa.state = ea.state; sa.count = ea.count;
    sa.stream = stream.as<uint8_t>(); sa.head_bytes = tw.head_bytes; sa.ntiles = (uint32_t)ntiles; sa.max_ncols = max_ncols;
    if (launch_tile_scatter(sa, st) != 0) return EOQ_ERR_CUDA;
    CU_TRY(cudaStreamSynchronize(st));
    return EOQ_OK;
}

// A weight from symbols in device memory (this library's own allocation).  Falls back to the host encoder, through a
// copy of the symbols, where the device encoder declines.
static eoq_error_t weight_from_device_symbols(const uint8_t *d_sym, const uint16_t *scales_fp16, const eoq_b200_weight_opts_t *opts,
                                              eoq_b200_weight_t **out)
{
    TiledWeights tw;
    DeviceBuf stream;
    size_t stream_bytes = 0;
    eoq_error_t rc = build_tiled_device(d_sym, opts, tw, stream, stream_bytes, nullptr);
    if (rc == EOQ_ERR_UNSUPPORTED && tw.N != 0) {
        std::vector<uint8_t> host((size_t)opts->rows * opts->cols);
        CU_TRY(cudaMemcpy(host.data(), d_sym, host.size(), cudaMemcpyDeviceToHost));
        eoq_b200_tiles_t *t = nullptr;
        rc = eoq_b200_tiles_build(host.data(), opts, &t);
        if (rc != EOQ_OK) return rc;
        rc = upload_weight(t->tw, scales_fp16, opts->kind == EOQ_B200_KIND_Q5_POLAR ? opts->centroids : nullptr, out);
        eoq_b200_tiles_free(t);
        return rc;
    }
    if (rc != EOQ_OK) return rc;
    return upload_weight(tw, scales_fp16, opts->kind == EOQ_B200_KIND_Q5_POLAR ? opts->centroids : nullptr, out, &stream, stream_bytes);
}


extern "C" eoq_error_t eoq_b200_tiles_build(const uint8_t *symbols, const eoq_b200_weight_opts_t *opts, eoq_b200_tiles_t **out)
{
    if (!symbols || !opts || !out) return EOQ_ERR_NULL_PTR;
    *out = nullptr;
    uint32_t bits, G, p, target; uint8_t pad;
    eoq_error_t rc = resolve_opts(opts, bits, G, p, target, pad);
    if (rc != EOQ_OK) return rc;
    if (opts->rows == 0 || opts->cols == 0 || opts->group == 0) return EOQ_ERR_INVALID_HEADER;
    if (target == 0) target = default_target_tiles(opts, bits, G);
    std::unique_ptr<eoq_b200_tiles> t(new eoq_b200_tiles());
    // inside the library the integer widths are one family (the kernels are templated on the field width)
    const uint32_t family = opts->kind == EOQ_B200_KIND_Q5_POLAR ? EOQ_B200_KIND_Q5_POLAR : EOQ_B200_KIND_INT4_ABSMAX;
    rc = build_tiled(symbols, opts->rows, opts->cols, bits, G, p, opts->group, family, target, pad, t->tw);
    if (rc != EOQ_OK) return rc;
    *out = t.release();
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_tiles_view(const eoq_b200_tiles_t *t, eoq_b200_tiles_view_t *v)
{
    if (!t || !v) return EOQ_ERR_NULL_PTR;
    const TiledWeights &tw = t->tw;
    v->rows = tw.N; v->cols = tw.K; v->padded_rows = tw.Npad; v->group = tw.group; v->kind = public_kind(tw.kind, tw.bits); v->bits = tw.bits;
    v->symbols_per_step = tw.G; v->precision_bits = tw.p;
    v->num_tiles = (uint32_t)tw.tiles.size(); v->num_col_segments = tw.nseg;
    v->table = tw.table.data();
    static_assert(sizeof(eoq_b200_tile_desc_t) == sizeof(TileDesc), "tile descriptor layout");
    v->tiles = reinterpret_cast<const eoq_b200_tile_desc_t *>(tw.tiles.data());
    v->stream = tw.stream.data();
    v->stream_bytes = tw.stream.size();
    v->max_lane_drift = tw.max_drift;
    v->head_bytes = tw.head_bytes;
    return EOQ_OK;
}

extern "C" void eoq_b200_tiles_free(eoq_b200_tiles_t *t) { delete t; }

extern "C" eoq_error_t eoq_b200_weight_from_tiles(const eoq_b200_tiles_t *t, const uint16_t *scales_fp16, const float *centroids,
                                                  eoq_b200_weight_t **out)
{
    if (!t || !scales_fp16 || !out) return EOQ_ERR_NULL_PTR;
    *out = nullptr;
    if (t->tw.kind == EOQ_B200_KIND_Q5_POLAR && !centroids) return EOQ_ERR_NULL_PTR;
    if (!have_device()) return EOQ_ERR_CUDA;
    return upload_weight(t->tw, scales_fp16, t->tw.kind == EOQ_B200_KIND_Q5_POLAR ? centroids : nullptr, out);
}

extern "C" eoq_error_t eoq_b200_weight_from_symbols(const uint8_t *symbols, const uint16_t *scales_fp16,
                                                    const eoq_b200_weight_opts_t *opts, eoq_b200_weight_t **out)
{
    if (!symbols || !scales_fp16 || !opts || !out) return EOQ_ERR_NULL_PTR;
    *out = nullptr;
    if (!have_device()) {
        uint32_t bits, G, p, target; uint8_t pad;
        eoq_error_t rc = resolve_opts(opts, bits, G, p, target, pad);
        return rc != EOQ_OK ? rc : EOQ_ERR_CUDA;
    }
    // the symbols go to the device and the tiles are encoded there (the host encoder, which the device encoder matches
    // byte for byte, stays behind eoq_b200_tiles_build for callers without a device at hand)
    if (opts->rows == 0 || opts->cols == 0) return EOQ_ERR_INVALID_HEADER;
    const size_t n = (size_t)opts->rows * opts->cols;
    DeviceArena sym;
    if (sym.acquire(n) != cudaSuccess) return EOQ_ERR_ALLOC;
    CU_TRY(cudaMemcpy(sym.base(), symbols, n, cudaMemcpyHostToDevice));
    return weight_from_device_symbols(sym.base(), scales_fp16, opts, out);
}

extern "C" eoq_error_t eoq_b200_weight_from_device_symbols(const uint8_t *d_symbols, const uint16_t *scales_fp16,
                                                           const eoq_b200_weight_opts_t *opts, eoq_b200_weight_t **out)
{
    if (!d_symbols || !scales_fp16 || !opts || !out) return EOQ_ERR_NULL_PTR;
    *out = nullptr;
    if (!have_device()) return EOQ_ERR_CUDA;
    if (opts->rows == 0 || opts->cols == 0) return EOQ_ERR_INVALID_HEADER;
    if ((reinterpret_cast<uintptr_t>(d_symbols) & 3u) == 0) return weight_from_device_symbols(d_symbols, scales_fp16, opts, out);
    // the counting kernel reads four symbols at a time: an odd base address goes through an aligned copy
    const size_t n = (size_t)opts->rows * opts->cols;
    DeviceArena sym;
    if (sym.acquire(n) != cudaSuccess) return EOQ_ERR_ALLOC;
    CU_TRY(cudaMemcpy(sym.base(), d_symbols, n, cudaMemcpyDeviceToDevice));
    return weight_from_device_symbols(sym.base(), scales_fp16, opts, out);
}

extern "C" eoq_error_t eoq_b200_weight_from_rans(const uint8_t *c, size_t size, const uint16_t *scales_fp16,
                                                 const eoq_b200_weight_opts_t *opts, eoq_b200_weight_t **out)
{
    if (!c || !scales_fp16 || !opts || !out) return EOQ_ERR_NULL_PTR;
    *out = nullptr;
    // `RANS` container: magic, then 7 x u32 (version, num_symbols, block_size, num_blocks, alphabet,
    // precision_bits, data_size), u32 freq[alphabet], u32 offsets[num_blocks], data  (core/rans_blocked.py:176-214)
    if (size < 32 || std::memcmp(c, "RANS", 4) != 0) return EOQ_ERR_INVALID_HEADER;
    uint32_t h[7];
    std::memcpy(h, c + 4, 28);
    if (h[0] != 1) return EOQ_ERR_INVALID_HEADER;
    const uint32_t n = h[1], bs = h[2], nb = h[3], a = h[4], p = h[5], dsz = h[6];
    if ((uint64_t)32 + (uint64_t)a * 4 + (uint64_t)nb * 4 + dsz > size) return EOQ_ERR_CORRUPT_STREAM;
    if ((uint64_t)opts->rows * opts->cols != n) return EOQ_ERR_INVALID_HEADER;
    if (a == 0 || a > 256) return EOQ_ERR_UNSUPPORTED;
    std::vector<uint32_t> raw(a), freq, cdf;
    std::memcpy(raw.data(), c + 32, (size_t)a * 4);
    eoq_error_t rc = normalize_reference(raw.data(), a, p, freq, cdf);
    if (rc != EOQ_OK) return rc;
    if (!have_device()) return EOQ_ERR_CUDA;
    // decoded into device memory and encoded into tiles there: the symbols never visit the host
    DeviceArena sym;
    if (sym.acquire(n) != cudaSuccess) return EOQ_ERR_ALLOC;
    if (n) {
        V1Job job;
        const uint8_t *offsets = c + 32 + (size_t)a * 4;             // of any alignment: read on the host only from a copy
        std::vector<uint32_t> aligned(checks_on_device(nb) ? 0 : nb);
        if (!aligned.empty()) std::memcpy(aligned.data(), offsets, aligned.size() * 4);
        rc = blocked_job(freq.data(), a, p, offsets + (size_t)nb * 4, dsz, aligned.empty() ? reinterpret_cast<const uint32_t *>(offsets) : aligned.data(), nb, bs, n, 1,
                         job, true);
        if (rc != EOQ_OK) return rc;
        job.dev_out = sym.base();
        V1Job *one = &job;
        DeviceArena arena;
        rc = decode_jobs(&one, 1, nullptr, arena);
        if (rc == EOQ_OK && job.raw_offsets) rc = job_verdict(job, arena, nullptr);
        const cudaError_t e = cudaStreamSynchronize(nullptr);
        if (rc != EOQ_OK) return rc;
        CU_TRY(e);
    }
    return weight_from_device_symbols(sym.base(), scales_fp16, opts, out);
}

extern "C" void eoq_b200_weight_destroy(eoq_b200_weight_t *w) { delete w; }

extern "C" eoq_error_t eoq_b200_weight_info(const eoq_b200_weight_t *w, eoq_b200_weight_info_t *info)
{
    if (!w || !info) return EOQ_ERR_NULL_PTR;
    info->rows = w->N; info->cols = w->K; info->padded_rows = w->Npad; info->group = w->group; info->kind = public_kind(w->kind, w->bits);
    info->symbols_per_step = w->G; info->precision_bits = w->p; info->alphabet = w->alphabet;
    info->num_tiles = w->ntiles; info->num_col_segments = w->nseg;
    info->stream_bytes = w->stream_bytes;
    info->table_bytes = (uint64_t)4 << w->p;
    info->scale_bytes = w->scale_bytes;
    info->desc_bytes = (uint64_t)w->ntiles * sizeof(TileDesc);
    info->scratch_bytes = (w->partials.p ? w->partial_bytes : 0) + w->pair_partial_bytes + (uint64_t)w->nrb * 4;
    info->bits_per_weight = (double)w->stream_bytes * 8.0 / ((double)w->N * w->K);
    return EOQ_OK;
}

// The arguments every fused GEMV launch shares (inputs, outputs and scratch are the caller's to add).
static void weight_gemv_args(eoq_b200_weight_t *w, GemvArgs &a)
{
    a.table = w->table.as<uint32_t>(); a.tiles = w->tiles.as<TileDesc>(); a.stream = w->stream.as<uint8_t>();
    a.scales = w->scales.as<uint16_t>(); a.centroids = w->centroids.as<float>();
    a.status = w->status_word();
    a.N = w->N; a.K = w->K; a.Npad = w->Npad; a.group = w->group; a.p = w->p; a.ntiles = w->ntiles; a.nseg = w->nseg;
    a.nrb = w->nrb; a.stage_bytes = w->stage_bytes; a.max_ncols = w->max_ncols; a.head_bytes = w->head_bytes;
    a.scales_t = w->scales_t.as<uint2>();
}

// A weight lives on the device it was uploaded to; launching its kernels with another device current would hand
// that device pointers it cannot reach.  Refused on the host, before anything is launched.
static eoq_error_t check_device(const eoq_b200_weight_t *w, const char *where)
{
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return EOQ_ERR_CUDA;
    if (dev != w->device) {
        std::fprintf(stderr, "%s: the weight lives on device %d but device %d is current\n", where, w->device, dev);
        return EOQ_ERR_UNSUPPORTED;
    }
    return EOQ_OK;
}

// Scratch of the one-tile-per-warp GEMV kernel: one partial row per column segment.  Weights laid out for the pair
// kernel get it on the first call that falls back to the other kernel (an allocation: not inside stream capture).
static eoq_error_t ring_scratch(eoq_b200_weight_t *w)
{
    std::lock_guard<std::mutex> lock(w->scratch_mu);
    if (w->partials.p || w->partial_bytes == 0) return EOQ_OK;
    return w->partials.alloc(w->partial_bytes) == cudaSuccess ? EOQ_OK : EOQ_ERR_ALLOC;
}

extern "C" eoq_error_t eoq_b200_gemv(eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch, void *y, int y_dtype,
                                     const float *bias, void *stream)
{
    if (!w || !x || !y) return EOQ_ERR_NULL_PTR;
    if (batch == 0) return EOQ_OK;
    if (batch > 8) return EOQ_ERR_UNSUPPORTED;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    eoq_error_t drc = check_device(w, "eoq_b200_gemv");
    if (drc != EOQ_OK) return drc;
    GemvArgs a = {};
    weight_gemv_args(w, a);
    a.x = x; a.y = y; a.bias = bias; a.counters = w->counters.as<uint32_t>(); a.batch = batch;
    a.pair_partials = w->pair_partials.as<float>();
    a.x_dtype = x_dtype; a.y_dtype = y_dtype;
    if (!gemv_takes_pairs(a, w->G, w->bits, w->kind)) {
        const uint32_t bt = batch <= 1 ? 1 : batch <= 2 ? 2 : batch <= 4 ? 4 : 8;
        if (gemv_smem_bytes(w->K, w->p, bt, w->kind) > 227 * 1024) {
            // x for this many rows does not fit shared memory beside the table: run the rows in two halves
            if (bt == 1) return EOQ_ERR_UNSUPPORTED;
            static const size_t esz[3] = {2, 2, 4};
            const uint32_t half = bt / 2, first = std::min(batch, half);
            eoq_error_t rc = eoq_b200_gemv(w, x, x_dtype, first, y, y_dtype, bias, stream);
            if (rc != EOQ_OK || batch <= half) return rc;
            return eoq_b200_gemv(w, static_cast<const uint8_t *>(x) + (size_t)first * w->K * esz[x_dtype], x_dtype, batch - first,
                                 static_cast<uint8_t *>(y) + (size_t)first * w->N * esz[y_dtype], y_dtype, bias, stream);
        }
        eoq_error_t rc = ring_scratch(w);
        if (rc != EOQ_OK) return rc;
        a.partials = w->partials.as<float>();
    }
    int e = launch_gemv(a, w->G, w->bits, w->kind, stream);
    if (e != 0) { std::fprintf(stderr, "eoq_b200_gemv: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_gemm(eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t m, void *y, int y_dtype,
                                     const float *bias, void *stream)
{
    if (!w || !x || !y) return EOQ_ERR_NULL_PTR;
    if (m == 0) return EOQ_OK;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    // the tensor-core path is built for the default INT4 layout: 3 weights per step, 96-row tiles
    if (w->kind != EOQ_B200_KIND_INT4_ABSMAX || w->G != 3 || w->bits != 4 || w->Npad != w->nrb * 96u || (w->K & 15u)) return EOQ_ERR_UNSUPPORTED;
    if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15u) != 0) return EOQ_ERR_UNSUPPORTED;
    eoq_error_t drc = check_device(w, "eoq_b200_gemm");
    if (drc != EOQ_OK) return drc;
    static const size_t esz[3] = {2, 2, 4};
    const uint32_t per_pass = std::min(m, kGemmRowsPerPass);
    {
        std::lock_guard<std::mutex> lock(w->mu);
        if (!w->gemm_x.p || w->gemm_rows < per_pass) {
            // fp16 copy of one pass of fp32 or bf16 activation rows, one fp32 partial tile pair per CTA and 128-row token tile, one
            // arrival counter per row block.  Sized by the rows of a pass; a later call with more rows allocates again (outside
            // stream capture), after everything queued on the old scratch has finished.
            if (w->gemm_x.p) {
                CU_TRY(cudaDeviceSynchronize());
                cudaFree(w->gemm_x.p); w->gemm_x.p = nullptr;
                cudaFree(w->gemm_partials.p); w->gemm_partials.p = nullptr;
                cudaFree(w->gemm_counters.p); w->gemm_counters.p = nullptr;
            }
            const uint32_t rows = per_pass <= 128 ? 128 : kGemmRowsPerPass;
            CU_TRY(w->gemm_x.alloc((size_t)rows * w->K * 2));
            CU_TRY(w->gemm_partials.alloc(gemm_partial_bytes(gemm_grid(w->nrb, w->nseg), rows)));
            CU_TRY(w->gemm_counters.alloc((size_t)w->nrb * 4));
            CU_TRY(cudaMemset(w->gemm_counters.p, 0, (size_t)w->nrb * 4));
            w->gemm_rows = rows;
        }
    }
    for (uint32_t m0 = 0; m0 < m; m0 += kGemmRowsPerPass) {     // up to 512 activation rows share one pass over the compressed weight
        const uint32_t mb = std::min(kGemmRowsPerPass, m - m0);
        int e = launch_gemm_tc(w->table.as<uint32_t>(), w->tiles.as<TileDesc>(), w->stream.as<uint8_t>(), w->scales_t.as<uint2>(),
                               static_cast<const uint8_t *>(x) + (size_t)m0 * w->K * esz[x_dtype], w->gemm_x.p,
                               w->gemm_partials.as<float>(), w->gemm_counters.as<uint32_t>(),
                               static_cast<uint8_t *>(y) + (size_t)m0 * w->N * esz[y_dtype], bias, w->status_word(),
                               w->N, w->K, w->group, w->p, w->nseg, w->nrb, w->head_bytes, mb, x_dtype, y_dtype, stream);
        if (e != 0) { std::fprintf(stderr, "eoq_b200_gemm: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    }
    return EOQ_OK;
}

// =========================================================================
// Row-sharded GEMV with the all-gather fused into the kernel (peer stores over NVLink)
// =========================================================================
//
// Each rank owns one device allocation, opened by every other rank through CUDA IPC:
//   [slots x slot_bytes of output][slots x receive buffer of 8-byte words][slots epochs][slots done-counters]
// A gather sends into one slot of every peer's receive buffer; consecutive gathers must use different slots (a
// fast rank may already be sending the next gather while a slow one still unpacks the previous one).
struct eoq_b200_gather {
    uint32_t world = 0, rank = 0, slots = 0;
    size_t slot_bytes = 0, slot_elems = 0, total = 0;
    int device = 0;
    uint8_t *base[kMaxPeers] = {};      // base[rank] is the local allocation
    bool opened[kMaxPeers] = {};
    DeviceBuf status;
    long long limit_ticks = 1ll << 31;  // how long a kernel waits for the peers' words (about a second at 2 GHz)
    size_t ll_off(uint32_t slot) const { return (size_t)slots * slot_bytes + (size_t)slot * slot_elems * 8; }
    size_t epoch_off(uint32_t slot) const { return ll_off(slots) + (size_t)slot * 4; }
    size_t done_off(uint32_t slot) const { return epoch_off(slots) + (size_t)slot * 4; }
};

extern "C" eoq_error_t eoq_b200_gather_create(uint32_t world, uint32_t rank, uint32_t slots, size_t slot_bytes,
                                              eoq_b200_gather_t **out, void *ipc_handle_out)
{
    if (!out || !ipc_handle_out) return EOQ_ERR_NULL_PTR;
    if (world < 2 || world > kMaxPeers || rank >= world || slots < 2 || slots > 16 || slot_bytes == 0) return EOQ_ERR_UNSUPPORTED;
    static_assert(sizeof(cudaIpcMemHandle_t) == EOQ_B200_IPC_HANDLE_BYTES, "handle size");
    std::unique_ptr<eoq_b200_gather> g(new eoq_b200_gather());
    g->world = world; g->rank = rank; g->slots = slots;
    g->slot_bytes = (slot_bytes + 255) & ~(size_t)255;
    g->slot_elems = g->slot_bytes / 2;                      // the narrowest output element is 2 bytes
    g->total = g->done_off(slots);
    CU_TRY(cudaGetDevice(&g->device));
    void *p = nullptr;
    CU_TRY(cudaMalloc(&p, g->total));
    g->base[rank] = static_cast<uint8_t *>(p);
    g->opened[rank] = false;
    CU_TRY(cudaMemset(p, 0, g->total));
    CU_TRY(g->status.alloc(4));
    CU_TRY(cudaMemset(g->status.p, 0, 4));
    CU_TRY(cudaIpcGetMemHandle(reinterpret_cast<cudaIpcMemHandle_t *>(ipc_handle_out), p));
    CU_TRY(cudaDeviceSynchronize());
    *out = g.release();
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_gather_connect(eoq_b200_gather_t *g, const void *all_handles)
{
    if (!g || !all_handles) return EOQ_ERR_NULL_PTR;
    const cudaIpcMemHandle_t *h = reinterpret_cast<const cudaIpcMemHandle_t *>(all_handles);
    for (uint32_t p = 0; p < g->world; p++) {
        if (p == g->rank || g->base[p]) continue;
        void *ptr = nullptr;
        CU_TRY(cudaIpcOpenMemHandle(&ptr, h[p], cudaIpcMemLazyEnablePeerAccess));
        g->base[p] = static_cast<uint8_t *>(ptr);
        g->opened[p] = true;
    }
    return EOQ_OK;
}

extern "C" void eoq_b200_gather_destroy(eoq_b200_gather_t *g)
{
    if (!g) return;
    for (uint32_t p = 0; p < g->world; p++)
        if (g->opened[p] && g->base[p]) cudaIpcCloseMemHandle(g->base[p]);
    if (g->base[g->rank]) cudaFree(g->base[g->rank]);
    delete g;
}

extern "C" void *eoq_b200_gather_buffer(eoq_b200_gather_t *g, uint32_t slot)
{
    return g && slot < g->slots ? g->base[g->rank] + (size_t)slot * g->slot_bytes : nullptr;
}

extern "C" eoq_error_t eoq_b200_gather_status(eoq_b200_gather_t *g, void *stream)
{
    if (!g) return EOQ_ERR_NULL_PTR;
    uint32_t st = 0;
    CU_TRY(cudaMemcpyAsync(&st, g->status.p, 4, cudaMemcpyDeviceToHost, reinterpret_cast<cudaStream_t>(stream)));
    CU_TRY(cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream)));
    if (st) CU_TRY(cudaMemsetAsync(g->status.p, 0, 4, reinterpret_cast<cudaStream_t>(stream)));   // reported once; the object stays usable
    return st ? EOQ_ERR_CUDA : EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_gemv_gather(eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch, int y_dtype,
                                            const float *bias, eoq_b200_gather_t *g, uint32_t slot, uint32_t row_offset,
                                            uint32_t n_total, void *stream)
{
    if (!w || !x || !g) return EOQ_ERR_NULL_PTR;
    if (batch == 0) return EOQ_OK;
    if (batch > 8 || x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2 || slot >= g->slots) return EOQ_ERR_UNSUPPORTED;
    static const size_t esz[3] = {2, 2, 4};
    if ((size_t)row_offset + w->N > n_total || (size_t)batch * n_total * esz[y_dtype] > g->slot_bytes) return EOQ_ERR_BUFFER_TOO_SMALL;
    if (row_offset != g->rank * w->N || (size_t)w->N * g->world != n_total) return EOQ_ERR_UNSUPPORTED;   // equal, rank-ordered shards
    for (uint32_t p = 0; p < g->world; p++)
        if (!g->base[p]) return EOQ_ERR_UNSUPPORTED;                    // eoq_b200_gather_connect has not run
    eoq_error_t drc = check_device(w, "eoq_b200_gemv_gather");
    if (drc != EOQ_OK) return drc;
    if (g->device != w->device) return EOQ_ERR_UNSUPPORTED;
    GemvArgs a = {};
    weight_gemv_args(w, a);
    a.x = x; a.bias = bias; a.counters = w->counters.as<uint32_t>(); a.batch = batch;
    a.pair_partials = w->pair_partials.as<float>();
    a.x_dtype = x_dtype; a.y_dtype = y_dtype;
    a.world = g->world; a.rank = g->rank; a.row_offset = row_offset; a.n_total = n_total;
    for (uint32_t p = 0; p < g->world; p++) a.peer_ll[p] = reinterpret_cast<uint64_t *>(g->base[p] + g->ll_off(slot));
    a.y = g->base[g->rank] + (size_t)slot * g->slot_bytes;
    a.gather_epoch = reinterpret_cast<uint32_t *>(g->base[g->rank] + g->epoch_off(slot));
    a.gather_done = reinterpret_cast<uint32_t *>(g->base[g->rank] + g->done_off(slot));
    a.gather_status = g->status.as<uint32_t>();
    a.gather_g = w->G;
    a.gather_limit = g->limit_ticks;
    // words one sender occupies per activation row (see GemvArgs): must fit the slot's receive buffer
    const size_t wpr = y_dtype == EOQ_B200_F32 ? w->N : w->Npad / w->G;
    if ((size_t)batch * g->world * wpr > g->slot_elems) return EOQ_ERR_BUFFER_TOO_SMALL;
    if (!gemv_takes_pairs(a, w->G, w->bits, w->kind)) {
        const uint32_t bt = batch <= 1 ? 1 : batch <= 2 ? 2 : batch <= 4 ? 4 : 8;
        if (gemv_smem_bytes(w->K, w->p, bt, w->kind) > 227 * 1024) return EOQ_ERR_UNSUPPORTED;
        eoq_error_t rc = ring_scratch(w);
        if (rc != EOQ_OK) return rc;
        a.partials = w->partials.as<float>();
    }
    // one launch: the kernel sends this rank's rows, then waits for the others' and unpacks them
    int e = launch_gemv(a, w->G, w->bits, w->kind, stream);
    if (e != 0) { std::fprintf(stderr, "eoq_b200_gemv_gather: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_gather_set_timeout_ms(eoq_b200_gather_t *g, uint32_t milliseconds)
{
    if (!g) return EOQ_ERR_NULL_PTR;
    if (milliseconds == 0 || milliseconds > 60000) return EOQ_ERR_UNSUPPORTED;
    int khz = 0, dev = g->device;
    if (cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, dev) != cudaSuccess || khz <= 0) khz = 2000000;
    g->limit_ticks = (long long)milliseconds * khz;
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_gather_wait(eoq_b200_gather_t *g, uint32_t slot, uint32_t rows_per_rank, uint32_t batch,
                                            int y_dtype, uint32_t rows_per_word, void *stream)
{
    if (!g) return EOQ_ERR_NULL_PTR;
    if (slot >= g->slots || batch == 0 || batch > 8 || y_dtype < 0 || y_dtype > 2 || rows_per_rank == 0 ||
        rows_per_word < 1 || rows_per_word > 3)
        return EOQ_ERR_UNSUPPORTED;
    static const size_t esz[3] = {2, 2, 4};
    const size_t n_total = (size_t)rows_per_rank * g->world;
    if ((size_t)batch * n_total * esz[y_dtype] > g->slot_bytes) return EOQ_ERR_BUFFER_TOO_SMALL;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) return EOQ_ERR_CUDA;
    if (dev != g->device) return EOQ_ERR_UNSUPPORTED;
    GemvArgs a = {};
    a.N = rows_per_rank;
    a.Npad = (rows_per_rank + 32u * rows_per_word - 1u) / (32u * rows_per_word) * (32u * rows_per_word);
    a.batch = batch; a.y_dtype = y_dtype;
    a.world = g->world; a.rank = g->rank; a.row_offset = g->rank * rows_per_rank; a.n_total = (uint32_t)n_total;
    a.peer_ll[g->rank] = reinterpret_cast<uint64_t *>(g->base[g->rank] + g->ll_off(slot));
    a.y = g->base[g->rank] + (size_t)slot * g->slot_bytes;
    a.gather_epoch = reinterpret_cast<uint32_t *>(g->base[g->rank] + g->epoch_off(slot));
    a.gather_done = reinterpret_cast<uint32_t *>(g->base[g->rank] + g->done_off(slot));
    a.gather_status = g->status.as<uint32_t>();
    a.gather_g = rows_per_word;
    a.gather_limit = g->limit_ticks;
    const size_t wpr = y_dtype == EOQ_B200_F32 ? a.N : a.Npad / rows_per_word;
    if ((size_t)batch * g->world * wpr > g->slot_elems) return EOQ_ERR_BUFFER_TOO_SMALL;
    int e = launch_gather_wait(a, stream);
    if (e != 0) { std::fprintf(stderr, "eoq_b200_gather_wait: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_gemv_host_async(eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch, void *y, int y_dtype,
                                                const float *bias_host, void *stream)
{
    if (!w || !x || !y) return EOQ_ERR_NULL_PTR;
    if (batch == 0) return EOQ_OK;
    if (batch > 8 || x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    static const size_t esz[3] = {2, 2, 4};
    eoq_error_t drc = check_device(w, "eoq_b200_gemv_host");
    if (drc != EOQ_OK) return drc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lock(w->mu);
    CU_TRY(cudaMemcpyAsync(w->xbuf.p, x, (size_t)batch * w->K * esz[x_dtype], cudaMemcpyHostToDevice, st));
    if (bias_host) CU_TRY(cudaMemcpyAsync(w->biasbuf.p, bias_host, (size_t)w->N * 4, cudaMemcpyHostToDevice, st));
    // A pinned (page-locked) y is device-addressable: the kernel then stores its results straight into it and the
    // copy back is not needed.  Pageable memory goes through the weight's device buffer and a copy.
    void *y_direct = nullptr;
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, y) == cudaSuccess && attr.type == cudaMemoryTypeHost && attr.devicePointer) y_direct = attr.devicePointer;
    else (void)cudaGetLastError();
    eoq_error_t rc = eoq_b200_gemv(w, w->xbuf.p, x_dtype, batch, y_direct ? y_direct : w->ybuf.p, y_dtype,
                                   bias_host ? w->biasbuf.as<float>() : nullptr, stream);
    if (rc != EOQ_OK) return rc;
    if (!y_direct) CU_TRY(cudaMemcpyAsync(y, w->ybuf.p, (size_t)batch * w->N * esz[y_dtype], cudaMemcpyDeviceToHost, st));
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_gemv_host(eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch, void *y, int y_dtype,
                                          const float *bias_host, void *stream)
{
    eoq_error_t rc = eoq_b200_gemv_host_async(w, x, x_dtype, batch, y, y_dtype, bias_host, stream);
    if (rc != EOQ_OK || batch == 0) return rc;
    return eoq_b200_weight_status(w, stream);       // reads the status word and synchronises the stream
}

static eoq_error_t weight_decode(eoq_b200_weight_t *w, uint8_t *d_sym, int packed, void *d_dequant, int out_dtype, int early, void *stream)
{
    if (!w) return EOQ_ERR_NULL_PTR;
    if (!d_sym && !d_dequant) return EOQ_OK;
    if (packed && w->bits != 4) return EOQ_ERR_UNSUPPORTED;
    if (d_dequant && w->kind != EOQ_B200_KIND_INT4_ABSMAX) return EOQ_ERR_UNSUPPORTED;      // any integer width dequantises; polar does not
    if (out_dtype < 0 || out_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    eoq_error_t drc = check_device(w, "eoq_b200_weight_decode");
    if (drc != EOQ_OK) return drc;
    DecodeArgs a;
    a.head_bytes = w->head_bytes;
    a.table = w->table.as<uint32_t>(); a.tiles = w->tiles.as<TileDesc>(); a.stream = w->stream.as<uint8_t>();
    a.scales = w->scales.as<uint16_t>(); a.centroids = w->centroids.as<float>();
    a.status = w->status_word();
    a.out_sym = d_sym; a.out_deq = d_dequant; a.N = w->N; a.K = w->K; a.group = w->group; a.p = w->p; a.ntiles = w->ntiles;
    a.packed = packed; a.out_dtype = out_dtype; a.early = early;
    a.scales_t = w->scales_t.as<uint2>(); a.nseg = w->nseg; a.nrb = w->nrb; a.Npad = w->Npad; a.stage_bytes = w->stage_bytes;
    int e = launch_decode_tiles(a, w->G, w->bits, w->kind, stream);
    if (e != 0) { std::fprintf(stderr, "eoq_b200_weight_decode: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    return EOQ_OK;
}

extern "C" eoq_error_t eoq_b200_weight_decode(eoq_b200_weight_t *w, uint8_t *d_sym, int packed, void *d_dequant, int out_dtype, void *stream)
{
    return weight_decode(w, d_sym, packed != 0, d_dequant, out_dtype, 0, stream);
}

extern "C" eoq_error_t eoq_b200_dequant_packed(const uint8_t *d_packed, const uint16_t *d_scales_fp16, uint32_t rows, uint32_t cols,
                                               uint32_t bits, uint32_t group, uint32_t row_lo, uint32_t row_hi, void *d_out,
                                               int out_dtype, void *stream)
{
    if (!d_packed || !d_out || (!d_scales_fp16 && out_dtype != EOQ_B200_I8)) return EOQ_ERR_NULL_PTR;   // codes alone need no scales
    if (bits < 2 || bits > 8 || group == 0 || cols == 0) return EOQ_ERR_INVALID_HEADER;
    if (row_lo > row_hi || row_hi > rows) return EOQ_ERR_INVALID_HEADER;
    if (out_dtype < 0 || out_dtype > EOQ_B200_I8) return EOQ_ERR_UNSUPPORTED;
    if (!have_device()) return EOQ_ERR_CUDA;
    // row stride of QuantizedLinear.packed_weight (core/quantized_linear.py:49-66)
    const uint32_t row_bytes = bits == 4 ? (cols + 1) / 2 : bits == 2 ? (cols + 3) / 4 : cols;
    int e = launch_dequant_packed(d_packed, d_scales_fp16, cols, row_bytes, bits, group, row_lo, row_hi, d_out, out_dtype, stream);
    if (e != 0) { std::fprintf(stderr, "eoq_b200_dequant_packed: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    return EOQ_OK;
}

// What a launch of the product kernel came to.  A device that has no room for any cut of it (or a driver without tensor
// maps) is a call that is not supported, which other routes may take; everything else is a failed launch.
static eoq_error_t product_result(int e, const char *where)
{
    if (e == 0) return EOQ_OK;
    if (e == (int)cudaErrorNotSupported) return EOQ_ERR_UNSUPPORTED;
    std::fprintf(stderr, "%s: launch failed: %s\n", where, cudaGetErrorString((cudaError_t)e));
    return EOQ_ERR_CUDA;
}

static QmmCall packed_call(const uint8_t *d_packed, const uint16_t *d_scales_fp16, uint32_t rows, uint32_t cols, uint32_t bits, uint32_t group,
                           const void *x, int x_dtype, uint32_t batch, void *d_scratch, void *y, int y_dtype, const float *bias)
{
    QmmCall c = {};
    c.packed = d_packed; c.scales = d_scales_fp16; c.bias = bias; c.x = x; c.y = y; c.N = rows; c.K = cols; c.M = batch; c.bits = bits;
    c.group = group; c.bf16 = x_dtype == EOQ_B200_BF16; c.y_dtype = y_dtype;
    if (x_dtype == EOQ_B200_F32) { c.split_x = 1; c.x = d_scratch; }
    return c;
}

extern "C" eoq_error_t eoq_b200_gemv_packed(const uint8_t *d_packed, const uint16_t *d_scales_fp16, uint32_t rows, uint32_t cols,
                                            uint32_t bits, uint32_t group, const void *x, int x_dtype, uint32_t batch, void *d_scratch,
                                            void *y, int y_dtype, const float *bias, void *stream)
{
    if (!d_packed || !d_scales_fp16 || !x || !y) return EOQ_ERR_NULL_PTR;
    if (batch == 0 || rows == 0) return EOQ_OK;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    if (bits < 2 || bits > 8 || group == 0 || cols == 0) return EOQ_ERR_INVALID_HEADER;
    // a lane takes sixteen aligned bytes of a row, in pieces of eight columns of one scale group: other shapes go through
    // the dequantise kernel
    const uint32_t per16 = bits == 4 ? 32u : bits == 2 ? 64u : 16u;
    if (cols % per16 || group % 8u || cols % group || (reinterpret_cast<uintptr_t>(d_packed) & 15u)) return EOQ_ERR_UNSUPPORTED;
    const bool f32 = x_dtype == EOQ_B200_F32;
    // rows: 32 where a group is whole 128-column spans and the product kernel may take them, 8 otherwise
    const bool wide = cols % 128u == 0 && group % 128u == 0 &&
                      (f32 ? d_scratch && (reinterpret_cast<uintptr_t>(d_scratch) & 15u) == 0 : (reinterpret_cast<uintptr_t>(x) & 15u) == 0);
    if (batch > (wide ? 32u : 8u)) return EOQ_ERR_UNSUPPORTED;
    if (!have_device()) return EOQ_ERR_CUDA;
    int e = 0;
    if (wide && (f32 || batch > 8)) {
        // fp32 activations reach the tensor cores as two fp16 halves, written into the caller's scratch by one small launch
        if (f32) e = launch_polar_rotate(x, x_dtype, cols, 0, batch, nullptr, static_cast<uint16_t *>(d_scratch), stream);      // block of 1: no rotation, only the split
        if (e == 0) e = launch_qmm(packed_call(d_packed, d_scales_fp16, rows, cols, bits, group, x, x_dtype, batch, d_scratch, y, y_dtype, bias), stream);
    } else {
        PackedGemvArgs a = {};
        a.packed = d_packed; a.scales = d_scales_fp16; a.x = x; a.y = y; a.bias = bias;
        a.N = rows; a.K = cols; a.group = group; a.batch = batch; a.bits = bits; a.x_dtype = x_dtype; a.y_dtype = y_dtype;
        // row stride of QuantizedLinear.packed_weight (core/quantized_linear.py:49-66)
        a.row_bytes = bits == 4 ? cols / 2 : bits == 2 ? cols / 4 : cols;
        e = launch_gemv_packed(a, stream);
    }
    return product_result(e, "eoq_b200_gemv_packed");
}

// For the torch-facing front (not in the public header): whether up to eight rows of 16-bit activations are to go to
// eoq_b200_gemv_packed's tensor-core form.
extern "C" int eoq_b200_gemv_packed_preferred(uint32_t rows, uint32_t cols, uint32_t bits, uint32_t group) { return group && packed_mma_preferred(rows, cols, bits, group) ? 1 : 0; }

extern "C" eoq_error_t eoq_b200_linear_packed(const uint8_t *d_packed, const uint16_t *d_scales_fp16, uint32_t rows, uint32_t cols,
                                              uint32_t bits, uint32_t group, const void *x, int x_dtype, uint32_t batch, void *d_scratch,
                                              void *y, int y_dtype, const float *bias, void *stream)
{
    if (!d_packed || !d_scales_fp16 || !x || !y) return EOQ_ERR_NULL_PTR;
    if (batch == 0 || rows == 0) return EOQ_OK;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    if (bits < 2 || bits > 8 || group == 0 || cols == 0) return EOQ_ERR_INVALID_HEADER;
    const bool split = x_dtype == EOQ_B200_F32;
    if (split && !d_scratch) return EOQ_ERR_NULL_PTR;
    if (!qmm_takes(cols, bits, group, d_packed, split ? d_scratch : x) || (split && !split_rows_takes(cols, 1))) return EOQ_ERR_UNSUPPORTED;
    if (!have_device()) return EOQ_ERR_CUDA;
    QmmCall c = packed_call(d_packed, d_scales_fp16, rows, cols, bits, group, x, x_dtype, batch, d_scratch, y, y_dtype, bias);
    int e = 0;
    if (split) {
        float *factors = reinterpret_cast<float *>(static_cast<uint8_t *>(d_scratch) + (size_t)batch * cols * 4);
        c.tok_scale = factors;
        e = launch_split_rows(x, x_dtype, cols, batch, 1, d_scratch, factors, stream);
    }
    if (e == 0) e = launch_qmm(c, stream);
    return product_result(e, "eoq_b200_linear_packed");
}

// For the torch-facing front (not in the public header): whether eoq_b200_linear_packed takes the call and is to be
// preferred to a dequantised copy (1.2 T weights/s, and two launches: no call takes less than 5.5 us) and a library GEMM.
extern "C" int eoq_b200_linear_packed_preferred(const uint8_t *d_packed, uint32_t rows, uint32_t cols, uint32_t bits, uint32_t group,
                                                const void *x, int x_dtype, uint32_t batch)
{
    const bool split = x_dtype == EOQ_B200_F32;
    if (!qmm_takes(cols, bits, group, d_packed, x) || (split && !split_rows_takes(cols, 1))) return 0;
    return qmm_preferred(packed_call(d_packed, nullptr, rows, cols, bits, group, x, x_dtype, batch, nullptr, nullptr, x_dtype, nullptr),
                         (double)rows * cols / 1.2e6, 5.5) ? 1 : 0;
}

// Above 64 rows, and above 32 against weights of which several CTAs share the columns anyway (from 8192 rows on a block of 64
// columns costs some 1300 cycles when rotated, 900 to 1500 when not, by the rows).  14336 x 4096 has not been split, so it goes like
// 11008 x 4096: 64 rows 42.0 us / rotated 45.6, 80 rows 48.4 / 46.3, 512 rows 127 / 94.8; 4096 x 4096, 40 rows 16.9 / 16.6, 200
// rows 30.2 / 21.2; 1024 x 4096, 40 rows 12.0 / 9.0.  But not 113 to 128 rows (the other form's tile of 128 tokens, without its folds)
// where row tiles are many and long, 12288 x 4096 45.3 / 47.1, 14336 x 8192 94.1 / 97.6, 28672 x 8192 176 / 211 (11008 x 8192 86.2 / 84.1, 14336 x 2048
// 26.2 / 25.5, 18944 x 8192 101.0 / 101.5), and up to 144 where they are most, 28672 x 4096 101.8 / 104.4, 28672 x 8192 186 / 215 (24576 x 8192 161.7 /
// 162.8, 20480 x 8192 154.1 / 156.1, 18944 x 8192 106.3 / 102.4, 28672 x 11008 253 / 243).
static bool polar_rotates(uint32_t rows, uint32_t cols, uint32_t batch)
{
    if (batch > 112u && cols >= 4096u && (batch <= 128u ? rows >= 12288u : batch <= 144u && rows > 24576u && cols <= 8192u)) return false;
    return batch > 64u || (batch > 32u && rows <= 8192u);
}
extern "C" int eoq_b200_polar_rotates(uint32_t rows, uint32_t cols, uint32_t batch) { return polar_rotates(rows, cols, batch) ? 1 : 0; }      // (for the tests)

extern "C" eoq_error_t eoq_b200_linear_polar_codes(const uint8_t *d_codes, const uint16_t *d_norms_fp16, const float *d_centroids,
                                                   uint32_t rows, uint32_t cols, uint32_t bits, uint32_t block, const void *x, int x_dtype,
                                                   uint32_t batch, void *d_scratch, void *y, int y_dtype, const void *bias, int bias_dtype,
                                                   void *stream)
{
    if (!d_codes || !d_norms_fp16 || !d_centroids || !x || !y || !d_scratch) return EOQ_ERR_NULL_PTR;
    if (bias && bias_dtype != EOQ_B200_F32 && bias_dtype != EOQ_B200_F16) return EOQ_ERR_UNSUPPORTED;
    if (batch == 0 || rows == 0) return EOQ_OK;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    if (bits < 1 || bits > 8 || block == 0 || cols == 0) return EOQ_ERR_INVALID_HEADER;
    if (block < 64 || !qmm_takes(cols, 8, block, d_codes, d_scratch) || !split_rows_takes(cols, block)) return EOQ_ERR_UNSUPPORTED;
    if (!have_device()) return EOQ_ERR_CUDA;
    QmmCall c = {};
    float *factors = reinterpret_cast<float *>(static_cast<uint8_t *>(d_scratch) + (size_t)batch * cols * 4);
    c.packed = d_codes; c.scales = d_norms_fp16; c.centroids = d_centroids; c.bias = bias; c.x = d_scratch; c.tok_scale = factors; c.y = y;
    c.bias_half = bias_dtype == EOQ_B200_F16;
    c.N = rows; c.K = cols; c.M = batch; c.bits = bits; c.group = block; c.split_x = 1; c.y_dtype = y_dtype;
    // many 16-bit rows against blocks of 64: the weight is rotated on its way to the products instead of the activations, which
    // then are one fp16 plane (bf16 ones brought to fp16's range a row at a time) and need two products of a pair, not three
    c.rotate = block == 64 && polar_rotates(rows, cols, batch) && x_dtype != EOQ_B200_F32 && (x_dtype != EOQ_B200_F16 || (reinterpret_cast<uintptr_t>(x) & 15u) == 0);
    if (c.rotate) c.split_x = 0;
    if (c.rotate && x_dtype == EOQ_B200_F16) { c.x = x; c.tok_scale = nullptr; }
    int e = 0;
    if (c.x == d_scratch) e = launch_split_rows(x, x_dtype, cols, batch, c.rotate ? 1 : block, d_scratch, factors, stream);
    if (e == 0) e = launch_qmm(c, stream);
    return product_result(e, "eoq_b200_linear_polar_codes");
}

// Bytes of scratch eoq_b200_weight_linear needs in front of the activations' part: the weight's codes, two per byte.
static size_t weight_codes_bytes(const eoq_b200_weight_t *w) { return ((size_t)w->Npad * w->K / 2 + 255) & ~(size_t)255; }

// Layouts that eoq_b200_weight_linear takes: the pair layout (4-bit codes, three per step; tiles that the pair decoder
// stages whole), groups the product kernel takes.
static bool weight_linear_takes(const eoq_b200_weight_t *w, const void *x, int x_dtype)
{
    return w->kind == EOQ_B200_KIND_INT4_ABSMAX && w->bits == 4 && w->G == 3 && w->scales_t.p && w->stage_bytes <= 6144u && w->p <= 13u &&
           qmm_takes(w->K, 4, w->group, nullptr, x) && (x_dtype != EOQ_B200_F32 || split_rows_takes(w->K, 1));
}

extern "C" size_t eoq_b200_weight_linear_scratch(const eoq_b200_weight_t *w, uint32_t batch, int x_dtype)
{
    return w ? weight_codes_bytes(w) + (x_dtype == EOQ_B200_F32 ? (size_t)batch * (w->K + 1u) * 4u : 0u) : 0u;
}

extern "C" eoq_error_t eoq_b200_weight_linear(eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch, void *d_scratch, void *y,
                                              int y_dtype, const float *bias, void *stream)
{
    if (!w || !x || !y || !d_scratch) return EOQ_ERR_NULL_PTR;
    if (batch == 0) return EOQ_OK;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    if (!weight_linear_takes(w, x, x_dtype) || (reinterpret_cast<uintptr_t>(d_scratch) & 15u)) return EOQ_ERR_UNSUPPORTED;
    eoq_error_t rc = check_device(w, "eoq_b200_weight_linear");
    if (rc != EOQ_OK) return rc;
    uint8_t *codes = static_cast<uint8_t *>(d_scratch), *halves = codes + weight_codes_bytes(w);
    // the activations' halves first: the codes' kernel then is the one that the product follows directly and waits for
    int e = 0;
    float *factors = reinterpret_cast<float *>(halves + (size_t)batch * w->K * 4);
    if (x_dtype == EOQ_B200_F32) e = launch_split_rows(x, x_dtype, w->K, batch, 1, halves, factors, stream);
    if (e == 0) {
        rc = weight_decode(w, codes, 2, nullptr, 0, 1, stream);
        if (rc != EOQ_OK) return rc;
        QmmCall c = packed_call(codes, w->scales.as<uint16_t>(), w->N, w->K, 4, w->group, x, x_dtype, batch, halves, y, y_dtype, bias);
        if (x_dtype == EOQ_B200_F32) c.tok_scale = factors;
        c.late = 1;
        c.status = w->status_word();
        c.blocked_rows = w->Npad;
        e = launch_qmm(c, stream);
    }
    return product_result(e, "eoq_b200_weight_linear");
}

// For the torch-facing front (not in the public header): whether eoq_b200_weight_linear takes the call and is to be
// preferred to a dense decode and a library GEMM.  Both decode; the dense result takes longer to store and to read back
// (11008 x 4096: 30 us), the product 1 us longer to start.
extern "C" int eoq_b200_weight_linear_preferred(const eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch)
{
    if (!w || !weight_linear_takes(w, x, x_dtype)) return 0;
    QmmCall c = packed_call(nullptr, nullptr, w->N, w->K, 4, w->group, x, x_dtype, batch, nullptr, nullptr, x_dtype, nullptr);
    c.blocked_rows = w->Npad;
    return qmm_preferred(c, (double)w->N * w->K / 1.5e6 - 1.0, 0.0) ? 1 : 0;
}

extern "C" uint32_t eoq_b200_linear_status(void) { return qmm_status(); }

extern "C" eoq_error_t eoq_b200_gemv_polar_codes(const uint8_t *d_codes, const uint16_t *d_norms_fp16, const float *d_centroids,
                                                 uint32_t rows, uint32_t cols, uint32_t bits, uint32_t block, const void *x, int x_dtype,
                                                 uint32_t batch, void *d_scratch, void *y, int y_dtype, const float *bias,
                                                 int tensor_cores, void *stream)
{
    if (!d_codes || !d_norms_fp16 || !d_centroids || !x || !y || !d_scratch) return EOQ_ERR_NULL_PTR;
    if (batch == 0 || rows == 0) return EOQ_OK;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    if (bits < 1 || bits > 8 || block == 0 || cols == 0) return EOQ_ERR_INVALID_HEADER;
    // one row alone is quickest on the CUDA cores, several on the tensor cores (a quad of lanes takes 64 columns of one block)
    const bool split = tensor_cores < 0 ? batch >= 2 && block >= 64u : tensor_cores != 0;
    if (batch > (split ? 32u : 8u)) return EOQ_ERR_UNSUPPORTED;
    // a lane takes sixteen codes of one block with one aligned load
    if ((block & (block - 1u)) || block < (split ? 64u : 16u) || block > 4096u || cols % block ||
        ((reinterpret_cast<uintptr_t>(d_codes) | reinterpret_cast<uintptr_t>(d_scratch)) & 15u))
        return EOQ_ERR_UNSUPPORTED;
    if (!have_device()) return EOQ_ERR_CUDA;
    uint32_t shift = 4;
    while ((1u << shift) < block) shift++;
    int e = launch_polar_rotate(x, x_dtype, cols, shift, batch, split ? nullptr : static_cast<float *>(d_scratch),
                                split ? static_cast<uint16_t *>(d_scratch) : nullptr, stream);
    if (e == 0 && split) {
        QmmCall c = {};
        c.packed = d_codes; c.scales = d_norms_fp16; c.centroids = d_centroids; c.bias = bias; c.x = d_scratch; c.y = y;
        c.N = rows; c.K = cols; c.M = batch; c.bits = bits; c.group = block; c.split_x = 1; c.y_dtype = y_dtype;
        e = launch_qmm(c, stream);
    } else if (e == 0) {
        PolarCodesArgs a = {};
        a.codes = d_codes; a.norms = d_norms_fp16; a.centroids = d_centroids; a.y = y; a.bias = bias;
        a.xrot = static_cast<const float *>(d_scratch);
        a.N = rows; a.K = cols; a.batch = batch; a.entries = 1u << bits; a.y_dtype = y_dtype; a.block_shift = shift;
        e = launch_gemv_polar_codes(a, stream);
    }
    return product_result(e, "eoq_b200_gemv_polar_codes");
}

extern "C" eoq_error_t eoq_b200_weight_status(eoq_b200_weight_t *w, void *stream)
{
    if (!w) return EOQ_ERR_NULL_PTR;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    std::lock_guard<std::mutex> lock(w->mu);
    if (!w->status_host) return EOQ_ERR_ALLOC;
    CU_TRY(cudaStreamSynchronize(st));
    return *static_cast<volatile uint32_t *>(w->status_host) ? EOQ_ERR_CUDA : EOQ_OK;
}


// Test hook (not in the public header): copy a resident weight's tile stream (what = 0), tile descriptors (1) or decode
// table (2) to the host; returns the bytes that part has, copies min(bytes, capacity).
extern "C" uint64_t eoq_b200_weight_read(eoq_b200_weight_t *w, int what, void *host, uint64_t capacity)
{
    if (!w) return 0;
    const void *src = what == 0 ? w->stream.p : what == 1 ? w->tiles.p : what == 2 ? w->table.p : nullptr;
    const uint64_t bytes = what == 0 ? w->stream_bytes : what == 1 ? (uint64_t)w->ntiles * sizeof(TileDesc) : what == 2 ? ((uint64_t)4 << w->p) : 0;
    if (src && host && cudaMemcpy(host, src, (size_t)std::min(bytes, capacity), cudaMemcpyDeviceToHost) != cudaSuccess) return 0;
    return bytes;
}

extern "C" int eoq_b200_tune(const char *key, int value)
{
    if (!key) return -1;
    if (std::strcmp(key, "gemv_ctas_per_sm") == 0) { set_gemv_ctas_per_sm(value); return 0; }
    if (std::strcmp(key, "gemm_warps") == 0) { set_gemm_warps(value); return 0; }
    if (std::strcmp(key, "pdl") == 0) { set_pdl(value); return 0; }
    if (std::strcmp(key, "gemv_pairs") == 0) { set_gemv_pairs(value); return 0; }
    if (std::strcmp(key, "v1_lanes") == 0) { set_v1_lanes(value); return 0; }
    if (std::strcmp(key, "packed_warps") == 0) { set_packed_warps(value); return 0; }
    if (std::strcmp(key, "dequant_vec") == 0) { set_dequant_vec(value); return 0; }
    if (std::strcmp(key, "qmm_wait_us") == 0) { set_qmm_wait_us(value); return 0; }
    if (std::strcmp(key, "pinned_refused") == 0) { g_pinned_refused.store(value); return 0; }
    if (std::strcmp(key, "release_scratch") == 0) { DeviceArena::trim(); PinnedBlock::trim(); return 0; }
    if (std::strcmp(key, "symbols_refused") == 0) { g_symbols_refused.store(value); return 0; }
    return -1;
}

extern "C" uint64_t eoq_b200_launch_count(void) { return launch_counter(); }

// =========================================================================
// Fused GEMV for callers that must not allocate
// =========================================================================
//
// Some callers cannot let a library reach the device allocator: a serving loop that has
// handed all of HBM to its own arena, a real-time thread where an allocator lock is a
// latency hazard, or code running under a framework that forbids allocation while it
// replays recorded work.  For them the cross-tile scratch of the fused kernel (the partial
// row sums of the column segments and the per-row-block arrival counters) lives in one
// fixed array in device global memory that is part of the loaded library.  Every GPU that
// loads the library holds the array until the process exits.
//
// In host code `g_gemv_scratch` is only a handle for the symbol, never a device address: its
// address is looked up once per device with cudaGetSymbolAddress (with that device
// current) and the resulting pointer is what the kernel receives.
constexpr size_t kGemvStaticScratchBytes = EOQ_B200_GEMV_STATIC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_gemv_scratch[kGemvStaticScratchBytes];

namespace {
struct StaticScratchMap {
    std::mutex mu;
    void *dev_ptr[64] = {nullptr};
} g_static_scratch;

// First use on a device resolves the symbol; later calls are a table lookup.
eoq_error_t static_scratch_for_current_device(unsigned char **out)
{
    int dev = 0;
    CU_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return EOQ_ERR_UNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_static_scratch.mu);
    if (!g_static_scratch.dev_ptr[dev]) {
        void *p = nullptr;
        CU_TRY(cudaGetSymbolAddress(&p, g_gemv_scratch));
        g_static_scratch.dev_ptr[dev] = p;
    }
    *out = static_cast<unsigned char *>(g_static_scratch.dev_ptr[dev]);
    return EOQ_OK;
}
}  // namespace

extern "C" eoq_error_t eoq_b200_gemv_static_scratch(eoq_b200_weight_t *w, const void *x, int x_dtype, uint32_t batch,
                                                    void *y, int y_dtype, const float *bias, void *stream)
{
    if (!w || !x || !y) return EOQ_ERR_NULL_PTR;
    if (batch == 0) return EOQ_OK;
    if (batch > 8) return EOQ_ERR_UNSUPPORTED;
    if (x_dtype < 0 || x_dtype > 2 || y_dtype < 0 || y_dtype > 2) return EOQ_ERR_UNSUPPORTED;
    eoq_error_t drc = check_device(w, "eoq_b200_gemv_static_scratch");
    if (drc != EOQ_OK) return drc;
    GemvArgs a = {};
    weight_gemv_args(w, a);
    a.x = x; a.y = y; a.bias = bias; a.batch = batch;
    a.x_dtype = x_dtype; a.y_dtype = y_dtype;
    // The scratch request is sized for the kernel that will run.  Two tiles per warp (the default INT4 layout): a few
    // partial rows per pair of row blocks, at most four activation rows per launch.  One tile per warp: one partial row
    // per column segment.  Layout of the array: [arrival counters, one u32 per row block, padded to 256 B][partial sums].
    const bool pairs = gemv_takes_pairs(a, w->G, w->bits, w->kind);
    const uint32_t bt = batch <= 1 ? 1 : batch <= 2 ? 2 : batch <= 4 ? 4 : 8;
    if (!pairs && gemv_smem_bytes(w->K, w->p, bt, w->kind) > 227 * 1024) {
        // same rule as eoq_b200_gemv: rows that do not fit shared memory together run in two halves
        if (bt == 1) return EOQ_ERR_UNSUPPORTED;
        static const size_t esz[3] = {2, 2, 4};
        const uint32_t half = bt / 2, first = std::min(batch, half);
        eoq_error_t rc = eoq_b200_gemv_static_scratch(w, x, x_dtype, first, y, y_dtype, bias, stream);
        if (rc != EOQ_OK || batch <= half) return rc;
        return eoq_b200_gemv_static_scratch(w, static_cast<const uint8_t *>(x) + (size_t)first * w->K * esz[x_dtype], x_dtype,
                                            batch - first, static_cast<uint8_t *>(y) + (size_t)first * w->N * esz[y_dtype],
                                            y_dtype, bias, stream);
    }
    const size_t counter_bytes = (((size_t)w->nrb * 4) + 255) & ~(size_t)255;
    const size_t partial_bytes = pairs ? (size_t)pair_partial_slots(w->nrb, w->nseg) * w->Npad * std::min(bt, 4u) * sizeof(float)
                               : w->nseg > 1 ? (size_t)w->nseg * w->Npad * bt * sizeof(float) : 0;
    if (counter_bytes + partial_bytes > kGemvStaticScratchBytes) {
        std::fprintf(stderr,
                     "eoq_b200_gemv_static_scratch: this weight needs %zu bytes of scratch for %u rows of x, the built-in array holds %zu; "
                     "use eoq_b200_gemv\n",
                     counter_bytes + partial_bytes, batch, kGemvStaticScratchBytes);
        return EOQ_ERR_BUFFER_TOO_SMALL;
    }
    unsigned char *scratch = nullptr;
    eoq_error_t rc = static_scratch_for_current_device(&scratch);
    if (rc != EOQ_OK) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // the array keeps whatever the last call left; the counters are the only part that must start at zero
    CU_TRY(cudaMemsetAsync(scratch, 0, counter_bytes, st));
    // pair_partials stays null: the array cannot keep the "empty slot" pattern between calls, so the runs of a pair of row
    // blocks meet through store, fence and ticket in `partials`
    a.partials = reinterpret_cast<float *>(scratch + counter_bytes);
    a.counters = reinterpret_cast<uint32_t *>(scratch);
    int e = launch_gemv(a, w->G, w->bits, w->kind, stream);
    if (e != 0) { std::fprintf(stderr, "eoq_b200_gemv_static_scratch: launch failed: %s\n", cudaGetErrorString((cudaError_t)e)); return EOQ_ERR_CUDA; }
    return EOQ_OK;
}
