// Memory and copies of handle creation: large host arrays on 2 MB pages, copies between pageable host memory and the
// device through page-locked rings filled by all cores, and a small cache of device blocks for matrices that are
// assembled again and again.
//
// Measured on the B200 host (16 cores): a pageable cudaMemcpy moves 11-18 GB/s, single-threaded, and a fresh host array
// costs 1.1 us per 4 KB page on top (9 ms for 32 MB, 29 ms for 64 MB).  Four 4 MB page-locked chunks filled by OpenMP
// threads while the copy engine drains the others reach 40-44 GB/s of the 53 GB/s the link gives page-locked memory
// (chunks of 1 / 2 / 4 / 8 MB: 29 / 36 / 44 / 41 GB/s), and 2 MB pages bring the first touch of 64 MB from 2.5 to 1.3 ms
// with every core, 29 to 13 ms with one.  cudaMalloc and cudaFree take 0.3-3 ms each there.
#include <emmintrin.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include <omp.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "internal.h"

namespace asb {

constexpr size_t kHugePage = (size_t)2 << 20;

// Arrays of 32 MB and more are always mapped afresh by malloc: on 2 MB pages, with every page touched once by all cores
// (a 4 MB piece of an untouched array takes 350-500 us to copy into, however many threads share its two pages, 4 MB of
// touched memory 80 us).  Smaller arrays come from malloc as they are: it recycles them, and keeping them here instead
// made the caller's own arrays of the same sizes slower.
constexpr size_t kMappedBytes = (size_t)32 << 20;

void *host_alloc(size_t bytes) {
    void *p = nullptr;
    const bool huge = bytes >= kMappedBytes;
    if (posix_memalign(&p, huge ? kHugePage : 64, bytes ? bytes : 64) != 0) return nullptr;
    if (huge) {
        (void)madvise(p, bytes & ~(kHugePage - 1), MADV_HUGEPAGE);  // advice: where it is refused, small pages serve
        char *c = static_cast<char *>(p);
#pragma omp parallel for schedule(static)
        for (int64_t i = 0; i < (int64_t)(bytes >> 12); i++) c[i << 12] = 0;
    }
    return p;
}

// Copies past the caches: the destination is read next by the copy engine, or much later.  (What a core leaves dirty in
// its cache the copy engine has to fetch from there: the last chunks of an upload, read after the cores had gone idle,
// took 250-420 us per 4 MB instead of 80.)
static void copy_streaming(char *dst, const char *src, size_t bytes) {
    const size_t head = std::min<size_t>(bytes, (16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15);
    memcpy(dst, src, head);
    dst += head, src += head, bytes -= head;
    for (; bytes >= 64; bytes -= 64, dst += 64, src += 64) {
        const __m128i *s = reinterpret_cast<const __m128i *>(src);
        __m128i *d = reinterpret_cast<__m128i *>(dst);
        const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2), e = _mm_loadu_si128(s + 3);
        _mm_stream_si128(d, a), _mm_stream_si128(d + 1, b), _mm_stream_si128(d + 2, c), _mm_stream_si128(d + 3, e);
    }
    memcpy(dst, src, bytes);
    _mm_sfence();
}

// memcpy by all cores once the piece is worth waking them for.  The team is always the whole one, of which a smaller
// piece gives work to a few: a region that asks for fewer threads than the last one makes the OpenMP runtime end the
// others, and the next large piece starts them anew (190-550 us for a 4 MB piece that takes 30; fp64 1.1e6 power-law
// rows with x on the device and a pageable y, whose last piece is a smaller one, 1.13 ms, this way 0.48, plain copy 0.72).
void host_copy(void *dst, const void *src, size_t bytes) {
    constexpr size_t kPerThread = 128 << 10;
    const size_t pieces = std::min<size_t>((size_t)std::max(1, omp_get_max_threads()), bytes / kPerThread);
    if (pieces <= 1) {
        memcpy(dst, src, bytes);
        return;
    }
#pragma omp parallel
    {
        const size_t t = (size_t)omp_get_thread_num(), n = std::min(pieces, (size_t)omp_get_num_threads());
        if (t < n) {
            const size_t a = (bytes * t / n) & ~(size_t)63, e = t + 1 == n ? bytes : (bytes * (t + 1) / n) & ~(size_t)63;
            copy_streaming(static_cast<char *>(dst) + a, static_cast<const char *>(src) + a, e - a);
        }
    }
}

// ---- page-locked rings ------------------------------------------------------------------------------
//
// One ring per direction and device, made on first use and kept (2 x 16 MB page-locked per device in use).  A transfer
// holds its ring's lock; an upload returns once its last piece is in the ring (the source may go away), a download
// once everything is in host memory.
//
// Nobody waits here for another caller: whoever finds the ring taken, or its chunks full of copies queued on another
// stream behind who knows what, copies directly, as slow as CUDA moves pageable memory and as independent.

constexpr int kRingChunks = 4;
constexpr size_t kRingChunkBytes = (size_t)4 << 20;
constexpr size_t kRingMinBytes = 64 << 10;  // below this one pageable cudaMemcpyAsync is as fast
constexpr int kRingDevices = 64;

struct Ring {
    std::mutex mu;
    bool ready = false;
    char *buf[kRingChunks] = {};
    cudaEvent_t ev[kRingChunks] = {};
    unsigned long long by[kRingChunks] = {};  // number of the stream whose copy `ev` stands behind
    int next = 0;
    cudaStream_t side = nullptr;  // copy_to_device_beside
    cudaEvent_t side_done = nullptr;
};
static Ring g_up[kRingDevices], g_down[kRingDevices];

static cudaError_t ring_of_current_device(Ring *rings, Ring **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    *out = nullptr;
    if (e == cudaSuccess && dev < kRingDevices) *out = &rings[dev];
    return e;
}

// with the ring's lock held; a ring that cannot be made stays unready and the caller copies directly
static bool ring_ready(Ring &r) {
    if (r.ready) return true;
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < kRingChunks && e == cudaSuccess; k++) {
        if (!r.buf[k]) e = cudaHostAlloc(reinterpret_cast<void **>(&r.buf[k]), kRingChunkBytes, cudaHostAllocDefault);
        if (e == cudaSuccess && !r.ev[k]) e = cudaEventCreateWithFlags(&r.ev[k], cudaEventDisableTiming);
    }
    if (e != cudaSuccess) (void)cudaGetLastError();
    return r.ready = e == cudaSuccess;
}

// While a stream is being captured nothing of it may pass through a ring: the copy would be recorded, not made, and the
// chunk's event could not be waited for from then on, by anyone.  The caller then copies directly, and its wait for that
// copy, which no call here leaves out, ends the capture with an error.
bool being_captured(cudaStream_t st) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &status) == cudaSuccess) return status != cudaStreamCaptureStatusNone;
    (void)cudaGetLastError();  // the legacy stream beside a capturing one
    return true;
}

// Its number, which no other stream ever has; false while it is being captured.
static bool stream_number(cudaStream_t st, unsigned long long *number) {
    if (being_captured(st)) return false;  // (a graph runs where it is launched)
    if (cudaStreamGetId(st, number) == cudaSuccess) return true;
    (void)cudaGetLastError();
    return false;
}

bool page_locked(const void *p) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return at.type != cudaMemoryTypeUnregistered;
}

cudaError_t copy_to_device(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    if (bytes == 0) return cudaSuccess;
    Ring *ring = nullptr;
    unsigned long long number = 0;
    if (bytes >= kRingMinBytes && !page_locked(src) && stream_number(st, &number)) {
        cudaError_t e = ring_of_current_device(g_up, &ring);
        if (e != cudaSuccess) return e;
    }
    if (!ring) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    std::unique_lock<std::mutex> lock(ring->mu, std::try_to_lock);
    if (!lock.owns_lock() || !ring_ready(*ring)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    for (size_t off = 0; off < bytes; off += kRingChunkBytes) {
        const size_t n = std::min(kRingChunkBytes, bytes - off);
        int k = -1;
        for (int i = 0; i < kRingChunks && k < 0; i++) {  // the next chunk whose copy is done, or queued in front of ours
            const int at = (ring->next + i) % kRingChunks;
            if (ring->by[at] == number || cudaEventQuery(ring->ev[at]) == cudaSuccess) k = at;
            else (void)cudaGetLastError();
        }
        if (k < 0)
            return cudaMemcpyAsync(static_cast<char *>(dst) + off, static_cast<const char *>(src) + off, bytes - off,
                                   cudaMemcpyHostToDevice, st);
        ring->next = (k + 1) % kRingChunks;
        cudaError_t e = cudaEventSynchronize(ring->ev[k]);  // the copy that used this chunk last is done
        if (e != cudaSuccess) return e;
        host_copy(ring->buf[k], static_cast<const char *>(src) + off, n);
        ring->by[k] = number;
        e = cudaMemcpyAsync(static_cast<char *>(dst) + off, ring->buf[k], n, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(ring->ev[k], st);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t copy_to_device_beside(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    Ring *ring = nullptr;
    cudaError_t e = ring_of_current_device(g_up, &ring);
    if (e != cudaSuccess) return e;
    if (!ring || bytes < kRingMinBytes || being_captured(st)) return copy_to_device(dst, src, bytes, st);
    cudaStream_t side = nullptr;
    cudaEvent_t done = nullptr;
    {
        std::unique_lock<std::mutex> lock(ring->mu, std::try_to_lock);
        if (!lock.owns_lock()) return copy_to_device(dst, src, bytes, st);
        if (!ring->side_done) {
            e = cudaStreamCreateWithFlags(&ring->side, cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ring->side_done, cudaEventDisableTiming);
            if (e != cudaSuccess) return e;
        }
        side = ring->side, done = ring->side_done;
    }
    e = copy_to_device(dst, src, bytes, side);
    if (e != cudaSuccess) {  // nothing may be on its way to `dst` when the caller gives it up
        if (cudaStreamSynchronize(side) != cudaSuccess) (void)cudaGetLastError();
        return e;
    }
    // (two threads may record one after the other: both copies are then in front of the later record, and the earlier
    // waiter waits for at least its own)
    e = cudaEventRecord(done, side);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st, done, 0);
    return e;
}

cudaError_t copy_to_host(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    if (bytes < kRingMinBytes || page_locked(dst)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
    return Download({{dst, src, bytes}}, st).finish();
}

Download::Download(std::initializer_list<Piece> pieces, cudaStream_t st) : st_(st) {
    size_t total = 0;
    try {
        for (const Piece &p : pieces) {
            total += p.bytes;
            for (size_t off = 0; off < p.bytes; off += kRingChunkBytes)
                chunks_.push_back({static_cast<char *>(p.dst) + off, static_cast<const char *>(p.src) + off,
                                   std::min(kRingChunkBytes, p.bytes - off)});
        }
    } catch (...) {  // no memory for the list: nothing is copied, finish() says so
        error_ = cudaErrorMemoryAllocation;
        return;
    }
    if (total < kRingMinBytes || being_captured(st)) return;  // copied by finish()
    Ring *ring = nullptr;
    error_ = ring_of_current_device(g_down, &ring);
    if (error_ != cudaSuccess || !ring) return;
    if (!ring->mu.try_lock()) return;  // copied by finish()
    if (!ring_ready(*ring)) {
        ring->mu.unlock();
        return;
    }
    ring_ = ring;
    while (issued_ < chunks_.size() && issued_ < kRingChunks && error_ == cudaSuccess) issue();
}

void Download::issue() {
    const Piece &c = chunks_[issued_];
    const size_t k = issued_ % kRingChunks;
    error_ = cudaMemcpyAsync(ring_->buf[k], c.src, c.bytes, cudaMemcpyDeviceToHost, st_);
    if (error_ == cudaSuccess) error_ = cudaEventRecord(ring_->ev[k], st_);
    issued_++;
}

cudaError_t Download::finish() {
    for (; done_ < chunks_.size() && error_ == cudaSuccess; done_++) {
        const Piece &c = chunks_[done_];
        if (!ring_) {
            error_ = cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, st_);
            continue;
        }
        const size_t k = done_ % kRingChunks;
        error_ = cudaEventSynchronize(ring_->ev[k]);
        if (error_ != cudaSuccess) break;
        host_copy(c.dst, ring_->buf[k], c.bytes);
        if (issued_ < chunks_.size()) issue();
    }
    if (!ring_ && error_ == cudaSuccess) error_ = cudaStreamSynchronize(st_);
    return error_;
}

Download::~Download() {
    if (!ring_) return;
    // given up half-way: nothing may still write into the ring (and no error stays behind for the next call to find)
    if (done_ < issued_ && cudaStreamSynchronize(st_) != cudaSuccess) (void)cudaGetLastError();
    ring_->mu.unlock();
}

// ---- small page-locked blocks ---------------------------------------------------------------------------
//
// A call with host vectors of a few kilobytes spends its time on copies of pageable memory, each of which the driver
// stages and waits for by itself.  Such a call packs its vectors into one of these blocks instead: one copy in, results
// stored or copied straight back into the block, one wait.  Blocks are made on first use and kept, at most
// kHostBlocks of them (4 MB); a caller that finds none takes the ordinary way.

constexpr int kHostBlocks = 8;
static std::mutex g_host_block_mu;
static HostBlock g_host_block[kHostBlocks];
static bool g_host_block_taken[kHostBlocks];

bool host_block_take(HostBlock *out) {
    std::lock_guard<std::mutex> lock(g_host_block_mu);
    for (int k = 0; k < kHostBlocks; k++) {
        if (g_host_block_taken[k]) continue;
        HostBlock &b = g_host_block[k];
        if (!b.p && cudaHostAlloc(&b.p, kHostBlockBytes, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
            (void)cudaGetLastError();
            b.p = nullptr;
            return false;
        }
        b.index = k;
        *out = b;
        return g_host_block_taken[k] = true;
    }
    return false;
}

void host_block_give(const HostBlock &b) {
    std::lock_guard<std::mutex> lock(g_host_block_mu);
    g_host_block_taken[b.index] = false;
}

void host_pools_trim() {
    for (Ring *rings : {g_up, g_down})
        for (int d = 0; d < kRingDevices; d++) {
            Ring &r = rings[d];
            std::unique_lock<std::mutex> lock(r.mu, std::try_to_lock);
            if (!lock.owns_lock() || !r.ready) continue;
            for (int k = 0; k < kRingChunks; k++) {  // (its copies may still be queued)
                cudaError_t e = cudaEventSynchronize(r.ev[k]);
                if (e == cudaSuccess) e = cudaFreeHost(r.buf[k]);
                if (e == cudaSuccess) r.buf[k] = nullptr, r.ready = false;
                else (void)cudaGetLastError();
            }
        }
    std::lock_guard<std::mutex> lock(g_host_block_mu);
    for (int k = 0; k < kHostBlocks; k++) {
        if (g_host_block_taken[k] || !g_host_block[k].p) continue;
        if (cudaFreeHost(g_host_block[k].p) != cudaSuccess) (void)cudaGetLastError();
        g_host_block[k].p = nullptr;
    }
}

// ---- device blocks of assembled matrices ---------------------------------------------------------------
//
// Converting triples needs scratch for the sort and one block for the resulting arrays.  A program that assembles its
// matrix at every step would pay cudaMalloc and cudaFree for both each time (1-6 ms of a 5 ms conversion), so blocks
// given back here are kept for the next conversion: at most kCacheBytes over all devices, the oldest leave first, and
// all of them when an allocation fails.
//
// A handle may be destroyed while products with it are still queued.  Nothing is waited for then: waiting for the device
// would end every capture in progress in the process with an error, whoever is recording it, and the stream of the
// products may be gone.  A block whose work was all queued on one stream goes out again only to a taker on that stream,
// which waits for it; one that cannot be told is given to CUDA, which waits for everything.

constexpr size_t kCacheBytes = (size_t)512 << 20;
constexpr size_t kCacheGrain = (size_t)256 << 10;

struct CacheBlock {
    void *p;
    size_t bytes;
    int device;
    BlockUse use;  // kNowhere or kOneStream
};
static std::mutex g_cache_mu;
static std::vector<CacheBlock> g_cache;  // oldest first

static void cache_free(const CacheBlock &b) {
    int prev = -1;
    cudaGetDevice(&prev);
    if (prev != b.device) cudaSetDevice(b.device);
    if (cudaFree(b.p) != cudaSuccess) (void)cudaGetLastError();
    if (prev >= 0 && prev != b.device) cudaSetDevice(prev);
}

bool device_cache_trim() {
    std::vector<CacheBlock> out;
    {
        std::lock_guard<std::mutex> lock(g_cache_mu);
        out.swap(g_cache);
    }
    for (const CacheBlock &b : out) cache_free(b);
    return !out.empty();
}

void BlockUse::add(cudaStream_t st) {
    unsigned long long number = 0;
    if (where == kAnywhere) return;
    if (!stream_number(st, &number) || (where == kOneStream && number != stream)) where = kAnywhere;
    else where = kOneStream, stream = number;
}

cudaError_t device_block_take(size_t bytes, cudaStream_t st, bool kept, DeviceBlock *out) {
    *out = DeviceBlock{};
    const size_t want = (std::max<size_t>(bytes, 1) + kCacheGrain - 1) / kCacheGrain * kCacheGrain;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (device_alloc_denied()) return cudaErrorMemoryAllocation;
    unsigned long long number = 0;
    const bool numbered = stream_number(st, &number);
    const size_t most = kept ? want + want / 4 : 2 * want;
    bool wait = false;
    {
        std::lock_guard<std::mutex> lock(g_cache_mu);
        size_t best = g_cache.size();
        for (size_t i = 0; i < g_cache.size(); i++) {
            const CacheBlock &c = g_cache[i];
            if (c.device != dev || c.bytes < want || c.bytes > most) continue;
            if (c.use.where != BlockUse::kNowhere && !(numbered && c.use.stream == number)) continue;
            if (best == g_cache.size() || c.bytes < g_cache[best].bytes) best = i;
        }
        if (best < g_cache.size()) {
            out->p = g_cache[best].p, out->bytes = g_cache[best].bytes, out->device = dev;
            wait = g_cache[best].use.where != BlockUse::kNowhere;
            g_cache.erase(g_cache.begin() + (ptrdiff_t)best);
        }
    }
    if (out->p) {
        e = wait ? cudaStreamSynchronize(st) : cudaSuccess;
        if (e != cudaSuccess) {
            BlockUse use;
            use.where = BlockUse::kAnywhere;
            device_block_give(out, use);
        }
        return e;
    }
    e = cudaMalloc(&out->p, want);
    if (e == cudaErrorMemoryAllocation && device_cache_trim()) {
        (void)cudaGetLastError();
        e = cudaMalloc(&out->p, want);
    }
    if (e == cudaSuccess) out->bytes = want, out->device = dev;
    return e;
}

void device_block_give(DeviceBlock *b, const BlockUse &use) {
    if (!b->p) return;
    const CacheBlock mine{b->p, b->bytes, b->device, use};
    *b = DeviceBlock{};
    if (mine.bytes > kCacheBytes / 2 || use.where == BlockUse::kAnywhere) {
        cache_free(mine);
        return;
    }
    std::vector<CacheBlock> out;
    bool kept = false;
    try {
        std::lock_guard<std::mutex> lock(g_cache_mu);
        out.reserve(g_cache.size() + 1);  // (this and the next line are all that needs memory)
        g_cache.push_back(mine), kept = true;
        size_t total = 0;
        for (const CacheBlock &c : g_cache) total += c.bytes;
        while (total > kCacheBytes) {
            total -= g_cache.front().bytes;
            out.push_back(g_cache.front());
            g_cache.erase(g_cache.begin());
        }
    } catch (...) {
    }
    if (!kept) cache_free(mine);
    for (const CacheBlock &c : out) cache_free(c);
}

}  // namespace asb
