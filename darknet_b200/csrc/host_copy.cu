// Uploads of images that live in ordinary (pageable) host memory, which is where Darknet's load_image and network_predict's
// callers keep them (src/image.c, calloc).  The driver's own path for such memory copies through its staging buffers on one
// thread, about 15-20 GB/s on this hardware, and the caller waits for it; here a few threads copy chunks into a page-locked
// ring and each chunk's DMA (55 GB/s) starts as soon as it is there.  The ring belongs to the pool: at most 16 MB per process, whatever
// the number and the batch of its networks, and as many slots of it as the largest batch so far had chunks.  Measured on this
// path, 2 / 16.6 / 71 MB: driver 211 / 1351 / 6386 us, this 86 / 484 / 1911 us.
#include "host_copy.h"

#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <atomic>
#include <condition_variable>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

#include "common.h"

namespace dnb {

// Small enough that the first transfer starts early, large enough that what a transfer costs beside its bytes (5-6 us) stays
// a fraction of its time on the bus (9 us per 512 KB); larger ones where there are many.
constexpr size_t COPY_CHUNK = 512 * 1024, COPY_CHUNK_MAX = 1024 * 1024, COPY_MANY = 8 * 1024 * 1024;
// A slot is as long as the longest chunk, whatever the upload's own: its event then guards the same bytes for every upload, and one
// of another chunk length cannot reach bytes whose transfer has not been waited for.
constexpr size_t COPY_RING = 16, COPY_GROUP = 2 * COPY_CHUNK_MAX;   // slots; page-locked memory is taken in multiples of two
// Below this a second thread cannot be awake before the copy is over.
constexpr size_t COPY_ALONE = 1024 * 1024;

// Copies past the cache.  Chunks that stayed dirty in the copying cores' caches were read by the copy engine at 7 GB/s.
static void copy_streaming(char *dst, const char *src, size_t bytes)
{
#if defined(__SSE2__)
    const size_t whole = ((uintptr_t)dst % 16) ? 0 : bytes / 64 * 64;
    for (size_t i = 0; i < whole; i += 64) {
        const __m128i a = _mm_loadu_si128((const __m128i *)(src + i)), b = _mm_loadu_si128((const __m128i *)(src + i + 16));
        const __m128i c = _mm_loadu_si128((const __m128i *)(src + i + 32)), d = _mm_loadu_si128((const __m128i *)(src + i + 48));
        _mm_stream_si128((__m128i *)(dst + i), a);
        _mm_stream_si128((__m128i *)(dst + i + 16), b);
        _mm_stream_si128((__m128i *)(dst + i + 32), c);
        _mm_stream_si128((__m128i *)(dst + i + 48), d);
    }
    if (whole < bytes) memcpy(dst + whole, src + whole, bytes - whole);
    _mm_sfence();
#else
    memcpy(dst, src, bytes);
#endif
}

class CopyPool {
public:
    ~CopyPool()
    {
        {
            std::lock_guard<std::mutex> g(lock_);
            quit_ = true;
        }
        wake_.notify_all();
        for (std::thread &t : threads_) t.join();
        drop_events();
        for (char *g : blocks_) {
            cudaHostUnregister(g);
            free(g);
        }
    }

    int upload(char *dst, const char *src, size_t bytes, size_t of, cudaStream_t s)
    {
        std::lock_guard<std::mutex> turn(turn_);
        const size_t chunk = bytes > COPY_MANY ? COPY_CHUNK_MAX : COPY_CHUNK, n = (bytes + chunk - 1) / chunk;
        const size_t step = (of + chunk - 1) / chunk, depth = grow(step < COPY_RING ? step : COPY_RING);
        if (!depth || !ready()) return NOT_STAGED;
        const bool helped = bytes > COPY_ALONE && start_threads();
        auto job = std::make_shared<Job>();   // a worker may still look at it after the last chunk is taken
        for (size_t i = 0; i < depth; ++i) job->slot[i] = slot_[i];
        job->depth = depth; job->src = src; job->bytes = bytes; job->chunk = chunk; job->chunks = n;
        job->done.reset(new std::atomic<bool>[n]);
        for (size_t i = 0; i < n; ++i) job->done[i].store(false, std::memory_order_relaxed);
        if (helped) {
            {
                std::lock_guard<std::mutex> g(lock_);
                job_ = job;
                ++generation_;
            }
            wake_.notify_all();
        }
        size_t told = 0, open = 0;             // chunks enqueued; chunks that may be copied (their ring slots are free)
        cudaError_t err = cudaSuccess;
        while (told < n) {
            while (open < n && open < told + depth) {   // a slot is free when its last transfer has left it
                const cudaError_t q = cudaEventQuery(sent_[open % depth]);
                if (q == cudaErrorNotReady) break;
                if (q != cudaSuccess) err = q;
                job->limit.store(++open, std::memory_order_release);
            }
            if (told < open && job->done[told].load(std::memory_order_acquire)) {
                const size_t at = told * chunk, len = bytes - at < chunk ? bytes - at : chunk, slot = told % depth;
                if (err == cudaSuccess) err = cudaMemcpyAsync(dst + at, slot_[slot], len, cudaMemcpyHostToDevice, s);
                if (err == cudaSuccess) err = cudaEventRecord(sent_[slot], s);
                ++told;
            } else if (!job->one()) {
                std::this_thread::yield();     // another thread is about to finish this chunk, or the ring is full
            }
        }
        if (helped) {
            std::lock_guard<std::mutex> g(lock_);
            job_.reset();
        }
        DNB_CUDA(err);
        return DNB_OK;
    }

private:
    struct Job {
        char *slot[COPY_RING] = {};
        const char *src = nullptr;
        size_t depth = 0, bytes = 0, chunk = 0, chunks = 0;
        std::atomic<size_t> next{0}, limit{0};
        std::unique_ptr<std::atomic<bool>[]> done;
        bool taken() const { return next.load(std::memory_order_relaxed) >= chunks; }
        bool one()   // copies the next chunk, if one may be copied now
        {
            size_t i = next.load(std::memory_order_relaxed);
            do {
                if (i >= chunks || i >= limit.load(std::memory_order_acquire)) return false;
            } while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
            const size_t at = i * chunk, len = bytes - at < chunk ? bytes - at : chunk;
            copy_streaming(slot[i % depth], src + at, len);
            done[i].store(true, std::memory_order_release);
            return true;
        }
    };

    // Slots of the ring up to `want`, as many as there are to be had: what is missing at once, else two slots at a time.  Pages of 2 MB
    // where the system has them: taking and locking 16 MB takes 3.7 ms with them, 13 to 20 with 4 KB pages.
    size_t grow(size_t want)
    {
        for (size_t bytes; slots_ < want && !full_;) {
            blocks_.reserve(COPY_RING);
            bytes = (want - slots_ + 1) / 2 * COPY_GROUP;
            char *g = lock_pages(bytes);
            if (!g && bytes > COPY_GROUP) g = lock_pages(bytes = COPY_GROUP);
            full_ = !g;                        // no more page-locked memory: go on with what there is
            if (!g) break;
            blocks_.push_back(g);
            for (size_t at = 0; at < bytes; at += COPY_CHUNK_MAX) slot_[slots_++] = g + at;
        }
        return slots_ < want ? slots_ : want;
    }

    static char *lock_pages(size_t bytes)
    {
        char *g = (char *)aligned_alloc(COPY_GROUP, bytes);
        if (g) madvise(g, bytes, MADV_HUGEPAGE);
        if (g && cudaHostRegister(g, bytes, cudaHostRegisterPortable) == cudaSuccess) return g;
        cudaGetLastError();
        free(g);
        return nullptr;
    }

    bool start_threads()
    {
        if (threads_.empty() && !alone_) {
            const unsigned cores = std::thread::hardware_concurrency();
            const unsigned n = cores > 4 ? 3 : cores > 1 ? 1 : 0;   // beside the caller
            try {
                for (unsigned i = 0; i < n; ++i) threads_.emplace_back([this] { work(); });
            } catch (const std::exception &) {}                     // no more threads to be had: those that there are, or the caller alone
            alone_ = threads_.empty();
        }
        return !alone_;
    }

    // The ring's events, on the current device.
    bool ready()
    {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return false; }
        if (device_ == dev) return true;
        drop_events();
        for (cudaEvent_t &e : sent_)
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); return false; }
        device_ = dev;
        return true;
    }
    void drop_events()
    {
        for (cudaEvent_t &e : sent_) {
            if (e) { cudaEventSynchronize(e); cudaEventDestroy(e); }
            e = nullptr;
        }
        device_ = -1;
    }

    void work()
    {
        unsigned long long seen = 0;
        for (;;) {
            std::shared_ptr<Job> job;
            {
                std::unique_lock<std::mutex> g(lock_);
                wake_.wait(g, [&] { return quit_ || generation_ != seen; });
                if (quit_) return;
                seen = generation_;
                job = job_;
            }
            // (Sleeping where there is nothing to copy for a while frees little, the threads copy most of the time, and made 284 MB
            // take 10.0 ms instead of 9.4.)
            while (job && !job->taken())
                if (!job->one()) std::this_thread::yield();
        }
    }

    std::vector<char *> blocks_;   // the ring's memory
    char *slot_[COPY_RING] = {};
    size_t slots_ = 0;
    bool full_ = false, alone_ = false;
    cudaEvent_t sent_[COPY_RING] = {};
    int device_ = -1;
    std::mutex turn_, lock_;
    std::condition_variable wake_;
    std::shared_ptr<Job> job_;
    unsigned long long generation_ = 0;
    bool quit_ = false;
    std::vector<std::thread> threads_;
};

std::shared_ptr<CopyPool> copy_pool(bool make)
{
    static std::mutex lock;
    static std::weak_ptr<CopyPool> pool;
    std::lock_guard<std::mutex> g(lock);
    std::shared_ptr<CopyPool> p = pool.lock();
    if (p || !make) return p;
    try {
        p = std::make_shared<CopyPool>();
    } catch (const std::exception &) {}
    pool = p;
    return p;
}

int upload_staged(CopyPool *pool, void *dst, const void *src, size_t bytes, size_t of, cudaStream_t s)
{
    try {
        return pool ? pool->upload((char *)dst, (const char *)src, bytes, of, s) : NOT_STAGED;
    } catch (const std::exception &) {   // of what an upload sets up, before it does anything
        return NOT_STAGED;
    }
}

}  // namespace dnb
