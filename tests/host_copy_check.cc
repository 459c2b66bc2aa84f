// Uploads through darknet_b200/csrc/host_copy.cu against a CUDA runtime made of host memory: transfers wait in a queue and move one
// at a time, only when somebody asks whether an event has completed, so whatever may still be unread in the staging ring is.
//   host_copy_check in_turn     small, large, small ... uploads from one thread, nothing waited for in between
//   host_copy_check threads     the same from two threads, a stream each
//   host_copy_check no_threads  the system refuses every thread: the caller copies alone
//   host_copy_check no_memory   there is no page-locked memory: nothing is staged, and the caller is told so
//   host_copy_check little_memory   there are two slots of it
//   host_copy_check small       a few small images: little page-locked memory is taken, and no thread started
// Prints "ok" and returns 0, or says what is wrong.
#include <cuda_runtime.h>
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <deque>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../darknet_b200/csrc/host_copy.h"

namespace {
struct Event { int pending = 0; };
struct Op { Event *event; char *dst; const char *src; size_t bytes; };
std::mutex engine;
std::deque<Op> queued;
bool no_threads;
int threads_asked;
size_t locked, may_lock = 16 << 20;   // bytes of page-locked memory: taken, and to be had

void step()   // with the engine's lock
{
    if (queued.empty()) return;
    const Op op = queued.front();
    queued.pop_front();
    if (op.event) --op.event->pending;
    else memcpy(op.dst, op.src, op.bytes);
}
}  // namespace

extern "C" {
int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x)
{
    typedef int (*Create)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static const Create create = (Create)dlsym(RTLD_NEXT, "pthread_create");
    ++threads_asked;
    return no_threads ? EAGAIN : create(t, a, f, x);
}
cudaError_t cudaHostRegister(void *, size_t bytes, unsigned)
{
    if (locked + bytes > may_lock) return cudaErrorMemoryAllocation;
    locked += bytes;
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t) new Event(); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event *)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
    std::lock_guard<std::mutex> g(engine);
    ++((Event *)e)->pending;
    queued.push_back(Op{(Event *)e, nullptr, nullptr, 0});
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e)
{
    std::lock_guard<std::mutex> g(engine);
    if (!((Event *)e)->pending) return cudaSuccess;
    step();
    return cudaErrorNotReady;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    std::lock_guard<std::mutex> g(engine);
    while (((Event *)e)->pending) step();
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t bytes, cudaMemcpyKind, cudaStream_t)
{
    std::lock_guard<std::mutex> g(engine);
    queued.push_back(Op{nullptr, (char *)dst, (const char *)src, bytes});
    return cudaSuccess;
}
}

namespace dnb {
static thread_local std::string error_text;
void set_error(const char *fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    error_text = buf;
}
const char *get_error() { return error_text.c_str(); }
int sm_count() { return 148; }
bool pdl_enabled() { return true; }
}  // namespace dnb

namespace {
struct Upload {
    std::vector<unsigned> src, want, dst;
    Upload(size_t words, unsigned seed) : src(words), dst(words)
    {
        for (size_t i = 0; i < words; ++i) src[i] = (unsigned)i * 2654435761u + seed;
        want = src;
    }
    bool run(dnb::CopyPool *pool, cudaStream_t s)
    {
        const int rc = dnb::upload_staged(pool, dst.data(), src.data(), src.size() * 4, src.size() * 4, s);
        std::fill(src.begin(), src.end(), 0u);   // the images have been read when the call returns
        if (rc) printf("upload failed with %d: %s\n", rc, dnb::get_error());
        return rc == 0;
    }
};

bool right(std::vector<std::unique_ptr<Upload>> &all)
{
    {
        std::lock_guard<std::mutex> g(engine);
        while (!queued.empty()) step();
    }
    for (size_t k = 0; k < all.size(); ++k)
        for (size_t i = 0; i < all[k]->want.size(); ++i)
            if (all[k]->dst[i] != all[k]->want[i]) {
                printf("upload %zu of %zu bytes: wrong from byte %zu on\n", k, all[k]->want.size() * 4, i * 4);
                return false;
            }
    return true;
}

// Sizes on both sides of what changes the chunk's length and the number of threads; ragged ones among them.
const size_t SIZES[] = {1 << 20, 5000001, 100, 300000, 2097152, 4194304, 131073, 2097153, 7};

bool sequence(dnb::CopyPool *pool, std::vector<std::unique_ptr<Upload>> &all, int rounds, unsigned seed, cudaStream_t s)
{
    for (int r = 0; r < rounds; ++r)
        for (size_t words : SIZES) {
            all.emplace_back(new Upload(words, seed++));
            if (!all.back()->run(pool, s)) return false;
        }
    return true;
}
}  // namespace

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    std::vector<std::unique_ptr<Upload>> a, b;
    no_threads = what == "no_threads";
    if (what == "no_memory") may_lock = 0;
    if (what == "little_memory") may_lock = 3 << 20;
    {
        std::shared_ptr<dnb::CopyPool> pool = dnb::copy_pool(true);
        if (what == "in_turn") {
            if (!sequence(pool.get(), a, 2, 1, nullptr) || !right(a)) return 1;
        } else if (what == "threads") {
            bool ok[2] = {false, false};
            std::thread t([&] { ok[0] = sequence(pool.get(), a, 2, 1, (cudaStream_t)1); });
            ok[1] = sequence(pool.get(), b, 2, 1000, (cudaStream_t)2);
            t.join();
            if (!ok[0] || !ok[1] || !right(a) || !right(b)) return 1;
        } else if (what == "small") {
            no_threads = true;   // refused, and counted
            for (unsigned k = 0; k < 5; ++k) {
                a.emplace_back(new Upload(196608, k));   // 256 x 256 pixels
                if (!a.back()->run(pool.get(), nullptr)) return 1;
            }
            if (!right(a) || locked > 2 << 20 || threads_asked) return 1;
        } else if (what == "no_threads" || what == "little_memory") {
            if (!sequence(pool.get(), a, 1, 1, nullptr) || !right(a)) return 1;
        } else if (what == "no_memory") {
            for (size_t words : SIZES) {
                Upload u(words, 1);
                if (dnb::upload_staged(pool.get(), u.dst.data(), u.src.data(), words * 4, words * 4, nullptr) != dnb::NOT_STAGED || !queued.empty()) return 1;
            }
        } else {
            printf("what?\n");
            return 2;
        }
    }
    printf("ok\n");
    return 0;
}
