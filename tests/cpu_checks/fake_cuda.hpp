// A stand-in for the CUDA runtime calls of the host layer, so that its copies can be checked without a GPU.  "Device"
// memory is host memory; a stream is a thread that carries out its work in order, every item some milliseconds after its
// turn came; a call can be made to fail by its number.
#pragma once
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <sys/mman.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <set>
#include <thread>

namespace fake {

static const int DELAY_MS = 10;
static std::atomic<int> fail_download{0};      // the n-th copy to the host from now on fails
static std::atomic<int> fail_sync{0};          // the n-th stream synchronisation from now on waits and then fails
static std::atomic<int> fail_thread{0};        // threads cannot be started while this is set
static std::atomic<int> frees{0}, freeing{0};
static std::atomic<int> free_ms{0};            // what giving back page-locked memory takes

static std::mutex pinned_mu;
static std::set<std::thread::id> copiers;      // threads that have queued a copy
static std::map<char *, size_t> pinned;

inline bool is_pinned(const void *p)
{
    std::lock_guard<std::mutex> lk(pinned_mu);
    auto it = pinned.upper_bound((char *)p);
    if (it == pinned.begin()) return false;
    --it;
    return (char *)p < it->first + it->second;
}

class Stream {
  public:
    Stream() : thread_([this] { work(); }) { thread_.detach(); }
    uint64_t push(std::function<void()> fn)
    {
        std::lock_guard<std::mutex> lk(mu_);
        items_.push_back(std::move(fn));
        cv_.notify_all();
        return ++pushed_;
    }
    void wait(uint64_t upto)
    {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return done_ >= upto; });
    }
    void wait() { wait(pushed()); }
    uint64_t pushed()
    {
        std::lock_guard<std::mutex> lk(mu_);
        return pushed_;
    }

  private:
    void work()
    {
        std::unique_lock<std::mutex> lk(mu_);
        while (true) {
            cv_.wait(lk, [this] { return !items_.empty(); });
            auto fn = std::move(items_.front());
            items_.pop_front();
            lk.unlock();
            std::this_thread::sleep_for(std::chrono::milliseconds(DELAY_MS));
            fn();
            lk.lock();
            done_++;
            cv_.notify_all();
        }
    }
    std::mutex mu_;
    std::condition_variable cv_;
    std::deque<std::function<void()>> items_;
    uint64_t pushed_ = 0, done_ = 0;
    std::thread thread_;
};

struct Event {
    Stream *stream = nullptr;
    uint64_t at = 0;
};

inline Stream *of(cudaStream_t st) { return (Stream *)st; }
inline Stream &library_stream()
{
    static Stream &s = *new Stream;
    return s;
}
inline bool due(std::atomic<int> &n) { return n.load() > 0 && n.fetch_sub(1) == 1; }

}  // namespace fake

// --- the library's own runtime --------------------------------------------------------------------------------------
namespace cb200 {
static thread_local char g_err[1024] = "";
int fail(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return 1;
}
void clear_error() { g_err[0] = 0; }
void trace(const char *, ...) {}
cudaStream_t lib_stream() { return (cudaStream_t)&fake::library_stream(); }
}  // namespace cb200

// --- CUDA -------------------------------------------------------------------------------------------------------------
extern "C" {

cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { *p = malloc(n); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeAsync(void *p, cudaStream_t st)
{
    fake::of(st)->push([p] { free(p); });
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned)
{
    // mapped shared, as the driver does it
    *p = mmap(nullptr, (n + 4095) / 4096 * 4096, PROT_READ | PROT_WRITE, MAP_SHARED | MAP_ANONYMOUS, -1, 0);
    std::lock_guard<std::mutex> lk(fake::pinned_mu);
    fake::pinned[(char *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void *p, size_t n, unsigned)
{
    std::lock_guard<std::mutex> lk(fake::pinned_mu);
    fake::pinned[(char *)p] = n;
    return cudaSuccess;
}
static void fake_unpin(void *p)
{
    fake::freeing++;
    std::this_thread::sleep_for(std::chrono::milliseconds(fake::free_ms.load()));
    fake::freeing--;
    fake::frees++;
    std::lock_guard<std::mutex> lk(fake::pinned_mu);
    fake::pinned.erase((char *)p);
}
cudaError_t cudaHostUnregister(void *p) { fake_unpin(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p)
{
    fake_unpin(p);                                      // the pages stay mapped: nobody looks
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p)
{
    a->type = fake::is_pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *dst, size_t dp, const void *src, size_t sp, size_t w, size_t h, cudaMemcpyKind kind, cudaStream_t st)
{
    if (kind == cudaMemcpyDeviceToHost && fake::due(fake::fail_download)) return cudaErrorUnknown;
    {
        std::lock_guard<std::mutex> lk(fake::pinned_mu);
        fake::copiers.insert(std::this_thread::get_id());
    }
    auto copy = [=] {
        for (size_t r = 0; r < h; r++) memcpy((char *)dst + r * dp, (const char *)src + r * sp, w);
    };
    fake::of(st)->push(copy);
    if (!fake::is_pinned(kind == cudaMemcpyDeviceToHost ? dst : src)) fake::of(st)->wait();      // pageable memory: done on return
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind kind, cudaStream_t st)
{
    return cudaMemcpy2DAsync(dst, n, src, n, n, 1, kind, st);
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t st)
{
    fake::of(st)->push([=] { memset(p, v, n); });
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st)
{
    fake::of(st)->wait();
    return fake::due(fake::fail_sync) ? cudaErrorUnknown : cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = (cudaEvent_t) new fake::Event; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st)
{
    ((fake::Event *)e)->stream = fake::of(st);
    ((fake::Event *)e)->at = fake::of(st)->pushed();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e)
{
    fake::Event *ev = (fake::Event *)e;
    if (ev->stream) ev->stream->wait(ev->at);
    std::this_thread::sleep_for(std::chrono::milliseconds(fake::DELAY_MS));      // the waiter is late
    return cudaSuccess;
}

}
