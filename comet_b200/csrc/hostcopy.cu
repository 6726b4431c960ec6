// Copies between HOST memrefs and the device for the host-memref entry points.
//
// COMET's generated code gets its memrefs from memref.alloc, i.e. malloc: pageable memory.  A
// cudaMemcpyAsync on pageable memory is staged by the driver through one internal buffer on the
// calling thread and reaches a fraction of the PCIe rate, and it is not asynchronous.  Here copies on pageable
// memory go through a ring of page-locked chunks owned by the library instead: a few worker threads, and
// the calling thread while it has to wait, move the bytes between the caller's array and the chunks (several
// chunks in flight, so the memcpy bandwidth of several cores adds up) while the DMA engine moves chunks that
// are already filled, in stream order.  Page-locked (or registered) host memory and copies of a few pages take
// the plain cudaMemcpyAsync path.
//
//   h2d / h2d_2d : return when every byte of the host array has been read (like cudaMemcpyAsync on
//                  pageable memory); the device side is complete in stream order.  Between uploads_begin() and
//                  uploads_join() they return at once and the join waits for all of them, so that the arrays of an
//                  operand are copied side by side; work that reads them is launched after the join.
//   d2h / d2h_2d : return when every chunk's DMA has been enqueued; the bytes reach the host array
//                  on the worker threads.  copies_drain() waits for them and must be called (after
//                  the stream has been synchronised or not -- it waits on each chunk's own event)
//                  before the entry point returns to its caller.
#include <atomic>
#include <condition_variable>
#include <deque>
#include <functional>
#include <mutex>
#include <string.h>
#include <system_error>
#include <thread>
#include <vector>

#include "common.cuh"
#include "hostcopy.cuh"
#include "streamcopy.cuh"

namespace cb200 {

namespace {

// Measured on this host (16 virtual cores): one core copies 16 GB/s, eight 35 to 40, PCIe moves 53; the driver's own
// staging 14.  Waking a worker takes 12 us and the DMA engine reads the chunks while others are written, so few threads with
// large pieces beat many with small ones (4.3 MB / 17 MB / 70 MB in and out: five threads and pieces of 1.5 MB 225 / 601 /
// 3500 us, eight and 512 KB 272 / 639 / 3580).
//
// What a worker reads of the caller's arrays is in its core's caches afterwards, and the caller's next writes there have to
// take the lines back.  A program that rewrites its operands before each call pays for that what the workers saved, and more
// while the arrays fit the caches.  Microseconds to write operands of 4.2 / 10.2 / 25.6 MB and to multiply by them (SpMV,
// rows of 16), by number of workers: none 249 + 375 / 612 + 735 / 1590 + 1940, one 409 + 310 / 890 + 530 / 2000 + 1220, two
// 690 + 309 / 1193 + 481 / 2085 + 915, five 890 + 332 / 1820 + 520 / 2730 + 890; the driver's own copies 252 + 410 / 610 +
// 767 / 1810 + 1980.  So the calling thread copies the first WORKERS_FROM bytes of what it is given alone, and there is one
// more worker for every BYTES_PER_WORKER after them (with 4 MB instead of 8 the 25.6 MB take as long as the driver's copies).
const size_t WORKERS_FROM = (size_t)8 << 20, BYTES_PER_WORKER = (size_t)8 << 20;
const size_t CHUNK = (size_t)2 << 20;     // bytes per page-locked chunk
const int SLAB_CHUNKS = 8;                // chunks are allocated 16 MiB at a time (7 ms each),
const int MAX_SLABS = 4;                  // at most 64 MiB per device
const size_t PIECE_MIN = (size_t)1536 << 10;
const size_t STAGE_MIN_DEFAULT = (size_t)96 << 10;  // smaller copies are left to the driver

struct Slot {
    char *buf = nullptr;
    cudaEvent_t ev = nullptr;
    bool dma_pending = false;             // an H2D copy out of this chunk may still be running
};

struct Batch {                            // the chunks of one upload call
    int left = 0;
};

class Pool {
  public:
    explicit Pool(int device) : device_(device)
    {
        // half of the cores this process can count on (16 cores, five / eight / eleven workers: 20.5 GB of results 612 / 520 /
        // 527 ms, 2.4 GB in and out 60.5 / 55.3 / 55.8, 100 MB 3.58 / 3.66 / 3.73 ms): launchers that start one process per
        // GPU export LOCAL_WORLD_SIZE, and the processes of one node share its cores
        int share = 1;
        const char *lws = getenv("LOCAL_WORLD_SIZE");
        if (lws && atoi(lws) > 1) share = atoi(lws);
        int n = (int)std::thread::hardware_concurrency() / (2 * share);
        const char *env = getenv("COMET_B200_COPY_THREADS");
        if (env) n = atoi(env);
        if (n < 2) n = 2;
        if (n > 12) n = 12;
        slots_.reserve(SLAB_CHUNKS * MAX_SLABS);
        grow(1);
        try {
            for (int i = 0; i < n; i++) workers_.emplace_back([this] { work(); });
        } catch (const std::system_error &) {  // no more threads to be had: whoever waits for a copy carries queued ones out
        }
    }
    bool usable() const { return slots_.size() >= 2; }
    int threads() const { return (int)workers_.size() + 1; }

    // more chunks for a copy that would wait for them
    void grow(int slabs)
    {
        std::lock_guard<std::mutex> lk(mu_);
        while (slabs_ < slabs && slabs_ < MAX_SLABS) {
            char *buf = nullptr;
            slabs_++;
            if (cudaHostAlloc((void **)&buf, CHUNK * SLAB_CHUNKS, cudaHostAllocDefault) != cudaSuccess) {
                (void)cudaGetLastError();
                slabs_ = MAX_SLABS;        // do not try again
                return;
            }
            for (int i = 0; i < SLAB_CHUNKS; i++) {
                Slot s;
                s.buf = buf + i * CHUNK;
                if (cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming) != cudaSuccess) return;
                slots_.push_back(s);       // reserved above: the elements never move
                free_.push_back((int)slots_.size() - 1);
            }
        }
    }

    // a free chunk; while there is none the calling thread does queued copies itself
    int acquire()
    {
        std::unique_lock<std::mutex> lk(mu_);
        while (free_.empty())
            if (!run_one(lk)) cv_free_.wait(lk, [this] { return !free_.empty() || !tasks_.empty(); });
        const int i = free_.front();
        free_.pop_front();
        lk.unlock();
        if (slots_[i].dma_pending) {
            if (cudaEventSynchronize(slots_[i].ev) != cudaSuccess) failed_ = true;
            slots_[i].dma_pending = false;
        }
        return i;
    }
    void release(int i)
    {
        {
            std::lock_guard<std::mutex> lk(mu_);
            free_.push_back(i);
        }
        cv_free_.notify_one();
    }
    Slot &slot(int i) { return slots_[i]; }

    void submit(std::function<void()> fn, size_t bytes, Batch *batch = nullptr)
    {
        bool wake;
        {
            std::lock_guard<std::mutex> lk(mu_);
            tasks_.push_back(Task{std::move(fn), batch});
            if (pending_++ == 0) busy_bytes_ = 0;
            busy_bytes_ += bytes;
            if (batch) batch->left++;
            wake = awake_ < workers_.size() && WORKERS_FROM + awake_ * BYTES_PER_WORKER <= busy_bytes_;
            if (wake) {
                awake_++;
                calls_++;
            }
        }
        if (wake) cv_task_.notify_one();
    }
    // waits until the tasks of one batch have run, doing queued ones meanwhile
    void wait(Batch *batch)
    {
        std::unique_lock<std::mutex> lk(mu_);
        while (batch->left > 0)
            if (!run_one(lk)) cv_done_.wait(lk, [batch] { return batch->left == 0; });
    }
    bool take_failure() { return failed_.exchange(false); }
    // waits until every submitted task has run; returns non-zero if one of them failed
    int drain()
    {
        std::unique_lock<std::mutex> lk(mu_);
        while (pending_ > 0)
            if (!run_one(lk)) cv_done_.wait(lk, [this] { return pending_ == 0; });
        const bool f = failed_.exchange(false);
        return f ? 1 : 0;
    }
    void fail_flag() { failed_ = true; }

  private:
    // takes the first task of the queue and runs it without the lock; false if there is none
    bool run_one(std::unique_lock<std::mutex> &lk)
    {
        if (tasks_.empty()) return false;
        Task t = std::move(tasks_.front());
        tasks_.pop_front();
        lk.unlock();
        t.fn();
        lk.lock();
        pending_--;
        if (t.batch) t.batch->left--;
        if (pending_ == 0 || (t.batch && t.batch->left == 0)) cv_done_.notify_all();
        return true;
    }
    void work()
    {
        cudaSetDevice(device_);
        std::unique_lock<std::mutex> lk(mu_);
        while (true) {
            cv_task_.wait(lk, [this] { return calls_ > 0; });
            calls_--;
            while (run_one(lk)) {
            }
            awake_--;
        }
    }
    struct Task {
        std::function<void()> fn;
        Batch *batch = nullptr;
    };
    int device_;
    std::vector<Slot> slots_;
    std::deque<int> free_;
    std::deque<Task> tasks_;
    std::vector<std::thread> workers_;     // live until the process exits
    std::mutex mu_;
    std::condition_variable cv_free_, cv_task_, cv_done_;
    int pending_ = 0, slabs_ = 0;
    size_t busy_bytes_ = 0;                // given since there was nothing to do
    size_t awake_ = 0, calls_ = 0;         // workers at work or called, calls not heard yet
    std::atomic<bool> failed_{false};
};

std::mutex g_pool_mu;
Pool *g_pool[64] = {nullptr};

Pool *pool()
{
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (!g_pool[d]) g_pool[d] = new Pool(d);
    return g_pool[d]->usable() ? g_pool[d] : nullptr;
}

// COMET_B200_STAGED_COPIES=0 leaves every copy to the driver; COMET_B200_STAGE_MIN_BYTES moves the size from
// which pageable copies are staged (both read at every call: they are test and tuning knobs)
bool staging_enabled()
{
    const char *e = getenv("COMET_B200_STAGED_COPIES");
    return !(e && e[0] == '0');
}

size_t stage_min()
{
    const char *e = getenv("COMET_B200_STAGE_MIN_BYTES");
    if (e) {
        const long long v = atoll(e);
        if (v >= 0) return (size_t)v;
    }
    return STAGE_MIN_DEFAULT;
}

// rows x row_bytes, host rows `host_pitch` apart, device rows `dev_pitch` apart (a 1-D copy is one row cut
// into chunk-sized pieces by the callers below)
struct Piece {
    char *host;
    char *dev;
    size_t rows, row_bytes, host_pitch, dev_pitch;
};

void copy_rows(char *dst, size_t dpitch, const char *src, size_t spitch, size_t row_bytes, size_t rows)
{
    if (dpitch == row_bytes && spitch == row_bytes) {
        memcpy(dst, src, row_bytes * rows);
        return;
    }
    for (size_t r = 0; r < rows; r++) memcpy(dst + r * dpitch, src + r * spitch, row_bytes);
}

thread_local bool g_scope = false;        // between uploads_begin() and uploads_join()
thread_local Batch g_scope_batch;
thread_local Pool *g_scope_pool = nullptr;

int staged(Pool *p, bool to_device, const Piece &pc, cudaStream_t st)
{
    Batch own;
    Batch *batch = to_device ? (g_scope ? &g_scope_batch : &own) : nullptr;
    if (to_device && g_scope) g_scope_pool = p;
    const size_t total = pc.rows * pc.row_bytes;
    p->grow((int)(1 + total / (CHUNK * SLAB_CHUNKS)));
    // pieces small enough that every thread gets some, large enough to be worth a thread
    size_t piece = total / (2 * (size_t)p->threads());
    piece = (piece + 4095) & ~(size_t)4095;
    piece = piece < PIECE_MIN ? PIECE_MIN : (piece > CHUNK ? CHUNK : piece);
    // a chunk carries whole rows (packed), or a part of one row when a row is longer than a piece
    const size_t rows_per_chunk = pc.row_bytes >= piece ? 1 : piece / pc.row_bytes;
    for (size_t r0 = 0; r0 < pc.rows; r0 += rows_per_chunk) {
        const size_t nr = pc.rows - r0 < rows_per_chunk ? pc.rows - r0 : rows_per_chunk;
        for (size_t b0 = 0; b0 < pc.row_bytes; b0 += piece) {
            const size_t nb = pc.row_bytes - b0 < piece ? pc.row_bytes - b0 : piece;
            const int si = p->acquire();
            Slot &s = p->slot(si);
            char *host = pc.host + r0 * pc.host_pitch + b0;
            char *dev = pc.dev + r0 * pc.dev_pitch + b0;
            const size_t host_pitch = pc.host_pitch, dev_pitch = pc.dev_pitch;
            const bool flat = nr == 1 || dev_pitch == nb;      // one run of bytes on the device
            if (to_device) {
                p->submit([p, si, host, dev, nr, nb, host_pitch, dev_pitch, flat, st] {
                    Slot &sl = p->slot(si);
                    fill_chunk(sl.buf, host, host_pitch, nb, nr);
                    cudaError_t e = flat ? cudaMemcpyAsync(dev, sl.buf, nb * nr, cudaMemcpyHostToDevice, st)
                                         : cudaMemcpy2DAsync(dev, dev_pitch, sl.buf, nb, nb, nr, cudaMemcpyHostToDevice, st);
                    if (e == cudaSuccess) e = cudaEventRecord(sl.ev, st);
                    if (e != cudaSuccess) p->fail_flag();
                    sl.dma_pending = true;
                    p->release(si);
                }, nb * nr, batch);
            } else {
                cudaError_t e = flat ? cudaMemcpyAsync(s.buf, dev, nb * nr, cudaMemcpyDeviceToHost, st)
                                     : cudaMemcpy2DAsync(s.buf, nb, dev, dev_pitch, nb, nr, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) {
                    e = cudaEventRecord(s.ev, st);
                    if (e != cudaSuccess) cudaStreamSynchronize(st);        // the copy into the chunk
                }
                if (e != cudaSuccess) {
                    p->release(si);
                    return fail("staged copy to the host failed: %s", cudaGetErrorString(e));
                }
                p->submit([p, si, host, nr, nb, host_pitch] {
                    Slot &sl = p->slot(si);
                    if (cudaEventSynchronize(sl.ev) != cudaSuccess) p->fail_flag();
                    else copy_rows(host, host_pitch, sl.buf, nb, nb, nr);
                    p->release(si);
                }, nb * nr);
            }
        }
    }
    // uploads: the host array must have been read, and every chunk's DMA enqueued, before the caller goes on
    if (batch == &own) {
        p->wait(&own);
        if (p->take_failure()) return fail("staged copy to the device failed");
    }
    return 0;
}

}  // namespace

bool host_is_pageable(const void *p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

int h2d_2d(void *dev, size_t dev_pitch, const void *host, size_t host_pitch, size_t row_bytes, size_t rows,
           cudaStream_t st)
{
    if (rows == 0 || row_bytes == 0) return 0;
    Pool *p = nullptr;
    if (staging_enabled() && row_bytes * rows >= stage_min() && host_is_pageable(host)) p = pool();
    if (!p) {
        CB_CUDA(cudaMemcpy2DAsync(dev, dev_pitch, host, host_pitch, row_bytes, rows, cudaMemcpyHostToDevice, st));
        return 0;
    }
    Piece pc = {(char *)host, (char *)dev, rows, row_bytes, host_pitch, dev_pitch};
    return staged(p, true, pc, st);
}

int d2h_2d(void *host, size_t host_pitch, const void *dev, size_t dev_pitch, size_t row_bytes, size_t rows,
           cudaStream_t st)
{
    if (rows == 0 || row_bytes == 0) return 0;
    Pool *p = nullptr;
    if (staging_enabled() && row_bytes * rows >= stage_min() && host_is_pageable(host)) p = pool();
    if (!p) {
        CB_CUDA(cudaMemcpy2DAsync(host, host_pitch, dev, dev_pitch, row_bytes, rows, cudaMemcpyDeviceToHost, st));
        return 0;
    }
    Piece pc = {(char *)host, (char *)dev, rows, row_bytes, host_pitch, dev_pitch};
    return staged(p, false, pc, st);
}

int h2d(void *dev, const void *host, size_t bytes, cudaStream_t st)
{
    if (bytes == 0) return 0;
    if (bytes < stage_min() || !staging_enabled() || !host_is_pageable(host)) {
        CB_CUDA(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, st));
        return 0;
    }
    return h2d_2d(dev, bytes, host, bytes, bytes, 1, st);
}

int d2h(void *host, const void *dev, size_t bytes, cudaStream_t st)
{
    if (bytes == 0) return 0;
    if (bytes < stage_min() || !staging_enabled() || !host_is_pageable(host)) {
        CB_CUDA(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st));
        return 0;
    }
    return d2h_2d(host, bytes, dev, bytes, bytes, 1, st);
}

static std::mutex g_words_mu;
static std::vector<void *> g_words;

PinnedWords::PinnedWords() : p(nullptr)
{
    std::lock_guard<std::mutex> lk(g_words_mu);
    if (g_words.empty()) {
        char *page = nullptr;
        if (cudaHostAlloc((void **)&page, 4096, cudaHostAllocPortable) != cudaSuccess) return;
        for (int i = 0; i < 64; i++) g_words.push_back(page + 64 * i);
    }
    p = g_words.back();
    g_words.pop_back();
}

PinnedWords::~PinnedWords()
{
    if (!p) return;
    std::lock_guard<std::mutex> lk(g_words_mu);
    g_words.push_back(p);
}

bool uploads_begin()
{
    if (g_scope) return false;
    g_scope = true;
    g_scope_pool = nullptr;
    return true;
}

int uploads_join()
{
    g_scope = false;
    Pool *p = g_scope_pool;
    g_scope_pool = nullptr;
    if (!p) return 0;
    p->wait(&g_scope_batch);
    return p->take_failure() ? fail("staged copy to the device failed") : 0;
}

int copies_drain()
{
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= 64) return 0;
    Pool *p;
    {
        std::lock_guard<std::mutex> lk(g_pool_mu);
        p = g_pool[d];
    }
    if (p && p->drain()) return fail("a staged copy between host and device failed");
    return 0;
}

}  // namespace cb200
