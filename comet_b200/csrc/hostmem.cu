// Page-locked memory for results that the library's callers get as new arrays (the Python layer's return values).
//
// A new 64 MB array costs its user 37 ms of page faults on one core (4 KB pages; 2.5 ms on eight cores with large
// ones) before or while the result is copied into it, and a pageable destination is staged on top; the DMA engine
// writes a page-locked one in 1.2 ms.  Page-locking itself takes 11 ms per 64 MB, so blocks are kept for the next
// result of about the same size.  A block is private memory that is page-locked afterwards, not cudaHostAlloc's: that is
// mapped shared, so that a forked child would write to its parent's results (and takes 24 ms per 64 MB).  The pool never makes a caller wait: a request it has no block for is answered with
// null (the caller uses ordinary memory), and from the second such request of a size on a background thread
// page-locks one more block.  Blocks in use and kept together stay below 1 GiB and an eighth of the machine's memory;
// beyond that kept blocks of other sizes are given up, which is the background thread's work too (it waits for
// the device), and then requests are refused.  comet_b200_release_scratch() gives back every block that is not in use.
#include <sys/mman.h>
#include <unistd.h>

#include <map>
#include <mutex>
#include <system_error>
#include <thread>
#include <unordered_map>
#include <vector>

#include "common.cuh"

namespace cb200 {

namespace {

struct Sizes {
    std::vector<void *> kept;
    int misses = 0;
};
// never destroyed: blocks may be given back while the process ends
std::mutex &g_mu = *new std::mutex;
std::map<size_t, Sizes> &g_sizes = *new std::map<size_t, Sizes>;
std::unordered_map<void *, size_t> &g_used = *new std::unordered_map<void *, size_t>;
size_t g_held = 0;                        // bytes in use, kept and being allocated
bool g_growing = false;
std::thread &g_grower = *new std::thread;

size_t limit()
{
    static const size_t bytes = [] {
        const long pages = sysconf(_SC_PHYS_PAGES), page = sysconf(_SC_PAGESIZE);
        const size_t eighth = pages > 0 && page > 0 ? (size_t)pages * (size_t)page / 8 : (size_t)1 << 28;
        return eighth < ((size_t)1 << 30) ? eighth : (size_t)1 << 30;
    }();
    return bytes;
}

// sizes are rounded up to whole pages and eight steps per power of two
size_t rounded(size_t bytes)
{
    static const size_t page = sysconf(_SC_PAGESIZE) > 0 ? (size_t)sysconf(_SC_PAGESIZE) : 4096;
    size_t step = page;
    while (step * 16 < bytes) step <<= 1;
    return (bytes + step - 1) / step * step;
}

// Page-locked memory of whole pages, large ones where they fit.
void *make_block(size_t size)
{
    const size_t large = (size_t)2 << 20, align = size >= large ? large : 0;
    char *m = (char *)mmap(nullptr, size + align, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (m == (char *)MAP_FAILED) return nullptr;
    char *p = align ? (char *)(((uintptr_t)m + align - 1) & ~(uintptr_t)(align - 1)) : m;
    if (p > m) munmap(m, p - m);
    if (m + align > p) munmap(p + size, m + align - p);
    if (align) madvise(p, size, MADV_HUGEPAGE);
    if (cudaHostRegister(p, size, cudaHostRegisterPortable) == cudaSuccess) return p;
    (void)cudaGetLastError();
    munmap(p, size);
    return nullptr;
}

void free_block(void *p, size_t size)
{
    cudaHostUnregister(p);
    munmap(p, size);
}

using Blocks = std::vector<std::pair<void *, size_t>>;

// gives blocks back that are on no list any more; without the lock
void give_back(const Blocks &blocks)
{
    if (blocks.empty()) return;
    size_t bytes = 0;
    for (const auto &b : blocks) {
        free_block(b.first, b.second);
        bytes += b.second;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    g_held -= bytes;
}

void grow(size_t size, int device, Blocks given_up)
{
    give_back(given_up);
    void *p = cudaSetDevice(device) == cudaSuccess ? make_block(size) : nullptr;
    std::lock_guard<std::mutex> lk(g_mu);
    if (p) g_sizes[size].kept.push_back(p);
    else g_held -= size;
    g_growing = false;                     // last: the lock's release is all that follows
}

}  // namespace

void result_release_kept()
{
    Blocks all;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        for (auto &s : g_sizes) {
            for (void *p : s.second.kept) all.emplace_back(p, s.first);
            s.second.kept.clear();
            s.second.misses = 0;
        }
    }
    give_back(all);
}

}  // namespace cb200

extern "C" void *comet_b200_result_alloc(int64_t bytes)
{
    using namespace cb200;
    if (bytes <= 0) return nullptr;
    const size_t size = rounded((size_t)bytes);
    std::lock_guard<std::mutex> lk(g_mu);
    Sizes &s = g_sizes[size];
    if (!s.kept.empty()) {
        void *p = s.kept.back();
        s.kept.pop_back();
        g_used[p] = size;
        return p;
    }
    if (++s.misses < 2 || g_growing || size > limit()) return nullptr;
    size_t kept = 0;
    for (const auto &o : g_sizes) kept += o.first * o.second.kept.size();
    int device = 0;
    if (g_held - kept + size > limit() || cudaGetDevice(&device) != cudaSuccess) return nullptr;
    // a process that ends waits for the block being made (registered after the CUDA runtime's own handler, so run before it)
    static const bool registered = std::atexit([] { if (g_grower.joinable()) g_grower.join(); }) == 0;
    if (!registered) return nullptr;
    if (g_grower.joinable()) g_grower.join();          // g_growing is false: it has ended, or is about to return
    Blocks given_up;                                   // they count as held until they are free
    size_t over = g_held + size > limit() ? g_held + size - limit() : 0;
    for (auto it = g_sizes.begin(); over && it != g_sizes.end(); ++it)
        while (over && !it->second.kept.empty()) {
            given_up.emplace_back(it->second.kept.back(), it->first);
            it->second.kept.pop_back();
            over = over > it->first ? over - it->first : 0;
        }
    try {
        g_grower = std::thread(grow, size, device, given_up);
        g_held += size;                                // it waits for the lock before it looks at either
        g_growing = true;
    } catch (const std::system_error &) {              // no thread to be had: everything stays as it was
        for (const auto &b : given_up) g_sizes[b.second].kept.push_back(b.first);
    }
    return nullptr;
}

extern "C" void comet_b200_result_free(void *p)
{
    using namespace cb200;
    if (!p) return;
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_used.find(p);
    if (it == g_used.end()) return;
    g_sizes[it->second].kept.push_back(p);
    g_used.erase(it);
}

extern "C" int64_t comet_b200_result_size(void *p)
{
    using namespace cb200;
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_used.find(p);
    return it == g_used.end() ? 0 : (int64_t)it->second;
}
