// The pool of page-locked result blocks never makes a caller wait, also while blocks are given up for others.
#include "fake_cuda.hpp"

#include <sys/wait.h>
#include <unistd.h>

#include "../../include/comet_b200.h"

// a machine of 64 MB: the pool keeps 8 MB at most
extern "C" long sysconf(int name) { return name == _SC_PHYS_PAGES ? 16384 : name == _SC_PAGESIZE ? 4096 : -1; }

namespace cb200 { void result_release_kept(); }

using Clock = std::chrono::steady_clock;

#define CHECK(cond, ...)                         \
    do {                                         \
        if (!(cond)) {                           \
            printf(__VA_ARGS__);                 \
            printf("\n");                        \
            fflush(stdout);                      \
            _Exit(1);                            \
        }                                        \
    } while (0)

static const int SLOW_MS = 400;
static double worst = 0.0;

template <typename F>
static auto timed(F f)
{
    const auto t = Clock::now();
    auto r = f();
    const double ms = std::chrono::duration<double, std::milli>(Clock::now() - t).count();
    if (ms > worst) worst = ms;
    return r;
}

// asks until the background thread has made a block
static void *block(int64_t bytes)
{
    for (int i = 0; i < 400; i++) {
        if (void *p = timed([&] { return comet_b200_result_alloc(bytes); })) return p;
        std::this_thread::sleep_for(std::chrono::milliseconds(5));
    }
    return nullptr;
}

int main()
{
    const int64_t MB = 1 << 20;
    CHECK(!comet_b200_result_alloc(4 * MB), "a first request is answered with a block");
    void *a = block(4 * MB), *b = block(4 * MB);
    CHECK(a && b && a != b, "no two blocks of 4 MB");
    comet_b200_result_free(a);
    CHECK(comet_b200_result_alloc(4 * MB) == a, "a block given back is not taken again");
    // a forked child has a copy of the block, as of any other array
    memset(a, 1, 4 * MB);
    const pid_t child = fork();
    if (child == 0) {
        const bool same = ((char *)a)[5 * 4096] == 1;
        memset(a, 2, 4 * MB);
        _exit(same ? 0 : 1);
    }
    int status = 0;
    CHECK(waitpid(child, &status, 0) == child && WIFEXITED(status) && WEXITSTATUS(status) == 0, "a child cannot read a block");
    CHECK(((char *)a)[5 * 4096] == 1, "a child's writes are seen by its parent");
    comet_b200_result_free(a);
    comet_b200_result_free(b);
    // 8 MB are kept; a block of another size takes their place
    fake::free_ms = SLOW_MS;
    std::atomic<bool> stop{false};
    double other = 0.0;
    std::thread t([&] {                                  // another thread's requests meanwhile
        while (!stop) {
            const auto at = Clock::now();
            comet_b200_result_alloc(9 * MB);              // more than the pool may hold: refused
            other = std::max(other, std::chrono::duration<double, std::milli>(Clock::now() - at).count());
            std::this_thread::sleep_for(std::chrono::milliseconds(1));
        }
    });
    void *c = block(6 * MB);
    stop = true;
    t.join();
    CHECK(c, "no block of 6 MB");
    CHECK(fake::frees == 2, "%d blocks were given up", fake::frees.load());
    CHECK(worst < SLOW_MS / 2 && other < SLOW_MS / 2, "a request took %.0f ms, another thread's %.0f", worst, other);
    // blocks in use are never given up
    for (int i = 0; i < 20; i++) {
        CHECK(!comet_b200_result_alloc(5 * MB), "more than 8 MB are held");
        std::this_thread::sleep_for(std::chrono::milliseconds(5));
    }
    comet_b200_result_free(c);
    cb200::result_release_kept();
    CHECK(fake::frees == 3, "a kept block was not given back");
    printf("ok\n");
    fflush(stdout);
    _Exit(0);
}
