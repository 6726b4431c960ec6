// A process that may not start another thread: nothing is thrown through the C entry points, copies are carried out by the
// calling thread, and the result pool makes blocks again once it can.
#include "fake_cuda.hpp"

#include <dlfcn.h>
#include <errno.h>

#include <vector>

#include "../../comet_b200/csrc/hostcopy.cuh"
#include "../../include/comet_b200.h"

extern "C" int pthread_create(pthread_t *t, const pthread_attr_t *a, void *(*f)(void *), void *x)
{
    using Fn = int (*)(pthread_t *, const pthread_attr_t *, void *(*)(void *), void *);
    static const Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
    if (fake::fail_thread) return EAGAIN;
    return real(t, a, f, x);
}

#define CHECK(cond, ...)                         \
    do {                                         \
        if (!(cond)) {                           \
            printf(__VA_ARGS__);                 \
            printf("\n");                        \
            fflush(stdout);                      \
            _Exit(1);                            \
        }                                        \
    } while (0)

int main()
{
    cudaStream_t st = cb200::lib_stream();              // its thread stands for the device
    fake::fail_thread = 1;
    const size_t n = (size_t)6 << 20;                   // more pieces than one
    std::vector<char> src(n), back(n, 0), dev(n, 0);
    for (size_t i = 0; i < n; i++) src[i] = (char)(i * 7 + i / 4096);
    CHECK(cb200::uploads_begin(), "an upload scope is open");
    CHECK(cb200::h2d(dev.data(), src.data(), n, st) == 0 && cb200::uploads_join() == 0, "the upload failed");
    CHECK(cb200::d2h(back.data(), dev.data(), n, st) == 0, "the download failed");
    cudaStreamSynchronize(st);
    CHECK(cb200::copies_drain() == 0 && src == back, "the bytes differ");
    for (int i = 0; i < 4; i++) CHECK(!comet_b200_result_alloc(1 << 20), "a block without a thread that makes it");
    fake::fail_thread = 0;
    void *p = nullptr;
    for (int i = 0; i < 400 && !p; i++) {
        p = comet_b200_result_alloc(1 << 20);
        std::this_thread::sleep_for(std::chrono::milliseconds(5));
    }
    CHECK(p, "no block");
    comet_b200_result_free(p);
    printf("ok\n");
    fflush(stdout);
    _Exit(0);
}
