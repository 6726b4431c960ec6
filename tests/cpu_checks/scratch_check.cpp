// Scratch memory on a device with little of it: what a call can do without is refused without an error, grows with head-room, and is given
// back when another call finds no room, but not while it is in use.
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>

#include <map>

#include "../../comet_b200/csrc/common.cuh"

static size_t room = 1 << 20, used = 0;
static int mallocs = 0, fail_sync = 0;
static cudaError_t last = cudaSuccess;
static std::map<void *, size_t> blocks;
static cudaError_t set(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaMalloc(void **p, size_t n)
{
    mallocs++;
    if (used + n > room) return set(cudaErrorMemoryAllocation);
    *p = malloc(n);
    used += n;
    blocks[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    used -= blocks[p];
    blocks.erase(p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return set(fail_sync && fail_sync-- == 1 ? cudaErrorUnknown : cudaSuccess); }
}
namespace cb200 { void result_release_kept() {} }

#define CHECK(cond)                                          \
    do {                                                     \
        if (!(cond)) {                                       \
            printf("line %d: %s\n", __LINE__, #cond);        \
            return 1;                                        \
        }                                                    \
    } while (0)

using namespace cb200;

int main()
{
    comet_b200_set_error_mode(1);
    void *p = nullptr;
    {
        ScratchIfRoom a;                                     // fits, grows slowly: two allocations in all
        for (size_t n = 100000; n <= 112000; n += 1000) {
            ScratchIfRoom s;
            s.take(SLOT_TRIANGLES, n);
            CHECK(s.p);
        }
        CHECK(mallocs == 1);
        a.take(SLOT_TRIANGLES, 2 << 20);                     // does not
        CHECK(!a.p && last == cudaSuccess && used == 0);
        ScratchIfRoom b;                                     // exactly, without head-room
        b.take(SLOT_TRIANGLES, 1 << 20);
        CHECK(b.p && used == 1 << 20);
        CHECK(scratch(SLOT_MISC, 300, &p) != 0);             // in use: stays
        CHECK(used == 1 << 20);
        cudaGetLastError();
    }
    CHECK(scratch(SLOT_MISC, 300, &p) == 0 && used == 512);  // no longer
    {
        ScratchIfRoom s;
        s.take(SLOT_TRIANGLES, 1000);
        CHECK(s.p);
    }
    const size_t before = used;
    fail_sync = 1;
    ScratchIfRoom s;
    s.take(SLOT_TRIANGLES, 100000);                          // the old buffer cannot be released: nothing leaks, no error stays
    CHECK(!s.p && last == cudaSuccess && used == before);
    printf("ok\n");
    return 0;
}
