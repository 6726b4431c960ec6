// A stand-in for the CUDA runtime under objects built by nvcc, so that what the host side allocates and launches can be checked
// without a GPU.  "Device" memory is host memory; a launch runs nothing, but is shown to the check, by the kernel's name, with its arguments.
#pragma once
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <functional>
#include <map>
#include <string>
#include <vector>

#include "../../comet_b200/csrc/common.cuh"

namespace fake {

struct Launch {
    std::string name;
    dim3 grid, block;
};
static std::map<const void *, std::string> &names()
{
    static std::map<const void *, std::string> &n = *new std::map<const void *, std::string>;      // objects register before main
    return n;
}
static std::vector<Launch> launches;
static std::function<void(const std::string &, void **)> on_launch;
static size_t pool_room = ~(size_t)0;               // what one cudaMallocAsync may ask for

static int launched(const char *name)
{
    int n = 0;
    for (auto &l : launches) n += l.name.find(name) != std::string::npos;
    return n;
}
static cudaError_t launch(const void *f, dim3 grid, dim3 block, void **args)
{
    launches.push_back({names()[f], grid, block});
    if (on_launch) on_launch(launches.back().name, args);
    return cudaSuccess;
}

}  // namespace fake

namespace cb200 {
static char g_err[1024] = "";
int fail(const char *fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return 1;
}
void clear_error() { g_err[0] = 0; }
int sm_count() { return 148; }
}  // namespace cb200

extern "C" {

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *)
{
    fake::names()[host] = name;
}
static struct { dim3 grid, block; size_t smem; void *stream; } fake_config;
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *st)
{
    fake_config = {grid, block, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *st)
{
    *grid = fake_config.grid;
    *block = fake_config.block;
    *smem = fake_config.smem;
    *(void **)st = fake_config.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3 block, void **args, size_t, cudaStream_t) { return fake::launch(f, grid, block, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **args) { return fake::launch(f, c->gridDim, c->blockDim, args); }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "made to fail"; }
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t)
{
    *p = n > fake::pool_room ? nullptr : malloc(n);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(dst, src, n); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }

}
