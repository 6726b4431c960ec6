// A stand-in for a thread block, so that kernels' own text can be compiled with g++ and watched by ThreadSanitizer: every thread of the
// block is a host thread.  Only barriers order memory; shuffles, votes, reductions and atomics exchange values and make the
// lanes wait for each other, but order nothing else, which is what CUDA promises.
#pragma once
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <functional>
#include <string>
#include <thread>
#include <type_traits>
#include <vector>

using std::max;
using std::min;

#define __global__ static
#define __device__
#define __host__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __shared__ static
#define __align__(n) __attribute__((aligned(n)))
#define CB_UNUSED __attribute__((unused))

struct int2 { int x, y; };
struct int4 { int x, y, z, w; };
struct uint4 { unsigned x, y, z, w; };
struct longlong2 { long long x, y; };
inline int2 make_int2(int x, int y) { return {x, y}; }
inline int4 make_int4(int x, int y, int z, int w) { return {x, y, z, w}; }
inline uint4 make_uint4(unsigned x, unsigned y, unsigned z, unsigned w) { return {x, y, z, w}; }

struct Dim { unsigned x, y, z; };
static thread_local Dim threadIdx, blockIdx;
static Dim blockDim, gridDim;

namespace fake {

struct Barrier {
    std::atomic<unsigned long long> arrived{0};
    void wait(unsigned long long upto)
    {
        arrived.fetch_add(1, std::memory_order_acq_rel);
        while (arrived.load(std::memory_order_acquire) < upto) std::this_thread::yield();
    }
};
struct Warp {
    std::atomic<unsigned long long> slot[2][32], step[32];
    Barrier barrier;
};
static std::vector<Warp> *warps;
static Barrier *block;
static thread_local unsigned long long steps, warp_waits, block_waits;

inline Warp &own() { return (*warps)[threadIdx.x >> 5]; }
inline unsigned lane() { return threadIdx.x & 31; }

// all lanes' values; the next call may not begin to write before every lane has read, hence two sets of slots
inline const std::atomic<unsigned long long> *exchange(unsigned long long v)
{
    Warp &w = own();
    const unsigned long long now = ++steps;
    w.slot[now & 1][lane()].store(v, std::memory_order_relaxed);
    w.step[lane()].store(now, std::memory_order_relaxed);
    for (int l = 0; l < 32; l++)
        while (w.step[l].load(std::memory_order_relaxed) < now) std::this_thread::yield();
    return w.slot[now & 1];
}
template <typename T>
unsigned long long bits_of(T v)
{
    unsigned long long b = 0;
    memcpy(&b, &v, sizeof(T));
    return b;
}
template <typename T>
T from_bits(unsigned long long b)
{
    T v;
    memcpy(&v, &b, sizeof(T));
    return v;
}

// runs one block (number b of n, in row y) of `threads` threads
inline void run_block(unsigned threads, unsigned b, unsigned n, const std::function<void()> &kernel, unsigned y = 0)
{
    std::vector<Warp> w(threads / 32);
    for (auto &x : w)
        for (int l = 0; l < 32; l++) x.step[l] = 0;
    Barrier bar;
    warps = &w;
    block = &bar;
    blockDim = {threads, 1, 1};
    gridDim = {n, 1, 1};
    std::vector<std::thread> t;
    for (unsigned i = 0; i < threads; i++)
        t.emplace_back([&, i] {
            threadIdx = {i, 0, 0};
            blockIdx = {b, y, 0};
            kernel();
        });
    for (auto &x : t) x.join();
}

}  // namespace fake

inline void __syncwarp(unsigned = 0xffffffffu) { fake::own().barrier.wait(32 * ++fake::warp_waits); }
inline void __syncthreads() { fake::block->wait(blockDim.x * ++fake::block_waits); }
inline void wait_for_previous() {}

template <typename T> T __shfl_sync(unsigned, T v, int src, int = 32)
{
    return fake::from_bits<T>(fake::exchange(fake::bits_of(v))[src & 31].load(std::memory_order_relaxed));
}
template <typename T> T __shfl_up_sync(unsigned, T v, int d)
{
    const int l = (int)fake::lane() - d;
    return fake::from_bits<T>(fake::exchange(fake::bits_of(v))[l < 0 ? fake::lane() : l].load(std::memory_order_relaxed));
}
template <typename T> T __shfl_xor_sync(unsigned, T v, int d)
{
    return fake::from_bits<T>(fake::exchange(fake::bits_of(v))[fake::lane() ^ d].load(std::memory_order_relaxed));
}
inline double shfl_f64(double v, int src, int) { return __shfl_sync(0u, v, src); }
inline unsigned __ballot_sync(unsigned, bool v)
{
    auto *s = fake::exchange(v);
    unsigned m = 0;
    for (int l = 0; l < 32; l++) m |= (unsigned)(s[l].load(std::memory_order_relaxed) & 1) << l;
    return m;
}
inline bool __all_sync(unsigned, bool v) { return __ballot_sync(0, v) == 0xffffffffu; }
inline bool __any_sync(unsigned, bool v) { return __ballot_sync(0, v) != 0u; }
template <typename T, typename F> T fake_reduce(T v, F f)
{
    auto *s = fake::exchange(fake::bits_of(v));
    T r = fake::from_bits<T>(s[0].load(std::memory_order_relaxed));
    for (int l = 1; l < 32; l++) r = f(r, fake::from_bits<T>(s[l].load(std::memory_order_relaxed)));
    return r;
}
template <typename T> T __reduce_add_sync(unsigned, T v) { return fake_reduce(v, [](T a, T b) { return a + b; }); }
template <typename T> T __reduce_max_sync(unsigned, T v) { return fake_reduce(v, [](T a, T b) { return a > b ? a : b; }); }
template <typename T> T __reduce_min_sync(unsigned, T v) { return fake_reduce(v, [](T a, T b) { return a < b ? a : b; }); }

template <typename T, typename U> T atomicOr(T *p, U v) { return __atomic_fetch_or(p, (T)v, __ATOMIC_RELAXED); }
template <typename T, typename U> T atomicAdd(T *p, U v) { return __atomic_fetch_add(p, (T)v, __ATOMIC_RELAXED); }
inline double atomicAdd(double *p, double v)
{
    unsigned long long *a = (unsigned long long *)p, old = __atomic_load_n(a, __ATOMIC_RELAXED);
    while (!__atomic_compare_exchange_n(a, &old, fake::bits_of(fake::from_bits<double>(old) + v), false, __ATOMIC_RELAXED, __ATOMIC_RELAXED)) {}
    return fake::from_bits<double>(old);
}
template <typename T, typename U> T atomicExch(T *p, U v) { return __atomic_exchange_n(p, (T)v, __ATOMIC_RELAXED); }
template <typename T, typename U, typename V> T atomicCAS(T *p, U cmp, V v)
{
    T old = (T)cmp;
    __atomic_compare_exchange_n(p, &old, (T)v, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED);
    return old;
}
template <typename T, typename U> T atomicMax(T *p, U v)
{
    T old = __atomic_load_n(p, __ATOMIC_RELAXED);
    while (old < (T)v && !__atomic_compare_exchange_n(p, &old, (T)v, false, __ATOMIC_RELAXED, __ATOMIC_RELAXED)) {}
    return old;
}

inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(int v) { return __builtin_ffs(v); }
inline int __clz(int v) { return v ? __builtin_clz((unsigned)v) : 32; }
template <typename T> T __ldg(const T *p) { return *p; }
template <typename T> T __ldcs(const T *p) { return *p; }
template <typename T> T __ldcg(const T *p) { return *p; }
template <typename T, typename U> void __stcs(T *p, U v) { *p = (T)v; }
