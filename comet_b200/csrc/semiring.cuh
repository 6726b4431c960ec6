#pragma once
#include "common.cuh"

namespace cb200 {

// --------------------------------------------------------------------------
// Semiring arithmetic (codes of include/comet_b200.h).  The second operator
// combines A[i,k] and B[k,j]; the first one folds the products of one output.
// "any" is only offered with "pair", where every product is 1, so it can share
// the min fold.
// --------------------------------------------------------------------------
__device__ __forceinline__ double sr_combine(int semi, double a, double b)
{
    switch (semi) {
    case COMET_B200_PLUS_PAIR: case COMET_B200_ANY_PAIR: return 1.0;
    case COMET_B200_PLUS_FIRST: case COMET_B200_MIN_FIRST: return a;
    case COMET_B200_PLUS_SECOND: case COMET_B200_MIN_SECOND: return b;
    case COMET_B200_MIN_PLUS: return a + b;
    default: return a * b;
    }
}

__host__ __device__ __forceinline__ bool sr_is_min(int semi) { return semi >= COMET_B200_MIN_PLUS; }

__device__ __forceinline__ double sr_identity(int semi) { return sr_is_min(semi) ? __longlong_as_double(0x7ff0000000000000LL) : 0.0; }

// min fold on an f64 in shared or global memory (there is no native one)
__device__ __forceinline__ void atomic_min_f64(double *addr, double v)
{
    unsigned long long *a = (unsigned long long *)addr;
    unsigned long long old = *a;
    while (v < __longlong_as_double((long long)old)) {
        const unsigned long long assumed = old;
        old = atomicCAS(a, assumed, (unsigned long long)__double_as_longlong(v));
        if (old == assumed) break;
    }
}

__device__ __forceinline__ double sr_fold_value(int semi, double a, double b)
{
    return sr_is_min(semi) ? (b < a ? b : a) : a + b;
}

__device__ __forceinline__ void sr_fold(int semi, double *addr, double v)
{
    if (sr_is_min(semi)) atomic_min_f64(addr, v);
    else atomicAdd(addr, v);
}

}  // namespace cb200
