// Long rows of C = A*B when B has long rows itself (spgemm.cu, bin 2 without a mask).
//
// In a power-law product nearly all of the work comes from a few rows of B: R-MAT scale 18, 16 entries per row, squared has
// 2.93 G products, 88 % of them with the 988 rows of 512 entries and more.  Prepared once per product:
//   columns   B's columns are renumbered to those that B stores, in order (scale 18: 148,500 of 262,144), so that a row's
//             bitmap, its ranks and the walk over them shrink by as much
//   bitmaps   of those rows of B ("hubs"): the symbolic call ORs them into a row's bitmap in registers, 128 bits a load,
//             instead of marking their columns bit by bit with atomics (5.3 -> 3.7 ms, 3.3 with four CTAs an SM).  The line of 512 entries: 256 6.1 ms,
//             384 3.8, 768 3.8, 1024 4.1; on scale 15 0.30, 0.27 (512: 0.27), 0.37, 0.37.  With wide bitmaps an OR takes longer than the
//             marks of 512 entries, hence at least an eighth of an entry per word.
// Tried and not kept: sums by rank in shared memory, a range of columns per warp and the part of every hub that falls into it
// added without atomics.  The parts are too short (13 entries with 512 accumulators a warp, and fewer warps with more): 21.5 ms
// against 20.1 for the atomics in L2 at the time.
#pragma once
#include "common.cuh"
#include "semiring.cuh"
#include "stream.cuh"

namespace cb200 {

static const int HUB_MIN_ENTRIES = 512;
// Products per word of the rows' bitmaps from which on long rows, and columns of which between 5/8 and 7/8 are stored, are worth it where the
// numeric kernel gains no CTA on an SM: coordinates cost a look-up each, which few products pay for.  R-MAT scale 15 squared has 22 (70 % stored,
// both calls 1316 us renumbered, 1430 not); 12,351 rows of 13,000 products in 791,000 columns, 74 % stored, 0.5 (4199 and 3951); min-plus, 115,713
// rows of 1900 in 268,835 columns, 75 %, 0.2 (7760 and 7060); long rows in columns that keep their numbers, 3300 rows of 13,200 in 800,000 columns,
// 0.5 (with bitmaps of them 1550, without 1250).
static const int HUB_PRODUCTS = 4;
static const int HUB_MAX_WORDS = 25600;             // with their ranks, what bin 2 holds in shared memory
static const int64_t HUB_MAX_COLS = (int64_t)1 << 23;
static const size_t HUB_MEMORY = (size_t)128 << 20; // bitmaps of all hubs

struct HubPrep {             // filled on the device, read by the host
    unsigned ncols;          // columns that B stores
    unsigned pad;
    long long nrows_b;       // rows of B that A can name
    long long longest;       // entries of the longest of them
    long long products;      // of A and B
};

struct Hubs {
    void *mem, *mem2;
    int words, stride;       // words of a bitmap, rounded up to a multiple of 4: `stride`
    unsigned cap;            // hubs there is room for
    int64_t nrows_b;
    int32_t *crd;            // B's columns, renumbered unless B stores nearly all of them
    int32_t *colmap;         // their numbers in B (null: the same)
    uint32_t *present;
    int32_t *before;
    HubPrep *prep;
    unsigned *count;         // hubs found (more than cap: the others are ordinary rows)
    int32_t *id;             // of a row of B: number of the hub, or -1
    uint32_t *bm;            // hub -> bitmap, `stride` words each
};

#ifdef __CUDACC__

// Columns that B stores (a bit each), the largest row that A names, the longest, and the number of products.  SMEM: the bits are collected per CTA, so that the hub
// columns' words are not a queue for the whole chip.
template <bool SMEM>
__global__ void __launch_bounds__(1024)
hub_present_kernel(int64_t nnz_b, const int32_t *__restrict__ bcrd, int64_t words, uint32_t *__restrict__ present, int64_t nrows,
                   const int64_t *__restrict__ apos, const int64_t *__restrict__ acrd, const int64_t *__restrict__ bpos,
                   HubPrep *prep)
{
    extern __shared__ uint32_t s_bits[];
    if (SMEM) {
        for (int64_t w = threadIdx.x; w < words; w += blockDim.x) s_bits[w] = 0;
        __syncthreads();
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t q = t0; q < nnz_b; q += stride) {
        const int32_t j = bcrd[q];
        const uint32_t bit = 1u << (j & 31);
        if (SMEM) {
            if (!(s_bits[j >> 5] & bit)) atomicOr(&s_bits[j >> 5], bit);
        } else {
            if (!(__ldcg(present + (j >> 5)) & bit)) atomicOr(present + (j >> 5), bit);
        }
    }
    const int64_t nnz_a = apos[nrows];
    long long top = 0, longest = 0, products = 0;
    for (int64_t p = t0; p < nnz_a; p += stride) {
        const long long k = acrd[p] + 1, len = bpos[k] - bpos[k - 1];
        top = k > top ? k : top;
        longest = len > longest ? len : longest;
        products += len;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long v = __shfl_xor_sync(0xffffffffu, top, o);
        top = v > top ? v : top;
        const long long l = __shfl_xor_sync(0xffffffffu, longest, o);
        longest = l > longest ? l : longest;
        products += __shfl_xor_sync(0xffffffffu, products, o);
    }
    if ((threadIdx.x & 31) == 0 && top) {
        atomicMax(&prep->nrows_b, top);
        atomicMax(&prep->longest, longest);
        atomicAdd((unsigned long long *)&prep->products, (unsigned long long)products);
    }
    if (SMEM) {
        __syncthreads();
        for (int64_t w = threadIdx.x; w < words; w += blockDim.x) {
            const uint32_t v = s_bits[w];
            if (v) atomicOr(present + w, v);
        }
    }
}

// before[w] = stored columns before word w; one CTA.
__global__ void __launch_bounds__(1024)
hub_before_kernel(int64_t words, const uint32_t *__restrict__ present, int32_t *__restrict__ before, HubPrep *prep)
{
    __shared__ int s_sum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int carry = 0;
    for (int64_t base = 0; base < words; base += 4096) {
        int c[4], incl[4];
        int mine = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t w = base + 4 * threadIdx.x + i;
            c[i] = w < words ? __popc(present[w]) : 0;
            incl[i] = mine;
            mine += c[i];
        }
        int sum = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        if (lane == 31) s_sum[warp] = sum;
        __syncthreads();
        int run = carry + sum - mine, total = 0;
        for (int i = 0; i < 32; i++) {
            if (i < warp) run += s_sum[i];
            total += s_sum[i];
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t w = base + 4 * threadIdx.x + i;
            if (w < words) before[w] = run + incl[i];
        }
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) prep->ncols = (unsigned)carry;
}

// the new numbers of B's entries, and the columns they stand for
__global__ void __launch_bounds__(256)
hub_renumber_kernel(int64_t nnz_b, const int32_t *__restrict__ bcrd, int64_t words, const uint32_t *__restrict__ present,
                    const int32_t *__restrict__ before, int32_t *__restrict__ crd, int32_t *__restrict__ colmap)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t q = t0; q < nnz_b; q += stride) {
        const int32_t j = bcrd[q];
        crd[q] = before[j >> 5] + __popc(present[j >> 5] & ((1u << (j & 31)) - 1u));
    }
    for (int64_t w = t0; w < words; w += stride) {
        uint32_t v = present[w];
        for (int32_t at = before[w]; v; v &= v - 1, at++) colmap[at] = (int32_t)(w * 32 + __ffs(v) - 1);
    }
}

__global__ void __launch_bounds__(256)
hub_find_kernel(int64_t nrows_b, const int64_t *__restrict__ bpos, int64_t least, unsigned cap, unsigned *count,
                int32_t *__restrict__ id, int32_t *__restrict__ rows)
{
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nrows_b) return;
    int32_t h = -1;
    if (bpos[k + 1] - bpos[k] >= least) {
        const unsigned at = atomicAdd(count, 1u);
        if (at < cap) {
            h = (int32_t)at;
            rows[at] = (int32_t)k;
        }
    }
    id[k] = h;
}

// a CTA per hub: its bitmap
__global__ void __launch_bounds__(512)
hub_build_kernel(const unsigned *__restrict__ count, unsigned cap, const int32_t *__restrict__ rows,
                 const int64_t *__restrict__ bpos, const int32_t *__restrict__ crd, int stride, uint32_t *__restrict__ bm)
{
    extern __shared__ uint32_t s_bits[];
    const unsigned n = min(*count, cap);
    for (unsigned h = blockIdx.x; h < n; h += gridDim.x) {
        const int64_t s = bpos[rows[h]], e = bpos[rows[h] + 1];
        for (int w = threadIdx.x; w < stride; w += 512) s_bits[w] = 0;
        __syncthreads();
        for (int64_t q = s + threadIdx.x; q < e; q += 512) atomicOr(&s_bits[crd[q] >> 5], 1u << (crd[q] & 31));
        __syncthreads();
        for (int w = threadIdx.x; w < stride; w += 512) bm[(size_t)h * stride + w] = s_bits[w];
        __syncthreads();
    }
}

#endif

}  // namespace cb200
