// Gustavson SpGEMM  C = A*B  (optionally C<M,push> = A*B), all CSR, f64 / i64,
// as a symbolic call (fills C.pos) and a numeric call (fills C.crd sorted, C.val).
//
// Rows are binned by an upper bound on their number of distinct columns
// (sum of the lengths of the B rows they touch, capped by the mask row):
//   bin 0  no products                     -> empty row
//   bin 1  bound <= HASH_ROW_MAX           -> one warp per row.  The symbolic call counts distinct columns with a bitmap (few
//          columns) or a hash table in shared memory; the numeric call sorts column and place of the products in registers and adds equal
//          neighbours (with a mask: the hash table again, its keys sorted in registers)
//   bin 3  bound <= MID_ROW_MAX, no mask, not too many columns -> 128 or 256 threads per row, a bitmap over the columns of B and
//          sums by rank in shared memory
//   bin 2  everything else                 -> one CTA per row, a bitmap over the
//          columns of B in shared memory (global memory when B has too many
//          columns); popcounts give the row's count, prefix popcounts give each
//          column's rank, so crd comes out sorted with no sort and val[rank] is
//          accumulated in place with f64 atomics on the output row, which the
//          CTA has just zeroed and which therefore sits in L2.
//          From HUB_WORK bytes of bitmaps on, without a mask, B's long rows are prepared first (hubs.cuh).
// This mirrors COMET's workspace transformation (dense row workspace + mark
// array, sort of the touched columns) with a bit per column instead of a mark
// word per column, and replaces std::sort by ranking.
//
// The bitmaps of bin-2 rows found by the symbolic call are kept (when they fit
// a budget) so that the numeric call does not have to traverse the products a
// second time to rebuild them.
//
// Accumulation order inside a row is not fixed (atomics); structure (pos, crd)
// is exact and values agree with a sequential sum to rounding.
#include <mutex>
#include <type_traits>
#include <unordered_map>

#include "common.cuh"
#include "stream.cuh"
#include "hostcopy.cuh"
#include "hubs.cuh"
#include "masked.cuh"
#include "semiring.cuh"

namespace cb200 {

static const int HASH_ROW_MAX = 256;        // bound for bin 1
static const int HASH_SLOTS = 512;          // table size per warp with sums (load factor <= 0.5); twice that without
static const int HASH_WARPS = 4;            // warps per CTA in the hash kernels
static const int BM_THREADS = 512;          // CTA size of the bitmap kernels
static const size_t BM_SMEM_LIMIT = 200 * 1024;
static const size_t BM_STORE_BUDGET = (size_t)12 << 30;
static const size_t BM_STORE_SMALL = (size_t)64 << 20;
static const size_t HUB_WORK = (size_t)32 << 20;      // bytes of bitmaps of bin-2 rows from which on hubs.cuh takes them
// and bytes of them per entry of B: looking B over takes some 10 us per million entries, in vain where it has no long rows and stores nearly all
// of its columns. B of 8 M entries, bytes per entry and both calls without / with it: 9 560 / 700 us, 12 397 / 464, 25 714 / 789, 50 1959 / 2070.
// Where it pays there are 83 (20,000 rows of 300 times 300 of 8) and more.
static const size_t HUB_ENTRY = 64;

struct Plan {
    int kind;                // 0 = spgemm, 1 = elementwise CSR .* CSR
    int64_t nrows, ncols, nnz_b;
    const int64_t *apos, *acrd, *bpos, *bcrd, *mpos, *mcrd;
    const double *aval, *bval;
    int semi;                // semiring code
    int64_t *cpos;           // caller's array
    int64_t nnz_c;
    void *mem;               // owned device memory: the next five arrays
    unsigned *bin_counts;    // [3]
    int64_t *cnt;            // per-row distinct count
    int32_t *bcrd32;
    int32_t *list1, *list2, *list3;  // rows of bins 1, 2 and 3
    unsigned n1, n2, n3;
    uint32_t *bm_store;      // n2 * stride words (without hubs n2 * words), or null
    int words;
    Hubs *hubs;              // not null: bin 2 goes by hubs.cuh
    MaskedPlan *masked;      // not null: the product is formed by dot products over the mask
    cudaStream_t last;       // stream of the latest call on this plan: its arrays are released in that stream's order
};

static std::mutex g_plans_mu;
static std::unordered_map<int64_t, Plan *> g_plans;
static int64_t g_next_handle = 1;

static void plan_free(Plan *p, cudaStream_t st)
{
    if (!p) return;
    if (p->mem) cudaFreeAsync(p->mem, st);
    if (p->bm_store) cudaFreeAsync(p->bm_store, st);
    if (p->hubs) {
        if (p->hubs->mem) cudaFreeAsync(p->hubs->mem, st);
        if (p->hubs->mem2) cudaFreeAsync(p->hubs->mem2, st);
        delete p->hubs;
    }
    masked_free(p->masked, st);
    delete p;
}

static int pool_setup()
{
    static bool done[64] = {false};
    int d = 0;
    CB_CUDA(cudaGetDevice(&d));
    if (d >= 0 && d < 64 && !done[d]) {
        cudaMemPool_t pool;
        CB_CUDA(cudaDeviceGetDefaultMemPool(&pool, d));
        uint64_t keep = ~(uint64_t)0;   // keep freed blocks cached for the next call
        CB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        done[d] = true;
    }
    return 0;
}

template <typename T>
static int dev_alloc(T **p, size_t n, cudaStream_t st)
{
    if (n == 0) n = 1;
    cudaError_t e = cudaMallocAsync((void **)p, n * sizeof(T), st);
    if (e != cudaSuccess) {
        *p = nullptr;
        return fail("device allocation of %zu bytes failed: %s", n * sizeof(T), cudaGetErrorString(e));
    }
    return 0;
}

// --------------------------------------------------------------------------
// mask membership: is column j stored in the (ascending) mask row [ms, me)?
// --------------------------------------------------------------------------
__device__ __forceinline__ bool in_mask(const int64_t *__restrict__ mcrd, int64_t ms, int64_t me,
                                        int64_t j)
{
    while (ms < me) {
        int64_t mid = (ms + me) >> 1;
        int64_t v = mcrd[mid];
        if (v == j) return true;
        if (v < j) ms = mid + 1; else me = mid;
    }
    return false;
}

// --------------------------------------------------------------------------
// Binning: 8 lanes per row sum the lengths of the B rows it touches, 32 of them at a time, and stop when the sum has left
// bin 1: a row's bin does not depend on more, and the hub rows of a power-law matrix leave it at once (R-MAT scale 13, 59,000
// entries: 82 -> 6 us; scale 16 125 -> 9).  The CTAs behind those of the rows copy B's columns as 32-bit numbers.
// --------------------------------------------------------------------------
static const int BIN_THREADS = 256;
static const int BIN_PASS = BIN_THREADS / 8;            // rows at a time
static const int BIN_ROWS = BIN_PASS * 4;
static const int64_t BIN_LONG_ROW = 1024;
static const int64_t NARROW_PART = 4096;                // entries per CTA

__global__ void __launch_bounds__(BIN_THREADS)
bin_rows_kernel(int64_t nrows, int passes, unsigned row_ctas, const int64_t *__restrict__ apos, const int64_t *__restrict__ acrd,
                const int64_t *__restrict__ bpos, const int64_t *__restrict__ mpos,
                int64_t stop, int64_t *__restrict__ cnt, int32_t *__restrict__ list1, int32_t *__restrict__ list2,
                int32_t *__restrict__ list3, unsigned *__restrict__ bin_counts, const int64_t *__restrict__ bcrd, int32_t *__restrict__ bcrd32, int64_t nnz_b)
{
    if (blockIdx.x >= row_ctas) {
        const int64_t first = (int64_t)(blockIdx.x - row_ctas) * NARROW_PART;
        for (int64_t q = first + 2 * threadIdx.x; q < first + NARROW_PART && q < nnz_b; q += 2 * BIN_THREADS) {
            if (q + 1 < nnz_b) {
                const longlong2 c = __ldcs((const longlong2 *)(bcrd + q));
                *(int2 *)(bcrd32 + q) = make_int2((int)c.x, (int)c.y);
            } else {
                bcrd32[q] = (int32_t)bcrd[q];
            }
        }
        return;
    }
    __shared__ unsigned char bin_of[BIN_ROWS];
    __shared__ unsigned short local_at[BIN_ROWS];
    __shared__ unsigned local_cnt[3], base[3], n_long;
    __shared__ unsigned short long_slot[BIN_ROWS];
    const int g = threadIdx.x / 8, l = threadIdx.x % 8;
    const unsigned gmask = 0xffu << ((threadIdx.x & 31) & ~7);
    if (threadIdx.x < 3) local_cnt[threadIdx.x] = 0;
    if (threadIdx.x == 3) n_long = 0;
    __syncthreads();
    const int64_t row0 = (int64_t)blockIdx.x * (BIN_PASS * passes);
    // the bin of a row from ub: its products, or more than `stop` if it has more
    auto place = [&](int slot, int64_t r, int64_t ub) {
        if (mpos) {
            int64_t ml = mpos[r + 1] - mpos[r];
            if (ml < ub) ub = ml;
        }
        int b = ub == 0 ? 0 : (ub <= HASH_ROW_MAX ? 1 : ub <= stop ? 3 : 2);
        bin_of[slot] = (unsigned char)b;
        if (b == 0) cnt[r] = 0;
        else local_at[slot] = (unsigned short)atomicAdd(&local_cnt[b - 1], 1u);
    };
    // lengths of the rows of B of entries p, p + lanes, ... (four of them) before `end`
    auto four = [&](int64_t p, int64_t end, int lanes) {
        int64_t k[4], sum = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) k[i] = p + i * lanes < end ? acrd[p + i * lanes] : -1;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (k[i] >= 0) sum += bpos[k[i] + 1] - bpos[k[i]];
        return sum;
    };
    for (int pass = 0; pass < passes; pass++) {
        const int slot = pass * BIN_PASS + g;
        const int64_t r = row0 + slot;
        if (r >= nrows) break;
        const int64_t as = apos[r], ae = apos[r + 1];
        int64_t ub = 0;
        bool later = false;
        for (int64_t p = as; p < ae; p += 32) {
            if (p - as >= 64 && ae - p > BIN_LONG_ROW) {       // many entries and hardly a product: left to the whole CTA below
                later = true;
                break;
            }
            int64_t part = four(p + l, ae, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) part += __shfl_xor_sync(gmask, (long long)part, o, 8);
            ub += part;
            if (ub > stop) break;
        }
        if (l == 0) {
            if (later) long_slot[atomicAdd(&n_long, 1u)] = (unsigned short)slot;
            else place(slot, r, ub);
        }
    }
    __syncthreads();
    const unsigned nl = n_long;
    for (unsigned i = 0; i < nl; i++) {
        const int slot = long_slot[i];
        const int64_t r = row0 + slot, ae = apos[r + 1];
        int64_t ub = 0;
        bool over = false;
        for (int64_t p = apos[r]; p < ae && !over; p += 4 * BIN_THREADS) {
            ub += four(p + threadIdx.x, ae, BIN_THREADS);
            over = __syncthreads_or(ub > stop);
        }
        // without a thread over the limit, the sum of all: no more than 256 * stop
        int64_t total = over ? stop + 1 : 0;
        if (!over) {
            __shared__ unsigned sum;
            if (threadIdx.x == 0) sum = 0;
            __syncthreads();
            if (ub) atomicAdd(&sum, (unsigned)ub);
            __syncthreads();
            total = sum;
        }
        if (threadIdx.x == 0) place(slot, r, total);
        __syncthreads();
    }
    __syncthreads();
    if (threadIdx.x < 3 && local_cnt[threadIdx.x]) base[threadIdx.x] = atomicAdd(&bin_counts[threadIdx.x], local_cnt[threadIdx.x]);
    __syncthreads();
    for (int slot = threadIdx.x; slot < BIN_PASS * passes; slot += BIN_THREADS) {
        int64_t r = row0 + slot;
        if (r >= nrows) break;
        int b = bin_of[slot];
        if (b == 1) list1[base[0] + local_at[slot]] = (int32_t)r;
        else if (b == 2) list2[base[1] + local_at[slot]] = (int32_t)r;
        else if (b == 3) list3[base[2] + local_at[slot]] = (int32_t)r;
    }
}

// What the host waits for, written straight to its page-locked words (three copies cost 5 us more).
__global__ void publish_kernel(const unsigned *__restrict__ bin_counts, const int64_t *__restrict__ nnz, unsigned *host)
{
    wait_for_previous();
    host[0] = bin_counts[0];
    host[1] = bin_counts[1];
    host[2] = bin_counts[2];
    *(int64_t *)(host + 4) = *nnz;
}

// --------------------------------------------------------------------------
// Bin 1: warp per row, hash table in shared memory.
//
// The products of 32 entries of the A row at a time are laid end to end and dealt to the lanes, 32 per step (short rows
// of B would otherwise leave most lanes idle, and every one of them cost its own chain of dependent loads), the next
// step's loads ahead of the current step's insertions.  The keys that an insertion created are numbered and listed, so a
// row ends by clearing its own slots and not the table, and the sums are kept by number.  The numeric call sorts key |
// number in registers (a bitonic network of 32 x E words; 64-bit ones from 2^24 columns on); ranking each key against
// all others was two thirds of the kernel before (16384 rows of 256 products: 207 us).
// --------------------------------------------------------------------------

// Inserts j; returns the slot, sets *fresh when this call created the entry.
template <int SLOTS>
__device__ __forceinline__ int hash_insert(int32_t *keys, int32_t j, bool *fresh)
{
    int h = (int)(((uint64_t)((uint32_t)j * 0x9E3779B1u) * SLOTS) >> 32);
    *fresh = false;
    for (int probe = 0; probe < SLOTS; probe++) {
        int32_t old = atomicCAS(&keys[h], -1, j);
        if (old == -1) { *fresh = true; return h; }
        if (old == j) return h;
        h = (h + 1) & (SLOTS - 1);
    }
    return -1;   // cannot happen: at most HASH_ROW_MAX distinct keys in two or four times as many slots
}

// Sorts the 32 * E words v[r] of lane l (place l * E + r) ascending: a bitonic network.  The blocks that a level sorts
// downwards are complemented for its duration, so that every exchange puts the smaller word first.
template <int E, typename T>
__device__ __forceinline__ void warp_sort(T (&v)[E], int lane)
{
#pragma unroll
    for (int k = 2; k <= 32 * E; k <<= 1) {
        // complemented at the level before: place & (k / 2); at this one: place & k
#pragma unroll
        for (int r = 0; r < E; r++) {
            const int place = lane * E + r;
            v[r] ^= (T)0 - (T)(((place & k) != 0) != (k > 2 && (place & (k >> 1)) != 0));
        }
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= E) {
                const bool low = (lane & (j / E)) == 0;
#pragma unroll
                for (int r = 0; r < E; r++) {
                    const T o = __shfl_xor_sync(0xffffffffu, v[r], j / E);
                    v[r] = low ? min(v[r], o) : max(v[r], o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < E; r++) {
                    if (r & j) continue;
                    const T a = min(v[r], v[r | j]), b = max(v[r], v[r | j]);
                    v[r] = a;
                    v[r | j] = b;
                }
            }
        }
    }
    // the last level complemented nothing (place < 32 E), the one before it the upper half, taken back above
}

// Writes a row's n listed keys in ascending order, and the value of each, to C.  The sorted words go through `list` so
// that the stores are coalesced.
template <int E, typename T>
__device__ __forceinline__ void write_sorted(T *list, const int32_t *row_keys, const double *vals, int n, int lane,
                                             int64_t *__restrict__ ccrd, double *__restrict__ cval)
{
    T v[E];
#pragma unroll
    for (int r = 0; r < E; r++) {
        const int at = lane + 32 * r;                  // any order goes in
        v[r] = at < n ? (T)row_keys[at] << 8 | (T)at : ~(T)0;
    }
    __syncwarp();
    warp_sort<E>(v, lane);
#pragma unroll
    for (int r = 0; r < E; r++)
        if (lane * E + r < n) list[lane * E + r] = v[r];
    __syncwarp();
    for (int i = lane; i < n; i += 32) {
        const T x = list[i];
        ccrd[i] = (int64_t)(x >> 8);
        cval[i] = vals[(int)(x & 255)];
    }
}

template <typename T>
__device__ __forceinline__ void write_row(T *list, const int32_t *row_keys, const double *vals, int n, int lane,
                                          int64_t *__restrict__ ccrd, double *__restrict__ cval)
{
    if (n <= 32) write_sorted<1>(list, row_keys, vals, n, lane, ccrd, cval);
    else if (n <= 64) write_sorted<2>(list, row_keys, vals, n, lane, ccrd, cval);
    else if (n <= 128) write_sorted<4>(list, row_keys, vals, n, lane, ccrd, cval);
    else write_sorted<8>(list, row_keys, vals, n, lane, ccrd, cval);
}

// WIDE: columns from 2^24 on, sorted as 64-bit words.
template <bool NUMERIC, bool WIDE>
__global__ void __launch_bounds__(HASH_WARPS * 32, NUMERIC && !WIDE ? 7 : 1)
hash_rows_kernel(const unsigned *__restrict__ nlist_dev, const int32_t *__restrict__ list, const int64_t *__restrict__ apos,
                 const int64_t *__restrict__ acrd, const double *__restrict__ aval,
                 const int64_t *__restrict__ bpos, const int32_t *__restrict__ bcrd,
                 const double *__restrict__ bval, const int64_t *__restrict__ mpos,
                 const int64_t *__restrict__ mcrd, int semi, int64_t *__restrict__ cnt,
                 const int64_t *__restrict__ cpos, int64_t *__restrict__ ccrd,
                 double *__restrict__ cval)
{
    using Word = typename std::conditional<WIDE, unsigned long long, unsigned>::type;
    constexpr int SLOTS = NUMERIC ? HASH_SLOTS : 2 * HASH_SLOTS;
    __shared__ int32_t s_keys[HASH_WARPS][SLOTS];
    __shared__ unsigned short s_slot[HASH_WARPS][HASH_ROW_MAX];      // slots of the row's keys, by number
    __shared__ unsigned short s_number[NUMERIC ? HASH_WARPS : 1][NUMERIC ? SLOTS : 1];
    __shared__ double s_vals[NUMERIC ? HASH_WARPS : 1][NUMERIC ? HASH_ROW_MAX : 1];
    __shared__ int32_t s_list[NUMERIC ? HASH_WARPS : 1][NUMERIC ? HASH_ROW_MAX : 1];
    __shared__ Word s_sorted[NUMERIC ? HASH_WARPS : 1][NUMERIC ? HASH_ROW_MAX : 1];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, wn = NUMERIC ? w : 0;
    const unsigned below = (1u << lane) - 1u;
    int32_t *keys = s_keys[w];
    double *vals = s_vals[wn];
    int32_t *row_keys = s_list[wn];
    const double ident = sr_identity(semi);
    for (int s = lane; s < SLOTS; s += 32) keys[s] = -1;
    if (NUMERIC)
        for (int s = lane; s < HASH_ROW_MAX; s += 32) vals[s] = ident;
    __syncwarp();
    wait_for_previous();
    const unsigned nwarps = gridDim.x * HASH_WARPS, nlist = *nlist_dev;
    for (unsigned it = blockIdx.x * HASH_WARPS + w; it < nlist; it += nwarps) {
        const int64_t r = list[it];
        int64_t ms = 0, me = 0;
        if (mpos) { ms = mpos[r]; me = mpos[r + 1]; }
        int n = 0;                                     // distinct columns so far
        const int64_t ae = apos[r + 1];
        for (int64_t p0 = apos[r]; p0 < ae; p0 += 32) {
            int64_t s = 0;
            int len = 0;
            double av = 0.0;
            if (p0 + lane < ae) {
                const int64_t k = acrd[p0 + lane];
                if (NUMERIC) av = aval[p0 + lane];
                s = bpos[k];
                len = (int)(bpos[k + 1] - s);
            }
            int upto = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const int total = __shfl_sync(0xffffffffu, upto, 31);
            const int64_t rel = s - (upto - len);      // product x of the batch is entry rel + x of B, for its own A entry
            auto fetch = [&](int x, int32_t &j, double &bv, double &a) {
                int t = 0;                             // first A entry whose prefix sum exceeds x
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, upto, t + step - 1) <= x) t += step;
                const int64_t q = __shfl_sync(0xffffffffu, (long long)rel, t) + x;
                if (NUMERIC) a = shfl_f64(av, t, 32);
                j = -1;
                if (x < total) {
                    j = bcrd[q];
                    if (NUMERIC) bv = bval[q];
                }
            };
            int32_t j1;
            double bv1 = 0.0, a1 = 0.0;
            fetch(lane, j1, bv1, a1);
            for (int x0 = 0; x0 < total; x0 += 32) {
                const int32_t j = j1;
                const double bv = bv1, a = a1;
                if (x0 + 32 < total) fetch(x0 + 32 + lane, j1, bv1, a1);
                bool fresh = false;
                int h = -1;
                if (j >= 0 && (!mpos || in_mask(mcrd, ms, me, j))) {
                    h = hash_insert<SLOTS>(keys, j, &fresh);
                }
                const unsigned made = __ballot_sync(0xffffffffu, fresh);
                if (fresh) {
                    const int at = n + __popc(made & below);
                    s_slot[w][at] = (unsigned short)h;
                    if (NUMERIC) {
                        row_keys[at] = j;
                        s_number[wn][h] = (unsigned short)at;
                    }
                }
                n += __popc(made);
                if (NUMERIC) {
                    __syncwarp();                      // the new keys' numbers
                    if (h >= 0) sr_fold(semi, &vals[s_number[wn][h]], sr_combine(semi, a, bv));
                }
            }
        }
        __syncwarp();
        if (!NUMERIC) {
            if (lane == 0) cnt[r] = n;
        } else {
            const int64_t base = cpos[r];
            write_row(s_sorted[wn], row_keys, vals, n, lane, ccrd + base, cval + base);
            __syncwarp();
        }
        for (int i = lane; i < n; i += 32) {
            keys[s_slot[w][i]] = -1;
            if (NUMERIC) vals[i] = ident;
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------------------
// Bin 1 without a mask, numeric call: the row has at most HASH_ROW_MAX products, so they are sorted by column in registers, and equal
// neighbours are added up.  A word is column | place of the product in the row (8 bits), so equal columns keep the order
// of the products and the sums are those of the sequential loop.  Products are dealt to the lanes as in the hash
// kernel.  Against hashing and sorting the distinct keys: no insertion loops, no atomics (16384 rows of 256
// products: 66 -> 47 us; counting alone, the table is the faster one: 26 against 34 us).
// --------------------------------------------------------------------------
template <int E, typename T>
__device__ __forceinline__ void sort_words(T *list, int n, int lane)
{
    T v[E];
#pragma unroll
    for (int r = 0; r < E; r++) v[r] = lane + 32 * r < n ? list[lane + 32 * r] : ~(T)0;      // any order goes in
    __syncwarp();
    warp_sort<E>(v, lane);
#pragma unroll
    for (int r = 0; r < E; r++) list[lane * E + r] = v[r];
    __syncwarp();
}

template <bool WIDE>
__global__ void __launch_bounds__(HASH_WARPS * 32)
short_rows_kernel(const unsigned *__restrict__ nlist_dev, const int32_t *__restrict__ rows, const int64_t *__restrict__ apos,
                  const int64_t *__restrict__ acrd, const double *__restrict__ aval, const int64_t *__restrict__ bpos,
                  const int32_t *__restrict__ bcrd, const double *__restrict__ bval, int semi,
                  const int64_t *__restrict__ cpos, int64_t *__restrict__ ccrd, double *__restrict__ cval)
{
    using Word = typename std::conditional<WIDE, unsigned long long, unsigned>::type;
    __shared__ Word s_list[HASH_WARPS][HASH_ROW_MAX];
    __shared__ double s_vals[HASH_WARPS][HASH_ROW_MAX];
    __shared__ unsigned short s_head[HASH_WARPS][HASH_ROW_MAX + 1];     // first word of every column
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    Word *list = s_list[w];
    double *vals = s_vals[w];
    unsigned short *head = s_head[w];
    wait_for_previous();
    const unsigned nwarps = gridDim.x * HASH_WARPS, nlist = *nlist_dev;
    for (unsigned it = blockIdx.x * HASH_WARPS + w; it < nlist; it += nwarps) {
        const int64_t r = rows[it];
        const int64_t ae = apos[r + 1];
        int n = 0;                                     // products so far
        for (int64_t p0 = apos[r]; p0 < ae; p0 += 32) {
            int64_t s = 0;
            int len = 0;
            double av = 0.0;
            if (p0 + lane < ae) {
                const int64_t k = acrd[p0 + lane];
                av = aval[p0 + lane];
                s = bpos[k];
                len = (int)(bpos[k + 1] - s);
            }
            int upto = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const int total = __shfl_sync(0xffffffffu, upto, 31);
            const int64_t rel = s - (upto - len);      // product x of the batch is entry rel + x of B, for its own A entry
#pragma unroll 2
            for (int x0 = 0; x0 < total; x0 += 32) {
                const int x = x0 + lane;
                int t = 0;                             // first A entry whose prefix sum exceeds x
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, upto, t + step - 1) <= x) t += step;
                const int64_t q = __shfl_sync(0xffffffffu, (long long)rel, t) + x;
                const double a = shfl_f64(av, t, 32);
                if (x < total) {
                    list[n + x] = (Word)bcrd[q] << 8 | (Word)(n + x);
                    vals[n + x] = sr_combine(semi, a, bval[q]);
                }
            }
            n += total;
        }
        __syncwarp();
        if (n <= 32) sort_words<1>(list, n, lane);
        else if (n <= 64) sort_words<2>(list, n, lane);
        else if (n <= 128) sort_words<4>(list, n, lane);
        else sort_words<8>(list, n, lane);
        int distinct = 0;
        for (int x0 = 0; x0 < n; x0 += 32) {
            const int x = x0 + lane;
            const bool first = x < n && (x == 0 || (list[x] >> 8) != (list[x - 1] >> 8));
            const unsigned firsts = __ballot_sync(0xffffffffu, first);
            if (first) head[distinct + __popc(firsts & below)] = (unsigned short)x;
            distinct += __popc(firsts);
        }
        if (lane == 0) head[distinct] = (unsigned short)n;
        __syncwarp();
        const int64_t base = cpos[r];
        for (int i = lane; i < distinct; i += 32) {
            const int b = head[i], e = head[i + 1];
            const Word x = list[b];
            double sum = vals[(int)(x & 255)];
            for (int y = b + 1; y < e; y++) sum = sr_fold_value(semi, sum, vals[(int)(list[y] & 255)]);
            ccrd[base + i] = (int64_t)(x >> 8);
            cval[base + i] = sum;
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------------------
// Bin 1 without a mask, symbolic call, where a bitmap over B's columns fits a warp's share of shared memory: FEW_COLUMNS columns.
//
// A warp per row; the products are dealt to the lanes as above, mark their columns and count the bits they are the first to set;
// then they clear the words of the columns they have kept.  Against the hash table: one atomic per product that always succeeds (16,384 rows of
// 256 products in as many columns 25 -> 18 us, 32,768 47 -> 39).  The numeric call by ranks from such a bitmap takes longer than the
// sort (51 us against 46: two shared-memory atomics per product and the words' counts).
// --------------------------------------------------------------------------
static const int64_t FEW_COLUMNS = 32768;               // 20 KB a CTA, which leaves the occupancy to the registers

__global__ void __launch_bounds__(HASH_WARPS * 32)
few_columns_kernel(const unsigned *__restrict__ nlist_dev, const int32_t *__restrict__ rows, int words,
                   const int64_t *__restrict__ apos, const int64_t *__restrict__ acrd, const int64_t *__restrict__ bpos,
                   const int32_t *__restrict__ bcrd, int64_t *__restrict__ cnt)
{
    extern __shared__ uint32_t s_few[];                 // a bitmap per warp
    __shared__ int32_t s_cols[HASH_WARPS][HASH_ROW_MAX];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *bits = s_few + w * words;
    int32_t *cols = s_cols[w];
    for (int t = lane; t < words; t += 32) bits[t] = 0;
    __syncwarp();
    wait_for_previous();
    const unsigned nwarps = gridDim.x * HASH_WARPS, nlist = *nlist_dev;
    for (unsigned it = blockIdx.x * HASH_WARPS + w; it < nlist; it += nwarps) {
        const int64_t r = rows[it];
        const int64_t ae = apos[r + 1];
        int n = 0;                                     // products so far
        unsigned fresh = 0;
        for (int64_t p0 = apos[r]; p0 < ae; p0 += 32) {
            int64_t s = 0;
            int len = 0;
            if (p0 + lane < ae) {
                const int64_t k = acrd[p0 + lane];
                s = bpos[k];
                len = (int)(bpos[k + 1] - s);
            }
            int upto = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const int total = __shfl_sync(0xffffffffu, upto, 31);
            const int64_t rel = s - (upto - len);      // product x of the batch is entry rel + x of B, for its own A entry
#pragma unroll 4
            for (int x0 = 0; x0 < total; x0 += 32) {
                const int x = x0 + lane;
                int t = 0;                             // first A entry whose prefix sum exceeds x
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, upto, t + step - 1) <= x) t += step;
                const int64_t q = __shfl_sync(0xffffffffu, (long long)rel, t) + x;
                if (x < total) {
                    const int32_t j = bcrd[q];
                    const uint32_t bit = 1u << (j & 31);
                    cols[n + x] = j;
                    fresh += !(atomicOr(&bits[j >> 5], bit) & bit);
                }
            }
            n += total;
        }
        fresh = __reduce_add_sync(0xffffffffu, fresh);
        if (lane == 0) cnt[r] = fresh;
        __syncwarp();                                  // the other lanes' columns and marks: a reduction orders no memory
        for (int x = lane; x < n; x += 32) bits[cols[x] >> 5] = 0;
        __syncwarp();
    }
}

// --------------------------------------------------------------------------
// Bin 3, without a mask: rows of up to MID_ROW_MAX products where a bitmap over B's columns fits beside them.
//
// A CTA of 128 or 256 threads per row.  The lengths of as many rows of B are scanned and their products dealt to the threads one
// by one, so that short and long rows of B cost the same per product.  A product marks its column and is kept; popcounts
// of the words give every column its rank; the products are added up by rank in shared memory, and the row is written
// in one coalesced pass.  The kept products also clear the bitmap.  Against a bin-2 CTA: no bitmap stored by one call
// and read by the other, no cleared and re-read output, four times as many rows at a time.
//
// Bound: instructions, two passes over the words and about 60 per product.  50,000 rows of 900 products in 50,000 columns:
// 1374 -> 845 us for both calls; the numeric one has the shared-memory pipe busy two thirds of the time.  A second bitmap of
// the words with columns, to skip the others, cost more than it saved (966).
// --------------------------------------------------------------------------
static const int MID_MANY_WORDS = 2048;     // 256 threads from here on, as fewer CTAs fit: 180,000 rows of 20, 4250 -> 3410 us (at 50,000 columns 845 -> 900)
static const int MID_ROW_MAX = 1024;
// The bitmap and its ranks, beside the 29 KB the kernel has anyway in 227: 1,070,400 columns.  It is the faster one as far as it
// goes, where one CTA is left on an SM too.  Both calls, rows of 20, in milliseconds here and in bin 2: 262,200 columns 7.1 and
// 12.0, 400,000 12.0 and 25.5, 700,000 48 and 100, 1,000,000 90 and 287; rows of 30 and 1,000,000 columns 113 and 301.
static const size_t MID_SMEM = 196 * 1024;

template <int THREADS, bool NUMERIC>
__global__ void __launch_bounds__(THREADS)
mid_rows_kernel(const unsigned *__restrict__ nlist_dev, const int32_t *__restrict__ rows, int words,
                const int64_t *__restrict__ apos, const int64_t *__restrict__ acrd, const double *__restrict__ aval,
                const int64_t *__restrict__ bpos, const int32_t *__restrict__ bcrd, const double *__restrict__ bval, int semi,
                int64_t *__restrict__ cnt, const int64_t *__restrict__ cpos, int64_t *__restrict__ ccrd,
                double *__restrict__ cval)
{
    constexpr int NW = THREADS / 32, KEEP = NUMERIC ? MID_ROW_MAX : 1;
    extern __shared__ uint32_t bm[];                   // words, then (numeric) a 16-bit rank for each
    __shared__ int64_t s_rel[THREADS];
    __shared__ double s_av[NUMERIC ? THREADS : 1], s_vals[KEEP], s_sums[KEEP];
    __shared__ int s_upto[THREADS], s_cols[MID_ROW_MAX], s_out[KEEP];
    __shared__ unsigned s_warp[NW], s_count;
    unsigned short *pre = (unsigned short *)(bm + words);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const double ident = sr_identity(semi);
    for (int w = tid; w < words; w += THREADS) bm[w] = 0;
    wait_for_previous();
    const unsigned nlist = *nlist_dev;
    for (unsigned it = blockIdx.x; it < nlist; it += gridDim.x) {
        const int64_t r = rows[it], ae = apos[r + 1];
        int n = 0;                                     // products so far
        unsigned fresh = 0;
        for (int64_t p0 = apos[r]; p0 < ae; p0 += THREADS) {
            int64_t s = 0;
            int len = 0;
            if (p0 + tid < ae) {
                const int64_t k = acrd[p0 + tid];
                if (NUMERIC) s_av[tid] = aval[p0 + tid];
                s = bpos[k];
                len = (int)(bpos[k + 1] - s);
            }
            int upto = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            if (lane == 31) s_warp[warp] = upto;
            __syncthreads();
            int total = 0;
#pragma unroll
            for (int w = 0; w < NW; w++) {
                if (w < warp) upto += s_warp[w];
                total += s_warp[w];
            }
            s_upto[tid] = upto;
            s_rel[tid] = s - (upto - len);             // product x of the batch is entry s_rel[t] + x of B, for its own A entry
            __syncthreads();
#pragma unroll 2
            for (int x = tid; x < total; x += THREADS) {
                int t = 0;                             // first A entry whose prefix sum exceeds x
#pragma unroll
                for (int step = THREADS / 2; step > 0; step >>= 1)
                    if (s_upto[t + step - 1] <= x) t += step;
                const int64_t q = s_rel[t] + x;
                const int32_t j = bcrd[q];
                s_cols[n + x] = j;
                if (NUMERIC) {
                    s_vals[n + x] = sr_combine(semi, s_av[t], bval[q]);
                    atomicOr(&bm[j >> 5], 1u << (j & 31));
                } else {
                    fresh += !((atomicOr(&bm[j >> 5], 1u << (j & 31)) >> (j & 31)) & 1u);
                }
            }
            n += total;
            __syncthreads();                           // the batch's arrays and the warps' sums are free again
        }
        if (!NUMERIC) {
            if (tid == 0) s_count = 0;
            fresh = __reduce_add_sync(0xffffffffu, fresh);
            __syncthreads();
            if (lane == 0 && fresh) atomicAdd(&s_count, fresh);
        } else {
            // words in runs of an odd number per thread: every bank once
            const int per = ((words + THREADS - 1) / THREADS) | 1;
            const int w0 = min(tid * per, words), w1 = min(w0 + per, words);
            unsigned c = 0;
            for (int w = w0; w < w1; w++) c += __popc(bm[w]);
            unsigned incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) s_warp[warp] = incl;
            const int64_t base = cpos[r];
            const int out = (int)(cpos[r + 1] - base);
            for (int i = tid; i < out; i += THREADS) s_sums[i] = ident;
            __syncthreads();
            unsigned run = incl - c;
#pragma unroll
            for (int w = 0; w < NW; w++)
                if (w < warp) run += s_warp[w];
            for (int w = w0; w < w1; w++) {
                pre[w] = (unsigned short)run;
                run += __popc(bm[w]);
            }
            __syncthreads();
            for (int i = tid; i < n; i += THREADS) {
                const int j = s_cols[i];
                const unsigned rank = pre[j >> 5] + __popc(bm[j >> 5] & ((1u << (j & 31)) - 1u));
                s_out[rank] = j;
                sr_fold(semi, &s_sums[rank], s_vals[i]);
            }
            __syncthreads();
            for (int i = tid; i < out; i += THREADS) {
                __stcs((long long *)ccrd + base + i, (long long)s_out[i]);
                __stcs(cval + base + i, s_sums[i]);
            }
        }
        for (int i = tid; i < n; i += THREADS) bm[s_cols[i] >> 5] = 0;
        __syncthreads();
        if (!NUMERIC && tid == 0) cnt[r] = s_count;
    }
}

static size_t mid_smem(int words, bool numeric) { return (size_t)words * (numeric ? 6 : 4); }

// --------------------------------------------------------------------------
// Bin 2: CTA per row, bitmap over B's columns.
// --------------------------------------------------------------------------
__device__ __forceinline__ unsigned block_sum_u32(unsigned v, unsigned *s_warp)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    unsigned t = 0;
    for (int i = 0; i < BM_THREADS / 32; i++) t += s_warp[i];
    return t;
}

// Rows of B longer than this are walked by the whole CTA instead of one warp: in a power-law
// product a few such rows hold most of the work of an output row, and one warp working alone while
// fifteen wait at the next barrier was the largest stall of both passes.
static const int64_t LONG_B_ROW = 1024;

static const unsigned BM_DENSE_ROW = 512;   // bits in 32 consecutive bitmap words from which crd is written word by word (measured: 96 / 192 / 320 / 512 / 768 / never = 22.9 / 21.8 / 21.5 / 21.45 / 21.65 / 21.7 ms numeric at config 4)
// Columns that need a look-up: the least that a warp's stage is worth having for.  Rows of 32 words with more than it holds go out like those
// of BM_DENSE_ROW, one word at a time (one by one with a look-up each 2000 rows of 100,000 products in 350,000 columns took 3.08 ms; 2.42
// so, and 2.53 before columns were renumbered).
static const unsigned STAGE_MIN = 128;
static const int LONG_LIST = 1024;          // long rows of B remembered per pass over a row of A
// Steps of 32 products whose loads are in flight, with 3 CTAs of 512 threads on an SM (R-MAT scale 18 squared, numeric / symbolic kernel in
// ms): 1 19.3 / 4.6, 2 18.1 / 4.0, 4 17.4 / 3.8.  More of them with fewer warps is slower (2 CTAs, 6 steps 20.1), and so are more
// warps with fewer steps (4 CTAs, 2 steps 20.1).
static const int WALK_DEPTH = 4;
// Where the fold is a loop, and where the bitmaps are in memory, steps side by side only meet in it: one is folded with the next one's
// loads ahead.  Numeric kernel in ms with 1 (nothing ahead) / 2 / 4: min-plus, R-MAT scale 14, 16 per row 0.85 / 0.93 / 0.94; scale 17, 5 per
// row 2.4 / 2.4 / 2.6.  Both calls in us with nothing and with the next step ahead: min-plus, scale 13, 16 per row 566, 526; plus-times, 40 rows
// of 24,000 products in 8,000,000 columns 930, 852.
static const int WALK_DEPTH_FOLD = 1;

// Calls f(j, bv, av) for every product of row r of A with B in this CTA's share: j and bv are the column and
// value of an entry of row acrd[p] of B (bv = 0 when bval is null), av = aval[p] (0 when aval is null).  A team
// of `team` CTAs deals the entries of the A row out over its warps one by one.  The loads are arranged so that
// no warp waits on a chain: 32 entries of a warp's share look up their rows of B lane-parallel (acrd, then
// bpos, once per batch), and DEPTH steps of 32 products are fetched before the first of them is worked on.
// hub_id (null: none): rows of B with a number >= 0 there are left out.
// Short rows of B are walked by one warp; long ones are remembered in s_long and then walked by the
// whole CTA.  s_ctl: [0] entries in s_long, [1] set when the list was too small (then the share is
// scanned again for long rows).  All threads of the CTA must call this.
template <int DEPTH, typename F>
__device__ __forceinline__ void for_each_product(int64_t r, unsigned part, unsigned team,
                                                 const int64_t *__restrict__ apos,
                                                 const int64_t *__restrict__ acrd,
                                                 const double *__restrict__ aval,
                                                 const int64_t *__restrict__ bpos,
                                                 const int32_t *__restrict__ bcrd,
                                                 const double *__restrict__ bval, const int32_t *__restrict__ hub_id,
                                                 int *s_long, unsigned *s_ctl, F f)
{
    constexpr int NW = BM_THREADS / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t as = apos[r], ae = apos[r + 1];
    if (threadIdx.x == 0) { s_ctl[0] = 0; s_ctl[1] = 0; }
    __syncthreads();
    // this warp's entries of the A row: first, first + stride, ... (dealt one by one, so that the warps of a
    // team share a row of any length evenly); 32 of them at a time are looked up lane-parallel
    const int64_t stride = (int64_t)team * NW;
    const int64_t first = as + (int64_t)part * NW + warp;
    for (int64_t p0 = first; p0 < ae; p0 += 32 * stride) {
        const int64_t p = p0 + lane * stride;
        int64_t s_l = 0;
        int n_l = 0;                     // entries of this lane's row of B; 0 for lanes past the A row and long rows
        double av_l = 0.0;
        if (p < ae) {
            const int64_t k = acrd[p];
            s_l = bpos[k];
            int64_t len = bpos[k + 1] - s_l;
            if (hub_id && hub_id[k] >= 0) len = 0;
            if (aval) av_l = aval[p];
            if (len > LONG_B_ROW) {
                const unsigned at = atomicAdd(&s_ctl[0], 1u);
                if (at < (unsigned)LONG_LIST) s_long[at] = (int)(p - as);
                else s_ctl[1] = 1;
            } else {
                n_l = (int)len;
            }
        }
        // the rows' entries in steps of 32, DEPTH steps' loads in flight whether they belong to one row or to several
        unsigned left = __ballot_sync(0xffffffffu, n_l > 0);
        int64_t at = 0;
        int rem = 0;
        double av = 0.0;
        auto step = [&](int32_t &j, double &v, double &a) {
            if (rem <= 0 && left) {
                const int t = __ffs(left) - 1;
                left &= left - 1;
                at = __shfl_sync(0xffffffffu, (long long)s_l, t) + lane;
                rem = __shfl_sync(0xffffffffu, n_l, t);
                av = shfl_f64(av_l, t, 32);
            }
            a = av;
            j = -1;
            v = 0.0;
            if (lane < rem) {
                j = bcrd[at];
                if (bval) v = bval[at];
            }
            at += 32;
            rem -= 32;
        };
        if (DEPTH == 1) {
            int32_t j = -1;
            double v = 0.0, a = 0.0;
            if (left) step(j, v, a);
            for (bool more = true; more;) {
                more = left || rem > 0;
                int32_t j1 = -1;
                double v1 = 0.0, a1 = 0.0;
                if (more) step(j1, v1, a1);
                if (j >= 0) f(j, v, a);
                j = j1; v = v1; a = a1;
            }
        } else {
            while (left || rem > 0) {
                int32_t j[DEPTH];
                double v[DEPTH], am[DEPTH];
#pragma unroll
                for (int i = 0; i < DEPTH; i++) step(j[i], v[i], am[i]);
#pragma unroll
                for (int i = 0; i < DEPTH; i++)
                    if (j[i] >= 0) f(j[i], v[i], am[i]);
            }
        }
    }
    __syncthreads();
    auto whole_cta = [&](int64_t sl, int64_t el, double avl) {
        for (int64_t q = sl + threadIdx.x; q < el; q += 2 * BM_THREADS) {
            const bool two = q + BM_THREADS < el;
            const int32_t ja = bcrd[q];
            const int32_t jb = two ? bcrd[q + BM_THREADS] : 0;
            const double va = bval ? bval[q] : 0.0;
            const double vb = (bval && two) ? bval[q + BM_THREADS] : 0.0;
            f(ja, va, avl);
            if (two) f(jb, vb, avl);
        }
    };
    if (!s_ctl[1]) {
        const unsigned n = s_ctl[0];
        for (unsigned i = 0; i < n; i++) {
            const int64_t pl = as + s_long[i];
            const int64_t k = acrd[pl];
            whole_cta(bpos[k], bpos[k + 1], aval ? aval[pl] : 0.0);
        }
    } else {
        for (int64_t p0 = as + (int64_t)part * NW; p0 < ae; p0 += stride)
            for (int64_t pl = p0; pl < p0 + NW && pl < ae; pl++) {
                const int64_t k = acrd[pl];
                const int64_t sl = bpos[k], el = bpos[k + 1];
                if (el - sl <= LONG_B_ROW || (hub_id && hub_id[k] >= 0)) continue;
                whole_cta(sl, el, aval ? aval[pl] : 0.0);
            }
    }
}

// marks the columns of row r's products in bm (bm cleared by the caller)
__device__ __forceinline__ void mark_products(uint32_t *bm, int64_t r, const int64_t *__restrict__ apos,
                                              const int64_t *__restrict__ acrd,
                                              const int64_t *__restrict__ bpos,
                                              const int32_t *__restrict__ bcrd,
                                              const int64_t *__restrict__ mpos,
                                              const int64_t *__restrict__ mcrd, int *s_long, unsigned *s_ctl)
{
    int64_t ms = 0, me = 0;
    if (mpos) { ms = mpos[r]; me = mpos[r + 1]; }
    for_each_product<WALK_DEPTH>(r, 0u, 1u, apos, acrd, nullptr, bpos, bcrd, nullptr, nullptr, s_long, s_ctl, [&](int32_t j, double, double) {
        if (mpos && !in_mask(mcrd, ms, me, j)) return;
        atomicOr(&bm[j >> 5], 1u << (j & 31));          // testing the bit first was measured slower (6.4 vs 5.2 ms)
    });
}

template <bool SMEM>
__global__ void __launch_bounds__(BM_THREADS)
bitmap_symbolic_kernel(const unsigned *__restrict__ nlist_dev, const int32_t *__restrict__ list, int words,
                       uint32_t *__restrict__ gbm, const int64_t *__restrict__ apos,
                       const int64_t *__restrict__ acrd, const int64_t *__restrict__ bpos,
                       const int32_t *__restrict__ bcrd, const int64_t *__restrict__ mpos,
                       const int64_t *__restrict__ mcrd, int64_t *__restrict__ cnt,
                       uint32_t *__restrict__ bm_store)
{
    extern __shared__ uint32_t s_dyn[];
    __shared__ unsigned s_warp[BM_THREADS / 32];
    __shared__ int s_long[LONG_LIST];
    __shared__ unsigned s_ctl[2];
    uint32_t *bm = SMEM ? s_dyn : gbm + (size_t)blockIdx.x * words;
    wait_for_previous();
    const unsigned nlist = *nlist_dev;
    for (unsigned it = blockIdx.x; it < nlist; it += gridDim.x) {
        const int64_t r = list[it];
        for (int w = threadIdx.x; w < words; w += BM_THREADS) bm[w] = 0;
        __syncthreads();
        mark_products(bm, r, apos, acrd, bpos, bcrd, mpos, mcrd, s_long, s_ctl);
        __syncthreads();
        unsigned c = 0;
        uint32_t *keep = bm_store ? bm_store + (size_t)it * words : nullptr;
        for (int w = threadIdx.x; w < words; w += BM_THREADS) {
            uint32_t v = bm[w];
            c += __popc(v);
            if (keep) keep[w] = v;
        }
        unsigned total = block_sum_u32(c, s_warp);
        if (threadIdx.x == 0) cnt[r] = total;
        __syncthreads();
    }
}

// --------------------------------------------------------------------------
// Teams for the numeric pass of bin-2 rows.
//
// f64 atomics run at ~200 G/s while their targets stay in L2 and at 20-80 G/s once the rows being
// accumulated no longer fit (measured on this part with a stand-alone probe).  With one CTA per row
// the rows in flight of a power-law product hold far more than L2, so a row whose output is large
// is given to a team of T CTAs instead: they split the entries of the A row, add into the same
// output row, and T is chosen so that (CTAs in flight / T) rows of that size fit the budget.
// Teams are laid out contiguously in an item list and CTAs draw items in order, so the members of a
// team run at about the same time.  The values of team rows are cleared by a separate launch
// (a member must not start adding before another has cleared); single-CTA rows clear their own.
// --------------------------------------------------------------------------
struct TeamHeader {
    unsigned nitems;
    unsigned next;
    unsigned overflow;
    unsigned pad;
};
static const unsigned TEAM_MAX = 64;
// Shares of the L2 that one CTA's row may take: a team of two clears and scans the row twice, which is more than what it saves where the row is
// a little above one share. Rows of 1.06 shares 4.95 ms in teams and 4.25 alone, 1.2 1.91 and 1.73, 1.33 2.06 and 1.94, 1.45 2.23 and
// 2.29, 1.6 2.58 and 3.13 (6000 and 20,000 rows of 20,000 to 35,000 products in 300,000 columns, both calls).
static const double TEAM_ALONE = 1.4;
// With fewer rows than twice the CTAs that run, teams also fill the chip: any row above one share gets one, with shares as for four CTAs an SM.
// Rows of 18,000 entries in 120,000 columns, both calls, before columns were renumbered, without and with this: 20 rows 110, 140, 113; 300 170, 172, 166;
// 500 220, 222, 206; 900 340, 316, 326; 1800 580, 521, 548.  20,000 in 60,000: 20 rows 122, 138, 106; 500 258, 285, 252; 900 386, 390, 385; 1800 675, 648, 652.
static const unsigned TEAM_FEW = 2;

__device__ __forceinline__ uint64_t team_pack(unsigned it, unsigned part, unsigned t)
{
    return (uint64_t)it | ((uint64_t)part << 32) | ((uint64_t)t << 48);
}

__global__ void __launch_bounds__(256)
team_items_kernel(unsigned nlist, const int32_t *__restrict__ list, const int64_t *__restrict__ cpos,
                  double ctas_per_budget_entry, double alone_to, TeamHeader *th, uint64_t *items, unsigned cap)
{
    // consecutive list entries in consecutive slots (one warp-wide scan per 32 rows keeps the list ordered)
    const unsigned it = blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    unsigned t = 0;
    if (it < nlist) {
        const int64_t r = list[it];
        const double want = (double)(cpos[r + 1] - cpos[r]) * ctas_per_budget_entry;
        t = want <= alone_to ? 1u : (want >= (double)TEAM_MAX ? TEAM_MAX : (unsigned)ceil(want));
    }
    unsigned incl = t;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    unsigned base = 0;
    if (lane == 31) base = atomicAdd(&th->nitems, incl);
    base = __shfl_sync(0xffffffffu, base, 31) + incl - t;
    if (t) {
        if (base + t <= cap) {
            for (unsigned i = 0; i < t; i++) items[base + i] = team_pack(it, i, t);
        } else {
            th->overflow = 1;
        }
    }
}

__global__ void __launch_bounds__(256)
team_clear_kernel(const TeamHeader *th, const uint64_t *__restrict__ items, unsigned cap,
                  const int32_t *__restrict__ list, const int64_t *__restrict__ cpos, int semi,
                  double *__restrict__ cval)
{
    wait_for_previous();
    unsigned n = th->nitems;
    if (n > cap) n = 0;
    const double ident = sr_identity(semi);
    for (unsigned i = blockIdx.x; i < n; i += gridDim.x) {
        const uint64_t v = items[i];
        const unsigned t = (unsigned)(v >> 48), part = (unsigned)(v >> 32) & 0xffffu;
        if (t <= 1) continue;
        const int64_t r = list[(unsigned)v];
        const int64_t base = cpos[r], n_out = cpos[r + 1] - base;
        const int64_t per = (n_out + t - 1) / t;
        const int64_t s = base + (int64_t)part * per;
        int64_t e = s + per;
        if (e > base + n_out) e = base + n_out;
        for (int64_t q = s + threadIdx.x; q < e; q += blockDim.x) cval[q] = ident;
    }
}

// stride: words from one stored bitmap to the next.  MAPPED: colmap has the column of each number in bcrd.
template <bool SMEM, bool PLUS_TIMES, bool MAPPED>
__global__ void __launch_bounds__(BM_THREADS, SMEM ? 3 : 1)
bitmap_numeric_kernel(unsigned nlist, const int32_t *__restrict__ list, int words, int stride, unsigned stage_n,
                      const int32_t *__restrict__ colmap,
                      uint32_t *__restrict__ gbm, const int64_t *__restrict__ apos,
                      const int64_t *__restrict__ acrd, const double *__restrict__ aval,
                      const int64_t *__restrict__ bpos, const int32_t *__restrict__ bcrd,
                      const double *__restrict__ bval, const int64_t *__restrict__ mpos,
                      const int64_t *__restrict__ mcrd, int semi,
                      const uint32_t *__restrict__ bm_store, const int64_t *__restrict__ cpos,
                      int64_t *__restrict__ ccrd, double *__restrict__ cval, TeamHeader *th,
                      const uint64_t *__restrict__ items)
{
    extern __shared__ uint32_t s_dyn[];
    __shared__ unsigned s_item;
    __shared__ unsigned s_scan[BM_THREADS / 32];
    __shared__ int s_long[LONG_LIST];
    __shared__ unsigned s_ctl[2];
    uint32_t *bm = SMEM ? s_dyn : gbm + (size_t)blockIdx.x * 2 * words;
    uint32_t *pre = bm + words;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int32_t *stage = (int32_t *)s_dyn + (SMEM ? 2 * words : 0) + warp * stage_n;
    constexpr int NW = BM_THREADS / 32;
    wait_for_previous();
    for (unsigned iter = blockIdx.x;; iter += gridDim.x) {
        // one row per CTA, or (with an item list) the next member of a team
        unsigned it = iter, part = 0, team = 1;
        if (th) {
            if (threadIdx.x == 0) s_item = atomicAdd(&th->next, 1u);
            __syncthreads();
            const unsigned idx = s_item;
            if (idx >= (items ? th->nitems : nlist)) break;
            it = idx;
            if (items) {
                const uint64_t v = items[idx];
                it = (unsigned)v;
                part = (unsigned)(v >> 32) & 0xffffu;
                team = (unsigned)(v >> 48);
            }
        } else if (iter >= nlist) {
            break;
        }
        const int64_t r = list[it];
        if (bm_store) {
            const uint32_t *keep = bm_store + (size_t)it * stride;
            for (int w = threadIdx.x; w < words; w += BM_THREADS) bm[w] = __ldcs(keep + w);     // read once per member
            __syncthreads();
        } else {
            for (int w = threadIdx.x; w < words; w += BM_THREADS) bm[w] = 0;
            __syncthreads();
            mark_products(bm, r, apos, acrd, bpos, bcrd, mpos, mcrd, s_long, s_ctl);
            __syncthreads();
        }
        // Exclusive prefix popcount per word, and the row's coordinates.  A warp owns a run of whole rows of 32
        // consecutive words; lane l of the warp holds word l of the current row, so every shared-memory access
        // below is conflict-free and the prefix inside a row is a warp scan.
        const int nrow32 = (words + 31) >> 5;
        const int rows_per_warp = (nrow32 + NW - 1) / NW;
        const int i0 = warp * rows_per_warp, i1 = min(i0 + rows_per_warp, nrow32);
        unsigned mine = 0;
        for (int i = i0; i < i1; i++) {
            const int w = i * 32 + lane;
            if (w < words) mine += __popc(bm[w]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
        if (lane == 0) s_scan[warp] = mine;
        __syncthreads();
        unsigned run = 0;
        for (int w2 = 0; w2 < warp; w2++) run += s_scan[w2];
        const int64_t base = cpos[r];
        const int64_t rown = cpos[r + 1] - base;
        unsigned held = 0;                             // columns in the stage: those of the outputs before `upto`
        auto flush = [&](unsigned upto) {
            __syncwarp();
            long long *out = (long long *)ccrd + base + upto - held;
#pragma unroll 4
            for (unsigned o = lane; o < held; o += 32) {
                __stcs(out + o, (long long)__ldg(colmap + stage[o]));               // written once, not read here again
            }
            __syncwarp();
            held = 0;
        };
        for (int i = i0; i < i1; i++) {
            const int w = i * 32 + lane;
            uint32_t v = w < words ? bm[w] : 0u;
            const unsigned c = __popc(v);
            unsigned incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            const unsigned excl = run + incl - c;
            if (w < words) pre[w] = excl;
            const unsigned rowtotal = __shfl_sync(0xffffffffu, incl, 31);
            const unsigned before = run;
            run += rowtotal;
            if (rowtotal == 0) continue;
            // the members of a team share the writing of crd by rows of 32 words
            const bool ours = team == 1 || (unsigned)i % team == part;
            if (MAPPED && held && (!ours || held + rowtotal > stage_n)) flush(before);
            if (!ours) continue;
            if (rowtotal >= BM_DENSE_ROW || (MAPPED && rowtotal > stage_n)) {
                if (MAPPED && held) flush(before);
                // many bits per word: one word at a time, lane b writes column 32 w + b at its rank, so a
                // store instruction covers consecutive addresses
                // (all 32 words in a fixed-trip loop: the shuffles of different words do not depend on each
                // other, so they overlap; a loop over the non-empty words only ran one word per shuffle latency)
                long long *out = (long long *)ccrd + base;
                const unsigned below = (1u << lane) - 1u;
#pragma unroll 8
                for (int l = 0; l < 32; l++) {
                    const uint32_t wv = __shfl_sync(0xffffffffu, v, l);
                    const unsigned wp = __shfl_sync(0xffffffffu, excl, l);
                    if ((wv >> lane) & 1u) {
                        const int j = (i * 32 + l) * 32 + lane;
                        __stcs(out + wp + __popc(wv & below), (long long)(MAPPED ? __ldg(colmap + j) : j));
                    }
                }
            } else if (!MAPPED) {
                unsigned at = excl;
                for (; v; v &= v - 1, at++) {
                    const int j = w * 32 + __ffs(v) - 1;
                    __stcs((long long *)ccrd + base + at, (long long)j);
                }
            } else {
                // the columns go through shared memory, so that the stores are coalesced and the look-ups independent (R-MAT scale
                // 18 squared 21.5 -> 18.6 ms)
                unsigned at = held + excl - before;
                for (; v; v &= v - 1) stage[at++] = w * 32 + __ffs(v) - 1;
                held += rowtotal;
            }
        }
        if (MAPPED && held) flush(run);
        if (team == 1)
            for (int64_t t = threadIdx.x; t < rown; t += BM_THREADS) cval[base + t] = sr_identity(semi);
        __syncthreads();
        // accumulate every product at the rank of its column
        double *crow = cval + base;
        for_each_product<PLUS_TIMES ? WALK_DEPTH : WALK_DEPTH_FOLD>(r, part, team, apos, acrd, aval, bpos, bcrd, bval, nullptr, s_long, s_ctl, [&](int32_t j, double bv, double av) {
            uint32_t word = bm[j >> 5];
            uint32_t bit = 1u << (j & 31);
            if (!(word & bit)) return;          // filtered out by the mask
            unsigned rank = pre[j >> 5] + __popc(word & (bit - 1u));
            if (PLUS_TIMES) atomicAdd(crow + rank, av * bv);
            else sr_fold(semi, crow + rank, sr_combine(semi, av, bv));
        });
        __syncthreads();
    }
    (void)mpos; (void)mcrd;
}

// --------------------------------------------------------------------------
// Bin 2 by hubs (hubs.cuh).
// --------------------------------------------------------------------------

// The hubs that the next entries of a row of A name, from *p on, to s_hub, their count to *s_n, in any order.  Stops when a further
// step of BM_THREADS entries might not fit.  Called by the whole CTA.
__device__ __forceinline__ int hub_list(int64_t *p, int64_t ae, const int64_t *__restrict__ acrd, const int32_t *__restrict__ hub_id,
                                        int *s_hub, unsigned *s_n)
{
    __syncthreads();                                   // the list is no longer read
    if (threadIdx.x == 0) *s_n = 0;
    __syncthreads();
    int64_t at = *p;
    for (; at < ae && (int)*s_n <= LONG_LIST - BM_THREADS; at += BM_THREADS) {
        __syncthreads();                               // all have read the count
        if (at + threadIdx.x < ae) {
            const int h = hub_id[acrd[at + threadIdx.x]];
            if (h >= 0) s_hub[atomicAdd(s_n, 1u)] = h;
        }
        __syncthreads();
    }
    *p = at;
    return (int)*s_n;
}

// bm = the columns of row r's products; hub_id == null: B has no hubs
__device__ __forceinline__ void hub_mark_row(uint32_t *bm, int stride, int64_t r, const int64_t *__restrict__ apos,
                                             const int64_t *__restrict__ acrd, const int64_t *__restrict__ bpos,
                                             const int32_t *__restrict__ bcrd, const int32_t *__restrict__ hub_id,
                                             const uint32_t *__restrict__ hub_bm, int *s_long, unsigned *s_n,
                                             unsigned *s_ctl)
{
    int *s_hub = s_long;                               // one list after the other
    const int64_t ae = apos[r + 1];
    int64_t p = apos[r];
    for (bool first = true; first || (hub_id && p < ae); first = false) {
        const int n = hub_id ? hub_list(&p, ae, acrd, hub_id, s_hub, s_n) : 0;
        for (int g = threadIdx.x; g < stride / 4; g += BM_THREADS) {
            uint4 v = first ? make_uint4(0, 0, 0, 0) : ((uint4 *)bm)[g];
#pragma unroll 8
            for (int i = 0; i < n; i++) {
                const uint4 o = __ldg((const uint4 *)(hub_bm + (size_t)s_hub[i] * stride) + g);
                v.x |= o.x; v.y |= o.y; v.z |= o.z; v.w |= o.w;
            }
            ((uint4 *)bm)[g] = v;
        }
    }
    __syncthreads();
    for_each_product<WALK_DEPTH>(r, 0u, 1u, apos, acrd, nullptr, bpos, bcrd, nullptr, hub_id, s_long, s_ctl,
                     [&](int32_t j, double, double) { atomicOr(&bm[j >> 5], 1u << (j & 31)); });
    __syncthreads();
}

// Four CTAs on an SM: rows of a few thousand products wait for barriers and for loads, so that registers for a fourth CTA are worth more than
// the 24 bytes they put on the stack.  Both calls with three (39 registers) and four (32): 200,000 rows of 2000 products in 100,000
// columns 8.13 and 7.64 ms (7.89 before there were hubs), R-MAT scale 18 squared 23.3 and 22.3.
__global__ void __launch_bounds__(BM_THREADS, 4)
hub_symbolic_kernel(unsigned nlist, const int32_t *__restrict__ list, Hubs hb, const int64_t *__restrict__ apos,
                    const int64_t *__restrict__ acrd, const int64_t *__restrict__ bpos, int64_t *__restrict__ cnt,
                    uint32_t *__restrict__ bm_store)
{
    extern __shared__ __align__(16) uint32_t s_dyn[];
    __shared__ unsigned s_warp[BM_THREADS / 32];
    __shared__ int s_long[LONG_LIST];
    __shared__ unsigned s_ctl[2], s_n;
    const int32_t *id = *hb.count ? hb.id : nullptr;
    for (unsigned it = blockIdx.x; it < nlist; it += gridDim.x) {
        const int64_t r = list[it];
        hub_mark_row(s_dyn, hb.stride, r, apos, acrd, bpos, hb.crd, id, hb.bm, s_long, &s_n, s_ctl);
        unsigned c = 0;
        uint4 *keep = bm_store ? (uint4 *)(bm_store + (size_t)it * hb.stride) : nullptr;
        for (int g = threadIdx.x; g < hb.stride / 4; g += BM_THREADS) {
            const uint4 v = ((const uint4 *)s_dyn)[g];
            c += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
            if (keep) __stcs(keep + g, v);
        }
        const unsigned total = block_sum_u32(c, s_warp);
        if (threadIdx.x == 0) cnt[r] = total;
    }
}

// --------------------------------------------------------------------------
// Elementwise CSR .* CSR: two-pointer intersection, one thread per row.
// --------------------------------------------------------------------------
template <bool NUMERIC>
__global__ void __launch_bounds__(256)
elews_ss_kernel(int64_t nrows, const int64_t *__restrict__ apos, const int64_t *__restrict__ acrd,
                const double *__restrict__ aval, const int64_t *__restrict__ bpos,
                const int64_t *__restrict__ bcrd, const double *__restrict__ bval,
                int64_t *__restrict__ cnt, const int64_t *__restrict__ cpos,
                int64_t *__restrict__ ccrd, double *__restrict__ cval)
{
    int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= nrows) return;
    int64_t p = apos[r], pe = apos[r + 1], q = bpos[r], qe = bpos[r + 1];
    int64_t n = 0, at = NUMERIC ? cpos[r] : 0;
    while (p < pe && q < qe) {
        int64_t ca = acrd[p], cb = bcrd[q];
        if (ca == cb) {
            if (NUMERIC) { ccrd[at + n] = ca; cval[at + n] = aval[p] * bval[q]; }
            n++;
        }
        if (ca <= cb) p++;
        if (cb <= ca) q++;
    }
    if (!NUMERIC) cnt[r] = n;
}

// --------------------------------------------------------------------------
// Host side
// --------------------------------------------------------------------------
static int64_t register_plan(Plan *p)
{
    std::lock_guard<std::mutex> lk(g_plans_mu);
    int64_t h = g_next_handle++;
    g_plans[h] = p;
    return h;
}

static Plan *find_plan(int64_t h, bool remove)
{
    std::lock_guard<std::mutex> lk(g_plans_mu);
    auto it = g_plans.find(h);
    if (it == g_plans.end()) return nullptr;
    Plan *p = it->second;
    if (remove) g_plans.erase(it);
    return p;
}

static int bitmap_grid(unsigned nlist, size_t smem_bytes)
{
    int per_sm = smem_bytes ? (int)((220 * 1024) / (smem_bytes + 1024)) : 2;
    if (per_sm < 1) per_sm = 1;
    if (per_sm > 2048 / BM_THREADS) per_sm = 2048 / BM_THREADS;
    int64_t g = (int64_t)sm_count() * per_sm;
    if (g > nlist) g = nlist;
    return (int)(g < 1 ? 1 : g);
}

static unsigned cnt_grid(unsigned rows)
{
    const unsigned cap = (unsigned)sm_count() * 16;
    return rows < cap ? rows : cap;
}

template <bool NUMERIC>
static int launch_mid(const Plan *p, unsigned grid, int64_t *ccrd, double *cval, cudaStream_t st)
{
    const size_t smem = mid_smem(p->words, NUMERIC);
    const bool many = p->words >= MID_MANY_WORDS;
    auto kernel = many ? mid_rows_kernel<256, NUMERIC> : mid_rows_kernel<128, NUMERIC>;
    CB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CB_CUDA(launch_behind(kernel, dim3(grid), many ? 256 : 128, smem, st, p->bin_counts + 2, p->list3, p->words, p->apos, p->acrd,
                          p->aval, p->bpos, p->bcrd32, p->bval, p->semi, p->cnt, p->cpos, ccrd, cval));
    return 0;
}

// CTAs of the numeric kernel on an SM, and the columns of a warp's stage that are left room for where columns need a look-up (mapped)
struct NumericCtas {
    size_t per_sm, stage;
};
static NumericCtas numeric_ctas(int64_t words, bool mapped)
{
    // three CTAs are what the registers leave room for; coordinates are staged in the shared memory that is left
    // (200,000 rows of up to 60: 4.2 ms with three and what is left, 5.2 with a full stage and two).  Columns that need no
    // look-up are written as they are found (3.3 against 3.5).  A stage of a few columns is worth less than a CTA: 2000 rows of
    // 100,000 products in 450,000 columns 2.39 ms with three CTAs and 43 columns, 2.27 with two and 512.
    const size_t smem = (size_t)words * sizeof(uint32_t) * 2, sm = (size_t)228 * 1024, own = 6 * 1024;
    if (smem > BM_SMEM_LIMIT) return {0, 0};
    size_t per_sm = sm / (smem + own);
    per_sm = per_sm < 1 ? 1 : per_sm > 3 ? 3 : per_sm;
    auto stage_of = [&](size_t ctas) { return (sm / ctas - own - smem) / (BM_THREADS / 32 * 4); };
    while (mapped && per_sm > 1 && stage_of(per_sm) < STAGE_MIN) per_sm--;
    const size_t stage = mapped ? stage_of(per_sm) : 0;
    return {per_sm, stage > BM_DENSE_ROW ? (size_t)BM_DENSE_ROW : stage};
}

// Prepares B's long rows (p->hubs stays null where the columns that B stores are too many, or where these keep their numbers and B has no long
// rows or A names few).  Synchronises.  In vain that costs 20 to 65 us.
static int hub_prepare(Plan *p, int64_t nrows, int64_t nnz_a, cudaStream_t st)
{
    Hubs *hb = new Hubs();
    memset(hb, 0, sizeof(Hubs));
    p->hubs = hb;                                      // freed with the plan
    const int64_t words = ceil_div(p->ncols, 32);
    auto pad = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
    const size_t b_bits = pad((size_t)words * 4), b_map = pad((size_t)p->ncols * 4), b_crd = pad((size_t)p->nnz_b * 4 + 16);
    auto without = [&]() {                             // no hubs: bin 2 as it is
        if (hb->mem) cudaFreeAsync(hb->mem, st);
        delete hb;
        p->hubs = nullptr;
        (void)cudaGetLastError();
        return 0;
    };
    char *m = nullptr;
    if (cudaMallocAsync((void **)&m, 256 + 2 * b_bits + b_map + b_crd, st) != cudaSuccess) return without();
    hb->mem = m;
    hb->prep = (HubPrep *)m;
    hb->count = (unsigned *)(m + 128);
    hb->present = (uint32_t *)(m + 256);
    hb->before = (int32_t *)(m + 256 + b_bits);
    hb->colmap = (int32_t *)(m + 256 + 2 * b_bits);
    hb->crd = (int32_t *)(m + 256 + 2 * b_bits + b_map);
    CB_CUDA(cudaMemsetAsync(m, 0, 256 + b_bits, st));
    // the kernel walks A as well as B: a tall A times a small B has its work there (100,000 rows of 300 times 600 of 6, both calls
    // 15.6 ms with the one CTA that B alone would get)
    const int64_t least = ceil_div(nnz_a > p->nnz_b ? nnz_a : p->nnz_b, 4096), most = (int64_t)sm_count() * 2;
    const unsigned grid = (unsigned)(least < most ? least : most);
    if (words * 4 <= 96 * 1024) {
        CB_CUDA(cudaFuncSetAttribute(hub_present_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(words * 4)));
        hub_present_kernel<true><<<grid, 1024, (size_t)words * 4, st>>>(p->nnz_b, p->bcrd32, words, hb->present, nrows, p->apos,
                                                                      p->acrd, p->bpos, hb->prep);
    } else {
        hub_present_kernel<false><<<grid, 1024, 0, st>>>(p->nnz_b, p->bcrd32, words, hb->present, nrows, p->apos, p->acrd,
                                                          p->bpos, hb->prep);
    }
    CB_LAUNCH_CHECK();
    hub_before_kernel<<<1, 1024, 0, st>>>(words, hb->present, hb->before, hb->prep);
    CB_LAUNCH_CHECK();
    HubPrep prep;
    {
        PinnedWords host;
        if (!host.p) return fail("spgemm: no page-locked memory");
        CB_CUDA(cudaMemcpyAsync(host.p, hb->prep, sizeof(prep), cudaMemcpyDeviceToHost, st));
        CB_CUDA(cudaStreamSynchronize(st));
        memcpy(&prep, host.p, sizeof(prep));
    }
    // the look-up of every coordinate costs what an eighth of the words does (200,000 columns, all stored: 3.3 -> 4.0 ms), and more where rows
    // have few products for their words: HUB_PRODUCTS
    const bool much = prep.products / HUB_PRODUCTS >= (long long)p->n2 * words;
    const int64_t stored = (int64_t)prep.ncols * 8;
    const bool renumber = stored <= p->ncols * 5 ||
                          (stored <= p->ncols * 7 &&
                           (much || numeric_ctas(ceil_div((int64_t)prep.ncols, 32), true).per_sm > numeric_ctas(words, false).per_sm));
    hb->words = (int)(renumber ? ceil_div((int64_t)prep.ncols, 32) : words);
    hb->stride = (hb->words + 3) & ~3;
    hb->nrows_b = prep.nrows_b;
    const int64_t entries = hb->words / 8 > HUB_MIN_ENTRIES ? hb->words / 8 : HUB_MIN_ENTRIES;
    if (hb->words > HUB_MAX_WORDS || (!renumber && (!much || prep.longest < entries))) return without();
    if (renumber) {
        hub_renumber_kernel<<<(unsigned)sm_count() * 8, 256, 0, st>>>(p->nnz_b, p->bcrd32, words, hb->present, hb->before, hb->crd,
                                                                      hb->colmap);
        CB_LAUNCH_CHECK();
    } else {
        hb->crd = p->bcrd32;
        hb->colmap = nullptr;
    }
    const size_t each = (size_t)hb->stride * 4 + 4;
    size_t cap = (size_t)(p->nnz_b / entries) + 1;
    if (cap > HUB_MEMORY / each) cap = HUB_MEMORY / each;
    hb->cap = (unsigned)cap;
    const size_t b_id = pad((size_t)hb->nrows_b * 4), b_rows = pad(cap * 4);
    m = nullptr;
    if (cudaMallocAsync((void **)&m, b_id + b_rows + cap * hb->stride * 4, st) != cudaSuccess) return without();
    hb->mem2 = m;
    hb->id = (int32_t *)m;
    int32_t *rows = (int32_t *)(m + b_id);
    hb->bm = (uint32_t *)(m + b_id + b_rows);
    hub_find_kernel<<<(unsigned)ceil_div(hb->nrows_b, 256), 256, 0, st>>>(hb->nrows_b, p->bpos, entries, hb->cap, hb->count, hb->id,
                                                                        rows);
    CB_LAUNCH_CHECK();
    CB_CUDA(cudaFuncSetAttribute(hub_build_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, hb->stride * 4));
    hub_build_kernel<<<(unsigned)(cap < (size_t)sm_count() * 2 ? cap : (size_t)sm_count() * 2), 512, (size_t)hb->stride * 4, st>>>(
        hb->count, hb->cap, rows, p->bpos, hb->crd, hb->stride, hb->bm);
    CB_LAUNCH_CHECK();
    return 0;
}

int spgemm_symbolic(int64_t nrows, int64_t ncols_b, int64_t nnz_b, const int64_t *apos,
                    const int64_t *acrd, const double *aval, const int64_t *bpos,
                    const int64_t *bcrd, const double *bval, const int64_t *mpos,
                    const int64_t *mcrd, int semiring, int64_t *cpos, int64_t *nnz_host,
                    int64_t *handle_out, cudaStream_t st)
{
    if (ncols_b >= 0x7fffffffLL || nrows >= 0x7fffffffLL)
        return fail("spgemm: more than 2^31-1 rows or columns is not supported");
    if (((uintptr_t)bcrd & 15) != 0) return fail("spgemm: B.crd must be 16-byte aligned");
    CB_TRY(pool_setup());
    Plan *p = new Plan();
    memset(p, 0, sizeof(Plan));
    p->kind = 0; p->nrows = nrows; p->ncols = ncols_b; p->nnz_b = nnz_b;
    p->last = st;
    p->apos = apos; p->acrd = acrd; p->aval = aval; p->bpos = bpos; p->bcrd = bcrd; p->bval = bval;
    p->mpos = mpos; p->mcrd = mpos ? mcrd : nullptr; p->semi = semiring;
    p->cpos = cpos;
    p->words = (int)ceil_div(ncols_b, 32);
    int rc = 0;
#define STEP(expr) do { if (!rc) rc = (expr); } while (0)
#define STEP_CUDA(expr) do { if (!rc) { cudaError_t e_ = (expr); if (e_ != cudaSuccess) rc = fail("%s failed: %s", #expr, cudaGetErrorString(e_)); } } while (0)
    if (mpos) {
        STEP(masked_symbolic(nrows, ncols_b, nnz_b, apos, acrd, bpos, bcrd, mpos, mcrd, cpos, &p->masked, st));
        if (!rc && p->masked) {
            PinnedWords words;
            if (!rc && !words.p) rc = fail("spgemm: no page-locked memory");
            STEP_CUDA(cudaMemcpyAsync(words.p, cpos + nrows, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
            STEP_CUDA(cudaMemcpyAsync((int64_t *)words.p + 1, masked_checks(p->masked), 3 * sizeof(int), cudaMemcpyDeviceToHost, st));
            STEP_CUDA(cudaStreamSynchronize(st));
            if (rc) { plan_free(p, st); return rc; }
            const int *ok = (const int *)((int64_t *)words.p + 1);
            if (ok[0] == 0 && ok[1] == ok[2]) {
                p->nnz_c = *(int64_t *)words.p;
                *nnz_host = p->nnz_c;
                *handle_out = register_plan(p);
                return 0;
            }
            masked_free(p->masked, st);    // rows of B that do not ascend strictly: push
            p->masked = nullptr;
        }
    }
    auto pad = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
    const size_t b_cnt = pad(((size_t)nrows + 1) * 8), b_crd = pad((size_t)nnz_b * 4 + 8), b_list = pad((size_t)nrows * 4);
    char *mem = nullptr;
    const bool mid = !mpos && mid_smem(p->words, true) <= MID_SMEM;
    STEP(dev_alloc(&mem, 256 + b_cnt + b_crd + (mid ? 3 : 2) * b_list, st));
    p->mem = mem;
    p->bin_counts = (unsigned *)mem;
    p->cnt = (int64_t *)(mem + 256);
    p->bcrd32 = (int32_t *)(mem + 256 + b_cnt);
    p->list1 = (int32_t *)(mem + 256 + b_cnt + b_crd);
    p->list2 = (int32_t *)((char *)p->list1 + b_list);
    p->list3 = (int32_t *)((char *)p->list2 + b_list);
    STEP_CUDA(cudaMemsetAsync(p->bin_counts, 0, 3 * sizeof(unsigned), st));
    if (!rc && nrows + nnz_b > 0) {
        const int passes = nrows >= (int64_t)sm_count() * 8 * BIN_ROWS ? 4 : 1;
        const int64_t row_ctas = ceil_div(nrows, (int64_t)BIN_PASS * passes), ctas = row_ctas + ceil_div(nnz_b, NARROW_PART);
        if (ctas > 0x7fffffffLL) rc = fail("spgemm: too many entries");
        if (!rc)
            bin_rows_kernel<<<(unsigned)ctas, BIN_THREADS, 0, st>>>(nrows, passes, (unsigned)row_ctas, apos, acrd, bpos, mpos,
                                                                   mid ? MID_ROW_MAX : HASH_ROW_MAX, p->cnt, p->list1, p->list2,
                                                                   p->list3, p->bin_counts, bcrd, p->bcrd32, nnz_b);
        STEP_CUDA(cudaGetLastError());
    }
    PinnedWords words;
    if (!rc && !words.p) rc = fail("spgemm: no page-locked memory");
    unsigned *counts = (unsigned *)words.p;
    // The bitmaps of the bin-2 rows are kept for the numeric call, so their number is needed to allocate them: after a
    // synchronisation, unless bitmaps for every row are small change (then the kernels read the bin sizes themselves).
    p->n1 = p->n2 = (unsigned)nrows;
    p->n3 = mid ? (unsigned)nrows : 0;
    bool counted = false;
    int64_t nnz_a = 0;
    if ((size_t)nrows * p->words * 4 > BM_STORE_SMALL) {
        STEP_CUDA(launch_behind(publish_kernel, dim3(1), 1, 0, st, p->bin_counts, apos + nrows, counts));
        STEP_CUDA(cudaStreamSynchronize(st));
        if (!rc) { p->n1 = counts[0]; p->n2 = counts[1]; p->n3 = counts[2]; nnz_a = *(int64_t *)(counts + 4); counted = true; }
    }
    if (!rc && p->n1) {
        unsigned grid = (unsigned)ceil_div(p->n1, HASH_WARPS);
        unsigned cap = (unsigned)sm_count() * 16;
        if (grid > cap) grid = cap;
        if (!mpos && ncols_b <= FEW_COLUMNS)
            STEP_CUDA(launch_behind(few_columns_kernel, dim3(grid), HASH_WARPS * 32, (size_t)p->words * HASH_WARPS * 4, st, p->bin_counts,
                                    p->list1, p->words, apos, acrd, bpos, p->bcrd32, p->cnt));
        else
            STEP_CUDA(launch_behind(hash_rows_kernel<false, false>, dim3(grid), HASH_WARPS * 32, 0, st, p->bin_counts, p->list1, apos, acrd,
                                aval, bpos, p->bcrd32, bval, mpos, p->mcrd, p->semi, p->cnt, nullptr, nullptr, nullptr));
    }
    if (!rc && p->n3) STEP(launch_mid<false>(p, cnt_grid(p->n3), nullptr, nullptr, st));
    const size_t hub_bytes = counted && !mpos ? (size_t)p->n2 * p->words * 4 : 0;
    if (hub_bytes >= HUB_WORK && hub_bytes / HUB_ENTRY >= (size_t)nnz_b && ncols_b <= HUB_MAX_COLS && nnz_b < 0x7fffffffLL)
        STEP(hub_prepare(p, nrows, nnz_a, st));
    if (!rc && p->n2) {
        size_t store = (size_t)p->n2 * (p->hubs ? p->hubs->stride : p->words) * sizeof(uint32_t);
        // the symbolic pass's bitmaps are kept for the numeric pass while they fit the budget
        // (COMET_B200_SPGEMM_BITMAP_GB overrides it; 0 makes the numeric pass mark its rows again)
        size_t budget = BM_STORE_BUDGET;
        if (const char *e = getenv("COMET_B200_SPGEMM_BITMAP_GB")) budget = (size_t)(atof(e) * (double)(1ull << 30));
        if (store <= budget) {
            cudaError_t e = cudaMallocAsync((void **)&p->bm_store, store, st);
            if (e != cudaSuccess) { p->bm_store = nullptr; (void)cudaGetLastError(); }
        }
        size_t smem = (size_t)(p->hubs ? p->hubs->stride : p->words) * sizeof(uint32_t);
        if (p->hubs) {
            STEP_CUDA(cudaFuncSetAttribute(hub_symbolic_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            if (!rc)
                hub_symbolic_kernel<<<bitmap_grid(p->n2, smem + 5 * 1024), BM_THREADS, smem, st>>>(p->n2, p->list2, *p->hubs, apos,
                                                                                                  acrd, bpos, p->cnt, p->bm_store);
        } else if (2 * smem <= BM_SMEM_LIMIT) {
            int grid = bitmap_grid(p->n2, smem);
            STEP_CUDA(cudaFuncSetAttribute(bitmap_symbolic_kernel<true>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            STEP_CUDA(launch_behind(bitmap_symbolic_kernel<true>, dim3(grid), BM_THREADS, smem, st, p->bin_counts + 1, p->list2,
                                    p->words, nullptr, apos, acrd, bpos, p->bcrd32, mpos, p->mcrd, p->cnt, p->bm_store));
        } else {
            int grid = bitmap_grid(p->n2, 0);
            void *gbm = nullptr;
            STEP(scratch(SLOT_BITMAP, (size_t)grid * 2 * smem, &gbm));
            if (!rc)
                bitmap_symbolic_kernel<false><<<grid, BM_THREADS, 0, st>>>(
                    p->bin_counts + 1, p->list2, p->words, (uint32_t *)gbm, apos, acrd, bpos, p->bcrd32, mpos,
                    p->mcrd, p->cnt, p->bm_store);
        }
        STEP_CUDA(cudaGetLastError());
    }
    STEP(exclusive_scan_i64(p->cnt, cpos, nrows, st));
    STEP_CUDA(launch_behind(publish_kernel, dim3(1), 1, 0, st, p->bin_counts, cpos + nrows, counts));
    STEP_CUDA(cudaStreamSynchronize(st));
    if (!rc) {
        p->n1 = counts[0]; p->n2 = counts[1]; p->n3 = counts[2];
        p->nnz_c = *(int64_t *)(counts + 4);
    }
#undef STEP
#undef STEP_CUDA
    if (rc) { plan_free(p, st); return rc; }
    *nnz_host = p->nnz_c;
    *handle_out = register_plan(p);
    return 0;
}

int elews_ss_symbolic(int64_t nrows, const int64_t *apos, const int64_t *acrd, const double *aval,
                      const int64_t *bpos, const int64_t *bcrd, const double *bval, int64_t *cpos,
                      int64_t *nnz_host, int64_t *handle_out, cudaStream_t st)
{
    CB_TRY(pool_setup());
    Plan *p = new Plan();
    memset(p, 0, sizeof(Plan));
    p->kind = 1; p->nrows = nrows;
    p->last = st;
    p->apos = apos; p->acrd = acrd; p->aval = aval; p->bpos = bpos; p->bcrd = bcrd; p->bval = bval;
    p->cpos = cpos;
    int rc = dev_alloc(&p->cnt, (size_t)nrows + 1, st);
    p->mem = p->cnt;
    if (!rc && nrows > 0) {
        elews_ss_kernel<false><<<(unsigned)ceil_div(nrows, 256), 256, 0, st>>>(
            nrows, apos, acrd, aval, bpos, bcrd, bval, p->cnt, nullptr, nullptr, nullptr);
        if (cudaGetLastError() != cudaSuccess) rc = fail("elews symbolic launch failed");
    }
    if (!rc) rc = exclusive_scan_i64(p->cnt, cpos, nrows, st);
    if (!rc && cudaMemcpyAsync(&p->nnz_c, cpos + nrows, sizeof(int64_t), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        rc = fail("elews symbolic: copy of nnz failed");
    if (!rc && cudaStreamSynchronize(st) != cudaSuccess) rc = fail("elews symbolic: synchronize failed");
    if (rc) { plan_free(p, st); return rc; }
    *nnz_host = p->nnz_c;
    *handle_out = register_plan(p);
    return 0;
}

int sparse_out_numeric(int64_t handle, int64_t *ccrd, double *cval, int keep, cudaStream_t st)
{
    Plan *p = find_plan(handle, !keep);
    if (!p) return fail("numeric phase: unknown handle %lld", (long long)handle);
    p->last = st;
    int rc = 0;
    if (p->masked) {
        rc = masked_numeric(p->masked, p->aval, p->bval, p->mcrd, p->semi, ccrd, cval, st);
    } else if (p->kind == 1) {
        if (p->nrows > 0) {
            elews_ss_kernel<true><<<(unsigned)ceil_div(p->nrows, 256), 256, 0, st>>>(
                p->nrows, p->apos, p->acrd, p->aval, p->bpos, p->bcrd, p->bval, nullptr, p->cpos, ccrd,
                cval);
            if (cudaGetLastError() != cudaSuccess) rc = fail("elews numeric launch failed");
        }
    } else {
        if (p->n1) {
            unsigned grid = (unsigned)ceil_div(p->n1, HASH_WARPS);
            unsigned cap = (unsigned)sm_count() * 16;
            if (grid > cap) grid = cap;
            if (!p->mpos) {
                auto k = p->ncols <= (1 << 24) ? short_rows_kernel<false> : short_rows_kernel<true>;
                k<<<grid, HASH_WARPS * 32, 0, st>>>(p->bin_counts, p->list1, p->apos, p->acrd, p->aval, p->bpos, p->bcrd32,
                                                    p->bval, p->semi, p->cpos, ccrd, cval);
            } else {
                auto k = p->ncols <= (1 << 24) ? hash_rows_kernel<true, false> : hash_rows_kernel<true, true>;
                k<<<grid, HASH_WARPS * 32, 0, st>>>(p->bin_counts, p->list1, p->apos, p->acrd, p->aval, p->bpos, p->bcrd32,
                                                    p->bval, p->mpos, p->mcrd, p->semi, nullptr, p->cpos, ccrd, cval);
            }
            if (cudaGetLastError() != cudaSuccess) rc = fail("spgemm numeric (hash) launch failed");
        }
        if (!rc && p->n3) rc = launch_mid<true>(p, cnt_grid(p->n3), ccrd, cval, st);
        if (!rc && p->n2) {
            const int words = p->hubs ? p->hubs->words : p->words, stride = p->hubs ? p->hubs->stride : p->words;
            const int32_t *colmap = p->hubs ? p->hubs->colmap : nullptr, *bcrd32 = p->hubs ? p->hubs->crd : p->bcrd32;
            size_t smem = (size_t)words * sizeof(uint32_t) * 2;
            if (smem <= BM_SMEM_LIMIT) {
                // full occupancy grid even for few rows: teams give every CTA work
                const NumericCtas ctas = numeric_ctas(words, colmap != nullptr);
                const size_t stage_n = ctas.stage;
                smem += stage_n * (BM_THREADS / 32 * 4);
                const int grid = sm_count() * (int)ctas.per_sm;
                // team size of a row = its output entries * 8 bytes * CTAs in flight / budget
                double budget_mb = 60.0;                 // measured best on R-MAT scale 18 (25 / 40 / 60 / 160 MB)
                if (const char *e = getenv("COMET_B200_SPGEMM_TEAM_MB")) budget_mb = atof(e);
                if (budget_mb < 0.001) budget_mb = 0.001;
                const bool few = p->n2 < (unsigned)grid * TEAM_FEW;
                const double alone_to = few ? 1.0 : TEAM_ALONE;
                const double per_entry = 8.0 * (few ? bitmap_grid(0xffffffffu, (size_t)words * 8) : grid) / (budget_mb * 1048576.0);
                // no row of so few columns wants a team: two launches less
                const bool alone = (double)words * 32 * per_entry <= alone_to;
                const size_t cap = (size_t)p->n2 + (size_t)((double)p->nnz_c * per_entry) + 64;
                void *tm = nullptr;
                rc = cap > 0xfffffff0u ? fail("spgemm numeric: too many team items")
                                       : scratch(SLOT_TEAMS, sizeof(TeamHeader) + cap * sizeof(uint64_t), &tm);
                TeamHeader *th = (TeamHeader *)tm;
                uint64_t *items = (uint64_t *)((char *)tm + sizeof(TeamHeader));
                if (!rc && cudaMemsetAsync(th, 0, sizeof(TeamHeader), st) != cudaSuccess)
                    rc = fail("spgemm numeric: clearing the team header failed");
                if (!rc) {
                    if (alone) items = nullptr;
                    else
                        team_items_kernel<<<(unsigned)ceil_div(p->n2, 256), 256, 0, st>>>(
                            p->n2, p->list2, p->cpos, per_entry, alone_to, th, items, (unsigned)cap);
                    if (!alone) launch_behind(team_clear_kernel, dim3((unsigned)sm_count() * 8), 256, 0, st, th, items, (unsigned)cap, p->list2,
                                  p->cpos, p->semi, cval);
                    const bool times = p->semi == COMET_B200_PLUS_TIMES;
                    auto kernel = colmap ? (times ? bitmap_numeric_kernel<true, true, true> : bitmap_numeric_kernel<true, false, true>)
                                         : (times ? bitmap_numeric_kernel<true, true, false> : bitmap_numeric_kernel<true, false, false>);
                    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
                    launch_behind(kernel, dim3(grid), BM_THREADS, smem, st, p->n2, p->list2, words, stride, (unsigned)stage_n, colmap,
                                  nullptr, p->apos, p->acrd, p->aval, p->bpos, bcrd32, p->bval, p->mpos, p->mcrd, p->semi, p->bm_store,
                                  p->cpos, ccrd, cval, th, items);
                }
            } else {
                int grid = bitmap_grid(p->n2, 0);
                void *gbm = nullptr;
                rc = scratch(SLOT_BITMAP, (size_t)grid * smem, &gbm);
                if (!rc)
                    bitmap_numeric_kernel<false, false, false><<<grid, BM_THREADS, 0, st>>>(
                        p->n2, p->list2, words, stride, 0, nullptr, (uint32_t *)gbm, p->apos, p->acrd, p->aval, p->bpos,
                        bcrd32, p->bval, p->mpos, p->mcrd, p->semi, p->bm_store, p->cpos, ccrd, cval, nullptr,
                        nullptr);
            }
            if (!rc && cudaGetLastError() != cudaSuccess) rc = fail("spgemm numeric (bitmap) launch failed");
        }
    }
    if (!keep) plan_free(p, st);
    return rc;
}

void destroy_plan(int64_t handle)
{
    // a numeric launch of a kept plan may still be running: free behind it, in its own stream's order
    Plan *p = find_plan(handle, true);
    if (p) plan_free(p, p->last);
}

}  // namespace cb200

extern "C" {

int32_t comet_b200_dev_spgemm_symbolic_f64_i64(int64_t nrows, int64_t ncols_b, int64_t nnz_b,
                                               const int64_t *apos, const int64_t *acrd,
                                               const double *aval, const int64_t *bpos,
                                               const int64_t *bcrd, const double *bval,
                                               const int64_t *mpos, const int64_t *mcrd,
                                               int32_t semiring, int64_t *cpos, int64_t *nnz_host,
                                               int64_t *handle_out, void *stream)
{
    cb200::clear_error();
    if (semiring < COMET_B200_PLUS_TIMES || semiring > COMET_B200_ANY_PAIR)
        return cb200::fail("spgemm: unsupported semiring %d", semiring);
    return cb200::spgemm_symbolic(nrows, ncols_b, nnz_b, apos, acrd, aval, bpos, bcrd, bval, mpos, mcrd,
                                  semiring, cpos, nnz_host, handle_out, (cudaStream_t)stream);
}

int32_t comet_b200_dev_elews_mul_sparse_sparse_symbolic_f64_i64(
    int64_t nrows, const int64_t *apos, const int64_t *acrd, const double *aval,
    const int64_t *bpos, const int64_t *bcrd, const double *bval, int64_t *cpos, int64_t *nnz_host,
    int64_t *handle_out, void *stream)
{
    cb200::clear_error();
    return cb200::elews_ss_symbolic(nrows, apos, acrd, aval, bpos, bcrd, bval, cpos, nnz_host,
                                    handle_out, (cudaStream_t)stream);
}

int32_t comet_b200_dev_spgemm_numeric_f64_i64(int64_t handle, int64_t *ccrd, double *cval,
                                              int32_t keep, void *stream)
{
    cb200::clear_error();
    return cb200::sparse_out_numeric(handle, ccrd, cval, keep, (cudaStream_t)stream);
}

void comet_b200_handle_destroy(int64_t handle) { cb200::destroy_plan(handle); }

}
