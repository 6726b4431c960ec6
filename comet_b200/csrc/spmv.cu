// SpMV  y[a] = y[a] (+) sum_b A[a,b] (x) x[b]   (CSR / DCSR rows, f64 values, i64 indices).
//
// A group of T lanes (T chosen from the mean row length) walks one row with
// 128-bit loads of crd and val (two entries per load), the next row's pointers on their way.
//
// One launch of lane groups, while A's path of entries and row ends has fewer tiles of 2^11 steps than the chip has SMs; no
// scratch memory.  Rows of more than 16 T entries are left to the end of the CTA, where a warp, or for very long ones all 256
// threads, walk them.
// From there to 2^20 entries: the tiles, a CTA each, in one launch and without scratch memory too.  A power-law matrix of this
// size has its hub rows in a CTA or two of lane groups, which the launch waits for.
// Both give the same sums to the bit in every call.
// From 2^20 on: rows longer than DEFER_ROW entries are cut into chunks that
// go to a work list in scratch memory, and a second launch gives each chunk to
// a warp that adds its partial sum to y with one f64 atomic -- on a power-law
// matrix the long rows sit next to each other and would otherwise all land in
// the first few CTAs.
// From 2^23 on a first kernel looks for long rows (3 us): without them the lane groups take the call and need no list, with
// them planned tiles do.
//
// Microseconds of back-to-back calls in a CUDA graph, lane groups in one launch / tiles in one launch:
//   even rows of 16:  60,000 entries 2.8 / 5.5    262,144 3.8 / 6.2    600,000 5.3 / 8.6    960,000 7.3 / 10.3
//   rows of 0 to 20:  500,000 6.5 / 7.1           rows of 60: 300,000 3.8 / 5.8
//   R-MAT:            25,500 8 / 6.3    120,000 17 / 8.4    228,000 20 / 8.1    468,000 51 / 8.8    728,000 88 / 10.9
//   100,000 rows of 4 and one of 300,000: 269 / 10.3
// (launched one by one the calls are 8 to 10 apart either way).  Only the device knows how long the rows are, and tiles are
// the ones that no matrix makes slow, so they take over as soon as they fill the chip.
// With a list / planned tiles: even rows 3.2 M entries 25 / 29, 36 M 182 / 232; R-MAT 3 M 43 / 28, 16 M 133 / 107.
//
// Bound: HBM, 8(n+1) + 16 nnz + 8 ncols + 8 nrows bytes per call, and the L1's rate for the gathered x, one line per entry
// (57 us at one line a clock for 16 M entries of a power-law matrix).  Row pointers fetched a row ahead: R-MAT scale 20
// 146 -> 133 us, 36 M entries in even rows 202 -> 182.
#include <atomic>

#include "common.cuh"
#include "stream.cuh"

namespace cb200 {

static const int SPMV_THREADS = 256;
static const int SPMV_PASSES = 4;          // most rows per lane group per CTA (fewer on small matrices)
static const int64_t LONG_ROW = 2048;
static const int64_t DEFER_ROW = 64;       // with a work list: rows above this go to it
static const int64_t SPMV_CHUNK = 256;     // entries per work-list chunk
static const int64_t DEFER_MIN_NNZ = 1 << 20;
static const int64_t LOOK_MIN_NNZ = 1 << 23;      // the look and two launches that return at once: 5 us, too much of 40
static const int TILE_ITEMS = 8;           // steps per thread of a tile's CTA
static const int TILE_SHIFT = 11;          // 2^11 per tile
static const int ONCE_PAST = SPMV_THREADS; // one launch: a row that ends so many steps behind a tile is not cut
static const int ONCE_TILES = 1024;        // one launch: most tiles
static const int ONCE_SLOTS = 16;          // one launch: calls in a row that use memory of their own

template <bool PAIR>
__device__ __forceinline__ double combine(double a, double b)
{
    return PAIR ? 1.0 : a * b;
}

// Partial dot product of one row over entries handled by this lane; `nl` lanes
// share the row, lane index `l`.  VEC: crd/val are 16-byte aligned arrays.
template <bool PAIR, bool VEC>
__device__ __forceinline__ double row_partial(const int64_t *__restrict__ crd,
                                              const double *__restrict__ val,
                                              const double *__restrict__ x, int64_t s, int64_t e,
                                              int l, int nl)
{
    double sum0 = 0.0, sum1 = 0.0;
    if (VEC) {
        for (int64_t q = (s & ~(int64_t)1) + 2 * l; q < e; q += 2 * nl) {
            if (q >= s && q + 1 < e) {
                longlong2 c = __ldcs((const longlong2 *)(crd + q));
                double2 v = __ldcs((const double2 *)(val + q));
                sum0 += combine<PAIR>(v.x, PAIR ? 0.0 : __ldg(x + c.x));
                sum1 += combine<PAIR>(v.y, PAIR ? 0.0 : __ldg(x + c.y));
            } else {
                if (q >= s) sum0 += combine<PAIR>(val[q], PAIR ? 0.0 : __ldg(x + crd[q]));
                if (q + 1 < e) sum1 += combine<PAIR>(val[q + 1], PAIR ? 0.0 : __ldg(x + crd[q + 1]));
            }
        }
    } else {
        for (int64_t q = s + l; q < e; q += nl)
            sum0 += combine<PAIR>(val[q], PAIR ? 0.0 : __ldg(x + crd[q]));
    }
    return sum0 + sum1;
}

template <int T, bool PAIR, bool VEC>
__global__ void __launch_bounds__(SPMV_THREADS)
spmv_kernel(int64_t nrows, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
            const int64_t *__restrict__ crd, const double *__restrict__ val,
            const double *__restrict__ x, double *__restrict__ y, int accumulate, int passes,
            WorkHeader *hdr, Chunk *chunks, unsigned chunk_cap, LongRows lr)
{
    constexpr int GROUPS = SPMV_THREADS / T;
    constexpr int ROWS = GROUPS * SPMV_PASSES;
    __shared__ int64_t long_rows[ROWS];
    __shared__ int n_long;
    __shared__ unsigned n_chunks, first[ROWS];
    __shared__ double warp_part[SPMV_THREADS / 32];

    const int g = threadIdx.x / T, l = threadIdx.x % T;
    const int lane = threadIdx.x & 31;
    const unsigned gmask = (T == 32) ? 0xffffffffu : (((1u << T) - 1u) << (lane & ~(T - 1)));
    if (threadIdx.x == 0) n_long = n_chunks = 0;
    // Programmatic dependent launch: when the launch carries that attribute this grid may be set up while the
    // kernel before it in the stream is still running; nothing that kernel may have written (x, y, even A) is
    // touched before the wait, and the next kernel in the stream is allowed to set up from here on.  Without
    // the attribute both instructions do nothing.
    wait_for_previous();
    if (lr.flag && *lr.flag == lr.call) return;        // a matrix with long rows: the tiles'
    __syncthreads();

    const int64_t row0 = (int64_t)blockIdx.x * (GROUPS * passes);
    int64_t s1 = 0, e1 = 0;
    if (row0 + g < nrows) { s1 = pos[row0 + g]; e1 = pos[row0 + g + 1]; }
    for (int pass = 0; pass < passes; pass++) {
        int64_t r = row0 + pass * GROUPS + g;
        if (r >= nrows) break;
        const int64_t s = s1, e = e1;
        if (pass + 1 < passes && r + GROUPS < nrows) { s1 = pos[r + GROUPS]; e1 = pos[r + GROUPS + 1]; }   // on their way meanwhile
        if (e - s > (hdr ? DEFER_ROW : T * 16)) {      // left to the end of the CTA, or to the chunks' kernel
            if (l == 0) long_rows[atomicAdd(&n_long, 1)] = r;
            continue;
        }
        double sum = row_partial<PAIR, VEC>(crd, val, x, s, e, l, T);
#pragma unroll
        for (int o = T / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(gmask, sum, o, T);
        if (l == 0) {
            int64_t out = row_ids ? row_ids[r] : r;
            y[out] = accumulate ? y[out] + sum : sum;
        }
    }
    __syncthreads();
    const int nl = n_long;
    if (hdr) {
        // chunks of the CTA's long rows: room for all of them is taken at once (a counter that 50,000 rows went to one by
        // one took 60 us), a warp writes a row's
        for (int i = threadIdx.x; i < nl; i += SPMV_THREADS) {
            const int64_t r = long_rows[i];
            first[i] = atomicAdd(&n_chunks, (unsigned)((pos[r + 1] - pos[r] + SPMV_CHUNK - 1) / SPMV_CHUNK));
            if (!accumulate) y[row_ids ? row_ids[r] : r] = 0.0;         // the chunks add into it
        }
        __syncthreads();
        if (threadIdx.x == 0 && nl) n_chunks = atomicAdd(&hdr->count, n_chunks);
        __syncthreads();
        for (int i = threadIdx.x >> 5; i < nl; i += SPMV_THREADS / 32) {
            const int64_t r = long_rows[i], s = pos[r], n = (pos[r + 1] - s + SPMV_CHUNK - 1) / SPMV_CHUNK;
            const unsigned at = n_chunks + first[i];
            if (at + n > chunk_cap) continue;          // cannot be: its capacity is a bound
            for (int64_t k = lane; k < n; k += 32) {
                chunks[at + k].row = r;
                chunks[at + k].begin = s + k * SPMV_CHUNK;
            }
        }
        return;
    }
    for (int i = threadIdx.x >> 5; i < nl; i += SPMV_THREADS / 32) {
        const int64_t r = long_rows[i], s = pos[r], e = pos[r + 1];
        if (e - s > LONG_ROW) continue;
        double sum = row_partial<PAIR, VEC>(crd, val, x, s, e, lane, 32);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) {
            const int64_t out = row_ids ? row_ids[r] : r;
            y[out] = accumulate ? y[out] + sum : sum;
        }
    }
    for (int i = 0; i < nl; i++) {
        int64_t r = long_rows[i];
        if (pos[r + 1] - pos[r] <= LONG_ROW) continue;
        double sum = row_partial<PAIR, VEC>(crd, val, x, pos[r], pos[r + 1], threadIdx.x, SPMV_THREADS);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) warp_part[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < SPMV_THREADS / 32; w++) t += warp_part[w];
            int64_t out = row_ids ? row_ids[r] : r;
            y[out] = accumulate ? y[out] + t : t;
        }
        __syncthreads();
    }
}

// Equal tiles of A's path (one step per stored entry and one per row end; the merge path of Merrill and Garland, Merge-based
// Parallel Sparse Matrix-Vector Multiplication, 2016), a CTA each.  The products of a tile's entries are
// made with all loads in flight and put into shared memory; every thread then walks eight or nine steps of the merged list of
// entries and row ends, and sums of rows that reach over threads travel by a segmented scan.
//
// With a plan (piece_plan) a row cut by a tile boundary is added with atomics onto a zero that the plan has written.
//
// ONCE, for matrices of up to ONCE_TILES tiles: one launch.  A CTA finds its rows itself: a first round of probes looks at
// the rows around where they would lie if all were alike and at places spread over the rest, which is all that even rows
// take; a second is enough below 100,000 rows.  A row that ends up to ONCE_PAST steps behind a boundary stays with the tile
// before it, so only long rows are cut: their tiles leave the parts in `cuts`, and the last one to do so adds them up in
// order.  Nobody waits, and the sums of every call are the same to the bit.
//
// Bound: up to 2^20 entries the chain of probes, row ends, entries and gathers of a CTA (6 us); beyond, the L1's rate of line
// accesses.
struct CutRows {
    double part[2 * ONCE_TILES];           // [2 b] of the row from before tile b, [2 b + 1] of the row that goes on behind it
    unsigned arrived[ONCE_TILES];          // by the tile that the row starts in; zero between calls
};
static __device__ CutRows g_cut_rows[ONCE_SLOTS];

// The rows and entries in which a tile and the next one start.  128 threads look for each, two probes at a time.
__device__ __forceinline__ void once_bounds(int64_t tile, int nrows, int64_t nnz, const int64_t *__restrict__ pos, int64_t (&row)[2],
                                            int64_t (&ent)[2])
{
    __shared__ int s_lo[2][2], s_hi[2][2];             // by round, so that one barrier does
    __shared__ int64_t s_end[2];
    const int which = threadIdx.x >> 7, i = threadIdx.x & 127;
    const int64_t steps = nnz + nrows, d = (tile + which) << TILE_SHIFT;
    if (threadIdx.x < 4) {
        s_lo[threadIdx.x >> 1][threadIdx.x & 1] = 0;
        s_hi[threadIdx.x >> 1][threadIdx.x & 1] = nrows;
    }
    if (i == 0) s_end[which] = -1;
    __syncthreads();
    // the row in whose steps (its entries, then its end) step d lies: the first with pos[r + 1] + r >= d
    int lo = 0, hi = nrows;
    for (int round = 0; round < 32; round++) {
        if (lo < hi) {
            const int64_t span = hi - lo;
            int p[2];
            if (round == 0) {
                p[0] = (int)((double)d / (double)steps * nrows) - 64 + i;
                p[1] = (int)(span * i / 128);
            } else {
                p[0] = lo + (int)(span * (2 * i) / 256);
                p[1] = lo + (int)(span * (2 * i + 1) / 256);
            }
            int64_t b[2], e[2];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                p[j] = p[j] < lo ? lo : p[j] >= hi ? hi - 1 : p[j];
                b[j] = pos[p[j]] + p[j] - 1;           // last step of the row before
                e[j] = pos[p[j] + 1] + p[j];
            }
#pragma unroll
            for (int j = 0; j < 2; j++) {
                if (e[j] < d) lo = p[j] + 1 > lo ? p[j] + 1 : lo;
                else hi = p[j] < hi ? p[j] : hi;
                if (e[j] >= d && b[j] < d) {           // this one
                    lo = hi = p[j];
                    s_end[which] = e[j];
                }
            }
            lo = __reduce_max_sync(0xffffffffu, lo);
            hi = __reduce_min_sync(0xffffffffu, hi);
            if ((threadIdx.x & 31) == 0) {
                atomicMax(&s_lo[round & 1][which], lo);
                atomicMin(&s_hi[round & 1][which], hi);
            }
        }
        __syncthreads();
        lo = s_lo[round & 1][which];
        hi = s_hi[round & 1][which];
        if (s_lo[round & 1][0] >= s_hi[round & 1][0] && s_lo[round & 1][1] >= s_hi[round & 1][1]) {
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int64_t r = s_lo[round & 1][j], end = s_end[j], at = (tile + j) << TILE_SHIFT;     // end -1: behind the last row
                const bool past = end >= 0 && end + 1 - at <= ONCE_PAST && at > 0;
                row[j] = end < 0 ? nrows : past ? r + 1 : r;
                ent[j] = end < 0 ? nnz : past ? end - r : at - r;
            }
            return;
        }
        // the other buffer starts the next round from these: it can only narrow
        if (i == 0) {
            s_lo[(round + 1) & 1][which] = lo;
            s_hi[(round + 1) & 1][which] = hi;
        }
        __syncthreads();
    }
}

// ONCE: this tile's part of row r, which is cut.  A warp; true for the last one to come, which has the sum of all tiles' parts.
__device__ __forceinline__ bool once_add(CutRows *cuts, int64_t tile, int after, double part, int64_t r,
                                            const int64_t *__restrict__ pos, double *total)
{
    const int lane = threadIdx.x & 31;
    const int64_t first = (pos[r] + r) >> TILE_SHIFT, last = (pos[r + 1] + r - ONCE_PAST) >> TILE_SHIFT;
    unsigned n = 0;
    if (lane == 0) {
        cuts->part[2 * tile + after] = part;
        __threadfence();
        n = atomicAdd(&cuts->arrived[first], 1u);
    }
    n = __shfl_sync(0xffffffffu, n, 0);
    if (n != (unsigned)(last - first)) return false;
    __threadfence();
    double sum = 0.0;
    for (int64_t q = first + lane; q <= last; q += 32) sum += __ldcg(&cuts->part[2 * q + (q == first)]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) cuts->arrived[first] = 0;
    *total = sum;
    return true;
}

template <bool PAIR, bool ONCE>
__global__ void __launch_bounds__(SPMV_THREADS, 4)
spmv_tiles_kernel(int64_t nrows, int64_t nnz, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                  const int64_t *__restrict__ crd, const double *__restrict__ val, const double *__restrict__ x,
                  double *__restrict__ y, int accumulate, const int64_t *__restrict__ tile_row,
                  const int64_t *__restrict__ tile_ent, LongRows lr, int slot)
{
    constexpr int ITEMS = ONCE ? ((1 << TILE_SHIFT) + ONCE_PAST) / SPMV_THREADS : TILE_ITEMS, STEPS = SPMV_THREADS * ITEMS;
    constexpr int PAD = ITEMS % 2 ? STEPS : ITEMS;     // entry i at i + i / PAD: a thread's run of ITEMS hits every bank once
    __shared__ double prod[STEPS + STEPS / PAD];
    __shared__ int ends[STEPS + 2];                    // ends of the rows that end in the tile, counted from its first entry
    __shared__ double warp_sum[SPMV_THREADS / 32];
    __shared__ int warp_end[SPMV_THREADS / 32];
    __shared__ double cut_part[2];                     // ONCE: of the row from before, of the row that goes on
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    wait_for_previous();
    if (not_this(lr)) return;
    int64_t row[2], ent[2];
    if (ONCE) {
        once_bounds(blockIdx.x, (int)nrows, nnz, pos, row, ent);
    } else {
        row[0] = tile_row[blockIdx.x];
        row[1] = tile_row[blockIdx.x + 1];
        ent[0] = tile_ent[blockIdx.x];
        ent[1] = tile_ent[blockIdx.x + 1];
    }
    const int64_t r0 = row[0], e0 = ent[0];
    const int m = (int)(row[1] - r0), n = (int)(ent[1] - e0);

    int64_t c[ITEMS];
    double v[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const int p = tid + i * SPMV_THREADS;
        c[i] = 0;
        v[i] = 0.0;
        if (p < n) {
            if (!PAIR) c[i] = ld_stream(crd + e0 + p);
            v[i] = PAIR ? 1.0 : ld_stream(val + e0 + p);
        }
    }
    for (int a = tid; a < m; a += SPMV_THREADS) ends[a] = (int)(pos[r0 + a + 1] - e0);
    const bool cut = r0 < nrows && pos[r0] < e0;       // the first row starts in an earlier tile
#pragma unroll
    for (int i = 0; i < ITEMS; i++) {
        const int p = tid + i * SPMV_THREADS;
        if (p < n) prod[p + p / PAD] = PAIR ? 1.0 : v[i] * __ldg(x + c[i]);
    }
    __syncthreads();

    // where this thread's steps start: after `a` row ends and `e` entries
    const int d = tid * ITEMS < n + m ? tid * ITEMS : n + m;
    const int last = tid == SPMV_THREADS - 1 || d + ITEMS > n + m ? n + m : d + ITEMS;
    int lo = d > n ? d - n : 0, hi = d < m ? d : m;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ends[mid] <= d - 1 - mid) lo = mid + 1;
        else hi = mid;
    }
    int a = lo, e = d - lo;
    const int a0 = a;
    double acc = 0.0, head = 0.0;                      // head: what this thread adds to the first row that ends here
    auto store = [&](int64_t r, double sum, bool add) {
        double *at = y + (row_ids ? row_ids[r] : r);
        if (add) atomicAdd(at, sum);
        else *at = accumulate ? *at + sum : sum;
    };
    int next = a < m ? ends[a] : n + 1;
    for (int t = d; t < last; t++) {
        if (e < next) {
            acc += prod[e + e / PAD];
            e++;
        } else {
            if (a == a0) head = acc;
            else store(r0 + a, acc, false);
            acc = 0.0;
            a++;
            next = a < m ? ends[a] : n + 1;
        }
    }
    // sums of unfinished rows travel to the thread in which the row ends
    const bool has = a > a0;
    double sum = acc;
    bool stop = has;                                   // the sum starts in this thread
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, sum, o);
        const bool ups = __shfl_up_sync(0xffffffffu, (int)stop, o);
        if (lane >= o && !stop) {
            sum += up;
            stop = ups;
        }
    }
    if (lane == 31) {
        warp_sum[warp] = sum;
        warp_end[warp] = stop;
    }
    double in = __shfl_up_sync(0xffffffffu, sum, 1);
    bool in_stop = __shfl_up_sync(0xffffffffu, (int)stop, 1);
    if (lane == 0) { in = 0.0; in_stop = false; }
    __syncthreads();
    if (!in_stop)
        for (int w = warp - 1; w >= 0; w--) {
            in += warp_sum[w];
            if (warp_end[w]) break;
        }
    if (!ONCE) {
        if (has) store(r0 + a0, in + head, a0 == 0 && cut);
        if (tid == SPMV_THREADS - 1 && r0 + m < nrows && e0 + n > pos[r0 + m]) store(r0 + m, has ? acc : in + acc, true);
        return;
    }
    const bool goes_on = r0 + m < nrows && e0 + n > pos[r0 + m], through = goes_on && cut && m == 0;
    if (has) {
        if (a0 == 0 && cut) cut_part[0] = in + head;
        else store(r0 + a0, in + head, false);
    }
    if (tid == SPMV_THREADS - 1 && goes_on) cut_part[through ? 0 : 1] = has ? acc : in + acc;
    __syncthreads();
    if (warp == 0 ? cut : warp == 1 && goes_on && !through) {
        const int64_t r = warp == 0 ? r0 : r0 + m;
        double total = 0.0;
        if (once_add(g_cut_rows + slot, blockIdx.x, warp, cut_part[warp], r, pos, &total) && lane == 0) store(r, total, false);
    }
}

template <bool PAIR, bool VEC>
__global__ void __launch_bounds__(SPMV_THREADS)
spmv_chunks_kernel(const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                   const int64_t *__restrict__ crd, const double *__restrict__ val,
                   const double *__restrict__ x, double *__restrict__ y, const WorkHeader *hdr,
                   const Chunk *chunks, unsigned chunk_cap)
{
    const int lane = threadIdx.x & 31;
    const unsigned warp = (blockIdx.x * SPMV_THREADS + threadIdx.x) >> 5;
    const unsigned nwarps = (gridDim.x * SPMV_THREADS) >> 5;
    wait_for_previous();
    unsigned count = hdr->count;
    if (count > chunk_cap) count = 0;
    for (unsigned w = warp; w < count; w += nwarps) {
        const Chunk ch = chunks[w];
        int64_t e = pos[ch.row + 1];
        if (e > ch.begin + SPMV_CHUNK) e = ch.begin + SPMV_CHUNK;
        double sum = row_partial<PAIR, VEC>(crd, val, x, ch.begin, e, lane, 32);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) atomicAdd(y + (row_ids ? row_ids[ch.row] : ch.row), sum);
    }
}

template <int T>
static int launch_spmv(int64_t nrows, const int64_t *row_ids, const int64_t *pos, const int64_t *crd,
                       const double *val, const double *x, double *y, bool pair, bool vec,
                       int accumulate, int64_t nnz, LongRows lr, cudaStream_t st)
{
    WorkHeader *hdr = nullptr;
    Chunk *chunks = nullptr;
    size_t cap = 0;
    if (nnz >= DEFER_MIN_NNZ && !lr.flag) {
        cap = (size_t)(nnz / SPMV_CHUNK + nnz / DEFER_ROW + 16);
        void *wl = nullptr;
        CB_TRY(scratch(SLOT_WORKLIST, sizeof(WorkHeader) + cap * sizeof(Chunk), &wl));
        hdr = (WorkHeader *)wl;
        chunks = (Chunk *)((char *)wl + sizeof(WorkHeader));
        CB_CUDA(cudaMemsetAsync(hdr, 0, sizeof(WorkHeader), st));
    }
    // small matrices: fewer rows per CTA so that the grid still covers every SM a few times
    constexpr int GROUPS = SPMV_THREADS / T;
    int passes = SPMV_PASSES;
    while (passes > 1 && ceil_div(nrows, (int64_t)GROUPS * passes) < (int64_t)sm_count() * 4) passes--;
    unsigned grid = (unsigned)ceil_div(nrows, (int64_t)GROUPS * passes);
    const unsigned ucap = (unsigned)cap;
    auto kernel = pair ? (vec ? spmv_kernel<T, true, true> : spmv_kernel<T, true, false>)
                       : (vec ? spmv_kernel<T, false, true> : spmv_kernel<T, false, false>);
    if (lr.flag)
        CB_CUDA(launch_behind(kernel, dim3(grid), SPMV_THREADS, 0, st, nrows, row_ids, pos, crd, val, x, y, accumulate, passes, hdr,
                              chunks, ucap, lr));
    else
        kernel<<<grid, SPMV_THREADS, 0, st>>>(nrows, row_ids, pos, crd, val, x, y, accumulate, passes, hdr, chunks, ucap, lr);
    CB_LAUNCH_CHECK();
    if (hdr) {
        const unsigned g2 = (unsigned)sm_count() * 8;
#define GO2(P, V) CB_CUDA(launch_behind(spmv_chunks_kernel<P, V>, dim3(g2), SPMV_THREADS, 0, st, row_ids, pos, crd, val, x, y, hdr, chunks, (unsigned)cap))
        if (pair) { if (vec) GO2(true, true); else GO2(true, false); }
        else      { if (vec) GO2(false, true); else GO2(false, false); }
#undef GO2
        CB_LAUNCH_CHECK();
    }
    return 0;
}

int spmv_rows(int64_t nrows, int64_t nnz, const int64_t *row_ids, const int64_t *pos,
              const int64_t *crd, const double *val, const double *x, double *y, int semiring,
              int accumulate, cudaStream_t st)
{
    if (nrows <= 0) return 0;
    bool vec = (((uintptr_t)crd | (uintptr_t)val) & 15) == 0;
    bool pair = semiring == COMET_B200_PLUS_PAIR;
    double mean = (double)nnz / (double)nrows;
    int t = mean <= 4.0 ? 2 : mean <= 8.0 ? 4 : mean <= 24.0 ? 8 : mean <= 48.0 ? 16 : 32;
    if (nnz < DEFER_MIN_NNZ) {
        // lanes that would idle otherwise shorten the longest rows (R-MAT scale 14: 28 -> 18 us)
        while (t < 32 && nrows * t * 2 <= (int64_t)sm_count() * 2048) t *= 2;
    }
    if (const char *env = getenv("COMET_B200_SPMV_LANES")) {        // tuning knob: lanes per row
        const int want = atoi(env);
        if (want == 2 || want == 4 || want == 8 || want == 16 || want == 32) t = want;
    }
    auto tiles = [&](LongRows lr) {
        StreamPlan plan;
        static_assert(SPMV_THREADS * TILE_ITEMS == 1 << TILE_SHIFT, "steps per tile");
        CB_TRY(piece_plan(nrows, nnz, TILE_SHIFT, row_ids, pos, y, 1, 1, accumulate, lr, st, &plan));
        if (plan.nblocks > 0x7fffffffLL) return fail("spmv: too many rows");
        CB_CUDA(launch_behind(pair ? spmv_tiles_kernel<true, false> : spmv_tiles_kernel<false, false>, dim3((unsigned)plan.nblocks),
                              SPMV_THREADS, 0, st, nrows, nnz, row_ids, pos, crd, val, x, y, accumulate, plan.block_row,
                              plan.block_ent, lr, 0));
        return 0;
    };
    const int64_t ntiles = ceil_div(nnz + nrows, (int64_t)1 << TILE_SHIFT);
    if (nnz < DEFER_MIN_NNZ && ntiles >= sm_count() && ntiles <= ONCE_TILES) {
        static std::atomic<unsigned> calls{0};
        CB_CUDA(launch_behind(pair ? spmv_tiles_kernel<true, true> : spmv_tiles_kernel<false, true>, dim3((unsigned)ntiles),
                              SPMV_THREADS, 0, st, nrows, nnz, row_ids, pos, crd, val, x, y, accumulate, nullptr, nullptr,
                              LongRows{nullptr, 0}, (int)(calls++ % ONCE_SLOTS)));
        return 0;
    }
    LongRows lr = {nullptr, 0};
    if (nnz >= LOOK_MIN_NNZ) {
        lr = next_mark();
        if (!lr.flag) return -1;
        // a lane group finishes 64 entries, or four times the mean, while its neighbours are still busy
        CB_TRY(mark_long_rows(nrows, pos, nnz / nrows * 4 > 64 ? nnz / nrows * 4 : 64, lr, st));
    }
    auto rows = t == 2 ? launch_spmv<2> : t == 4 ? launch_spmv<4> : t == 8 ? launch_spmv<8> : t == 16 ? launch_spmv<16> : launch_spmv<32>;
    CB_TRY(rows(nrows, row_ids, pos, crd, val, x, y, pair, vec, accumulate, nnz, lr, st));
    return lr.flag ? tiles(lr) : 0;
}

}  // namespace cb200

extern "C" int32_t comet_b200_dev_spmv_f64_i64(int64_t nrows, int64_t nnz, const int64_t *row_ids,
                                               const int64_t *pos, const int64_t *crd,
                                               const double *val, const double *x, double *y,
                                               int32_t semiring, int32_t accumulate, void *stream)
{
    cb200::clear_error();
    if (semiring != COMET_B200_PLUS_TIMES && semiring != COMET_B200_PLUS_PAIR)
        return cb200::fail("spmv: unsupported semiring %d", semiring);
    return cb200::spmv_rows(nrows, nnz, row_ids, pos, crd, val, x, y, semiring, accumulate,
                            (cudaStream_t)stream);
}
