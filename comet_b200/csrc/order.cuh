// The masked count of one strictly triangular matrix with itself (tc.cu): the triangles of a graph, counted in another order of
// its vertices.
//
// L strictly lower (or strictly upper) triangular, ascending, no coordinate twice: SUM(L*L .* L) is the number of triangles of the
// undirected graph L + L^T, whatever the order its vertices are numbered in.  So the vertices are renumbered by falling degree and every
// edge becomes an entry (hi, lo) of another strictly lower triangular matrix.  The hubs come first, no row is long any more
// (R-MAT scale 22, 64 M edges: 50,542 -> 1046 entries), and most entries are in the first HUBS columns.  Triangles i > k > j are
// counted in two parts by their lowest vertex:
//   j < HUBS    a warp per row i with a bitmap of its entries below HUBS in shared memory; for every entry k of the row, row k's part
//               below HUBS is intersected with it.  Rows with TRI_BITMAP and more such entries have their bitmap in memory: 128
//               columns a lane and step.  Where row i has few entries they are looked up in row k's bitmap instead (a sector each), and
//               rows k without a bitmap are streamed past row i's.
//   j >= HUBS   the rest of the rows, by the kernels of pairs.cuh (which need neither sorted rows nor the cut at column k).
// Nothing is sorted: entries are put into their rows in any order.
//
// Bound: the first part issues 2.9 of four instructions a clock (scale 20), 35 per step of 4096 columns; with fewer of them (row i's bits in
// registers, four rows k a step 7.1 ms; only the groups of 128 columns that row i has 7.3) it waits for the L2 instead.  At scale 22 the
// renumbering takes 2.8 ms of 11.3, the first part 5.5, the rest 2.9.
//
// Whether a matrix is triangular, and skewed enough for this to pay, is found out on the device (TcHeader::ordered); if not, the rest
// is the whole matrix as it is, and the kernels of the first part have nothing to do.
#pragma once
#include "pairs.cuh"
#include "stream.cuh"

namespace cb200 {

// A warp's bitmap is 2 KB of shared memory.  R-MAT scale 22, the first part / the rest, ms: 8192 4.5 / 4.3, 16384 5.5 / 2.8, 32768 8.2 / 1.4
// (more bitmaps than the L2 holds).
static const int TRI_HUBS = 16384;
static const int TRI_BITMAP = 64;               // entries from which on a row has a bitmap (32 5.7 ms at scale 22, 64 and 96 5.5)
static const int TRI_LOOK = 1;                  // look-ups of 32 entries against steps of 4096 columns: 1 to 1 5.5 ms, 2 to 1 6.2, none 9.9
static const int TRI_SAMPLE = 16;
static const int TRI_BUCKETS = 512;             // degrees: 16 per octave
// Where it pays (us before and after, R-MAT scale x edges per vertex): 18x5 322 566, 19x9 873 999, 20x6 1119 1375, 21x6 2533 2431,
// 19x13 1280 1128, 19x16 1745 1230, 20x16 3200 2378, 21x16 7760 4765, 22x16 18480 11250.
static const int64_t TRI_MIN_ENTRIES = 6000000;
static const int64_t TRI_MIN_PER_ROW = 10;
static const int TRI_WARPS = 8;
static const int TRI_SINGLE = 1 << 17;

struct TriCounters {                            // cleared before
    unsigned not_lower, not_upper;              // rows that are not (some of them counted twice)
    unsigned desc_all, desc_edge;               // places where the coordinates do not ascend: all, and those at row starts
    unsigned next, pad;
    unsigned long long words;                   // of the bitmaps given out
    unsigned long long columns;                 // of the rest
    unsigned hist[TRI_BUCKETS];                 // vertices per bucket, then the next place in it
    unsigned long long held[TRI_BUCKETS];       // their degrees
};

__device__ __forceinline__ int tri_bucket(unsigned degree)      // larger degrees, smaller numbers
{
    if (degree < 16) return TRI_BUCKETS - 1 - (int)degree;
    const int e = 31 - __clz(degree);
    return TRI_BUCKETS - 1 - (e * 16 - 48 + (int)((degree >> (e - 4)) & 15));
}

// Column counts, of one entry in TRI_SAMPLE (the order has to be about right; all of them take 1.3 ms on 64 M entries, where the hubs'
// counters are a queue, this 0.17).  Of 64 entries four neighbours are taken, any four: a column that is always at the same place of its row is met
// as often as others.  A CTA looks at the ends of rows from all over the matrix first and counts nothing if that cannot be triangular, which
// nearly all CTAs find out where it is not.
static __global__ void __launch_bounds__(256)
tri_degree_kernel(int64_t nrows, int64_t n, const int64_t *__restrict__ pos, const int64_t *__restrict__ crd, uint32_t *__restrict__ degree,
                  TriCounters *tc)
{
    __shared__ unsigned s_lower, s_upper;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (threadIdx.x == 0) s_lower = s_upper = 0;
    __syncthreads();
    const int64_t r = ((int64_t)threadIdx.x * gridDim.x + blockIdx.x) * nrows / stride, s = pos[r], e = pos[r + 1];
    const unsigned lower = __reduce_add_sync(0xffffffffu, (unsigned)(e > s && crd[e - 1] >= r));
    const unsigned upper = __reduce_add_sync(0xffffffffu, (unsigned)(e > s && crd[s] <= r));
    if ((threadIdx.x & 31) == 0) {
        if (lower) atomicAdd(&s_lower, lower);
        if (upper) atomicAdd(&s_upper, upper);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (s_lower) atomicAdd(&tc->not_lower, s_lower);
        if (s_upper) atomicAdd(&tc->not_upper, s_upper);
    }
    if (s_lower && s_upper) return;
    for (int64_t g = t0; g * (4 * TRI_SAMPLE) < n; g += stride) {
        const int64_t p = (g * TRI_SAMPLE + ((unsigned)g * 0x9E3779B1u >> 28)) * 4;
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (p + i < n) atomicAdd(degree + crd[p + i], (unsigned)TRI_SAMPLE);
    }
}
static_assert(TRI_SAMPLE == 16, "four bits of the hash");

// Row lengths to the degrees, their histogram, and the checks by row.
static __global__ void __launch_bounds__(512)
tri_hist_kernel(int64_t nrows, const int64_t *__restrict__ pos, const int64_t *__restrict__ crd, uint32_t *__restrict__ degree,
                TriCounters *tc)
{
    __shared__ unsigned s_hist[TRI_BUCKETS], s_held[TRI_BUCKETS];      // of 2^32 degrees at most
    __shared__ bool s_neither;
    wait_for_previous();
    if (threadIdx.x == 0) s_neither = *(volatile unsigned *)&tc->not_lower && *(volatile unsigned *)&tc->not_upper;
    for (int t = threadIdx.x; t < TRI_BUCKETS; t += blockDim.x) s_hist[t] = s_held[t] = 0;
    __syncthreads();
    if (s_neither) return;
    unsigned edge = 0, lower = 0, upper = 0;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t s = pos[r], e = pos[r + 1];
        unsigned d = degree[r];
        if (e > s) {
            const int64_t first = crd[s];
            lower += crd[e - 1] >= r;
            upper += first <= r;
            edge += s > 0 && first <= crd[s - 1];
            d += (unsigned)(e - s);
            degree[r] = d;
        }
        atomicAdd(&s_hist[tri_bucket(d)], 1u);
        if (d) atomicAdd(&s_held[tri_bucket(d)], d);
    }
    lower = __reduce_add_sync(0xffffffffu, lower);
    upper = __reduce_add_sync(0xffffffffu, upper);
    edge = __reduce_add_sync(0xffffffffu, edge);
    if ((threadIdx.x & 31) == 0) {
        if (lower) atomicAdd(&tc->not_lower, lower);
        if (upper) atomicAdd(&tc->not_upper, upper);
        if (edge) atomicAdd(&tc->desc_edge, edge);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < TRI_BUCKETS; t += blockDim.x)
        if (s_hist[t]) {
            atomicAdd(&tc->hist[t], s_hist[t]);
            atomicAdd(&tc->held[t], (unsigned long long)s_held[t]);
        }
}

// Decides, and turns the histogram into places.  One CTA of TRI_BUCKETS threads.
static __global__ void __launch_bounds__(TRI_BUCKETS)
tri_decide_kernel(int64_t nnz, TcHeader *hdr, TriCounters *tc)
{
    __shared__ unsigned s_n[TRI_BUCKETS];
    __shared__ unsigned long long s_h[TRI_BUCKETS];
    const int t = threadIdx.x;
    wait_for_previous();
    s_n[t] = tc->hist[t];
    s_h[t] = tc->held[t];
    __syncthreads();
    for (int o = 1; o < TRI_BUCKETS; o <<= 1) {
        const unsigned n = t >= o ? s_n[t - o] : 0u;
        const unsigned long long h = t >= o ? s_h[t - o] : 0ull;
        __syncthreads();
        s_n[t] += n;
        s_h[t] += h;
        __syncthreads();
    }
    const unsigned before = t ? s_n[t - 1] : 0u;
    tc->hist[t] = before;
    // the first TRI_HUBS vertices hold a quarter of all degrees, or there are no more vertices than that.  Of the bucket that reaches TRI_HUBS
    // as many count as still fit: where all vertices are alike it holds every one of them (12 entries in each of 700,000 rows, counted
    // in another order: 713 -> 960 us).
    const bool last = s_n[t] >= TRI_HUBS || t == TRI_BUCKETS - 1;
    if (last && before < TRI_HUBS) {
        const double of = s_n[t] > TRI_HUBS ? (double)(TRI_HUBS - before) / (s_n[t] - before) : 1.0;
        const double held = (t ? (double)s_h[t - 1] : 0.0) + of * (double)(s_h[t] - (t ? s_h[t - 1] : 0ull));
        const bool skewed = s_n[TRI_BUCKETS - 1] <= TRI_HUBS || held * 4.0 >= 2.0 * (double)nnz;
        hdr->ordered = skewed && (tc->not_lower == 0 || tc->not_upper == 0);       // if the coordinates ascend, see tri_totals_kernel
    }
}

// A vertex's new number: by falling degree, any order within a bucket.  Clears the rows' counts.
static __global__ void __launch_bounds__(512)
tri_rank_kernel(int64_t nrows, const uint32_t *__restrict__ degree, const TcHeader *hdr, TriCounters *tc, int32_t *__restrict__ rank,
                int32_t *__restrict__ hub_count, int32_t *__restrict__ rest_count)
{
    wait_for_previous();
    if (!hdr->ordered) return;
    __shared__ unsigned s_count[TRI_BUCKETS], s_base[TRI_BUCKETS];
    const int64_t stride = (int64_t)gridDim.x * 2048;
    for (int64_t r0 = (int64_t)blockIdx.x * 2048; r0 < nrows; r0 += stride) {
        for (int t = threadIdx.x; t < TRI_BUCKETS; t += 512) s_count[t] = 0;
        __syncthreads();
        int bucket[4];
        unsigned at[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t r = r0 + i * 512 + threadIdx.x;
            bucket[i] = r < nrows ? tri_bucket(degree[r]) : -1;
            if (r < nrows) {
                at[i] = atomicAdd(&s_count[bucket[i]], 1u);
                hub_count[r] = rest_count[r] = 0;
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < TRI_BUCKETS; t += 512)
            if (s_count[t]) s_base[t] = atomicAdd(&tc->hist[t], s_count[t]);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (bucket[i] >= 0) rank[r0 + i * 512 + threadIdx.x] = (int32_t)(s_base[bucket[i]] + at[i]);
        __syncthreads();
    }
}

// The edges in their new numbers, how many entries every row will have in the hub columns and in the others, and each entry's place
// among them; and the places where the coordinates do not ascend.  A warp takes 512 entries, 128 of them in flight, and finds their rows among 32 row ends in the lanes.
static __global__ void __launch_bounds__(256)
tri_edges_kernel(int64_t nrows, int64_t nnz, const int64_t *__restrict__ pos, const int64_t *__restrict__ crd,
                 const int32_t *__restrict__ rank, const TcHeader *hdr, TriCounters *tc, int2 *__restrict__ edge,
                 int32_t *__restrict__ place, int32_t *__restrict__ hub_count, int32_t *__restrict__ rest_count)
{
    wait_for_previous();
    if (!hdr->ordered) return;
    const int lane = threadIdx.x & 31;
    const int64_t first = (((int64_t)blockIdx.x * 256 + threadIdx.x) >> 5) * 512;
    if (first >= nnz) return;
    const int n = nnz - first < 512 ? (int)(nnz - first) : 512;
    crd += first;
    edge += first;
    place += first;
    int64_t w0 = 0;
    int end = 0;                                 // lane l: where row w0 + l ends, counted from `first`; the first of them ends behind p
    int32_t own = 0;                             // and its number
    auto rows_from = [&](int p) {
        int64_t lo = 0, hi = nrows - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (pos[mid + 1] <= first + p) lo = mid + 1; else hi = mid;
        }
        w0 = lo;
        const int64_t e = w0 + lane < nrows ? pos[w0 + lane + 1] - first : n;
        end = e < n ? (int)e : n;
        own = w0 + lane < nrows ? rank[w0 + lane] : 0;
    };
    rows_from(0);
    unsigned top = 0, desc = 0;
    for (int p0 = 0; p0 < n; p0 += 128) {
        int32_t rj[4], ri[4], at[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int p = p0 + u * 32 + lane;
            const int64_t j = crd[p < n ? p : n - 1];
            rj[u] = rank[j];
            desc += p < n && first + p + 1 < nnz && crd[p + 1] <= j;
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int p = min(p0 + u * 32 + lane, n - 1);
            bool open = true;
            while (true) {
                int lo = 0;
#pragma unroll
                for (int step = 16; step > 0; step >>= 1)
                    if (__shfl_sync(0xffffffffu, end, lo + step - 1) <= p) lo += step;
                if (__shfl_sync(0xffffffffu, end, lo) <= p) lo++;
                const int32_t number = __shfl_sync(0xffffffffu, own, lo & 31);
                if (open && lo < 32) {
                    ri[u] = number;
                    open = false;
                }
                const unsigned left = __ballot_sync(0xffffffffu, open);
                if (!left) break;
                rows_from(__shfl_sync(0xffffffffu, p, __ffs(left) - 1));
            }
        }
        // the entries that stay in their row are neighbours and add to its count together (one by one 1.4 ms on 64 M entries)
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const bool in = p0 + u * 32 + lane < n;
            const int32_t hi = max(ri[u], rj[u]), lo = min(ri[u], rj[u]);
            const bool is_hub = lo < TRI_HUBS, stays = in && hi == ri[u];
            const int32_t before = __shfl_up_sync(0xffffffffu, ri[u], 1);
            const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || before != ri[u]);
            const unsigned stay_hub = __ballot_sync(0xffffffffu, stays && is_hub), stay_rest = __ballot_sync(0xffffffffu, stays && !is_hub);
            const unsigned upto = 0xffffffffu >> (31 - lane), later = heads & ~upto;
            const unsigned run = (later ? (1u << (__ffs(later) - 1)) - 1u : 0xffffffffu) & (0xffffffffu << (31 - __clz(heads & upto)));
            const unsigned group = stays ? run & (is_hub ? stay_hub : stay_rest) : 1u << lane;
            const int leader = __ffs(group) - 1;
            int32_t got = 0;
            if (in && lane == leader) got = atomicAdd((is_hub ? hub_count : rest_count) + hi, __popc(group));
            at[u] = __shfl_sync(0xffffffffu, got, leader) + __popc(group & (upto >> 1));
            if (in && !is_hub) top = max(top, (unsigned)(lo - TRI_HUBS + 1));
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int p = p0 + u * 32 + lane;
            if (p >= n) continue;
            __stcs(edge + p, make_int2(max(ri[u], rj[u]), min(ri[u], rj[u])));
            __stcs(place + p, at[u]);
        }
    }
    top = __reduce_max_sync(0xffffffffu, top);
    desc = __reduce_add_sync(0xffffffffu, desc);
    if (lane == 0 && desc) atomicAdd(&tc->desc_all, desc);
    if (lane == 0 && top > (unsigned)*(volatile unsigned long long *)&tc->columns) atomicMax(&tc->columns, (unsigned long long)top);
}

// Where the rows' entries begin in the hub columns (blockIdx.y 0) and in the others (1): sums of TRI_TILE rows, the sums before them, places.
// Where the order stays, the rest is the whole matrix as it is.
static const int TRI_TILE = 2048;

static __global__ void __launch_bounds__(256)
tri_sums_kernel(int64_t nrows, const int32_t *__restrict__ hub_count, const int32_t *__restrict__ rest_count, const TcHeader *hdr,
                int64_t *__restrict__ sums)
{
    __shared__ int64_t s_sum[8];
    wait_for_previous();
    if (!hdr->ordered) return;
    const int32_t *in = blockIdx.y ? rest_count : hub_count;
    int64_t sum = 0;
#pragma unroll
    for (int i = 0; i < TRI_TILE / 256; i++) {
        const int64_t r = (int64_t)blockIdx.x * TRI_TILE + i * 256 + threadIdx.x;
        if (r < nrows) sum += in[r];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, (long long)sum, o);
    if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; w++) sum += s_sum[w];
        sums[(int64_t)blockIdx.y * gridDim.x + blockIdx.x] = sum;
    }
}

// One CTA.  The edges' kernel has been through all coordinates: if they do not ascend, the order stays.
static __global__ void __launch_bounds__(1024)
tri_totals_kernel(int64_t nrows, int64_t tiles, TcHeader *hdr, const TriCounters *tc, int64_t *__restrict__ sums, int64_t *__restrict__ hub_pos,
                  int64_t *__restrict__ rest_pos)
{
    __shared__ int64_t s_sum[32];
    wait_for_previous();
    if (!hdr->ordered) return;
    __syncthreads();                             // all have read it
    if (tc->desc_all != tc->desc_edge) {
        if (threadIdx.x == 0) hdr->ordered = 0;
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int y = 0; y < 2; y++, sums += tiles) {
        int64_t carry = 0;
        for (int64_t base = 0; base < tiles; base += 1024) {
            const int64_t t = base + threadIdx.x, own = t < tiles ? sums[t] : 0;
            int64_t incl = own;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t v = __shfl_up_sync(0xffffffffu, (long long)incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) s_sum[warp] = incl;
            __syncthreads();
            int64_t before = carry + incl - own;
            for (int w = 0; w < 32; w++) {
                if (w < warp) before += s_sum[w];
                carry += s_sum[w];
            }
            if (t < tiles) sums[t] = before;
            __syncthreads();
        }
        if (threadIdx.x == 0) (y ? rest_pos : hub_pos)[nrows] = carry;
    }
}

static __global__ void __launch_bounds__(256)
tri_places_kernel(int64_t nrows, const int32_t *__restrict__ hub_count, const int32_t *__restrict__ rest_count, const int64_t *__restrict__ pos,
                  const TcHeader *hdr, const int64_t *__restrict__ sums, int64_t *__restrict__ hub_pos, int64_t *__restrict__ rest_pos)
{
    __shared__ int64_t s_sum[8];
    wait_for_previous();
    const int64_t base = (int64_t)blockIdx.x * TRI_TILE;
    if (!hdr->ordered) {
        if (blockIdx.y == 0) return;
#pragma unroll
        for (int i = 0; i < TRI_TILE / 256; i++) {
            const int64_t r = base + i * 256 + threadIdx.x;
            if (r <= nrows) rest_pos[r] = pos[r];
        }
        return;
    }
    const int32_t *in = blockIdx.y ? rest_count : hub_count;
    int64_t *out = blockIdx.y ? rest_pos : hub_pos;
    const int64_t r0 = base + threadIdx.x * (TRI_TILE / 256);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t own[TRI_TILE / 256];
    int64_t incl = 0;
#pragma unroll
    for (int i = 0; i < TRI_TILE / 256; i++) {
        own[i] = r0 + i < nrows ? in[r0 + i] : 0;
        incl += own[i];
    }
    int64_t at = -incl;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t v = __shfl_up_sync(0xffffffffu, (long long)incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    at += incl + sums[(int64_t)blockIdx.y * gridDim.x + blockIdx.x];
    for (int w = 0; w < warp; w++) at += s_sum[w];
#pragma unroll
    for (int i = 0; i < TRI_TILE / 256; i++) {
        if (r0 + i < nrows) out[r0 + i] = at;
        at += own[i];
    }
}

// The entries into their rows.  columns != null: where pairs.cuh looks for the number of columns.  m32 may be a32 (columns keep their numbers).
static __global__ void __launch_bounds__(256)
tri_scatter_kernel(int64_t nnz, const int2 *__restrict__ edge, const int32_t *__restrict__ place, const int64_t *__restrict__ hub_pos,
                   const int64_t *__restrict__ rest_pos, const TcHeader *hdr, const TriCounters *tc,
                   unsigned short *__restrict__ hub, int32_t *a32, int32_t *m32, int64_t *columns)
{
    wait_for_previous();
    if (!hdr->ordered) return;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (t0 == 0 && columns) *columns = (int64_t)tc->columns;
    for (int64_t p0 = t0; p0 < nnz; p0 += 4 * stride) {
        int2 e[4];
        int64_t at[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (p0 + u * stride < nnz) {
                e[u] = __ldcs(edge + p0 + u * stride);
                at[u] = __ldcs(place + p0 + u * stride);
            }
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (p0 + u * stride < nnz) at[u] += (e[u].y < TRI_HUBS ? hub_pos : rest_pos)[e[u].x];
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (p0 + u * stride < nnz) {
                if (e[u].y < TRI_HUBS) {
                    hub[at[u]] = (unsigned short)e[u].y;
                } else {
                    a32[at[u]] = e[u].y;
                    if (m32 != a32) m32[at[u]] = e[u].y - TRI_HUBS;
                }
            }
    }
}

// words of row k's bitmap: its hub columns are below k
__device__ __forceinline__ int tri_words(int64_t k) { return (int)(((k < TRI_HUBS ? k : TRI_HUBS) + 127) >> 7) * 4; }

// Bitmaps of the rows with TRI_BITMAP and more hub columns, while there is room: bits_at[k] in units of four words, or -1.
static __global__ void __launch_bounds__(TRI_WARPS * 32)
tri_bitmap_kernel(int64_t nrows, const int64_t *__restrict__ hub_pos, const unsigned short *__restrict__ hub, const TcHeader *hdr,
                  TriCounters *tc, unsigned long long room, int32_t *__restrict__ bits_at, uint32_t *__restrict__ bits)
{
    __shared__ __align__(16) uint32_t s_bits[TRI_WARPS][TRI_HUBS / 32];
    wait_for_previous();
    if (!hdr->ordered) return;
    const int lane = threadIdx.x & 31;
    uint32_t *bm = s_bits[threadIdx.x >> 5];
    for (int w = lane; w < TRI_HUBS / 32; w += 32) bm[w] = 0;
    __syncwarp();
    const int64_t warps = (int64_t)gridDim.x * TRI_WARPS;
    for (int64_t base = ((int64_t)blockIdx.x * TRI_WARPS + (threadIdx.x >> 5)) * 32; base < nrows; base += warps * 32) {
        int64_t s = 0;
        int len = 0;
        if (base + lane < nrows) {
            s = hub_pos[base + lane];
            len = (int)(hub_pos[base + lane + 1] - s);
            if (len < TRI_BITMAP) bits_at[base + lane] = -1;
        }
        unsigned left = __ballot_sync(0xffffffffu, len >= TRI_BITMAP);
        while (left) {
            const int t = __ffs(left) - 1;
            left &= left - 1;
            const int64_t k = base + t, ks = __shfl_sync(0xffffffffu, (long long)s, t);
            const int n = __shfl_sync(0xffffffffu, len, t), words = tri_words(k);
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(&tc->words, (unsigned long long)words);
            at = __shfl_sync(0xffffffffu, at, 0);
            const bool fits = at + words <= room;
            if (lane == 0) bits_at[k] = fits ? (int32_t)(at >> 2) : -1;
            if (!fits) continue;
            for (int q = lane; q < n; q += 32) {
                const unsigned j = hub[ks + q];
                atomicOr(&bm[j >> 5], 1u << (j & 31));
            }
            __syncwarp();
            for (int w = lane; w < words / 4; w += 32) {
                ((uint4 *)(bits + at))[w] = ((uint4 *)bm)[w];
                ((uint4 *)bm)[w] = make_uint4(0, 0, 0, 0);
            }
            __syncwarp();
        }
    }
}

// The triangles whose lowest vertex is a hub column.  Steps of one kind from several entries k are in flight together.
static __global__ void __launch_bounds__(TRI_WARPS * 32, 5)
tri_count_kernel(int64_t nrows, const int64_t *__restrict__ hub_pos, const unsigned short *__restrict__ hub,
                 const int64_t *__restrict__ rest_pos, const int32_t *__restrict__ a32, const int32_t *__restrict__ bits_at,
                 const uint32_t *__restrict__ bits, const TcHeader *hdr, TriCounters *tc, unsigned long long *count)
{
    __shared__ __align__(16) uint32_t s_bits[TRI_WARPS][TRI_HUBS / 32];
    __shared__ unsigned long long s_part[TRI_WARPS];
    wait_for_previous();
    if (!hdr->ordered) return;
    const int lane = threadIdx.x & 31;
    uint32_t *bm = s_bits[threadIdx.x >> 5];
    for (int w = lane; w < TRI_HUBS / 32; w += 32) bm[w] = 0;
    __syncwarp();
    unsigned long long total = 0;
    while (true) {
        // the first rows, where the long ones are, one by one, the others 32 at a time
        unsigned ticket = 0;
        if (lane == 0) ticket = atomicAdd(&tc->next, 1u);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        const bool single = ticket < (unsigned)TRI_SINGLE;
        const int64_t i0 = single ? ticket : TRI_SINGLE + (int64_t)(ticket - TRI_SINGLE) * 32;
        if (i0 >= nrows) break;
        int64_t s_l = 0, rs_l = 0;
        int n_l = 0, pairs_l = 0;
        if (i0 + lane < nrows && (lane == 0 || !single)) {
            s_l = hub_pos[i0 + lane];
            rs_l = rest_pos[i0 + lane];
            n_l = (int)(hub_pos[i0 + lane + 1] - s_l);
            pairs_l = n_l + (int)(rest_pos[i0 + lane + 1] - rs_l);
        }
        unsigned rows = __ballot_sync(0xffffffffu, n_l > 0 && pairs_l > 1);
        while (rows) {
            const int mine = __ffs(rows) - 1;
            rows &= rows - 1;
            const int64_t s = __shfl_sync(0xffffffffu, (long long)s_l, mine), rs = __shfl_sync(0xffffffffu, (long long)rs_l, mine);
            const int n = __shfl_sync(0xffffffffu, n_l, mine), pairs = __shfl_sync(0xffffffffu, pairs_l, mine);
            for (int q = lane; q < n; q += 32) {
                const unsigned j = hub[s + q];
                atomicOr(&bm[j >> 5], 1u << (j & 31));
            }
            __syncwarp();
            unsigned hits = 0;
            const int probes = (n + 31) >> 5;
            for (int b = 0; b < pairs; b += 32) {
                int64_t ks = 0;
                int len = 0, groups = 0, at = -1;
                if (b + lane < pairs) {
                    const int64_t k = b + lane < n ? hub[s + b + lane] : a32[rs + b + lane - n];
                    ks = hub_pos[k];
                    len = (int)(hub_pos[k + 1] - ks);
                    if (len >= TRI_BITMAP) {
                        at = bits_at[k];
                        groups = tri_words(k) >> 2;
                    }
                }
                // rows k without a bitmap: past row i's
                {
                    unsigned left = __ballot_sync(0xffffffffu, len > 0 && at < 0);
                    const unsigned short *q = hub;
                    int rem = 0;
                    while (left || rem > 0) {
                        int j[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            if (rem <= 0 && left) {
                                const int t = __ffs(left) - 1;
                                left &= left - 1;
                                q = hub + __shfl_sync(0xffffffffu, (long long)ks, t) + lane;
                                rem = __shfl_sync(0xffffffffu, len, t);
                            }
                            j[u] = -1;
                            if (lane < rem) j[u] = __ldg(q);
                            q += 32;
                            rem -= 32;
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            if (j[u] >= 0) hits += (bm[j[u] >> 5] >> (j[u] & 31)) & 1u;
                    }
                }
                // a row i of few entries: looked up in row k's bitmap, four rows k at a time
                const bool look = at >= 0 && probes * TRI_LOOK < (groups + 31) / 32;
                unsigned left = __ballot_sync(0xffffffffu, look);
                for (int q = 0; left && q < n; q += 32) {
                    const int j = q + lane < n ? hub[s + q + lane] : INT32_MAX;
                    for (unsigned now = left; now;) {
                        uint32_t v[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            v[u] = 0;
                            if (!now) continue;
                            const int t = __ffs(now) - 1;
                            now &= now - 1;
                            const int64_t kat = __shfl_sync(0xffffffffu, at, t);
                            const int kw = __shfl_sync(0xffffffffu, groups, t);
                            if ((j >> 7) < kw) v[u] = __ldg(bits + kat * 4 + (j >> 5));
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++) hits += (v[u] >> (j & 31)) & 1u;
                    }
                }
                // bitmap against bitmap, steps of 4096 columns of one row k or of several in flight
                left = __ballot_sync(0xffffffffu, at >= 0 && !look);
                const uint4 *q = (const uint4 *)bits;
                int rem = 0, w = 0;
                while (left || rem > 0) {
                    uint4 v[4];
                    int o[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (rem <= 0 && left) {
                            const int t = __ffs(left) - 1;
                            left &= left - 1;
                            q = (const uint4 *)bits + __shfl_sync(0xffffffffu, at, t) + lane;
                            rem = __shfl_sync(0xffffffffu, groups, t);
                            w = lane;
                        }
                        o[u] = w;
                        v[u] = make_uint4(0, 0, 0, 0);
                        if (lane < rem) v[u] = __ldg(q);
                        q += 32;
                        w += 32;
                        rem -= 32;
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const uint4 x = ((const uint4 *)bm)[o[u] & (TRI_HUBS / 128 - 1)];
                        hits += __popc(v[u].x & x.x) + __popc(v[u].y & x.y) + __popc(v[u].z & x.z) + __popc(v[u].w & x.w);
                    }
                }
            }
            total += hits;
            __syncwarp();
            for (int q = lane; q < n; q += 32) bm[hub[s + q] >> 5] = 0;
            __syncwarp();
        }
    }
    tc_add_count(total, s_part, TRI_WARPS, count);
}

}  // namespace cb200
