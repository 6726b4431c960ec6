// Format conversions on the device: stable sort of coordinate entries, COO -> CSR, and the
// transpose of a CSR matrix (CSR of the transposed matrix, i.e. the CSC arrays of the input).
//
// COMET does these on the host with one thread: the reader sorts the parsed entries with
// std::stable_sort by (row, col) and keeps duplicates (lib/ExecutionEngine/SparseUtils.cpp:360-367,
// 404-533), and transpose_2D turns CSR into coordinates, sorts them by (col, row) and rebuilds the
// row pointer (lib/ExecutionEngine/TransposeUtils.cpp:738-812).  Here both are one radix sort (least significant
// digit first, stable, so equal coordinates keep their input order like stable_sort) of keys major | minor in as
// many bits as the two extents need, carrying the entry's position, then a gather of the values and
// the row pointer by binary search in the sorted keys.  A CSR matrix is already in row order, so its
// transpose sorts by the column alone.
//
// The sort is this file's own code for published methods: least-significant-digit passes of one kernel each (Adinets and
// Merrill, Onesweep, 2022) whose tiles find their places by decoupled look-back (Merrill and Garland, Single-pass Parallel
// Prefix Scan with Decoupled Look-back, 2016).  One kernel makes the keys and counts the digits of all passes; a pass is one kernel:
// a CTA ranks a tile of keys by their digit, learns from the tiles before it where its runs of equal digits
// start (each tile publishes its digit counts, then their sums over all tiles so far, and looks back until it meets
// such a sum), orders the tile in shared memory and writes it out run by run.  Tiles are numbered in the order in
// which CTAs start, so the tiles looked back at are running or done; the wait is bounded all the same.  Ranking
// is what makes it stable: a warp walks its part of the tile 32 consecutive keys at a time, `__match_any_sync`
// names the lanes that hold the same digit, a key's rank is the number of such lanes below it plus the
// count its warp has already seen for the digit, and warps are ordered by a prefix over their counts.
//
// Bound: HBM or L2 (a pass reads and writes key and position once: 2 x 12 bytes per entry for keys above 32 bits and fewer
// than 2^32 entries; passes = key bits / 8, rounded up).  Measured on B200: 4.2 M entries with 36-bit keys 28 us for the keys,
// 67 us a pass, 47 us for gather and row pointer (a count, three scan and a scatter kernel per pass before); 1000 entries
// from and to host arrays 735 -> 141 us.
#include "common.cuh"
#include "hostcopy.cuh"

namespace cb200 {

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, position) pairs.
// ---------------------------------------------------------------------------
static const int RS_THREADS = 256;                    // 8 warps
static const int RS_WARPS = RS_THREADS / 32;
static const int RS_ROUNDS = 16;                      // rounds of 32 keys per warp
static const int RS_TILE = RS_THREADS * RS_ROUNDS;    // keys per CTA
static const int RS_DIGITS = 256;
static const int RS_MAX_PASSES = 8;
static const int RS_COPIES = 8;                       // histograms a CTA keeps while counting: equal digits meet 4 lanes at most
static const uint64_t RS_COUNT = 1ull << 62;          // state word: the tile's own count
static const uint64_t RS_SUM = 2ull << 62;            // state word: sum over all tiles up to this one
static const int RS_SPIN_LIMIT = 1 << 24;

struct SortPlan {
    int passes, width;                                // digits of `width` bits
    int64_t ntiles;
    int *bad;                                         // [0] coordinate outside the matrix, [1] a look-back gave up
    unsigned *ticket;                                 // one per pass
    uint64_t *hist;                                   // [pass][digit] counts, then their exclusive sums
    uint64_t *state;                                  // [pass][tile][digit]
};

// Counts the digits of every pass of one key into the CTA's histograms.
template <typename KeyT>
__device__ __forceinline__ void rs_count_key(unsigned *h, KeyT key, int passes, int width)
{
    const int copy = threadIdx.x & (RS_COPIES - 1);
    for (int p = 0; p < passes; p++)
        atomicAdd(&h[((p * RS_DIGITS) + ((unsigned)(key >> (p * width)) & ((1u << width) - 1u))) * RS_COPIES + copy], 1u);
}

__device__ __forceinline__ void rs_count_flush(const unsigned *h, int passes, uint64_t *hist)
{
    for (int i = threadIdx.x; i < passes * RS_DIGITS; i += blockDim.x) {
        unsigned t = 0;
        for (int c = 0; c < RS_COPIES; c++) t += h[i * RS_COPIES + c];
        if (t) atomicAdd((unsigned long long *)hist + i, (unsigned long long)t);
    }
}

// keys of coordinate entries; `minor` null: the major coordinate alone; entries from *limit on (limit not null) get the last
// major coordinate
template <typename KeyT>
__global__ void __launch_bounds__(256)
rs_make_keys_kernel(int64_t n, const int64_t *__restrict__ major, const int64_t *__restrict__ minor, int64_t nmajor,
                    int64_t nminor, int minor_bits, const int64_t *limit, KeyT *__restrict__ keys, SortPlan sp)
{
    extern __shared__ unsigned s_hist[];
    for (int i = threadIdx.x; i < sp.passes * RS_DIGITS * RS_COPIES; i += blockDim.x) s_hist[i] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t a = __ldcs((const long long *)major + i), b = minor ? __ldcs((const long long *)minor + i) : 0;
        KeyT key = 0;                                 // reported by the host; the key stays in range
        if (limit && i >= *limit) key = (KeyT)(nmajor - 1);
        else if (a < 0 || a >= nmajor || b < 0 || b >= nminor) *sp.bad = 1;
        else key = (KeyT)(((uint64_t)a << minor_bits) | (uint64_t)b);
        keys[i] = key;
        rs_count_key(s_hist, key, sp.passes, sp.width);
    }
    __syncthreads();
    rs_count_flush(s_hist, sp.passes, sp.hist);
}

// counts -> exclusive sums, a CTA per pass
__global__ void __launch_bounds__(RS_DIGITS)
rs_scan_kernel(uint64_t *hist)
{
    __shared__ uint64_t s[RS_DIGITS];
    uint64_t *h = hist + blockIdx.x * RS_DIGITS;
    const uint64_t own = h[threadIdx.x];
    s[threadIdx.x] = own;
    __syncthreads();
    for (int o = 1; o < RS_DIGITS; o <<= 1) {
        const uint64_t v = (int)threadIdx.x >= o ? s[threadIdx.x - o] : 0;
        __syncthreads();
        s[threadIdx.x] += v;
        __syncthreads();
    }
    h[threadIdx.x] = s[threadIdx.x] - own;
}

// One pass.  FIRST: the position of key i is i.
template <typename KeyT, typename IdxT, bool FIRST>
__global__ void __launch_bounds__(RS_THREADS)
rs_pass_kernel(int64_t n, const KeyT *__restrict__ keys, const IdxT *__restrict__ idx, KeyT *__restrict__ keys_out,
               IdxT *__restrict__ idx_out, int pass, SortPlan sp)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    KeyT *s_keys = (KeyT *)s_raw;
    IdxT *s_idx = (IdxT *)(s_keys + RS_TILE);
    __shared__ unsigned cnt[RS_WARPS][RS_DIGITS];
    __shared__ unsigned local[RS_DIGITS];             // first place of the digit's run in the ordered tile
    __shared__ int64_t start[RS_DIGITS];              // first place of the tile's run of the digit in the output
    __shared__ unsigned warp_sum[RS_WARPS];
    __shared__ unsigned s_tile;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, d0 = threadIdx.x;
    const int shift = pass * sp.width;
    const unsigned mask = (1u << sp.width) - 1u, below = (1u << lane) - 1u;
    if (threadIdx.x == 0) s_tile = atomicAdd(sp.ticket + pass, 1u);
    for (int i = threadIdx.x; i < RS_WARPS * RS_DIGITS; i += RS_THREADS) (&cnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t base = tile * RS_TILE + (int64_t)w * 32 * RS_ROUNDS + lane;
    KeyT k[RS_ROUNDS];
    IdxT v[RS_ROUNDS];
    unsigned rank[RS_ROUNDS];
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; r++) {
        const int64_t i = base + r * 32;
        k[r] = i < n ? keys[i] : 0;
        v[r] = FIRST ? (IdxT)i : (i < n ? idx[i] : 0);
    }
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; r++) {
        const bool live = base + r * 32 < n;
        const unsigned d = live ? (unsigned)(k[r] >> shift) & mask : RS_DIGITS;    // dead lanes form their own group
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(peers) - 1;
        unsigned old = 0;
        if (live && lane == leader) {
            old = cnt[w][d];
            cnt[w][d] = old + __popc(peers);
        }
        old = __shfl_sync(0xffffffffu, old, leader);
        __syncwarp();
        rank[r] = old + __popc(peers & below);
    }
    __syncthreads();
    unsigned total = 0;                               // this thread's digit: keys of it in the tile
    for (int i = 0; i < RS_WARPS; i++) {
        const unsigned c = cnt[i][d0];
        cnt[i][d0] = total;
        total += c;
    }
    volatile uint64_t *state = sp.state + ((int64_t)pass * sp.ntiles) * RS_DIGITS;
    state[tile * RS_DIGITS + d0] = (tile == 0 ? RS_SUM : RS_COUNT) | total;
    unsigned incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sum[w] = incl;
    __syncthreads();
    unsigned off = incl - total;
    for (int i = 0; i < w; i++) off += warp_sum[i];
    local[d0] = off;
    uint64_t before = 0;                              // keys of the digit in earlier tiles
    for (int64_t t = tile - 1; t >= 0; t--) {
        uint64_t s = 0;
        for (int spin = 0; (s = state[t * RS_DIGITS + d0]) < RS_COUNT; spin++)
            if (spin > RS_SPIN_LIMIT) {
                sp.bad[1] = 1;
                s = RS_SUM;
                break;
            }
        before += s & (RS_COUNT - 1);
        if (s >= RS_SUM) break;
    }
    if (tile > 0) state[tile * RS_DIGITS + d0] = RS_SUM | (before + total);
    start[d0] = (int64_t)(sp.hist[pass * RS_DIGITS + d0] + before) - off;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; r++) {
        if (base + r * 32 >= n) continue;
        const unsigned d = (unsigned)(k[r] >> shift) & mask;
        const unsigned at = local[d] + cnt[w][d] + rank[r];
        s_keys[at] = k[r];
        s_idx[at] = v[r];
    }
    __syncthreads();
    const int64_t left = n - tile * RS_TILE;
    const int live = left < RS_TILE ? (int)left : RS_TILE;
    for (int i = threadIdx.x; i < live; i += RS_THREADS) {
        const KeyT key = s_keys[i];
        const int64_t at = start[(unsigned)(key >> shift) & mask] + i;
        if (at >= 0 && at < n) {                      // always, unless a look-back gave up
            keys_out[at] = key;
            idx_out[at] = s_idx[i];
        }
    }
}

template <typename KeyT, typename IdxT>
__global__ void __launch_bounds__(256)
rs_gather_kernel(int64_t n, const KeyT *__restrict__ keys, const IdxT *__restrict__ idx, int minor_bits,
                 const double *__restrict__ vals, const int64_t *__restrict__ payload, int64_t *__restrict__ major_out,
                 int64_t *__restrict__ minor_out, double *__restrict__ vals_out)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = keys[i];
        const int64_t from = vals_out || payload ? (int64_t)idx[i] : 0;
        if (major_out) major_out[i] = (int64_t)(k >> minor_bits);
        if (minor_out) minor_out[i] = payload ? payload[from] : (int64_t)(k & ((1ull << minor_bits) - 1ull));
        if (vals_out) vals_out[i] = vals[from];
    }
}

// pos[r] = first sorted key whose major coordinate is r or more
template <typename KeyT>
__global__ void __launch_bounds__(256)
rs_pos_kernel(int64_t n, const KeyT *__restrict__ keys, int minor_bits, int64_t nmajor, int64_t *__restrict__ pos)
{
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= nmajor; r += (int64_t)gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = n;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if ((int64_t)((uint64_t)keys[mid] >> minor_bits) < r) lo = mid + 1; else hi = mid;
        }
        pos[r] = lo;
    }
}

// row of every stored entry of a CSR matrix: 8 lanes per row
__global__ void __launch_bounds__(256)
expand_rows_kernel(int64_t nrows, const int64_t *__restrict__ pos, int64_t *__restrict__ rows)
{
    const int l = threadIdx.x & 7;
    const int64_t g = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int64_t ng = ((int64_t)gridDim.x * blockDim.x) >> 3;
    for (int64_t r = g; r < nrows; r += ng)
        for (int64_t p = pos[r] + l; p < pos[r + 1]; p += 8) rows[p] = r;
}

static unsigned grid_for(int64_t work)
{
    int64_t blocks = ceil_div(work > 0 ? work : 1, 256);
    const int64_t cap = (int64_t)sm_count() * 16;
    return (unsigned)(blocks > cap ? cap : blocks);
}

static int extent_bits(int64_t n)
{
    int b = 0;
    while (b < 63 && ((int64_t)1 << b) < n) b++;
    return b;
}

struct SortOut {
    int64_t *major, *minor, *pos;                     // pos: row pointer over the major coordinate
    double *vals;
};

// Sorted keys and positions of n entries in memory that the caller frees (sp.bad is its first byte).
template <typename KeyT, typename IdxT>
struct Sorted {
    char *mem = nullptr;
    SortPlan sp;
    KeyT *keys;
    IdxT *idx;
};

template <typename KeyT, typename IdxT>
static int sort_keys(int64_t n, int64_t nmajor, int64_t nminor, int bits, int minor_bits, const int64_t *major,
                     const int64_t *minor, const int64_t *limit, Sorted<KeyT, IdxT> *out, cudaStream_t st)
{
    SortPlan sp;
    sp.passes = bits > 0 ? (bits + 7) / 8 : 1;
    sp.width = bits > 0 ? (bits + sp.passes - 1) / sp.passes : 1;
    sp.ntiles = ceil_div(n, RS_TILE);
    auto pad = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t head = 256, hist = sizeof(uint64_t) * RS_DIGITS * sp.passes,
                 state = sizeof(uint64_t) * RS_DIGITS * sp.passes * (size_t)sp.ntiles, cleared = pad(head + hist + state);
    char *mem = nullptr;
    const size_t bytes = cleared + 2 * pad((size_t)n * sizeof(KeyT)) + 2 * pad((size_t)n * sizeof(IdxT));
    if (cudaMallocAsync((void **)&mem, bytes, st) != cudaSuccess) return fail("sort: device allocation of %zu bytes failed", bytes);
    sp.bad = (int *)mem;
    sp.ticket = (unsigned *)(mem + 64);
    sp.hist = (uint64_t *)(mem + head);
    sp.state = sp.hist + RS_DIGITS * sp.passes;
    KeyT *keys[2];
    IdxT *idx[2];
    keys[0] = (KeyT *)(mem + cleared);
    keys[1] = (KeyT *)((char *)keys[0] + pad((size_t)n * sizeof(KeyT)));
    idx[0] = (IdxT *)((char *)keys[1] + pad((size_t)n * sizeof(KeyT)));
    idx[1] = (IdxT *)((char *)idx[0] + pad((size_t)n * sizeof(IdxT)));
    cudaMemsetAsync(mem, 0, cleared, st);
    int64_t grid = ceil_div(n, 2048);
    if (grid > sm_count() * 4) grid = sm_count() * 4;
    const size_t hist_smem = sizeof(unsigned) * sp.passes * RS_DIGITS * RS_COPIES;
    const size_t tile_smem = (size_t)RS_TILE * (sizeof(KeyT) + sizeof(IdxT));
    cudaFuncSetAttribute(rs_make_keys_kernel<KeyT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist_smem);
    cudaFuncSetAttribute(rs_pass_kernel<KeyT, IdxT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem);
    cudaFuncSetAttribute(rs_pass_kernel<KeyT, IdxT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_smem);
    rs_make_keys_kernel<KeyT><<<(unsigned)grid, 256, hist_smem, st>>>(n, major, minor, nmajor, nminor, minor_bits, limit, keys[0], sp);
    rs_scan_kernel<<<(unsigned)sp.passes, RS_DIGITS, 0, st>>>(sp.hist);
    int from = 0;
    for (int p = 0; p < sp.passes; p++, from ^= 1) {
        if (p == 0)
            rs_pass_kernel<KeyT, IdxT, true><<<(unsigned)sp.ntiles, RS_THREADS, tile_smem, st>>>(
                n, keys[0], nullptr, keys[1], idx[1], p, sp);
        else
            rs_pass_kernel<KeyT, IdxT, false><<<(unsigned)sp.ntiles, RS_THREADS, tile_smem, st>>>(
                n, keys[from], idx[from], keys[from ^ 1], idx[from ^ 1], p, sp);
    }
    out->mem = mem;
    out->sp = sp;
    out->keys = keys[from];
    out->idx = idx[from];
    return 0;
}

template <typename KeyT, typename IdxT>
static int sort_entries(int64_t n, int64_t nmajor, int64_t nminor, int bits, int minor_bits, const int64_t *major,
                        const int64_t *minor, const double *vals, const int64_t *payload, const SortOut &out, cudaStream_t st)
{
    Sorted<KeyT, IdxT> s;
    CB_TRY((sort_keys<KeyT, IdxT>(n, nmajor, nminor, bits, minor_bits, major, minor, nullptr, &s, st)));
    char *mem = s.mem;
    const SortPlan sp = s.sp;
    rs_gather_kernel<KeyT, IdxT><<<grid_for(n), 256, 0, st>>>(n, s.keys, s.idx, minor_bits, vals, payload, out.major,
                                                             out.minor, vals ? out.vals : nullptr);
    if (out.pos) rs_pos_kernel<KeyT><<<grid_for(nmajor + 1), 256, 0, st>>>(n, s.keys, minor_bits, nmajor, out.pos);
    int rc = 0;
    PinnedWords words;
    int *bad = (int *)words.p;
    if (!bad || cudaMemcpyAsync(bad, sp.bad, 2 * sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess || cudaGetLastError() != cudaSuccess)
        rc = fail("sort: kernels failed");
    else if (bad[1])
        rc = fail("sort: a tile did not see its predecessors' counts");
    else if (bad[0])
        rc = fail("sort: a coordinate lies outside %lld x %lld", (long long)nmajor, (long long)nminor);
    cudaFreeAsync(mem, st);
    return rc;
}

// Entries sorted by (major, minor), equal coordinates in input order; `minor` null: by the major coordinate alone, and the
// minor output is payload[] of the entry.  Any of the outputs may be null.
static int sort_into(int64_t n, int64_t nmajor, int64_t nminor, const int64_t *major, const int64_t *minor, const double *vals,
                     const int64_t *payload, const SortOut &out, cudaStream_t st)
{
    if (nmajor <= 0 || nminor <= 0) return fail("sort: empty coordinate space");
    const int minor_bits = minor ? extent_bits(nminor) : 0, bits = minor_bits + extent_bits(nmajor);
    if (bits > 64) return fail("sort: rows x cols = %lld x %lld does not fit a 64-bit key", (long long)nmajor, (long long)nminor);
    const bool wide = n >= 0xffffffffLL;
#define GO(K, I) return sort_entries<K, I>(n, nmajor, nminor, bits, minor_bits, major, minor, vals, payload, out, st)
    if (bits <= 32) { if (wide) GO(uint32_t, uint64_t); GO(uint32_t, uint32_t); }
    if (wide) GO(uint64_t, uint64_t);
    GO(uint64_t, uint32_t);
#undef GO
}

int sort_coo(int64_t n, int64_t nmajor, int64_t nminor, const int64_t *major, const int64_t *minor,
             const double *vals, int64_t *major_out, int64_t *minor_out, double *vals_out, cudaStream_t st)
{
    if (n <= 0) return 0;
    return sort_into(n, nmajor, nminor, major, minor, vals, nullptr, {major_out, minor_out, nullptr, vals_out}, st);
}

// trow[q], tidx[q]: row and place of the q-th entry in column order; *err = 1 if the sort failed
__global__ void __launch_bounds__(256)
rs_index_kernel(int64_t n, const uint32_t *__restrict__ idx, const int32_t *__restrict__ row_of, int32_t *__restrict__ trow,
                int32_t *__restrict__ tidx, const int *bad, int *err)
{
    if (blockIdx.x == 0 && threadIdx.x == 0 && (bad[0] || bad[1])) *err = 1;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t from = idx[i];
        trow[i] = row_of[from];
        tidx[i] = (int32_t)from;
    }
}

int transpose_index(int64_t n, const int64_t *limit, int64_t ncols, const int64_t *crd, const int32_t *row_of, int64_t *tpos,
                    int32_t *trow, int32_t *tidx, int *err, cudaStream_t st)
{
    Sorted<uint32_t, uint32_t> s;
    CB_TRY((sort_keys<uint32_t, uint32_t>(n, ncols + 1, 1, extent_bits(ncols + 1), 0, crd, nullptr, limit, &s, st)));
    rs_index_kernel<<<grid_for(n), 256, 0, st>>>(n, s.idx, row_of, trow, tidx, s.sp.bad, err);
    rs_pos_kernel<uint32_t><<<grid_for(ncols + 1), 256, 0, st>>>(n, s.keys, 0, ncols, tpos);
    cudaFreeAsync(s.mem, st);
    CB_LAUNCH_CHECK();
    return 0;
}

}  // namespace cb200

using namespace cb200;

extern "C" int32_t comet_b200_dev_sort_coo_f64_i64(int64_t n, int64_t nmajor, int64_t nminor, const int64_t *major,
                                                   const int64_t *minor, const double *vals, int64_t *major_out,
                                                   int64_t *minor_out, double *vals_out, void *stream)
{
    clear_error();
    return sort_coo(n, nmajor, nminor, major, minor, vals, major_out, minor_out, vals_out, (cudaStream_t)stream);
}

extern "C" int32_t comet_b200_dev_coo_to_csr_f64_i64(int64_t nrows, int64_t ncols, int64_t nnz, const int64_t *rows,
                                                     const int64_t *cols, const double *vals, int64_t *pos,
                                                     int64_t *crd, double *val, void *stream)
{
    clear_error();
    cudaStream_t st = (cudaStream_t)stream;
    if (nrows < 0 || ncols < 0 || nnz < 0) return fail("coo_to_csr: negative size");
    if (nnz == 0) {
        CB_CUDA(cudaMemsetAsync(pos, 0, (size_t)(nrows + 1) * 8, st));
        return 0;
    }
    return sort_into(nnz, nrows, ncols, rows, cols, vals, nullptr, {nullptr, crd, pos, val}, st);
}

extern "C" int32_t comet_b200_dev_csr_transpose_f64_i64(int64_t nrows, int64_t ncols, int64_t nnz, const int64_t *pos,
                                                        const int64_t *crd, const double *val, int64_t *tpos,
                                                        int64_t *tcrd, double *tval, void *stream)
{
    clear_error();
    cudaStream_t st = (cudaStream_t)stream;
    if (nrows < 0 || ncols < 0 || nnz < 0) return fail("transpose: negative size");
    if (nnz == 0) {
        CB_CUDA(cudaMemsetAsync(tpos, 0, (size_t)(ncols + 1) * 8, st));
        return 0;
    }
    int64_t *rows = nullptr;
    CB_CUDA(cudaMallocAsync((void **)&rows, (size_t)nnz * 8, st));
    expand_rows_kernel<<<grid_for(nrows * 8), 256, 0, st>>>(nrows, pos, rows);
    // the entries are in row order already: a stable sort by column leaves every column's rows ascending
    const int rc = sort_into(nnz, ncols, nrows, crd, nullptr, val, rows, {nullptr, tcrd, tpos, tval}, st);
    cudaFreeAsync(rows, st);
    return rc;
}
