// Masked SpGEMM reduced to a scalar under plus-pair:
//   count = sum over stored A[i,k] of the number of entries of row k of B whose
//           column is stored in row i of M
// which is SUM(C<M,push> = A*B) with every product worth 1.  With A = B = M = L
// (strict lower triangle of a symmetric graph) it is the triangle count.
//
// Every stored A[i,k] asks for the size of the intersection of two sorted lists, M_i and B_k.  One of them is
// held as a SET in shared memory and the other is streamed past it, and it is the SHORTER one that is streamed:
// the reference's push mask always streams B_k, which on a power-law graph is usually the hub's list (R-MAT
// scale 22: 57.6 G elements streamed that way, 14.1 G the shorter way).  So the pairs (i,k) are split:
//   mask side   M_i is the set; the lists are the B_k of row i with |B_k| <= |M_i|, found by walking row i of A
//   B side      B_k is the set (more than TC_WARP_MAX entries and longer than M_i); the lists are the M_i of
//               all such i, found through a transposed list of these pairs (count, scan, scatter by k)
// All lists of one set are streamed against it without keeping them apart: only the total counts.
//
// Sets of more than TC_WARP_MAX entries are bitmaps over the columns: one shared-memory load per probe (the
// cuckoo table of earlier versions needed two, and shared-memory bank conflicts are what bounds the probing).
// A set's bits are put in before and taken out after its lists, so the whole bitmap is cleared once per CTA.
// The bitmap covers TC_MAX_COLS columns; a wider column space is first compacted to the columns that M stores
// (scale 22: 1.42 M of 4.19 M), and what still does not fit is walked segment by segment.
// Shorter sets take a cuckoo hash set per warp: two tables, two hash functions, every coordinate in one of its
// two slots, a probe is two loads and two compares with no loop (if an insertion chain does not end the set
// falls back to linear probing in the same memory).
//
// Repeated coordinates: one in M counts once (a bit), one in A or B per occurrence.  A bitmap of B_k would lose
// B's repeats and a streamed M_i count M's twice.  So the B side is switched off when M repeats a coordinate (a
// flag found while M is narrowed), and a B_k that sets a bit twice has its hits counted by a linear scan.
//
// Counts are exact int64; no floating point is involved.
// A matrix counted with itself that is large and triangular, as a graph's lower triangle, is renumbered first (order.cuh); only what lies
// beyond its hub columns is left to the kernels here.
//
// Measured on B200, R-MAT edge factor 16 lower triangles (mask side only, cuckoo sets in every bin -> both sides, bitmaps -> renumbered):
// scale 14 0.27 -> 0.16 ms, scale 18 1.96 -> 0.76, scale 20 10.2 -> 3.15 -> 2.38, scale 22 61.9 -> 18.4 -> 11.3.
#include "order.cuh"
#include "pairs.cuh"

namespace cb200 {

// present[j] = column j is stored in M (a bit each).  Most entries name a few hub columns, whose words would be a queue
// for the whole chip (0.9 ms on 64 M entries with a test before the atomic, 1.9 ms with plain byte stores), so a
// CTA remembers the columns it met last.  The table is read and written without order: a lost entry only repeats a test.
static const int TC_SEEN_SLOTS = 8192;

__global__ void __launch_bounds__(512)
tc_present_kernel(int64_t n, const int64_t *__restrict__ mcrd, uint32_t *__restrict__ present, const TcHeader *mode)
{
    if (mode && mode->ordered) return;
    __shared__ int32_t s_seen[TC_SEEN_SLOTS];
    for (int t = threadIdx.x; t < TC_SEEN_SLOTS; t += blockDim.x) s_seen[t] = -1;
    __syncthreads();
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const int32_t j = (int32_t)__ldcs((const long long *)mcrd + p);
        volatile int32_t *seen = s_seen + (((uint32_t)j * 0x9E3779B1u) >> 19);
        if (*seen == j) continue;
        *seen = j;
        const uint32_t bit = 1u << (j & 31);
        if (!(__ldcg(present + (j >> 5)) & bit)) atomicOr(present + (j >> 5), bit);
    }
}

__global__ void __launch_bounds__(256)
tc_popc_kernel(int64_t words, const uint32_t *__restrict__ present, int32_t *__restrict__ cnt)
{
    for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += (int64_t)gridDim.x * blockDim.x)
        cnt[w] = __popc(present[w]);
}

// int64 -> int32 coordinates.  present != null: columns are renumbered to their rank among the columns M stores, and
// the others to the number of those (a column no mask row has).  hdr != null: also counts the places inside rows
// [row_lo, row_hi) of `pos` where the coordinates do not ascend.
__global__ void __launch_bounds__(256)
tc_narrow_kernel(int64_t n, const int64_t *__restrict__ crd, int32_t *__restrict__ out,
                 const uint32_t *__restrict__ present, const int64_t *__restrict__ before, int64_t words,
                 const int64_t *__restrict__ pos, int64_t row_lo, int64_t row_hi, TcHeader *hdr, const TcHeader *mode)
{
    if (mode && mode->ordered) return;
    int64_t lo = 0, hi = 0;
    if (hdr) { lo = pos[row_lo]; hi = pos[row_hi] - 1; }
    unsigned desc = 0;
    for (int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 2; p < n; p += (int64_t)gridDim.x * blockDim.x * 2) {
        int64_t a, b = -1;
        if (p + 1 < n) {
            const longlong2 v = __ldcs((const longlong2 *)(crd + p));
            a = v.x; b = v.y;
        } else {
            a = crd[p];
        }
        if (hdr) {
            if (p >= lo && p < hi && b <= a) desc++;
            if (p + 1 >= lo && p + 1 < hi && crd[p + 2] <= b) desc++;
        }
        if (present) {
            auto rank = [&](int64_t j) {
                const uint32_t w = present[j >> 5], bit = 1u << (j & 31);
                return (w & bit) ? (int32_t)(before[j >> 5] + __popc(w & (bit - 1u))) : (int32_t)before[words];
            };
            a = rank(a);
            if (p + 1 < n) b = rank(b);
        }
        if (p + 1 < n) *(int2 *)(out + p) = make_int2((int)a, (int)b);
        else out[p] = (int32_t)a;
    }
    if (hdr && desc) atomicAdd(&hdr->desc_all, desc);
}

struct TriArrays {
    TriCounters *counters;
    uint32_t *degree, *bits;
    int32_t *rank, *hub_count, *rest_count, *bits_at;
    int64_t *hub_pos, *rest_pos, *sums;
    unsigned short *hub;
    int2 *edge;
    int32_t *place;
    unsigned long long room;               // words of `bits`
};

// eight bytes an entry hold all bitmaps of R-MAT graphs; rows that find no room do without
static size_t tri_room(int64_t nnz) { return nnz * 2 < ((int64_t)1 << 28) ? (size_t)nnz * 2 : (size_t)1 << 28; }
static size_t tri_pad(size_t bytes) { return (bytes + 255) & ~(size_t)255; }
static int64_t tri_tiles(int64_t nrows) { return ceil_div(nrows + 1, TRI_TILE); }
static size_t tri_bytes(int64_t nrows, int64_t nnz)
{
    return tri_pad(sizeof(TriCounters)) + 5 * tri_pad((size_t)nrows * 4) + 2 * tri_pad((size_t)(nrows + 1) * 8) +
           tri_pad((size_t)tri_tiles(nrows) * 16) + tri_pad((size_t)nnz * 2) + tri_room(nnz) * 4;
}

// Decides whether the matrix is counted in another order, and numbers its vertices and edges (mem: tri_bytes; edge, place: room for n of them).
// The kernels start while the one before them ends, so that those that find nothing to do cost little.  What a matrix pays that keeps its
// order, us without all this / with every kernel launched behind the whole of the one before it, all coordinates read for the degrees and
// six launches for two scans / now: uniform rows, 500,000 of 14 601 / 746 / 631, 1,000,000 of 16 1181 / 1440 / 1228, 3,000,000 of 12
// 3683 / 4187 / 3740; their lower triangles 598 / 704 / 640, 1231 / 1387 / 1301, 3476 / 3759 / 3617; R-MAT scale 20 x 16, not triangular,
// 7190 / 7300 / 7190.
static int tri_prepare(int64_t nrows, int64_t nnz, const int64_t *pos, const int64_t *crd, TcHeader *hdr, void *mem, int2 *edge, int32_t *place,
                       TriArrays *t, cudaStream_t st)
{
    const size_t b_n = tri_pad((size_t)nrows * 4), b_pos = tri_pad((size_t)(nrows + 1) * 8), b_tc = tri_pad(sizeof(TriCounters)),
                 b_hub = tri_pad((size_t)nnz * 2);
    t->room = tri_room(nnz);
    char *at = (char *)mem;
    auto take = [&](size_t bytes) { char *q = at; at += bytes; return (void *)q; };
    t->counters = (TriCounters *)take(b_tc);
    t->degree = (uint32_t *)take(b_n);
    t->hub_count = (int32_t *)take(b_n);
    t->rest_count = (int32_t *)take(b_n);
    t->rank = (int32_t *)take(b_n);
    t->bits_at = (int32_t *)take(b_n);
    t->hub_pos = (int64_t *)take(b_pos);
    t->rest_pos = (int64_t *)take(b_pos);
    t->sums = (int64_t *)take(tri_pad((size_t)tri_tiles(nrows) * 16));
    t->hub = (unsigned short *)take(b_hub);
    t->bits = (uint32_t *)at;
    t->edge = edge;
    t->place = place;
    CB_CUDA(cudaMemsetAsync(mem, 0, b_tc + b_n, st));             // counters, degrees
    const unsigned full = (unsigned)sm_count() * 8;
    auto grid = [&](int64_t items, int per) {
        const int64_t n = ceil_div(items, per);
        return (unsigned)(n < (int64_t)full ? n : (int64_t)full);
    };
    tri_degree_kernel<<<grid(nnz, 256 * 4 * TRI_SAMPLE), 256, 0, st>>>(nrows, nnz, pos, crd, t->degree, t->counters);
    CB_LAUNCH_CHECK();
    CB_CUDA(launch_behind(tri_hist_kernel, dim3(grid(nrows, 2048)), 512, 0, st, nrows, pos, crd, t->degree, t->counters));
    CB_CUDA(launch_behind(tri_decide_kernel, dim3(1), TRI_BUCKETS, 0, st, nnz, hdr, t->counters));
    CB_CUDA(launch_behind(tri_rank_kernel, dim3(grid(nrows, 2048)), 512, 0, st, nrows, t->degree, hdr, t->counters, t->rank,
                          t->hub_count, t->rest_count));
    CB_CUDA(launch_behind(tri_edges_kernel, dim3((unsigned)ceil_div(nnz, 4096)), 256, 0, st, nrows, nnz, pos, crd, t->rank, hdr, t->counters,
                          t->edge, t->place, t->hub_count, t->rest_count));
    const dim3 tiles((unsigned)tri_tiles(nrows), 2);
    CB_CUDA(launch_behind(tri_sums_kernel, tiles, 256, 0, st, nrows, t->hub_count, t->rest_count, hdr, t->sums));
    CB_CUDA(launch_behind(tri_totals_kernel, dim3(1), 1024, 0, st, nrows, (int64_t)tiles.x, hdr, t->counters, t->sums, t->hub_pos, t->rest_pos));
    CB_CUDA(launch_behind(tri_places_kernel, tiles, 256, 0, st, nrows, t->hub_count, t->rest_count, pos, hdr, t->sums, t->hub_pos, t->rest_pos));
    return 0;
}

// Counts the triangles of the hub columns; the rest of the rows goes to a32 and, where that is another array, counted from the first of its
// columns, to m32.
static int tri_count(int64_t nrows, int64_t nnz, TcHeader *hdr, TriArrays *t, int32_t *a32, int32_t *m32,
                     int64_t *columns, int64_t *count_dev, cudaStream_t st)
{
    const unsigned sms = (unsigned)sm_count();
    CB_CUDA(launch_behind(tri_scatter_kernel, dim3(sms * 8), 256, 0, st, nnz, t->edge, t->place, t->hub_pos, t->rest_pos, hdr, t->counters,
                          t->hub, a32, m32, columns));
    CB_CUDA(launch_behind(tri_bitmap_kernel, dim3(sms * 6), TRI_WARPS * 32, 0, st, nrows, t->hub_pos, t->hub, hdr, t->counters, t->room,
                          t->bits_at, t->bits));
    CB_CUDA(launch_behind(tri_count_kernel, dim3(sms * 5), TRI_WARPS * 32, 0, st, nrows, t->hub_pos, t->hub, t->rest_pos, a32, t->bits_at, t->bits,
                          hdr, t->counters, (unsigned long long *)count_dev));
    return 0;
}

int masked_pair_count(int64_t row_lo, int64_t row_hi, int64_t ncols, int64_t nnz_a, int64_t nnz_b,
                      int64_t nnz_m, const int64_t *apos, const int64_t *acrd, const int64_t *bpos,
                      const int64_t *bcrd, const int64_t *mpos, const int64_t *mcrd,
                      int64_t *count_dev, cudaStream_t st)
{
    CB_CUDA(cudaMemsetAsync(count_dev, 0, sizeof(int64_t), st));
    if (row_hi <= row_lo || nnz_a <= 0 || nnz_b <= 0 || nnz_m <= 0) return 0;
    if (ncols >= 0x7fffffffLL || row_hi >= 0x7fffffffLL)
        return fail("masked count: more than 2^31-1 rows or columns is not supported");
    if ((((uintptr_t)acrd | (uintptr_t)bcrd | (uintptr_t)mcrd) & 15) != 0)
        return fail("masked count: crd arrays must be 16-byte aligned");
    const int64_t nrows = row_hi - row_lo;
    // rows of B the B side keeps a list for: B's row count is not among the arguments, its column count is, and the
    // two agree for the square operands this is called with (pairs beyond it stay on the mask side)
    const int64_t bcap = ncols > row_hi ? ncols : row_hi;
    const bool compact = ncols > TC_MAX_COLS;
    const int64_t words = ceil_div(ncols, 32);
    auto grid_for = [](int64_t n) {
        const int64_t blocks = ceil_div(n, 256), cap = (int64_t)sm_count() * 16;
        return (unsigned)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
    };
    const bool same_bm = bcrd == mcrd && nnz_b == nnz_m, same_am = acrd == mcrd && nnz_a == nnz_m;
    const bool same_ab = acrd == bcrd && nnz_a == nnz_b;
    // one matrix in all three places: its triangles, if it is triangular, in another order of the vertices
    const bool suits = same_am && same_bm && apos == mpos && bpos == mpos && row_lo == 0 && row_hi == ncols &&
                       nnz_a >= TRI_MIN_ENTRIES && nnz_a / TRI_MIN_PER_ROW >= ncols && nnz_a < 0x7fffffffLL;

    // scratch: header, rows of A, list places, B side lists and their pointers, unit list
    const size_t nunits = (size_t)(nnz_a / 16 + (nnz_m < nrows * TC_WARP_MAX ? nnz_m / TC_WARP_MAX : nrows) +
                                   (nnz_b < bcap * TC_WARP_MAX ? nnz_b / TC_WARP_MAX : bcap) + 64);
    void *hdrp = nullptr, *a32 = nullptr, *b32 = nullptr, *m32 = nullptr, *rows = nullptr, *bins = nullptr;
    auto pad = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
    const size_t counts_bytes = pad(sizeof(TcHeader)) + pad((size_t)bcap * 4) + (compact ? pad((size_t)words * 4) : 0);
    const size_t hdr_bytes = counts_bytes + pad((size_t)(bcap + 1) * 8) +
                             (compact ? pad((size_t)words * 4) + pad((size_t)(words + 1) * 8) : 0);
    CB_TRY(scratch(SLOT_MISC, hdr_bytes, &hdrp));
    char *at = (char *)hdrp;
    auto take = [&](size_t bytes) { char *q = at; at += pad(bytes); return (void *)q; };
    TcHeader *hdr = (TcHeader *)take(sizeof(TcHeader));
    int32_t *bcount = (int32_t *)take((size_t)bcap * 4);
    uint32_t *present = compact ? (uint32_t *)take((size_t)words * 4) : nullptr;
    int64_t *bptr = (int64_t *)take((size_t)(bcap + 1) * 8);
    int32_t *popc = compact ? (int32_t *)take((size_t)words * 4) : nullptr;
    int64_t *before = compact ? (int64_t *)take((size_t)(words + 1) * 8) : nullptr;
    CB_TRY(scratch(SLOT_ROWINFO, pad((size_t)nnz_a * 4) * 2 + pad((size_t)nnz_a * 8), &rows));
    int32_t *arow = (int32_t *)rows, *slot = (int32_t *)((char *)rows + pad((size_t)nnz_a * 4));
    int2 *blist = (int2 *)((char *)rows + 2 * pad((size_t)nnz_a * 4));
    CB_TRY(scratch(SLOT_BINS, pad((size_t)nrows * 4) + 2 * nunits * sizeof(TcUnit), &bins));
    int32_t *small = (int32_t *)bins;
    TcUnit *units = (TcUnit *)((char *)bins + pad((size_t)nrows * 4)), *mids = units + nunits;
    CB_TRY(scratch(SLOT_NARROW_M, (size_t)nnz_m * 4 + 16, &m32));
    if (same_bm) b32 = m32;
    else CB_TRY(scratch(SLOT_NARROW_B, (size_t)nnz_b * 4 + 16, &b32));
    if (same_am && !compact) a32 = m32;
    else if (same_ab && !compact) a32 = b32;
    else CB_TRY(scratch(SLOT_NARROW_A, (size_t)nnz_a * 4 + 16, &a32));
    CB_TRY(exclusive_scan_room(bcap > words ? bcap : words));
    // after all that the count cannot do without
    ScratchIfRoom tri_mem;
    if (suits) tri_mem.take(SLOT_TRIANGLES, tri_bytes(row_hi, nnz_a));
    const bool order = tri_mem.p != nullptr;               // else in the order it has
    const TcShape sh = {bcap, acrd == mcrd && apos == mpos, false, false, order};
    CB_CUDA(cudaMemsetAsync(hdr, 0, counts_bytes, st));           // header, list counts, column bits

    TriArrays tri;
    if (order) CB_TRY(tri_prepare(row_hi, nnz_a, apos, acrd, hdr, tri_mem.p, blist, slot, &tri, st));

    if (compact) {
        tc_present_kernel<<<(unsigned)sm_count() * 4, 512, 0, st>>>(nnz_m, mcrd, present, order ? hdr : nullptr);
        CB_LAUNCH_CHECK();
        tc_popc_kernel<<<grid_for(words), 256, 0, st>>>(words, present, popc);
        CB_LAUNCH_CHECK();
        CB_TRY(exclusive_scan_i32(popc, before, words, st));
    }
    auto narrow = [&](const int64_t *crd, int64_t n, void *out, bool columns, bool check) {
        tc_narrow_kernel<<<grid_for(ceil_div(n, 2)), 256, 0, st>>>(n, crd, (int32_t *)out, columns ? present : nullptr, before,
                                                                  words, mpos, row_lo, row_hi, check ? hdr : nullptr, order ? hdr : nullptr);
        return cudaGetLastError() == cudaSuccess ? 0 : fail("masked count: narrowing failed");
    };
    CB_TRY(narrow(mcrd, nnz_m, m32, true, true));
    if (b32 != m32) CB_TRY(narrow(bcrd, nnz_b, b32, true, false));
    if (a32 != m32 && a32 != b32) CB_TRY(narrow(acrd, nnz_a, a32, false, false));
    const int32_t *A = (const int32_t *)a32, *B = (const int32_t *)b32, *M = (const int32_t *)m32;
    if (order) {
        CB_TRY(tri_count(row_hi, nnz_a, hdr, &tri, (int32_t *)a32, (int32_t *)m32, compact ? before + words : nullptr, count_dev, st));
        apos = bpos = mpos = tri.rest_pos;
    }
    tc_rows_kernel<<<grid_for(nrows * 16), 256, 0, st>>>(row_lo, row_hi, apos, mpos, mcrd, arow, hdr);
    CB_LAUNCH_CHECK();
    tc_route_kernel<<<grid_for(nnz_a), 256, 0, st>>>(row_lo, row_hi, apos, A, arow, bpos, mpos, sh, hdr, slot, bcount);
    CB_LAUNCH_CHECK();
    CB_TRY(exclusive_scan_i32(bcount, bptr, bcap, st));
    tc_scatter_kernel<<<grid_for(nnz_a), 256, 0, st>>>(row_lo, row_hi, apos, A, arow, slot, bptr, blist);
    CB_LAUNCH_CHECK();
    const int64_t most = nrows > bcap ? nrows : bcap;
    auto clamp = [](int64_t v, int64_t lo, int64_t hi) { return (unsigned)(v < lo ? lo : (v > hi ? hi : v)); };
    tc_units_kernel<<<(unsigned)ceil_div(most, 256), 256, 0, st>>>(row_lo, row_hi, bcap, apos, mpos, bpos, bptr, hdr, small,
                                                                  mids, units, clamp(nnz_a / (sm_count() * 192), 32, 512),
                                                                  clamp(nnz_a / (sm_count() * 64), 64, 4096));
    CB_LAUNCH_CHECK();
    const TcCountAll out = {(unsigned long long *)count_dev, 0};
    const int width = (int)(compact ? TC_MAX_COLS : ncols);
    const size_t smem = (size_t)2 * TC_SET_BUF * 4 + (size_t)((width >> 5) + 1) * 4;
    const int64_t *ncols_dev = compact ? before + words : nullptr;
    // one CTA of 32 warps per SM where two bitmaps do not fit well, otherwise two of 16
    if (compact)
        CB_TRY((launch_bitmap<1024, true>(smem, hdr, units, apos, A, bpos, B, mpos, M, bptr, blist, sh, width, ncols_dev,
                                          out, st)));
    else if (smem > 52 * 1024)
        CB_TRY((launch_bitmap<1024, false>(smem, hdr, units, apos, A, bpos, B, mpos, M, bptr, blist,
                                           sh, width, ncols_dev, out, st)));
    else
        CB_TRY((launch_bitmap<512, false>(smem, hdr, units, apos, A, bpos, B, mpos, M, bptr, blist, sh, width, ncols_dev,
                                          out, st)));
    tc_mid_kernel<<<(unsigned)sm_count() * 6, TC_MID_WARPS * 32, 0, st>>>(hdr, mids, apos, A, bpos, B, mpos, M, bptr, blist,
                                                                          sh, out);
    CB_LAUNCH_CHECK();
    tc_warp_kernel<<<(unsigned)sm_count() * 8, TC_WARPS * 32, 0, st>>>(hdr, small, apos, A, bpos, B, mpos, M, sh, out);
    CB_LAUNCH_CHECK();
    return 0;
}

}  // namespace cb200

extern "C" int32_t comet_b200_dev_masked_spgemm_count_f64_i64(
    int64_t row_lo, int64_t row_hi, int64_t ncols, int64_t nnz_a, int64_t nnz_b, int64_t nnz_m,
    const int64_t *apos, const int64_t *acrd, const int64_t *bpos, const int64_t *bcrd,
    const int64_t *mpos, const int64_t *mcrd, int64_t *count_dev, void *stream)
{
    cb200::clear_error();
    return cb200::masked_pair_count(row_lo, row_hi, ncols, nnz_a, nnz_b, nnz_m, apos, acrd, bpos, bcrd,
                                    mpos, mcrd, count_dev, (cudaStream_t)stream);
}
