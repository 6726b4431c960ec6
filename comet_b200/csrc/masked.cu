// C<M,push> = A * B with C stored: one dot product of row i of A and column j of B per mask entry (i,j).
//
// The push form walks the products of row i and looks every product's column up in the mask row; the sum over the rows
// is what the unmasked product costs, and the look-up was a binary search.  Here B is transposed once (a sort of its
// entries by column) and every mask entry intersects two ascending lists, A_i and B_j, with the machinery of the masked
// count (pairs.cuh): the longer list is a set in shared memory, the shorter one is streamed past it.  An R-MAT graph of
// scale 15, edge factor 16, squared under itself as mask has 442 M products and 125 M elements in the shorter lists.
//
// Symbolic: the number of common positions of every mask entry (kept: it is the value under plus-pair, and where it is
// zero there is no entry of C); a mask entry that repeats the one before it counts as none.  Numeric: under another
// semiring a second pass over the mask entries with hits folds the products; then every row's entries are written in
// mask order, which is ascending.
//
// Where A, B and M are one symmetric pattern (the adjacency matrix of a graph: the device looks every entry's mate up, 39 us), B needs
// no transposing, the entries (i,j) and (j,i) have the same count and are counted once, with the longer list as the set, so nothing has
// to be routed to the other side; a second pass folds the values of both.
//
// Taken when A's rows ascend strictly (checked on the device; a set or a list with repeats would count them wrong, and
// so would B's, whose check is part of the transpose), when the bitmaps cover A's columns, and when the bound
// sum |M_i| |A_i| on the elements streamed is at most MASKED_DOT_COST times the products of the push form: a mask much
// denser than the product it masks is cheaper to push.
// Measured on B200, push form and now: a symmetric graph of scale 15, edge factor 16, under plus-pair 18.7 -> 0.36 ms, under plus-times
// 19.5 -> 1.21.  Of the 0.36 the set kernels take 0.21 (bitmaps 0.105, hash sets 0.076 and 0.031), the checks and the mates 0.06.  Not
// symmetric, of the same scale: 0.42 and 0.88; set kernels 0.19, transposing 0.06, routing 0.03.  Scale 9, edge factor 8: 0.16 and 0.33
// symmetric, 0.19 and 0.28 not (13 or 24 launches in the symbolic call, two synchronisations).
#include <string.h>

#include "hostcopy.cuh"
#include "masked.cuh"
#include "pairs.cuh"
#include "stream.cuh"

namespace cb200 {

static const double MASKED_DOT_COST = 4.0;

struct MaskedStats {
    unsigned long long nrows_b;            // rows of B that A names
    unsigned long long products, bound;
    unsigned long long desc_all, desc_edge;           // places where A's coordinates do not ascend: all, and at row starts
    unsigned nnz_a, nnz_m;                 // 0xffffffff: that or more
    unsigned long long one_sided;          // not 0: some entry of A has no mate, see masked_mates_kernel
    unsigned long long balance;            // not 0: some vertex has not as many entries in its row as in its column
};
static_assert(sizeof(MaskedStats) <= 64, "fits a page-locked word block");

struct MaskedPlan {
    char *mem;
    int64_t nrows, ncols, nnz_m, nnz_b;
    int64_t width;                         // columns of A that occur
    TcHeader *hdr;
    int *err;                              // [0] the sort failed, [1] and [2] see masked_rows_kernel
    int32_t *a32, *m32, *trow, *tidx, *cnt, *small;
    int2 *blist;
    int64_t *tpos, *bptr, *place;
    TcUnit *units, *mids;
    const int64_t *apos, *mpos;
    int32_t *mate;                         // not null: A, B and M are one symmetric pattern; place of (j,i) for every entry (i,j)
};

static unsigned flat_grid(int64_t n)
{
    const int64_t blocks = ceil_div(n, 256), cap = (int64_t)sm_count() * 8;
    return (unsigned)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

// a vertex's weight in MaskedStats::balance
__device__ __forceinline__ unsigned long long masked_weight(int64_t k)
{
    unsigned long long h = (unsigned long long)(k + 1) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 29;
    return h * 0xBF58476D1CE4E5B9ull;
}

// same: A, B and M are one square matrix.  It cannot be symmetric unless the weights of its entries' columns add up to those of their
// rows, which rules out nearly every other one without a look-up (masked_mates_kernel took 130 us of 1847 on a lower triangle of 4 M entries).
__global__ void __launch_bounds__(256)
masked_stats_kernel(int64_t nrows, const int64_t *__restrict__ apos, const int64_t *__restrict__ acrd,
                    const int64_t *__restrict__ bpos, const int64_t *__restrict__ mpos, bool same, MaskedStats *stats)
{
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t n = apos[nrows];
    unsigned long long top = 0, products = 0, bound = 0, balance = 0;
    unsigned desc = 0, edge = 0;
    for (int64_t p = t0; p < n; p += stride) {
        const int64_t k = acrd[p];
        if ((unsigned long long)(k + 1) > top) top = (unsigned long long)(k + 1);
        products += (unsigned long long)(bpos[k + 1] - bpos[k]);
        if (p + 1 < n && acrd[p + 1] <= k) desc++;
        if (same) balance += masked_weight(k);
    }
    for (int64_t r = t0; r < nrows; r += stride) {
        const int64_t s = apos[r], e = apos[r + 1];
        bound += (unsigned long long)(e - s) * (unsigned long long)(mpos[r + 1] - mpos[r]);
        if (s > 0 && e > s && acrd[s] <= acrd[s - 1]) edge++;
        if (same) balance -= (unsigned long long)(e - s) * masked_weight(r);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, top, o);
        top = v > top ? v : top;
        products += __shfl_xor_sync(0xffffffffu, products, o);
        bound += __shfl_xor_sync(0xffffffffu, bound, o);
        balance += __shfl_xor_sync(0xffffffffu, balance, o);
    }
    desc = __reduce_add_sync(0xffffffffu, desc);
    edge = __reduce_add_sync(0xffffffffu, edge);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&stats->nrows_b, top);
        if (products) atomicAdd(&stats->products, products);
        if (bound) atomicAdd(&stats->bound, bound);
        if (balance) atomicAdd(&stats->balance, balance);
        if (desc) atomicAdd(&stats->desc_all, (unsigned long long)desc);
        if (edge) atomicAdd(&stats->desc_edge, (unsigned long long)edge);
    }
    if (t0 == 0) {
        const int64_t m = mpos[nrows];
        stats->nnz_a = n < 0xffffffffLL ? (unsigned)n : 0xffffffffu;
        stats->nnz_m = m < 0xffffffffLL ? (unsigned)m : 0xffffffffu;
    }
}

// Row of every entry of the rows of B that are used (16 lanes per row), and the places where their coordinates do not
// ascend: all (desc[0]) and those at row starts (desc[1]).  The two differ where a row repeats or misorders a coordinate.
__global__ void __launch_bounds__(256)
masked_rows_kernel(int64_t nrows, const int64_t *__restrict__ bpos, const int64_t *__restrict__ bcrd, int32_t *__restrict__ rows,
                   unsigned *desc)
{
    const int l = threadIdx.x & 15;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned all = 0, edge = 0;
    for (int64_t r = t0 >> 4; r < nrows; r += stride >> 4) {
        const int64_t s = bpos[r], e = bpos[r + 1];
        for (int64_t p = s + l; p < e; p += 16) rows[p] = (int32_t)r;
        if (l == 0 && s > 0 && e > s && bcrd[s] <= bcrd[s - 1]) edge++;
    }
    const int64_t n = bpos[nrows];
    for (int64_t p = t0; p + 1 < n; p += stride) all += bcrd[p + 1] <= bcrd[p] ? 1u : 0u;
    all = __reduce_add_sync(0xffffffffu, all);
    edge = __reduce_add_sync(0xffffffffu, edge);
    if ((threadIdx.x & 31) == 0) {
        if (all) atomicAdd(desc, all);
        if (edge) atomicAdd(desc + 1, edge);
    }
}

// A square pattern of strictly ascending rows: the place of (j,i) for every entry (i,j), or that some entry has none.
// A thread per entry: its row by a search in the row pointer, its mate by one in row j.  Ends with the first entry that has none (as many in
// every row as in every column, but not symmetric: 16 neighbours on one side of each of 200,000 vertices of a ring, plus-pair, without a
// search 648 us, with all of them 755, so 672).
__global__ void __launch_bounds__(256)
masked_mates_kernel(int64_t nrows, const int64_t *__restrict__ pos, const int64_t *__restrict__ crd, int64_t room,
                    int32_t *__restrict__ mate, MaskedStats *stats)
{
    wait_for_previous();
    const int64_t n = pos[nrows];
    if (stats->balance) {                              // some entry has none
        if (blockIdx.x == 0 && threadIdx.x == 0) stats->one_sided = 1;
        return;
    }
    unsigned none = n > room;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n && p < room; p += (int64_t)gridDim.x * blockDim.x) {
        const bool found = *(volatile unsigned long long *)&stats->one_sided != 0;       // looked at when this entry is done
        int64_t lo = 0, hi = nrows - 1;
        while (lo < hi) {                              // the first row that ends behind p
            const int64_t mid = (lo + hi) >> 1;
            if (pos[mid + 1] <= p) lo = mid + 1; else hi = mid;
        }
        const int64_t i = lo, j = crd[p], e = pos[j + 1];
        lo = pos[j];
        hi = e;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (crd[mid] < i) lo = mid + 1; else hi = mid;
        }
        if (lo < e && crd[lo] == i) mate[p] = (int32_t)lo;
        else none = 1;
        if (none || found) break;
    }
    none = __reduce_add_sync(0xffffffffu, none);
    if ((threadIdx.x & 31) == 0 && none) atomicAdd(&stats->one_sided, (unsigned long long)none);
}

// the entries left out have their mates' counts (an entry and its mate write the same)
__global__ void __launch_bounds__(256)
masked_mirror_kernel(int64_t n, const int32_t *__restrict__ mate, int32_t *cnt)
{
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const int32_t c = cnt[mate[p]];
        if (c > cnt[p]) cnt[p] = c;
    }
}

// row pointer of C: entries of C before row r = mask entries with hits before it
__global__ void __launch_bounds__(256)
masked_pos_kernel(int64_t nrows, const int64_t *__restrict__ mpos, const int64_t *__restrict__ place, int64_t *__restrict__ cpos)
{
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r <= nrows; r += (int64_t)gridDim.x * blockDim.x)
        cpos[r] = place[mpos[r]];
}

// the mask entries with hits are C's entries, in their order
__global__ void __launch_bounds__(256)
masked_compact_kernel(int64_t n, const int64_t *__restrict__ mcrd, const int32_t *__restrict__ cnt,
                      const int64_t *__restrict__ place, const double *__restrict__ val, bool any, int64_t *__restrict__ ccrd,
                      double *__restrict__ cval)
{
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const int32_t c = cnt[p];
        if (c == 0) continue;
        const int64_t q = place[p];
        ccrd[q] = mcrd[p];
        cval[q] = val ? val[p] : (any ? 1.0 : (double)c);
    }
}

__global__ void __launch_bounds__(256)
masked_gather_kernel(int64_t n, const int32_t *__restrict__ idx, const double *__restrict__ val, double *__restrict__ out)
{
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
        out[p] = val[idx[p]];
}

template <class Out>
static int run_pairs(MaskedPlan *m, const Out &out, cudaStream_t st)
{
    // "A" of the pairs is the mask, "M" is A, "B" is the transposed B
    const TcShape sh = {m->mate ? 0 : m->ncols, false, true, m->mate != nullptr, false};
    const int width = (int)m->width;
    const size_t smem = (size_t)2 * TC_SET_BUF * 4 + (size_t)((width >> 5) + 1) * 4;
    if (smem > 52 * 1024)
        CB_TRY((launch_bitmap<1024, false>(smem, m->hdr, m->units, m->mpos, m->m32, m->tpos, m->trow,
                                           m->apos, m->a32, m->bptr, m->blist, sh, width, nullptr, out, st)));
    else
        CB_TRY((launch_bitmap<512, false>(smem, m->hdr, m->units, m->mpos, m->m32, m->tpos, m->trow, m->apos, m->a32, m->bptr,
                                          m->blist, sh, width, nullptr, out, st)));
    tc_mid_kernel<<<(unsigned)sm_count() * 6, TC_MID_WARPS * 32, 0, st>>>(m->hdr, m->mids, m->mpos, m->m32, m->tpos, m->trow,
                                                                          m->apos, m->a32, m->bptr, m->blist, sh, out);
    CB_LAUNCH_CHECK();
    tc_warp_kernel<<<(unsigned)sm_count() * 8, TC_WARPS * 32, 0, st>>>(m->hdr, m->small, m->mpos, m->m32, m->tpos, m->trow,
                                                                       m->apos, m->a32, sh, out);
    CB_LAUNCH_CHECK();
    return 0;
}

const int *masked_checks(const MaskedPlan *plan) { return plan->err; }

void masked_free(MaskedPlan *plan, cudaStream_t st)
{
    if (!plan) return;
    if (plan->mem) cudaFreeAsync(plan->mem, st);
    if (plan->mate) cudaFreeAsync(plan->mate, st);
    delete plan;
}

int masked_symbolic(int64_t nrows, int64_t ncols_b, int64_t nnz_b, const int64_t *apos, const int64_t *acrd, const int64_t *bpos,
                    const int64_t *bcrd, const int64_t *mpos, const int64_t *mcrd, int64_t *cpos, MaskedPlan **plan,
                    cudaStream_t st)
{
    *plan = nullptr;
    if (nrows <= 0 || ncols_b <= 0 || nnz_b <= 0 || nnz_b >= 0x7fffffffLL) return 0;
    void *sp = nullptr;
    CB_TRY(scratch(SLOT_MISC, sizeof(MaskedStats), &sp));
    CB_CUDA(cudaMemsetAsync(sp, 0, sizeof(MaskedStats), st));
    // one matrix in all three places: it may be symmetric, as the adjacency matrix of a graph is
    const bool same = nrows == ncols_b && apos == bpos && apos == mpos && acrd == bcrd && acrd == mcrd;
    masked_stats_kernel<<<(unsigned)sm_count() * 4, 256, 0, st>>>(nrows, apos, acrd, bpos, mpos, same, (MaskedStats *)sp);
    CB_LAUNCH_CHECK();
    int32_t *mate = nullptr;
    if (same && cudaMallocAsync((void **)&mate, (size_t)nnz_b * 4, st) != cudaSuccess) {
        (void)cudaGetLastError();
        mate = nullptr;
    }
    MaskedPlan *m = new MaskedPlan();
    m->mate = mate;                        // freed with the plan
    if (mate) launch_behind(masked_mates_kernel, dim3(flat_grid(nnz_b)), 256, 0, st, nrows, apos, acrd, nnz_b, mate, (MaskedStats *)sp);
    MaskedStats s;
    {
        PinnedWords words;
        int rc = words.p ? 0 : fail("spgemm: no page-locked memory");
        if (!rc && (cudaGetLastError() != cudaSuccess || cudaMemcpyAsync(words.p, sp, sizeof(s), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                    cudaStreamSynchronize(st) != cudaSuccess))
            rc = fail("spgemm: looking the operands over failed");
        if (rc) {
            masked_free(m, st);
            return rc;
        }
        memcpy(&s, words.p, sizeof(s));
    }
    if (s.nnz_a == 0 || s.nnz_m == 0 || s.nnz_a >= 0x7fffffffu || s.nnz_m >= 0x7fffffffu || s.desc_all != s.desc_edge ||
        (int64_t)s.nrows_b > TC_MAX_COLS || (double)s.bound > MASKED_DOT_COST * (double)s.products) {
        masked_free(m, st);
        return 0;
    }
    if (m->mate && s.one_sided) {
        cudaFreeAsync(m->mate, st);
        m->mate = nullptr;
    }
    const bool sym = m->mate != nullptr;
    m->nrows = nrows; m->ncols = ncols_b; m->nnz_m = s.nnz_m; m->width = (int64_t)s.nrows_b; m->nnz_b = nnz_b;
    m->apos = apos; m->mpos = mpos;
    const size_t nunits = (size_t)(s.nnz_m / 16 + (s.nnz_a < nrows * TC_WARP_MAX ? s.nnz_a / TC_WARP_MAX : nrows) +
                                   (nnz_b < ncols_b * TC_WARP_MAX ? nnz_b / TC_WARP_MAX : ncols_b) + 64);
    auto pad = [](size_t bytes) { return (bytes + 255) & ~(size_t)255; };
    size_t total = 0;
    auto want = [&](size_t bytes) { const size_t at = total; total += pad(bytes); return at; };
    // cleared: headers (the second one only collects what tc_rows_kernel counts), list counts, hits
    const size_t o_hdr = want(3 * sizeof(TcHeader)), o_bcount = want((size_t)ncols_b * 4), o_cnt = want((size_t)s.nnz_m * 4);
    const size_t cleared = total;
    const size_t o_a32 = want((size_t)s.nnz_a * 4 + 16), o_small = want((size_t)nrows * 4), o_place = want(((size_t)s.nnz_m + 1) * 8),
                 o_units = want(nunits * sizeof(TcUnit)), o_mids = want(nunits * sizeof(TcUnit));
    // not needed for a symmetric pattern, which is its own transpose and has no B side
    auto want_too = [&](size_t bytes) { return sym ? 0 : want(bytes); };
    const size_t o_m32 = want_too((size_t)s.nnz_m * 4 + 16), o_trow = want_too((size_t)nnz_b * 4 + 16), o_tidx = want_too((size_t)nnz_b * 4),
                 o_tpos = want_too((size_t)(ncols_b + 1) * 8), o_bptr = want_too((size_t)(ncols_b + 1) * 8),
                 o_blist = want_too((size_t)s.nnz_m * 8), o_rows = want_too((size_t)(nnz_b > s.nnz_m ? nnz_b : s.nnz_m) * 4),
                 o_slot = want_too((size_t)s.nnz_m * 4);
    if (cudaMallocAsync((void **)&m->mem, total, st) != cudaSuccess) {
        (void)cudaGetLastError();
        m->mem = nullptr;
        masked_free(m, st);
        return 0;                          // the push form needs less memory
    }
    auto at = [&](size_t o) { return (void *)(m->mem + o); };
    m->hdr = (TcHeader *)at(o_hdr);
    m->err = (int *)(m->hdr + 2);
    m->cnt = (int32_t *)at(o_cnt);
    m->a32 = (int32_t *)at(o_a32); m->m32 = (int32_t *)at(o_m32);
    m->trow = (int32_t *)at(o_trow); m->tidx = (int32_t *)at(o_tidx); m->tpos = (int64_t *)at(o_tpos);
    m->bptr = (int64_t *)at(o_bptr); m->blist = (int2 *)at(o_blist); m->small = (int32_t *)at(o_small);
    m->place = (int64_t *)at(o_place);
    m->units = (TcUnit *)at(o_units); m->mids = (TcUnit *)at(o_mids);
    if (sym) {
        m->m32 = m->trow = m->a32;
        m->tidx = m->mate;
        m->tpos = const_cast<int64_t *>(apos);
    }
    int32_t *bcount = (int32_t *)at(o_bcount), *rows = (int32_t *)at(o_rows), *slot = (int32_t *)at(o_slot);

    auto build = [&]() {
        CB_CUDA(cudaMemsetAsync(m->mem, 0, cleared, st));
        CB_TRY(narrow_any_i64_to_i32(acrd, m->a32, s.nnz_a, st));
        const TcShape sh = {ncols_b, false, true, false, false};
        if (!sym) {
            CB_TRY(narrow_any_i64_to_i32(mcrd, m->m32, s.nnz_m, st));
            masked_rows_kernel<<<flat_grid(m->width * 16), 256, 0, st>>>(m->width, bpos, bcrd, rows, (unsigned *)m->err + 1);
            CB_LAUNCH_CHECK();
            CB_TRY(transpose_index(nnz_b, bpos + m->width, ncols_b, bcrd, rows, m->tpos, m->trow, m->tidx, m->err, st));
            tc_rows_kernel<<<flat_grid(nrows * 16), 256, 0, st>>>(0, nrows, mpos, apos, acrd, rows, m->hdr + 1);
            CB_LAUNCH_CHECK();
            tc_route_kernel<<<flat_grid(s.nnz_m), 256, 0, st>>>(0, nrows, mpos, m->m32, rows, m->tpos, apos, sh, m->hdr, slot, bcount);
            CB_LAUNCH_CHECK();
            CB_TRY(exclusive_scan_i32(bcount, m->bptr, ncols_b, st));
            tc_scatter_kernel<<<flat_grid(s.nnz_m), 256, 0, st>>>(0, nrows, mpos, m->m32, rows, slot, m->bptr, m->blist);
            CB_LAUNCH_CHECK();
        }
        auto clamp = [](int64_t v, int64_t lo, int64_t hi) { return (unsigned)(v < lo ? lo : (v > hi ? hi : v)); };
        const int64_t most = nrows > ncols_b ? nrows : ncols_b;
        tc_units_kernel<<<(unsigned)ceil_div(most, 256), 256, 0, st>>>(0, nrows, sym ? 0 : ncols_b, mpos, apos, m->tpos, m->bptr, m->hdr,
                                                                      m->small, m->mids, m->units,
                                                                      clamp(s.nnz_m / (sm_count() * 192), 32, 512),
                                                                      clamp(s.nnz_m / (sm_count() * 64), 64, 4096));
        CB_LAUNCH_CHECK();
        const TcCountPairs out = {m->cnt};
        CB_TRY(run_pairs(m, out, st));
        if (sym) {
            masked_mirror_kernel<<<flat_grid(s.nnz_m), 256, 0, st>>>(s.nnz_m, m->mate, m->cnt);
            CB_LAUNCH_CHECK();
        }
        CB_TRY(exclusive_scan_nonzero(m->cnt, m->place, s.nnz_m, st));
        masked_pos_kernel<<<flat_grid(nrows + 1), 256, 0, st>>>(nrows, mpos, m->place, cpos);
        CB_LAUNCH_CHECK();
        return 0;
    };
    if (build()) {
        masked_free(m, st);
        return 1;
    }
    *plan = m;
    return 0;
}

int masked_numeric(MaskedPlan *m, const double *aval, const double *bval, const int64_t *mcrd, int semi, int64_t *ccrd, double *cval,
                   cudaStream_t st)
{
    const bool any = semi == COMET_B200_ANY_PAIR;
    double *val = nullptr, *tval = nullptr;
    if (semi != COMET_B200_PLUS_PAIR && !any) {
        if (cudaMallocAsync((void **)&val, (size_t)(m->nnz_m + m->nnz_b) * 8, st) != cudaSuccess)
            return fail("spgemm numeric: device allocation failed");
        tval = val + m->nnz_m;             // B's values in column order
        masked_gather_kernel<<<flat_grid(m->nnz_b), 256, 0, st>>>(m->nnz_b, m->tidx, bval, tval);
        int rc = cudaMemsetAsync(&m->hdr->next_small, 0, 3 * sizeof(unsigned), st) == cudaSuccess ? 0 : fail("spgemm numeric: clearing the counters failed");
        if (!rc) rc = m->mate ? run_pairs(m, TcValuePairs<true>{m->cnt, m->mate, val, aval, tval, semi}, st)
                              : run_pairs(m, TcValuePairs<false>{m->cnt, nullptr, val, aval, tval, semi}, st);
        if (rc) {
            cudaFreeAsync(val, st);
            return rc;
        }
    }
    masked_compact_kernel<<<flat_grid(m->nnz_m), 256, 0, st>>>(m->nnz_m, mcrd, m->cnt, m->place, val, any, ccrd, cval);
    if (val) cudaFreeAsync(val, st);
    CB_LAUNCH_CHECK();
    return 0;
}

}  // namespace cb200
