// Intersections of pairs of sorted lists, one of each pair held as a set in shared memory and the other streamed past it
// (tc.cu: the masked count; masked.cu: the masked product).  The names are those of the masked count: pairs are
// the stored entries (i,k) of A, and the lists are row i of M and row k of B.
#pragma once
#include "common.cuh"
#include "semiring.cuh"

namespace cb200 {

static const int TC_WARP_MAX = 128;      // mask rows up to this length stay on the mask side, a warp per row
static const int TC_WARP_LOG2 = 9;       // log2 slots of their hash sets (both tables together)
static const int TC_WARPS = 8;           // warps per CTA in that kernel
static const int TC_MID_MAX = 512;       // sets up to this length are hash sets, a warp per unit
static const int TC_MID_LOG2 = 11;
static const int TC_MID_WARPS = 4;
static const int TC_CUCKOO_CHAIN = 48;   // longest eviction chain before the row falls back
static const int64_t TC_MAX_COLS = 1500000;   // columns of a bitmap: 183 KB, which leaves room for the set buffers
static const int TC_SET_BUF = 2048;      // sets up to this length are fetched while the one before is worked on
static const unsigned TC_UNIT_PROBES = 1u << 22;      // lists x set length a bitmap unit is cut to (64 lists at least)

struct TcUnit {           // a set and some of its lists
    int32_t row;          // mask side: row i of M; B side: row k of B
    uint32_t off;         // first list
    uint32_t count;       // lists; the top bit marks the B side
};
static const uint32_t TC_B_SIDE = 0x80000000u;

struct TcHeader {
    unsigned nsmall, nmid, nunits;         // short mask rows, hash-set units, bitmap units
    unsigned next_small, next_mid, next_unit;         // next one to hand out
    unsigned desc_all, desc_edge;          // positions where M's coordinates do not ascend: all, and those at row starts
    unsigned ordered;                      // A, B and M are the rest of a matrix in another order (order.cuh): rows in any order
};

struct TcShape {
    int64_t bcap;         // rows of B that can be sets
    bool cut;             // A and M are one matrix
    bool distinct;        // a coordinate that row i of A repeats is one pair (otherwise one per occurrence)
    bool half;            // A, M and B (rows of B as the pairs have them) are one symmetric pattern: of the pairs (i,k) and (k,i) the one
                          // whose set is the longer list is taken, and none goes to the B side
    bool ask;             // `cut` is off if TcHeader::ordered
};

__device__ __forceinline__ bool tc_left_out(const TcShape &sh, int64_t i, int64_t k, int64_t ml, int64_t bl)
{
    return sh.half && (bl > ml || (bl == ml && k > i));
}

// M repeats no coordinate: every place where its coordinates do not ascend is the start of a row
__device__ __forceinline__ bool tc_swap_ok(const TcHeader *hdr) { return hdr->desc_all == hdr->desc_edge; }

// The pair of entry number o of row i of A goes to the B side: B_k is the longer one.  What is compared is the part of
// M_i that would be streamed: when A and M are one matrix whose row i is cut at column k (`cut`: a strict lower
// triangle squared, where no column of B_k reaches k), that is its first o entries.
__device__ __forceinline__ bool tc_b_side(bool swap, int64_t ml, int64_t o, int64_t bl, int64_t k, const TcShape &sh, bool cut)
{
    return swap && bl > TC_WARP_MAX && bl > (cut ? o : ml) && k < sh.bcap;
}

// --- cuckoo set: tables T0 = tab[0, H) and T1 = tab[H, 2H), H = 2^(LOG2-1) -------------------------
template <int LOG2>
__device__ __forceinline__ unsigned tc_h0(int32_t j)
{
    return ((uint32_t)j * 0x9E3779B1u) >> (33 - LOG2);
}

template <int LOG2>
__device__ __forceinline__ unsigned tc_h1(int32_t j)
{
    return (1u << (LOG2 - 1)) + (((uint32_t)j * 0x85EBCA6Bu + 0x6D2B79F5u) >> (33 - LOG2));
}

// Returns false if the eviction chain did not end.
template <int LOG2>
__device__ __forceinline__ bool tc_cuckoo_insert(int32_t *tab, int32_t key)
{
    bool second = false;
    for (int it = 0; it < TC_CUCKOO_CHAIN; it++) {
        const unsigned pos = second ? tc_h1<LOG2>(key) : tc_h0<LOG2>(key);
        const int32_t old = atomicExch(&tab[pos], key);
        if (old == -1 || old == key) return true;
        key = old;                 // the evicted coordinate moves to its slot in the other table
        second = !second;
    }
    return false;
}

// --- fallback: linear probing over all 2^LOG2 slots -------------------------------------------
template <int LOG2>
__device__ __forceinline__ unsigned tc_slot(int32_t j)
{
    return ((uint32_t)j * 0x9E3779B1u) >> (32 - LOG2);
}

template <int LOG2>
__device__ __forceinline__ bool tc_linear_insert(int32_t *tab, int32_t j)     // true: it was there already
{
    unsigned h = tc_slot<LOG2>(j);
    for (int probe = 0; probe < (1 << LOG2); probe++) {
        int32_t old = atomicCAS(&tab[h], -1, j);
        if (old == -1 || old == j) return old == j;
        h = (h + 1) & ((1u << LOG2) - 1u);
    }
    return false;
}

template <int LOG2>
__device__ __forceinline__ unsigned tc_linear_probe(const int32_t *tab, int32_t j)
{
    unsigned h = tc_slot<LOG2>(j);
    for (int probe = 0; probe < (1 << LOG2); probe++) {
        int32_t k = tab[h];
        if (k == j) return 1u;
        if (k == -1) return 0u;
        h = (h + 1) & ((1u << LOG2) - 1u);
    }
    return 0u;
}

// Clears and fills the warp's set with crd[ms .. me).  Returns TC_CUCKOO, or TC_LINEAR when an insertion chain did
// not end; with `repeats` also TC_LINEAR for coordinates that do not ascend, and TC_REPEATS when one occurs twice.
enum { TC_CUCKOO = 0, TC_LINEAR = 1, TC_REPEATS = 3 };

template <int LOG2>
__device__ __forceinline__ unsigned tc_fill(int32_t *tab, const int32_t *__restrict__ crd, int64_t ms, int64_t me, int lane,
                                            bool repeats)
{
    auto clear = [&]() {
#pragma unroll 4
        for (int s = lane; s < (1 << LOG2) / 4; s += 32) ((int4 *)tab)[s] = make_int4(-1, -1, -1, -1);
        __syncwarp();
    };
    clear();
    bool ok = true;
    for (int64_t t = ms + lane; t < me; t += 32) {
        const int32_t key = crd[t];
        if (repeats && t > ms && crd[t - 1] >= key) ok = false;
        ok = tc_cuckoo_insert<LOG2>(tab, key) && ok;
    }
    __syncwarp();                          // the other lanes' columns: a vote orders no memory
    if (__all_sync(0xffffffffu, ok)) return TC_CUCKOO;
    clear();
    bool twice = false;
    for (int64_t t = ms + lane; t < me; t += 32) twice |= tc_linear_insert<LOG2>(tab, crd[t]);
    __syncwarp();
    return __any_sync(0xffffffffu, twice) && repeats ? TC_REPEATS : TC_LINEAR;
}

// Row starts of M where the coordinates do not ascend, and the row of every entry of A: 16 lanes per row.
static __global__ void __launch_bounds__(256)
tc_rows_kernel(int64_t row_lo, int64_t row_hi, const int64_t *__restrict__ apos, const int64_t *__restrict__ mpos,
               const int64_t *__restrict__ mcrd, int32_t *__restrict__ arow, TcHeader *hdr)
{
    const int l = threadIdx.x & 15;
    const int64_t first = mpos[row_lo];
    const bool check = l == 0 && !hdr->ordered;
    unsigned desc = 0;
    const int64_t ng = ((int64_t)gridDim.x * blockDim.x) >> 4;
    for (int64_t r = row_lo + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4); r < row_hi; r += ng) {
        const int64_t e = apos[r + 1];
        for (int64_t p = apos[r] + l; p < e; p += 16) arow[p] = (int32_t)r;
        if (check) {
            const int64_t s = mpos[r];
            if (s > first && mpos[r + 1] > s && mcrd[s] <= mcrd[s - 1]) desc++;
        }
    }
    if (desc) atomicAdd(&hdr->desc_edge, desc);
}

// Pairs of the B side counted per row of B; slot[p] = the pair's place in its row's list (-1: mask side).
static __global__ void __launch_bounds__(256)
tc_route_kernel(int64_t row_lo, int64_t row_hi, const int64_t *__restrict__ apos, const int32_t *__restrict__ acrd,
                const int32_t *__restrict__ arow, const int64_t *__restrict__ bpos, const int64_t *__restrict__ mpos,
                TcShape sh, const TcHeader *hdr, int32_t *__restrict__ slot, int32_t *__restrict__ bcount)
{
    const bool swap = tc_swap_ok(hdr);
    const bool cut = sh.cut && !(sh.ask && hdr->ordered);
    const int64_t end = apos[row_hi];
    for (int64_t p = apos[row_lo] + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < end;
         p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = arow[p], k = acrd[p];
        const int64_t ml = mpos[i + 1] - mpos[i], bl = bpos[k + 1] - bpos[k];
        int32_t at = -1;
        const bool again = sh.distinct && p > apos[i] && acrd[p - 1] == k;
        if (ml > 0 && !again && tc_b_side(swap, ml, p - apos[i], bl, k, sh, cut)) at = atomicAdd(bcount + k, 1);
        slot[p] = at;
    }
}

static __global__ void __launch_bounds__(256)
tc_scatter_kernel(int64_t row_lo, int64_t row_hi, const int64_t *__restrict__ apos, const int32_t *__restrict__ acrd,
                  const int32_t *__restrict__ arow, const int32_t *__restrict__ slot,
                  const int64_t *__restrict__ bptr, int2 *__restrict__ blist)
{
    const int64_t end = apos[row_hi];
    for (int64_t p = apos[row_lo] + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < end;
         p += (int64_t)gridDim.x * blockDim.x) {
        const int32_t at = slot[p];
        if (at >= 0) blist[bptr[acrd[p]] + at] = make_int2(arow[p], (int)(p - apos[arow[p]]));
    }
}

// The rows of the warp kernel and the units of the bitmap kernel.  Thread t looks at row row_lo + t of the mask side
// and at row t of the B side.
static __global__ void __launch_bounds__(256)
tc_units_kernel(int64_t row_lo, int64_t row_hi, int64_t bcap, const int64_t *__restrict__ apos,
                const int64_t *__restrict__ mpos, const int64_t *__restrict__ bpos, const int64_t *__restrict__ bptr,
                TcHeader *hdr, int32_t *__restrict__ small, TcUnit *__restrict__ mids, TcUnit *__restrict__ units,
                unsigned mid_lists, unsigned unit_lists)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    auto cut = [&](int64_t row, int64_t lists, int64_t set, uint32_t side) {
        const bool mid = set <= TC_MID_MAX;
        unsigned per = mid ? mid_lists : TC_UNIT_PROBES / (unsigned)(set < (int64_t)TC_UNIT_PROBES ? set : (int64_t)TC_UNIT_PROBES);
        if (!mid) per = per > unit_lists ? unit_lists : (per < 64 ? 64 : per);
        const unsigned n = (unsigned)((lists + per - 1) / per);
        const unsigned at = atomicAdd(mid ? &hdr->nmid : &hdr->nunits, n);
        for (unsigned u = 0; u < n; u++) {
            TcUnit v;
            v.row = (int32_t)row;
            v.off = u * per;
            const int64_t left = lists - (int64_t)v.off;
            v.count = (unsigned)(left < (int64_t)per ? left : (int64_t)per) | side;
            (mid ? mids : units)[at + u] = v;
        }
    };
    const int64_t r = row_lo + t;
    int64_t al = 0, ml = 0;
    if (r < row_hi) {
        al = apos[r + 1] - apos[r];
        ml = mpos[r + 1] - mpos[r];
    }
    const bool is_small = al > 0 && ml > 0 && ml <= TC_WARP_MAX;
    const unsigned m = __ballot_sync(0xffffffffu, is_small);
    if (m) {
        unsigned base = 0;
        const int leader = __ffs(m) - 1;
        if (lane == leader) base = atomicAdd(&hdr->nsmall, (unsigned)__popc(m));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (is_small) small[base + __popc(m & ((1u << lane) - 1u))] = (int32_t)r;
    }
    if (al > 0 && ml > TC_WARP_MAX) cut(r, al, ml, 0u);
    if (t < bcap) {
        const int64_t lists = bptr[t + 1] - bptr[t];
        if (lists > 0) cut(t, lists, bpos[t + 1] - bpos[t], TC_B_SIDE);
    }
}

// ---------------------------------------------------------------------------
// Streaming: lane l of the warp holds a list, crd[s .. s + len) (len 0: none).  probe(j) is 1 for a column in the set;
// `dead` is a column that is not.  The lists are walked one after another in groups of 32 elements, the last group of a
// list partly idle, with eight groups in flight whether they belong to one list or to several: a list is only a few
// hundred elements long, so waiting for the first load of each would leave the warp idle most of the time.
// Consecutive lanes hold consecutive elements: an ascending list's neighbours share bitmap words, which costs 3.2
// shared-memory cycles per 32 probes on R-MAT scale 20 where lanes four elements apart (128-bit loads) cost 5.5.
// ---------------------------------------------------------------------------
template <typename P>
__device__ __forceinline__ unsigned tc_stream(const int32_t *__restrict__ crd, int64_t s, int len, int lane, int32_t dead,
                                              P probe)
{
    unsigned hits = 0;
    unsigned left = __ballot_sync(0xffffffffu, len > 0);
    const int32_t *q = crd;
    int rem = 0;
    while (left || rem > 0) {
        int32_t j[8];
        if (rem >= 256) {
#pragma unroll
            for (int i = 0; i < 8; i++) j[i] = __ldg(q + i * 32);
            q += 256;
            rem -= 256;
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                if (rem <= 0 && left) {
                    const int t = __ffs(left) - 1;
                    left &= left - 1;
                    q = crd + __shfl_sync(0xffffffffu, (long long)s, t) + lane;
                    rem = __shfl_sync(0xffffffffu, len, t);
                }
                j[i] = dead;
                if (lane < rem) j[i] = __ldg(q);
                q += 32;
                rem -= 32;
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++) hits += probe(j[i]);
    }
    return hits;
}

// The same with the hits of each list kept apart: lane l returns those of its own list.
template <typename P>
__device__ __forceinline__ unsigned tc_stream_each(const int32_t *__restrict__ crd, int64_t s, int len, int lane,
                                                   int32_t dead, P probe)
{
    unsigned own = 0;
    unsigned left = __ballot_sync(0xffffffffu, len > 0);
    const int32_t *q = crd;
    int rem = 0, t = 0;
    while (left || rem > 0) {
        int32_t j[8];
        int of[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            if (rem <= 0 && left) {
                t = __ffs(left) - 1;
                left &= left - 1;
                q = crd + __shfl_sync(0xffffffffu, (long long)s, t) + lane;
                rem = __shfl_sync(0xffffffffu, len, t);
            }
            of[i] = t;
            j[i] = dead;
            if (lane < rem) j[i] = __ldg(q);
            q += 32;
            rem -= 32;
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const unsigned hit = __ballot_sync(0xffffffffu, probe(j[i]) != 0u);
            if (lane == of[i]) own += __popc(hit);
        }
    }
    return own;
}

__device__ __forceinline__ void tc_add_count(unsigned long long hits, unsigned long long *s_part, int nwarps,
                                             unsigned long long *count)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) hits += __shfl_xor_sync(0xffffffffu, hits, o);
    if (lane == 0) s_part[threadIdx.x >> 5] = hits;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int i = 0; i < nwarps; i++) t += s_part[i];
        if (t) atomicAdd(count, t);
    }
}

// ---------------------------------------------------------------------------
// What becomes of the hits.  stream() is called by a warp with a list per lane; p is the list's pair (entry of A), set_at
// the set's first entry.
// ---------------------------------------------------------------------------
struct TcCountAll {                        // one total
    static const bool PAIRS = false, VALUES = false;
    unsigned long long *count;
    unsigned long long hits;
    __device__ bool wanted(int64_t) const { return true; }
    template <typename P, typename W>
    __device__ void stream(const int32_t *crd, int64_t s, int len, int lane, int32_t dead, P probe, W, int64_t, bool, int64_t)
    {
        hits += tc_stream(crd, s, len, lane, dead, probe);
    }
    __device__ void finish(unsigned long long *s_part, int nwarps) { tc_add_count(hits, s_part, nwarps, count); }
};

struct TcCountPairs {                      // cnt[p], cleared before
    static const bool PAIRS = true, VALUES = false;
    int32_t *cnt;
    __device__ bool wanted(int64_t) const { return true; }
    template <typename P, typename W>
    __device__ void stream(const int32_t *crd, int64_t s, int len, int lane, int32_t dead, P probe, W, int64_t p, bool, int64_t)
    {
        const unsigned own = tc_stream_each(crd, s, len, lane, dead, probe);
        if (own) cnt[p] = (int32_t)own;
    }
    __device__ void finish(unsigned long long *, int) {}
};

// val[p] for the pairs with hits: the products of equal positions, folded.  BOTH: a pair taken for two (TcShape::half): val[mate[p]] too,
// from the values of A along the list and of B along the set.
template <bool BOTH>
struct TcValuePairs {
    static const bool PAIRS = true, VALUES = true;
    const int32_t *cnt, *mate;
    double *val;
    const double *aval, *bval;             // values of the rows of A (the lists "M_i") and of the transposed B ("B_k")
    int semi;
    __device__ bool wanted(int64_t p) const { return cnt[p] != 0; }
    // as tc_stream_each; where(j) is the place of a column in the set.  The lanes' parts of a list are added up when the walk
    // goes on to the next list.
    template <typename P, typename W>
    __device__ void stream(const int32_t *crd, int64_t s, int len, int lane, int32_t dead, P probe, W where, int64_t p, bool bside,
                           int64_t set_at)
    {
        const double *sval = (bside ? bval : aval) + set_at, *lval = bside ? aval : bval;
        double own = 0.0, part = sr_identity(semi), own2 = 0.0, part2 = part;
        unsigned left = __ballot_sync(0xffffffffu, len > 0);
        int64_t at = 0;
        int rem = 0, t = -1, cur = -1;
        auto flush = [&]() {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                part = sr_fold_value(semi, part, __shfl_xor_sync(0xffffffffu, part, o));
                if (BOTH) part2 = sr_fold_value(semi, part2, __shfl_xor_sync(0xffffffffu, part2, o));
            }
            if (lane == cur) { own = part; own2 = part2; }
            part = part2 = sr_identity(semi);
        };
        while (left || rem > 0) {
            int32_t j[4];
            int64_t from[4];
            int of[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (rem <= 0 && left) {
                    t = __ffs(left) - 1;
                    left &= left - 1;
                    at = __shfl_sync(0xffffffffu, (long long)s, t) + lane;
                    rem = __shfl_sync(0xffffffffu, len, t);
                }
                of[i] = t;
                from[i] = at;
                j[i] = dead;
                if (lane < rem) j[i] = __ldg(crd + at);
                at += 32;
                rem -= 32;
            }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if (of[i] != cur) {
                    if (cur >= 0) flush();
                    cur = of[i];
                }
                if (probe(j[i])) {
                    const int at_set = where(j[i]);
                    const double sv = __ldg(sval + at_set), lv = __ldg(lval + from[i]);
                    part = sr_fold_value(semi, part, bside ? sr_combine(semi, lv, sv) : sr_combine(semi, sv, lv));
                    if (BOTH)
                        part2 = sr_fold_value(semi, part2, sr_combine(semi, __ldg(aval + from[i]), __ldg(bval + set_at + at_set)));
                }
            }
        }
        if (cur >= 0) flush();
        if (len > 0) {
            val[p] = own;
            if (BOTH) val[mate[p]] = own2;
        }
    }
    __device__ void finish(unsigned long long *, int) {}
};

// place of j in an ascending set that holds it
__device__ __forceinline__ int tc_search(const int32_t *set, int len, int32_t j)
{
    int lo = 0, hi = len;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (set[mid] < j) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// probe function of a warp's hash set handed to stream()
template <int LOG2, class Out>
__device__ __forceinline__ void tc_stream_set(Out &out, const int32_t *tab, const unsigned short *place, unsigned how,
                                              const int32_t *__restrict__ crd, int64_t s, int len, int lane,
                                              const int32_t *__restrict__ set, int64_t p, bool bside, int64_t set_at, int set_len)
{
    if (how == TC_CUCKOO) {
        out.stream(crd, s, len, lane, -2, [&](int32_t j) {
            return (unsigned)(tab[tc_h0<LOG2>(j)] == j) | (unsigned)(tab[tc_h1<LOG2>(j)] == j);
        }, [&](int32_t j) { return place[tab[tc_h0<LOG2>(j)] == j ? tc_h0<LOG2>(j) : tc_h1<LOG2>(j)]; }, p, bside, set_at);
        return;
    }
    out.stream(crd, s, len, lane, -2, [&](int32_t j) {
        unsigned c = tc_linear_probe<LOG2>(tab, j);
        if (how == TC_REPEATS && c) {       // a hit counts as often as the set's row stores it
            c = 0;
            for (int t = 0; t < set_len; t++) c += set[t] == j ? 1u : 0u;
        }
        return c;
    }, [&](int32_t j) { return tc_search(set, set_len, j); }, p, bside, set_at);
}

// where in the set every slot's coordinate comes from (after tc_fill returned TC_CUCKOO)
template <int LOG2>
__device__ __forceinline__ void tc_fill_places(const int32_t *tab, unsigned short *place, const int32_t *__restrict__ crd,
                                               int64_t s, int64_t e, int lane)
{
    for (int64_t t = s + lane; t < e; t += 32) {
        const int32_t j = crd[t];
        place[tab[tc_h0<LOG2>(j)] == j ? tc_h0<LOG2>(j) : tc_h1<LOG2>(j)] = (unsigned short)(t - s);
    }
    __syncwarp();
}

// Mask rows of at most TC_WARP_MAX entries: a warp per row, its set built when the first list turns up.
template <class Out>
__global__ void __launch_bounds__(TC_WARPS * 32)
tc_warp_kernel(TcHeader *hdr, const int32_t *__restrict__ small, const int64_t *__restrict__ apos,
               const int32_t *__restrict__ acrd, const int64_t *__restrict__ bpos,
               const int32_t *__restrict__ bcrd, const int64_t *__restrict__ mpos,
               const int32_t *__restrict__ mcrd, TcShape sh, Out out)
{
    __shared__ __align__(16) int32_t s_tab[TC_WARPS][1 << TC_WARP_LOG2];
    __shared__ unsigned short s_place[Out::VALUES ? TC_WARPS : 1][Out::VALUES ? 1 << TC_WARP_LOG2 : 1];
    __shared__ unsigned long long s_part[TC_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool swap = tc_swap_ok(hdr);
    const bool cut = sh.cut && !(sh.ask && hdr->ordered);
    const unsigned n = hdr->nsmall;
    // Four rows a draw keep the counter from being a queue; fewer than all warps would draw go one by one, or most warps have none (a symmetric
    // graph of 1934 vertices and 70,000 entries, plus-times 790 -> 456 us; R-MAT scale 13 x 16, plus-pair 330 -> 280).
    const unsigned step = n >= gridDim.x * TC_WARPS * 4 ? 4u : 1u;
    while (true) {
        unsigned idx = 0;
        if (lane == 0) idx = atomicAdd(&hdr->next_small, step);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= n) break;
        const unsigned stop = idx + step < n ? idx + step : n;
        for (; idx < stop; idx++) {
            const int64_t i = small[idx];
            const int64_t as = apos[i], ae = apos[i + 1], ms = mpos[i], me = mpos[i + 1];
            bool filled = false;
            unsigned how = TC_CUCKOO;
            for (int64_t p0 = as; p0 < ae; p0 += 32) {
                int64_t s = 0;
                int len = 0;
                if (p0 + lane < ae) {
                    const int64_t k = acrd[p0 + lane];
                    s = bpos[k];
                    const int64_t bl = bpos[k + 1] - s;
                    const bool again = sh.distinct && p0 + lane > as && acrd[p0 + lane - 1] == k;
                    if (!again && out.wanted(p0 + lane) && !(Out::PAIRS && tc_left_out(sh, i, k, me - ms, bl)) &&
                        !tc_b_side(swap, me - ms, p0 + lane - as, bl, k, sh, cut))
                        len = (int)bl;
                }
                if (!__any_sync(0xffffffffu, len > 0)) continue;
                if (!filled) {
                    how = tc_fill<TC_WARP_LOG2>(s_tab[w], mcrd, ms, me, lane, false);
                    if (Out::VALUES && how == TC_CUCKOO) tc_fill_places<TC_WARP_LOG2>(s_tab[w], s_place[w], mcrd, ms, me, lane);
                }
                filled = true;
                tc_stream_set<TC_WARP_LOG2>(out, s_tab[w], s_place[Out::VALUES ? w : 0], how, bcrd, s, len, lane, mcrd + ms,
                                            p0 + lane, false, ms, (int)(me - ms));
            }
            __syncwarp();
        }
    }
    out.finish(s_part, TC_WARPS);
}

// A unit's next lists: lane l < n gets list number b + l of the unit (mask side: length 0 if it belongs to the B side).
// `first` is the unit's first entry of A's row (mask side) or first place in blist.  On the B side a list ends, at the
// latest, where the entry of M_i at the pair's own place o in row i already lies behind the set's last column.
template <class Out>
__device__ __forceinline__ void tc_unit_lists(const Out &out, int64_t row, bool bside, int64_t first, int64_t off, int b, int n, int lists,
                                              int lane, bool swap, bool cut, int64_t ml, int32_t last, const TcShape &sh,
                                              const int64_t *__restrict__ apos, const int32_t *__restrict__ acrd,
                                              const int64_t *__restrict__ bpos, const int64_t *__restrict__ mpos,
                                              const int32_t *__restrict__ mcrd, const int2 *__restrict__ blist, int64_t &s,
                                              int &len, int64_t &p)
{
    s = 0;
    len = 0;
    p = 0;
    if (lane >= n || b + lane >= lists) return;
    if (bside) {
        const int2 io = __ldg(blist + first + b + lane);
        if (Out::PAIRS) {
            p = __ldg(apos + io.x) + io.y;
            if (!out.wanted(p)) return;
        }
        s = __ldg(mpos + io.x);
        len = (int)(__ldg(mpos + io.x + 1) - s);
        if (cut && io.y < len && __ldg(mcrd + s + io.y) > last) len = io.y;
    } else {
        p = first + b + lane;
        const int64_t k = __ldg(acrd + p);
        if (!out.wanted(p) || (sh.distinct && off + b + lane > 0 && __ldg(acrd + p - 1) == k)) return;
        s = __ldg(bpos + k);
        const int64_t bl = __ldg(bpos + k + 1) - s;
        len = (Out::PAIRS && tc_left_out(sh, row, k, ml, bl)) || tc_b_side(swap, ml, off + b + lane, bl, k, sh, cut) ? 0 : (int)bl;
    }
}

// Units whose set has at most TC_MID_MAX entries: a warp per unit, the set as a hash set.
template <class Out>
__global__ void __launch_bounds__(TC_MID_WARPS * 32)
tc_mid_kernel(TcHeader *hdr, const TcUnit *__restrict__ mids, const int64_t *__restrict__ apos,
              const int32_t *__restrict__ acrd, const int64_t *__restrict__ bpos, const int32_t *__restrict__ bcrd,
              const int64_t *__restrict__ mpos, const int32_t *__restrict__ mcrd, const int64_t *__restrict__ bptr,
              const int2 *__restrict__ blist, TcShape sh, Out out)
{
    __shared__ __align__(16) int32_t s_tab[TC_MID_WARPS][1 << TC_MID_LOG2];
    __shared__ unsigned short s_place[Out::VALUES ? TC_MID_WARPS : 1][Out::VALUES ? 1 << TC_MID_LOG2 : 1];
    __shared__ unsigned long long s_part[TC_MID_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool swap = tc_swap_ok(hdr);
    const bool cut = sh.cut && !(sh.ask && hdr->ordered);
    const unsigned n = hdr->nmid;
    while (true) {
        unsigned idx = 0;
        if (lane == 0) idx = atomicAdd(&hdr->next_mid, 1u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= n) break;
        const TcUnit u = mids[idx];
        const bool bside = (u.count & TC_B_SIDE) != 0;
        const int lists = (int)(u.count & ~TC_B_SIDE);
        const int32_t *scrd = bside ? bcrd : mcrd, *lcrd = bside ? mcrd : bcrd;
        const int64_t *spos = bside ? bpos : mpos;
        const int64_t ss = spos[u.row], se = spos[u.row + 1];
        const int64_t row_at = (bside ? bptr : apos)[u.row] + u.off;
        int32_t last = -1;
        for (int64_t t = ss + lane; t < se; t += 32) last = max(last, scrd[t]);
        last = __reduce_max_sync(0xffffffffu, last);
        const unsigned how = tc_fill<TC_MID_LOG2>(s_tab[w], scrd, ss, se, lane, bside);
        if (Out::VALUES && how == TC_CUCKOO) tc_fill_places<TC_MID_LOG2>(s_tab[w], s_place[w], scrd, ss, se, lane);
        __syncwarp();
        for (int b = 0; b < lists; b += 32) {
            int64_t s;
            int len;
            int64_t p;
            tc_unit_lists(out, u.row, bside, row_at, u.off, b, 32, lists, lane, swap, cut, se - ss, last, sh, apos, acrd, bpos, mpos, mcrd,
                          blist, s, len, p);
            tc_stream_set<TC_MID_LOG2>(out, s_tab[w], s_place[Out::VALUES ? w : 0], how, lcrd, s, len, lane, scrd + ss, p, bside,
                                       ss, (int)(se - ss));
        }
        __syncwarp();
    }
    out.finish(s_part, TC_MID_WARPS);
}

// Units: a bitmap of the set, its lists drawn by the warps in batches of 32.  SEGMENTED: the columns do not fit one
// bitmap, the unit is repeated per segment of `width` columns.  The next unit's set is fetched into shared memory by
// warp 0 while the others stream, so that between two units only the bits change.
// 32 warps an SM, as many as are launched: 64 registers a thread, which no variant spills for.  With the 109 that the value pass for both
// halves takes otherwise, one CTA of 16 warps ran (R-MAT scale 15 / 16, 16 per row, symmetric, under itself, plus-times 1450 -> 1235 and
// 3000 -> 2300 us); the one-sided pass spilled 112 bytes (not symmetric, 15 / 16, 1000 -> 985 and 1715 -> 1695).  Three CTAs of 16 warps for
// counts cost 96 bytes of spills and gain nothing (plus-pair at scale 15 373 and 373 us).
template <int THREADS, bool SEGMENTED, class Out>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS)
tc_bitmap_kernel(TcHeader *hdr, const TcUnit *__restrict__ units, const int64_t *__restrict__ apos,
                 const int32_t *__restrict__ acrd, const int64_t *__restrict__ bpos, const int32_t *__restrict__ bcrd,
                 const int64_t *__restrict__ mpos, const int32_t *__restrict__ mcrd, const int64_t *__restrict__ bptr,
                 const int2 *__restrict__ blist, TcShape sh, int width, const int64_t *ncols_dev,
                 bool with_prefix, Out out)
{
    extern __shared__ __align__(16) int32_t s_tc[];
    __shared__ unsigned long long s_part[THREADS / 32];
    __shared__ TcUnit s_unit[2];
    __shared__ int64_t s_at[2];            // first entry of the unit's set
    __shared__ int s_len[2];               // its length
    __shared__ unsigned s_batch, s_dup;
    __shared__ int32_t s_last;             // largest column of the set
    int32_t *buf = s_tc;                   // two set buffers of TC_SET_BUF
    uint32_t *bm = (uint32_t *)(s_tc + 2 * TC_SET_BUF);
    const int words = (width >> 5) + 1;    // covers bit `width`, which stands for "no such column"
    uint32_t *pre = Out::VALUES && with_prefix ? bm + words : nullptr;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool swap = tc_swap_ok(hdr);
    const bool cut = sh.cut && !(sh.ask && hdr->ordered);
    const unsigned nunits = hdr->nunits;
    for (int t = threadIdx.x; t < words; t += THREADS) bm[t] = 0;

    auto fetch = [&](int to) {             // warp 0: the next unit and its set
        unsigned idx = 0;
        if (lane == 0) idx = atomicAdd(&hdr->next_unit, 1u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= nunits) {
            if (lane == 0) s_unit[to].row = -1;
            return;
        }
        const TcUnit u = units[idx];
        const bool bside = (u.count & TC_B_SIDE) != 0;
        const int64_t *pos = bside ? bpos : mpos;
        const int32_t *crd = bside ? bcrd : mcrd;
        const int64_t s = pos[u.row];
        const int len = (int)(pos[u.row + 1] - s);
        if (lane == 0) {
            s_unit[to] = u;
            s_at[to] = s;
            s_len[to] = len;
        }
        if (len <= TC_SET_BUF)
#pragma unroll 4
            for (int t = lane; t < len; t += 32) buf[to * TC_SET_BUF + t] = __ldg(crd + s + t);
    };
    if (w == 0) fetch(0);
    if (threadIdx.x == 0) { s_batch = 0; s_dup = 0; s_last = -1; }
    __syncthreads();
    for (int cur = 0;; cur ^= 1) {
        const TcUnit u = s_unit[cur];
        if (u.row < 0) break;
        const bool bside = (u.count & TC_B_SIDE) != 0;
        const int lists = (int)(u.count & ~TC_B_SIDE);
        const int len = s_len[cur];
        const int32_t *set = len <= TC_SET_BUF ? buf + cur * TC_SET_BUF : (bside ? bcrd : mcrd) + s_at[cur];
        const int32_t *lcrd = bside ? mcrd : bcrd;
        const int64_t row_at = bside ? bptr[u.row] + u.off : apos[u.row] + u.off;
        const int64_t ml = len;            // mask side: the length of the mask row
        const int64_t ncols = SEGMENTED ? *ncols_dev : 0;
        for (int64_t base = 0;; base += width) {
            int32_t top = -1;
            for (int t = threadIdx.x; t < len; t += THREADS) {
                const int64_t j = (int64_t)set[t] - base;
                if (SEGMENTED && (j < 0 || j >= width || set[t] >= ncols)) continue;
                const uint32_t bit = 1u << (j & 31);
                if (atomicOr(&bm[j >> 5], bit) & bit) s_dup = 1;
                top = max(top, set[t]);
            }
            top = __reduce_max_sync(0xffffffffu, top);
            if (lane == 0) atomicMax(&s_last, top);
            __syncthreads();
            if (Out::VALUES && pre) {
                // pre[w] = set columns before word w: a thread sums a run of words, the CTA scans the sums
                const int per = (words + THREADS - 1) / THREADS, w0 = min((int)threadIdx.x * per, words), w1 = min(w0 + per, words);
                unsigned sum = 0;
                for (int t = w0; t < w1; t++) sum += __popc(bm[t]);
                unsigned incl = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                if (lane == 31) s_part[w] = incl;
                __syncthreads();
                unsigned run = incl - sum;
                for (int t = 0; t < w; t++) run += (unsigned)s_part[t];
                for (int t = w0; t < w1; t++) {
                    pre[t] = run;
                    run += __popc(bm[t]);
                }
                __syncthreads();
            }
            const bool dup = bside && s_dup;
            if (w == 0 && base == 0) fetch(cur ^ 1);
            while (true) {
                // lists in ever smaller draws (a share of what is left), so that the warps end together
                unsigned b = 0;
                int step = 0;
                if (lane == 0) {
                    step = min(32, max(1, (lists - (int)*(volatile unsigned *)&s_batch) / (THREADS / 16)));
                    b = atomicAdd(&s_batch, (unsigned)step);
                }
                b = __shfl_sync(0xffffffffu, b, 0);
                step = __shfl_sync(0xffffffffu, step, 0);
                if ((int)b >= lists) break;
                int64_t s, p;
                int n;
                tc_unit_lists(out, u.row, bside, row_at, u.off, (int)b, step, lists, lane, swap, cut, ml, bside ? s_last : 0, sh, apos, acrd,
                              bpos, mpos, mcrd, blist, s, n, p);
                auto where = [&](int32_t x) {
                    if (!Out::VALUES || !pre) return tc_search(set, len, x);
                    const unsigned bits = bm[x >> 5] & ((1u << (x & 31)) - 1u);
                    return (int)pre[x >> 5] + __popc(bits);
                };
                auto bit_of = [&](int32_t x) { return (bm[x >> 5] >> (x & 31)) & 1u; };
                if (SEGMENTED && ncols > width) {
                    out.stream(lcrd, s, n, lane, INT32_MAX, [&](int32_t j) {
                        const int64_t x = (int64_t)j - base;
                        unsigned c = x < 0 || x >= width ? 0u : bit_of((int32_t)x);
                        if (c && dup) {
                            c = 0;
                            for (int t = 0; t < len; t++) c += set[t] == j ? 1u : 0u;
                        }
                        return c;
                    }, where, p, bside, s_at[cur]);
                    continue;
                }
                if (!dup)
                    out.stream(lcrd, s, n, lane, width, bit_of, where, p, bside, s_at[cur]);
                else                       // B_k repeats a coordinate: a hit counts as often as it is stored
                    out.stream(lcrd, s, n, lane, width, [&](int32_t j) {
                        unsigned c = 0;
                        if (bit_of(j)) for (int t = 0; t < len; t++) c += set[t] == j ? 1u : 0u;
                        return c;
                    }, where, p, bside, s_at[cur]);
            }
            __syncthreads();
            for (int t = threadIdx.x; t < len; t += THREADS) {
                const int64_t j = (int64_t)set[t] - base;
                if (SEGMENTED && (j < 0 || j >= width)) continue;
                bm[j >> 5] = 0;
            }
            if (threadIdx.x == 0) { s_batch = 0; s_dup = 0; s_last = -1; }
            __syncthreads();
            if (!SEGMENTED || base + width >= ncols) break;
        }
    }
    out.finish(s_part, THREADS / 32);
}

template <int THREADS, bool SEGMENTED, class Out>
static int launch_bitmap(size_t smem, TcHeader *hdr, const TcUnit *units, const int64_t *apos,
                         const int32_t *acrd, const int64_t *bpos, const int32_t *bcrd, const int64_t *mpos,
                         const int32_t *mcrd, const int64_t *bptr, const int2 *blist, TcShape sh, int width,
                         const int64_t *ncols_dev, const Out &out, cudaStream_t st)
{
    auto k = tc_bitmap_kernel<THREADS, SEGMENTED, Out>;
    // places in the set come from prefix counts beside the bitmap where both fit, else from a search
    const size_t both = smem + (size_t)((width >> 5) + 1) * 4;
    const bool with_prefix = Out::VALUES && both <= (size_t)210 * 1024;
    if (with_prefix) smem = both;
    CB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<(unsigned)(sm_count() * (1024 / THREADS)), THREADS, smem, st>>>(hdr, units, apos, acrd, bpos, bcrd, mpos, mcrd, bptr, blist,
                                                             sh, width, ncols_dev, with_prefix, out);
    CB_LAUNCH_CHECK();
    return 0;
}

}  // namespace cb200
