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
// Measured on B200, R-MAT edge factor 16 lower triangles (mask side only, cuckoo sets in every bin -> this):
// scale 14 0.27 -> 0.16 ms, scale 18 1.96 -> 0.76, scale 20 10.2 -> 3.15, scale 22 61.9 -> 18.3.  At scale 22 the bitmap kernel takes 12.0 of
// it (shared-memory pipe and issue slots both near 70 %: 6.7 wavefronts and 25 instructions per 32 probes), the hash
// sets 3.6, routing and scattering the pairs 1.4, narrowing and renumbering 1.1.
#include "common.cuh"

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
};

struct TcShape {
    int64_t bcap;         // rows of B that can be sets
    bool cut;             // A and M are one matrix
};

// M repeats no coordinate: every place where its coordinates do not ascend is the start of a row
__device__ __forceinline__ bool tc_swap_ok(const TcHeader *hdr) { return hdr->desc_all == hdr->desc_edge; }

// The pair of entry number o of row i of A goes to the B side: B_k is the longer one.  What is compared is the part of
// M_i that would be streamed: when A and M are one matrix whose row i is cut at column k (`cut`: a strict lower
// triangle squared, where no column of B_k reaches k), that is its first o entries.
__device__ __forceinline__ bool tc_b_side(bool swap, int64_t ml, int64_t o, int64_t bl, int64_t k, const TcShape &sh)
{
    return swap && bl > TC_WARP_MAX && bl > (sh.cut ? o : ml) && k < sh.bcap;
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
    if (__all_sync(0xffffffffu, ok)) return TC_CUCKOO;
    clear();
    bool twice = false;
    for (int64_t t = ms + lane; t < me; t += 32) twice |= tc_linear_insert<LOG2>(tab, crd[t]);
    return __any_sync(0xffffffffu, twice) && repeats ? TC_REPEATS : TC_LINEAR;
}

// ---------------------------------------------------------------------------
// Preparation
// ---------------------------------------------------------------------------

// present[j] = column j is stored in M (a bit each).  Most entries name a few hub columns, whose words would be a queue
// for the whole chip (0.9 ms on 64 M entries with a test before the atomic, 1.9 ms with plain byte stores), so a
// CTA remembers the columns it met last.  The table is read and written without order: a lost entry only repeats a test.
static const int TC_SEEN_SLOTS = 8192;

__global__ void __launch_bounds__(512)
tc_present_kernel(int64_t n, const int64_t *__restrict__ mcrd, uint32_t *__restrict__ present)
{
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
                 const int64_t *__restrict__ pos, int64_t row_lo, int64_t row_hi, TcHeader *hdr)
{
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

// Row starts of M where the coordinates do not ascend, and the row of every entry of A: 16 lanes per row.
__global__ void __launch_bounds__(256)
tc_rows_kernel(int64_t row_lo, int64_t row_hi, const int64_t *__restrict__ apos, const int64_t *__restrict__ mpos,
               const int64_t *__restrict__ mcrd, int32_t *__restrict__ arow, TcHeader *hdr)
{
    const int l = threadIdx.x & 15;
    const int64_t first = mpos[row_lo];
    unsigned desc = 0;
    const int64_t ng = ((int64_t)gridDim.x * blockDim.x) >> 4;
    for (int64_t r = row_lo + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4); r < row_hi; r += ng) {
        const int64_t e = apos[r + 1];
        for (int64_t p = apos[r] + l; p < e; p += 16) arow[p] = (int32_t)r;
        if (l == 0) {
            const int64_t s = mpos[r];
            if (s > first && mpos[r + 1] > s && mcrd[s] <= mcrd[s - 1]) desc++;
        }
    }
    if (desc) atomicAdd(&hdr->desc_edge, desc);
}

// Pairs of the B side counted per row of B; slot[p] = the pair's place in its row's list (-1: mask side).
__global__ void __launch_bounds__(256)
tc_route_kernel(int64_t row_lo, int64_t row_hi, const int64_t *__restrict__ apos, const int32_t *__restrict__ acrd,
                const int32_t *__restrict__ arow, const int64_t *__restrict__ bpos, const int64_t *__restrict__ mpos,
                TcShape sh, const TcHeader *hdr, int32_t *__restrict__ slot, int32_t *__restrict__ bcount)
{
    const bool swap = tc_swap_ok(hdr);
    const int64_t end = apos[row_hi];
    for (int64_t p = apos[row_lo] + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < end;
         p += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = arow[p], k = acrd[p];
        const int64_t ml = mpos[i + 1] - mpos[i], bl = bpos[k + 1] - bpos[k];
        int32_t at = -1;
        if (ml > 0 && tc_b_side(swap, ml, p - apos[i], bl, k, sh)) at = atomicAdd(bcount + k, 1);
        slot[p] = at;
    }
}

__global__ void __launch_bounds__(256)
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
__global__ void __launch_bounds__(256)
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

// probe function of a warp's hash set handed to tc_stream
template <int LOG2>
__device__ __forceinline__ unsigned tc_stream_set(const int32_t *tab, unsigned how, const int32_t *__restrict__ crd,
                                                  int64_t s, int len, int lane,
                                                  const int32_t *__restrict__ set, int set_len)
{
    if (how == TC_CUCKOO)
        return tc_stream(crd, s, len, lane, -2, [&](int32_t j) {
            return (unsigned)(tab[tc_h0<LOG2>(j)] == j) | (unsigned)(tab[tc_h1<LOG2>(j)] == j);
        });
    return tc_stream(crd, s, len, lane, -2, [&](int32_t j) {
        unsigned c = tc_linear_probe<LOG2>(tab, j);
        if (how == TC_REPEATS && c) {       // a hit counts as often as the set's row stores it
            c = 0;
            for (int t = 0; t < set_len; t++) c += set[t] == j ? 1u : 0u;
        }
        return c;
    });
}

// Mask rows of at most TC_WARP_MAX entries: a warp per row, its set built when the first list turns up.
__global__ void __launch_bounds__(TC_WARPS * 32)
tc_warp_kernel(TcHeader *hdr, const int32_t *__restrict__ small, const int64_t *__restrict__ apos,
               const int32_t *__restrict__ acrd, const int64_t *__restrict__ bpos,
               const int32_t *__restrict__ bcrd, const int64_t *__restrict__ mpos,
               const int32_t *__restrict__ mcrd, TcShape sh, unsigned long long *__restrict__ count)
{
    __shared__ __align__(16) int32_t s_tab[TC_WARPS][1 << TC_WARP_LOG2];
    __shared__ unsigned long long s_part[TC_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool swap = tc_swap_ok(hdr);
    const unsigned n = hdr->nsmall;
    unsigned long long hits = 0;
    while (true) {
        unsigned idx = 0;
        if (lane == 0) idx = atomicAdd(&hdr->next_small, 4u);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= n) break;
        const unsigned stop = idx + 4 < n ? idx + 4 : n;
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
                    if (!tc_b_side(swap, me - ms, p0 + lane - as, bl, k, sh)) len = (int)bl;
                }
                if (!__any_sync(0xffffffffu, len > 0)) continue;
                if (!filled) how = tc_fill<TC_WARP_LOG2>(s_tab[w], mcrd, ms, me, lane, false);
                filled = true;
                hits += tc_stream_set<TC_WARP_LOG2>(s_tab[w], how, bcrd, s, len, lane, nullptr, 0);
            }
            __syncwarp();
        }
    }
    tc_add_count(hits, s_part, TC_WARPS, count);
}

// A unit's next lists: lane l < n gets list number b + l of the unit (mask side: length 0 if it belongs to the B side).
// `first` is the unit's first entry of A's row (mask side) or first place in blist.  On the B side a list ends, at the
// latest, where the entry of M_i at the pair's own place o in row i already lies behind the set's last column.
__device__ __forceinline__ void tc_unit_lists(bool bside, int64_t first, int64_t off, int b, int n, int lists, int lane,
                                              bool swap, int64_t ml, int32_t last, TcShape sh,
                                              const int32_t *__restrict__ acrd, const int64_t *__restrict__ bpos,
                                              const int64_t *__restrict__ mpos, const int32_t *__restrict__ mcrd,
                                              const int2 *__restrict__ blist, int64_t &s, int &len)
{
    s = 0;
    len = 0;
    if (lane >= n || b + lane >= lists) return;
    if (bside) {
        const int2 io = __ldg(blist + first + b + lane);
        s = __ldg(mpos + io.x);
        len = (int)(__ldg(mpos + io.x + 1) - s);
        if (io.y < len && __ldg(mcrd + s + io.y) > last) len = io.y;
    } else {
        const int64_t k = __ldg(acrd + first + b + lane);
        s = __ldg(bpos + k);
        const int64_t bl = __ldg(bpos + k + 1) - s;
        len = tc_b_side(swap, ml, off + b + lane, bl, k, sh) ? 0 : (int)bl;
    }
}

// Units whose set has at most TC_MID_MAX entries: a warp per unit, the set as a hash set.
__global__ void __launch_bounds__(TC_MID_WARPS * 32)
tc_mid_kernel(TcHeader *hdr, const TcUnit *__restrict__ mids, const int64_t *__restrict__ apos,
              const int32_t *__restrict__ acrd, const int64_t *__restrict__ bpos, const int32_t *__restrict__ bcrd,
              const int64_t *__restrict__ mpos, const int32_t *__restrict__ mcrd, const int64_t *__restrict__ bptr,
              const int2 *__restrict__ blist, TcShape sh, unsigned long long *__restrict__ count)
{
    __shared__ __align__(16) int32_t s_tab[TC_MID_WARPS][1 << TC_MID_LOG2];
    __shared__ unsigned long long s_part[TC_MID_WARPS];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool swap = tc_swap_ok(hdr);
    const unsigned n = hdr->nmid;
    unsigned long long hits = 0;
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
        __syncwarp();
        for (int b = 0; b < lists; b += 32) {
            int64_t s;
            int len;
            tc_unit_lists(bside, row_at, u.off, b, 32, lists, lane, swap, se - ss, last, sh, acrd, bpos, mpos, mcrd, blist, s, len);
            hits += tc_stream_set<TC_MID_LOG2>(s_tab[w], how, lcrd, s, len, lane, scrd + ss, (int)(se - ss));
        }
        __syncwarp();
    }
    tc_add_count(hits, s_part, TC_MID_WARPS, count);
}

// Units: a bitmap of the set, its lists drawn by the warps in batches of 32.  SEGMENTED: the columns do not fit one
// bitmap, the unit is repeated per segment of `width` columns.  The next unit's set is fetched into shared memory by
// warp 0 while the others stream, so that between two units only the bits change.
template <int THREADS, bool SEGMENTED>
__global__ void __launch_bounds__(THREADS)
tc_bitmap_kernel(TcHeader *hdr, const TcUnit *__restrict__ units, const int64_t *__restrict__ apos,
                 const int32_t *__restrict__ acrd, const int64_t *__restrict__ bpos, const int32_t *__restrict__ bcrd,
                 const int64_t *__restrict__ mpos, const int32_t *__restrict__ mcrd, const int64_t *__restrict__ bptr,
                 const int2 *__restrict__ blist, TcShape sh, int width, const int64_t *ncols_dev,
                 unsigned long long *__restrict__ count)
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
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool swap = tc_swap_ok(hdr);
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
    unsigned long long hits = 0;
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
                int64_t s;
                int n;
                tc_unit_lists(bside, row_at, u.off, (int)b, step, lists, lane, swap, ml, bside ? s_last : 0, sh, acrd, bpos, mpos, mcrd,
                              blist, s, n);
                auto bit_of = [&](int32_t x) { return (bm[x >> 5] >> (x & 31)) & 1u; };
                if (SEGMENTED && ncols > width) {
                    hits += tc_stream(lcrd, s, n, lane, INT32_MAX, [&](int32_t j) {
                        const int64_t x = (int64_t)j - base;
                        unsigned c = x < 0 || x >= width ? 0u : bit_of((int32_t)x);
                        if (c && dup) {
                            c = 0;
                            for (int t = 0; t < len; t++) c += set[t] == j ? 1u : 0u;
                        }
                        return c;
                    });
                    continue;
                }
                if (!dup)
                    hits += tc_stream(lcrd, s, n, lane, width, bit_of);
                else                       // B_k repeats a coordinate: a hit counts as often as it is stored
                    hits += tc_stream(lcrd, s, n, lane, width, [&](int32_t j) {
                        unsigned c = 0;
                        if (bit_of(j)) for (int t = 0; t < len; t++) c += set[t] == j ? 1u : 0u;
                        return c;
                    });
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
    tc_add_count(hits, s_part, THREADS / 32, count);
}

template <int THREADS, bool SEGMENTED>
static int launch_bitmap(size_t smem, int per_sm, TcHeader *hdr, const TcUnit *units, const int64_t *apos,
                         const int32_t *acrd, const int64_t *bpos, const int32_t *bcrd, const int64_t *mpos,
                         const int32_t *mcrd, const int64_t *bptr, const int2 *blist, TcShape sh, int width,
                         const int64_t *ncols_dev, unsigned long long *count, cudaStream_t st)
{
    auto k = tc_bitmap_kernel<THREADS, SEGMENTED>;
    CB_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k<<<(unsigned)(sm_count() * per_sm), THREADS, smem, st>>>(hdr, units, apos, acrd, bpos, bcrd, mpos, mcrd, bptr, blist,
                                                             sh, width, ncols_dev, count);
    CB_LAUNCH_CHECK();
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
    const TcShape sh = {bcap, acrd == mcrd && apos == mpos};
    const int64_t words = ceil_div(ncols, 32);
    auto grid_for = [](int64_t n) {
        const int64_t blocks = ceil_div(n, 256), cap = (int64_t)sm_count() * 16;
        return (unsigned)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
    };
    const bool same_bm = bcrd == mcrd && nnz_b == nnz_m, same_am = acrd == mcrd && nnz_a == nnz_m;
    const bool same_ab = acrd == bcrd && nnz_a == nnz_b;

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
    CB_CUDA(cudaMemsetAsync(hdr, 0, counts_bytes, st));           // header, list counts, column bits

    if (compact) {
        tc_present_kernel<<<(unsigned)sm_count() * 4, 512, 0, st>>>(nnz_m, mcrd, present);
        CB_LAUNCH_CHECK();
        tc_popc_kernel<<<grid_for(words), 256, 0, st>>>(words, present, popc);
        CB_LAUNCH_CHECK();
        CB_TRY(exclusive_scan_i32(popc, before, words, st));
    }
    auto narrow = [&](const int64_t *crd, int64_t n, void *out, bool columns, bool check) {
        tc_narrow_kernel<<<grid_for(ceil_div(n, 2)), 256, 0, st>>>(n, crd, (int32_t *)out, columns ? present : nullptr, before,
                                                                  words, mpos, row_lo, row_hi, check ? hdr : nullptr);
        return cudaGetLastError() == cudaSuccess ? 0 : fail("masked count: narrowing failed");
    };
    CB_TRY(scratch(SLOT_NARROW_M, (size_t)nnz_m * 4 + 16, &m32));
    CB_TRY(narrow(mcrd, nnz_m, m32, true, true));
    if (same_bm) b32 = m32;
    else {
        CB_TRY(scratch(SLOT_NARROW_B, (size_t)nnz_b * 4 + 16, &b32));
        CB_TRY(narrow(bcrd, nnz_b, b32, true, false));
    }
    if (same_am && !compact) a32 = m32;
    else if (same_ab && !compact) a32 = b32;
    else {
        CB_TRY(scratch(SLOT_NARROW_A, (size_t)nnz_a * 4 + 16, &a32));
        CB_TRY(narrow(acrd, nnz_a, a32, false, false));
    }
    const int32_t *A = (const int32_t *)a32, *B = (const int32_t *)b32, *M = (const int32_t *)m32;
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
    unsigned long long *cnt = (unsigned long long *)count_dev;
    const int width = (int)(compact ? TC_MAX_COLS : ncols);
    const size_t smem = (size_t)2 * TC_SET_BUF * 4 + (size_t)((width >> 5) + 1) * 4;
    const int64_t *ncols_dev = compact ? before + words : nullptr;
    // one CTA of 32 warps per SM when the bitmap fills the shared memory, otherwise two of 32 or four of 16
    if (compact)
        CB_TRY((launch_bitmap<1024, true>(smem, 1, hdr, units, apos, A, bpos, B, mpos, M, bptr, blist, sh, width, ncols_dev,
                                          cnt, st)));
    else if (smem > 52 * 1024)
        CB_TRY((launch_bitmap<1024, false>(smem, smem > 108 * 1024 ? 1 : 2, hdr, units, apos, A, bpos, B, mpos, M, bptr, blist,
                                           sh, width, ncols_dev, cnt, st)));
    else
        CB_TRY((launch_bitmap<512, false>(smem, 4, hdr, units, apos, A, bpos, B, mpos, M, bptr, blist, sh, width, ncols_dev,
                                          cnt, st)));
    tc_mid_kernel<<<(unsigned)sm_count() * 6, TC_MID_WARPS * 32, 0, st>>>(hdr, mids, apos, A, bpos, B, mpos, M, bptr, blist,
                                                                          sh, cnt);
    CB_LAUNCH_CHECK();
    tc_warp_kernel<<<(unsigned)sm_count() * 8, TC_WARPS * 32, 0, st>>>(hdr, small, apos, A, bpos, B, mpos, M, sh, cnt);
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
