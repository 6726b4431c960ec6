// SpMM over equal pieces of A's path, one group of lanes per piece.
//
// The path walks A row by row, one step per stored entry and one per row end.  It is cut into equal pieces, and a group of
// T lanes takes one: T lanes x NI vectors cover the columns of B and C, so a warp holds 32 / T pieces and narrow
// operands still use every lane.  A group loads up to eight entries of its piece at a time (a lane one to four of
// them), hands them round with shuffles and keeps U rows of B in flight.  Rows inside a piece are stored; rows that a
// boundary cuts are added with f64 atomics onto zeros that the plan kernel has written, so hub rows are shared by as many
// groups as they have pieces and no row waits for another.
//
// FIXED, for small matrices: a piece leaves its part of a cut row in scratch memory instead (the part of a row that started
// before it in one slot, of a row that goes on after it in another), and a last kernel adds the parts up in the order of
// the pieces, so the sums of every call are the same to the bit.  It costs 2 us.
//
// V = double2 where K, both leading dimensions and both addresses allow 16-byte accesses, otherwise double: an odd
// number of columns costs twice the load instructions and no more.  K beyond one pass is walked in slices.
//
// Bound: the L2 -> SM rate (17 TB/s) for the gathered rows of B and the latency of a group's entry -> row of B chain.
// R-MAT scale 20, 16 entries per row, against the lane group per row (even K) or thread per row (odd K) it took over from:
// K = 4 1052 -> 230 us, K = 8 810 -> 260, K = 13 9586 -> 440, K = 33 10214 -> 820, K = 48 1259 -> 860, K = 127 14030 -> 2400.
#include "common.cuh"
#include "spmm.cuh"

namespace cb200 {

static const int SP_THREADS = 256;

// CTAs per SM that the registers of a lane's accumulators and rows in flight allow
template <typename V>
constexpr int pieces_ctas(int ni)
{
    return ni * (int)sizeof(V) <= 16 ? 4 : ni * (int)sizeof(V) < 64 ? 3 : 2;
}

// Boundary b of the plan lies b * 2^s steps along the path: in row piece_row[b], before entry piece_ent[b] (a boundary
// behind a row's last entry counts as the next row's start).  A thread per row writes the boundaries that fall into
// its row's steps (a search per boundary took as long as the product of a small matrix); a warp shares the boundaries of
// a long row.  Rows that a boundary cuts get zeros when their parts are going to be added up.
//
// A warp takes four neighbouring rows from each of eight places evenly spread over the matrix: graphs keep their long rows
// together, and a warp with 32 of them was what the kernel waited for.
__global__ void __launch_bounds__(256)
spmm_plan_kernel(int64_t nrows, int s, int64_t npieces, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                 double *__restrict__ c, int64_t ldc, int64_t k, bool clear, LongRows lr, int64_t *__restrict__ piece_row,
                 int64_t *__restrict__ piece_ent, WorkHeader *hdr)
{
    wait_for_previous();
    let_next_start();
    if (not_this(lr)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) hdr->pad[0] = 0;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5), mask = ((int64_t)1 << s) - 1;
    const int64_t part = ((nrows + 3) / 4 + 7) / 8;    // groups of four rows per place
    for (int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < part; g += warps) {
        const int64_t r = ((lane >> 2) * part + g) * 4 + (lane & 3);
        bool cut = false;
        int64_t ps = 0, pe = 0, b0 = 0, b1 = 0;        // boundaries b0 .. b1 - 1 lie in row r
        // steps of the row: (ps + r, pe + r + 1]; step pe + r + 1 is its end, and so is a boundary behind its last entry
        auto put = [&](int64_t b, int64_t row, int64_t end) {
            const int64_t e = (b << s) - row;          // entries before the boundary
            const bool next = b > 0 && e == end;
            piece_row[b] = next ? row + 1 : row;
            piece_ent[b] = e;
            return !next;
        };
        if (r < nrows) {
            ps = pos[r];
            pe = pos[r + 1];
            b0 = (ps + r + mask) >> s;
            b1 = (pe + r + 1 + mask) >> s;
            if (b1 > npieces) b1 = npieces;
            if (r == nrows - 1)
                for (int64_t b = (pe + nrows + mask) >> s; b <= npieces; b++) {
                    piece_row[b] = nrows;
                    piece_ent[b] = pe;
                }
            if (b1 - b0 <= 4)
                for (int64_t b = b0; b < b1; b++)
                    if (put(b, r, pe) && (b << s) - r > ps) cut = true;
        }
        unsigned many = __ballot_sync(0xffffffffu, b1 - b0 > 4);
        if (b1 - b0 > 4) cut = true;
        while (many) {
            const int t = __ffs(many) - 1;
            many &= many - 1;
            const int64_t tb = __shfl_sync(0xffffffffu, (long long)b0, t), te = __shfl_sync(0xffffffffu, (long long)b1, t),
                          tp = __shfl_sync(0xffffffffu, (long long)pe, t), tr = __shfl_sync(0xffffffffu, (long long)r, t);
            for (int64_t b = tb + lane; b < te; b += 32) put(b, tr, tp);
        }
        unsigned cuts = __ballot_sync(0xffffffffu, cut && clear);
        while (cuts) {
            const int64_t rr = __shfl_sync(0xffffffffu, (long long)r, __ffs(cuts) - 1);
            cuts &= cuts - 1;
            double *crow = c + (row_ids ? row_ids[rr] : rr) * ldc;
            for (int64_t j = lane; j < k; j += 32) crow[j] = 0.0;
        }
    }
}

int piece_plan(int64_t nrows, int64_t nnz, int s, const int64_t *row_ids, const int64_t *pos, double *c, int64_t ldc,
               int64_t k, int accumulate, LongRows lr, cudaStream_t st, StreamPlan *out)
{
    out->nblocks = ceil_div(nnz + nrows, (int64_t)1 << s);
    void *wl = nullptr;
    CB_TRY(scratch(SLOT_WORKLIST, sizeof(WorkHeader) + (size_t)(out->nblocks + 1) * 2 * sizeof(int64_t), &wl));
    out->hdr = (WorkHeader *)wl;
    out->block_row = (int64_t *)((char *)wl + sizeof(WorkHeader));
    out->block_ent = out->block_row + (out->nblocks + 1);
    int64_t grid = ceil_div(nrows, 256);
    if (grid > sm_count() * 8) grid = sm_count() * 8;
    CB_CUDA(launch_behind(spmm_plan_kernel, dim3((unsigned)grid), 256, 0, st, nrows, s, out->nblocks, row_ids, pos, c, ldc, k,
                          c && !accumulate, lr, out->block_row, out->block_ent, out->hdr));
    return 0;
}

// Pieces of 2^6 to 2^9 steps, the longest that still leave eight for each warp: short ones keep a small matrix's warps busy
// (R-MAT scale 14, K = 128: 30 us with 2^6, 43 with 2^7, 117 with 2^9), long ones cut fewer rows (scale 20: 2^6 1560, 2^9 1290).
int stream_plan(int64_t nrows, int64_t nnz, int64_t warps, const int64_t *row_ids, const int64_t *pos, double *c,
                int64_t ldc, int64_t k, int accumulate, LongRows lr, cudaStream_t st, StreamPlan *out)
{
    int s = 6;
    while ((nnz + nrows) >> (s + 1) >= warps * 8) s++;
    if ((nnz + nrows) >> s > 0x7ffffff0LL) return 0;
    return piece_plan(nrows, nnz, s, row_ids, pos, c, ldc, k, accumulate, lr, st, out) ? -1 : 1;
}

template <typename V, int T, int NI, bool PAIR, bool FIXED>
__global__ void __launch_bounds__(SP_THREADS, pieces_ctas<V>(NI))
spmm_pieces_kernel(int64_t nrows, int64_t npieces, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                   const int64_t *__restrict__ crd, const double *__restrict__ val, const double *__restrict__ b0, uint32_t ldb8,
                   double *__restrict__ c0, int64_t ldc, int k, int accumulate, const int64_t *__restrict__ piece_row,
                   const int64_t *__restrict__ piece_ent, LongRows lr, double *__restrict__ parts, int64_t all_k)
{
    wait_for_previous();
    if (not_this(lr)) return;
    constexpr int EPL = T >= 8 ? 1 : 8 / T;            // entries a lane loads at a time
    constexpr int BATCH = T * EPL;
    constexpr int U = NI >= 3 ? 2 : 4;                 // rows of B in flight
    constexpr int VN = Vec<V>::N;
    const int lane = threadIdx.x & 31, l = threadIdx.x & (T - 1);
    const unsigned gmask = (T == 32) ? 0xffffffffu : (((1u << T) - 1u) << (lane & ~(T - 1)));
    const int64_t piece = ((int64_t)blockIdx.x * SP_THREADS + threadIdx.x) / T;
    if (piece >= npieces) return;
    const int col0 = blockIdx.y * (T * NI * VN);       // columns of this slice
    const int kv = (k - col0 < T * NI * VN ? k - col0 : T * NI * VN) / VN;
    const char *b = (const char *)((const V *)(b0 + col0) + l);
    double *c = c0 + col0;
    bool on[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) on[i] = l + i * T < kv;

    // entries and row ends are counted from the piece's first entry
    const int64_t e0 = piece_ent[piece], rend = piece_row[piece + 1];              // rows before rend end in this piece
    const int n_ent = (int)(piece_ent[piece + 1] - e0);
    const int64_t *crd_p = crd + e0;
    const double *val_p = val + e0;
    int64_t r = piece_row[piece];
    bool whole = true;                                 // row r starts in this piece
    auto end_of = [&](int64_t row) {
        if (row >= nrows) return n_ent + 1;
        const int64_t d = pos[row + 1] - e0;
        return d > n_ent ? n_ent + 1 : (int)d;         // n_ent + 1: it ends behind the piece
    };
    if (r < nrows) whole = pos[r] >= e0;
    int re = end_of(r);
    V acc[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) acc[i] = Vec<V>::zero();

    auto flush = [&](bool store) {
        V *crow = FIXED && !store ? (V *)(parts + (2 * piece + (whole ? 1 : 0)) * all_k + col0)
                                  : (V *)(c + (row_ids ? row_ids[r] : r) * ldc);
#pragma unroll
        for (int i = 0; i < NI; i++) {
            if (on[i]) {
                V *at = crow + l + i * T;
                if (!store && FIXED) *at = acc[i];
                else if (!store) Vec<V>::atomic_to(at, acc[i]);
                else {
                    if (accumulate) Vec<V>::add_to(acc[i], *at);
                    __stcs(at, acc[i]);                // written once, not read again here
                }
            }
            acc[i] = Vec<V>::zero();
        }
    };
    auto next_row = [&]() {
        flush(whole);
        r += 1;
        whole = true;
        re = end_of(r);
    };

    uint32_t cl[EPL];
    double vl[EPL];
    auto load = [&](int at) {
#pragma unroll
        for (int i = 0; i < EPL; i++) {
            const int p = at + l + i * T;
            cl[i] = 0;
            vl[i] = 0.0;
            if (p < n_ent) {
                cl[i] = (uint32_t)ld_stream(crd_p + p);
                if (!PAIR) vl[i] = ld_stream(val_p + p);
            }
        }
    };
    load(0);
    for (int e = 0; e < n_ent; e += BATCH) {
        uint32_t cc[EPL];
        double vv[EPL];
#pragma unroll
        for (int i = 0; i < EPL; i++) { cc[i] = cl[i]; vv[i] = vl[i]; }
        load(e + BATCH);                               // the next batch's entries are on their way meanwhile
#pragma unroll
        for (int t0 = 0; t0 < BATCH; t0 += U) {
            const int left = n_ent - e - t0;
            if (left <= 0) break;
            V bv[U][NI];
            double av[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int t = t0 + u;
                const uint32_t col = __shfl_sync(gmask, cc[t / T], t % T, T);
                av[u] = PAIR ? 1.0 : __shfl_sync(gmask, vv[t / T], t % T, T);
                const char *src = b + (uint64_t)col * ldb8;
#pragma unroll
                for (int i = 0; i < NI; i++)
                    bv[u][i] = PAIR ? Vec<V>::ones(1.0) : (u < left && on[i]) ? __ldg((const V *)src + i * T) : Vec<V>::zero();
            }
            if (e + t0 + U <= re && left >= U) {       // all of them belong to the row in progress
#pragma unroll
                for (int u = 0; u < U; u++)
#pragma unroll
                    for (int i = 0; i < NI; i++) Vec<V>::fma_to(acc[i], av[u], bv[u][i]);
            } else {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (u < left) {
                        while (e + t0 + u >= re) next_row();
#pragma unroll
                        for (int i = 0; i < NI; i++) Vec<V>::fma_to(acc[i], av[u], bv[u][i]);
                    }
                }
            }
        }
    }
    // rows that end in this piece (the one in progress, empty ones after it), then the part of row rend that it holds
    while (r < rend) next_row();
    if (rend < nrows && e0 + n_ent > pos[rend]) flush(false);
}

// FIXED: the row that piece b starts and does not end, its parts in order.  A warp per piece.
__global__ void __launch_bounds__(256)
spmm_parts_kernel(int64_t nrows, int64_t npieces, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                  double *__restrict__ c, int64_t ldc, int64_t k, int accumulate, const int64_t *__restrict__ piece_row,
                  const int64_t *__restrict__ piece_ent, LongRows lr, const double *__restrict__ parts)
{
    wait_for_previous();
    if (not_this(lr)) return;
    const int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (b >= npieces) return;
    const int64_t r = piece_row[b + 1];
    if (r >= nrows) return;
    const int64_t start = pos[r];
    if (start < piece_ent[b] || start >= piece_ent[b + 1]) return;      // starts in another piece, or none of it is in this one
    int64_t last = b + 1;
    while (last + 1 < npieces && piece_row[last + 1] <= r) last++;      // the piece in which the row ends
    double *crow = c + (row_ids ? row_ids[r] : r) * ldc;
    for (int64_t j = threadIdx.x & 31; j < k; j += 32) {
        double sum = parts[(2 * b + 1) * k + j];
#pragma unroll 4
        for (int64_t q = b + 1; q <= last; q++) sum += parts[2 * q * k + j];
        crow[j] = accumulate ? crow[j] + sum : sum;
    }
}

template <typename V, int T, int NI>
static int launch_pieces(const SpmmCall &a, LongRows lr)
{
    const int64_t kv = a.k / Vec<V>::N;
    const int64_t groups = (int64_t)sm_count() * SP_THREADS * pieces_ctas<V>(NI) / T;      // on the chip at a time
    int s = 5;                                         // 2^5 to 2^8 steps, the longest that still give eight rounds (four: 2 to 6 % slower)
    // The same pieces at every K, so that a product taken in panels has the sums of the whole one
    const bool fixed = a.nnz < SPMM_FIXED_NNZ && !a.pair;
    double *parts = nullptr;
    if (fixed) {
        while ((a.nnz + a.nrows) >> s >= (1 << 13)) s++;               // parts of 64 MB at most
        void *mem = nullptr;
        CB_TRY(scratch(SLOT_MISC, (size_t)(ceil_div(a.nnz + a.nrows, (int64_t)1 << s) + 1) * 2 * (size_t)a.k * sizeof(double), &mem));
        parts = (double *)mem;
    } else {
        while (s < 8 && (a.nnz + a.nrows) >> (s + 1) >= groups * 8) s++;
        while ((a.nnz + a.nrows) >> s >= (1LL << 31)) s++;
    }
    StreamPlan plan;
    CB_TRY(piece_plan(a.nrows, a.nnz, s, a.row_ids, a.pos, fixed ? nullptr : a.c, a.ldc, a.k, a.accumulate, lr, a.st, &plan));
    const int64_t blocks = ceil_div(plan.nblocks * T, SP_THREADS), slices = ceil_div(kv, T * NI);
    auto kernel = a.pair  ? spmm_pieces_kernel<V, T, NI, true, false>
                  : fixed ? spmm_pieces_kernel<V, T, NI, false, true>
                          : spmm_pieces_kernel<V, T, NI, false, false>;
    for (int64_t first = 0; first < slices; first += 65535) {
        const int64_t n = slices - first < 65535 ? slices - first : 65535, col0 = first * T * NI * Vec<V>::N;
        CB_CUDA(launch_behind(kernel, dim3((unsigned)blocks, (unsigned)n), SP_THREADS, 0, a.st, a.nrows, plan.nblocks, a.row_ids,
                              a.pos, a.crd, a.val, a.b + col0, (uint32_t)(a.ldb * 8), a.c + col0, a.ldc, (int)(a.k - col0),
                              a.accumulate, plan.block_row, plan.block_ent, lr, parts ? parts + col0 : nullptr, a.k));
    }
    if (fixed)
        CB_CUDA(launch_behind(spmm_parts_kernel, dim3((unsigned)ceil_div(plan.nblocks * 32, 256)), 256, 0, a.st, a.nrows, plan.nblocks,
                              a.row_ids, a.pos, a.c, a.ldc, a.k, a.accumulate, plan.block_row, plan.block_ent, lr, parts));
    return 0;
}

// As few lanes as cover the columns with one vector each up to 16, then more vectors a lane: at 17 to 32 vectors 16 lanes x 2
// beat 32 x 1 (R-MAT scale 20, K = 48: 890 against 1030 us), at 33 to 48 vectors 16 x 3 beat 32 x 2 (scale 17, K = 96: 128
// against 227).  On a small matrix narrow rows get lanes that would idle anyway: 16 of them load a piece's entries at once
// (R-MAT scale 14, K = 4: 49 -> 27 us).  Beyond 128 vectors in slices as even as they go.
template <typename V>
static int dispatch_pieces(const SpmmCall &a, LongRows lr)
{
    const int64_t kv = a.k / Vec<V>::N;
    int64_t t = kv <= 2 ? 2 : kv <= 4 ? 4 : kv <= 8 ? 8 : 16;
    while (t < 16 && ((a.nnz + a.nrows) >> 5) * t * 2 <= (int64_t)sm_count() * 1024) t *= 2;
    if (t == 2) return launch_pieces<V, 2, 1>(a, lr);
    if (t == 4) return launch_pieces<V, 4, 1>(a, lr);
    if (t == 8) return launch_pieces<V, 8, 1>(a, lr);
    if (kv <= 16) return launch_pieces<V, 16, 1>(a, lr);
    if (kv <= 32) return launch_pieces<V, 16, 2>(a, lr);
    if (kv <= 48) return launch_pieces<V, 16, 3>(a, lr);
    const int64_t width = ceil_div(kv, ceil_div(kv, 128));
    if (width <= 64) return launch_pieces<V, 32, 2>(a, lr);
    if (width <= 96) return launch_pieces<V, 32, 3>(a, lr);
    return launch_pieces<V, 32, 4>(a, lr);
}

int spmm_pieces(const SpmmCall &a, LongRows lr)
{
    if (a.k > 512 && a.nnz < SPMM_FIXED_NNZ) {         // the parts' memory grows with the columns
        for (int64_t col0 = 0; col0 < a.k; col0 += 512) {
            SpmmCall slab = a;
            slab.k = a.k - col0 < 512 ? a.k - col0 : 512;
            slab.b += col0;
            slab.c += col0;
            CB_TRY(spmm_pieces(slab, lr));
        }
        return 0;
    }
    return a.vec ? dispatch_pieces<double2>(a, lr) : dispatch_pieces<double>(a, lr);
}

}  // namespace cb200
