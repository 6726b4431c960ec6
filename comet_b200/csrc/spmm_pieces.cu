// SpMM over equal pieces of A's path, one group of lanes per piece.
//
// The path walks A row by row, one step per stored entry and one per row end (the merge path of Merrill and Garland,
// Merge-based Parallel Sparse Matrix-Vector Multiplication, 2016).  It is cut into equal pieces, and a group of
// T lanes takes one: T lanes x NI vectors cover the columns of B and C, so a warp holds 32 / T pieces and narrow
// operands still use every lane.  A group loads up to eight entries of its piece at a time (a lane one to four of
// them), hands them round with shuffles and keeps U rows of B in flight.  Rows inside a piece are stored; of a row that a
// boundary cuts, every piece leaves its part in scratch memory (the part of a row that started before it in one slot, of a
// row that goes on after it in another), and a last kernel adds the parts up in the order of the pieces.  So hub rows are
// shared by as many groups as they have pieces, no row waits for another, and the sums of every call are the same to the
// bit.  (Adding the parts of a CTA's pieces up in shared memory first made the pieces' kernel 10 to 60 % slower.)
//
// V = double2 where K, both leading dimensions and both addresses allow 16-byte accesses, otherwise double: an odd
// number of columns costs twice the load instructions and no more.  K beyond one pass is walked in slices.
//
// Bound: the L2 -> SM rate (17 TB/s) for the gathered rows of B and the latency of a group's entry -> row of B chain.
// R-MAT scale 20, 16 entries per row, against the lane group per row (even K) or thread per row (odd K) it took over from:
// K = 4 1052 -> 268 us, K = 8 810 -> 314, K = 13 9586 -> 467, K = 33 10214 -> 865, K = 48 1259 -> 917, K = 63 12343 -> 1149.
// Atomics in the place of the parts, whose order is another one in every call: 251, 272, 435, 835, 882, 1152; at scale 17
// K = 33 107 against 128, K = 63 148 against 167.
#include "common.cuh"
#include "spmm.cuh"

namespace cb200 {

static const int SP_THREADS = 256;
static const int MANY = 8;                 // parts of a row that one thread adds up at most
static const int RUN_SUMS = 2048;          // rows x runs x columns that a CTA holds sums of

// CTAs per SM that the registers of a lane's accumulators and rows in flight allow
template <typename V>
constexpr int pieces_ctas(int ni)
{
    return ni * (int)sizeof(V) <= 24 ? 4 : ni * (int)sizeof(V) < 64 ? 3 : 2;
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
    out->s = s;
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
int stream_plan(int64_t nrows, int64_t nnz, int64_t warps, int64_t most, const int64_t *row_ids, const int64_t *pos, double *c,
                int64_t ldc, int64_t k, int accumulate, LongRows lr, cudaStream_t st, StreamPlan *out)
{
    int s = 6;
    while ((nnz + nrows) >> (s + 1) >= warps * 8 || (nnz + nrows) >> s >= most) s++;
    if ((nnz + nrows) >> s > 0x7ffffff0LL) return 0;
    return piece_plan(nrows, nnz, s, row_ids, pos, c, ldc, k, accumulate, lr, st, out) ? -1 : 1;
}

template <typename V, int T, int NI, bool PAIR>
__global__ void __launch_bounds__(SP_THREADS, pieces_ctas<V>(NI))
spmm_pieces_kernel(int64_t nrows, int64_t npieces, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                   const int64_t *__restrict__ crd, const double *__restrict__ val, const double *__restrict__ b0, uint32_t ldb8,
                   double *__restrict__ c0, int64_t ldc, int k, int accumulate, const int64_t *__restrict__ piece_row,
                   const int64_t *__restrict__ piece_ent, LongRows lr, double *__restrict__ parts, unsigned all_k)
{
    wait_for_previous();
    if (not_this(lr)) return;
    constexpr int EPL = T >= 8 ? 1 : 8 / T;            // entries a lane loads at a time
    constexpr int BATCH = T * EPL;
    constexpr int U = NI >= 3 ? 2 : 4;                 // rows of B in flight
    constexpr int VN = Vec<V>::N;
    const int lane = threadIdx.x & 31, l = threadIdx.x & (T - 1);
    const unsigned gmask = (T == 32) ? 0xffffffffu : (((1u << T) - 1u) << (lane & ~(T - 1)));
    const unsigned piece = blockIdx.x * (SP_THREADS / T) + threadIdx.x / T;
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

    auto flush = [&](bool ends) {
        if (whole && ends) {
            V *crow = (V *)(c + (row_ids ? row_ids[r] : r) * ldc) + l;
#pragma unroll
            for (int i = 0; i < NI; i++) {
                if (on[i]) {
                    if (accumulate) Vec<V>::add_to(acc[i], crow[i * T]);
                    __stcs(crow + i * T, acc[i]);      // written once, not read again here
                }
                acc[i] = Vec<V>::zero();
            }
        } else {
            // the piece's number is made again: kept in a register it costs some kernels a CTA per SM (PARTS_BYTES: 32 bits do)
            const unsigned at = 2 * (blockIdx.x * (SP_THREADS / T) + threadIdx.x / T) + (whole ? 1 : 0);
            V *crow = (V *)(parts + (at * all_k + blockIdx.y * (T * NI * VN))) + l;
#pragma unroll
            for (int i = 0; i < NI; i++) {
                if (on[i]) crow[i * T] = acc[i];
                acc[i] = Vec<V>::zero();
            }
        }
    };
    auto next_row = [&]() {
        flush(true);
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

// The row that a piece starts and does not end, its parts in order.  W lanes take four neighbouring pieces at a time, as the
// chain from the plan to the parts is all there is to wait for.  Rows of more than MANY parts are left to the whole CTA, which
// works on all that it has at a time (one by one the hub rows of a power-law matrix, which lie together, took 50 us): `runs` runs
// of a row's parts first, then their sums; the order depends on `runs` and the number of parts alone.
template <int W>
__global__ void __launch_bounds__(SP_THREADS)
spmm_parts_kernel(int64_t nrows, int64_t npieces, int s, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                  double *__restrict__ c, int64_t ldc, int k, int accumulate, const int64_t *__restrict__ piece_row,
                  const int64_t *__restrict__ piece_ent, LongRows lr, int runs, const double *__restrict__ parts)
{
    constexpr int U = 4, GROUPS = SP_THREADS / W, LONG = GROUPS * U / MANY + 1;      // a long row covers MANY pieces after its first
    __shared__ int64_t s_piece[LONG], s_row[LONG];
    __shared__ int s_parts[LONG], n_long;
    __shared__ double s_sum[RUN_SUMS];
    wait_for_previous();
    if (not_this(lr)) return;
    if (threadIdx.x == 0) n_long = 0;
    __syncthreads();
    const int l = threadIdx.x % W;
    const int64_t b0 = ((int64_t)blockIdx.x * GROUPS + threadIdx.x / W) * U;
    auto put = [&](int64_t row, int j, double sum) {
        double *at = c + (row_ids ? row_ids[row] : row) * ldc + j;
        *at = accumulate ? *at + sum : sum;
    };
    int64_t r[U];
    int m[U], most = 0;                                // parts; 0: the row starts elsewhere, or none of it is in this piece
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int64_t b = b0 + u < npieces ? b0 + u : npieces - 1;
        r[u] = piece_row[b + 1];
        const int64_t start = b0 + u < npieces && r[u] < nrows ? pos[r[u]] : -1;
        m[u] = 0;
        if (start >= piece_ent[b] && start < piece_ent[b + 1])
            m[u] = (int)(((pos[r[u] + 1] + r[u] - 1) >> s) - b + 1);   // up to the piece of its last entry
        if (m[u] > MANY) {
            if (l == 0) {
                const int i = atomicAdd(&n_long, 1);
                s_piece[i] = b;
                s_row[i] = r[u];
                s_parts[i] = m[u];
            }
            m[u] = 0;
        }
        most = m[u] > most ? m[u] : most;
    }
    for (int j = l; j < k; j += W) {
        const double *at = parts + 2 * b0 * k + j;
        double sum[U];
#pragma unroll
        for (int u = 0; u < U; u++) sum[u] = m[u] ? at[(2 * u + 1) * k] + at[2 * (u + 1) * k] : 0.0;
#pragma unroll 2
        for (int t = 2; t < most; t++)
#pragma unroll
            for (int u = 0; u < U; u++)
                if (t < m[u]) sum[u] += at[2 * (u + t) * k];
#pragma unroll
        for (int u = 0; u < U; u++)
            if (m[u]) put(r[u], j, sum[u]);
    }
    __syncthreads();
    const int cols_most = k < RUN_SUMS / runs ? k : RUN_SUMS / runs, rows_most = RUN_SUMS / (runs * cols_most);
    for (int i0 = 0; i0 < n_long; i0 += rows_most) {
        const int rows = n_long - i0 < rows_most ? n_long - i0 : rows_most;
        for (int c0 = 0; c0 < k; c0 += cols_most) {
            const int cols = k - c0 < cols_most ? k - c0 : cols_most, items = rows * runs * cols;
            for (int t0 = threadIdx.x; t0 < items; t0 += U * SP_THREADS) {
                const double *at[U];
                int n[U], longest = 0;
                double sum[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int t = t0 + u * SP_THREADS, i = t / (runs * cols), w = t / cols - i * runs, j = t % cols;
                    n[u] = 0;
                    sum[u] = 0.0;
                    if (t < items) {
                        const int all = s_parts[i0 + i] - 1, len = (all + runs - 1) / runs, q0 = w * len;
                        n[u] = all - q0 < len ? all - q0 : len;
                        at[u] = parts + 2 * (s_piece[i0 + i] + 1 + q0) * k + c0 + j;
                    }
                    longest = n[u] > longest ? n[u] : longest;
                }
#pragma unroll 2
                for (int64_t q = 0; q < longest; q++)
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (q < n[u]) sum[u] += at[u][2 * q * k];
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (t0 + u * SP_THREADS < items) s_sum[t0 + u * SP_THREADS] = sum[u];
            }
            __syncthreads();
            for (int t = threadIdx.x; t < rows * cols; t += SP_THREADS) {
                const int i = t / cols, j = t - i * cols;
                double sum = parts[(2 * s_piece[i0 + i] + 1) * k + c0 + j];
                for (int w = 0; w < runs; w++) sum += s_sum[(i * runs + w) * cols + j];
                put(s_row[i0 + i], c0 + j, sum);
            }
            __syncthreads();
        }
    }
}

int piece_parts(int64_t npieces, int64_t k, double **parts)
{
    void *mem = nullptr;
    CB_TRY(scratch(SLOT_MISC, (size_t)npieces * 2 * (size_t)k * sizeof(double), &mem));
    *parts = (double *)mem;
    return 0;
}

int add_parts(const SpmmCall &a, const StreamPlan &plan, LongRows lr, const double *parts)
{
    // as many runs as there are threads for; a small product's sums do not depend on its columns
    int runs = 32;
    while (a.nnz >= SPMM_SMALL_NNZ && runs > 4 && runs * a.k > RUN_SUMS / 2) runs /= 2;
    auto kernel = a.k <= 4 ? spmm_parts_kernel<4> : a.k <= 8 ? spmm_parts_kernel<8> : a.k <= 16 ? spmm_parts_kernel<16> : spmm_parts_kernel<32>;
    const int w = a.k <= 4 ? 4 : a.k <= 8 ? 8 : a.k <= 16 ? 16 : 32;
    CB_CUDA(launch_behind(kernel, dim3((unsigned)ceil_div(plan.nblocks, SP_THREADS / w * 4)), SP_THREADS, 0, a.st, a.nrows, plan.nblocks,
                          plan.s, a.row_ids, a.pos, a.c, a.ldc, (int)a.k, a.accumulate, plan.block_row, plan.block_ent, lr, runs, parts));
    return 0;
}

template <typename V, int T, int NI>
static int launch_pieces(const SpmmCall &a, LongRows lr)
{
    const int64_t kv = a.k / Vec<V>::N;
    const int64_t groups = (int64_t)sm_count() * SP_THREADS * pieces_ctas<V>(NI) / T;      // on the chip at a time
    int s = 5;                                         // 2^5 to 2^8 steps, the longest that still give four rounds (eight: more parts; R-MAT scale 17, K = 48 138 -> 148 us)
    if (a.nnz < SPMM_SMALL_NNZ) {                      // the same pieces at every K, so that a product taken in panels has the sums of the whole one
        while ((a.nnz + a.nrows) >> s >= (1 << 13)) s++;
    } else {
        while (s < 8 && (a.nnz + a.nrows) >> (s + 1) >= groups * 4) s++;
        while ((a.nnz + a.nrows) >> s >= PARTS_BYTES / (16 * a.k)) s++;
    }
    StreamPlan plan;
    CB_TRY(piece_plan(a.nrows, a.nnz, s, a.row_ids, a.pos, nullptr, 0, 0, 0, lr, a.st, &plan));
    const int64_t blocks = ceil_div(plan.nblocks * T, SP_THREADS), slices = ceil_div(kv, T * NI);
    double *parts = nullptr;
    CB_TRY(piece_parts(plan.nblocks, a.k, &parts));
    auto kernel = a.pair ? spmm_pieces_kernel<V, T, NI, true> : spmm_pieces_kernel<V, T, NI, false>;
    CB_CUDA(launch_behind(kernel, dim3((unsigned)blocks, (unsigned)slices), SP_THREADS, 0, a.st, a.nrows, plan.nblocks, a.row_ids, a.pos,
                          a.crd, a.val, a.b, (uint32_t)(a.ldb * 8), a.c, a.ldc, (int)a.k, a.accumulate, plan.block_row, plan.block_ent,
                          lr, parts, (unsigned)a.k));
    return add_parts(a, plan, lr, parts);
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
    for (int64_t col0 = 0; col0 < a.k; col0 += 512) {  // the parts' memory grows with the columns
        SpmmCall slab = a;
        slab.k = a.k - col0 < 512 ? a.k - col0 : 512;
        slab.b += col0;
        slab.c += col0;
        CB_TRY(slab.vec ? dispatch_pieces<double2>(slab, lr) : dispatch_pieces<double>(slab, lr));
    }
    return 0;
}

}  // namespace cb200
