// SDDMM  out[p] = S.val[p] * sum_k X[i,k] * Y[j,k]   for every stored (i,j) of S (CSR).
//
// Every entry is a dot product of its own, so the entries are cut into equal pieces whatever rows they belong to, one warp
// per piece.  A warp takes 32 entries at a time: a lane each loads their columns and values, one batch ahead, and finds
// their rows among 32 row ends that the lanes hold (six shuffles; the ends are replaced when a batch runs past them).
// Groups of G lanes then take G consecutive entries each: NI vectors per lane cover the columns, X[i,:] stays in registers
// while the row does not change, and the products of U entries are in flight.  An entry's sum is finished with
// xor-shuffles and lands in the lane that holds its place, so results leave in one coalesced store.
//
// A batch of one row (long rows: most of a power-law matrix) takes a path with X[i,:] loaded once and nothing but Y in flight.
//
// V = double2 where K, both leading dimensions and both addresses allow 16-byte accesses, otherwise double: an odd number of
// columns costs twice the load instructions and no more.  K beyond one pass of a warp is walked in slices (LOOP).
//
// Bound: HBM for the arrays, 8(n+1) + 24 nnz + 8 K (nrows + ncols) bytes; with wide rows the L2 -> SM rate (17 TB/s) for the
// gathered rows of Y.
#include "common.cuh"
#include "stream.cuh"

namespace cb200 {

static const int SD_THREADS = 256;

// piece_row[b]: the row of entry b * 2^s.  A thread per row, a warp together for a row with many pieces.
__global__ void __launch_bounds__(256)
sddmm_plan_kernel(int64_t nrows, int s, int64_t npieces, const int64_t *__restrict__ pos, int32_t *__restrict__ piece_row)
{
    let_next_start();
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, mask = ((int64_t)1 << s) - 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) piece_row[npieces] = (int32_t)(nrows - 1);
    for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; r0 < nrows; r0 += stride) {
        int64_t b0 = 0, b1 = 0;
        if (r0 + lane < nrows) {
            b0 = (pos[r0 + lane] + mask) >> s;
            b1 = (pos[r0 + lane + 1] + mask) >> s;
            if (b1 > npieces) b1 = npieces;
        }
        if (b1 - b0 <= 4)
            for (int64_t b = b0; b < b1; b++) piece_row[b] = (int32_t)(r0 + lane);
        unsigned many = __ballot_sync(0xffffffffu, b1 - b0 > 4);
        while (many) {
            const int t = __ffs(many) - 1;
            many &= many - 1;
            const int64_t tb = __shfl_sync(0xffffffffu, (long long)b0, t), te = __shfl_sync(0xffffffffu, (long long)b1, t);
            for (int64_t b = tb + lane; b < te; b += 32) piece_row[b] = (int32_t)(r0 + t);
        }
    }
}

__device__ __forceinline__ void dot_to(double (&d)[2], double2 a, double2 b) { d[0] = fma(a.x, b.x, d[0]); d[1] = fma(a.y, b.y, d[1]); }
__device__ __forceinline__ void dot_to(double (&d)[2], double a, double b) { d[0] = fma(a, b, d[0]); }

// A column number.  Y has more than 2^32 rows only if they are short.
template <bool SHORT>
struct Columns { using type = uint32_t; };
template <>
struct Columns<true> { using type = unsigned long long; };

template <typename V, int G, int NI, int U, int UF, int MINB, bool LOOP>
__global__ void __launch_bounds__(SD_THREADS, MINB)
sddmm_kernel(int64_t nrows, int64_t nnz, int s, const int64_t *__restrict__ pos, const int64_t *__restrict__ crd,
             const double *__restrict__ sval, const double *__restrict__ x0, uint32_t ldx8, const double *__restrict__ y0,
             uint32_t ldy8, double *__restrict__ out, int kv, const int32_t *__restrict__ piece_row, int64_t npieces)
{
    using Col = typename Columns<(G * NI <= 8)>::type;
    const int lane = threadIdx.x & 31, g = lane / G, l = lane % G;
    const int64_t piece = ((int64_t)blockIdx.x * SD_THREADS + threadIdx.x) >> 5;
    const char *x = (const char *)((const V *)x0 + l), *y = (const char *)((const V *)y0 + l);
    bool on[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) on[i] = LOOP || l + i * G < kv;
    wait_for_previous();
    if (piece >= npieces) return;

    const int64_t p0 = piece << s;
    const int n = nnz - p0 < ((int64_t)1 << s) ? (int)(nnz - p0) : 1 << s;
    const int rlast = piece_row[piece + 1];            // no entry of the piece lies in a later row
    int w0 = piece_row[piece];                         // lane i holds the end of row w0 + i, counted from the piece's start
    int end;
    auto load_ends = [&]() {
        const int64_t e = w0 + lane < nrows ? pos[w0 + lane + 1] - p0 : n;
        end = e < n ? (int)e : n;
    };
    load_ends();
    crd += p0;
    sval += p0;
    out += p0;

    // columns, values and rows of the batch at e
    auto fetch = [&](int e, Col &c, double &v, int &row) {
        const int p = e + lane < n ? e + lane : n - 1;
        c = (Col)ld_stream(crd + p);
        v = ld_stream(sval + p);
        bool open = true;
        while (true) {
            int lo = 0;                                // ends at or before p
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
                if (__shfl_sync(0xffffffffu, end, lo + step - 1) <= p) lo += step;
            if (__shfl_sync(0xffffffffu, end, lo) <= p) lo++;
            if (open && lo < 32) {
                row = w0 + lo;
                open = false;
            }
            const unsigned left = __ballot_sync(0xffffffffu, open);
            if (!left) break;
            // the first row whose end lies behind the first entry without a row: 32 probes at a time where empty rows lie between
            const int64_t want = p0 + __shfl_sync(0xffffffffu, p, __ffs(left) - 1);
            int64_t a = (int64_t)w0 + 32, b = (int64_t)rlast + 1;
            while (b - a > 32) {
                const int64_t step = (b - a + 31) / 32, at = a + lane * step;
                const int k = __popc(__ballot_sync(0xffffffffu, at < b && pos[at < b ? at + 1 : a] <= want));
                if (k == 0) break;                     // row a itself
                b = a + k * step + 1 < b ? a + k * step + 1 : b;
                a += (k - 1) * step + 1;
            }
            w0 = (int)a;
            load_ends();
        }
    };

    Col cn;
    double vn;
    int rn, cur = -1;
    V xr[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) xr[i] = Vec<V>::zero();
    fetch(0, cn, vn, rn);
    for (int e = 0; e < n; e += 32) {
        const Col c = cn;
        const double v = vn;
        const int row = rn;
        if (e + 32 < n) fetch(e + 32, cn, vn, rn);
        const int m = n - e;
        double mine = 0.0;
        if (LOOP) {
            for (int t = 0; t < G; t++) {
                const int idx = g * G + t;
                const Col cc = __shfl_sync(0xffffffffu, c, idx);
                const int rr = __shfl_sync(0xffffffffu, row, idx);
                double d[2] = {0.0, 0.0};
                for (int k = 0; k < kv && idx < m; k += G * NI) {
                    V a[NI], b[NI];
#pragma unroll
                    for (int i = 0; i < NI; i++) {
                        const bool in = l + i * G + k < kv;
                        a[i] = in ? __ldg((const V *)(x + (uint64_t)(uint32_t)rr * ldx8) + i * G + k) : Vec<V>::zero();
                        b[i] = in ? __ldg((const V *)(y + (uint64_t)cc * ldy8) + i * G + k) : Vec<V>::zero();
                    }
#pragma unroll
                    for (int i = 0; i < NI; i++) dot_to(d, a[i], b[i]);
                }
                double sum = d[0] + d[1];
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if (l == t) mine = sum;
            }
        } else if (UF > 0 && __all_sync(0xffffffffu, row == __shfl_sync(0xffffffffu, row, 0))) {
            if (row != cur)
#pragma unroll
                for (int i = 0; i < NI; i++)
                    xr[i] = on[i] ? __ldg((const V *)(x + (uint64_t)(uint32_t)row * ldx8) + i * G) : Vec<V>::zero();
            cur = row;
            constexpr int UU = UF > 0 ? UF : 1;
#pragma unroll 1
            for (int t0 = 0; t0 < G; t0 += UU) {
                V yv[UU][NI];
#pragma unroll
                for (int u = 0; u < UU; u++) {
                    const int idx = g * G + t0 + u;
                    const Col cc = __shfl_sync(0xffffffffu, c, idx);
#pragma unroll
                    for (int i = 0; i < NI; i++)
                        yv[u][i] = on[i] && idx < m ? __ldg((const V *)(y + (uint64_t)cc * ldy8) + i * G) : Vec<V>::zero();
                }
#pragma unroll
                for (int u = 0; u < UU; u++) {
                    double d[2] = {0.0, 0.0};
#pragma unroll
                    for (int i = 0; i < NI; i++) dot_to(d, xr[i], yv[u][i]);
                    double sum = d[0] + d[1];
#pragma unroll
                    for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (l == t0 + u) mine = sum;
                }
            }
        } else {
#pragma unroll 1
            for (int t0 = 0; t0 < G; t0 += U) {
                V yv[U][NI], xv[U][NI];
                int rr[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int idx = g * G + t0 + u;
                    const Col cc = __shfl_sync(0xffffffffu, c, idx);
                    rr[u] = __shfl_sync(0xffffffffu, row, idx);
#pragma unroll
                    for (int i = 0; i < NI; i++)
                        yv[u][i] = on[i] && idx < m ? __ldg((const V *)(y + (uint64_t)cc * ldy8) + i * G) : Vec<V>::zero();
                    if (rr[u] != (u ? rr[u - 1] : cur))
#pragma unroll
                        for (int i = 0; i < NI; i++)
                            xv[u][i] = on[i] ? __ldg((const V *)(x + (uint64_t)(uint32_t)rr[u] * ldx8) + i * G) : Vec<V>::zero();
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    if (rr[u] != (u ? rr[u - 1] : cur))
#pragma unroll
                        for (int i = 0; i < NI; i++) xr[i] = xv[u][i];
                    double d[2] = {0.0, 0.0};
#pragma unroll
                    for (int i = 0; i < NI; i++) dot_to(d, xr[i], yv[u][i]);
                    double sum = d[0] + d[1];
#pragma unroll
                    for (int o = G / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (l == t0 + u) mine = sum;
                }
                cur = rr[U - 1];
            }
        }
        if (lane < m) out[e + lane] = v * mine;
    }
}

// Any size: one thread per row.  For operands beyond 32-bit row and column numbers or row offsets.
__global__ void __launch_bounds__(256)
sddmm_scalar_kernel(int64_t nrows, const int64_t *__restrict__ pos, const int64_t *__restrict__ crd,
                    const double *__restrict__ sval, const double *__restrict__ x, int64_t ldx,
                    const double *__restrict__ y, int64_t ldy, double *__restrict__ out, int64_t k)
{
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows;
         r += (int64_t)gridDim.x * blockDim.x) {
        for (int64_t p = pos[r]; p < pos[r + 1]; p++) {
            const double *xr = x + r * ldx, *yr = y + crd[p] * ldy;
            double t = 0.0;
            for (int64_t kk = 0; kk < k; kk++) t = fma(xr[kk], yr[kk], t);
            out[p] = sval[p] * t;
        }
    }
}

struct SddmmCall {
    int64_t nrows, nnz, k;
    const int64_t *pos, *crd;
    const double *sval, *x;
    int64_t ldx;
    const double *y;
    int64_t ldy;
    double *out;
    cudaStream_t st;
};

template <typename V, int G, int NI, int U, int UF, int MINB, bool LOOP>
static int launch_sddmm(const SddmmCall &a)
{
    const int64_t warps = (int64_t)sm_count() * 32;    // about what the registers let run at a time
    int s = 5;                                         // 2^5 to 2^8 entries a piece, the most that still give four rounds
    while (s < 8 && a.nnz >> (s + 1) >= warps * 4) s++;
    const int64_t npieces = ceil_div(a.nnz, (int64_t)1 << s), blocks = ceil_div(npieces, SD_THREADS / 32);
    if (blocks > 0x7fffffffLL) return fail("sddmm: too many entries");
    void *rows = nullptr;
    CB_TRY(scratch(SLOT_WORKLIST, (size_t)(npieces + 1) * sizeof(int32_t), &rows));
    int64_t grid = ceil_div(a.nrows, 256);
    if (grid > sm_count() * 8) grid = sm_count() * 8;
    sddmm_plan_kernel<<<(unsigned)grid, 256, 0, a.st>>>(a.nrows, s, npieces, a.pos, (int32_t *)rows);
    CB_LAUNCH_CHECK();
    CB_CUDA(launch_behind(sddmm_kernel<V, G, NI, U, UF, MINB, LOOP>, dim3((unsigned)blocks), SD_THREADS, 0, a.st, a.nrows, a.nnz, s, a.pos,
                          a.crd, a.sval, a.x, (uint32_t)(a.ldx * 8), a.y, (uint32_t)(a.ldy * 8), a.out,
                          (int)(a.k / Vec<V>::N), (const int32_t *)rows, npieces));
    return 0;
}

// G lanes x NI vectors just cover the columns; many vectors per lane and few lanes mean fewer shuffles per entry, as long as
// a group's loads still fill whole 128-byte lines.  U and UF (0: no path of its own for batches of one row) are entries in
// flight, MINB the CTAs per SM that the registers are limited for; taken from sweeps over R-MAT graphs of scale 14, 17 and
// 20, 400,000 rows of 8 and ragged rectangles.  Microseconds, R-MAT scale 20 / scale 14 / 400,000 rows of 8, with the lane
// group per 32 entries of short rows and chunk list for the others (even K) or the thread per row (odd K) before:
//   K = 4   331 28 66 -> 199 14 34    K = 16  ...  29 95 -> 334 15 82      K = 13  53290 1549 ... -> 372 15 80
//   K = 64  852 .. 320 -> 808 19 259  K = 128 1551 .. 589 -> 1406 25 535   K = 127 430553 11377 2469 -> 1846 27 625
template <typename V>
static int dispatch_sddmm(const SddmmCall &a)
{
    const int64_t kv = a.k / Vec<V>::N;
    constexpr bool pairs = Vec<V>::N == 2;
    if (kv <= 1) return launch_sddmm<V, 1, 2, 1, 0, 1, false>(a);
    if (kv <= 2) return launch_sddmm<V, 2, 1, 2, 2, 1, false>(a);
    if (kv <= 4) return launch_sddmm<V, 2, 2, 2, 0, 1, false>(a);
    if (kv <= 8) return pairs ? launch_sddmm<V, 4, 2, 1, 2, 4, false>(a) : launch_sddmm<V, 4, 2, 2, 2, 1, false>(a);
    if (kv <= (pairs ? 12 : 16)) return launch_sddmm<V, 4, 4, 1, 1, 1, false>(a);
    if (kv <= 16) return launch_sddmm<V, 8, 2, 1, 2, 4, false>(a);
    if (kv <= 32) return pairs ? launch_sddmm<V, 8, 4, 1, 1, 1, false>(a) : launch_sddmm<V, 8, 4, 2, 2, 4, false>(a);
    if (kv <= 48) return pairs ? launch_sddmm<V, 16, 3, 1, 1, 1, false>(a) : launch_sddmm<V, 16, 3, 2, 2, 4, false>(a);
    if (kv <= 64) return launch_sddmm<V, 16, 4, 1, 2, 3, false>(a);
    if (!pairs && kv <= 96) return launch_sddmm<V, 32, 3, 2, 2, 4, false>(a);
    if (kv <= 128) return pairs ? launch_sddmm<V, 32, 4, 2, 2, 1, false>(a) : launch_sddmm<V, 32, 4, 1, 2, 3, false>(a);
    if (kv <= 192) return launch_sddmm<V, 32, 6, 1, 1, 1, false>(a);
    if (kv <= 256) return launch_sddmm<V, 32, 8, 1, 1, 1, false>(a);
    return launch_sddmm<V, 32, 4, 1, 0, 1, true>(a);
}

int sddmm_csr(int64_t nrows, int64_t nnz, int64_t k, const int64_t *pos, const int64_t *crd,
              const double *sval, const double *x, int64_t ldx, const double *y, int64_t ldy,
              double *out, cudaStream_t st)
{
    if (nrows <= 0 || nnz <= 0) return 0;
    if (k <= 0 || k > (1 << 24) || nrows >= 0x7fffffe0LL || ldx >= (1LL << 29) || ldy >= (1LL << 29)) {
        int64_t blocks = ceil_div(nrows, 256);
        if (blocks > 0x7fffffffLL) blocks = 0x7fffffffLL;
        sddmm_scalar_kernel<<<(unsigned)blocks, 256, 0, st>>>(nrows, pos, crd, sval, x, ldx, y, ldy, out, k);
        CB_LAUNCH_CHECK();
        return 0;
    }
    const SddmmCall a = {nrows, nnz, k, pos, crd, sval, x, ldx, y, ldy, out, st};
    const bool vec = k % 2 == 0 && ldx % 2 == 0 && ldy % 2 == 0 && (((uintptr_t)x | (uintptr_t)y) & 15) == 0;
    return vec ? dispatch_sddmm<double2>(a) : dispatch_sddmm<double>(a);
}

}  // namespace cb200

extern "C" int32_t comet_b200_dev_sddmm_f64_i64(int64_t nrows, int64_t nnz, int64_t k,
                                                const int64_t *pos, const int64_t *crd,
                                                const double *sval, const double *x, int64_t ldx,
                                                const double *y, int64_t ldy, double *out,
                                                void *stream)
{
    cb200::clear_error();
    if (ldx < k || ldy < k) return cb200::fail("sddmm: leading dimension smaller than K");
    return cb200::sddmm_csr(nrows, nnz, k, pos, crd, sval, x, ldx, y, ldy, out, (cudaStream_t)stream);
}
