// SpMM for matrices without long rows: a few threads per row, every row finished by them.
//
// tp = ceil(kv / NI) consecutive threads take a row of kv vectors, whatever K is, so a CTA works on 256 / tp rows at a time
// and few of its lanes idle.  Each thread reads the row's entries itself (one address for all threads of a row: one access
// of a warp for each row that it holds) instead of getting them by shuffles, and keeps U entries' rows of B in flight, NI
// vectors of each, with the next U entries loaded meanwhile.
//
// Bound: the L1's rate of line accesses (every load of a warp touches the lines of each row that the warp holds) and the
// latency of the chain row pointer -> entry -> row of B.  Both fall with more vectors per thread, as long as the rows still
// fill the chip; dispatch_short has the split, and what it was chosen from.
//
// Whether a matrix has long rows is seen on the device: a first kernel reads the row pointer and marks the call, and the
// kernels for the two kinds of matrices return at once when the mark is not theirs (about 1 us each).
#include <atomic>

#include "common.cuh"
#include "spmm.cuh"

namespace cb200 {

static const int SHORT_THREADS = 256;
static const int SHORT_CTAS = 4;                       // resident per SM: 64 registers a thread
static const int SHORT_SLICE = 512;                    // columns per pass over A: 128 threads a row at most

__global__ void __launch_bounds__(256)
spmm_long_rows_kernel(int64_t nrows, const int64_t *__restrict__ pos, int64_t limit, int64_t *flag, int64_t call)
{
    let_next_start();
    bool any = false;
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * blockDim.x)
        any |= pos[r + 1] - pos[r] > limit;
    if (__syncthreads_or(any) && threadIdx.x == 0) *flag = call;       // 50,000 stores to one address took 100 us
}

template <typename V, int NI, int U, bool PAIR>
__global__ void __launch_bounds__(SHORT_THREADS, SHORT_CTAS)
spmm_short_rows_kernel(int64_t nrows, const int64_t *__restrict__ row_ids, const int64_t *__restrict__ pos,
                       const int64_t *__restrict__ crd, const double *__restrict__ val, const double *__restrict__ b0,
                       uint32_t ldb8, double *__restrict__ c0, int64_t ldc, int64_t k, int accumulate, LongRows lr)
{
    wait_for_previous();
    if (*lr.flag == lr.call) return;
    const int64_t col0 = (int64_t)blockIdx.y * SHORT_SLICE;
    const int kv = (int)(k - col0 < SHORT_SLICE ? k - col0 : SHORT_SLICE) / Vec<V>::N;
    const int tp = (kv + NI - 1) / NI, per = SHORT_THREADS / tp;
    const int g = threadIdx.x / tp, l = threadIdx.x - g * tp;
    if (g >= per) return;
    const char *b = (const char *)((const V *)(b0 + col0) + l);
    bool on[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) on[i] = i == 0 || l + i * tp < kv;
    const int64_t stride = (int64_t)gridDim.x * per;
    for (int64_t r = (int64_t)blockIdx.x * per + g; r < nrows; r += stride) {
        const int64_t s = pos[r];
        const int n = (int)(pos[r + 1] - s);
        const int64_t *cp = crd + s;
        const double *vp = val + s;
        V acc[NI];
#pragma unroll
        for (int i = 0; i < NI; i++) acc[i] = Vec<V>::zero();
        uint32_t col[U];
        double v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            col[u] = u < n ? (uint32_t)__ldg(cp + u) : 0;
            v[u] = u < n && !PAIR ? __ldg(vp + u) : 1.0;
        }
        for (int p = 0; p < n; p += U) {
            V x[U][NI];
#pragma unroll
            for (int u = 0; u < U; u++)
#pragma unroll
                for (int i = 0; i < NI; i++)
                    x[u][i] = p + u >= n || !on[i] ? Vec<V>::zero()
                              : PAIR               ? Vec<V>::ones(1.0)
                                                   : __ldg((const V *)(b + (uint64_t)col[u] * ldb8) + i * tp);
            double w[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                w[u] = v[u];
                if (p + U + u < n) {
                    col[u] = (uint32_t)__ldg(cp + p + U + u);
                    if (!PAIR) v[u] = __ldg(vp + p + U + u);
                }
            }
#pragma unroll
            for (int u = 0; u < U; u++)
                if (p + u < n)
#pragma unroll
                    for (int i = 0; i < NI; i++) Vec<V>::fma_to(acc[i], w[u], x[u][i]);
        }
        if (accumulate && n == 0) continue;
        V *at = (V *)(c0 + col0 + (row_ids ? row_ids[r] : r) * ldc) + l;
#pragma unroll
        for (int i = 0; i < NI; i++)
            if (on[i]) {
                if (accumulate) Vec<V>::add_to(acc[i], __ldcs(at + i * tp));
                __stcs(at + i * tp, acc[i]);           // written once, not read again here
            }
    }
}

// A call marks the word with its own number, so the word need not be cleared.  What an earlier use left there can only
// be equal by chance, and then the kernels that take every matrix do the work.
LongRows next_mark()
{
    static std::atomic<int64_t> calls{1};
    void *flag = nullptr;
    if (scratch(SLOT_FLAG, sizeof(int64_t), &flag)) return {nullptr, 0};
    return {(const int64_t *)flag, calls.fetch_add(1) * 0x9e3779b97f4a7c1 + 0x5bd1e995};
}

int mark_long_rows(int64_t nrows, const int64_t *pos, int64_t limit, LongRows lr, cudaStream_t st)
{
    int64_t grid = ceil_div(nrows, 256);
    if (grid > sm_count() * 8) grid = sm_count() * 8;
    spmm_long_rows_kernel<<<(unsigned)grid, 256, 0, st>>>(nrows, pos, limit, (int64_t *)lr.flag, lr.call);
    CB_LAUNCH_CHECK();
    return 0;
}

template <typename V, int NI, int U, bool PAIR>
static int launch_short(const SpmmCall &a, LongRows *lr)
{
    const int64_t kv = (a.k < SHORT_SLICE ? a.k : SHORT_SLICE) / Vec<V>::N, tp = ceil_div(kv, NI);
    const int64_t resident = (int64_t)sm_count() * SHORT_CTAS * SHORT_THREADS;
    // Rows are short when none is far above the mean (the threads of a warp wait for its longest row) and when none takes
    // much longer than the threads' share of all the work, 128 entries (about 15 us) being always all right.
    int64_t limit = a.nnz * tp * 2 / resident;
    if (limit < 128) limit = 128;
    if (limit > a.nnz / a.nrows * 3 + 16) limit = a.nnz / a.nrows * 3 + 16;
    if (limit > 0x7ffffff0) limit = 0x7ffffff0;        // a row's entries are counted in 32 bits
    *lr = next_mark();
    if (!lr->flag) return -1;
    CB_TRY(mark_long_rows(a.nrows, a.pos, limit, *lr, a.st));
    int64_t blocks = ceil_div(a.nrows, SHORT_THREADS / tp);
    if (blocks > resident / SHORT_THREADS) blocks = resident / SHORT_THREADS;
    const dim3 grid((unsigned)blocks, (unsigned)ceil_div(a.k, SHORT_SLICE));
    CB_CUDA(launch_behind(spmm_short_rows_kernel<V, NI, U, PAIR>, grid, SHORT_THREADS, 0, a.st, a.nrows, a.row_ids, a.pos, a.crd,
                          a.val, a.b, (uint32_t)(a.ldb * 8), a.c, a.ldc, a.k, a.accumulate, *lr));
    return 0;
}

// Vectors per thread NI, entries in flight U.  Microseconds of the row kernel with (1, 4), (2, 2) [odd K: (2, 4)] and (4, 1)
// [odd K: (4, 2)] on 50,021 rows of 0 to 24 entries and on 400,000 rows of 8:
//   K = 8   10.4 11.5 16.4    33  41  49      odd 13   18.6 16.8 18.6    82  64  62
//   K = 16  14.5 14.5 18.6    58  51  57      odd 33   39   31   29     259 152 127
//   K = 48  33   25   29     195 164 156      odd 65   66   52   45     554 328 255
//   K = 96  53   41   41     396 355 344      odd 127 105   75   64    1030 621 516
//   K = 256 128  91   84    1089 1015 996
template <typename V>
static int dispatch_short(const SpmmCall &a, LongRows *lr)
{
    const int64_t kv = a.k / Vec<V>::N;
    if (a.pair) return kv <= 64 ? launch_short<V, 1, 4, true>(a, lr) : launch_short<V, 4, 1, true>(a, lr);   // no rows of B are read
    if (Vec<V>::N == 2) {
        if (kv <= 8) return launch_short<V, 1, 4, false>(a, lr);
        if (kv < 48) return launch_short<V, 2, 2, false>(a, lr);
        return launch_short<V, 4, 1, false>(a, lr);
    }
    if (kv <= 4) return launch_short<V, 1, 4, false>(a, lr);
    if (kv < 24) return launch_short<V, 2, 4, false>(a, lr);
    return launch_short<V, 4, 2, false>(a, lr);
}

int spmm_short_rows(const SpmmCall &a, LongRows *lr)
{
    return a.vec ? dispatch_short<double2>(a, lr) : dispatch_short<double>(a, lr);
}

}  // namespace cb200
