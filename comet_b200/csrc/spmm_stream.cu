// SpMM over the entry stream, rows of B staged in shared memory by asynchronous copies.
//
// Every warp owns a ring of shared-memory stages (G rows of B each) and a piece of
// the ENTRY stream of A: per stored entry its lanes issue 16-byte cp.async
// copies of B[crd, :] into the ring, several stages ahead of the stage being
// multiplied, so the gather runs ahead of the arithmetic without holding
// registers (the row panels of spmm.cu keep them in flight in registers, so
// that the bytes in flight follow occupancy).  (One bulk copy per row -- cp.async.bulk completing on an
// mbarrier -- was measured first and was slower: 1 KB per copy is too little
// work per copy instruction, 6.1 ms against 1.2 ms on R-MAT scale 20, K = 128.)
//
// Work is cut along the path that walks A row by row, one step per stored entry
// and one per row end, into equal pieces; persistent warps draw pieces from a
// counter.  A hub row is therefore shared by many warps and a run of empty rows
// by several, with no separate long-row pass.  A row that lies inside one piece
// is written with plain stores; a row cut by a boundary is added with f64
// atomics (onto zeros written by the plan kernel when the call does not
// accumulate), so its summation order is not fixed and differences stay at
// rounding level.  With 8-byte vectors (odd widths or addresses) the pieces
// leave their parts of such rows in scratch memory instead, where
// spmm_pieces.cu adds them up in order.
//
// Bound: the L2 -> SM rate (17 TB/s) for the gathered rows of B; the arrays alone would take 370 us of HBM time at R-MAT
// scale 20, K = 128, the gather 960 us.  That rate goes with the SM clock: calls with pauses between them take 1165 us at
// 1965 MHz, calls one after the other for seconds 1340, as the power cap (1000 W) then holds the clock at 1470 MHz.  Constant
// offsets in the ring, short pieces for small matrices (stream_plan) and a plan kernel with a thread per row instead of a search
// per piece: 111 -> 28 us at scale 14, at scale 20 no more than the runs of one side differ (1336 -> 1324 in long alternation).
#include "common.cuh"
#include "spmm.cuh"

namespace cb200 {

static const int SB_WARPS = 16;                // warps per CTA, one CTA per SM
static const int SB_RING_BYTES = 12 * 1024;    // per warp
static const int SB_SIDE_BYTES = 512;           // per warp: 32 column indices, 32 values of A, 32 row ends

// One copy of sizeof(V) bytes global -> shared.  16-byte ones bypass L1; operands with odd widths or addresses take 8.
template <typename V>
__device__ __forceinline__ void sb_copy(uint32_t dst, const void *src);
template <>
__device__ __forceinline__ void sb_copy<double2>(uint32_t dst, const void *src) { sb_copy16(dst, src); }
template <>
__device__ __forceinline__ void sb_copy<double>(uint32_t dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// NI vectors V per lane cover the columns; FULLK: exactly.  A row takes 32 NI vectors in the ring whether it fills them or
// not, so that every offset is a constant; a stage is four rows, two when rows are longer than 1 KB.
template <typename V, int NI>
struct StreamShape {
    static const int ROW = 32 * NI * (int)sizeof(V);
    static const int G = ROW <= 1024 ? 4 : 2;
    static const int STAGE = ROW * G;
    static const int STAGES = SB_RING_BYTES / STAGE;
    static const int RING = STAGE * STAGES;
    static const int WARP = RING + SB_SIDE_BYTES;
    static const bool FIXED = Vec<V>::N == 1;
};

template <typename V, int NI, bool FULLK>
__global__ void __launch_bounds__(SB_WARPS * 32, 1)
spmm_stream_kernel(int64_t nrows, unsigned nblocks, const int64_t *__restrict__ row_ids,
                   const int64_t *__restrict__ pos, const int64_t *__restrict__ crd, const double *__restrict__ val,
                   const double *__restrict__ b, int64_t ldb, double *__restrict__ c, int64_t ldc, int k,
                   int accumulate, WorkHeader *hdr, const int64_t *__restrict__ block_row,
                   const int64_t *__restrict__ block_ent, LongRows lr, double *__restrict__ parts)
{
    wait_for_previous();
    if (not_this(lr)) return;
    using S = StreamShape<V, NI>;
    constexpr int SB_G = S::G, stages = S::STAGES;
    constexpr bool FIXED = StreamShape<V, NI>::FIXED;
    constexpr uint32_t rowbytes = S::ROW, stagebytes = S::STAGE, ringbytes = S::RING;
    // per warp: a ring of `stages` stages of SB_G rows of B, then 32 column indices and 32 values of A
    extern __shared__ __align__(128) unsigned char sb_smem_raw[];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int kv = FULLK ? NI * 32 : k / Vec<V>::N;     // vectors per row
    unsigned char *ring = sb_smem_raw + (size_t)warp * S::WARP;
    int32_t *cs = (int32_t *)(ring + S::RING);
    double *vs = (double *)(cs + 32);
    int *ps = (int *)(vs + 32);                         // block-local end positions of 32 consecutive rows
    const uint32_t ring_s = sb_smem(ring) + (uint32_t)lane * (uint32_t)sizeof(V);
    const char *bl = (const char *)b + lane * sizeof(V);
    const int64_t ldb8 = ldb * 8;
    bool on[NI];
#pragma unroll
    for (int i = 0; i < NI; i++) on[i] = FULLK || (lane + i * 32 < kv);

    uint32_t pofs = 0;               // byte offset of the stage the next issue fills
    uint32_t cofs = 0;               // byte offset of the stage the next wait reads

    while (true) {
        unsigned blk = 0;
        if (lane == 0) blk = atomicAdd(&hdr->pad[0], 1u);
        blk = __shfl_sync(0xffffffffu, blk, 0);
        if (blk >= nblocks) break;
        const int64_t n0 = block_ent[blk];
        const int cnt = (int)(block_ent[blk + 1] - n0);
        const int64_t rend = block_row[blk + 1];        // rows before rend end in this block
        const int ngroups = (cnt + SB_G - 1) / SB_G;
        const int64_t *crd0 = crd + n0;
        const double *val0 = val + n0;

        // rows: r is the row of the entry being consumed; its entries are [rs, re) in block-local positions
        int64_t r = block_row[blk];
        const int64_t far = (int64_t)cnt + 1;
        const int64_t d = pos[r] - n0;
        int rs = d < -1 ? -1 : (int)d;                  // -1: the row starts before the block
        int64_t rb = r;                                 // ps[i] = end of row rb + i; cnt + 1: it ends after the block
        auto load_ends = [&]() {
            __syncwarp();
            int64_t e = far;
            if (rb + lane < nrows) {
                e = pos[rb + lane + 1] - n0;
                if (e > far) e = far;
            }
            ps[lane] = (int)e;
            __syncwarp();
        };
        load_ends();
        int re = ps[0];

        int32_t cnext = (lane < cnt) ? (int32_t)ld_stream(crd0 + lane) : 0;
        double vnext = (lane < cnt) ? ld_stream(val0 + lane) : 0.0;

        V acc[NI];
#pragma unroll
        for (int i = 0; i < NI; i++) acc[i] = Vec<V>::zero();

        // write out the finished row r and clear the accumulators
        auto flush = [&](bool whole) {
            const int64_t out = row_ids ? row_ids[r] : r;
            double *crow = FIXED && !whole ? parts + (2 * (int64_t)blk + (rs >= 0 ? 1 : 0)) * k : c + out * ldc;
            if (whole && accumulate && rs == re) return;       // an empty row adds nothing
#pragma unroll
            for (int i = 0; i < NI; i++) {
                V *at = (V *)crow + lane + i * 32;
                if (on[i]) {
                    if (!whole && FIXED) *at = acc[i];
                    else if (!whole) Vec<V>::atomic_to(at, acc[i]);
                    else {
                        if (accumulate) Vec<V>::add_to(acc[i], __ldcs(at));
                        __stcs(at, acc[i]);
                    }
                }
                acc[i] = Vec<V>::zero();
            }
        };
        auto next_row = [&]() {
            flush(rs >= 0);
            r += 1;
            rs = re;
            if (r - rb == 32) {
                rb = r;
                load_ends();
            }
            re = ps[r - rb];
        };

        // every call commits one copy group (an empty one past the end of the block), so "all but
        // stages-1 groups have landed" always means the stage about to be read has landed
        auto issue = [&](int g) {
            if (g < ngroups) {
                const int off = (g * SB_G) & 31;
                if (off == 0) {
                    cs[lane] = cnext;
                    const int nb = g * SB_G + 32 + lane;
                    cnext = (nb < cnt) ? (int32_t)ld_stream(crd0 + nb) : 0;
                    __syncwarp();
                }
                int cc[SB_G];                                       // broadcast read of the column indices
                if (SB_G == 4) {
                    const int4 c4 = *(const int4 *)(cs + off);
                    cc[0] = c4.x; cc[1] = c4.y; cc[SB_G - 2] = c4.z; cc[SB_G - 1] = c4.w;
                } else {
                    const int2 c2 = *(const int2 *)(cs + off);
                    cc[0] = c2.x; cc[1] = c2.y;
                }
                const uint32_t dst = ring_s + pofs;
                const int m = cnt - g * SB_G;
                if (m >= SB_G) {
#pragma unroll
                    for (int t = 0; t < SB_G; t++) {
                        const char *src = bl + (int64_t)cc[t] * ldb8;
#pragma unroll
                        for (int i = 0; i < NI; i++)
                            if (on[i]) sb_copy<V>(dst + (uint32_t)t * rowbytes + (uint32_t)(i * 32 * (int)sizeof(V)), src + i * 32 * (int)sizeof(V));
                    }
                } else {
#pragma unroll
                    for (int t = 0; t < SB_G; t++) {
                        if (t < m) {
                            const char *src = bl + (int64_t)cc[t] * ldb8;
#pragma unroll
                            for (int i = 0; i < NI; i++)
                                if (on[i]) sb_copy<V>(dst + (uint32_t)t * rowbytes + (uint32_t)(i * 32 * (int)sizeof(V)), src + i * 32 * (int)sizeof(V));
                        }
                    }
                }
                pofs += stagebytes;
                if (pofs == ringbytes) pofs = 0;
            }
            sb_commit();
        };

        for (int g = 0; g < stages - 1; g++) issue(g);

        for (int g = 0; g < ngroups; g++) {
            const int off = (g * SB_G) & 31;
            if (off == 0) {
                vs[lane] = vnext;
                const int nb = g * SB_G + 32 + lane;
                vnext = (nb < cnt) ? ld_stream(val0 + nb) : 0.0;
            }
            issue(g + stages - 1);
            sb_wait<stages - 1>();
            __syncwarp();                               // the other lanes' copies of this stage have landed too
            const V *src = (const V *)(ring + cofs) + lane;
            V bv[SB_G][NI];
#pragma unroll
            for (int t = 0; t < SB_G; t++)
#pragma unroll
                for (int i = 0; i < NI; i++) bv[t][i] = on[i] ? src[(t * NI + i) * 32] : Vec<V>::zero();
            double vv[SB_G];
#pragma unroll
            for (int t = 0; t < SB_G; t += 2) {
                const double2 v2 = *(const double2 *)(vs + off + t);
                vv[t] = v2.x; vv[t + 1] = v2.y;
            }
            const int j0 = g * SB_G;
            if (j0 + SB_G <= re && j0 + SB_G <= cnt) {  // the four entries belong to the row in progress
#pragma unroll
                for (int t = 0; t < SB_G; t++)
#pragma unroll
                    for (int i = 0; i < NI; i++) Vec<V>::fma_to(acc[i], vv[t], bv[t][i]);
            } else {
#pragma unroll
                for (int t = 0; t < SB_G; t++) {
                    if (j0 + t < cnt) {
                        while (j0 + t >= re) next_row();
#pragma unroll
                        for (int i = 0; i < NI; i++) Vec<V>::fma_to(acc[i], vv[t], bv[t][i]);
                    }
                }
            }
            cofs += stagebytes;
            if (cofs == ringbytes) cofs = 0;
            __syncwarp();                               // every lane has read the stage before it is refilled
        }

        // rows that end in this block (the one in progress, empty ones after it), then the part of
        // row rend this block holds, if the boundary cuts that row
        while (r < rend) next_row();
        if (rend < nrows && n0 + cnt > pos[rend]) flush(false);
    }
}

template <typename V, int NI, bool FULLK>
static int launch_stream(const SpmmCall &a, LongRows lr)
{
    constexpr bool FIXED = StreamShape<V, NI>::FIXED;
    StreamPlan plan;
    const int planned = stream_plan(a.nrows, a.nnz, (int64_t)sm_count() * SB_WARPS, FIXED ? PARTS_BYTES / (16 * a.k) : INT64_MAX,
                                    a.row_ids, a.pos, FIXED ? nullptr : a.c, a.ldc, a.k, a.accumulate, lr, a.st, &plan);
    if (planned <= 0) return planned;
    double *parts = nullptr;
    if (FIXED && piece_parts(plan.nblocks, a.k, &parts)) return -1;
    auto kernel = spmm_stream_kernel<V, NI, FULLK>;
    const size_t smem = (size_t)SB_WARPS * StreamShape<V, NI>::WARP;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        fail("spmm: shared memory size refused");
        return -1;
    }
    int64_t grid = ceil_div(plan.nblocks, SB_WARPS);
    if (grid > sm_count()) grid = sm_count();
    const cudaError_t e = launch_behind(kernel, dim3((unsigned)grid), SB_WARPS * 32, smem, a.st, a.nrows, (unsigned)plan.nblocks,
                                        a.row_ids, a.pos, a.crd, a.val, a.b, a.ldb, a.c, a.ldc, (int)a.k, a.accumulate,
                                        plan.hdr, plan.block_row, plan.block_ent, lr, parts);
    if (e != cudaSuccess) {
        fail("spmm: launch failed: %s", cudaGetErrorString(e));
        return -1;
    }
    if (FIXED && add_parts(a, plan, lr, parts)) return -1;
    return 1;
}

int spmm_stream(const SpmmCall &a, LongRows lr)
{
    if (a.k < 1 || a.k > 256 || a.nnz < 1 || a.nrows <= 0 || a.ncols > 0x7fffffffLL) return 0;    // columns travel as int32
    if (a.vec) {
        if (a.k == 64) return launch_stream<double2, 1, true>(a, lr);
        if (a.k < 64) return launch_stream<double2, 1, false>(a, lr);
        if (a.k == 128) return launch_stream<double2, 2, true>(a, lr);
        if (a.k < 128) return launch_stream<double2, 2, false>(a, lr);
        if (a.k <= 192) return launch_stream<double2, 3, false>(a, lr);
        if (a.k == 256) return launch_stream<double2, 4, true>(a, lr);
        return launch_stream<double2, 4, false>(a, lr);
    }
    if (a.k <= 64) return launch_stream<double, 2, false>(a, lr);
    if (a.k <= 96) return launch_stream<double, 3, false>(a, lr);
    if (a.k <= 128) return launch_stream<double, 4, false>(a, lr);
    if (a.k <= 192) return launch_stream<double, 6, false>(a, lr);
    return launch_stream<double, 8, false>(a, lr);
}

}  // namespace cb200
