// Shared by the entry-stream kernels (SpMM, SDDMM): asynchronous 16-byte copies into shared memory and the
// plan that cuts a CSR matrix into equal pieces of its (entries + rows) path.
#pragma once
#include "common.cuh"

namespace cb200 {

// Whether a matrix has long rows is found out on the device (spmm_short.cu): the word holds the call's number if it has.
// A kernel for matrices with long rows returns at once if it has not; flag == null: it takes every matrix.
struct LongRows {
    const int64_t *flag;
    int64_t call;
};
#ifdef __CUDACC__
__device__ __forceinline__ bool not_this(const LongRows &lr) { return lr.flag && *lr.flag != lr.call; }

// The kernels of one call are launched behind each other with their start-up overlapping the end of the one before
// (programmatic dependent launch): a kernel that finds nothing to do then costs 1 us instead of 2.5.  Each of them waits for
// the whole of the one before it before it touches memory, so the order is that of plain launches.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_behind(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif

struct StreamPlan {
    WorkHeader *hdr;          // hdr->pad[0]: counter the persistent warps draw pieces from
    int64_t *block_row;       // piece b starts in row block_row[b] ...
    int64_t *block_ent;       // ... at entry block_ent[b]; both have nblocks + 1 entries
    int64_t nblocks;
    int s;                    // a piece has 2^s steps
};

// Cuts the (entries + rows) path into pieces of 2^s steps (spmm_pieces.cu) and clears the counter.  c != null and
// accumulate == 0: rows cut by a boundary get zeros (k columns).  The plan lives in the device's work-list slot.
int piece_plan(int64_t nrows, int64_t nnz, int s, const int64_t *row_ids, const int64_t *pos, double *c, int64_t ldc,
               int64_t k, int accumulate, LongRows lr, cudaStream_t st, StreamPlan *out);
// A word for a call's mark and the call's number (spmm_short.cu); flag == null on error.
LongRows next_mark();
// Marks the call if a row has more than `limit` entries.
int mark_long_rows(int64_t nrows, const int64_t *pos, int64_t limit, LongRows lr, cudaStream_t st);
// Pieces for `warps` persistent warps, fewer than `most`.  Returns 1, 0 when the piece count does not fit 32 bits, -1 on error.
int stream_plan(int64_t nrows, int64_t nnz, int64_t warps, int64_t most, const int64_t *row_ids, const int64_t *pos, double *c,
                int64_t ldc, int64_t k, int accumulate, LongRows lr, cudaStream_t st, StreamPlan *out);

#ifdef __CUDACC__
// A row of B or C as vectors: two columns at a time where widths and addresses allow it, one otherwise.
template <typename V>
struct Vec;
template <>
struct Vec<double2> {
    static const int N = 2;
    static __device__ __forceinline__ double2 zero() { return make_double2(0.0, 0.0); }
    static __device__ __forceinline__ void fma_to(double2 &a, double v, double2 b) { a.x = fma(v, b.x, a.x); a.y = fma(v, b.y, a.y); }
    static __device__ __forceinline__ void add_to(double2 &a, double2 b) { a.x += b.x; a.y += b.y; }
    static __device__ __forceinline__ void atomic_to(double2 *p, double2 a) { atomicAdd(&p->x, a.x); atomicAdd(&p->y, a.y); }
    static __device__ __forceinline__ double2 ones(double v) { return make_double2(v, v); }
};
template <>
struct Vec<double> {
    static const int N = 1;
    static __device__ __forceinline__ double zero() { return 0.0; }
    static __device__ __forceinline__ void fma_to(double &a, double v, double b) { a = fma(v, b, a); }
    static __device__ __forceinline__ void add_to(double &a, double b) { a += b; }
    static __device__ __forceinline__ void atomic_to(double *p, double a) { atomicAdd(p, a); }
    static __device__ __forceinline__ double ones(double v) { return v; }
};

// wait until at most N of this thread's copy groups are still in flight
template <int N>
__device__ __forceinline__ void sb_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ uint32_t sb_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16 bytes global -> shared without passing through registers or L1
__device__ __forceinline__ void sb_copy16(uint32_t dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void sb_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
#endif

}  // namespace cb200
