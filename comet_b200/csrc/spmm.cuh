// The automatic SpMM: a call's operands, and the kernels that take it.
#pragma once
#include "common.cuh"
#include "stream.cuh"

namespace cb200 {

// Fewer entries: the launches themselves are what a call takes.
static const int64_t SPMM_SMALL_NNZ = 65536;
// Most memory for the parts of rows that are cut (2 k doubles a piece); more entries than this allows get longer pieces.
static const int64_t PARTS_BYTES = (int64_t)128 << 20;

struct SpmmCall {
    int64_t nrows, ncols, nnz, k;
    const int64_t *row_ids, *pos, *crd;
    const double *val, *b;
    int64_t ldb;
    double *c;
    int64_t ldc;
    bool pair;
    bool vec;                 // K, both leading dimensions and both addresses allow 16-byte accesses
    int accumulate;
    cudaStream_t st;
};

// Takes the call if no row is long, which only the device knows; `lr` is for the kernels that take it otherwise (spmm_short.cu).
int spmm_short_rows(const SpmmCall &a, LongRows *lr);
// Equal pieces of A's path, a group of lanes each; any K and alignment (spmm_pieces.cu).
int spmm_pieces(const SpmmCall &a, LongRows lr);
// Scratch memory for the parts of the rows that pieces cut, two rows of k sums a piece: [0] of a row that started before it,
// [1] of one that starts in it and goes on; and the kernel that adds them up, in order.
int piece_parts(int64_t npieces, int64_t k, double **parts);
int add_parts(const SpmmCall &a, const StreamPlan &plan, LongRows lr, const double *parts);
// Rows of B staged in shared memory (spmm_stream.cu).  Returns 1 when it took the call, 0 when the shape is not one that
// it handles, -1 on error.
int spmm_stream(const SpmmCall &a, LongRows lr);

}  // namespace cb200
