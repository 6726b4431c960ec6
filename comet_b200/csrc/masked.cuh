// Masked sparse product through dot products (masked.cu), used by the sparse product's symbolic and numeric calls.
#pragma once
#include "common.cuh"

namespace cb200 {

struct MaskedPlan;

// Fills the row pointer of C<M,push> = A * B, cpos[nrows + 1].  *plan stays null when the operands are
// not ones for this form (then nothing was written).  Synchronises the stream once.
int masked_symbolic(int64_t nrows, int64_t ncols_b, int64_t nnz_b, const int64_t *apos, const int64_t *acrd, const int64_t *bpos,
                    const int64_t *bcrd, const int64_t *mpos, const int64_t *mcrd, int64_t *cpos, MaskedPlan **plan,
                    cudaStream_t st);
// Three device integers to be read with the next synchronisation: the plan is good when the first is 0 and the others agree.
const int *masked_checks(const MaskedPlan *plan);
int masked_numeric(MaskedPlan *plan, const double *aval, const double *bval, const int64_t *mcrd, int semi, int64_t *ccrd,
                   double *cval, cudaStream_t st);
void masked_free(MaskedPlan *plan, cudaStream_t st);

}  // namespace cb200
