// A host call that returns an error has stopped writing to its caller's arrays: the arrays go back to their owner, who
// may use or free them at once.
//
//   download_errors_check <pinned|pageable> <copy|sync> <n>
//
// runs comet_b200_host_coo_to_csr (three downloads) with the n-th copy to the host, or the n-th synchronisation of the
// stream, failing, and watches the result arrays after it has returned.
#include "fake_cuda.hpp"

#include <vector>

#include "../../include/comet_b200.h"

extern "C" int32_t comet_b200_dev_coo_to_csr_f64_i64(int64_t nrows, int64_t, int64_t nnz, const int64_t *, const int64_t *,
                                                     const double *, int64_t *pos, int64_t *crd, double *val, void *stream)
{
    cudaMemsetAsync(pos, 0x5a, (size_t)(nrows + 1) * 8, (cudaStream_t)stream);
    cudaMemsetAsync(crd, 0x5a, (size_t)nnz * 8, (cudaStream_t)stream);
    cudaMemsetAsync(val, 0x5a, (size_t)nnz * 8, (cudaStream_t)stream);
    return 0;
}

int main(int argc, char **argv)
{
    if (argc != 4) return 2;
    const bool page_locked = strcmp(argv[1], "pinned") == 0;
    const int64_t nrows = 40000, nnz = 500000;          // 4 MB an array: three staged pieces
    std::vector<int64_t> rows(nnz, 0), cols(nnz, 0);
    std::vector<double> vals(nnz, 0.0);
    char *out[3];
    const size_t bytes[3] = {(size_t)(nrows + 1) * 8, (size_t)nnz * 8, (size_t)nnz * 8};
    for (int i = 0; i < 3; i++) {
        if (page_locked) cudaHostAlloc((void **)&out[i], bytes[i], 0);
        else out[i] = (char *)malloc(bytes[i]);
        memset(out[i], 0, bytes[i]);
    }
    (strcmp(argv[2], "copy") == 0 ? fake::fail_download : fake::fail_sync) = atoi(argv[3]);
    const int rc = comet_b200_host_coo_to_csr(nrows, nrows, nnz, rows.data(), cols.data(), vals.data(), (int64_t *)out[0],
                                              (int64_t *)out[1], (double *)out[2]);
    std::vector<char> seen[3];
    for (int i = 0; i < 3; i++) seen[i].assign(out[i], out[i] + bytes[i]);
    std::this_thread::sleep_for(std::chrono::milliseconds(30 * fake::DELAY_MS));
    for (int i = 0; i < 3; i++)
        if (memcmp(seen[i].data(), out[i], bytes[i])) {
            printf("array %d was written after the call had returned %d\n", i, rc);
            return 1;
        }
    printf("returned %d\n", rc);
    fflush(stdout);
    _Exit(0);                                           // the streams' threads go with the process
}
