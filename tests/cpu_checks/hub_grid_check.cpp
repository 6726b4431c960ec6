// The kernel that looks A and B over before a product with long rows walks both of them: a tall A times a small B must not be walked by
// the few blocks that B alone would get.
#include "fake_launch.hpp"

#include "../../comet_b200/csrc/hostcopy.cuh"

namespace cb200 {
PinnedWords::PinnedWords() { p = calloc(64, 1); }
PinnedWords::~PinnedWords() { free(p); }
int scratch(Slot, size_t bytes, void **ptr) { *ptr = malloc(bytes); return 0; }
int exclusive_scan_i64(const int64_t *, int64_t *, int64_t, cudaStream_t) { return 0; }
}  // namespace cb200

int main(int argc, char **argv)
{
    const int64_t nrows = atoll(argv[1]), nnz_a = atoll(argv[2]), nnz_b = atoll(argv[3]), ncols = atoll(argv[4]);
    std::vector<int64_t> apos((size_t)nrows + 1, 0), bcrd((size_t)nnz_b + 2, 0), cpos((size_t)nrows + 1, 0);
    apos[(size_t)nrows] = nnz_a;
    fake::on_launch = [&](const std::string &name, void **args) {
        if (name.find("publish_kernel") != std::string::npos) {        // every row is one of the long ones
            unsigned *host = *(unsigned **)args[2];
            const int64_t *n = *(const int64_t **)args[1];
            host[1] = (unsigned)nrows;
            if (n) *(int64_t *)(host + 4) = *n;
        }
    };
    int64_t nnz = 0, handle = 0;
    if (comet_b200_dev_spgemm_symbolic_f64_i64(nrows, ncols, nnz_b, apos.data(), nullptr, nullptr, apos.data(), bcrd.data(), nullptr, nullptr,
                                               nullptr, COMET_B200_PLUS_TIMES, cpos.data(), &nnz, &handle, nullptr)) {
        printf("%s\n", cb200::g_err);
        return 1;
    }
    unsigned grid = 0;
    for (auto &l : fake::launches)
        if (l.name.find("hub_present_kernel") != std::string::npos) grid = l.grid.x;
    printf("%u\n", grid);
    return 0;
}
