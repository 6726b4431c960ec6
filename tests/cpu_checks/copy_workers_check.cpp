// Operands of a few MB are copied by the thread that makes the call, large ones by workers too.
#include "fake_cuda.hpp"

#include <vector>

#include "../../comet_b200/csrc/hostcopy.cuh"

// uploads two arrays of `bytes` side by side and one back; returns how many threads copied
static size_t threads_for(size_t bytes)
{
    cudaStream_t st = cb200::lib_stream();
    std::vector<char> a(bytes, 1), b(bytes, 2), back(bytes, 0), da(bytes), db(bytes);
    {
        std::lock_guard<std::mutex> lk(fake::pinned_mu);
        fake::copiers.clear();
    }
    int rc = !cb200::uploads_begin();
    rc |= cb200::h2d(da.data(), a.data(), bytes, st) | cb200::h2d(db.data(), b.data(), bytes, st) | cb200::uploads_join();
    rc |= cb200::d2h(back.data(), db.data(), bytes, st);
    cudaStreamSynchronize(st);
    rc |= cb200::copies_drain();
    if (rc || da != a || db != b || back != b) return 0;
    std::lock_guard<std::mutex> lk(fake::pinned_mu);
    return fake::copiers.size();
}

int main()
{
    setenv("COMET_B200_COPY_THREADS", "4", 1);
    const size_t small = threads_for((size_t)3 << 20), large = threads_for((size_t)40 << 20);
    printf("%zu %s\n", small, large > 2 ? "several" : "few");
    fflush(stdout);
    _Exit(0);
}
