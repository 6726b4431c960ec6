// Intersections of lists with the sets that a warp builds in shared memory: sets that the cuckoo tables hold, and sets that they do not.
#include "fake_warp.hpp"

#include <comet_b200.h>

inline double __longlong_as_double(long long v) { return fake::from_bits<double>((unsigned long long)v); }
inline long long __double_as_longlong(double v) { return (long long)fake::bits_of(v); }
#include "kernels.inc"
using namespace cb200;

struct Matrix {
    std::vector<int64_t> pos = {0};
    std::vector<int32_t> crd;
    void row(std::vector<int32_t> r)
    {
        std::sort(r.begin(), r.end());
        crd.insert(crd.end(), r.begin(), r.end());
        pos.push_back((int64_t)crd.size());
    }
    int64_t rows() const { return (int64_t)pos.size() - 1; }
};

template <int LOG2>
static std::vector<int32_t> meeting(int n)         // columns that share both of their slots
{
    std::vector<int32_t> c;
    for (int32_t j = 0; (int)c.size() < n; j++)
        if (tc_h0<LOG2>(j) == tc_h0<LOG2>(1) && tc_h1<LOG2>(j) == tc_h1<LOG2>(1)) c.push_back(j);
    return c;
}

int main(int argc, char **argv)
{
    const bool mid = argc > 1 && !strcmp(argv[1], "mid");
    const char *what = argc > 2 ? argv[2] : "all";
    const int longest = mid ? TC_MID_MAX : TC_WARP_MAX, cols = 3000;
    Matrix A, B, M;
    uint32_t seed = 1;
    auto draw = [&](int n) { return (int32_t)((seed = seed * 1664525u + 1013904223u) >> 8) % n; };
    auto some = [&](int n, int below) {
        std::vector<bool> in(below, false);
        std::vector<int32_t> r;
        while ((int)r.size() < n) {
            const int32_t j = draw(below);
            if (!in[j]) { in[j] = true; r.push_back(j); }
        }
        return r;
    };
    const int nb = 40, nm = 12;
    const std::vector<int32_t> tight = mid ? meeting<TC_MID_LOG2>(5) : meeting<TC_WARP_LOG2>(5);
    for (int k = 0; k < nb; k++) {
        std::vector<int32_t> r = some(draw(90), cols);
        if (k % 4 == 0)
            for (int i = 0; i < 4; i++)
                if (std::find(r.begin(), r.end(), tight[i]) == r.end()) r.push_back(tight[i]);
        B.row(r);
    }
    for (int i = 0; i < nm; i++) {
        A.row(some(1 + draw(nb), nb));
        if (i % 3 == 0) M.row(tight);              // linear probing
        else M.row(some(i == 1 ? longest : 1 + draw(longest), cols));
    }
    const int64_t na = (int64_t)A.crd.size();
    std::vector<int32_t> cnt(na, 0), small;
    std::vector<TcUnit> units;
    std::vector<double> val(na, 0.0), aval(M.crd.size()), bval(B.crd.size());
    for (size_t i = 0; i < aval.size(); i++) aval[i] = 1 + draw(1000);
    for (size_t i = 0; i < bval.size(); i++) bval[i] = 1 + draw(1000);
    for (int i = 0; i < nm; i++) {
        small.push_back(i);
        TcUnit u = {i, 0, (uint32_t)(A.pos[i + 1] - A.pos[i])};
        units.push_back(u);
    }
    TcHeader hdr = {};
    hdr.nsmall = hdr.nmid = nm;
    TcShape sh = {};
    unsigned long long total = 0;
    std::vector<unsigned> want(na, 0);
    std::vector<double> sum(na, 0.0);
    unsigned long long all = 0;
    for (int i = 0; i < nm; i++)
        for (int64_t p = A.pos[i]; p < A.pos[i + 1]; p++)
            for (int64_t q = B.pos[A.crd[p]]; q < B.pos[A.crd[p] + 1]; q++)
                for (int64_t t = M.pos[i]; t < M.pos[i + 1]; t++)
                    if (M.crd[t] == B.crd[q]) {
                        want[p]++;
                        all++;
                        sum[p] += aval[t] * bval[q];
                    }
    auto go = [&](auto out) {
        fake::run_block(32 * (mid ? TC_MID_WARPS : TC_WARPS), 0, 1, [&] {
            if (mid)
                tc_mid_kernel(&hdr, units.data(), A.pos.data(), A.crd.data(), B.pos.data(), B.crd.data(), M.pos.data(), M.crd.data(), nullptr,
                              nullptr, sh, out);
            else
                tc_warp_kernel(&hdr, small.data(), A.pos.data(), A.crd.data(), B.pos.data(), B.crd.data(), M.pos.data(), M.crd.data(), sh, out);
        });
    };
    bool ok = all > 0;
    if (!strcmp(what, "all")) {
        go(TcCountAll{&total, 0});
        ok = ok && total == all;
    } else if (!strcmp(what, "pairs")) {
        go(TcCountPairs{cnt.data()});
        for (int64_t p = 0; p < na; p++) ok = ok && (unsigned)cnt[p] == want[p];
    } else {
        for (int64_t p = 0; p < na; p++) cnt[p] = (int32_t)want[p];
        go(TcValuePairs<false>{cnt.data(), nullptr, val.data(), aval.data(), bval.data(), COMET_B200_PLUS_TIMES});
        for (int64_t p = 0; p < na; p++) ok = ok && (!want[p] || val[p] == sum[p]);     // whole numbers
    }
    printf(ok ? "ok\n" : "results differ\n");
    return ok ? 0 : 1;
}
