// The mates of a symmetric pattern's entries, and patterns that are not symmetric: found out without a look-up where a vertex has not as many
// entries in its row as in its column.
#include "fake_warp.hpp"

#include "kernels.inc"

static bool symmetric, looked;
static int mates;

static void run(const std::vector<std::vector<int>> &rows)
{
    const int64_t n = (int64_t)rows.size();
    std::vector<int64_t> pos = {0}, crd;
    for (auto &r : rows) {
        crd.insert(crd.end(), r.begin(), r.end());
        pos.push_back((int64_t)crd.size());
    }
    MaskedStats stats = {};
    std::vector<int32_t> mate(crd.size(), -1);
    for (unsigned b = 0; b < 2; b++)
        fake::run_block(64, b, 2, [&] { masked_stats_kernel(n, pos.data(), crd.data(), pos.data(), pos.data(), true, &stats); });
    for (unsigned b = 0; b < 2; b++)
        fake::run_block(64, b, 2, [&] { masked_mates_kernel(n, pos.data(), crd.data(), (int64_t)crd.size(), mate.data(), &stats); });
    symmetric = stats.one_sided == 0;
    looked = false;
    mates = 0;
    for (size_t p = 0; p < mate.size(); p++) {
        looked = looked || mate[p] >= 0;
        mates += mate[p] >= 0;
        const int64_t i = std::upper_bound(pos.begin(), pos.end(), (int64_t)p) - pos.begin() - 1;
        if (symmetric && (mate[p] < pos[crd[p]] || mate[p] >= pos[crd[p] + 1] || crd[(size_t)mate[p]] != i)) {
            printf("entry %d\n", (int)p);
            exit(1);
        }
    }
}

int main()
{
    const int n = 90;
    std::vector<std::vector<int>> sym(n), lower(n), cycle(n);
    for (int i = 0; i < n; i++)
        for (int j = 0; j < n; j++) {
            if ((i * j + i + j) % 7 < 2) sym[i].push_back(j);
            if (j < i && (i + 3 * j) % 5 == 0) lower[i].push_back(j);
        }
    for (int i = 0; i < n; i++) cycle[i].push_back((i + 1) % n);
    run(sym);
    if (!symmetric || !looked) { printf("symmetric\n"); return 1; }
    run(lower);
    if (symmetric || looked) { printf("a lower triangle\n"); return 1; }
    sym[40].pop_back();
    run(sym);
    if (symmetric || looked) { printf("one entry without a mate\n"); return 1; }
    run(cycle);                                   // as many in every row as in every column
    if (symmetric) { printf("a cycle\n"); return 1; }
    cycle.resize(3000);                           // and a ring without a direction behind it, whose entries need not be looked up after a thread's first
    for (int i = n; i < 3000; i++) cycle[i] = {i > n ? i - 1 : n + 1, i + 1 < 3000 ? i + 1 : i - 1};
    cycle[n] = {n + 1};
    cycle[2999] = {2998};
    run(cycle);
    if (symmetric || mates > 128) { printf("a cycle and a ring\n"); return 1; }
    printf("ok\n");
    return 0;
}
