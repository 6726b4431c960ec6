// The kernels that count a triangular matrix in another order of its vertices, on small graphs and with 256 hub columns: whether a graph
// is taken, where its longest vertex goes, and the count, with and without room for bitmaps; and matrices that keep their order, because
// they are not skewed, not triangular, or do not ascend.
#include "fake_warp.hpp"

#include <comet_b200.h>

inline double __longlong_as_double(long long v) { return fake::from_bits<double>((unsigned long long)v); }
inline long long __double_as_longlong(double v) { return (long long)fake::bits_of(v); }
#include "kernels.inc"
using namespace cb200;

struct Graph {
    int64_t n;
    std::vector<std::vector<int64_t>> rows;
    std::vector<int64_t> pos, crd;
    int64_t nnz() const { return (int64_t)crd.size(); }
};

static Graph finish(int64_t n, std::vector<std::pair<int64_t, int64_t>> edges, bool upper)
{
    Graph g;
    g.n = n;
    g.rows.resize((size_t)n);
    std::sort(edges.begin(), edges.end());
    edges.erase(std::unique(edges.begin(), edges.end()), edges.end());
    for (auto &e : edges) g.rows[(size_t)(upper ? e.second : e.first)].push_back(upper ? e.first : e.second);     // first > second
    g.pos.push_back(0);
    for (auto &r : g.rows) {
        std::sort(r.begin(), r.end());
        g.crd.insert(g.crd.end(), r.begin(), r.end());
        g.pos.push_back((int64_t)g.crd.size());
    }
    return g;
}

static uint32_t seed = 7;
static int64_t draw(int64_t n) { return (int64_t)((seed = seed * 1664525u + 1013904223u) >> 8) % n; }
static double unit() { return (double)draw(1 << 20) / (1 << 20); }

static Graph skewed(int64_t n, int m, int power, bool upper)
{
    std::vector<std::pair<int64_t, int64_t>> e;
    for (int k = 0; k < m; k++) {
        double u = unit(), v = unit();
        for (int p = 1; p < power; p++) u *= unit();
        const int64_t i = (int64_t)(n * v), j = (int64_t)(n * u);
        if (i != j) e.push_back({std::max(i, j), std::min(i, j)});
    }
    return finish(n, e, upper);
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "skewed";
    Graph g;
    if (what == "skewed" || what == "no room" || what == "unordered" || what == "repeats") g = skewed(700, 9000, 3, false);
    else if (what == "upper" || what == "one below") g = skewed(700, 9000, 3, true);
    else if (what == "even") g = skewed(4000, 60000, 1, false);
    else if (what == "regular") {                    // a ring of 8000 vertices with 6 neighbours on either side
        std::vector<std::pair<int64_t, int64_t>> e;
        for (int64_t i = 0; i < 8000; i++)
            for (int64_t d = 1; d <= 6; d++) e.push_back({std::max(i, (i + d) % 8000), std::min(i, (i + d) % 8000)});
        g = finish(8000, e, false);
    } else {                                         // rows of even length, all of which end in the last column
        g = skewed(700, 9000, 3, true);
        std::vector<std::pair<int64_t, int64_t>> e;
        for (int64_t r = 0; r + 1 < g.n; r++) {
            std::vector<int64_t> row = g.rows[(size_t)r];
            if (!row.empty() && row.back() == g.n - 1) row.pop_back();
            if (row.size() % 2 == 0 && !row.empty()) row.pop_back();
            if (row.empty() && r + 2 < g.n) row.push_back(r + 1);
            for (int64_t j : row) e.push_back({j, r});
            e.push_back({g.n - 1, r});
        }
        g = finish(g.n, e, true);
        for (int64_t r = 0; r + 2 < g.n; r++)
            if ((g.pos[(size_t)r + 1] - g.pos[(size_t)r]) % 2) { printf("row %ld is odd\n", (long)r); return 1; }
    }
    const int64_t n = g.n, nnz = g.nnz();
    auto long_row = [&](int64_t from) {              // a row behind `from` of 5 entries and more
        while (g.pos[(size_t)from + 1] - g.pos[(size_t)from] < 5) from++;
        return from;
    };
    if (what == "unordered") std::swap(g.crd[(size_t)g.pos[(size_t)long_row(333)] + 1], g.crd[(size_t)g.pos[(size_t)long_row(333)] + 2]);
    if (what == "repeats") g.crd[(size_t)g.pos[(size_t)long_row(333)] + 1] = g.crd[(size_t)g.pos[(size_t)long_row(333)]];
    if (what == "one below") g.crd[(size_t)g.pos[(size_t)long_row(333)]] = 5;
    const int64_t *pos = g.pos.data(), *crd = g.crd.data();
    TcHeader hdr = {};
    TriCounters tc = {};
    std::vector<uint32_t> degree((size_t)n, 0), bits((size_t)nnz * 2);
    std::vector<int32_t> hub_count((size_t)n, -9), rest_count((size_t)n, -9), rank((size_t)n, -1), bits_at((size_t)n, -5), place((size_t)nnz);
    std::vector<int2> edge((size_t)nnz);
    std::vector<int64_t> hub_pos((size_t)n + 1), rest_pos((size_t)n + 1);
    std::vector<unsigned short> hub((size_t)nnz);
    std::vector<int32_t> a32((size_t)nnz, -1), m32((size_t)nnz, -1);
    unsigned long long count = 0;
    const unsigned long long room = what == "no room" ? 300 : (unsigned long long)nnz * 2;
    fake::run_block(64, 0, 1, [&] { tri_degree_kernel(n, nnz, pos, crd, degree.data(), &tc); });
    fake::run_block(512, 0, 1, [&] { tri_hist_kernel(n, pos, crd, degree.data(), &tc); });
    fake::run_block(512, 0, 1, [&] { tri_decide_kernel(nnz, &hdr, &tc); });
    const bool taken = hdr.ordered;
    if (taken != (what != "even" && what != "regular" && what != "one below")) {
        printf("taken: %d\n", (int)taken);
        return 1;
    }
    const int64_t tiles = (n + 1 + TRI_TILE - 1) / TRI_TILE;
    std::vector<int64_t> sums((size_t)tiles * 2);
    auto places = [&] {
        for (unsigned y = 0; y < 2; y++)
            for (unsigned b = 0; b < (unsigned)tiles; b++)
                fake::run_block(256, b, (unsigned)tiles, [&] { tri_sums_kernel(n, hub_count.data(), rest_count.data(), &hdr, sums.data()); }, y);
        fake::run_block(1024, 0, 1, [&] { tri_totals_kernel(n, tiles, &hdr, &tc, sums.data(), hub_pos.data(), rest_pos.data()); });
        for (unsigned y = 0; y < 2; y++)
            for (unsigned b = 0; b < (unsigned)tiles; b++)
                fake::run_block(256, b, (unsigned)tiles, [&] {
                    tri_places_kernel(n, hub_count.data(), rest_count.data(), pos, &hdr, sums.data(), hub_pos.data(), rest_pos.data());
                }, y);
    };
    if (!taken) {
        places();
        printf(hdr.ordered || rest_pos != g.pos ? "rows\n" : "ok\n");
        return 0;
    }
    fake::run_block(512, 0, 1, [&] { tri_rank_kernel(n, degree.data(), &hdr, &tc, rank.data(), hub_count.data(), rest_count.data()); });
    std::vector<int64_t> whole((size_t)n, 0);
    for (int64_t i = 0; i < n; i++)
        for (int64_t j : g.rows[(size_t)i]) { whole[(size_t)i]++; whole[(size_t)j]++; }
    const int64_t top = std::max_element(whole.begin(), whole.end()) - whole.begin();
    if (rank[(size_t)top] > n / 20) {
        printf("the vertex of %ld neighbours is number %d\n", (long)whole[(size_t)top], rank[(size_t)top]);
        return 1;
    }
    const unsigned blocks = (unsigned)((nnz + 4095) / 4096);
    for (unsigned b = 0; b < blocks; b++)
        fake::run_block(256, b, blocks, [&] {
            tri_edges_kernel(n, nnz, pos, crd, rank.data(), &hdr, &tc, edge.data(), place.data(), hub_count.data(), rest_count.data());
        });
    places();
    if (what == "unordered" || what == "repeats") {
        printf(hdr.ordered || rest_pos != g.pos ? "rows\n" : "ok\n");
        return 0;
    }
    if (!hdr.ordered) { printf("given up\n"); return 1; }
    for (int64_t k = 0, hubs = 0, others = 0; k <= n; k++) {
        if (hub_pos[(size_t)k] != hubs || rest_pos[(size_t)k] != others) { printf("row %ld\n", (long)k); return 1; }
        if (k < n) { hubs += hub_count[(size_t)k]; others += rest_count[(size_t)k]; }
    }
    fake::run_block(64, 0, 1, [&] {
        tri_scatter_kernel(nnz, edge.data(), place.data(), hub_pos.data(), rest_pos.data(), &hdr, &tc, hub.data(), a32.data(), m32.data(), nullptr);
    });
    fake::run_block(TRI_WARPS * 32, 0, 1, [&] { tri_bitmap_kernel(n, hub_pos.data(), hub.data(), &hdr, &tc, room, bits_at.data(), bits.data()); });
    fake::run_block(TRI_WARPS * 32, 0, 1, [&] {
        tri_count_kernel(n, hub_pos.data(), hub.data(), rest_pos.data(), a32.data(), bits_at.data(), bits.data(), &hdr, &tc, &count);
    });
    int with = 0, without = 0;
    for (int64_t k = 0; k < n; k++)
        if (hub_count[(size_t)k] >= TRI_BITMAP) (bits_at[(size_t)k] >= 0 ? with : without)++;
    // the rest, one by one, and the whole
    std::vector<std::vector<bool>> in((size_t)n, std::vector<bool>((size_t)n, false));
    unsigned long long rest = 0, want = 0;
    for (int64_t i = 0; i < n; i++)
        for (int64_t p = rest_pos[(size_t)i]; p < rest_pos[(size_t)i + 1]; p++) {
            if (m32[(size_t)p] != a32[(size_t)p] - TRI_HUBS) { printf("columns\n"); return 1; }
            in[(size_t)i][(size_t)a32[(size_t)p]] = true;
        }
    for (int64_t i = 0; i < n; i++)
        for (int64_t p = rest_pos[(size_t)i]; p < rest_pos[(size_t)i + 1]; p++)
            for (int64_t q = rest_pos[(size_t)a32[(size_t)p]]; q < rest_pos[(size_t)a32[(size_t)p] + 1]; q++) rest += in[(size_t)i][(size_t)a32[(size_t)q]];
    std::vector<std::vector<bool>> adj((size_t)n, std::vector<bool>((size_t)n, false));
    for (int64_t i = 0; i < n; i++)
        for (int64_t j : g.rows[(size_t)i]) adj[(size_t)i][(size_t)j] = true;
    for (int64_t i = 0; i < n; i++)
        for (int64_t k : g.rows[(size_t)i])
            for (int64_t j : g.rows[(size_t)k]) want += adj[(size_t)i][(size_t)j];
    const bool mixed = what == "no room" ? with > 0 && without > 0 : without == 0 && with > 0;
    if (count + rest != want || count == 0 || rest == 0 || !mixed) {
        printf("%llu and %llu triangles instead of %llu, %d bitmaps, %d rows without\n", count, rest, want, with, without);
        return 1;
    }
    printf("ok\n");
    return 0;
}
