// One warp counts rows of up to 256 products by its bitmap: batches that do not end on a multiple of 32, columns that meet.
#include "fake_warp.hpp"

static uint32_t s_few[4096];
#include "kernels.inc"

int main()
{
    const int ncols = 70, words = 3;
    // rows of B of 0 to 69 columns
    std::vector<int64_t> bpos = {0};
    std::vector<int32_t> bcrd;
    for (int k = 0; k < ncols; k++) {
        for (int j = 0; j < k; j++) bcrd.push_back((j * 7 + k) % ncols);
        bpos.push_back((int64_t)bcrd.size());
    }
    // rows of A: a warp takes every fourth one
    std::vector<std::vector<int64_t>> rows;
    for (int r = 0; r < 24; r++) {
        std::vector<int64_t> row;
        int n = 0;
        for (int i = 0; i < 80; i++) {
            const int k = r % 3 == 0 ? 1 + i % 3 : r % 3 == 1 ? (r * 5 + i * 11) % ncols : 69 - r;
            if (n + k > HASH_ROW_MAX) break;
            row.push_back(k);
            n += k;
        }
        rows.push_back(row);
    }
    std::vector<int64_t> apos = {0}, acrd, cnt(rows.size(), -1);
    std::vector<int32_t> list;
    for (auto &r : rows) {
        acrd.insert(acrd.end(), r.begin(), r.end());
        apos.push_back((int64_t)acrd.size());
        list.push_back((int32_t)list.size());
    }
    const unsigned nlist = (unsigned)rows.size();
    fake::run_block(32 * HASH_WARPS, 0, 1, [&] {
        few_columns_kernel(&nlist, list.data(), words, apos.data(), acrd.data(), bpos.data(), bcrd.data(), cnt.data());
    });
    for (size_t r = 0; r < rows.size(); r++) {
        std::vector<bool> seen(ncols, false);
        int64_t want = 0;
        for (int64_t k : rows[r])
            for (int64_t q = bpos[k]; q < bpos[k + 1]; q++) {
                want += !seen[bcrd[q]];
                seen[bcrd[q]] = true;
            }
        if (cnt[r] != want) {
            printf("row %d: %ld columns instead of %ld\n", (int)r, (long)cnt[r], (long)want);
            return 1;
        }
    }
    printf("ok\n");
    return 0;
}
