// What a count of triangles asks for.  Scratch is limited: a count for which just enough is there beside the memory that it can do without
// has to go on without that.
#include "fake_launch.hpp"

static size_t room = ~(size_t)0, held[cb200::SLOT_COUNT], total = 0;
static int refused = 0;

static bool grow(int slot, size_t bytes)
{
    if (held[slot] >= bytes) return true;
    if (total + bytes - held[slot] > room) return false;
    total += bytes - held[slot];
    held[slot] = bytes;
    return true;
}

namespace cb200 {
static char *some = (char *)malloc((size_t)64 << 20);           // headers are cleared
int scratch(Slot slot, size_t bytes, void **ptr)
{
    *ptr = some;
    return grow(slot, bytes) ? 0 : fail("no room for slot %d", (int)slot);
}
void ScratchIfRoom::take(Slot slot, size_t bytes)
{
    if (grow(slot, bytes)) p = some;
    else refused++;
}
ScratchIfRoom::~ScratchIfRoom() {}
int exclusive_scan_room(int64_t n) { return grow(SLOT_SCAN, (size_t)n / 256) ? 0 : fail("no room for a scan"); }
int exclusive_scan_i32(const int32_t *, int64_t *, int64_t n, cudaStream_t) { return exclusive_scan_room(n); }
}  // namespace cb200

int main(int argc, char **argv)
{
    const int64_t n = atoll(argv[1]), nnz = atoll(argv[2]);
    alignas(16) static int64_t pos[2], crd[2], count;
    auto call = [&] {
        total = 0;
        memset(held, 0, sizeof(held));
        fake::launches.clear();
        refused = 0;
        return comet_b200_dev_masked_spgemm_count_f64_i64(0, n, n, nnz, nnz, nnz, pos, crd, pos, crd, pos, crd, &count, nullptr);
    };
    // rows [1, n) are never counted in another order: what they take is what the count cannot do without (one row less of bins)
    if (comet_b200_dev_masked_spgemm_count_f64_i64(1, n, n, nnz, nnz, nnz, pos, crd, pos, crd, pos, crd, &count, nullptr)) return 1;
    const size_t least = total + 65536;
    if (call() || !fake::launched("tri_count_kernel")) {
        printf("with room: %s\n", cb200::g_err);
        return 1;
    }
    const size_t all = total;
    for (size_t limit : {least, least + (all - least) / 2, all - 1}) {
        room = limit;
        if (call() || refused != 1 || fake::launched("tri_count_kernel") || !fake::launched("tc_warp_kernel")) {
            printf("with %zu of %zu bytes: %s, %d refused\n", limit, all, cb200::g_err, refused);
            return 1;
        }
    }
    printf("ok\n");
    return 0;
}
