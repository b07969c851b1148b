// The list scan's plan against a restatement in 64 bits: for queries over one or several lists, the rows that the
// first pass takes of the list it ends in must survive the record that carries them, and no row may be taken twice
// or left out.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "list_plan.cuh"

using namespace gbivf;

static long bad = 0, cuts = 0, cases = 0;

static void check(const std::vector<int64_t>& lens, uint32_t rows, int step_log) {
    int64_t total = 0;
    for (int64_t n : lens) total += n;
    const uint32_t target = lc_first_rows(rows, (uint32_t)total, true);
    uint64_t before = 0;
    cases++;
    for (int64_t n : lens) {
        if (before + n < target) {
            before += n;
            continue;
        }
        const uint32_t need = (target - (uint32_t)before + 15u) & ~15u;
        if (!lc_ends_inside((uint32_t)n, need)) return;  // the whole list
        cuts++;
        const int packed = lc_pack_skip(step_log, need);
        if ((uint32_t)lc_skip(packed) != need || lc_step_log(packed) != step_log || need >= (uint64_t)n || packed < 0) {
            if (bad++ < 10)
                std::printf("list of %lld rows, total %lld: first pass %u, read back %d, step %d as %d\n", (long long)n,
                            (long long)total, need, lc_skip(packed), step_log, lc_step_log(packed));
        }
        return;
    }
}

int main() {
    const int64_t most = (1ll << 31) - 1;
    for (const int64_t n : {1ll, 511ll, 512ll, 592ll, 593ll, 4096ll, 1ll << 20, 1ll << 24, (1ll << 24) + 1, (1ll << 30) - 1, 1ll << 30,
                      (1ll << 30) + 1024, 1200000000ll, 2147483647ll})
        for (uint32_t rows : {1u, 65u, 4096u, (1u << 24) - 17, (1u << 24) - 16, (1u << 24) - 15, 1u << 24, 1u << 28})
            for (int step : {5, 8, 10}) {
                check({n}, rows, step);
                for (int64_t lead : {1ll, 15ll, 16ll, 100ll, 1ll << 24})
                    if (lead + n <= most) check({lead, n}, rows, step);
            }
    for (int n : {1, 31, 32, 33, 64, 65, 4096})
        for (int nmax : {32, 64})
            for (int seg : {1024, 8192})
                for (int64_t len : {int64_t{1}, int64_t{1023}, int64_t{1024}, int64_t{1025}, int64_t{8192}, int64_t{8193}, most - 8192,
                                    most - 1, most}) {
                    const int64_t gs = tc_group_size(n, nmax), want = (n + gs - 1) / gs * ((len + seg - 1) / seg);
                    cases++;
                    if (gs < 1 || gs > nmax || gs % 16 || tc_items(n, (int)len, nmax, seg) != want) bad++;
                }
    std::printf("cases %ld cuts %ld mismatches %ld\n", cases, cuts, bad);
    return bad != 0 || cuts == 0;
}
