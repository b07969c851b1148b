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

// batches drawn at random: their work items against the bound that the workspace is sized by
static void check_items(unsigned seed) {
    srand(seed);
    auto draw = [](int n) { return (int)(((int64_t)rand() << 15 ^ rand()) % n); };
    const int C = 1 + draw(40), nq = 1 + draw(200), w = 1 + draw(C), nmax = seed & 1 ? 32 : 64;
    const int seg = seed & 2 ? TC_SEG_FEW : TC_SEG_MANY;
    std::vector<int32_t> lens(C), n(C, 0), order(C);
    for (int l = 0; l < C; l++) {
        lens[l] = draw(4) ? draw(100) : draw(4) ? draw(100000) : draw(2147483647);
        order[l] = l;
    }
    ListPieces p;
    p.build(lens);
    for (int q = 0; q < nq; q++) {  // w different lists, the longest for half of the batches
        if (seed & 4) std::sort(order.begin(), order.end(), [&](int a, int b) { return lens[a] > lens[b]; });
        else for (int i = 0; i < w; i++) std::swap(order[i], order[i + draw(C - i)]);
        for (int i = 0; i < w; i++)
            if (lens[order[i]] > 0) n[order[i]]++;
    }
    int64_t items = 0, each = 0;
    for (int l = 0; l < C; l++) {
        if (n[l] == 0) continue;
        items += tc_items(n[l], lens[l], nmax, seg);
        each += (int64_t)n[l] * tc_segs(lens[l], seg);
    }
    const int64_t bound = p.max_items(nq, w, nmax, seg);
    cases++;
    if (items > bound || ((seed & 4) && bound > each + C + nq * w)) {
        if (bad++ < 10) std::printf("seed %u: %lld items, bound %lld\n", seed, (long long)items, (long long)bound);
    }
}

int main() {
    for (unsigned s = 0; s < 4000; s++) check_items(s);
    {   // 32,768 queries x 256 probes, one list of a million rows among 262,143 of 400: the headers' bytes
        std::vector<int32_t> lens(262144, 400);
        lens[77] = 1000000;
        ListPieces p;
        p.build(lens);
        if (p.max_items(32768, 256, 32, TC_SEG_MANY) * 32 > 32 << 20) bad++;
        // 600,000 queries x 4,096 probes: more pairs than an int counts
        if (list_plan_fits(600000ll * 4096, p.max_items(600000, 4096, 64, TC_SEG_MANY)) || !list_plan_fits(2147483647, 1)) bad++;
        // a flat index of 1e9 codes, 10,000 queries
        p.build({1000000000});
        if (p.max_items(10000, 1, 64, TC_SEG_FEW) * 32 > 6ll << 30) bad++;
    }
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
