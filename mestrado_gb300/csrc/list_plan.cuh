// The integer arithmetic of the list scan's plan, for the host and the device: work items of a list, where the
// first pass ends inside a list, and the record that tells the scan so. No CUDA headers: it also builds as plain
// C++.
#pragma once
#include <algorithm>
#include <cstdint>
#include <functional>
#include <vector>

#ifdef __CUDACC__
#define GB_PLAN __host__ __device__ __forceinline__
#else
#define GB_PLAN inline
#endif

namespace gbivf {

// queries per work item of a list probed by n queries, nmax (32 or 64) at most: the fewest items, evenly
// filled, in steps of 16
GB_PLAN int tc_group_size(int n, int nmax) {
    const int items = (n + nmax - 1) / nmax;
    return ((n + items - 1) / items + 15) / 16 * 16;
}
// pieces of at most seg rows of a list (len >= 1, up to 2^31 - 1)
GB_PLAN int tc_segs(int len, int seg) { return (len - 1) / seg + 1; }
// work items of a list of len rows probed by n queries
GB_PLAN int tc_items(int n, int len, int nmax, int seg) {
    if (n == 0) return 0;
    const int gs = tc_group_size(n, nmax);
    return ((n + gs - 1) / gs) * tc_segs(len, seg);
}

// rows per work item, at most: of few lists (tc_scan_shape), of many
constexpr int TC_SEG_FEW = 1024, TC_SEG_MANY = 8192;

// The most work items that a batch can have on an index's lists. A query probes a list at most once, so the n_l
// queries of list l satisfy sum_l n_l segs_l <= nq S, S = the pieces of the w longest lists, and
//     items = sum_l ceil(n_l / gs) segs_l <= sum_l min(n_l, n_l / nmax + 1) segs_l.
class ListPieces {
public:
    void build(const std::vector<int32_t>& lens) {
        for (int i = 0; i < 2; i++) {
            std::vector<int64_t>& e = more_[i];  // pieces beyond the first of the lists that have several, longest first
            e.clear();
            for (const int32_t n : lens)
                if (n > seg_of(i)) e.push_back(tc_segs(n, seg_of(i)) - 1);
            std::sort(e.begin(), e.end(), std::greater<int64_t>());
            for (size_t j = 1; j < e.size(); j++) e[j] += e[j - 1];
        }
        lists_ = (int64_t)lens.size();
    }
    int64_t max_items(int64_t nq, int64_t w, int nmax, int seg) const {
        const std::vector<int64_t>& e = more_[seg == TC_SEG_FEW ? 0 : 1];
        auto longest = [&](int64_t n) { return n > 0 && !e.empty() ? e[(size_t)std::min<int64_t>(n, (int64_t)e.size()) - 1] : 0; };
        const int64_t all = nq * (w + longest(w)), touched = std::min(nq * w, lists_);
        return std::min(all, (all + nmax - 1) / nmax + touched + longest(touched));
    }

private:
    static int seg_of(int i) { return i == 0 ? TC_SEG_FEW : TC_SEG_MANY; }
    std::vector<int64_t> more_[2];  // (prefix sums)
    int64_t lists_ = 0;
};

// pairs and work items are counted in 32 bits on the device
inline bool list_plan_fits(int64_t pairs, int64_t items) { return pairs <= INT32_MAX && items <= INT32_MAX; }

// The first pass ends inside a list when more rows of it than this are left for the list scan (which
// reads the list from its start and skips the rows already seen).
constexpr uint32_t LC_CUT_ROWS = 512;
// The rows that it took of that list, a multiple of 16, share a word with the logarithm of the emissions after
// which the bound is lowered: LC_SKIP_BITS bits.
constexpr int LC_SKIP_BITS = 24;
constexpr uint32_t LC_SKIP_MAX = (1u << LC_SKIP_BITS) - 16;

// rows of the first pass: `rows`, and with cut a 64th of the query's total (as far as the record holds it)
GB_PLAN uint32_t lc_first_rows(uint32_t rows, uint32_t total, bool cut) {
    uint32_t t = cut ? total / 64 : 0u;
    t = t < LC_SKIP_MAX ? t : LC_SKIP_MAX;
    return rows > t ? rows : t;
}
// whether the first pass ends after `need` rows of a list of n
GB_PLAN bool lc_ends_inside(uint32_t n, uint32_t need) { return n > need && n - need > LC_CUT_ROWS && need <= LC_SKIP_MAX; }

GB_PLAN int lc_pack_skip(int step_log, uint32_t skip) { return step_log << LC_SKIP_BITS | (int)skip; }
GB_PLAN int lc_skip(int packed) { return packed & ((1 << LC_SKIP_BITS) - 1); }
GB_PLAN int lc_step_log(int packed) { return packed >> LC_SKIP_BITS; }

}  // namespace gbivf
