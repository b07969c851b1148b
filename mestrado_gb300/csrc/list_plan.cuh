// The integer arithmetic of the list scan's plan, for the host and the device: work items of a list, where the
// first pass ends inside a list, and the record that tells the scan so. No CUDA headers: it also builds as plain
// C++.
#pragma once
#include <cstdint>

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
