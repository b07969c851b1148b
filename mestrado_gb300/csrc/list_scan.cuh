// Pieces shared by the planning and selection of the list-centric scan (scan_lists.cu) and its kernel
// (scan_tc.cu).
#pragma once
#include "kernels.cuh"
#include "list_plan.cuh"

namespace gbivf {

constexpr int LC_HIST_SHIFT = 15;   // histogram bucket width: 2^15 float ulps below the first bound
constexpr int TC_CB_BYTES = 65536;  // its FP16 codebook: 256 codes x 16 units x 16 bytes

#ifdef __CUDACC__
// candidates selected for query q
__device__ __forceinline__ int lc_ksel(const ScanArgs& a, int q) {
    const int kq0 = (a.flags & (SCAN_RERANK | SCAN_REFINE)) ? a.kl : query_k(a, q);
    return (a.flags & SCAN_MIXED) ? mixed_sel(a, kq0) : kq0;
}

// One warp: the lowest bucket edge of query q's histogram with at least k_sel emitted keys at or below
// it; tau_q drops to that edge. Bucket i counts keys whose float key lies 2^15 i .. 2^15 (i + 1) - 1
// ulps below the first bound t0 (the last bucket everything lower), so the keys at or below edge j,
// t0 - 2^15 j, are exactly those in buckets j and up.
__device__ __forceinline__ void lc_lower_bound(const ListScanWork& w, int q, uint32_t t0, int ksel, int lane) {
    constexpr int PER = LC_HIST_BUCKETS / 32;
    const unsigned int* hq = w.hist + (int64_t)q * LC_HIST_BUCKETS;
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        c[i] = __ldcg(hq + lane * PER + i);
        sum += c[i];
    }
    // keys in the buckets of higher lanes (suffix sum over the warp, exclusive)
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_down_sync(0xffffffffu, incl, o);
        if (lane + o < 32) incl += v;
    }
    uint32_t above = incl - sum;
    int best = -1;  // the largest bucket index j with sum over buckets >= j of at least ksel
#pragma unroll
    for (int i = PER - 1; i >= 0; i--) {
        above += c[i];
        if (best < 0 && above >= (uint32_t)ksel) best = lane * PER + i;
    }
    const unsigned cand = __ballot_sync(0xffffffffu, best >= 0);
    if (!cand) return;
    const int src = 31 - __clz(cand);  // the highest lane that found one holds the largest j
    const int j = __shfl_sync(0xffffffffu, best, src);
    const uint32_t edge = t0 - ((uint32_t)j << LC_HIST_SHIFT);
    if (lane == 0 && j > 0 && edge > 0x80000000u) atomicMin(w.tau + q, ((unsigned long long)edge << 32) | 0xffffffffull);
}
#endif

}  // namespace gbivf
