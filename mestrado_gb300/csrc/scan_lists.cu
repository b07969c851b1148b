// List-centric IVF-PQ scan: the (query, list) pairs of a batch grouped by
// list, one work item per (list, group of queries).
//
// The reference scans list by list inside each query (sumidxtab2 per probe,
// sequential/ivf_pq/ivf_search.cpp:182-203; the MPI pipeline dispatches the
// same per-list unit, parallel/ivf_pq/ivf_search.cpp:178-228, and the Xeon Phi
// variant per probe, phi2/ivf_pq/ivf_parallel.cpp:276-278). In a large batch
// most code bytes belong to lists that many queries probe, so here a list is
// decoded once for a group of queries and multiplied with their residuals on
// the tensor cores (scan_tc.cu). This file plans that scan and selects from
// its results.
//
// Both forms of the search use it as a screen: its distances are approximate
// (bounded error), the selected candidates are re-scored in the reference's
// FP32 arithmetic (scan_persistent.cu), and a query is proven when nothing
// outside the selection can enter its result. The exact form scans the queries
// that are not proven again with the per-query kernel, so its results are that
// kernel's bit for bit; the precision form counts them.
//
// Top-k without per-query state in the CTA: a first pass (the query-centric
// kernel, exact tables, SCAN_KEYS_ONLY) scans each query's nearest rows until it
// holds k_sel of them and hands off its k_sel best keys and the k_sel-th key
// tau_q. The list-centric pass appends only keys below tau_q, to a per-query
// buffer in global memory. That first bound is loose (in 128 dimensions the
// nearest lists are hardly closer than the 200th), so the bound moves: the first
// pass's keys and every emitted key are counted in a per-query histogram of
// their distance below the first bound (256 buckets of 2^15 float ulps, about
// 0.4 % each), and each time a query's emissions pass a power of two of about
// k_sel / 4 the emitting warp finds the lowest bucket edge with k_sel counted
// keys below it and lowers tau_q to it (atomicMin). Any such edge bounds the
// k_sel-th key from above, so every work item read afterwards filters harder
// and none loses a true candidate. The select kernel takes the k_sel smallest of
// both sets (exact radix select) and writes the finalize kernels' hand-off; a
// query whose buffer still overflowed is scanned again by the query-centric
// kernel.
#include "block_topk.cuh"
#include "list_scan.cuh"
#include "scan_common.cuh"

namespace gbivf {

constexpr int LC_SEL_NT = 256;    // threads of the select kernel (one CTA per query)
constexpr int LC_SEL_STAGE = 3072;  // keys of a query's pool the select kernel stages in shared memory

// ---------------------------------------------------------------------------
// planning: prefix probes per query, pairs per list, groups
// ---------------------------------------------------------------------------

// One warp per query: the first pass's extent -- the fewest leading probes holding beta * k_sel rows (and, with w.cut,
// a 64th of all, up to LC_SKIP_MAX; all of them when the query has fewer), the last of them cut at the next multiple
// of 16 rows when that leaves more than LC_CUT_ROWS -- and one count per probe with rows beyond it on its list. Zeroes the query's
// emission counter.
__global__ void lc_plan_kernel(DevIndex ix, ScanArgs a, ListScanWork w, int beta) {
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (q >= a.nq) return;
    const int wq = query_w(a, q);
    uint32_t total = 0;
    for (int j = lane; w.cut && j < wq; j += 32) {
        const int l = __ldg(a.probes + (int64_t)q * a.w + j);
        total += l >= 0 ? (uint32_t)__ldg(ix.list_len + l) : 0u;
    }
    total = __reduce_add_sync(0xffffffffu, total);
    // (a 64th of the rows at least: the items of a few long lists run side by side, and all of them filter
    // by this first bound)
    const uint32_t target = lc_first_rows((uint32_t)(beta * lc_ksel(a, q)), total, w.cut);
    uint32_t carry = 0, lim = 0xffffffffu;
    int p = wq;
    bool cut = false;
    for (int j0 = 0; j0 < wq && p == wq; j0 += 32) {
        const int j = j0 + lane;
        const int l = j < wq ? __ldg(a.probes + (int64_t)q * a.w + j) : -1;
        const uint32_t len = l >= 0 ? (uint32_t)__ldg(ix.list_len + l) : 0u;
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, j < wq && carry + incl >= target);
        if (hit) {
            const int src = __ffs(hit) - 1;
            p = j0 + src + 1;  // probes 0 .. p - 1
            const uint32_t n = __shfl_sync(0xffffffffu, len, src), end = carry + __shfl_sync(0xffffffffu, incl, src);
            const uint32_t need = (target - (end - n) + 15u) & ~15u;  // rows of the last of them
            cut = w.cut && lc_ends_inside(n, need);
            lim = cut ? end - n + need : end;
        }
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) {
        w.w0[q] = p;
        w.plim[q] = lim;
        w.ecnt[q] = 0;
    }
    for (int j = p - (cut ? 1 : 0) + lane; j < wq; j += 32) {
        const int l = __ldg(a.probes + (int64_t)q * a.w + j);
        if (l >= 0 && __ldg(ix.list_len + l) > 0) atomicAdd(&w.pcnt[l], 1);
    }
}

// Prefix sums over the C lists of their pair counts (pbeg) and of their work items (gbeg); fill cursors start at
// pbeg; the totals go to pbeg[C], gbeg[C], counters[0]. Two launches
// over blocks of LC_PFX lists (4 per thread): the blocks' totals, then each block's own scan from the
// sum of the totals before it -- every block at once, instead of one block walking all C lists.
constexpr int LC_PFX = 4096;

__device__ __forceinline__ void lc_prefix_load(const DevIndex& ix, const ListScanWork& w, int i0, int (&c)[4],
                                               int (&g)[4], int& tp, int& tg) {
    tp = tg = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        c[j] = i0 + j < ix.C ? w.pcnt[i0 + j] : 0;
        g[j] = c[j] > 0 ? tc_items(c[j], __ldg(ix.list_len + i0 + j), w.tc_n, w.tc_seg) : 0;
        tp += c[j];
        tg += g[j];
    }
}

__global__ void __launch_bounds__(1024) lc_prefix_sums_kernel(DevIndex ix, ListScanWork w) {
    __shared__ int s_p[32], s_g[32];
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
    int c[4], g[4], tp, tg;
    lc_prefix_load(ix, w, blockIdx.x * LC_PFX + 4 * tid, c, g, tp, tg);
    tp = __reduce_add_sync(0xffffffffu, tp);
    tg = __reduce_add_sync(0xffffffffu, tg);
    if (lane == 0) {
        s_p[wp] = tp;
        s_g[wp] = tg;
    }
    __syncthreads();
    if (wp == 0) {
        const int vp = __reduce_add_sync(0xffffffffu, s_p[lane]), vg = __reduce_add_sync(0xffffffffu, s_g[lane]);
        if (lane == 0) {
            w.bsum[2 * blockIdx.x] = vp;
            w.bsum[2 * blockIdx.x + 1] = vg;
        }
    }
}

__global__ void __launch_bounds__(1024) lc_prefix_kernel(DevIndex ix, ListScanWork w) {
    const int C = ix.C;
    __shared__ int s_wp[32], s_wg[32], s_base[2];
    const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, b = blockIdx.x;
    if (wp == 0) {  // this block's base: the totals of the blocks before it
        int bp = 0, bg = 0;
        for (int j = lane; j < b; j += 32) {
            bp += w.bsum[2 * j];
            bg += w.bsum[2 * j + 1];
        }
        bp = __reduce_add_sync(0xffffffffu, bp);
        bg = __reduce_add_sync(0xffffffffu, bg);
        if (lane == 0) {
            s_base[0] = bp;
            s_base[1] = bg;
        }
    }
    const int i0 = b * LC_PFX + 4 * tid;
    int c[4], g[4], tp, tg;
    lc_prefix_load(ix, w, i0, c, g, tp, tg);
    int ip = tp, ig = tg;  // inclusive scan over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int vp = __shfl_up_sync(0xffffffffu, ip, o), vg = __shfl_up_sync(0xffffffffu, ig, o);
        if (lane >= o) {
            ip += vp;
            ig += vg;
        }
    }
    if (lane == 31) {
        s_wp[wp] = ip;
        s_wg[wp] = ig;
    }
    __syncthreads();
    if (wp == 0) {  // exclusive scan of the 32 warp totals
        const int vp = s_wp[lane], vg = s_wg[lane];
        int jp = vp, jg = vg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, jp, o), ug = __shfl_up_sync(0xffffffffu, jg, o);
            if (lane >= o) {
                jp += up;
                jg += ug;
            }
        }
        s_wp[lane] = jp - vp;
        s_wg[lane] = jg - vg;
    }
    __syncthreads();
    int rp = s_base[0] + s_wp[wp] + ip - tp, rg = s_base[1] + s_wg[wp] + ig - tg;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if (i0 + j < C) {
            w.pbeg[i0 + j] = rp;
            w.fill[i0 + j] = rp;
            w.gbeg[i0 + j] = rg;
        }
        rp += c[j];
        rg += g[j];
    }
    if (b == gridDim.x - 1 && tid == 1023) {  // the totals
        w.pbeg[C] = rp;
        w.gbeg[C] = rg;
        w.counters[0] = rg;
    }
}

// One warp per query: the position of each probe's first row in the query's candidate order (the
// prefix of list lengths over all its probes) and a pair record per probe the first pass left: (query,
// position of the probe's first row, skip, float key of the first pass's bound), everything the scan needs
// but the current bound. skip: the probe's rows that the first pass took, and the logarithm of the emissions
// after which the bound is lowered (lc_pack_skip).
// Also starts the query's bound at the first pass's, and its histogram with the first pass's keys.
__global__ void __launch_bounds__(256) lc_fill_kernel(DevIndex ix, ScanArgs a, ListScanWork w) {
    __shared__ unsigned int s_h[8][LC_HIST_BUCKETS];
    const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (q >= a.nq) return;
    const int wq = query_w(a, q), p = w.w0[q];
    const uint32_t lim = w.plim[q];
    const int step_log = 31 - __clz(max(lc_ksel(a, q) / 4, 32));
    const u64 t0k = w.tau0[q];
    if (lane == 0) w.tau[q] = t0k;
    for (int i = lane; i < LC_HIST_BUCKETS; i += 32) s_h[wp][i] = 0u;
    __syncwarp();
    if (t0k != KEY_MAX) {
        const uint32_t t0 = (uint32_t)(t0k >> 32);
        const int na = w.cntA[q];
        for (int i = lane; i < na; i += 32) {
            const uint32_t below = t0 - (uint32_t)(w.keysA[(int64_t)q * a.cand_stride + i] >> 32);
            atomicAdd(&s_h[wp][min(LC_HIST_BUCKETS - 1, (int)(below >> LC_HIST_SHIFT))], 1u);
        }
    }
    __syncwarp();
    for (int i = lane; i < LC_HIST_BUCKETS; i += 32) w.hist[(int64_t)q * LC_HIST_BUCKETS + i] = s_h[wp][i];
    uint32_t carry = 0;
    for (int j0 = 0; j0 < wq; j0 += 32) {
        const int j = j0 + lane;
        const int l = j < wq ? __ldg(a.probes + (int64_t)q * a.w + j) : -1;
        const uint32_t len = l >= 0 ? (uint32_t)__ldg(ix.list_len + l) : 0u;
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const uint32_t first = carry + incl - len;
        const bool cut = j == p - 1 && carry + incl > lim;
        if ((j >= p || cut) && j < wq && len > 0) {
            const int slot = atomicAdd(&w.fill[l], 1);
            w.pairs[slot] = make_int4(q, (int)first, lc_pack_skip(step_log, cut ? lim - first : 0u),
                                        (int)(uint32_t)(t0k >> 32));
        }
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// ---------------------------------------------------------------------------
// selection: the first pass's best keys and the emitted keys -> the finalize hand-off
// ---------------------------------------------------------------------------

// The ksel smallest of the na keys A and the ne keys B of query q (`real` of them keys, the others the largest
// key), with the rows they stand for, into the query's hand-off.
template <bool ROWS_OUT>
__device__ __forceinline__ void select_pool(const DevIndex& ix, const ScanArgs& a, int q, const u64* A, int na,
                                            const u64* B, int ne, int real, int ksel) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31;
    const int stride = a.cand_stride, wq = query_w(a, q), n = na + ne;
    u64* stage = reinterpret_cast<u64*>(smem);                                // LC_SEL_STAGE keys
    uint32_t* prefix = reinterpret_cast<uint32_t*>(stage + LC_SEL_STAGE);     // wq + 1
    int* plist = reinterpret_cast<int*>(prefix + a.w + 1);                    // wq
    unsigned char* work = reinterpret_cast<unsigned char*>(plist + a.w + 1);
    work = reinterpret_cast<unsigned char*>(((uintptr_t)work + 15) & ~(uintptr_t)15);
    __shared__ int s_cnt;
    TopKSmem s{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0, 0, work};
    // the pool: staged in shared memory when it fits, else read in place (the radix passes then go
    // to L2); a small stage keeps several CTAs per SM
    int nA = na, nB = ne;
    if (n <= LC_SEL_STAGE) {
        for (int i = tid; i < na; i += LC_SEL_NT) stage[i] = A[i];
        for (int i = tid; i < ne; i += LC_SEL_NT) stage[na + i] = B[i];
        A = stage;
        nA = n;
        nB = 0;
    }
    for (int j = tid; j < wq; j += LC_SEL_NT) {
        const int l = __ldg(a.probes + (int64_t)q * a.w + j);
        plist[j] = l;
        prefix[j] = l >= 0 ? (uint32_t)__ldg(ix.list_len + l) : 0u;
    }
    if (tid == 0) {
        s_cnt = 0;
        s.slots()[0] = 0;
    }
    __syncthreads();
    if (tid < 32) {  // exclusive prefix of the probe lengths
        uint32_t carry = 0;
        for (int j0 = 0; j0 < wq; j0 += 32) {
            const int j = j0 + lane;
            const uint32_t len = j < wq ? prefix[j] : 0u;
            uint32_t incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (j < wq) prefix[j] = carry + incl - len;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) prefix[wq] = carry;
    }
    const int K = min(ksel, real);
    u64 T = KEY_MAX;
    if (real > K && K > 0) T = block_kth(s, A, nA, B, nB, K);  // the K-th smallest key
    __syncthreads();
    const int64_t o0 = (int64_t)q * stride;
    for (int i0 = 0; i0 < n; i0 += LC_SEL_NT) {
        const int i = i0 + tid;
        const u64 key = i < nA ? A[i] : (i < n ? B[i - nA] : KEY_MAX);
        const bool keep = i < n && key <= T && key != KEY_MAX;
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (!m) continue;
        int base = 0;
        if (lane == __ffs(m) - 1) base = atomicAdd(&s_cnt, __popc(m));
        base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
        if (keep) {
            const int slot = base + __popc(m & ((1u << lane) - 1u));
            const uint32_t pos = key_payload(key);
            const int j = probe_of(prefix, wq, pos);
            const int l = plist[j];
            const int64_t row = ix.list_beg[l] + (int64_t)(pos - prefix[j]);
            a.cand_key[o0 + slot] = key;
            if (ROWS_OUT) {
                a.cand_id[o0 + slot] = (int32_t)(uint32_t)row;
                a.cand_list[o0 + slot] = l;
            } else {
                a.cand_id[o0 + slot] = ix.ids[row];
            }
        }
    }
    // (slots K .. stride - 1 stay unwritten: the finalize kernels read the first cand_cnt only)
    if (tid == 0) a.cand_cnt[q] = K;
}

template <bool ROWS_OUT>
__global__ void __launch_bounds__(LC_SEL_NT) lc_select_kernel(DevIndex ix, ScanArgs a, ListScanWork w) {
    const int q = blockIdx.x, na = w.cntA[q], ne = w.ecnt[q];
    if (ne > w.ecap) {  // the buffer overflowed: the query-centric kernel scans this query again
        if (threadIdx.x == 0) {
            if (a.flags & SCAN_PROVE) {
                a.unproven_list[atomicAdd(a.unproven, 1)] = q;
                a.cand_cnt[q] = -1;  // (no hand-off; on the list once)
                atomicAdd(&w.counters[2], 1);
            } else {
                w.ovf[atomicAdd(&w.counters[2], 1)] = q;
            }
        }
        return;
    }
    select_pool<ROWS_OUT>(ix, a, q, w.keysA + (int64_t)q * a.cand_stride, na, w.ebuf + (int64_t)q * w.ecap, ne, na + ne,
                          lc_ksel(a, q));
}

// the ranges' keys of a split scan (scan_split), padded with the largest key
template <bool ROWS_OUT>
__global__ void __launch_bounds__(LC_SEL_NT) split_select_kernel(DevIndex ix, ScanArgs a, const u64* keys,
                                                                 const int32_t* cnt, int split, int stride) {
    const int q = blockIdx.x;
    int real = 0;
    for (int i = 0; i < split; i++) real += __ldg(cnt + q * split + i);
    select_pool<ROWS_OUT>(ix, a, q, keys + (int64_t)q * split * stride, split * stride, nullptr, 0, real, lc_ksel(a, q));
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

bool list_scan_supported(const DevIndex& ix, const ScanArgs& a) {
    return scan_persistent_supported(ix, a) && !(a.flags & (SCAN_TABLE_DIRECT | SCAN_SRC_RESIDUAL | SCAN_OUT_PACKED));
}

// Keys a query may emit below its threshold. The first pass's k-th key ranks well beyond k over all
// probes for large k (measured at the 100M workload: with 2 k + 2048 slots about one query in seven
// overflowed), so the buffer holds 8 k + 2048; untouched slots cost nothing. Small batches, whose few long
// lists are scanned side by side against the first bound, take up to 65,536 within 64 MB in all.
int list_scan_ecap(const ScanArgs& a) {
    const int base = 8 * scan_persistent_stride(a) + 2048;
    return std::max(base, (int)std::min<int64_t>(65536, (8 << 20) / std::max(a.nq, 1)));
}

static size_t select_smem(int w) {
    return sizeof(u64) * LC_SEL_STAGE + sizeof(int) * (2 * (size_t)w + 2) + 16 + TOPK_WORK_BYTES;
}

cudaError_t launch_list_scan(const DevIndex& ix, const ScanArgs& a, const ListScanWork& w, int num_sms,
                             cudaStream_t st, cudaEvent_t* ev) {
    if (a.nq <= 0) return cudaSuccess;
    if (!list_scan_supported(ix, a) || ix.C > (1 << 24)) return cudaErrorNotSupported;
    if (!(a.flags & SCAN_MIXED) || w.ecap < 1 || w.ecap > list_scan_ecap(a) || w.tc_n < 1 || w.tc_seg < 1)
        return cudaErrorInvalidValue;
    const int C = ix.C, nq = a.nq;
    cudaError_t e;
    auto rec = [&](int i) { return ev && ev[i] ? cudaEventRecord(ev[i], st) : cudaSuccess; };
    if ((e = cudaMemsetAsync(w.pcnt, 0, sizeof(int) * C, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(w.counters, 0, sizeof(int) * 3, st)) != cudaSuccess) return e;
    const int wblocks = (nq * 32 + 255) / 256;
    lc_plan_kernel<<<wblocks, 256, 0, st>>>(ix, a, w, std::max(1, w.beta));
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // First pass: the query-centric kernel over each query's leading rows, keys only, from exact tables (FP16
    // ones saturate at partial distances of 2^18, where their bounds prove nothing; the tensor-core scan has
    // no such limit. 2.63 against 2.03 ms with FP16 tables at 100M rows and m = 16, no difference at 10M
    // rows and m = 8.)
    ScanArgs pa = a;
    pa.flags = (pa.flags & ~SCAN_MIXED) | SCAN_KEYS_ONLY | SCAN_WIDE_SEL;
    pa.w_per_q = w.w0;
    pa.row_lim = w.cut ? w.plim : nullptr;
    pa.cand_key = w.keysA;
    pa.cand_cnt = w.cntA;
    pa.cand_id = nullptr;
    pa.cand_list = nullptr;
    pa.tau_out = w.tau0;
    pa.queue = w.queue_a;
    if ((e = rec(0)) != cudaSuccess) return e;
    if ((e = launch_scan_persistent(ix, pa, num_sms, 512, st, nullptr, false)) != cudaSuccess) return e;
    if ((e = rec(1)) != cudaSuccess) return e;
    const int pblocks = (C + LC_PFX - 1) / LC_PFX;
    lc_prefix_sums_kernel<<<pblocks, 1024, 0, st>>>(ix, w);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    lc_prefix_kernel<<<pblocks, 1024, 0, st>>>(ix, w);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    lc_fill_kernel<<<wblocks, 256, 0, st>>>(ix, a, w);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = rec(2)) != cudaSuccess) return e;
    if ((e = launch_tc_scan(ix, a, w, num_sms, st)) != cudaSuccess) return e;
    if ((e = rec(3)) != cudaSuccess) return e;
    const size_t ssm = select_smem(a.w);
    if ((e = cudaFuncSetAttribute(lc_select_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm)) != cudaSuccess)
        return e;
    lc_select_kernel<true><<<nq, LC_SEL_NT, ssm, st>>>(ix, a, w);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = rec(4)) != cudaSuccess) return e;
    if (a.flags & SCAN_PROVE) return cudaSuccess;  // (overflowed queries are among the unproven ones)
    // queries whose buffer overflowed: the query-centric kernel, exact tables, all their probes, full hand-off
    ScanArgs fa = a;
    fa.flags = (fa.flags & ~SCAN_MIXED) | SCAN_WIDE_SEL;
    fa.qlist = w.ovf;
    fa.nqlist = w.counters + 2;
    fa.queue = w.queue_b;
    return launch_scan_persistent(ix, fa, num_sms, 512, st, nullptr, false);
}

cudaError_t launch_split_select(const DevIndex& ix, const ScanArgs& a, const u64* keys, const int32_t* cnt, int split,
                                int stride, cudaStream_t st) {
    if (!keys || !cnt || split < 1 || stride < 1) return cudaErrorInvalidValue;
    const bool rows_out = (a.flags & (SCAN_MIXED | SCAN_REFINE)) != 0;
    if (!a.cand_key || !a.cand_id || !a.cand_cnt || (rows_out && !a.cand_list)) return cudaErrorInvalidValue;
    const size_t ssm = select_smem(a.w);
    auto sel = rows_out ? split_select_kernel<true> : split_select_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(sel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ssm);
    if (e != cudaSuccess) return e;
    sel<<<a.nq, LC_SEL_NT, ssm, st>>>(ix, a, keys, cnt, split, stride);
    return cudaGetLastError();
}

}  // namespace gbivf
