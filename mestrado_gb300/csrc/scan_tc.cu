// The list-centric scan's screening distances on the tensor cores.
//
// The ADC distance of a code row to a query's residual r = x - y_list,
//     sum_s ||r_s - c_s[code_s]||^2 = ||r||^2 + ||c||^2 - 2 <r, c>,   c = the row's PQ reconstruction,
// is a contraction over the d = 128 dimensions once c is written out. A list scanned for N queries is
// then a (rows x 128) x (128 x N) product: 128 multiply-adds per (row, query) pair on the tensor cores
// in place of m table look-ups, and no per-query tables at all (look-ups took m x 256 FP16 entries per
// (list, query), built before the first of them). One work item is a list and up to 64 of the
// queries that probe it.
//
// Per 128-row tile of an item:
//   * 8 warps decode the rows (two groups of four, taking tiles in turn): a row's 16 units of 8 dimensions are copied from the FP16 codebook in
//     shared memory (64 KB, scaled by a power of two) into the tile's A operand. Four lanes share a
//     row; in every step the eight lanes of a quarter-warp read eight different bank quads of the
//     codebook (slot code * 16 + unit, units permuted by lane) and write eight different ones of the
//     128-byte-swizzled tile, so neither side has bank conflicts. That is 8 wavefronts per 32 units, 4
//     cycles per row: the kernel's bound, whatever N is;
//   * one thread issues 8 tcgen05.mma (M = 128, K = 16, N = twice the item's queries rounded up to 16)
//     into one of four TMEM accumulators. The B operand holds the queries' residuals as r_hi and r_lo,
//     two FP16 columns under one power-of-two scale whose sum is the FP32 residual to 2^-22. Both
//     halves in one MMA read the A tile once: at these N the MMA is bound by that read (4 KB per
//     K step), and with a second pass over it shared memory was the limit;
//   * 12 warps (three groups of four, taking tiles in turn) add the two halves and test every (row, query)
//     pair against the query's bound: packed adds and FMAs and a funnel shift that collects the sign
//     bits. Survivors are appended to the queries' emission buffers, one per lane at a time; the
//     position that an append returns is used two appends later, so the atomic's round trip is hidden;
//   * 6 warps build the next item's B operand (residuals, their norms and scales, the bounds)
//     meanwhile. Operands are double-buffered; every wait is bounded (tc_common.cuh).
//
// The approximate distance differs from the real one by the rounding of c to FP16 alone: at most
// 2^-11 ||c|| ||r|| 2 in the worst case, about 2e-5 of the distance on average; the FP16 table entries of the
// per-query kernel (4e-5) are further off. The exact re-score (scan_persistent.cu) decides the results.
//
// What bounds it: the chain from a decoded tile through its MMAs back to the free operand stage (two
// stages of 32 KB are what shared memory holds beside the codebook), about 1,700 cycles per 128-row tile
// at 6 queries per list; shared memory itself is busy for about half of that.
//
// Measured, list scan kernel alone, one GB300, look-ups -> this kernel:
//   100M rows, 262,144 lists of log-normal sizes, m = 16, 32,768 queries, 1.44M (query, probe) pairs: 10.13 -> 5.1 ms
//   100M rows in the lists that k-means makes of a Zipf-weighted mixture, the same shape: 12.3 -> 7.2 ms
//   10M rows, 65,536 lists, m = 8, 10,000 queries, 0.30M pairs: 2.70 -> 0.85 ms
#include <algorithm>

#include <cuda_fp16.h>

#include "block_topk.cuh"
#include "f32x2.cuh"
#include "list_scan.cuh"
#include "scan_common.cuh"
#include "tc_common.cuh"

namespace gbivf {

constexpr int TC_ROWS = 128;                       // code rows per tile (MMA M)
// 27 warps at 72 registers: every role is a chain of dependent instructions, so it is more warps that help
constexpr int TC_EPI_WARPS = 12, TC_DEC_WARPS = 8, TC_BLD_WARPS = 6;
constexpr int TC_DEC0 = TC_EPI_WARPS, TC_BLD0 = TC_DEC0 + TC_DEC_WARPS, TC_MMA_WARP = TC_BLD0 + TC_BLD_WARPS;
constexpr int TC_THREADS = 32 * (TC_MMA_WARP + 1);
constexpr int TC_DSTAGES = 4;                      // accumulators
constexpr uint32_t TC_TMEM_COLS = 512;
constexpr int TC_A_PANEL = TC_ROWS * 128, TC_A_BYTES = 2 * TC_A_PANEL;
constexpr int TC_N64_MIN_PAIRS = 48;               // (query, probe) pairs per list from which items hold 64
constexpr int TC_QCAP = 64;                        // survivor queue entries per epilogue warp
constexpr int TC_CHUNK = 8;                        // accumulator columns per epilogue step
constexpr int TC_SCR = TC_CHUNK + 4;               // scratch row stride (floats): conflict-free 16-byte stores
// tiles whose row norms are kept: the decoders copy tile n's at the end of tile n - 2, which waited for the MMAs of
// tile n - 4, and those for the reads of tile n - 4 - TC_DSTAGES (so TC_DSTAGES + 4 would do)
constexpr int TC_RN = TC_DSTAGES + 6;

// N: queries per item, at most (32 or 64); the B operands of 128 / N items fit
template <int N>
struct TcShape {
    static constexpr int NB = 128 / N;                         // items in flight
    static constexpr int B_PANEL = 2 * N * 128, B_BYTES = 2 * B_PANEL;  // rows: the queries' r_hi, then r_lo
    static constexpr int DCOLS = 2 * N;                        // accumulator columns: hi and lo products
    static_assert(TC_DSTAGES * DCOLS <= (int)TC_TMEM_COLS && NB % 2 == 0, "shape");
};

struct TcSmem {
    static constexpr int CB = 0;                                   // codebook, 64 KB
    static constexpr int A = CB + TC_CB_BYTES;                     // 2 tiles
    static constexpr int B = A + 2 * TC_A_BYTES;                   // NB x (hi, lo)
    static constexpr int SCR = B + 65536;                          // epilogue scratch
    static constexpr int QK = SCR + TC_EPI_WARPS * 32 * TC_SCR * 4;  // survivor queues: keys ...
    static constexpr int QG = QK + TC_EPI_WARPS * TC_QCAP * 8;     // ... and slots
    static constexpr int K1 = QG + TC_EPI_WARPS * TC_QCAP;         // [NB][N / 2] (beta, beta, theta, theta)
    static constexpr int K2 = K1 + 128 * 8;                   // [NB][N] (||r||^2, beta, pos0, t0)
    static constexpr int K3 = K2 + 128 * 16;                  // [NB][N] (query, skip: see lc_fill_kernel)
    static constexpr int RN = K3 + 128 * 8;                  // [TC_RN][128] row norms
    static constexpr int BARS = RN + TC_RN * TC_ROWS * 4;
    static constexpr int TOTAL = BARS + 256;
};
static_assert(TcSmem::TOTAL <= 232448, "shared memory");

// K-major operand in the 128-byte swizzle (8-row groups 1024 bytes apart), sm_100 version bits
__device__ __forceinline__ uint64_t tc_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr));
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// a whole warp waits; it gives up as one
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t phase, volatile int* abort) {
    return __all_sync(0xffffffffu, mbar_wait_or_abort(bar, phase, abort));
}

// Work item headers, 2 x 16 bytes: (list, queries, rows, first pair), first code row and its number in the
// list. A CTA takes
// items blockIdx.x, + gridDim.x, ...; each warp reads 32 of them at a time, one per lane.
struct TcItem {
    int list, np, len, pb, r0;
    int64_t beg;
};
struct TcItems {
    const int4* hdr;
    int nitems, base;  // base: ordinal of the first item of the batch
    int4 a, b;
    __device__ __forceinline__ void fetch() {
        const int64_t it = blockIdx.x + (int64_t)(base + (threadIdx.x & 31)) * gridDim.x;
        a = b = make_int4(0, 0, 0, 0);
        if (it < nitems) {
            a = __ldg(hdr + 2 * it);
            b = __ldg(hdr + 2 * it + 1);
        }
    }
    __device__ __forceinline__ TcItems(const int4* h, int n) : hdr(h), nitems(n), base(0) { fetch(); }
    // header of this CTA's item `ord` (ordinals rise by one at most; past the last: len = np = 0); warp-uniform
    __device__ __forceinline__ TcItem get(int ord) {
        if (ord >= base + 32) {
            base += 32;
            fetch();
        }
        const int src = ord - base;
        TcItem h;
        h.list = __shfl_sync(0xffffffffu, a.x, src);
        h.np = __shfl_sync(0xffffffffu, a.y, src);
        h.len = __shfl_sync(0xffffffffu, a.z, src);
        h.pb = __shfl_sync(0xffffffffu, a.w, src);
        const uint32_t lo = (uint32_t)__shfl_sync(0xffffffffu, b.x, src);
        const uint32_t hi = (uint32_t)__shfl_sync(0xffffffffu, b.y, src);
        h.beg = (int64_t)(((uint64_t)hi << 32) | lo);
        h.r0 = __shfl_sync(0xffffffffu, b.z, src);
        return h;
    }
};

// the queries q of the lanes in m have taken a multiple of their step of emitted keys: tighter bounds
__device__ __noinline__ void tc_lower_bounds(const ScanArgs& a, const ListScanWork& w, unsigned m, int q) {
    const int lane = threadIdx.x & 31;
    for (; m; m &= m - 1) {
        const int qq = __shfl_sync(0xffffffffu, q, __ffs(m) - 1);
        lc_lower_bound(w, qq, (uint32_t)(w.tau0[qq] >> 32), lc_ksel(a, qq), lane);
    }
}

// the code bytes of the four units 4i .. 4i+3 of one row, one byte per unit that the lane needs
template <int M>
__device__ __forceinline__ uint32_t tc_code_word(const uint8_t* codes, int64_t row, int i) {
    if constexpr (M == 16) return __ldg(reinterpret_cast<const uint32_t*>(codes + row * 16) + i);
    else if constexpr (M == 8) return __ldg(reinterpret_cast<const unsigned short*>(codes + row * 8) + i);
    else return __ldg(codes + row * 4 + i);
}

// headers of the work items: one thread per list, lists of more than 8 items by the whole warp
__global__ void tc_items_kernel(DevIndex ix, ListScanWork w) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const bool in = l < ix.C;
    const int pb = in ? w.pbeg[l] : 0, n = in ? w.pbeg[l + 1] - pb : 0;
    const int g0 = in ? w.gbeg[l] : 0, ng = in ? w.gbeg[l + 1] - g0 : 0;
    auto write = [&](int list, int pairs, int first_pair, int len, int64_t beg, int base, int i) {
        const int gs = tc_group_size(pairs, w.tc_n), segs = tc_segs(len, w.tc_seg);
        const int first = i / segs * gs, r0 = i % segs * w.tc_seg;  // pair and row of the list
        int4* d = w.groups + 2 * (int64_t)(base + i);
        d[0] = make_int4(list, min(gs, pairs - first), min(w.tc_seg, len - r0), first_pair + first);
        const int64_t b = beg + r0;
        d[1] = make_int4((int)(uint32_t)b, (int)(b >> 32), r0, 0);
    };
    if (n > 0 && ng <= 8) {
        const int len = ix.list_len[l];
        const int64_t beg = ix.list_beg[l];
        for (int i = 0; i < ng; i++) write(l, n, pb, len, beg, g0, i);
    }
    for (unsigned m = __ballot_sync(0xffffffffu, ng > 8); m; m &= m - 1) {
        const int src = __ffs(m) - 1, ll = __shfl_sync(0xffffffffu, l, src), nn = __shfl_sync(0xffffffffu, n, src),
                  pp = __shfl_sync(0xffffffffu, pb, src), gg = __shfl_sync(0xffffffffu, g0, src),
                  cc = __shfl_sync(0xffffffffu, ng, src);
        const int len = ix.list_len[ll];
        const int64_t beg = ix.list_beg[ll];
        for (int i = lane; i < cc; i += 32) write(ll, nn, pp, len, beg, gg, i);
    }
}

template <int M, int N>
__global__ void __launch_bounds__(TC_THREADS, 1) tc_scan_kernel(const __grid_constant__ DevIndex ix,
                                                            const __grid_constant__ ScanArgs a,
                                                            const __grid_constant__ ListScanWork w) {
    extern __shared__ __align__(1024) unsigned char smem[];
    using S = TcShape<N>;
    constexpr int NB = S::NB;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + TcSmem::BARS);
    uint64_t* a_full = bars;        // [2] tile decoded (the four warps of its group)
    uint64_t* a_empty = bars + 2;   // [2] its MMAs are done
    uint64_t* b_full = bars + 4;    // [NB] queries of an item ready (the three warps of its group)
    uint64_t* b_empty = bars + 8;   // [NB] its MMAs are done and every epilogue warp is past the item
    uint64_t* d_full = bars + 12;   // [4] accumulator ready
    uint64_t* d_empty = bars + 16;  // [4] accumulator read (the four warps of its group)
    uint64_t* cb_full = bars + 20;
    uint64_t* drain = bars + 21;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 22);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 23);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nitems = w.counters[0];

    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(&a_full[s], TC_DEC_WARPS / 2);
            mbar_init(&a_empty[s], 1);
        }
        for (int s = 0; s < NB; s++) {
            mbar_init(&b_full[s], TC_BLD_WARPS / 2);
            mbar_init(&b_empty[s], 1 + TC_EPI_WARPS);
        }
        for (int s = 0; s < TC_DSTAGES; s++) {
            mbar_init(&d_full[s], 1);
            mbar_init(&d_empty[s], 4);
        }
        mbar_init(cb_full, 1);
        mbar_init(drain, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_expect_tx(cb_full, TC_CB_BYTES);
        bulk_load(smem + TcSmem::CB, ix.tc_cb, TC_CB_BYTES, cb_full);
    }
    if (warp == 0) {
        __syncwarp();  // (lane 0 comes from the set-up)
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tslot)),
                     "r"(TC_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    bool ok = true;

    if (warp >= TC_DEC0 && warp < TC_BLD0) {
        // ---------------- decode code rows into the A operand ----------------
        // two groups of four warps take tiles in turn, each the stage of its number
        const int dw = (warp - TC_DEC0) & 3, grp = (warp - TC_DEC0) >> 2, rl = lane >> 2, i = lane & 3;
        const int x = ((rl & 1) << 1) | (i >> 1);  // this lane's permutation of its four units
        uint32_t sel = 0, cba[4], sta[4];
        const uint32_t cb = smem_addr(smem + TcSmem::CB), at = smem_addr(smem + TcSmem::A);
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const int uu = t ^ x, u = 4 * i + uu;
            const int byte = M == 16 ? uu : M == 8 ? uu >> 1 : 0;
            sel |= (uint32_t)byte << (4 * t);
            cba[t] = cb + u * 16;
            sta[t] = at + grp * TC_A_BYTES + (u >> 3) * TC_A_PANEL + rl * 128 + (((u & 7) ^ rl) << 4);
        }
        // The code words of a tile are loaded one tile of the group ahead of their use, its row norms copied
        // into their ring at the same time. The loads are unconditional and into the registers that the
        // loop carries: a merge or a copy of a loaded register would wait for it on the spot.
        constexpr int RG = TC_ROWS / 8 / 4;  // 8-row groups per warp
        uint32_t wd[RG];
        int rows;  // of the tile; 0: no more tiles
        TcItems items(w.groups, nitems);
        int po = 0, pt = 0, slot = grp;
        TcItem ph = items.get(0);
        auto next_tile = [&]() {
            if (++pt * TC_ROWS >= ph.len && ph.len > 0) {
                ph = items.get(++po);
                pt = 0;
            }
        };
        const int nr = dw * 8 + (lane & 7) + 32 * (lane >> 3);  // the row whose norm this lane copies
        const uint32_t rn = smem_addr(smem + TcSmem::RN) + nr * 4;
        auto fetch = [&]() {
            rows = max(0, min(TC_ROWS, ph.len - pt * TC_ROWS));
            const int64_t row0 = ph.beg + pt * TC_ROWS;  // (past the last tile: row 0)
            const uint32_t to = rn + slot * (TC_ROWS * 4);
            slot = slot + 2 >= TC_RN ? slot + 2 - TC_RN : slot + 2;
            next_tile();
            next_tile();  // (the other group's)
            if (nr < rows)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(ix.row_norm + row0 + nr) : "memory");
            else if (rows > 0)  // past the list: nothing passes
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(to), "f"(__int_as_float(0x7f800000)) : "memory");
            asm volatile("cp.async.commit_group;" ::: "memory");
            // rows past the list read its last row; their products are not used
#pragma unroll
            for (int j = 0; j < RG; j++)
                wd[j] = tc_code_word<M>(ix.codes, row0 + max(0, min((dw + 4 * j) * 8 + rl, rows - 1)), i);
        };
        ok = tc_wait(cb_full, 0, abort_flag);
        if (grp) next_tile();
        fetch();
        for (int u = 0; ok && rows > 0; u++) {
            if (!(ok = tc_wait(&a_empty[grp], (u & 1) ^ 1, abort_flag))) break;
            uint32_t cw[RG];
#pragma unroll
            for (int j = 0; j < RG; j++) cw[j] = __byte_perm(wd[j], 0u, sel);
#pragma unroll
            for (int j = 0; j < RG; j += 2) {
                // two row groups at a time
                if ((dw + 4 * j) * 8 >= rows) break;
                uint4 v[2][4];
#pragma unroll
                for (int jj = 0; jj < 2; jj++)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                     : "=r"(v[jj][k].x), "=r"(v[jj][k].y), "=r"(v[jj][k].z), "=r"(v[jj][k].w)
                                     : "r"(cba[k] + __byte_perm(cw[j + jj], 0u, 0x4404u | ((uint32_t)k << 4))));  // code * 256
#pragma unroll
                for (int jj = 0; jj < 2; jj++)
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(sta[k] + (dw + 4 * (j + jj)) * 1024),
                                     "r"(v[jj][k].x), "r"(v[jj][k].y), "r"(v[jj][k].z), "r"(v[jj][k].w)
                                     : "memory");
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");  // (the row norms)
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[grp]);
            fetch();  // the group's next tile, while this one is multiplied
        }
    } else if (warp >= TC_BLD0 && warp < TC_MMA_WARP) {
        // ---------------- build the B operand: residuals of the item's queries ----------------
        // two groups of three warps take items in turn; 8 lanes per query (16 dimensions each), 12
        // queries per step of a group
        constexpr int GW = TC_BLD_WARPS / 2, STEP = 4 * GW;
        const int gw = (warp - TC_BLD0) % GW, grp = (warp - TC_BLD0) / GW, e = lane & 7, sub = gw * 4 + (lane >> 3);
        TcItems items(w.groups, nitems);
        TcItem h = items.get(0);
        if (grp) h = items.get(1);
        int4 pr = sub < h.np ? __ldg(w.pairs + h.pb + sub) : make_int4(-1, 0, 1, 0);
        for (int u = 0; ok && h.np > 0; u++) {
            // the next item's first records, in flight meanwhile
            items.get(2 * u + grp + 1);
            const TcItem nh = items.get(2 * u + grp + 2);
            const int4 npr = sub < nh.np ? __ldg(w.pairs + nh.pb + sub) : make_int4(-1, 0, 1, 0);
            const int npad = (h.np + 15) & ~15, ib = 2 * u + grp, b = ib % NB;
            unsigned char* bt = smem + TcSmem::B + b * S::B_BYTES + (e >> 2) * S::B_PANEL;
            float* k1 = reinterpret_cast<float*>(smem + TcSmem::K1 + b * N * 8);
            const float4* y4 = reinterpret_cast<const float4*>(ix.coa + (int64_t)h.list * 128 + 16 * e);
            for (int g0 = 0; g0 < h.np; g0 += STEP) {
                const int g = g0 + sub;
                if (g0 > 0) pr = g < h.np ? __ldg(w.pairs + h.pb + g) : make_int4(-1, 0, 1, 0);
                const bool used = pr.x >= 0;
                float r[16];
                u64 tau = 0;
                if (used) tau = __ldcg(w.tau + pr.x);
                // (a caller's rows may start on any 4-byte boundary)
                const float* xp = a.queries + (int64_t)max(pr.x, 0) * 128 + 16 * e;
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    // bsxfunMINUS (ivf_search.cpp:155-172)
                    float4 xv;
                    if ((reinterpret_cast<uintptr_t>(a.queries) & 15) == 0) xv = __ldg(reinterpret_cast<const float4*>(xp) + t);
                    else xv = make_float4(__ldg(xp + 4 * t), __ldg(xp + 4 * t + 1), __ldg(xp + 4 * t + 2), __ldg(xp + 4 * t + 3));
                    const float4 yv = __ldg(y4 + t);
                    r[4 * t] = __fsub_rn(xv.x, yv.x);
                    r[4 * t + 1] = __fsub_rn(xv.y, yv.y);
                    r[4 * t + 2] = __fsub_rn(xv.z, yv.z);
                    r[4 * t + 3] = __fsub_rn(xv.w, yv.w);
                }
                float n2 = 0.0f, mx = 0.0f;
#pragma unroll
                for (int t = 0; t < 16; t++) {
                    n2 = __fmaf_rn(r[t], r[t], n2);
                    mx = fmaxf(mx, fabsf(r[t]));
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) {
                    n2 += __shfl_xor_sync(0xffffffffu, n2, o);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                }
                if (g0 == 0) {
                    if (!(ok = tc_wait(&b_empty[b], ((ib / NB) & 1) ^ 1, abort_flag))) break;
                    // slots without a query: nothing passes, whatever their columns hold
                    if (gw == 0 && lane < npad - h.np) k1[((h.np + lane) >> 1) * 4 + ((h.np + lane) & 1) + 2] = -__int_as_float(0x7f800000);
                }
                if (!used) continue;
                // power-of-two scale: the largest component to 2^14 .. 2^15 (FP16 holds 65504); the
                // exponent kept within what a float scale and its inverse can hold
                const int ex = mx > 0.0f ? min(max(14 - ilogbf(mx), -100), 100) : 0;
                const float sc = __uint_as_float((uint32_t)(127 + ex) << 23);
                unsigned char* dst = bt + (g >> 3) * 1024 + (g & 7) * 128;
#pragma unroll
                for (int c = 0; c < 2; c++) {
                    uint32_t hi[4], lo[4];
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        const float u0 = r[8 * c + 2 * t] * sc, u1 = r[8 * c + 2 * t + 1] * sc;
                        const __half2 hh = __floats2half2_rn(u0, u1);
                        const float2 hf = __half22float2(hh);
                        const __half2 ll = __floats2half2_rn(u0 - hf.x, u1 - hf.y);
                        hi[t] = *reinterpret_cast<const uint32_t*>(&hh);
                        lo[t] = *reinterpret_cast<const uint32_t*>(&ll);
                    }
                    // (npad is a multiple of 16: both rows have the same place in their 8-row groups)
                    unsigned char* dc = dst + ((((2 * e + c) & 7) ^ (g & 7)) << 4);
                    *reinterpret_cast<uint4*>(dc) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    *reinterpret_cast<uint4*>(dc + npad * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                }
                if (e == 0) {
                    // pass: ||c||^2 < acc * beta + theta, theta = tau - ||r||^2 (slack for its roundings)
                    const float beta = 2.0f * ix.tc_inv * __uint_as_float((uint32_t)(127 - ex) << 23);
                    const float td = tau == KEY_MAX ? __int_as_float(0x7f800000) : key_dist(tau);
                    float* k = k1 + (g >> 1) * 4 + (g & 1);
                    k[0] = beta;
                    k[2] = (td - n2) + 0x1p-20f * (fabsf(td) + n2);
                    reinterpret_cast<float4*>(smem + TcSmem::K2 + b * N * 16)[g] =
                        make_float4(n2, beta, __int_as_float(pr.y), __int_as_float(pr.w));
                    reinterpret_cast<int2*>(smem + TcSmem::K3 + b * N * 8)[g] = make_int2(pr.x, pr.z);
                }
            }
            if (!ok) break;
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&b_full[b]);
            h = nh;
            pr = npr;
        }
    } else if (warp == TC_MMA_WARP) {
        // ---------------- MMA issue ----------------
        const bool lead = elect_one();
        bool issued = false;
        int tc = 0;
        const uint32_t a0 = smem_addr(smem + TcSmem::A), b0 = smem_addr(smem + TcSmem::B);
        TcItems items(w.groups, nitems);
        for (int ib = 0; ok; ib++) {
            const int b = ib % NB;
            const TcItem h = items.get(ib);
            if (h.np == 0) break;
            const int nt = (h.len + TC_ROWS - 1) / TC_ROWS;
            // FP16 x FP16 -> FP32, K-major A and B, M = 128, N = twice the queries rounded up to 16
            const uint32_t idesc = (1u << 4) | ((uint32_t)((h.np + 15) >> 4) << 19) | ((uint32_t)(TC_ROWS >> 4) << 24);
            if (!(ok = tc_wait(&b_full[b], (ib / NB) & 1, abort_flag))) break;
            for (int t = 0; t < nt; t++, tc++) {
                const int s = tc & 1, d = tc % TC_DSTAGES;
                if (!(ok = tc_wait(&a_full[s], (tc >> 1) & 1, abort_flag)) ||
                    !(ok = tc_wait(&d_empty[d], ((tc / TC_DSTAGES) & 1) ^ 1, abort_flag)))
                    break;
                tc_fence_after();
                if (lead) {
#pragma unroll
                    for (int step = 0; step < 8; step++) {
                        const int panel = step >> 2, k = step & 3;
                        mma_bf16(tmem + (uint32_t)(d * S::DCOLS),
                                 tc_desc_sw128(a0 + s * TC_A_BYTES + panel * TC_A_PANEL + k * 32),
                                 tc_desc_sw128(b0 + b * S::B_BYTES + panel * S::B_PANEL + k * 32), idesc,
                                 step > 0 ? 1u : 0u);
                    }
                    mma_commit(&a_empty[s]);
                    mma_commit(&d_full[d]);
                }
                issued = true;
                __syncwarp();
            }
            if (!ok) break;
            if (lead) mma_commit(&b_empty[b]);
            __syncwarp();
        }
        if (issued && lead) {  // every MMA retired before TMEM is freed
            mma_commit(drain);
            mbar_wait_or_abort(drain, 0, nullptr);
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: group warp / 4 takes every third tile, TMEM lane quadrant warp % 4 ----------------
        const int qd = warp & 3, grp = warp >> 2;
        float* scr = reinterpret_cast<float*>(smem + TcSmem::SCR) + warp * 32 * TC_SCR + lane * TC_SCR;
        u64* qk = reinterpret_cast<u64*>(smem + TcSmem::QK) + warp * TC_QCAP;
        unsigned char* qg = smem + TcSmem::QG + warp * TC_QCAP;
        const unsigned lt = (1u << lane) - 1u;
        int qn = 0;  // queued survivors (warp-uniform)
        // this lane's last append, whose position has not been used yet (step 0: none)
        u64 pkey = 0;
        int pq = 0, pidx = 0, pstep = 0;
        auto retire = [&]() {
            bool cross = false;
            if (pstep) {
                if (pidx < w.ecap) w.ebuf[(int64_t)pq * w.ecap + pidx] = pkey;
                cross = ((pidx + 1) & (pstep - 1)) == 0;
            }
            pstep = 0;
            const unsigned m = __ballot_sync(0xffffffffu, cross);
            if (m) tc_lower_bounds(a, w, m, pq);
        };
        // append the first n (at most 32) queued survivors
        auto append = [&](int n, const float4* k2, const int2* k3) {
            retire();
            const bool in = lane < n;
            const int g = in ? qg[lane] : 0;
            const int2 c = k3[g];
            const u64 key = in ? qk[lane] : 0;
            pkey = key;
            pq = c.x;
            pstep = in ? 1 << lc_step_log(c.y) : 0;
            // (straight into the register that retire() reads: a merge of the two paths would wait for it)
            asm volatile("{\n .reg .pred p;\n setp.ne.s32 p, %2, 0;\n @p atom.global.add.u32 %0, [%1], 1;\n}\n"
                         : "+r"(pidx)
                         : "l"(w.ecnt + pq), "r"((int)in)
                         : "memory");
            if (in) {
                const uint32_t below = (uint32_t)__float_as_int(k2[g].w) - (uint32_t)(key >> 32);
                atomicAdd(w.hist + (int64_t)pq * LC_HIST_BUCKETS + min(LC_HIST_BUCKETS - 1, (int)(below >> LC_HIST_SHIFT)), 1u);
            }
            u64 mk = 0;
            unsigned char mg = 0;
            if (n + lane < qn) {  // (at most 31 entries stay)
                mk = qk[n + lane];
                mg = qg[n + lane];
            }
            __syncwarp();
            if (n + lane < qn) {
                qk[lane] = mk;
                qg[lane] = mg;
            }
            __syncwarp();
            qn -= n;
        };
        int tc = 0;
        const float* rn = reinterpret_cast<const float*>(smem + TcSmem::RN) + qd * 32 + lane;
        TcItems items(w.groups, nitems);
        for (int ib = 0; ok; ib++) {
            const int b = ib % NB;
            const TcItem h = items.get(ib);
            if (h.np == 0) break;
            const int nt = (h.len + TC_ROWS - 1) / TC_ROWS;
            const int npad = (h.np + 15) & ~15;
            const float4* k1 = reinterpret_cast<const float4*>(smem + TcSmem::K1 + b * N * 8);
            const float4* k2 = reinterpret_cast<const float4*>(smem + TcSmem::K2 + b * N * 16);
            const int2* k3 = reinterpret_cast<const int2*>(smem + TcSmem::K3 + b * N * 8);
            if (!(ok = tc_wait(&b_full[b], (ib / NB) & 1, abort_flag))) break;
            for (int t = 0; t < nt; t++, tc++) {
                if (tc % (TC_EPI_WARPS / 4) != grp) continue;
                const int d = tc % TC_DSTAGES;
                const int row = h.r0 + t * TC_ROWS + qd * 32 + lane;  // of the list
                if (!(ok = tc_wait(&d_full[d], (tc / TC_DSTAGES) & 1, abort_flag))) break;
                tc_fence_after();
                if (t * TC_ROWS + qd * 32 < h.len) {  // warp-uniform: some row of this slab
                    const float nrow = rn[tc % TC_RN * TC_ROWS];  // ||c||^2 of this lane's row
                    const f2_t nr2 = f2_pack(nrow, nrow);
                    for (int c0 = 0; c0 < h.np; c0 += TC_CHUNK) {
                        uint32_t r[TC_CHUNK], rl[TC_CHUNK];
                        const uint32_t ta = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(d * S::DCOLS + c0);
                        tmem_ld8_async(ta, r);
                        tmem_ld8_async(ta + npad, rl);
                        tmem_wait_ld();
                        if (c0 + TC_CHUNK >= h.np) {  // all of it is in registers
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&d_empty[d]);
                        }
                        uint32_t mask = 0;  // column j of the chunk at bit TC_CHUNK - 1 - j
#pragma unroll
                        for (int j = 0; j < TC_CHUNK; j += 2) {
                            const float4 k = k1[(c0 + j) >> 1];
                            const f2_t acc = f2_add(f2_pack(__uint_as_float(r[j]), __uint_as_float(r[j + 1])),
                                                    f2_pack(__uint_as_float(rl[j]), __uint_as_float(rl[j + 1])));
                            float s0, s1;
                            f2_unpack(acc, s0, s1);
                            r[j] = __float_as_uint(s0);
                            r[j + 1] = __float_as_uint(s1);
                            const f2_t v = f2_sub(nr2, f2_fma(acc, f2_pack(k.x, k.y), f2_pack(k.z, k.w)));
                            float v0, v1;
                            f2_unpack(v, v0, v1);
                            mask = __funnelshift_l(__float_as_uint(v0), mask, 1);
                            mask = __funnelshift_l(__float_as_uint(v1), mask, 1);
                        }
                        if (!__any_sync(0xffffffffu, mask != 0)) continue;
#pragma unroll
                        for (int j = 0; j < TC_CHUNK; j += 4)
                            *reinterpret_cast<uint4*>(scr + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
                        do {
                            bool in = false;
                            u64 key = 0;
                            const int col = mask ? __clz(mask) - (32 - TC_CHUNK) : 0;
                            if (mask) {
                                mask &= ~((1u << (TC_CHUNK - 1)) >> col);
                                const float4 k = k2[c0 + col];
                                const float dist = __fmaf_rn(-k.y, scr[col], k.x + nrow);
                                key = make_key(dist, (uint32_t)__float_as_int(k.z) + (uint32_t)row);
                                // (the test has slack; the first pass took the list's first rows)
                                in = (uint32_t)(key >> 32) <= (uint32_t)__float_as_int(k.w) &&
                                     row >= lc_skip(k3[c0 + col].y);
                            }
                            const unsigned m = __ballot_sync(0xffffffffu, in);
                            if (in) {
                                const int o = qn + __popc(m & lt);
                                qk[o] = key;
                                qg[o] = (unsigned char)(c0 + col);
                            }
                            qn += __popc(m);
                            __syncwarp();
                            if (qn >= 32) append(32, k2, k3);
                        } while (__any_sync(0xffffffffu, mask != 0));
                    }
                } else {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&d_empty[d]);
                }
            }
            if (!ok) break;
            if (qn > 0) append(qn, k2, k3);  // the slots' constants belong to this item
            __syncwarp();
            if (lane == 0) mbar_arrive(&b_empty[b]);
        }
        retire();
    }
    if (!ok) {
        *abort_flag = 1;
        atomicOr(w.err, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // (the codebook copy has landed: its waiters are past it, or it is waited for here)
    if (tid == 0) mbar_wait_or_abort(cb_full, 0, nullptr);
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS)
                     : "memory");
    }
}

template <int M, int N>
static cudaError_t launch_tc_mn(const DevIndex& ix, const ScanArgs& a, const ListScanWork& w, int num_sms,
                                cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(tc_scan_kernel<M, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcSmem::TOTAL);
    if (e != cudaSuccess) return e;
    tc_items_kernel<<<(ix.C + 255) / 256, 256, 0, st>>>(ix, w);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    tc_scan_kernel<M, N><<<num_sms, TC_THREADS, TcSmem::TOTAL, st>>>(ix, a, w);
    return cudaGetLastError();
}

template <int M>
static cudaError_t launch_tc_m(const DevIndex& ix, const ScanArgs& a, const ListScanWork& w, int num_sms,
                               cudaStream_t st) {
    return w.tc_n == 64 ? launch_tc_mn<M, 64>(ix, a, w, num_sms, st) : launch_tc_mn<M, 32>(ix, a, w, num_sms, st);
}

// Queries per work item, at most: with 64 a list is decoded for fewer items, with 32 the B operands of
// four items are in flight instead of two. Measured at 5 to 6 pairs per list: 32 gives 0.95 against 1.09 ms
// (10M rows) and 5.8 against 6.1 ms (100M); lists of 48 and more pairs fill items of 64.
static_assert(TC_SEG_FEW % TC_ROWS == 0 && TC_SEG_MANY % TC_ROWS == 0, "pieces of whole tiles");
// Rows per work item: lists are cut in pieces of 1,024 rows (8 tiles) when there would be fewer than 8 items
// per SM, so that a few long lists fill the GPU; otherwise only lists over 8,192 rows are cut.
// The first pass ends inside a list only where lists are long: its cost is per query (7 to 12 us on an SM),
// the rows of a short list hardly count, and the cut takes the slower form of the per-query kernel.
void tc_scan_shape(const DevIndex& ix, const ScanArgs& a, int num_sms, double mean_len, ListScanWork* w) {
    const int64_t pairs = (int64_t)a.nq * a.w;
    w->tc_n = pairs >= (int64_t)TC_N64_MIN_PAIRS * ix.C ? 64 : 32;
    w->tc_seg = std::min<int64_t>(pairs, ix.C) < 8 * (int64_t)num_sms ? TC_SEG_FEW : TC_SEG_MANY;
    w->cut = mean_len >= 4096.0;
}

cudaError_t launch_tc_scan(const DevIndex& ix, const ScanArgs& a, const ListScanWork& w, int num_sms, cudaStream_t st) {
    if (!ix.tc_cb || !ix.row_norm || (w.tc_n != 32 && w.tc_n != 64) || (w.tc_seg != TC_SEG_FEW && w.tc_seg != TC_SEG_MANY)) return cudaErrorInvalidValue;
    switch (ix.m) {
        case 4: return launch_tc_m<4>(ix, a, w, num_sms, st);
        case 8: return launch_tc_m<8>(ix, a, w, num_sms, st);
        case 16: return launch_tc_m<16>(ix, a, w, num_sms, st);
        default: return cudaErrorNotSupported;
    }
}

// ||c||^2 of every code row: the codes' centroid norms as FP32 pairs (48 bits), summed in pairs and rounded once. It
// runs in the index's first list scan; FP64 sums, at this GPU's FP64 rate, took 0.28 of its 0.35 ms for 10M rows.
__global__ void __launch_bounds__(256) row_norm_kernel(const uint8_t* __restrict__ codes, int64_t rows, int m,
                                                       const float* __restrict__ pq_hi, const float* __restrict__ pq_lo,
                                                       float* __restrict__ out) {
    extern __shared__ float2 sn[];
    for (int e = threadIdx.x; e < m * 256; e += 256) sn[e] = make_float2(pq_hi[e], pq_lo[e]);
    __syncthreads();
    for (int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x; r < rows; r += (int64_t)gridDim.x * 256) {
        float s = 0.0f, t = 0.0f;
        for (int j = 0; j < m; j += 4) {
            const uint32_t v = *reinterpret_cast<const uint32_t*>(codes + r * m + j);
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const float2 n = sn[(j + b) * 256 + ((v >> (8 * b)) & 0xff)];
                const float u = __fadd_rn(s, n.x), w = __fsub_rn(u, s);  // s + n.x = u + its error, exactly
                t = __fadd_rn(t, __fadd_rn(__fadd_rn(__fsub_rn(s, __fsub_rn(u, w)), __fsub_rn(n.x, w)), n.y));
                s = u;
            }
        }
        // (an infinite norm has no error term)
        out[r] = s <= 3.402823466e38f ? __fadd_rn(s, t) : s;
    }
}

cudaError_t launch_row_norms(const uint8_t* codes, int64_t rows, int m, const float* pq_hi, const float* pq_lo,
                             float* out, cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)std::min<int64_t>((rows + 255) / 256, 152 * 8);
    row_norm_kernel<<<grid, 256, sizeof(float2) * m * 256, st>>>(codes, rows, m, pq_hi, pq_lo, out);
    return cudaGetLastError();
}

}  // namespace gbivf
