// Index building on the GPU: synthetic mixture generation, k-means for the
// coarse quantizer and the sub-quantizers, assignment and PQ encoding.
//
// The reference trains with yael's k-means (sequential/yael_needs/kmeans.c:
// 209-443: Lloyd iterations, float centroid sums) and encodes with exact 1-NN
// (sequential/ivf_pq/ivf_assign.cpp:3-52, pq-utils/pq_assign.cpp:12-53), all
// single-threaded; at 10M-1B base vectors that is days of CPU. Here:
//   * assignment to d = 128 centroids runs on the tensor cores (the split-BF16
//     tcgen05 GEMM of coarse_gemm.cu, argmin fused into its epilogue, then a
//     reduction over centroid ranges); smaller dimensions use a SIMT kernel
//     with the centroids staged in shared memory;
//   * the sub-quantizers are trained together (one kernel per iteration assigns
//     and sums all of them) and encoded together (residual, m nearest centroids
//     and the code row in one kernel);
//   * centroid sums accumulate in FP64, then divide; an empty cluster is
//     re-seeded with a pseudo-random point;
//   * the generator is counter-based (a 64-bit mix of seed, stream, row and
//     dimension), so any chunk of a data set can be regenerated on its own.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "common.cuh"
#include "f32x2.cuh"
#include "kernels.cuh"

namespace gbivf {

__device__ __host__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ uint64_t hash4(uint64_t a, uint64_t b, uint64_t c, uint64_t d) {
    return mix64(a ^ mix64(b ^ mix64(c ^ mix64(d))));
}

// (double)x without the FP64 pipe, whose conversions take as long as its additions (normal numbers by their
// bits; the others convert)
__device__ __forceinline__ double widen(float x) {
    const uint32_t u = __float_as_uint(x), e = u & 0x7f800000u;
    if (e == 0u || e == 0x7f800000u) return (double)x;
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}

// ---------------------------------------------------------------------------
// mixture generator: x = clip(round(mean[comp] + sigma * N(0,1)), 0, 255)
// ---------------------------------------------------------------------------

__global__ void gen_components_kernel(int32_t* comp, int64_t row0, int64_t n, int ncomp, const double* cdf,
                                      uint64_t seed, uint64_t stream) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t h = hash4(seed, stream, 0xC0FFEEull, (uint64_t)(row0 + i));
    if (!cdf) {
        comp[i] = (int32_t)(h % (uint64_t)ncomp);
        return;
    }
    const double u = ((double)(h >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    int lo = 0, hi = ncomp - 1;  // first c with cdf[c] > u
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (cdf[mid] > u) hi = mid;
        else lo = mid + 1;
    }
    comp[i] = lo;
}

__global__ void gen_values_kernel(float* out, const int32_t* comp, int64_t row0, int64_t n, int d,
                                  const float* means, float sigma, uint64_t seed, uint64_t stream) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int pairs = d / 2;
    if (t >= n * pairs) return;
    const int64_t i = t / pairs;
    const int j = (int)(t % pairs);
    const uint64_t h = hash4(seed, stream, (uint64_t)(row0 + i), (uint64_t)j);
    const float u1 = ((float)(h >> 40) + 0.5f) * (1.0f / 16777216.0f);
    const float u2 = ((float)((h >> 16) & 0xFFFFFF) + 0.5f) * (1.0f / 16777216.0f);
    const float rad = sqrtf(-2.0f * logf(u1));
    float sn, cs;
    sincospif(2.0f * u2, &sn, &cs);
    const float* mu = means + (int64_t)comp[i] * d;
    const float a = fminf(fmaxf(rintf(mu[2 * j] + sigma * rad * cs), 0.0f), 255.0f);
    const float b = fminf(fmaxf(rintf(mu[2 * j + 1] + sigma * rad * sn), 0.0f), 255.0f);
    out[i * d + 2 * j] = a;
    out[i * d + 2 * j + 1] = b;
}

// ---------------------------------------------------------------------------
// assignment
// ---------------------------------------------------------------------------

// per row: the smallest key over the centroid tiles
__global__ void argmin_reduce_kernel(const u64* partial, int64_t n, int tiles, int32_t* assign) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    u64 b = KEY_MAX;
    for (int t = 0; t < tiles; t++) b = min(b, partial[i * tiles + t]);
    assign[i] = (int32_t)key_payload(b);
}

// SIMT nearest centroid for small dimensions: rows of x with stride ld, d <= 32;
// centroids (k x d) staged in shared memory in chunks
constexpr int AS_NT = 256, AS_CHUNK = 256;

template <int D>
__global__ void __launch_bounds__(AS_NT) assign_simt_kernel(const float* __restrict__ x, int64_t n, int64_t ld,
                                                            const float* __restrict__ cent, int k,
                                                            int32_t* __restrict__ assign) {
    __shared__ float sc[AS_CHUNK * D];
    __shared__ float sn[AS_CHUNK];
    const int64_t i = (int64_t)blockIdx.x * AS_NT + threadIdx.x;
    float v[D];
#pragma unroll
    for (int l = 0; l < D; l++) v[l] = i < n ? x[i * ld + l] : 0.0f;
    float best = INFINITY;
    int bi = 0;
    for (int c0 = 0; c0 < k; c0 += AS_CHUNK) {
        const int cn = min(AS_CHUNK, k - c0);
        __syncthreads();
        for (int e = threadIdx.x; e < cn * D; e += AS_NT) sc[e] = cent[(int64_t)c0 * D + e];
        __syncthreads();
        for (int c = threadIdx.x; c < cn; c += AS_NT) {
            float s = 0.0f;
#pragma unroll
            for (int l = 0; l < D; l++) s += sc[c * D + l] * sc[c * D + l];
            sn[c] = s;
        }
        __syncthreads();
        for (int c = 0; c < cn; c++) {
            float dot = 0.0f;
#pragma unroll
            for (int l = 0; l < D; l++) dot += v[l] * sc[c * D + l];
            const float dist = sn[c] - 2.0f * dot;
            if (dist < best) {
                best = dist;
                bi = c0 + c;
            }
        }
    }
    if (i < n) assign[i] = bi;
}

// ---------------------------------------------------------------------------
// centroid update in FP64
// ---------------------------------------------------------------------------

// Rows grouped by cluster (a counting sort), then summed by blocks of consecutive rows of that order: one
// FP64 atomic per (block, cluster, dimension) instead of one per element (100,000 rows x 128 dimensions,
// 1,024 clusters: about 0.25M instead of 12.8M; 140 -> 75 us an iteration).
__global__ void cluster_count_kernel(const int32_t* __restrict__ assign, int64_t n, int* __restrict__ counts) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) atomicAdd(&counts[assign[i]], 1);
}

// first[c]: rows of the clusters before c (one block); the counts are added to totals
__global__ void __launch_bounds__(1024) cluster_first_kernel(const int* __restrict__ counts, int k, int* __restrict__ first,
                                                             int* __restrict__ totals) {
    __shared__ int wsum[32];
    __shared__ int s_base;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_base = 0;
    __syncthreads();
    for (int c0 = 0; c0 < k; c0 += 4096) {
        int v[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = c0 + 4 * tid + j;
            v[j] = c < k ? counts[c] : 0;
            sum += v[j];
        }
        int incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        int run = s_base + incl - sum;
        for (int w = 0; w < warp; w++) run += wsum[w];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int c = c0 + 4 * tid + j;
            if (c < k) {
                first[c] = run;
                totals[c] += v[j];
            }
            run += v[j];
        }
        __syncthreads();
        if (tid == 1023) s_base = run;
        __syncthreads();
    }
}

__global__ void cluster_scatter_kernel(const int32_t* __restrict__ assign, int64_t n, int* __restrict__ cursor,
                                       int32_t* __restrict__ order) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) order[atomicAdd(&cursor[assign[i]], 1)] = (int32_t)i;
}

constexpr int KA_ROWS = 64;

__global__ void __launch_bounds__(128) cluster_sum_kernel(const float* __restrict__ x, int64_t n, int64_t ld, int d,
                                                          const int32_t* __restrict__ assign,
                                                          const int32_t* __restrict__ order, double* __restrict__ sums) {
    __shared__ int32_t s_row[KA_ROWS], s_cl[KA_ROWS];
    const int64_t r0 = (int64_t)blockIdx.x * KA_ROWS;
    const int nr = (int)min((int64_t)KA_ROWS, n - r0);
    for (int i = threadIdx.x; i < nr; i += 128) {
        s_row[i] = order[r0 + i];
        s_cl[i] = assign[s_row[i]];
    }
    __syncthreads();
    for (int l = threadIdx.x; l < d; l += 128) {
        double acc = 0.0;
        for (int i0 = 0; i0 < nr; i0 += 8) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = i0 + j < nr ? __ldg(x + (int64_t)s_row[i0 + j] * ld + l) : 0.0f;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int i = i0 + j;
                if (i >= nr) break;
                acc += widen(v[j]);
                if (i + 1 == nr || s_cl[i + 1] != s_cl[i]) {
                    atomicAdd(&sums[(int64_t)s_cl[i] * d + l], acc);
                    acc = 0.0;
                }
            }
        }
    }
}

__global__ void kmeans_finalize_kernel(const double* __restrict__ sums, const int* __restrict__ counts, int k, int d,
                                       float* __restrict__ cent, const float* __restrict__ x, int64_t n, int64_t ld,
                                       uint64_t seed, int iter) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)k * d) return;
    const int c = (int)(t / d), l = (int)(t % d);
    if (counts[c] > 0) {
        cent[t] = (float)(sums[t] / (double)counts[c]);
    } else {  // empty cluster: re-seed with a pseudo-random point
        const int64_t r = (int64_t)(hash4(seed, 0xE317ull, (uint64_t)iter, (uint64_t)c) % (uint64_t)n);
        cent[t] = x[r * ld + l];
    }
}

__global__ void init_centroids_kernel(const float* __restrict__ x, int64_t n, int64_t ld, int d, int k, uint64_t seed,
                                      float* __restrict__ cent) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)k * d) return;
    const int c = (int)(t / d), l = (int)(t % d);
    // one pseudo-random point from each of k equal slices of the data
    const uint64_t slice = n >= k ? (uint64_t)(n / k) : 0;
    const uint64_t h = hash4(seed, 0x1D17ull, (uint64_t)c, 0);
    const int64_t r = slice ? (int64_t)((uint64_t)c * slice + h % slice) : (int64_t)(h % (uint64_t)n);
    cent[t] = x[r * ld + l];
}

// ---------------------------------------------------------------------------
// sub-quantizers: nearest of 256 centroids in DS dimensions for R rows per thread
//
// The distance is ||c||^2 - 2 <v, c>, the dot product summed in order with every product and sum rounded on
// its own (assign_simt_kernel's arithmetic, bit for bit): two FP32 operations per dimension, and the FP32 rate
// is what bounds it. So the 256 centroids are screened with fused multiply-adds (one operation, more exact
// than the two), keeping the smallest distance of each group of 16 centroids only, and the group that holds
// the smallest is computed again in the defining arithmetic: the first of its smallest distances is the
// code. When another group comes within the two forms' difference, all 256 are computed so.
// Two centroids per instruction; in the defining arithmetic the products are fma(v, c, -0) with a -0 the
// compiler cannot see (f32x2.cuh). A 16-byte load of centroids occupies shared memory's return path for 4
// cycles per warp whatever it broadcasts: encoding takes 8 rows per thread (4 at DS = 16) to stay ahead of
// that. 500,003 rows, m = 16: 1.88 ms with 2 rows and no screen, 2.04 with 8, 1.52 with both.
// ---------------------------------------------------------------------------

constexpr int PQ_GROUP = 8;  // centroid pairs per group

// centroids (256 x DS) and their norms into shared memory: pair p's dimension l at sc[(p * DS + l) * 2 + h]
template <int DS>
__device__ __forceinline__ void pq_load_centroids(const float* __restrict__ cent, float* sc, float* sn) {
    for (int e = threadIdx.x; e < 256 * DS; e += blockDim.x) {
        const int c = e / DS, l = e % DS;
        sc[((c >> 1) * DS + l) * 2 + (c & 1)] = cent[e];
    }
    for (int c = threadIdx.x; c < 256; c += blockDim.x) {
        float s = 0.0f;
        for (int l = 0; l < DS; l++) {
            const float v = cent[c * DS + l];
            s += v * v;
        }
        sn[c] = s;
    }
}

template <int DS, int R, bool EXACT>
__device__ __forceinline__ void pq_pair(const float* sc, const float* sn, int p, const f2_t (&v)[R][DS], f2_t nz2,
                                        float (&d0)[R], float (&d1)[R]) {
    f2_t dot[R];
#pragma unroll
    for (int r = 0; r < R; r++) dot[r] = f2_pack(0.0f, 0.0f);
    const float4* c4 = reinterpret_cast<const float4*>(sc) + p * (DS / 2);
#pragma unroll
    for (int l = 0; l < DS; l += 2) {
        const float4 c = c4[l >> 1];
        const f2_t ca = f2_pack(c.x, c.y), cb = f2_pack(c.z, c.w);
#pragma unroll
        for (int r = 0; r < R; r++) {
            if constexpr (EXACT) {
                dot[r] = f2_add(dot[r], f2_fma(v[r][l], ca, nz2));
                dot[r] = f2_add(dot[r], f2_fma(v[r][l + 1], cb, nz2));
            } else {
                dot[r] = f2_fma(v[r][l + 1], cb, f2_fma(v[r][l], ca, dot[r]));
            }
        }
    }
    const float2 n = reinterpret_cast<const float2*>(sn)[p];
#pragma unroll
    for (int r = 0; r < R; r++) {
        if constexpr (EXACT) f2_unpack(f2_sub(f2_pack(n.x, n.y), f2_add(dot[r], dot[r])), d0[r], d1[r]);
        else f2_unpack(f2_fma(dot[r], f2_pack(-2.0f, -2.0f), f2_pack(n.x, n.y)), d0[r], d1[r]);
    }
}

// snmax: the largest centroid norm
template <int DS, int R>
__device__ __forceinline__ void pq_nearest(const float* sc, const float* sn, float snmax, const f2_t (&v)[R][DS],
                                           f2_t nz2, int (&code)[R]) {
    float best[R], second[R];  // the two smallest of the groups' minima
    int grp[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        best[r] = second[r] = INFINITY;
        grp[r] = 0;
    }
    for (int g = 0; g < 128 / PQ_GROUP; g++) {
        float mn[R];
#pragma unroll
        for (int r = 0; r < R; r++) mn[r] = INFINITY;
#pragma unroll
        for (int i = 0; i < PQ_GROUP; i++) {
            float d0[R], d1[R];
            pq_pair<DS, R, false>(sc, sn, g * PQ_GROUP + i, v, nz2, d0, d1);
#pragma unroll
            for (int r = 0; r < R; r++) mn[r] = fminf(mn[r], fminf(d0[r], d1[r]));
        }
#pragma unroll
        for (int r = 0; r < R; r++) {
            second[r] = fminf(second[r], fmaxf(mn[r], best[r]));
            grp[r] = mn[r] < best[r] ? g : grp[r];
            best[r] = fminf(best[r], mn[r]);
        }
    }
#pragma unroll
    for (int r = 0; r < R; r++) {
        f2_t u[1][DS];
        float vn = 0.0f;
#pragma unroll
        for (int l = 0; l < DS; l++) {
            u[0][l] = v[r][l];
            float a0, a1;
            f2_unpack(v[r][l], a0, a1);
            vn = __fmaf_rn(a0, a0, vn);
        }
        // The two forms differ by at most 2 (2 DS + 2) 2^-24 ||v|| ||c||, each distance's last rounding apart:
        // under 2^-17 (||v||^2 + ||c||^2) for DS <= 32, and twice that between two centroids. Subnormal products
        // and sums round by 2^-150 each whatever the norms are: 2 (4 DS + 2) of them.
        const float margin = __fmaf_rn(0x1p-16f, vn + snmax, 0x1p-140f);
        const bool one = second[r] - best[r] > margin;  // (false for anything not finite)
        const int p0 = one ? grp[r] * PQ_GROUP : 0, p1 = one ? p0 + PQ_GROUP : 128;
        float least = INFINITY;
        int c = 0;  // (no distance below infinity: the first centroid)
        for (int p = p0; p < p1; p++) {
            float d0[1], d1[1];
            pq_pair<DS, 1, true>(sc, sn, p, u, nz2, d0, d1);
            if (d0[0] < least) {
                least = d0[0];
                c = 2 * p;
            }
            if (d1[0] < least) {
                least = d1[0];
                c = 2 * p + 1;
            }
        }
        code[r] = c;
    }
}

// the largest of 256 norms (every thread of the block). One that is not a number does not count: its centroid is
// nobody's nearest, in either arithmetic.
__device__ __forceinline__ float pq_norm_max(const float* sn) {
    float m = 0.0f;
    for (int c = threadIdx.x & 31; c < 256; c += 32) m = fmaxf(m, sn[c]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}

// PQ codes of rows (of their residuals to coa[coarse] when coarse is given): every sub-quantizer's centroids
// resident in shared memory (m x 256 x DS floats: 128 KB at d = 128), one CTA per SM; a thread takes R rows
// through sub-quantizers s0 .. s0 + ms - 1. 500,003 rows, m = 16: 2.10 (residuals, a kernel per sub-quantizer
// and one to store its codes) -> 1.52 ms.
constexpr int PE_NT = 256;

template <int DS, int R>
__global__ void __launch_bounds__(PE_NT, 1) pq_encode_kernel(const float* __restrict__ x, int64_t n, int d,
                                                             const int32_t* __restrict__ coarse,
                                                             const float* __restrict__ coa, int m, int s0, int ms,
                                                             const float* __restrict__ pq, uint8_t* __restrict__ codes,
                                                             float neg_zero) {
    extern __shared__ __align__(16) float psm[];
    float* sn = psm + (int64_t)ms * 256 * DS;
    for (int s = 0; s < ms; s++) pq_load_centroids<DS>(pq + (int64_t)(s0 + s) * 256 * DS, psm + s * 256 * DS, sn + s * 256);
    __syncthreads();
    const f2_t nz2 = f2_pack(neg_zero, neg_zero);
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0 && (!coarse || (reinterpret_cast<uintptr_t>(coa) & 15) == 0);
    for (int64_t i0 = (int64_t)blockIdx.x * PE_NT * R; i0 < n; i0 += (int64_t)gridDim.x * PE_NT * R) {
        int64_t row[R];
        const float* y[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            row[r] = i0 + r * PE_NT + threadIdx.x;
            y[r] = coarse && row[r] < n ? coa + (int64_t)coarse[row[r]] * d : nullptr;
        }
        for (int s = 0; s < ms; s++) {
            f2_t v[R][DS];
#pragma unroll
            for (int r = 0; r < R; r++) {
                float t[DS];
                const int64_t at = (int64_t)(s0 + s) * DS;
#pragma unroll
                for (int l = 0; l < DS; l += 4) {
                    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
                    if (row[r] < n) {
                        const float* xp = x + row[r] * d + at + l;
                        if (vec) a = __ldg(reinterpret_cast<const float4*>(xp));
                        else a = make_float4(xp[0], xp[1], xp[2], xp[3]);
                        if (y[r]) {
                            const float* yp = y[r] + at + l;
                            if (vec) b = __ldg(reinterpret_cast<const float4*>(yp));
                            else b = make_float4(yp[0], yp[1], yp[2], yp[3]);
                        }
                    }
                    // x - 0 is x: rows without a coarse centroid are encoded as they are
                    t[l] = __fsub_rn(a.x, b.x);
                    t[l + 1] = __fsub_rn(a.y, b.y);
                    t[l + 2] = __fsub_rn(a.z, b.z);
                    t[l + 3] = __fsub_rn(a.w, b.w);
                }
#pragma unroll
                for (int l = 0; l < DS; l++) v[r][l] = f2_pack(t[l], t[l]);
            }
            int code[R];
            pq_nearest<DS, R>(psm + s * 256 * DS, sn + s * 256, pq_norm_max(sn + s * 256), v, nz2, code);
#pragma unroll
            for (int r = 0; r < R; r++)
                if (row[r] < n) codes[row[r] * m + s0 + s] = (uint8_t)code[r];
        }
    }
}

// One k-means iteration of all sub-quantizers (blockIdx.y): assignment of the block's rows and their sums.
// After a chunk of PK_R x 256 rows is assigned, thread c walks the chunk's rows of cluster c (a linked list in
// shared memory) and adds them to its own FP64 sums in registers; the block's sums are written once, for
// pq_centroids_kernel to add. 100,000 rows, m = 8: 675 us an iteration with a kernel per sub-quantizer and
// FP64 atomics -> 460 us (two blocks per SM; 515 with one and twice the rows per thread).
constexpr int PK_NT = 256;

template <int DS, int PK_R>
__global__ void __launch_bounds__(PK_NT, DS <= 16 ? 2 : 1) pq_kmeans_kernel(const float* __restrict__ x, int64_t n, int d,
                                                          const float* __restrict__ cent, double* __restrict__ sums,
                                                          int* __restrict__ counts, float neg_zero) {
    constexpr int CH = PK_NT * PK_R, LD = DS + 1;
    extern __shared__ __align__(16) float psm[];
    float* sc = psm;                       // 256 x DS centroids
    float* sn = sc + 256 * DS;             // 256 norms
    float* sx = sn + 256;                  // CH x LD rows
    int* head = reinterpret_cast<int*>(sx + CH * LD);  // 256
    int* next = head + 256;                // CH
    const int s = blockIdx.y, tid = threadIdx.x;
    pq_load_centroids<DS>(cent + (int64_t)s * 256 * DS, sc, sn);
    const f2_t nz2 = f2_pack(neg_zero, neg_zero);
    const float* xs = x + (int64_t)s * DS;
    const bool vec = (reinterpret_cast<uintptr_t>(x) & 15) == 0;  // (d and DS are multiples of 8)
    double acc[DS];
    int cnt = 0;
#pragma unroll
    for (int l = 0; l < DS; l++) acc[l] = 0.0;
    for (int64_t i0 = (int64_t)blockIdx.x * CH; i0 < n; i0 += (int64_t)gridDim.x * CH) {
        __syncthreads();  // the centroids; the previous chunk's walks
        head[tid] = -1;
        f2_t v[PK_R][DS];
#pragma unroll
        for (int r = 0; r < PK_R; r++) {
            const int64_t row = i0 + r * PK_NT + tid;
#pragma unroll
            for (int l = 0; l < DS; l += 4) {
                float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (row < n) {
                    const float* p = xs + row * d + l;
                    if (vec) a = __ldg(reinterpret_cast<const float4*>(p));
                    else a = make_float4(p[0], p[1], p[2], p[3]);
                }
                const float t[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    sx[(r * PK_NT + tid) * LD + l + j] = t[j];
                    v[r][l + j] = f2_pack(t[j], t[j]);
                }
            }
        }
        int code[PK_R];
        pq_nearest<DS, PK_R>(sc, sn, pq_norm_max(sn), v, nz2, code);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < PK_R; r++)
            if (i0 + r * PK_NT + tid < n) next[r * PK_NT + tid] = atomicExch(&head[code[r]], r * PK_NT + tid);
        __syncthreads();
        for (int e = head[tid]; e >= 0; e = next[e]) {
            cnt++;
#pragma unroll
            for (int l = 0; l < DS; l++) acc[l] += widen(sx[e * LD + l]);
        }
    }
    const int64_t o = ((int64_t)s * gridDim.x + blockIdx.x) * 256 + tid;
    counts[o] = cnt;
#pragma unroll
    for (int l = 0; l < DS; l++) sums[o * DS + l] = acc[l];
}

// the blocks' sums added, divided; an empty cluster is re-seeded with a pseudo-random point
__global__ void pq_centroids_kernel(const double* __restrict__ sums, const int* __restrict__ counts, int nb, int m, int ds,
                                    float* __restrict__ cent, const float* __restrict__ x, int64_t n, int d,
                                    uint64_t seed, int iter) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m * 256 * ds) return;
    const int s = t / (256 * ds), c = t / ds % 256, l = t % ds;
    double sum = 0.0;
    int cnt = 0;
    for (int b = 0; b < nb; b++) {
        const int64_t o = ((int64_t)s * nb + b) * 256 + c;
        sum += sums[o * ds + l];
        cnt += counts[o];
    }
    if (cnt > 0) {
        cent[t] = (float)(sum / (double)cnt);
    } else {
        const int64_t r = (int64_t)(hash4(seed + s, 0xE317ull, (uint64_t)iter, (uint64_t)c) % (uint64_t)n);
        cent[t] = x[r * d + (int64_t)s * ds + l];
    }
}

// e = x - coa[assign] - c1(codes): the residual error a refinement quantizer encodes
__global__ void pq_error_kernel(const float* __restrict__ x, int64_t n, int d, const int32_t* __restrict__ assign,
                                const float* __restrict__ coa, int m, const float* __restrict__ pq,
                                const uint8_t* __restrict__ codes, float* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * d) return;
    const int64_t i = t / d;
    const int l = (int)(t % d), ds = d / m, s = l / ds;
    const float y = assign ? coa[(int64_t)assign[i] * d + l] : 0.0f;
    out[t] = x[t] - y - pq[((int64_t)s * 256 + codes[i * m + s]) * ds + (l - s * ds)];
}

inline unsigned blocks(int64_t work, int nt) { return (unsigned)((work + nt - 1) / nt); }

static int device_sms() {
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 1;
    return sms;
}

// a device block freed with its scope, carved in 256-byte steps
struct Block {
    void* p = nullptr;
    size_t size = 0;
    ~Block() {
        if (p) cudaFree(p);
    }
    size_t take(size_t bytes) {
        const size_t at = size;
        size += (bytes + 255) / 256 * 256;
        return at;
    }
    cudaError_t alloc() { return cudaMalloc(&p, std::max<size_t>(size, 256)); }
    template <class T>
    T* at(size_t off) const { return reinterpret_cast<T*>(static_cast<unsigned char*>(p) + off); }
};

// Operands of the d = 128 assignment on the tensor cores (the persistent tcgen05 GEMM with the argmin
// epilogue), for blocks of up to 2^20 rows.
struct Assign128 {
    int64_t n = 0, bq = 0;
    int k = 0, sms = 1;
    size_t o_ct = 0, o_cn = 0, o_qt = 0, o_part = 0, o_err = 0;
    bool tiles_ready = false;  // all rows fit one block: their tiles are made once
    void plan(Block& b, int64_t rows, int kk) {
        n = rows;
        k = kk;
        sms = device_sms();
        bq = std::min<int64_t>(n, 1 << 20);
        const int64_t tail = n % bq;
        // partial-result slots for the largest need among the two block sizes used
        size_t slots = (size_t)bq * 2 * coarse_gemm_nsplit((int)bq, k, sms, nullptr);
        if (tail) slots = std::max(slots, (size_t)tail * 2 * coarse_gemm_nsplit((int)tail, k, sms, nullptr));
        o_ct = b.take(coarse_mma_tile_bytes(k, true));
        o_cn = b.take(sizeof(float) * k);
        o_qt = b.take(coarse_gemm_qtile_bytes((int)bq));
        o_part = b.take(sizeof(u64) * slots);
        o_err = b.take(sizeof(int));
    }
    cudaError_t start(const Block& b, cudaStream_t st) { return cudaMemsetAsync(b.at<int>(o_err), 0, sizeof(int), st); }
    // (centroids may change between runs, the rows may not)
    cudaError_t run(const Block& b, const float* x, const float* cent, int32_t* assign, cudaStream_t st, bool hi_only) {
        cudaError_t e = launch_bf16_split_tiles(cent, k, b.at<uint8_t>(o_ct), st);
        if (e == cudaSuccess) e = launch_norm_f(cent, k, 128, b.at<float>(o_cn), st);
        for (int64_t r0 = 0; r0 < n && e == cudaSuccess; r0 += bq) {
            const int nb = (int)std::min<int64_t>(bq, n - r0);
            const int ns = coarse_gemm_nsplit(nb, k, sms, nullptr);
            uint8_t* qt = b.at<uint8_t>(o_qt);
            if (!tiles_ready) {
                e = launch_bf16_tiles(x + r0 * 128, nb, MMA_QUERY_TILE, qt, st);
                const size_t written = coarse_mma_tile_bytes(nb, false), total = coarse_gemm_qtile_bytes(nb);
                if (e == cudaSuccess && total > written) e = cudaMemsetAsync(qt + written, 0, total - written, st);
            }
            if (e == cudaSuccess)
                e = launch_coarse_gemm_argmin(qt, b.at<uint8_t>(o_ct), nb, k, b.at<float>(o_cn), b.at<u64>(o_part), sms,
                                              b.at<int>(o_err), st, hi_only);
            if (e == cudaSuccess) {
                argmin_reduce_kernel<<<blocks(nb, 256), 256, 0, st>>>(b.at<u64>(o_part), nb, 2 * ns, assign + r0);
                e = cudaGetLastError();
            }
        }
        tiles_ready = e == cudaSuccess && bq == n;
        return e;
    }
    // waits for the stream; a bounded wait that ran out in any run
    cudaError_t finish(const Block& b, cudaStream_t st) {
        int herr = 0;
        cudaError_t e = cudaMemcpyAsync(&herr, b.at<int>(o_err), sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        return e == cudaSuccess && herr ? cudaErrorLaunchTimeout : e;
    }
};

// nearest centroid for every row: tensor cores for d = 128, SIMT for d <= 32
cudaError_t assign_rows(const float* x, int64_t n, int64_t ld, int d, const float* cent, int k, int32_t* assign,
                        cudaStream_t st, bool hi_only) {
    if (d == 128 && ld == 128) {
        Block b;
        Assign128 a;
        a.plan(b, n, k);
        cudaError_t e = b.alloc();
        if (e != cudaSuccess) return e;
        e = a.start(b, st);
        if (e == cudaSuccess) e = a.run(b, x, cent, assign, st, hi_only);
        const cudaError_t f = a.finish(b, st);
        return e != cudaSuccess ? e : f;
    }
    switch (d) {
        case 8: assign_simt_kernel<8><<<blocks(n, AS_NT), AS_NT, 0, st>>>(x, n, ld, cent, k, assign); break;
        case 16: assign_simt_kernel<16><<<blocks(n, AS_NT), AS_NT, 0, st>>>(x, n, ld, cent, k, assign); break;
        case 32: assign_simt_kernel<32><<<blocks(n, AS_NT), AS_NT, 0, st>>>(x, n, ld, cent, k, assign); break;
        default: return cudaErrorNotSupported;
    }
    return cudaGetLastError();
}

cudaError_t kmeans_rows(const float* x, int64_t n, int64_t ld, int d, int k, int niter, uint64_t seed, float* cent,
                        cudaStream_t st) {
    const bool tc = d == 128 && ld == 128;
    const int64_t chunk = std::min<int64_t>(n, 1 << 30);  // rows sorted at a time
    Block b;
    Assign128 a;
    const size_t o_as = b.take(sizeof(int32_t) * n), o_sum = b.take(sizeof(double) * k * d), o_tot = b.take(sizeof(int) * k),
                 o_cnt = b.take(sizeof(int) * k), o_cur = b.take(sizeof(int) * k), o_ord = b.take(sizeof(int32_t) * chunk);
    if (tc) a.plan(b, n, k);
    cudaError_t e = b.alloc();
    if (e != cudaSuccess) return e;
    int32_t* assign = b.at<int32_t>(o_as);
    if (tc) e = a.start(b, st);
    if (e == cudaSuccess) {
        init_centroids_kernel<<<blocks((int64_t)k * d, 256), 256, 0, st>>>(x, n, ld, d, k, seed, cent);
        e = cudaGetLastError();
    }
    for (int it = 0; it < niter && e == cudaSuccess; it++) {
        e = tc ? a.run(b, x, cent, assign, st, false) : assign_rows(x, n, ld, d, cent, k, assign, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(b.at<double>(o_sum), 0, sizeof(double) * k * d, st);
        if (e == cudaSuccess) e = cudaMemsetAsync(b.at<int>(o_tot), 0, sizeof(int) * k, st);
        for (int64_t r0 = 0; r0 < n && e == cudaSuccess; r0 += chunk) {
            const int64_t nb = std::min(chunk, n - r0);
            if ((e = cudaMemsetAsync(b.at<int>(o_cnt), 0, sizeof(int) * k, st)) != cudaSuccess) break;
            cluster_count_kernel<<<blocks(nb, 256), 256, 0, st>>>(assign + r0, nb, b.at<int>(o_cnt));
            cluster_first_kernel<<<1, 1024, 0, st>>>(b.at<int>(o_cnt), k, b.at<int>(o_cur), b.at<int>(o_tot));
            cluster_scatter_kernel<<<blocks(nb, 256), 256, 0, st>>>(assign + r0, nb, b.at<int>(o_cur), b.at<int32_t>(o_ord));
            cluster_sum_kernel<<<blocks(nb, KA_ROWS), 128, 0, st>>>(x + r0 * ld, nb, ld, d, assign + r0,
                                                                    b.at<int32_t>(o_ord), b.at<double>(o_sum));
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) {
            kmeans_finalize_kernel<<<blocks((int64_t)k * d, 256), 256, 0, st>>>(b.at<double>(o_sum), b.at<int>(o_tot), k, d,
                                                                                cent, x, n, ld, seed, it);
            e = cudaGetLastError();
        }
    }
    const cudaError_t f = tc ? a.finish(b, st) : cudaStreamSynchronize(st);
    return e != cudaSuccess ? e : f;
}

cudaError_t gen_mixture(float* out, int64_t n, int d, const float* means, int ncomp, const double* cdf, float sigma,
                        uint64_t seed, uint64_t stream_id, int64_t row0, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (d % 2) return cudaErrorInvalidValue;
    void* comp = nullptr;
    cudaError_t e = cudaMalloc(&comp, sizeof(int32_t) * n);
    if (e != cudaSuccess) return e;
    gen_components_kernel<<<blocks(n, 256), 256, 0, st>>>((int32_t*)comp, row0, n, ncomp, cdf, seed, stream_id);
    gen_values_kernel<<<blocks(n * (d / 2), 256), 256, 0, st>>>(out, (int32_t*)comp, row0, n, d, means, sigma, seed,
                                                                 stream_id);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(comp);
    return e;
}

template <int DS, int PK_R>
static cudaError_t pq_train_ds(const float* r, int64_t n, int d, int m, int niter, uint64_t seed, float* pq,
                               cudaStream_t st) {
    // one wave of blocks, two per SM (one with DS = 32): one assigns while the other adds
    const int nb = (int)std::max<int64_t>(1, std::min<int64_t>((n + PK_NT * PK_R - 1) / (PK_NT * PK_R), (DS <= 16 ? 2 : 1) * device_sms() / m));
    Block b;
    const size_t o_sum = b.take(sizeof(double) * (size_t)m * nb * 256 * DS), o_cnt = b.take(sizeof(int) * (size_t)m * nb * 256);
    const size_t smem = sizeof(float) * (256 * DS + 256 + PK_NT * PK_R * (DS + 1)) + sizeof(int) * (256 + PK_NT * PK_R);
    cudaError_t e = cudaFuncSetAttribute(pq_kmeans_kernel<DS, PK_R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = b.alloc();
    if (e != cudaSuccess) return e;
    for (int s = 0; s < m; s++)
        init_centroids_kernel<<<blocks(256 * DS, 256), 256, 0, st>>>(r + s * DS, n, d, DS, 256, seed + s,
                                                                     pq + (int64_t)s * 256 * DS);
    for (int it = 0; it < niter; it++) {
        pq_kmeans_kernel<DS, PK_R><<<dim3(nb, m), PK_NT, smem, st>>>(r, n, d, pq, b.at<double>(o_sum), b.at<int>(o_cnt), -0.0f);
        pq_centroids_kernel<<<blocks((int64_t)m * 256 * DS, 256), 256, 0, st>>>(b.at<double>(o_sum), b.at<int>(o_cnt), nb, m,
                                                                                DS, pq, r, n, d, seed, it);
    }
    e = cudaGetLastError();
    const cudaError_t f = cudaStreamSynchronize(st);
    return e != cudaSuccess ? e : f;
}

cudaError_t pq_train_rows(const float* r, int64_t n, int d, int m, int niter, uint64_t seed, float* pq,
                          cudaStream_t st) {
    switch (d / m) {
        case 8: return pq_train_ds<8, 4>(r, n, d, m, niter, seed + 1, pq, st);
        case 16: return pq_train_ds<16, 2>(r, n, d, m, niter, seed + 1, pq, st);
        case 32: return pq_train_ds<32, 1>(r, n, d, m, niter, seed + 1, pq, st);
        default: return cudaErrorNotSupported;
    }
}

template <int DS, int R>
static cudaError_t pq_encode_ds(const float* x, int64_t n, int d, const int32_t* coarse, const float* coa, int m,
                                const float* pq, uint8_t* codes, cudaStream_t st) {
    // as many sub-quantizers as fit shared memory at a time (all of them at d = 128)
    const size_t per = sizeof(float) * (256 * DS + 256);
    const int most = std::max(1, (int)((size_t)200 * 1024 / per));
    cudaError_t e = cudaFuncSetAttribute(pq_encode_kernel<DS, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(per * std::min(most, m)));
    const unsigned grid = (unsigned)std::min<int64_t>(device_sms(), (n + PE_NT * R - 1) / (PE_NT * R));
    for (int s0 = 0; s0 < m && e == cudaSuccess; s0 += most) {
        const int ms = std::min(most, m - s0);
        pq_encode_kernel<DS, R><<<grid, PE_NT, per * ms, st>>>(x, n, d, coarse, coa, m, s0, ms, pq, codes, -0.0f);
        e = cudaGetLastError();
    }
    const cudaError_t f = cudaStreamSynchronize(st);
    return e != cudaSuccess ? e : f;
}

cudaError_t pq_encode_rows(const float* x, int64_t n, int d, const int32_t* coarse, const float* coa, int m,
                           const float* pq, uint8_t* codes, cudaStream_t st) {
    switch (d / m) {
        case 8: return pq_encode_ds<8, 8>(x, n, d, coarse, coa, m, pq, codes, st);
        case 16: return pq_encode_ds<16, 4>(x, n, d, coarse, coa, m, pq, codes, st);
        case 32: return pq_encode_ds<32, 2>(x, n, d, coarse, coa, m, pq, codes, st);
        default: return cudaErrorNotSupported;
    }
}

cudaError_t pq_error_rows(const float* x, int64_t n, int d, const int32_t* coarse, const float* coa, int m,
                          const float* pq, const uint8_t* codes, float* out, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    pq_error_kernel<<<blocks(n * d, 256), 256, 0, st>>>(x, n, d, coarse, coa, m, pq, codes, out);
    return cudaGetLastError();
}

}  // namespace gbivf
