// Centroid probes ahead of the scan: reduced-precision (first part) and exact.
//
// Reduced-precision centroid probe (the precision form of GetClustersAccessOrderIVF,
// searcher.hpp:181-215, for flat and two-level indexes).
//
// The centroid scores come from one tensor-core GEMM per batch (pdxg_gemm.cu, BF16 or
// FP8-E4M3 operands, FP32 accumulation, epilogue |c|^2 - 2 q.c: the squared L2 distance up to
// the query's own |q|^2). Per query, probe_select_kernel takes the m' = ceil(1.1 nprobe)
// centroids with the smallest scores (the probe list widened by 10%), rescores them in FP32
// with the reference's own probe arithmetic (Horizontal, avx2_computers.hpp:47-98: 8 FMA lanes,
// pairwise double reduction) and keeps the nprobe nearest by (distance, id). A centroid the
// reduced-precision score pushes out of the widened list is the probe-set error of this form;
// whenever the exact nprobe nearest are all inside it, the visit order equals the reference's.
#include <cstdint>
#include <cuda_runtime.h>

#include "pdxg_block.cuh"
#include "pdxg_common.cuh"

namespace pdxg {

// |c|^2 of each row (FP32 result of an FP64 sum); one warp per row.
__global__ void row_sq_kernel(const float* __restrict__ x, uint32_t n, uint32_t d, float* __restrict__ out) {
    const uint32_t row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (row >= n) return;
    double s = 0.0;
    for (uint32_t i = lane; i < d; i += 32) {
        const double v = x[(size_t)row * d + i];
        s += v * v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) out[row] = (float)s;
}

constexpr int kSelectThreads = 128;

// Shared memory of one probe CTA: query, one key per centroid, candidates, sort keys.
size_t probe_select_smem(uint32_t d, uint32_t n1, uint32_t cand_cap, uint32_t sort_cap) {
    return ((size_t)d * 4 + 15) / 16 * 16 + (size_t)((n1 + 3) & ~3u) * 4 + (size_t)cand_cap * 4 + (size_t)sort_cap * 8;
}

// Order-preserving map of a float onto uint32 (negative scores included).
__device__ __forceinline__ uint32_t float_key(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// One CTA per query: widened candidate list from the approximate scores, FP32 rescore, the
// nprobe nearest sorted by (distance, id) into order[q * stride ..], count[q].
__global__ void __launch_bounds__(kSelectThreads) probe_select_kernel(const __grid_constant__ ProbeParams pp) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ Scalars s;
    const uint32_t q = blockIdx.x;
    const uint32_t n1 = pp.nclusters, d = pp.d;
    float* qf = reinterpret_cast<float*>(smem);                                         // [d]
    uint32_t* keys = reinterpret_cast<uint32_t*>(smem + ((size_t)d * 4 + 15) / 16 * 16);  // [n1]
    uint32_t* cand = keys + ((n1 + 3) & ~3u);                                            // [cand_cap]
    uint64_t* sortb = reinterpret_cast<uint64_t*>(cand + pp.cand_cap);                   // [sort_cap]
    const uint32_t np = pp.q_nprobe ? __ldg(pp.q_nprobe + q) : pp.nprobe;
    const uint32_t m = np < n1 ? np : n1;
    uint32_t mw = (uint32_t)ceilf(__fmul_rn(1.1f, (float)m));
    if (mw > n1) mw = n1;
    const float* src = pp.queries + (size_t)q * d;
    for (uint32_t i = threadIdx.x; i < d; i += kSelectThreads) qf[i] = __ldg(src + i);
    const float* sc = pp.scores + (size_t)q * pp.ld_scores;
    for (uint32_t c = threadIdx.x; c < n1; c += kSelectThreads) keys[c] = float_key(__ldg(sc + c));
    __syncthreads();
    // the mw smallest approximate scores: below the mw-th key, then ties in id order
    uint32_t kth, less;
    block_radix_select<kSelectThreads>(keys, n1, mw, s, kth, less);
    const uint32_t nl = block_compact<kSelectThreads>(
        n1, [&](uint32_t, uint32_t v) { return keys[v] < kth; }, [](uint32_t i) { return i; }, cand, s);
    const uint32_t nt = block_compact<kSelectThreads>(
        n1, [&](uint32_t, uint32_t v) { return keys[v] == kth; }, [](uint32_t i) { return i; }, cand + nl, s);
    (void)nt;
    // FP32 rescore of the candidates, 8 threads each (LevelOps::probe's arithmetic)
    const uint32_t N = next_pow2(mw);
    const uint32_t sub = threadIdx.x & 7;
    for (uint32_t base = 0; base < N; base += kSelectThreads / 8) {
        const uint32_t i = base + (threadIdx.x >> 3);
        const bool active = i < mw;
        const uint32_t c = active ? cand[i] : 0u;
        const float dd = horiz_f32_group8(qf, pp.centroids + (size_t)c * d, d, sub, active);
        if (sub == 0 && i < N) sortb[i] = active ? (((uint64_t)__float_as_uint(dd) << 32) | c) : ~0ull;
    }
    __syncthreads();
    block_bitonic_sort<kSelectThreads>(sortb, N);
    for (uint32_t i = threadIdx.x; i < m; i += kSelectThreads) pp.order[(size_t)q * pp.stride + i] = (uint32_t)sortb[i];
    if (threadIdx.x == 0) {
        pp.count[q] = m;
        if (pp.stats) {
            // the approximate scores read each centroid once per query (score_bytes per
            // centroid), the rescore the widened list in FP32
            const unsigned long long b = (unsigned long long)n1 * pp.score_bytes + (unsigned long long)mw * d * 4u;
            atomicAdd(pp.stats + 8, b);
            atomicAdd(pp.stats, b);
        }
    }
}

// ------------------------------------------------------------------------------------ exact
// Exact distances of a batch of queries to every centroid of a level (LevelOps::probe's values,
// searcher.hpp:181-215): FP32 in the AVX2 Horizontal order (8 FMA lanes over dims j, j + 8, ...,
// lanes j and j + 4 added in double, then pairs, then the d % 8 tail).
//
// A CTA takes 32 queries x 32 centroids and stages 64 dims of both with cp.async, two stages
// deep. Four threads share a tile of 4 x 4 pairs, each running two adjacent lanes of Horizontal
// as one packed chain, so a staged element feeds four chains. Bound by the FP32 pipe (two packed
// operations per pair of dims). Row stride 72 floats: the 16 lanes of a half warp read 4 rows x 8
// floats from distinct banks. With the pick below: 24 + 28 us for 300 queries x 895 centroids x 768
// dims (every centroid sorted), 15 + 11 us for 515 x 775 x 200; one CTA per query (8 threads a
// centroid, one load in flight per thread) took 405 and 65 us.
constexpr int kDistQ = 32, kDistC = 32, kDistD = 64, kDistRow = 72, kDistThreads = 256;

// VEC: d a multiple of 4 and both arrays 16-byte aligned (16-byte asynchronous copies); without it
// the stages are filled by plain loads.
template <bool VEC>
__global__ void __launch_bounds__(kDistThreads) centroid_dist_kernel(const float* __restrict__ queries,
                                                                     const uint32_t* __restrict__ q_list, uint32_t nq,
                                                                     uint32_t d, const float* __restrict__ cent,
                                                                     uint32_t n, uint32_t* __restrict__ keys) {
    __shared__ __align__(16) float qs[2][kDistQ * kDistRow];
    __shared__ __align__(16) float xs[2][kDistC * kDistRow];
    __shared__ uint32_t qrow[kDistQ];
    const uint32_t q0 = blockIdx.x * kDistQ, c0 = blockIdx.y * kDistC;
    const uint32_t full = d & ~7u;  // the tail dims are added at the end
    const uint32_t tid = threadIdx.x;
    if (tid < kDistQ) {
        const uint32_t q = q0 + tid < nq ? q0 + tid : q0;
        qrow[tid] = q_list ? __ldg(q_list + q) : q;
    }
    __syncthreads();
    const uint32_t nst = (full + kDistD - 1) / kDistD;
    auto issue = [&](uint32_t st) {
        const uint32_t j0 = st * kDistD;
        float* qb = qs[st & 1];
        float* xb = xs[st & 1];
        if constexpr (VEC) {
#pragma unroll
            for (int t = 0; t < kDistQ * kDistD / 4 / kDistThreads; ++t) {
                const uint32_t e = tid + t * kDistThreads, r = e >> 4, j = j0 + (e & 15) * 4;
                const bool in = j < full;  // full is a multiple of 8: a 16-byte piece never crosses it
                cp_async16_zfill(qb + r * kDistRow + (e & 15) * 4, queries + (size_t)qrow[r] * d + (in ? j : 0), in);
                const uint32_t c = c0 + r < n ? c0 + r : c0;
                cp_async16_zfill(xb + r * kDistRow + (e & 15) * 4, cent + (size_t)c * d + (in ? j : 0), in);
            }
        } else {
            for (uint32_t e = tid; e < kDistQ * kDistD; e += kDistThreads) {
                const uint32_t r = e >> 6, j = j0 + (e & 63);
                const uint32_t c = c0 + r < n ? c0 + r : c0;
                qb[r * kDistRow + (e & 63)] = j < full ? __ldg(queries + (size_t)qrow[r] * d + j) : 0.0f;
                xb[r * kDistRow + (e & 63)] = j < full ? __ldg(cent + (size_t)c * d + j) : 0.0f;
            }
        }
    };
    const uint32_t lane = tid & 31, warp = tid >> 5;
    const uint32_t sub = lane & 3, cg = (lane >> 2) & 3, qg = lane >> 4;
    const uint32_t qr0 = (warp & 3) * 8 + qg, cr0 = (warp >> 2) * 16 + cg;  // rows qr0 + 2 i, cr0 + 4 j
    uint64_t acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    if (nst) issue(0);
    cp_async_commit();
    for (uint32_t st = 0; st < nst; ++st) {
        if (st + 1 < nst) issue(st + 1);
        cp_async_commit();
        cp_async_wait1();
        __syncthreads();
        const float* qb = qs[st & 1] + 2 * sub;
        const float* xb = xs[st & 1] + 2 * sub;
#pragma unroll
        for (int t = 0; t < kDistD / 8; ++t) {  // dims past `full` are zero in both: nothing is added
            uint64_t qv[4], xv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                qv[i] = *reinterpret_cast<const uint64_t*>(qb + (qr0 + 2 * i) * kDistRow + 8 * t);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                xv[j] = *reinterpret_cast<const uint64_t*>(xb + (cr0 + 4 * j) * kDistRow + 8 * t);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint64_t df = f32x2_sub(qv[i], xv[j]);
                    acc[i][j] = f32x2_fma(df, df, acc[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float lo, hi;
            f32x2_unpack(acc[i][j], lo, hi);
            // threads 0 and 1 of the four: lanes 2 sub and 2 sub + 1 with their partners + 4
            double s0 = (double)lo + (double)__shfl_down_sync(0xffffffffu, lo, 2, 4);
            double s1 = (double)hi + (double)__shfl_down_sync(0xffffffffu, hi, 2, 4);
            s0 = s0 + __shfl_down_sync(0xffffffffu, s0, 1, 4);
            s1 = s1 + __shfl_down_sync(0xffffffffu, s1, 1, 4);
            const uint32_t r = qr0 + 2 * i, c = c0 + cr0 + 4 * j;
            if (sub == 0 && q0 + r < nq && c < n) {
                double s = s0 + s1;
                for (uint32_t k = full; k < d; ++k) {
                    const float t = __fsub_rn(__ldg(queries + (size_t)qrow[r] * d + k), __ldg(cent + (size_t)c * d + k));
                    s += (double)__fmul_rn(t, t);
                }
                keys[(size_t)(q0 + r) * n + c] = __float_as_uint((float)s);
            }
        }
    }
}

// keys[i x n]: distances (float bits) of query q_list[i] (query i without a list) to the n centroids.
cudaError_t launch_centroid_dist(const float* queries, const uint32_t* q_list, uint32_t nq, uint32_t d,
                                 const float* centroids, uint32_t n, uint32_t* keys, cudaStream_t st) {
    const dim3 grid((nq + kDistQ - 1) / kDistQ, (n + kDistC - 1) / kDistC);
    const bool vec = d % 4 == 0 && ((uintptr_t)queries & 15) == 0 && ((uintptr_t)centroids & 15) == 0;
    if (vec) centroid_dist_kernel<true><<<grid, kDistThreads, 0, st>>>(queries, q_list, nq, d, centroids, n, keys);
    else centroid_dist_kernel<false><<<grid, kDistThreads, 0, st>>>(queries, q_list, nq, d, centroids, n, keys);
    return cudaGetLastError();
}

// The nprobe nearest centroids by (distance, id), ascending, from the distances above: one CTA per
// query. Queries with an order ahead of the scan need no per-centroid arrays in the scan kernel.
template <int T>
__global__ void __launch_bounds__(T) probe_pick_kernel(const __grid_constant__ ProbeParams pp) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ Scalars s;
    const uint32_t q = pp.q_list ? __ldg(pp.q_list + blockIdx.x) : blockIdx.x;
    const uint32_t n1 = pp.nclusters;
    uint64_t* sortb = reinterpret_cast<uint64_t*>(smem);                    // [sort_cap]
    uint32_t* keys = reinterpret_cast<uint32_t*>(sortb + pp.sort_cap);      // [n1]
    uint32_t* cand = keys + ((n1 + 3) & ~3u);                               // [cand_cap]
    const uint32_t np = pp.q_nprobe ? __ldg(pp.q_nprobe + q) : pp.nprobe;
    const uint32_t m = np < n1 ? np : n1;
    const uint32_t N = next_pow2(m);
    const uint32_t* src = pp.keys + (size_t)blockIdx.x * n1;
    if (m < n1) {
        for (uint32_t c = threadIdx.x; c < n1; c += T) keys[c] = __ldg(src + c);
        __syncthreads();
        uint32_t kth, less;
        block_radix_select<T>(keys, n1, m, s, kth, less);
        const uint32_t nl = block_compact<T>(
            n1, [&](uint32_t, uint32_t v) { return keys[v] < kth; }, [](uint32_t i) { return i; }, cand, s);
        block_compact<T>(n1, [&](uint32_t, uint32_t v) { return keys[v] == kth; }, [](uint32_t i) { return i; },
                         cand + nl, s);
        for (uint32_t i = threadIdx.x; i < N; i += T)
            sortb[i] = (i < m) ? (((uint64_t)keys[cand[i]] << 32) | cand[i]) : ~0ull;
    } else {  // every centroid: sort them all
        for (uint32_t i = threadIdx.x; i < N; i += T)
            sortb[i] = (i < n1) ? (((uint64_t)__ldg(src + i) << 32) | i) : ~0ull;
    }
    __syncthreads();
    block_bitonic_sort<T>(sortb, N);
    for (uint32_t i = threadIdx.x; i < m; i += T) pp.order[(size_t)q * pp.stride + i] = (uint32_t)sortb[i];
    if (threadIdx.x == 0) {
        pp.count[q] = m;
        if (pp.stats) {
            const unsigned long long b = (unsigned long long)n1 * pp.d * 4u;
            atomicAdd(pp.stats + 8, b);
            atomicAdd(pp.stats, b);
        }
    }
}

// Shared memory of one pick CTA: sort keys, one key per centroid, candidates.
static size_t probe_pick_smem(const ProbeParams& pp) {
    return (size_t)pp.sort_cap * 8 + (size_t)((pp.nclusters + 3) & ~3u) * 4 + (size_t)pp.cand_cap * 4;
}

// Exact probe ahead of the scan: distances and pick, keys_rows queries at a time. Without a list
// the queries are rows 0 .. nq - 1.
cudaError_t launch_probe_exact(const ProbeParams& all, cudaStream_t st) {
    for (uint32_t q0 = 0; q0 < all.nq; q0 += all.keys_rows) {
        ProbeParams pp = all;
        pp.nq = all.nq - q0 < all.keys_rows ? all.nq - q0 : all.keys_rows;
        if (pp.q_list) {
            pp.q_list += q0;
        } else {
            pp.queries += (size_t)q0 * pp.d;
            pp.order += (size_t)q0 * pp.stride;
            pp.count += q0;
            if (pp.q_nprobe) pp.q_nprobe += q0;
        }
        cudaError_t e = launch_centroid_dist(pp.queries, pp.q_list, pp.nq, pp.d, pp.centroids, pp.nclusters, pp.keys, st);
        if (e != cudaSuccess) return e;
        const size_t smem = probe_pick_smem(pp);
        // sorts of a thousand keys or more, and selections from thousands: more threads per CTA
        auto kern = (pp.sort_cap >= 1024 || pp.nclusters > 2048) ? probe_pick_kernel<512> : probe_pick_kernel<128>;
        const int threads = (pp.sort_cap >= 1024 || pp.nclusters > 2048) ? 512 : 128;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<pp.nq, threads, smem, st>>>(pp);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_row_sq(const float* x, uint32_t n, uint32_t d, float* out, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    row_sq_kernel<<<(n * 32 + 255) / 256, 256, 0, st>>>(x, n, d, out);
    return cudaGetLastError();
}


cudaError_t launch_probe_select(const ProbeParams& pp, cudaStream_t st) {
    const size_t smem = probe_select_smem(pp.d, pp.nclusters, pp.cand_cap, pp.sort_cap);
    cudaError_t e = cudaFuncSetAttribute(probe_select_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    probe_select_kernel<<<pp.nq, kSelectThreads, smem, st>>>(pp);
    return cudaGetLastError();
}

}  // namespace pdxg
