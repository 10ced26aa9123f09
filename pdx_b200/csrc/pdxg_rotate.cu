// Query preparation: NormalizeQuery (scalar.hpp:23-40) and the ADSampling rotation
// y = M^T x of adsampling.hpp:225-245, batched as R[nq x d] = normalize(Q)[nq x d] @ M[d x d]
// (M row-major, as stored in the index file).
//
// The FP32 path is a register-tiled SIMT GEMM with FP32 accumulation (the reference's
// sgemm_ precision). Rotation parity against the reference is at FP32 rounding level, not
// bit-exact: the reference's own result depends on its BLAS build.
#include <cstdint>
#include <cuda_runtime.h>

namespace pdxg {

// Norm of one row by one warp: sqrt(sum x^2), the divisor of NormalizeQuery (1 for a zero row).
__device__ __forceinline__ float warp_row_norm(const float* __restrict__ row, uint32_t d) {
    float s = 0.0f;
    for (uint32_t i = threadIdx.x & 31; i < d; i += 32) s = __fmaf_rn(row[i], row[i], s);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    return (s == 0.0f) ? 1.0f : sqrtf(s);
}

__global__ void query_norms_kernel(const float* __restrict__ q, uint32_t nq, uint32_t d,
                                   float* __restrict__ norms) {
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (warp >= nq) return;
    const float norm = warp_row_norm(q + (size_t)warp * d, d);
    if ((threadIdx.x & 31) == 0) norms[warp] = norm;
}

// A few rows (nq <= kGemvRows, a single query or an appended row): C[nq x d] = (A / norm) @ B.
// Slice w of 32 takes rows w, w + 32, ... of B (FMA in that order, eight rows of B loaded before
// their FMAs); the 32 slices' partial sums are then added in slice order, so the result does not
// depend on timing. Bound by the latency of reading B once, so it is spread over the GPU: a CTA has
// 8 output columns, thread = (slice, column), 32 contiguous bytes per slice and row. Each CTA
// normalizes the rows itself, which saves the launch of the norms kernel.
// One row, d = 1024: 12 us; 2.6 + 14 with 32 columns per 1,024-thread CTA after the norms kernel.
constexpr uint32_t kGemvRows = 8;
constexpr uint32_t kGemvSlices = 32;
constexpr uint32_t kGemvCols = 8;

__global__ void __launch_bounds__(kGemvSlices * kGemvCols) rotate_gemv_kernel(const float* __restrict__ A, bool normalize,
                                                                              const float* __restrict__ B,
                                                                              float* __restrict__ C, uint32_t M,
                                                                              uint32_t N, uint32_t K) {
    __shared__ float part[kGemvSlices][kGemvRows][kGemvCols];
    __shared__ float norms[kGemvRows];
    const uint32_t slice = threadIdx.x / kGemvCols, lc = threadIdx.x % kGemvCols, warp = threadIdx.x >> 5;
    const uint32_t col = blockIdx.x * kGemvCols + lc;
    float b[8], bn[8];
    auto fetch = [&](uint32_t i0, float (&r)[8]) {
#pragma unroll
        for (uint32_t t = 0; t < 8; ++t) {
            const uint32_t i = i0 + kGemvSlices * t;
            r[t] = (i < K && col < N) ? __ldg(B + (size_t)i * N + col) : 0.0f;
        }
    };
    fetch(slice, b);  // in flight while the rows are normalized
    if (normalize) {
        static_assert(kGemvSlices * kGemvCols / 32 == kGemvRows, "a warp per row");
        if (warp < M) {
            const float norm = warp_row_norm(A + (size_t)warp * K, K);
            if ((threadIdx.x & 31) == 0) norms[warp] = norm;
        }
        __syncthreads();
    }
    float acc[kGemvRows];
#pragma unroll
    for (uint32_t r = 0; r < kGemvRows; ++r) acc[r] = 0.0f;
    for (uint32_t i0 = slice; i0 < K; i0 += kGemvSlices * 8) {
        fetch(i0 + kGemvSlices * 8, bn);
#pragma unroll
        for (uint32_t t = 0; t < 8; ++t) {
            const uint32_t i = i0 + kGemvSlices * t;
            if (i < K) {
#pragma unroll
                for (uint32_t r = 0; r < kGemvRows; ++r) {
                    if (r < M) {
                        float a = __ldg(A + (size_t)r * K + i);
                        if (normalize) a = __fdiv_rn(a, norms[r]);
                        acc[r] = __fmaf_rn(a, b[t], acc[r]);
                    }
                }
            }
            b[t] = bn[t];
        }
    }
#pragma unroll
    for (uint32_t r = 0; r < kGemvRows; ++r)
        if (r < M) part[slice][r][lc] = acc[r];
    __syncthreads();
    if (threadIdx.x < M * kGemvCols && col < N) {  // thread = (row, column)
        const uint32_t r = threadIdx.x / kGemvCols;
        float s = part[0][r][lc];
        for (uint32_t w = 1; w < kGemvSlices; ++w) s = __fadd_rn(s, part[w][r][lc]);
        C[(size_t)r * N + col] = s;
    }
}

// The GEMM below for batches that would give it fewer than two of its tiles per SM: 32x32 output
// tiles, 4x2 outputs per thread, K step 32 with the next step's loads in flight during the current
// one. Every output is one FMA chain over k in ascending order in both kernels, so they agree bit
// for bit. 515 rows of 200 dims: 14.5 us (45 with the tiles below, 20 CTAs of one round trip per K step),
// 2,048 of 256: 17 (60), 64 of 256: 9.5 (41), 1,000 of 128: 5 (16).
constexpr int SBM = 32, SBN = 32, SBK = 32;

__global__ void __launch_bounds__(128) rotate_sgemm_small_kernel(const float* __restrict__ A,
                                                                 const float* __restrict__ norms,
                                                                 const float* __restrict__ B,
                                                                 float* __restrict__ C, uint32_t M,
                                                                 uint32_t N, uint32_t K) {
    __shared__ __align__(16) float As[2][SBK][SBM + 4];
    __shared__ float Bs[2][SBK][SBN];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t row0 = blockIdx.y * SBM, col0 = blockIdx.x * SBN;
    const uint32_t tr = tid / 16, tc = tid % 16;  // 8 x 16 threads: 4 rows x 2 columns each
    // loads: A rows warp + 4 e (lane = k), B rows warp + 4 e (lane = column)
    float inv[8], a[8], b[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const uint32_t gr = row0 + warp + 4 * e;
        inv[e] = norms && gr < M ? __ldg(norms + gr) : 1.0f;
    }
    auto fetch = [&](uint32_t k0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t gr = row0 + warp + 4 * e, gk = k0 + lane, bk = k0 + warp + 4 * e, gc = col0 + lane;
            a[e] = (gr < M && gk < K) ? __ldg(A + (size_t)gr * K + gk) : 0.0f;
            b[e] = (bk < K && gc < N) ? __ldg(B + (size_t)bk * N + gc) : 0.0f;
        }
    };
    auto stage = [&](int buf) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            As[buf][lane][warp + 4 * e] = norms ? __fdiv_rn(a[e], inv[e]) : a[e];
            Bs[buf][warp + 4 * e][lane] = b[e];
        }
    };
    float acc[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0.0f;
    fetch(0);
    stage(0);
    __syncthreads();
    int buf = 0;
    for (uint32_t k0 = 0; k0 < K; k0 += SBK) {
        const bool more = k0 + SBK < K;
        if (more) fetch(k0 + SBK);
        const uint32_t len = K - k0 < (uint32_t)SBK ? K - k0 : (uint32_t)SBK;
#pragma unroll 8
        for (uint32_t kk = 0; kk < len; ++kk) {
            const float4 av = *reinterpret_cast<const float4*>(&As[buf][kk][tr * 4]);
            const float b0 = Bs[buf][kk][tc], b1 = Bs[buf][kk][tc + 16];
            acc[0][0] = __fmaf_rn(av.x, b0, acc[0][0]);
            acc[0][1] = __fmaf_rn(av.x, b1, acc[0][1]);
            acc[1][0] = __fmaf_rn(av.y, b0, acc[1][0]);
            acc[1][1] = __fmaf_rn(av.y, b1, acc[1][1]);
            acc[2][0] = __fmaf_rn(av.z, b0, acc[2][0]);
            acc[2][1] = __fmaf_rn(av.z, b1, acc[2][1]);
            acc[3][0] = __fmaf_rn(av.w, b0, acc[3][0]);
            acc[3][1] = __fmaf_rn(av.w, b1, acc[3][1]);
        }
        if (more) stage(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t gr = row0 + tr * 4 + i;
        if (gr >= M) continue;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t gc = col0 + tc + 16 * j;
            if (gc < N) C[(size_t)gr * N + gc] = acc[i][j];
        }
    }
}

// C[nq x d] = (A / norm)[nq x d] @ B[d x d]; 128x64 output tile per 256-thread CTA,
// 8x4 outputs per thread, K step 16, double-buffered through shared memory.
constexpr int RBM = 128, RBN = 64, RBK = 16;
constexpr uint32_t kRotateSMs = 148;  // of a B200

__global__ void __launch_bounds__(256) rotate_sgemm_kernel(const float* __restrict__ A,
                                                           const float* __restrict__ norms,
                                                           const float* __restrict__ B,
                                                           float* __restrict__ C, uint32_t M,
                                                           uint32_t N, uint32_t K) {
    __shared__ float As[2][RBK][RBM + 4];
    __shared__ float Bs[2][RBK][RBN];
    const uint32_t tid = threadIdx.x;
    const uint32_t row0 = blockIdx.y * RBM, col0 = blockIdx.x * RBN;
    const uint32_t tr = tid / 16, tc = tid % 16;  // 16 x 16 thread grid: 8 rows x 4 cols each
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    auto load_tile = [&](int buf, uint32_t k0) {
        // A tile: 128 rows x 16 k, 2048 elements, 8 per thread
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t idx = tid + e * 256;
            const uint32_t r = idx / RBK, kk = idx % RBK;
            const uint32_t gr = row0 + r, gk = k0 + kk;
            float v = 0.0f;
            if (gr < M && gk < K) {
                v = A[(size_t)gr * K + gk];
                if (norms) v = __fdiv_rn(v, norms[gr]);
            }
            As[buf][kk][r] = v;
        }
        // B tile: 16 k x 64 cols, 1024 elements, 4 per thread
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const uint32_t idx = tid + e * 256;
            const uint32_t kk = idx / RBN, c = idx % RBN;
            const uint32_t gk = k0 + kk, gc = col0 + c;
            Bs[buf][kk][c] = (gk < K && gc < N) ? B[(size_t)gk * N + gc] : 0.0f;
        }
    };

    int buf = 0;
    load_tile(0, 0);
    __syncthreads();
    for (uint32_t k0 = 0; k0 < K; k0 += RBK) {
        if (k0 + RBK < K) load_tile(buf ^ 1, k0 + RBK);
#pragma unroll
        for (int kk = 0; kk < RBK; ++kk) {
            float a[8], b[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = As[buf][kk][tr * 8 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[buf][kk][tc + 16 * j];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = __fmaf_rn(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t gr = row0 + tr * 8 + i;
        if (gr >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t gc = col0 + tc + 16 * j;
            if (gc < N) C[(size_t)gr * N + gc] = acc[i][j];
        }
    }
}

cudaError_t launch_prepare_queries(const float* q, uint32_t nq, uint32_t d, const float* rotation,
                                   bool normalize, float* norms_ws, float* out, cudaStream_t st) {
    if (nq == 0) return cudaSuccess;
    if (nq <= kGemvRows) {
        rotate_gemv_kernel<<<(d + kGemvCols - 1) / kGemvCols, kGemvSlices * kGemvCols, 0, st>>>(q, normalize, rotation, out,
                                                                                                nq, d, d);
        return cudaGetLastError();
    }
    if (normalize) {
        const uint32_t threads = 256;
        const uint32_t blocks = (nq * 32 + threads - 1) / threads;
        query_norms_kernel<<<blocks, threads, 0, st>>>(q, nq, d, norms_ws);
    }
    const dim3 grid((d + RBN - 1) / RBN, (nq + RBM - 1) / RBM);
    if ((uint64_t)grid.x * grid.y < 2u * kRotateSMs) {
        const dim3 small((d + SBN - 1) / SBN, (nq + SBM - 1) / SBM);
        rotate_sgemm_small_kernel<<<small, 128, 0, st>>>(q, normalize ? norms_ws : nullptr, rotation, out, nq, d, d);
        return cudaGetLastError();
    }
    rotate_sgemm_kernel<<<grid, 256, 0, st>>>(q, normalize ? norms_ws : nullptr, rotation, out, nq,
                                              d, d);
    return cudaGetLastError();
}

}  // namespace pdxg
