// Batched Start (PDXearch::Start, searcher.hpp:217-281), ahead of the scan.
//
// A query's first Start computes the full distance from the query to every vector of the first
// cluster it visits, then keeps the best k; while the heap is not full, the next clusters are
// Starts too (k 100 on clusters of 70 vectors takes two or more). In a batch many queries start in the same cluster,
// and the reference reads that whole cluster once per query. Here the queries of a batch are
// grouped by their first visited cluster and each cluster is read once per group of queries.
// U8 (groups of up to 16): the query-vector dot products run on the integer tensor cores; the
// distances are exact integer sums (no rounding): |q - x|^2 = |q|^2 + |x|^2 - 2 q.x holds
// exactly, so the values equal those of the per-query Start. F32 (groups of up to 8): the
// per-query Start's own chains, in its order. The search kernel then runs push_smallest on them
// (searcher.hpp:256-280) instead of recomputing.
//
//   start_count_kernel : the clusters that fill each unfiltered query's heap (up to sp.visits of
//                        them), counted per cluster; U8: the quantized query, once for the Start
//                        and the scan
//   start_plan_kernel  : one CTA -- per-cluster offsets, each query's row, work items
//   start_dist_kernel  : persistent CTAs over (cluster, <= kStartQ queries, 256 vectors) items,
//                        mma.sync m16n8k32 u8 x u8 -> s32 (a 16 x 8 x 32 tile per instruction)
//   start_f32_kernel   : the same over (cluster, <= kStartQF queries, 64 vectors) items
#include <cstdint>
#include <cuda_runtime.h>

#include "pdxg_block.cuh"
#include "pdxg_common.cuh"

namespace pdxg {

constexpr int kStartQ = 16;        // queries per work item
constexpr int kStartV = 256;       // vectors per work item (one per thread)
constexpr int kStartQF = 8;        // the same for F32 levels
constexpr int kStartVF = 64;
constexpr int kPlanThreads = 1024;

constexpr int kCountThreads = 256;

// Warp per query: lane 0 walks the first visits, all lanes quantize (U8).
__global__ void __launch_bounds__(kCountThreads) start_count_kernel(const __grid_constant__ StartParams sp) {
    const uint32_t q = (blockIdx.x * kCountThreads + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    for (uint32_t i = blockIdx.x * kCountThreads + threadIdx.x; i < sp.n_zero; i += gridDim.x * kCountThreads) sp.zero[i] = 0;
    if (q >= sp.nq) return;
    if (sp.l1.is_u8) {
        const float* qf = sp.queries + (size_t)q * sp.l1.d;
        uint32_t sq = 0;
        for (uint32_t w = lane; w < sp.nwords; w += 32) {
            const uint32_t word = quantize_word(qf, sp.l1, w);
            sp.qwords[(size_t)q * sp.nwords + w] = word;
            sq = __dp4a(word, word, sq);
        }
        sq = __reduce_add_sync(0xffffffffu, sq);
        if (lane == 0) sp.qsq[q] = sq;
    }
    if (lane) return;
    const size_t e0 = (size_t)q * sp.visits;
    for (uint32_t s = 0; s < sp.visits; ++s) {
        sp.row_of[e0 + s] = -1;
        sp.first_cl[e0 + s] = 0xFFFFFFFFu;
    }
    sp.full_at[q] = 0xFFFFFFFFu;
    if (sp.filter_of && sp.filter_of[q] != -1) return;
    const uint32_t cnt = sp.q_order_count[q], k = sp.q_k ? __ldg(sp.q_k + q) : sp.k;
    const uint32_t* ord = sp.q_order + (size_t)q * sp.q_order_stride;
    uint32_t s = 0, have = 0;
    for (uint32_t i = 0; i < cnt && s < sp.visits; ++i) {
        const uint32_t c = ord[i];
        const DevCluster& cl = sp.l1.clusters[c];
        if (cl.live == 0) continue;  // num_embeddings == 0 (searcher.hpp:662)
        sp.first_cl[e0 + s] = c;
        sp.slot_of[e0 + s] = atomicAdd(sp.cl_count + c, 1u);
        ++s;
        have += cl.n;
        if (have >= k) {
            sp.full_at[q] = i;
            return;
        }
    }
}

// Exclusive scan of n values in place with one CTA; returns the total.
__device__ uint32_t cta_exclusive_scan(uint32_t* a, uint32_t n, uint32_t* warp_tot) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < n; b0 += kPlanThreads) {
        const uint32_t i = b0 + threadIdx.x;
        const uint32_t x = i < n ? a[i] : 0u;
        uint32_t incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += t;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t v = warp_tot[lane];
            uint32_t wi = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= (uint32_t)o) wi += t;
            }
            warp_tot[lane] = wi - v;  // exclusive prefix of the warp totals
            if (lane == 31) warp_tot[32] = wi;
        }
        __syncthreads();
        if (i < n) a[i] = carry + warp_tot[warp] + incl - x;
        carry += warp_tot[32];
        __syncthreads();
    }
    return carry;
}

// Row of Start e. More than kPlanRows of them take their own launch: as a loop of the one planning
// CTA (two dependent reads a turn) 10,000 took 34 of its 37 us, 2,000 8 of 13.
constexpr uint32_t kPlanRows = 1024;

__device__ __forceinline__ void start_row(const StartParams& sp, uint32_t e) {
    const uint32_t c = sp.first_cl[e];
    if (c == 0xFFFFFFFFu) return;
    const uint32_t row = sp.cl_off[c] + sp.slot_of[e];
    sp.row_of[e] = (int32_t)row;
    sp.sorted_q[row] = e;
}

__global__ void __launch_bounds__(256) start_rows_kernel(const __grid_constant__ StartParams sp) {
    const uint32_t e = blockIdx.x * 256 + threadIdx.x;
    if (e < sp.nq * sp.visits) start_row(sp, e);
}

__global__ void __launch_bounds__(kPlanThreads) start_plan_kernel(const __grid_constant__ StartParams sp) {
    __shared__ uint32_t warp_tot[33];
    const uint32_t n1 = sp.l1.nclusters;
    const uint32_t iq = sp.l1.is_u8 ? kStartQ : kStartQF, iv = sp.l1.is_u8 ? kStartV : kStartVF;
    // cl_off[c] = first row of cluster c; cl_items[c] = first work item of cluster c
    for (uint32_t c = threadIdx.x; c < n1; c += kPlanThreads) {
        const uint32_t L = sp.cl_count[c];
        sp.cl_off[c] = L;
        const uint32_t nv = sp.l1.clusters[c].n;
        sp.cl_items[c] = L ? ((L + iq - 1) / iq) * ((nv + iv - 1) / iv) : 0u;
    }
    __syncthreads();
    const uint32_t total_rows = cta_exclusive_scan(sp.cl_off, n1, warp_tot);
    const uint32_t total_items = cta_exclusive_scan(sp.cl_items, n1, warp_tot);
    if (sp.nq * sp.visits <= kPlanRows)
        for (uint32_t e = threadIdx.x; e < sp.nq * sp.visits; e += kPlanThreads) start_row(sp, e);
    for (uint32_t c = threadIdx.x; c < n1; c += kPlanThreads) {
        const uint32_t L = sp.cl_count[c];
        if (!L) continue;
        const uint32_t nv = sp.l1.clusters[c].n;
        const uint32_t nqc = (L + iq - 1) / iq, nvc = (nv + iv - 1) / iv;
        uint32_t it = sp.cl_items[c];
        for (uint32_t a = 0; a < nqc; ++a)
            for (uint32_t b = 0; b < nvc; ++b, ++it) {
                sp.items[2 * it] = c;
                sp.items[2 * it + 1] = (a << 16) | b;
            }
    }
    if (threadIdx.x == 0) {
        sp.n_items[0] = total_items;
        sp.n_rows[0] = total_rows;
        sp.queue[0] = 0;
    }
}

// u8 x u8 -> s32 tensor-core product of a 16 x 32 query tile and a 32 x 8 vector tile,
// accumulated into c (exact: every product and partial sum is an integer below 2^31).
__device__ __forceinline__ void mma_u8_16x8x32(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// CTA = one work item: up to 16 queries x 256 vectors of one cluster. Warp w takes vectors
// [32 w, 32 w + 32) as four 8-vector tiles: column n of tile t is vector 4 n + t. The squared
// distance of an integer query q and vector x is |q|^2 + |x|^2 - 2 q.x exactly; q.x runs on the
// tensor cores, |x|^2 with dp4a on the same loaded words.
//
// The kernel reads every started cluster once from HBM and is bound by how that read is asked for.
// A dot product may take its dims in any order, so the k-groups are assigned for 16-byte loads: per
// 64 dims a lane (row gq, k-group gk) takes words 4 gk .. 4 gk + 3 of the query and of the four
// vectors 4 gq .. 4 gq + 3 -- four loads, which for a horizontal block cover 2 KB of contiguous
// memory per warp (word order as the fragments number it took 16 4-byte loads that used half of
// each sector) -- and the next 64 dims are loaded while these are computed. 10,000 queries on 1.02 GB
// of clusters (157 us at the copy rate): 248 us; 288 without the loads ahead, 333 with the 4-byte
// loads and each CTA quantizing its queries; 777 queries 134, 152 and 156.
__device__ __forceinline__ void start_mma_64(int (&acc)[4][4], uint32_t (&xsq)[4], const uint4& a0, const uint4& a1,
                                             const uint4 (&x)[4]) {
    const uint32_t lo[4] = {a0.x, a1.x, a0.y, a1.y}, hi[4] = {a0.z, a1.z, a0.w, a1.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        xsq[t] = __dp4a(x[t].x, x[t].x, xsq[t]);
        xsq[t] = __dp4a(x[t].y, x[t].y, xsq[t]);
        xsq[t] = __dp4a(x[t].z, x[t].z, xsq[t]);
        xsq[t] = __dp4a(x[t].w, x[t].w, xsq[t]);
        mma_u8_16x8x32(acc[t], lo, x[t].x, x[t].y);
        mma_u8_16x8x32(acc[t], hi, x[t].z, x[t].w);
    }
}

__host__ __device__ inline uint32_t start_row_words(uint32_t nwords) {
    return (nwords + 31) / 32 * 32 + 16;  // two rows of a 16-byte fragment load hit distinct banks
}

__global__ void __launch_bounds__(kStartV, 3) start_dist_kernel(const __grid_constant__ StartParams sp) {
    extern __shared__ __align__(16) uint32_t qw[];  // [kStartQ][qs] packed query words
    __shared__ uint32_t item;
    __shared__ uint32_t qsq[kStartQ];
    const DevLevel& lv = sp.l1;
    const uint32_t nwords = sp.nwords, qs = start_row_words(nwords);
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gq = lane >> 2, gk = lane & 3;  // fragment row / k-group of this lane
    const uint32_t* qa0 = qw + gq * qs + 4 * gk;
    const uint32_t* qa1 = qa0 + 8 * qs;
    for (;;) {
        if (threadIdx.x == 0) item = atomicAdd(sp.queue, 1u);
        __syncthreads();
        const uint32_t it = item;
        if (it >= sp.n_items[0]) break;
        const uint32_t c = sp.items[2 * it];
        const uint32_t ab = sp.items[2 * it + 1];
        const uint32_t qa = ab >> 16, vb = ab & 0xFFFFu;
        const uint32_t L = sp.cl_count[c];
        const uint32_t r0 = sp.cl_off[c] + qa * kStartQ;
        const uint32_t nqc = (L - qa * kStartQ) < (uint32_t)kStartQ ? (L - qa * kStartQ) : (uint32_t)kStartQ;
        // the item's query words; rows past nqc and words past the last are zero
        for (uint32_t j = warp; j < kStartQ; j += kStartV / 32) {
            const uint32_t q = j < nqc ? sp.sorted_q[r0 + j] / sp.visits : 0u;
            const uint32_t* src = sp.qwords + (size_t)q * nwords;
            for (uint32_t w = lane; w < qs; w += 32) qw[j * qs + w] = j < nqc && w < nwords ? __ldg(src + w) : 0u;
            if (lane == 0) qsq[j] = j < nqc ? sp.qsq[q] : 0u;
        }
        __syncthreads();
        const DevCluster cl = lv.clusters[c];
        const uint32_t vw = vb * kStartV + warp * 32;  // first vector of this warp; its 32 are inside n_pad
        if (vw < cl.n) {
            int acc[4][4];
            uint32_t xsq[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                xsq[t] = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[t][e] = 0;
            }
            const uint32_t* vert = reinterpret_cast<const uint32_t*>(sp.arena + cl.vert_off) + vw + 4 * gq;
            const uint4* hor = reinterpret_cast<const uint4*>(sp.arena + cl.hor_off) + (size_t)(vw + 4 * gq) * 4 + gk;
            const size_t bstride = (size_t)cl.n_pad * 4;  // 16-byte pieces per block
            // steps of 64 dims: the vertical words, then the horizontal blocks; the next step's loads
            // are in flight while one is computed
            const uint32_t nvs = (lv.n_vwords + 15) >> 4, steps = nvs + lv.n_hblocks;
            auto fetch = [&](uint32_t st, uint4 (&r)[4]) {
                if (st < nvs) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {  // word 16 st + 4 gk + i of the four vectors
                        const uint32_t w = st * 16 + 4 * gk + i;
                        r[i] = w < lv.n_vwords ? __ldg(reinterpret_cast<const uint4*>(vert + (size_t)w * cl.n_pad))
                                               : make_uint4(0u, 0u, 0u, 0u);
                    }
                } else {
                    const uint4* src = hor + (st - nvs) * bstride;
#pragma unroll
                    for (int t = 0; t < 4; ++t) r[t] = __ldg(src + 4 * t);
                }
            };
            auto compute = [&](uint32_t st, const uint4 (&r)[4]) {
                const uint32_t qo = st < nvs ? st * 16 : lv.qw_hoff + (st - nvs) * 16;
                const uint4 a0 = *reinterpret_cast<const uint4*>(qa0 + qo), a1 = *reinterpret_cast<const uint4*>(qa1 + qo);
                if (st < nvs) {
                    const uint4 x[4] = {make_uint4(r[0].x, r[1].x, r[2].x, r[3].x), make_uint4(r[0].y, r[1].y, r[2].y, r[3].y),
                                        make_uint4(r[0].z, r[1].z, r[2].z, r[3].z), make_uint4(r[0].w, r[1].w, r[2].w, r[3].w)};
                    start_mma_64(acc, xsq, a0, a1, x);
                } else {
                    start_mma_64(acc, xsq, a0, a1, r);
                }
            };
            uint4 ra[4], rb[4];
            fetch(0, ra);
            for (uint32_t st = 0; st < steps; st += 2) {
                if (st + 1 < steps) fetch(st + 1, rb);
                compute(st, ra);
                if (st + 1 < steps) {
                    if (st + 2 < steps) fetch(st + 2, ra);
                    compute(st + 1, rb);
                }
            }
            // |x|^2: the four lanes of a row's k-groups hold a quarter each
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                xsq[t] += __shfl_xor_sync(0xffffffffu, xsq[t], 1);
                xsq[t] += __shfl_xor_sync(0xffffffffu, xsq[t], 2);
            }
            // accumulator layout: acc[t][0..1] = (row gq, columns 2 gk, 2 gk + 1), acc[t][2..3] = row
            // gq + 8: over the tiles, four adjacent vectors per column
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t xs[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) xs[t] = __shfl_sync(0xffffffffu, xsq[t], (2 * gk + e) * 4);
                const uint32_t vx = vw + 4 * (2 * gk + e);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t j = gq + 8 * h, qq = qsq[j];
                    if (j < nqc && vx < cl.n)  // rows are a multiple of four long
                        *reinterpret_cast<uint4*>(sp.dist + (size_t)(r0 + j) * sp.stride + vx) =
                            make_uint4(qq + xs[0] - 2u * (uint32_t)acc[0][2 * h + e], qq + xs[1] - 2u * (uint32_t)acc[1][2 * h + e],
                                       qq + xs[2] - 2u * (uint32_t)acc[2][2 * h + e], qq + xs[3] - 2u * (uint32_t)acc[3][2 * h + e]);
                }
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------ F32
constexpr int kStartFD = 64;           // dims per stage
constexpr int kStartFRow = kStartFD + 4;  // floats per staged row: 16-byte reads of 8 rows hit distinct banks
constexpr int kStartFThreads = 128;

struct StartF32Smem {
    float x[2][kStartVF * kStartFRow];  // vertical: [dim][64 vectors]; horizontal: [vector][dim]
    float q[2][kStartQF * kStartFRow];  // [slot][dim]
    uint32_t qrow[kStartQF];
    uint32_t item;
};

// One stage for NQ query slots of a thread (vector v, slots slot0 .. slot0 + NQ - 1): vertical dims
// (one fused multiply-add per dimension, in dimension order) or one horizontal block
// (avx2_computers.hpp:47-98, lanes j and j + 1 as one packed chain), added to acc.
template <int NQ>
__device__ __forceinline__ void start_f32_stage(const float* xs, const float* qs, uint32_t v, uint32_t slot0,
                                                bool vertical, uint32_t len, float (&acc)[4]) {
    if (vertical) {
        for (uint32_t j = 0; j < len; ++j) {
            const float x = xs[j * kStartVF + v];
#pragma unroll
            for (int i = 0; i < NQ; ++i) {
                const float t = __fsub_rn(qs[(slot0 + i) * kStartFRow + j], x);
                acc[i] = __fmaf_rn(t, t, acc[i]);
            }
        }
        return;
    }
    uint64_t a[NQ][4];
#pragma unroll
    for (int i = 0; i < NQ; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) a[i][j] = 0ull;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const ulonglong2 x0 = *reinterpret_cast<const ulonglong2*>(xs + v * kStartFRow + 8 * t);
        const ulonglong2 x1 = *reinterpret_cast<const ulonglong2*>(xs + v * kStartFRow + 8 * t + 4);
        const uint64_t x[4] = {x0.x, x0.y, x1.x, x1.y};
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            const ulonglong2 q0 = *reinterpret_cast<const ulonglong2*>(qs + (slot0 + i) * kStartFRow + 8 * t);
            const ulonglong2 q1 = *reinterpret_cast<const ulonglong2*>(qs + (slot0 + i) * kStartFRow + 8 * t + 4);
            const uint64_t q[4] = {q0.x, q0.y, q1.x, q1.y};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint64_t df = f32x2_sub(q[j], x[j]);
                a[i][j] = f32x2_fma(df, df, a[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        float l[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) f32x2_unpack(a[i][j], l[2 * j], l[2 * j + 1]);
        const double s0 = (double)l[0] + (double)l[4], s1 = (double)l[1] + (double)l[5];
        const double s2 = (double)l[2] + (double)l[6], s3 = (double)l[3] + (double)l[7];
        acc[i] = __fadd_rn(acc[i], (float)((s0 + s2) + (s1 + s3)));
    }
}

// CTA = one work item: up to 8 queries x 64 vectors of one cluster; thread (vector tid & 63, half of
// the queries). A cluster's first visit by a batch reads it from HBM, and with a few queries per
// cluster that is what bounds the kernel, so the 64-dim stages are copied asynchronously, two deep,
// and small enough (39 KB) for five CTAs on an SM to keep 80 KB of copies in flight.
// 138 us for 2,000 queries on 200,000 x 768 (895 clusters, 614 MB: 94 us at the copy rate); the scan
// that begins with it takes 962 us in the per-query kernel, which reads a cluster once per query.
// VEC: d and d_v multiples of 4 and 16-byte aligned queries.
template <bool VEC>
__global__ void __launch_bounds__(kStartFThreads, 5) start_f32_kernel(const __grid_constant__ StartParams sp) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    StartF32Smem& S = *reinterpret_cast<StartF32Smem*>(smem_raw);
    const DevLevel& lv = sp.l1;
    const uint32_t tid = threadIdx.x, v = tid & (kStartVF - 1);
    const uint32_t d = lv.d, dv = lv.dv;
    const uint32_t nvc = (dv + kStartFD - 1) / kStartFD, nst = nvc + lv.n_hblocks;
    for (;;) {
        if (tid == 0) S.item = atomicAdd(sp.queue, 1u);
        __syncthreads();
        const uint32_t it = S.item;
        if (it >= sp.n_items[0]) break;
        const uint32_t c = sp.items[2 * it];
        const uint32_t ab = sp.items[2 * it + 1];
        const uint32_t qa = ab >> 16, v0 = (ab & 0xFFFFu) * kStartVF;
        const uint32_t L = sp.cl_count[c];
        const uint32_t r0 = sp.cl_off[c] + qa * kStartQF;
        const uint32_t nqc = (L - qa * kStartQF) < (uint32_t)kStartQF ? (L - qa * kStartQF) : (uint32_t)kStartQF;
        if (tid < kStartQF) S.qrow[tid] = sp.sorted_q[r0 + (tid < nqc ? tid : 0)] / sp.visits;
        __syncthreads();
        const DevCluster cl = lv.clusters[c];
        const float* vert = reinterpret_cast<const float*>(sp.arena + cl.vert_off);
        const float* hor = reinterpret_cast<const float*>(sp.arena + cl.hor_off);
        auto issue = [&](uint32_t st) {
            float* xb = S.x[st & 1];
            float* qb = S.q[st & 1];
            const bool vs = st < nvc;
            const uint32_t j0 = vs ? st * kStartFD : dv + (st - nvc) * kStartFD;
            const uint32_t len = vs && dv - j0 < (uint32_t)kStartFD ? dv - j0 : (uint32_t)kStartFD;
#pragma unroll
            for (int t = 0; t < kStartVF * kStartFD / 4 / kStartFThreads; ++t) {
                const uint32_t e = tid + t * kStartFThreads, r = e >> 4, c4 = (e & 15) * 4;
                if (vs) {  // dim j0 + r, vectors v0 + c4 ..: rows are n_pad long
                    const bool in = r < len && v0 + c4 < cl.n_pad;
                    cp_async16_zfill(xb + r * kStartVF + c4, vert + (in ? (size_t)(j0 + r) * cl.n_pad + v0 + c4 : 0), in);
                } else {   // vector v0 + r, dims c4 .. of the block
                    const bool in = v0 + r < cl.n_pad;
                    cp_async16_zfill(xb + r * kStartFRow + c4,
                                     hor + (in ? ((size_t)(st - nvc) * cl.n_pad + v0 + r) * kHDim + c4 : 0), in);
                }
            }
            if constexpr (VEC) {
                const uint32_t r = tid >> 4, c4 = (tid & 15) * 4;
                static_assert(kStartQF * kStartFD / 4 == kStartFThreads, "one piece per thread");
                const bool in = r < nqc && c4 < len;
                cp_async16_zfill(qb + r * kStartFRow + c4, sp.queries + (size_t)S.qrow[r] * d + (in ? j0 + c4 : 0), in);
            } else {
                for (uint32_t e = tid; e < kStartQF * kStartFD; e += kStartFThreads) {
                    const uint32_t r = e >> 6, j = e & 63;
                    qb[r * kStartFRow + j] = r < nqc && j < len ? __ldg(sp.queries + (size_t)S.qrow[r] * d + j0 + j) : 0.0f;
                }
            }
        };
        // the two thread halves split the queries: nq2 slots each
        const uint32_t nq2 = (nqc + 1) / 2, slot0 = (tid >> 6) * nq2;
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        issue(0);
        cp_async_commit();
        for (uint32_t st = 0; st < nst; ++st) {
            if (st + 1 < nst) issue(st + 1);
            cp_async_commit();
            cp_async_wait1();
            __syncthreads();
            const bool vs = st < nvc;
            const uint32_t len = vs && dv - st * kStartFD < (uint32_t)kStartFD ? dv - st * kStartFD : (uint32_t)kStartFD;
            const float* xs = S.x[st & 1];
            const float* qs = S.q[st & 1];
            if (nq2 == 1) start_f32_stage<1>(xs, qs, v, slot0, vs, len, acc);
            else if (nq2 == 2) start_f32_stage<2>(xs, qs, v, slot0, vs, len, acc);
            else if (nq2 == 3) start_f32_stage<3>(xs, qs, v, slot0, vs, len, acc);
            else start_f32_stage<4>(xs, qs, v, slot0, vs, len, acc);
            __syncthreads();
        }
        if (v0 + v < cl.n) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if ((uint32_t)i < nq2 && slot0 + i < nqc)
                    sp.dist[(size_t)(r0 + slot0 + i) * sp.stride + v0 + v] = __float_as_uint(acc[i]);
        }
    }
}

static bool start_f32_vec(const StartParams& sp) {
    return sp.l1.d % 4 == 0 && sp.l1.dv % 4 == 0 && ((uintptr_t)sp.queries & 15) == 0;
}

size_t start_dist_smem(const DevLevel& lv) {
    if (!lv.is_u8) return sizeof(StartF32Smem);
    return (size_t)kStartQ * start_row_words(lv.qw_hoff + lv.n_hblocks * 16) * 4;
}

cudaError_t launch_start_batched(const StartParams& sp, int grid, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(sp.cl_count, 0, sizeof(uint32_t) * sp.l1.nclusters, st);
    if (e != cudaSuccess) return e;
    start_count_kernel<<<(sp.nq + kCountThreads / 32 - 1) / (kCountThreads / 32), kCountThreads, 0, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    start_plan_kernel<<<1, kPlanThreads, 0, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (sp.nq * sp.visits > kPlanRows) {
        start_rows_kernel<<<(sp.nq * sp.visits + 255) / 256, 256, 0, st>>>(sp);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    const size_t smem = start_dist_smem(sp.l1);
    if (!sp.l1.is_u8) {
        auto kern = start_f32_vec(sp) ? start_f32_kernel<true> : start_f32_kernel<false>;
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
        kern<<<grid, kStartFThreads, smem, st>>>(sp);
        return cudaGetLastError();
    }
    e = cudaFuncSetAttribute(start_dist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    start_dist_kernel<<<grid, kStartV, smem, st>>>(sp);
    return cudaGetLastError();
}

int start_dist_occupancy(bool u8, size_t smem) {
    int blocks = 0;
    if (!u8) {
        cudaFuncSetAttribute(start_f32_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, start_f32_kernel<true>, kStartFThreads, smem);
        return blocks;
    }
    cudaFuncSetAttribute(start_dist_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, start_dist_kernel, kStartV, smem);
    return blocks;
}

// Starts of one launch at most: an item numbers its query and vector chunks in 16 bits each.
uint64_t start_max_starts(bool u8, uint32_t max_n) {
    const uint32_t iv = u8 ? kStartV : kStartVF;
    return ((uint64_t)max_n + iv - 1) / iv > 65536 ? 0 : 65536ull * (u8 ? kStartQ : kStartQF);
}

// Work items of `starts` Starts at most.
uint64_t start_item_bound(bool u8, uint32_t starts, uint32_t n1, uint32_t max_n) {
    const uint32_t iq = u8 ? kStartQ : kStartQF, iv = u8 ? kStartV : kStartVF;
    return (((uint64_t)starts + iq - 1) / iq + n1) * (((uint64_t)max_n + iv - 1) / iv);
}

}  // namespace pdxg
