// Tree top level for a whole batch (PDXTreeIndex::Search, index.hpp:545-566), tiled.
//
// The top-level search is a pruned F32 PDXearch over the meso clusters, whose "vectors" are
// the L1 centroids, with k = the L1 nprobe. On IVF2 indexes every query reads about half of
// all L1 centroids there (k is large against the few vectors per meso cluster, so the
// ADSampling bound prunes little), and thousands of queries of a batch read the same meso
// clusters. One CTA per query re-reads those centroids from L2 once per query and is bound by
// its load pipe. This form computes the exact per-pair quantities once, with reuse across
// queries, and then replays the reference's decisions on them:
//
//   1. centroid_dist_kernel (pdxg_probe.cu): exact centroid distances in the AVX2 order of
//      Horizontal (searcher.hpp:181-215); meso_list_kernel: the `top` nearest meso clusters per
//      query sorted by (distance, id), and per meso cluster the list of queries that probe it.
//   2. meso_partials_kernel: one CTA per (meso cluster, 128 of its queries, 32 of its
//      vectors). Query rows and cluster blocks are staged in shared memory with cp.async;
//      each thread keeps 4 queries x 4 vectors of FP32 chains in registers, so a staged
//      element feeds four chains. It writes, per (query, vector):
//        * the vertical chain (one fused multiply-add per dimension in dimension order,
//          Vertical of avx2_computers.hpp) at every warmup checkpoint: the cumulative
//          DIMENSIONS_FETCHING_SIZES steps from 0, capped at d_v, the last being d_v;
//        * the sum of every 64-dim horizontal block in the AVX2 order of Horizontal
//          (avx2_computers.hpp:47-98: 8 FMA lanes, lanes j and j + 4 added in double, then
//          pairs, then the total, rounded to float).
//   3. top_replay_kernel: one warp per query replays Start / Warmup / Prune / MergeIntoHeap
//      (searcher.hpp:217-566) on those values, so it takes the same decisions on the same
//      floats as the per-query kernel. A warmup that stops before d_v leaves vertical dims
//      for the vectors that survive every horizontal block; their chains continue from the
//      running distance and are recomputed here from the centroid data, in dimension order.
//      The sorted L1 visit order goes to l1_order for the search kernel.
#include <cfloat>
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "pdxg_block.cuh"
#include "pdxg_common.cuh"

namespace pdxg {

cudaError_t launch_centroid_dist(const float* queries, const uint32_t* q_list, uint32_t nq, uint32_t d,
                                 const float* centroids, uint32_t n, uint32_t* keys, cudaStream_t st);

// -------------------------------------------------------------------------------- probe
// Warp per query, on the distances of centroid_dist_kernel (pdxg_probe.cu): the `m` smallest
// (distance, id) pairs, ascending (the list of LevelOps::probe), the offsets of their partials,
// and the query's entry in the list of each. The entries of a CTA's queries are counted in shared
// memory first, so a meso cluster's counter takes one atomic per CTA: at 10,000 queries x 16 of 32
// clusters one atomic per entry queues 5,000 deep on each counter. Distances and lists were one
// kernel (8 queries x 32 centroids a CTA, one load in flight per thread): 95.6 us for 10,000
// queries x 32 centroids x 1024 dims and 34 us for 512, against 42.7 + 14.8 and 17.8 + 6.1 us.
__global__ void __launch_bounds__(512) meso_list_kernel(const __grid_constant__ TopLevelParams tp) {
    extern __shared__ __align__(16) uint8_t smem[];
    const DevLevel& l0 = tp.l0;
    const uint32_t nc = l0.nclusters, qp = tp.probe_q;
    const uint32_t N = next_pow2(nc);
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem);            // [qp][N]
    uint32_t* count = reinterpret_cast<uint32_t*>(keys + (size_t)qp * N);  // [nc]
    for (uint32_t c = threadIdx.x; c < nc; c += blockDim.x) count[c] = 0;
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t q = blockIdx.x * qp + warp;
    const bool mine = q < tp.nq && !(tp.filter_of && __ldg(tp.filter_of + q) != -1);  // warp-uniform
    uint64_t* kq = keys + (size_t)warp * N;
    uint32_t m = 0;
    if (mine) {
        const uint32_t* src = tp.probe_keys + (size_t)q * nc;
        for (uint32_t c = lane; c < N; c += 32) kq[c] = c < nc ? (((uint64_t)__ldg(src + c) << 32) | c) : ~0ull;
        __syncwarp();
        warp_sort_u64(kq, N);
        const uint32_t topq = tp.q_top ? __ldg(tp.q_top + q) : tp.top;
        m = topq < nc ? topq : nc;
        // offsets: exclusive prefix of nvals * stride over the probe list; the sort key's distance
        // half makes room for the entry's slot among the CTA's entries of that cluster
        uint32_t carry = 0;
        for (uint32_t r0 = 0; r0 < m; r0 += 32) {
            const uint32_t r = r0 + lane;
            const uint32_t c = r < m ? (uint32_t)kq[r] : 0u;
            const uint32_t sz = r < m ? tp.nvals * ((l0.clusters[c].n + 3u) & ~3u) : 0u;
            uint32_t total;
            const uint32_t at = carry + warp_exclusive_scan(sz, total);
            if (r < m) {
                tp.order[(size_t)q * tp.top + r] = c;
                tp.off[(size_t)q * tp.top + r] = at;
                kq[r] = ((uint64_t)atomicAdd(count + c, 1u) << 32) | c;
            }
            carry += total;
        }
    }
    if (q < tp.nq && lane == 0) tp.ntop[q] = m;
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < nc; c += blockDim.x)
        if (count[c]) count[c] = atomicAdd(tp.list_count + c, count[c]);
    __syncthreads();
    for (uint32_t r = lane; r < m; r += 32) {
        const uint32_t c = (uint32_t)kq[r];
        tp.lists[(size_t)c * tp.nq + count[c] + (uint32_t)(kq[r] >> 32)] = q * tp.top + r;
    }
}

// -------------------------------------------------------------------------------- partials
constexpr int kTQ = 128;          // queries per CTA
constexpr int kTV = 32;           // vectors per CTA
constexpr int kTD = 64;           // dimensions per stage
constexpr int kRow = kTD + 4;     // floats per staged row (16-byte aligned; conflict-free columns)
constexpr int kPartialsThreads = 256;

struct PartialsSmem {
    float q[2][kTQ * kRow];       // query rows [slot][dim]
    float x[2][kTV * kRow];       // vertical: [dim][32 vectors]; horizontal: [vector][dim]
    unsigned long long qoff[kTQ]; // float offset of each slot's partials (vals + qoff)
    uint32_t qrow[kTQ];           // query index of each slot
    uint32_t cp[kMaxCheckpoints]; // warmup checkpoints
};

// blockIdx.z: vector tile and part. With one part (large batches) a CTA runs all stages. A small
// batch has too few (cluster, query, vector) tiles to fill the GPU, and the stages are a chain of
// round trips there (about 5 us each): its horizontal blocks, which do not depend on each other or
// on the vertical chains, go to tp.parts - 1 CTAs beside the one that runs the vertical dims.
__global__ void __launch_bounds__(kPartialsThreads, 2) meso_partials_kernel(const __grid_constant__ TopLevelParams tp) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    PartialsSmem& S = *reinterpret_cast<PartialsSmem*>(smem_raw);
    const uint32_t m = blockIdx.y;
    const uint32_t cnt = tp.list_count[m];
    const uint32_t first = blockIdx.x * kTQ;
    if (first >= cnt) return;
    const DevLevel& l0 = tp.l0;
    const DevCluster c = l0.clusters[m];
    const uint32_t part = blockIdx.z % tp.parts;
    const uint32_t v0 = blockIdx.z / tp.parts * kTV;
    if (v0 >= c.n) return;
    const uint32_t n_pad = c.n_pad, stride = (c.n + 3u) & ~3u;
    const uint32_t d = l0.d, dv = l0.dv, nb = l0.n_hblocks, ncp = tp.ncp;
    const uint32_t ntile = (cnt - first) < (uint32_t)kTQ ? (cnt - first) : (uint32_t)kTQ;
    const uint32_t tid = threadIdx.x;
    if (tid < (uint32_t)kMaxCheckpoints) S.cp[tid] = tp.cp[tid];
    if (tid < kTQ) {
        if (tid < ntile) {
            const uint32_t e = tp.lists[(size_t)m * tp.nq + first + tid];
            const uint32_t q = e / tp.top;
            S.qrow[tid] = q;
            S.qoff[tid] = (unsigned long long)q * tp.per_query + tp.off[e];
        } else {
            S.qrow[tid] = 0;
            S.qoff[tid] = 0;
        }
    }
    __syncthreads();

    const float* vert = reinterpret_cast<const float*>(tp.arena + c.vert_off);
    const float* hor = reinterpret_cast<const float*>(tp.arena + c.hor_off);
    const uint32_t nvc = (dv + kTD - 1) / kTD;  // vertical stages
    const uint32_t nst = nvc + nb;
    // this CTA's stages: all; part 0 the vertical ones, parts 1 .. a share of the horizontal blocks each
    const uint32_t s_begin = part == 0 ? 0u : nvc + (part - 1) * nb / (tp.parts - 1);
    const uint32_t s_end = tp.parts == 1 ? nst : (part == 0 ? nvc : nvc + part * nb / (tp.parts - 1));
    if (s_begin == s_end) return;

    // stage s: query dims and the cluster block it covers, into buffer s & 1
    auto issue = [&](uint32_t st) {
        const uint32_t buf = st & 1;
        uint32_t j0, len;
        if (st < nvc) {
            j0 = st * kTD;
            len = (dv - j0) < (uint32_t)kTD ? (dv - j0) : (uint32_t)kTD;
        } else {
            j0 = dv + (st - nvc) * kTD;
            len = kTD;
        }
        const uint32_t n4 = len >> 2;  // float4 per row
        // query rows: 128 slots x 16 float4
#pragma unroll
        for (int t = 0; t < (kTQ * kTD / 4) / kPartialsThreads; ++t) {
            const uint32_t e = tid + t * kPartialsThreads;
            const uint32_t s = e >> 4, c4 = e & 15;
            if (s < ntile && c4 < n4)
                cp_async16(&S.q[buf][s * kRow + c4 * 4], tp.queries + (size_t)S.qrow[s] * d + j0 + c4 * 4);
        }
        if (st < nvc) {
            // vertical rows: len dims x 32 vectors (row stride n_pad: in bounds)
#pragma unroll
            for (int t = 0; t < (kTD * kTV / 4) / kPartialsThreads; ++t) {
                const uint32_t e = tid + t * kPartialsThreads;
                const uint32_t jj = e >> 3, c4 = e & 7;
                if (jj < len) cp_async16(&S.x[buf][jj * kTV + c4 * 4], vert + (size_t)(j0 + jj) * n_pad + v0 + c4 * 4);
            }
        } else {
            // horizontal block rows of the 32 vectors: 32 x 64 floats, contiguous in memory
            const float* hb = hor + ((size_t)(st - nvc) * n_pad + v0) * kHDim;
#pragma unroll
            for (int t = 0; t < (kTV * kTD / 4) / kPartialsThreads; ++t) {
                const uint32_t e = tid + t * kPartialsThreads;
                const uint32_t vv = e >> 4, c4 = e & 15;
                cp_async16(&S.x[buf][vv * kRow + c4 * 4], hb + (size_t)vv * kHDim + c4 * 4);
            }
        }
    };

    const uint32_t lane = tid & 31, warp = tid >> 5;
    const uint32_t vg = lane & 7, qg = lane >> 3;
    // thread tile: query slots slot0 + 4 i (i = 0..3; 4 consecutive rows per warp and load, so
    // distinct banks)
    const uint32_t slot0 = warp * 16 + qg;
    auto slot_ok = [&](int i) { return slot0 + 4 * i < ntile; };
    auto out_row = [&](int i, uint32_t row) { return tp.vals + S.qoff[slot0 + 4 * i] + (size_t)row * stride; };

    issue(s_begin);
    cp_async_commit();
    // Stage st is in buffer st & 1 once this returns; st + 1 is in flight.
    auto begin_stage = [&](uint32_t st) {
        if (st + 1 < s_end) issue(st + 1);
        cp_async_commit();
        cp_async_wait1();
        __syncthreads();
    };

    // vertical dims: one chain per (query, vector), stored at every checkpoint. Vectors
    // 2 vg + {0, 1} and 2 vg + 16 + {0, 1}, each adjacent pair in one packed register; a tile
    // with at most 16 vectors left (a cluster's tail) runs the first half only (NB = 1), as it
    // stores nothing from the second.
    auto vertical = [&](auto nb_tag) {
        constexpr int NB = decltype(nb_tag)::value;
        uint64_t acc[4][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = 0ull;
        uint32_t ck = 0;
        for (uint32_t st = 0; st < nvc; ++st) {
            begin_stage(st);
            const float* qs = S.q[st & 1];
            const float* xs = S.x[st & 1];
            const uint32_t j0 = st * kTD;
            const uint32_t len = (dv - j0) < (uint32_t)kTD ? (dv - j0) : (uint32_t)kTD;
            for (uint32_t jj = 0; jj < len; jj += 4) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    uint64_t qv[4], xv[2];
#pragma unroll
                    for (int i = 0; i < 4; ++i) qv[i] = f32x2_dup(qs[(slot0 + 4 * i) * kRow + jj + u]);
#pragma unroll
                    for (int b = 0; b < NB; ++b)
                        xv[b] = *reinterpret_cast<const uint64_t*>(xs + (jj + u) * kTV + 2 * vg + 16 * b);
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int b = 0; b < NB; ++b) {
                            const uint64_t t = f32x2_sub(qv[i], xv[b]);
                            acc[i][b] = f32x2_fma(t, t, acc[i][b]);
                        }
                }
                if (ck < ncp && j0 + jj + 4 == S.cp[ck]) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int b = 0; b < NB; ++b) {
                            const uint32_t v = v0 + 2 * vg + 16 * b;
                            if (slot_ok(i) && v < stride)
                                *reinterpret_cast<uint64_t*>(out_row(i, ck) + v) = acc[i][b];
                        }
                    ++ck;
                }
            }
            __syncthreads();
        }
    };
    const bool tail = c.n - v0 <= 16u;
    if (part != 0) {
        // another CTA's
    } else if (tail) vertical(std::integral_constant<int, 1>());
    else vertical(std::integral_constant<int, 2>());

    // horizontal blocks: per (query, vector) the AVX2 Horizontal sum of each block. Lanes
    // (j, j + 1) of Horizontal run as one packed chain: dims j + 8 t and j + 1 + 8 t are
    // adjacent in both staged rows. Passes of 4 queries x NB vectors (vg + 16 h, vg + 16 h + 8):
    // a tail tile with at most 16 vectors left runs pass 0 only, with at most 8 left one vector
    // per thread; it stores nothing from the rest.
    auto horizontal = [&](auto nb_tag, int passes) {
        constexpr int NB = decltype(nb_tag)::value;
        for (uint32_t st = s_begin > nvc ? s_begin : nvc; st < s_end; ++st) {
            begin_stage(st);
            const float* qs = S.q[st & 1];
            const float* xs = S.x[st & 1];
            const uint32_t row = ncp + (st - nvc);
#pragma unroll 1
            for (int h = 0; h < passes; ++h) {
                const uint32_t xo0 = (vg + 16 * h) * kRow, xo1 = (vg + 16 * h + 8) * kRow;
                double D0[4][2], D1[4][2], E0[4][2], E1[4][2];
                // lane pairs in the order they combine: (0,1) + (4,5) -> s0, s1; (2,3) + (6,7) -> s2, s3
#pragma unroll 1
                for (int cp2 = 0; cp2 < 4; ++cp2) {
                    const int c2 = ((cp2 & 1) << 2) | ((cp2 >> 1) << 1);  // 0, 4, 2, 6
                    uint64_t a[4][2];
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[i][0] = a[i][1] = 0ull;
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const int dim = c2 + 8 * t;
                        const uint64_t x0 = *reinterpret_cast<const uint64_t*>(xs + xo0 + dim);
                        uint64_t x1 = 0ull;
                        if constexpr (NB == 2) x1 = *reinterpret_cast<const uint64_t*>(xs + xo1 + dim);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint64_t qv = *reinterpret_cast<const uint64_t*>(qs + (slot0 + 4 * i) * kRow + dim);
                            uint64_t tt = f32x2_sub(qv, x0);
                            a[i][0] = f32x2_fma(tt, tt, a[i][0]);
                            if constexpr (NB == 2) {
                                tt = f32x2_sub(qv, x1);
                                a[i][1] = f32x2_fma(tt, tt, a[i][1]);
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int b = 0; b < NB; ++b) {
                            float lo, hi;
                            f32x2_unpack(a[i][b], lo, hi);
                            if (cp2 == 0) {          // lanes 0, 1
                                D0[i][b] = (double)lo;
                                D1[i][b] = (double)hi;
                            } else if (cp2 == 1) {   // lanes 4, 5: s0, s1
                                D0[i][b] = D0[i][b] + (double)lo;
                                D1[i][b] = D1[i][b] + (double)hi;
                            } else if (cp2 == 2) {   // lanes 2, 3
                                E0[i][b] = (double)lo;
                                E1[i][b] = (double)hi;
                            } else {                 // lanes 6, 7: s2, s3
                                E0[i][b] = E0[i][b] + (double)lo;
                                E1[i][b] = E1[i][b] + (double)hi;
                            }
                        }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        const uint32_t v = v0 + vg + 16 * h + 8 * b;
                        if (slot_ok(i) && v < stride)
                            out_row(i, row)[v] = (float)((D0[i][b] + E0[i][b]) + (D1[i][b] + E1[i][b]));
                    }
            }
            __syncthreads();
        }
    };
    if (c.n - v0 <= 8u) horizontal(std::integral_constant<int, 1>(), 1);
    else horizontal(std::integral_constant<int, 2>(), tail ? 1 : 2);
}

// -------------------------------------------------------------------------------- replay
// Bound by the latency of one warp's chain of visits and the instructions on it. So the heap is kept
// in registers once it is full (HR per lane: k <= 32 HR; HR = 0 keeps it in shared memory), a visit's
// cluster record, ids and partials are requested a visit ahead, the bounds of all checkpoints and
// blocks are computed once per visit, one a lane, four warmup steps and four horizontal blocks are
// read together and tested without branches, and a candidate that a merge has ruled out costs
// nothing. 235 us for 10,000 queries (16 of 32 meso clusters of 31 vectors each, k 32) and 61 us for
// 777; 292 and 81 with a bound computed per test and the Starts' order sorted, 344 and 94 with the
// heap in shared memory and everything read at its use.

// The full heap: slot j's distance bits and id in lane j % 32, register j / 32.
template <int HR>
struct TopHeap {
    uint32_t d[HR ? HR : 1], id[HR ? HR : 1];
    float* hd;
    uint32_t* hid;
    __device__ __forceinline__ void load(uint32_t k) {
        const uint32_t lane = threadIdx.x & 31;
        if constexpr (HR > 0) {
#pragma unroll
            for (int r = 0; r < HR; ++r) {
                const uint32_t j = 32 * r + lane;
                // an unused slot is never the lowest slot of the largest key
                d[r] = j < k ? __float_as_uint(hd[j]) : 0u;
                id[r] = j < k ? hid[j] : 0u;
            }
        }
    }
    // largest distance and its lowest slot, on every lane
    __device__ __forceinline__ void top(uint32_t k, float& t, uint32_t& slot) const {
        if constexpr (HR == 0) {
            warp_heap_top(hd, k, t, slot);
        } else {
            const uint32_t lane = threadIdx.x & 31;
            uint32_t best = d[0], bs = lane;
#pragma unroll
            for (int r = 1; r < HR; ++r)
                if (d[r] > best) {
                    best = d[r];
                    bs = 32 * r + lane;
                }
            const uint32_t gmax = __reduce_max_sync(0xffffffffu, best);
            if constexpr (HR == 1) slot = __ffs(__ballot_sync(0xffffffffu, best == gmax)) - 1;
            else slot = __reduce_min_sync(0xffffffffu, best == gmax ? bs : 0xFFFFFFFFu);
            t = __uint_as_float(gmax);
        }
    }
    __device__ __forceinline__ void set(uint32_t slot, float dist, uint32_t row) {
        const uint32_t lane = threadIdx.x & 31;
        if constexpr (HR == 0) {
            if (lane == 0) {
                hd[slot] = dist;
                hid[slot] = row;
            }
            __syncwarp();
        } else {
#pragma unroll
            for (int r = 0; r < HR; ++r)
                if (slot == 32 * r + lane) {
                    d[r] = __float_as_uint(dist);
                    id[r] = row;
                }
        }
    }
    __device__ __forceinline__ void store(uint32_t k) const {
        if constexpr (HR > 0) {
            const uint32_t lane = threadIdx.x & 31;
#pragma unroll
            for (int r = 0; r < HR; ++r) {
                const uint32_t j = 32 * r + lane;
                if (j < k) {
                    hd[j] = __uint_as_float(d[r]);
                    hid[j] = id[r];
                }
            }
            __syncwarp();
        }
    }
};

// Shared memory of the replay: the ratio table (d floats) for the CTA, then per warp
//   sortbuf [r_sort_cap] u64 | pre [2][r_pre_floats] | hd, hid [r_heap_cap] | dist [r_work_cap]
//   | meta [top] x {cluster, partials offset, vectors}
template <int HR>
__global__ void __launch_bounds__(128) top_replay_kernel(const __grid_constant__ TopLevelParams tp) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const DevLevel& l0 = tp.l0;
    const uint32_t d = l0.d, dv = l0.dv, nb = l0.n_hblocks, ncp = tp.ncp;
    float* ratios = reinterpret_cast<float*>(smem);
    for (uint32_t i = threadIdx.x; i < d; i += blockDim.x) ratios[i] = __ldg(tp.ratios + i);
    __syncthreads();  // the only block-wide barrier
    const uint32_t q = blockIdx.x * (blockDim.x >> 5) + warp;
    if (q >= tp.nq) return;  // whole warp
    if (tp.filter_of && __ldg(tp.filter_of + q) != -1) {
        if (lane == 0) tp.l1_count[q] = 0;
        return;
    }
    uint8_t* base = smem + ((size_t)d * 4 + 15) / 16 * 16 + (size_t)warp * tp.r_warp_bytes;
    uint64_t* sortbuf = reinterpret_cast<uint64_t*>(base);
    float* prebuf = reinterpret_cast<float*>(sortbuf + tp.r_sort_cap);
    float* hd = prebuf + 2 * tp.r_pre_floats;
    uint32_t* hid = reinterpret_cast<uint32_t*>(hd + tp.r_heap_cap);
    float* dist = reinterpret_cast<float*>(hid + tp.r_heap_cap);
    uint32_t* meta_c = reinterpret_cast<uint32_t*>(dist + tp.r_work_cap);  // [top] probed meso cluster
    uint32_t* meta_o = meta_c + tp.top;       // [top] offset of its partials
    uint32_t* meta_n = meta_o + tp.top;       // [top] its vectors

    const uint32_t k = tp.q_nprobe ? __ldg(tp.q_nprobe + q) : tp.k1;
    const uint32_t m_top = tp.ntop[q];
    const float* qf = tp.queries + (size_t)q * d;
    const float* qvals = tp.vals + (size_t)q * tp.per_query;
    unsigned long long bytes = (unsigned long long)l0.nclusters * d * 4u;  // centroid probe
    unsigned long long visits = 0;
    auto thr_at = [&](uint32_t cur, float top) {
        const float r = (cur == d) ? 1.0f : ratios[cur];
        return __fmul_rn(top, r);
    };
    for (uint32_t r = lane; r < m_top; r += 32) {
        const uint32_t c = tp.order[(size_t)q * tp.top + r];
        meta_c[r] = c;
        meta_o[r] = tp.off[(size_t)q * tp.top + r];
        meta_n[r] = l0.clusters[c].n;
    }
    __syncwarp();
    // next probed cluster with vectors at or after r (m_top if none)
    auto next_nonempty = [&](uint32_t r) {
        while (r < m_top && meta_n[r] == 0) ++r;
        return r;
    };
    // all partial rows of probed cluster r into buffer `buf`, asynchronously
    auto fetch = [&](uint32_t r, int buf) {
        const uint32_t n4 = tp.nvals * ((meta_n[r] + 3u) & ~3u) / 4;
        const float4* src = reinterpret_cast<const float4*>(qvals + meta_o[r]);
        float* dst = prebuf + (size_t)buf * tp.r_pre_floats;
        for (uint32_t i = lane; i < n4; i += 32) cp_async16(dst + 4 * i, src + i);
        cp_async_commit();
    };
    // cluster record and the ids of its first 32 vectors
    auto first_ids = [&](const DevCluster& c) {
        return lane < c.n ? __ldg(reinterpret_cast<const uint32_t*>(tp.arena + c.ids_off) + lane) : 0u;
    };

    const uint32_t cp_lane = lane < ncp ? tp.cp[lane] : 0u;  // at most 32 checkpoints
    uint32_t hsize = 0, slot = 0;
    float top = 0.0f;
    TopHeap<HR> heap;
    heap.hd = hd;
    heap.hid = hid;
    uint32_t r = next_nonempty(0);
    int buf = 0;
    DevCluster c{}, cn{};
    uint32_t id0 = 0;
    if (r < m_top) {
        fetch(r, 0);
        c = l0.clusters[meta_c[r]];
        id0 = first_ids(c);
    }
    while (r < m_top) {
        const uint32_t rn = next_nonempty(r + 1);
        if (rn < m_top) {
            fetch(rn, buf ^ 1);
            cn = l0.clusters[meta_c[rn]];
            cp_async_wait1();
        } else {
            cp_async_wait0();
        }
        __syncwarp();
        const float* pre = prebuf + (size_t)buf * tp.r_pre_floats;
        const uint32_t n = c.n;
        ++visits;
        const uint32_t stride = (n + 3u) & ~3u;
        const uint32_t* ids = reinterpret_cast<const uint32_t*>(tp.arena + c.ids_off);
        uint32_t id0n = 0;
        if (hsize < k) {
            // Start (searcher.hpp:217-281): full distances, push the best k - |heap| in the
            // order LevelOps::push_smallest uses (below the m-th key by position, then ties)
            bytes += (unsigned long long)n * d * 4u;
            uint32_t lo = 0xFFFFFFFFu, hi = 0;
            for (uint32_t v = lane; v < n; v += 32) {
                float a = pre[(size_t)(ncp - 1) * stride + v];
#pragma unroll 4
                for (uint32_t b = 0; b < nb; ++b) a = __fadd_rn(a, pre[(size_t)(ncp + b) * stride + v]);
                dist[v] = a;
                const uint32_t key = __float_as_uint(a);
                lo = key < lo ? key : lo;
                hi = key > hi ? key : hi;
            }
            __syncwarp();
            const uint32_t mm = (k - hsize) < n ? (k - hsize) : n;
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            uint32_t kth = hi;  // all of them
            if (mm < n) {  // the smallest key with at least mm keys not above it
                while (lo < hi) {
                    const uint32_t mid = lo + (hi - lo) / 2;
                    uint32_t c = 0;
                    for (uint32_t v = lane; v < n; v += 32) c += __float_as_uint(dist[v]) <= mid ? 1u : 0u;
                    if (__reduce_add_sync(0xffffffffu, c) >= mm) hi = mid;
                    else lo = mid + 1;
                }
                kth = lo;
            }
            uint32_t cntp = 0;
            for (int pass = 0; pass < 2; ++pass) {
                for (uint32_t b0 = 0; b0 < n; b0 += 32) {
                    const uint32_t v = b0 + lane;
                    const uint32_t key = v < n ? __float_as_uint(dist[v]) : 0u;
                    const bool sel = v < n && (pass == 0 ? key < kth : key == kth);
                    const unsigned bal = __ballot_sync(0xffffffffu, sel);
                    const uint32_t at = cntp + __popc(bal & ((1u << lane) - 1u));
                    if (sel && at < mm) {
                        hd[hsize + at] = dist[v];
                        hid[hsize + at] = b0 ? __ldg(ids + v) : id0;
                    }
                    cntp += __popc(bal);
                }
            }
            hsize += mm;
            __syncwarp();
            if (hsize >= k) {  // full: from here on only merges change it
                heap.load(k);
                heap.top(k, top, slot);
            }
            if (rn < m_top) id0n = first_ids(cn);
        } else {
            // Warmup (searcher.hpp:374-435): vertical checkpoints until >= ceil(0.8 n) fail the bound,
            // lane s holding the bound of checkpoint s
            const uint32_t needed = (uint32_t)ceilf(__fmul_rn(kSelectivity, (float)n));
            const float thr_cp = lane < ncp ? thr_at(cp_lane, top) : 0.0f;
            uint32_t step = 0;
            for (uint32_t s0 = 0, n_pruned = 0; n_pruned < needed && s0 < ncp; s0 += 4) {
                uint32_t cnt[4] = {0, 0, 0, 0};
                float thr[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) thr[u] = __shfl_sync(0xffffffffu, thr_cp, s0 + u);
                for (uint32_t v = lane; v - lane < n; v += 32) {
                    const float* col = pre + s0 * stride + v;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const bool on = v < n && s0 + u < ncp;
                        const float x = on ? col[u * stride] : 0.0f;
                        cnt[u] += __popc(__ballot_sync(0xffffffffu, on && x >= thr[u]));
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (n_pruned < needed && s0 + u < ncp) {
                        n_pruned = cnt[u];
                        step = s0 + u + 1;
                    }
            }
            const uint32_t cur = __shfl_sync(0xffffffffu, cp_lane, step - 1);
            bytes += (unsigned long long)n * cur * 4u;
            if (rn < m_top) id0n = first_ids(cn);
            // Prune (searcher.hpp:437-540) and MergeIntoHeap (searcher.hpp:542-566). The bound's heap
            // top is the one before the cluster's merges, so each vector's way through the
            // horizontal blocks and the remaining vertical dims depends on that vector alone: each
            // lane follows its own vectors, and the survivors of every step are the same, in the
            // same order, as with the step-by-step compaction.
            const float tc = top;
            // lane b holds the bound after horizontal block b (blocks past 32 read it)
            const float thr_hb = lane < nb ? thr_at(cur + kHDim * (lane + 1), tc) : 0.0f;
            const float* erow = pre + (size_t)(step - 1) * stride;
            const float* vert = reinterpret_cast<const float*>(tp.arena + c.vert_off);
            uint32_t lane_bytes = 0;
            for (uint32_t c0 = 0; c0 < n; c0 += 32) {
                const uint32_t v = c0 + lane;
                const bool in = v < n;
                float dd = in ? erow[v] : 0.0f;
                uint32_t cv = cur;
                bool alive = in && dd < thr_at(cv, tc);
                // four blocks at a time without branches: sums past a lane's failing test are not used
                const float* hrow = pre + ncp * stride + (in ? v : 0u);
                for (uint32_t b0 = 0; b0 < nb && __any_sync(0xffffffffu, alive); b0 += 4) {
                    float x[4], thr[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        x[u] = b0 + u < nb ? hrow[(b0 + u) * stride] : 0.0f;
                        thr[u] = __shfl_sync(0xffffffffu, thr_hb, (b0 + u) & 31);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (b0 + u < nb) {  // uniform
                            if (b0 + u >= 32) thr[u] = thr_at(cur + kHDim * (b0 + u + 1), tc);
                            if (tp.stats) lane_bytes += alive ? kHDim * 4u : 0u;
                            dd = __fadd_rn(dd, x[u]);
                            alive = alive && dd < thr[u];
                        }
                    }
                }
                if (alive) cv = cur + kHDim * nb;
                uint32_t cur_v = cur;
                while (alive && cur_v < dv) {
                    const uint32_t last = (cur_v + kHDim < dv) ? cur_v + kHDim : dv;
                    lane_bytes += (last - cur_v) * 4u;
                    for (uint32_t j = cur_v; j < last; ++j) {
                        const float t = __fsub_rn(__ldg(qf + j), __ldg(vert + (size_t)j * c.n_pad + v));
                        dd = __fmaf_rn(t, t, dd);
                    }
                    cv = (cv + kHDim < d) ? cv + kHDim : d;
                    cur_v = last;
                    alive = dd < thr_at(cv, tc);
                    if (cv == d) break;
                }
                // sequential, strict-<, in position order; the top only falls, so a vector that is
                // not below it once never is
                unsigned bal = __ballot_sync(0xffffffffu, alive && dd < top);
                if (bal) {
                    const uint32_t idv = c0 ? (alive ? __ldg(ids + v) : 0u) : id0;
                    while (bal) {
                        const int i = __ffs(bal) - 1;
                        const float ddi = __shfl_sync(0xffffffffu, dd, i);
                        const uint32_t idi = __shfl_sync(0xffffffffu, idv, i);
                        heap.set(slot, ddi, idi);
                        heap.top(k, top, slot);
                        bal &= bal - 1;
                        bal &= __ballot_sync(0xffffffffu, dd < top);
                    }
                }
            }
            if (tp.stats) bytes += __reduce_add_sync(0xffffffffu, lane_bytes);
        }
        __syncwarp();  // every lane is done with `pre` before the next fetch overwrites it
        r = rn;
        buf ^= 1;
        c = cn;
        id0 = id0n;
    }
    if (hsize >= k) heap.store(k);
    // BuildResultSetFromHeap (searcher.hpp:568-585): the L1 clusters, nearest first
    const uint32_t N = next_pow2(hsize ? hsize : 1);
    for (uint32_t i = lane; i < N; i += 32)
        sortbuf[i] = (i < hsize) ? (((uint64_t)__float_as_uint(hd[i]) << 32) | hid[i]) : ~0ull;
    __syncwarp();
    warp_sort_u64(sortbuf, N);
    uint32_t cnt = hsize;
    if (cnt && __uint_as_float((uint32_t)(sortbuf[cnt - 1] >> 32)) == FLT_MAX) --cnt;
    if (cnt > k) cnt = k;
    for (uint32_t i = lane; i < cnt; i += 32) tp.l1_order[(size_t)q * tp.k1 + i] = (uint32_t)sortbuf[i];
    if (lane == 0) {
        tp.l1_count[q] = cnt;
        if (tp.stats) {
            atomicAdd(tp.stats + 3, bytes);
            atomicAdd(tp.stats, bytes);
            atomicAdd(tp.stats + 1, visits);
        }
    }
}

// -------------------------------------------------------------------------------- launch
size_t partials_smem_bytes() { return sizeof(PartialsSmem); }

// ev (optional, 2 events): recorded after the meso probe and after the partials.
cudaError_t launch_top_level_tiled(const TopLevelParams& tp, uint32_t vtiles, int replay_warps,
                                   cudaStream_t st, const cudaEvent_t* ev) {
    cudaError_t e = cudaMemsetAsync(tp.list_count, 0, sizeof(uint32_t) * tp.l0.nclusters, st);
    if (e != cudaSuccess) return e;
    e = launch_centroid_dist(tp.queries, nullptr, tp.nq, tp.l0.d, tp.l0.centroids, tp.l0.nclusters, tp.probe_keys, st);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(meso_list_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tp.probe_smem);
    if (e != cudaSuccess) return e;
    meso_list_kernel<<<(tp.nq + tp.probe_q - 1) / tp.probe_q, 32 * tp.probe_q, tp.probe_smem, st>>>(tp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[0], st)) != cudaSuccess) return e;
    const int psmem = (int)sizeof(PartialsSmem);
    e = cudaFuncSetAttribute(meso_partials_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, psmem);
    if (e != cudaSuccess) return e;
    dim3 grid((tp.nq + kTQ - 1) / kTQ, tp.l0.nclusters, vtiles * tp.parts);
    meso_partials_kernel<<<grid, kPartialsThreads, psmem, st>>>(tp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[1], st)) != cudaSuccess) return e;
    const size_t rsmem = tp.r_smem;
    // heap registers a lane: k1 (the largest k of the batch) up to 32 or 128
    auto replay = tp.k1 <= 32 ? top_replay_kernel<1> : tp.k1 <= 128 ? top_replay_kernel<4> : top_replay_kernel<0>;
    e = cudaFuncSetAttribute(replay, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem);
    if (e != cudaSuccess) return e;
    replay<<<(tp.nq + replay_warps - 1) / replay_warps, 32 * replay_warps, rsmem, st>>>(tp);
    return cudaGetLastError();
}

}  // namespace pdxg
