// Cluster-major scan: PDXearch (searcher.hpp:217-566) for a whole batch, with the first warmup
// step computed once per cluster for all the queries that visit it. Instantiated for U8 and F32
// levels; "raw" distances are u32 integers or float bits.
//
// Per query, PDXearch visits its clusters in order. The first non-empty ones are Starts (full
// distances, the best pushed) until the heap holds k; every later one runs Warmup: partial distances over the
// vertical dims in steps of 16, 16, 32, ... (DIMENSIONS_FETCHING_SIZES), testing after each step
// how many vectors reach the ADSampling bound thr(top) = top * ratio[dims] (as raw distances)
// and stopping once ceil(0.8 n) do. On the IVF2 SQ8 workloads that exit comes after the first
// step almost always, so most of the scan is the first 16 dims of every vector of every visited
// cluster, one query at a time, each query re-reading the same clusters.
//
// The heap top only falls once the heap is full (MergeIntoHeap replaces the top with a smaller
// distance), and the bound is monotone in it. So the bound a query applies at any later cluster
// is at most tau0, its heap top right after the last Start, and a vector below that later bound at
// the first checkpoint is below the bound at tau0. That set -- the candidates -- is computed
// cluster-major: every cluster's first-checkpoint rows are read once per group of 64 queries and
// each (query, cluster) pair gets a bitmap of its candidates. Then one warp per query replays
// PDXearch in visit order with its true heap top: the vectors below the bound are the
// candidates whose exact first-checkpoint distance is below it, so the warmup's count and its
// survivors are exact; where the warmup would not stop after the first step the warp runs the
// whole warmup itself. Survivors then follow Prune (searcher.hpp:437-540) one per lane and are
// merged in position order (searcher.hpp:542-566), as in the per-query kernel.
//
//   scan_prep_kernel   : warp per query -- the Starts' pushes (the m
//                        smallest batched-Start distances, ties by position) and tau0's bound;
//                        every later visit appended to its cluster's list, with a work item per
//                        8 to 64 list entries; queries this path does not take go to a list for the
//                        per-query kernel
//   scan_bitmap_kernel : a CTA per item: candidate bitmaps over the first checkpoint's dims, with
//                        |q - x|^2 = |q|^2 + |x|^2 - 2 q.x and q.x on the tensor cores (U8 exact;
//                        F32 in TF32 with a margin for its error, so the candidates are a superset
//                        of that set); each visit is classed as empty (no candidate), light (its bitmap kept) or
//                        heavy (so many candidates that its warmup may pass the first step)
//   scan_replay_kernel : the values of all heavy visits, shared out over the GPU's warps; then warp
//                        per query -- Warmup / Prune / MergeIntoHeap / result, over the visits that
//                        are not empty
#include <cfloat>
#include <cstdint>
#include <cuda_runtime.h>

#include "pdxg_block.cuh"
#include "pdxg_common.cuh"

namespace pdxg {

constexpr uint32_t kScanCQ = 64;         // visits per bitmap work item at most
constexpr uint32_t kScanCQMin = 8;
constexpr uint32_t kScanDims = 16;       // dims of the first warmup step at most
constexpr int kBitmapThreads = 128;
constexpr int kScanWarps = 8;            // queries per prep / replay CTA
constexpr uint32_t kOffPath = 0xFFFFFFFFu;
constexpr uint32_t kHeavyBit = 0x80000000u;  // visit class: 0 empty, candidates of a light visit,
                                             // kHeavyBit | 1 + its first column / 32 in hv (0: no
                                             // room) a heavy one
constexpr uint32_t kHeavyPolls = 1u << 20;  // bound of the wait for the heavy values
constexpr uint32_t kHeavyBlocks = 2;  // horizontal blocks of a heavy work unit
constexpr uint32_t kBitmapTileMax = 64 * 1024;  // bytes of a work item's bitmaps in shared memory

// DIMENSIONS_FETCHING_SIZES (common.hpp:47-49)
__constant__ uint32_t c_scan_fetch[kNumFetchSizes] = {16, 16, 32, 32, 32, 32, 64, 64, 64, 64,
                                                     128, 128, 128, 128, 256, 256, 512, 1024, 2048, 16384};

// Visits per bitmap work item of a cluster of n vectors: cluster sizes differ by a factor of ten and
// the largest are visited most, so an item is at most about this many pairs, for its time not to
// stand out at the end of the kernel.
__host__ __device__ __forceinline__ uint32_t scan_chunk(uint32_t n) {
    uint32_t cq = kScanCQ;
    while (cq > kScanCQMin && cq * n > 65536u) cq >>= 1;
    return cq;
}

__device__ __forceinline__ uint32_t sq4(uint32_t a, uint32_t b, uint32_t acc) {
    const uint32_t d = __vabsdiffu4(a, b);
    return __dp4a(d, d, acc);
}

// GetPruningThreshold (searcher.hpp:75-91) for U8: top * ratio[cur] scaled to the raw domain,
// saturating (the same float steps as LevelOps::thr_raw).
__device__ __forceinline__ uint32_t thr_u8(float top, uint32_t cur, const DevLevel& lv, const float* ratios) {
    const float r = (cur == lv.d) ? 1.0f : __ldg(ratios + cur);
    const float scaled = __fmul_rn(__fmul_rn(top, r), lv.scale_sq);
    return scaled >= 4294967296.0f ? 0xFFFFFFFFu : __float2uint_rz(scaled);
}

// Raw distances of a level: their bound, comparisons and reported form. `below` is the pruning
// test, `reached` the warmup's count; a float distance that is not a number is neither.
template <bool U8>
struct Raw {
    static constexpr uint32_t kElem = U8 ? 1u : 4u;  // bytes per dimension
    static __device__ __forceinline__ uint32_t thr(float top, uint32_t cur, const DevLevel& lv, const float* ratios) {
        if constexpr (U8) return thr_u8(top, cur, lv, ratios);
        return __float_as_uint(__fmul_rn(top, (cur == lv.d) ? 1.0f : __ldg(ratios + cur)));
    }
    static __device__ __forceinline__ bool below(uint32_t raw, uint32_t t) {
        return U8 ? raw < t : __uint_as_float(raw) < __uint_as_float(t);
    }
    static __device__ __forceinline__ bool reached(uint32_t raw, uint32_t t) {
        return U8 ? raw >= t : __uint_as_float(raw) >= __uint_as_float(t);
    }
    static __device__ __forceinline__ float reported(uint32_t raw, const DevLevel& lv) {
        return U8 ? __fmul_rn(__uint2float_rn(raw), lv.inv_scale_sq) : __uint_as_float(raw);
    }
    static __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
        return U8 ? a + b : __float_as_uint(__fadd_rn(__uint_as_float(a), __uint_as_float(b)));
    }
    // one more vertical word: 4 U8 dims or one F32 dim
    static __device__ __forceinline__ uint32_t step(uint32_t q, uint32_t x, uint32_t raw) {
        if constexpr (U8) return sq4(q, x, raw);
        const float t = __fsub_rn(__uint_as_float(q), __uint_as_float(x));
        return __float_as_uint(__fmaf_rn(t, t, __uint_as_float(raw)));
    }
    // first word past vertical dim `dim` (U8: the d_v % 4 tail is a zero-padded word)
    static __device__ __forceinline__ uint32_t word(uint32_t dim) { return U8 ? (dim + 3) >> 2 : dim; }
    // words of a horizontal block's vector, and the first of block b in the query's words
    static constexpr uint32_t kHWords = U8 ? 16u : 64u;
    static __device__ __forceinline__ uint32_t hword(const DevLevel& lv, uint32_t b) {
        return (U8 ? lv.qw_hoff : lv.dv) + b * kHWords;
    }
};

// Sum of one horizontal block: `row` its 16-byte pieces, q the query's words of the block (F32: in
// the AVX2 order of avx2_computers.hpp:47-98).
template <bool U8>
__device__ __forceinline__ uint32_t hblock_sum(const uint32_t* q, const uint4* row);

__device__ __forceinline__ uint32_t sq16(const uint4& q, const uint4& x, uint32_t acc) {
    acc = sq4(q.x, x.x, acc);
    acc = sq4(q.y, x.y, acc);
    acc = sq4(q.z, x.z, acc);
    return sq4(q.w, x.w, acc);
}

template <>
__device__ __forceinline__ uint32_t hblock_sum<true>(const uint32_t* q, const uint4* row) {
    uint4 x[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) x[t] = __ldg(row + t);
    const uint4* qh = reinterpret_cast<const uint4*>(q);
    uint32_t sum = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) sum = sq16(qh[t], x[t], sum);
    return sum;
}

template <>
__device__ __forceinline__ uint32_t hblock_sum<false>(const uint32_t* q, const uint4* row) {
    float a[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    uint4 x[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) x[t] = __ldg(row + t);
    const float* qf = reinterpret_cast<const float*>(q);
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const uint32_t xw[4] = {x[t].x, x[t].y, x[t].z, x[t].w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float df = __fsub_rn(qf[4 * t + j], __uint_as_float(xw[j]));
            a[(4 * t + j) & 7] = __fmaf_rn(df, df, a[(4 * t + j) & 7]);
        }
    }
    const double s0 = (double)a[0] + (double)a[4], s1 = (double)a[1] + (double)a[5];
    const double s2 = (double)a[2] + (double)a[6], s3 = (double)a[3] + (double)a[7];
    return __float_as_uint((float)((s0 + s2) + (s1 + s3)));
}

__device__ __forceinline__ void add_stat(const ScanParams& sp, int idx, unsigned long long v) {
    if (v) atomicAdd(sp.stats + idx, v);
}

constexpr float kTf32Keep = 1.0f - 0.001953125f;  // 1 - 2^-9
constexpr float kTf32Tiny = 1e-36f;               // products below the normal range
__device__ __forceinline__ float nan_unless_finite(float x) {
    return fabsf(x) <= FLT_MAX ? x : __int_as_float(0x7fffffff);
}

// ------------------------------------------------------------------------------------ prep
constexpr int kRegKeys = 32;  // Start distances a prep lane keeps in registers (clusters <= 1024)

// The m-th smallest of the n keys (1 <= m <= n): the smallest key with at least m keys not above
// it, found bit by bit between the keys' common prefix and their lowest bit with one count of the
// keys below a trial value per bit.
template <class Key>
__device__ __forceinline__ uint32_t warp_select(uint32_t n, uint32_t m, const Key& key) {
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
    key.for_each(n, [&](uint32_t, uint32_t k) {
        lo = k < lo ? k : lo;
        hi = k > hi ? k : hi;
    });
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lo == hi) return lo;
    const int top = 31 - __clz(lo ^ hi);
    // every key agrees above bit `top`; the answer's bits from there down, high to low
    uint32_t prefix = top == 31 ? 0u : (hi >> (top + 1)) << (top + 1);
    for (int b = top; b >= 0; --b) {
        const uint32_t trial = prefix | (1u << b);
        uint32_t below = 0;
        key.for_each(n, [&](uint32_t, uint32_t k) { below += k < trial ? 1u : 0u; });
        if (__reduce_add_sync(0xffffffffu, below) < m) prefix = trial;
    }
    return prefix;
}

// Start distances held by the lanes: key j of a lane is vector 32 j + lane (all loads issued
// together).
struct RegKeys {
    uint32_t k[kRegKeys];
    __device__ __forceinline__ void load(const uint32_t* src, uint32_t n) {
        const uint32_t lane = threadIdx.x & 31;
#pragma unroll
        for (int j = 0; j < kRegKeys; ++j) {
            const uint32_t v = 32u * j + lane;
            k[j] = v < n ? __ldg(src + v) : 0xFFFFFFFFu;
        }
    }
    template <class F>
    __device__ __forceinline__ void for_each(uint32_t n, F f) const {
        const uint32_t lane = threadIdx.x & 31;
#pragma unroll
        for (int j = 0; j < kRegKeys; ++j)
            if (32u * j + lane < n) f(32u * j + lane, k[j]);
    }
    // f(v0, key of v0 + lane) for the 32-vector chunks v0 = 0, 32, ... below n, in order
    template <class F>
    __device__ __forceinline__ void for_chunks(uint32_t n, F f) const {
#pragma unroll
        for (int j = 0; j < kRegKeys; ++j)
            if (32u * j < n) f(32u * j, k[j]);
    }
};

// Start distances read from global memory (clusters larger than the register form).
struct MemKeys {
    const uint32_t* src;
    template <class F>
    __device__ __forceinline__ void for_each(uint32_t n, F f) const {
        for (uint32_t v = threadIdx.x & 31; v < n; v += 32) f(v, src[v]);
    }
    template <class F>
    __device__ __forceinline__ void for_chunks(uint32_t n, F f) const {
        for (uint32_t v0 = 0; v0 < n; v0 += 32) {
            const uint32_t v = v0 + (threadIdx.x & 31);
            f(v0, v < n ? src[v] : 0xFFFFFFFFu);
        }
    }
};

// Start (searcher.hpp:256-280): the m smallest keys pushed in the order of
// LevelOps::push_smallest -- the keys below the m-th in position order, then the ties at it.
// Returns the m-th key. This form walks all keys; start_push below needs it for long selections.
template <bool U8>
__device__ __noinline__ uint32_t start_push_all(MemKeys key, uint32_t n, uint32_t m, const uint32_t* ids,
                                                const DevLevel& lv, float* hd, uint32_t* hid) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t kth = warp_select(n, m, key);
    uint32_t pushed = 0;
    for (int pass = 0; pass < 2 && pushed < m; ++pass) {
        key.for_chunks(n, [&](uint32_t v0, uint32_t kv) {
            const uint32_t v = v0 + lane;
            const bool sel = pushed < m && v < n && (pass == 0 ? kv < kth : kv == kth);
            const unsigned b = __ballot_sync(0xffffffffu, sel);
            const uint32_t at = pushed + __popc(b & ((1u << lane) - 1u));
            if (sel && at < m) {
                hd[at] = Raw<U8>::reported(kv, lv);
                hid[at] = __ldg(ids + v);
            }
            pushed += __popc(b);
        });
    }
    return kth;
}

// A few counts bring a bound above at least m keys and at most kSelectList of them; those, in
// position order, are all that the selection and the pushes then look at. Selecting over all keys,
// bit by bit and with two passes of ballots, and quantizing the query here, took the warp about
// 9,000 instructions on 1,000 vectors: 200 us for the prep kernel on 10,000 queries, 58 us on 777,
// against 102 and 26.
constexpr uint32_t kSelectList = 128;

template <bool U8, class Key>
__device__ __forceinline__ uint32_t start_push(const Key& key, uint32_t n, uint32_t m, const uint32_t* ids,
                                               const DevLevel& lv, float* hd, uint32_t* hid, uint64_t* list,
                                               const uint32_t* src) {
    const uint32_t lane = threadIdx.x & 31;
    if (m > kSelectList) return start_push_all<U8>(MemKeys{src}, n, m, ids, lv, hd, hid);
    // bound T with m <= #(keys <= T) <= kSelectList, by bisection between the smallest and largest key
    uint32_t T = 0xFFFFFFFFu, cnt = n;
    if (n > kSelectList) {
        uint32_t lo = 0xFFFFFFFFu, hi = 0;
        key.for_each(n, [&](uint32_t, uint32_t k) {
            lo = k < lo ? k : lo;
            hi = k > hi ? k : hi;
        });
        lo = __reduce_min_sync(0xffffffffu, lo);
        T = hi = __reduce_max_sync(0xffffffffu, hi);
        while (cnt > kSelectList && lo < T) {
            const uint32_t mid = lo + (T - lo) / 2;
            uint32_t c = 0;
            key.for_each(n, [&](uint32_t, uint32_t k) { c += k <= mid ? 1u : 0u; });
            c = __reduce_add_sync(0xffffffffu, c);
            if (c >= m) {
                T = mid;
                cnt = c;
            } else {
                lo = mid + 1;
            }
        }
        // more ties at the m-th key than the list holds
        if (cnt > kSelectList) return start_push_all<U8>(MemKeys{src}, n, m, ids, lv, hd, hid);
    }
    uint32_t len = 0;
    key.for_chunks(n, [&](uint32_t v0, uint32_t kv) {
        const bool in = v0 + lane < n && kv <= T;
        const unsigned b = __ballot_sync(0xffffffffu, in);
        if (in) list[len + __popc(b & ((1u << lane) - 1u))] = ((uint64_t)kv << 32) | (v0 + lane);
        len += __popc(b);
    });
    __syncwarp();
    // the list in registers, entry 32 u + lane in register u; rows of the pushes requested already
    constexpr int R = kSelectList / 32;
    uint32_t k[R], id[R];
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
    for (int u = 0; u < R; ++u) {
        const bool in = 32u * u + lane < len;
        const uint64_t e = in ? list[32 * u + lane] : 0ull;
        k[u] = (uint32_t)(e >> 32);
        id[u] = in ? __ldg(ids + (uint32_t)e) : 0u;
        if (in) {
            lo = k[u] < lo ? k[u] : lo;
            hi = k[u] > hi ? k[u] : hi;
        }
    }
    __syncwarp();  // the list may be rewritten by the next Start
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    while (lo < hi) {  // kth in [lo, hi]
        const uint32_t mid = lo + (hi - lo) / 2;
        uint32_t c = 0;
#pragma unroll
        for (int u = 0; u < R; ++u) c += (32u * u + lane < len && k[u] <= mid) ? 1u : 0u;
        if (__reduce_add_sync(0xffffffffu, c) >= m) hi = mid;
        else lo = mid + 1;
    }
    const uint32_t kth = lo;
    uint32_t pushed = 0;
#pragma unroll
    for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const bool sel = 32u * u + lane < len && (pass == 0 ? k[u] < kth : k[u] == kth);
            const unsigned b = __ballot_sync(0xffffffffu, sel);
            const uint32_t at = pushed + __popc(b & ((1u << lane) - 1u));
            if (sel && at < m) {
                hd[at] = Raw<U8>::reported(k[u], lv);
                hid[at] = id[u];
            }
            pushed += __popc(b);
        }
    }
    return kth;
}

template <bool U8>
__global__ void __launch_bounds__(kScanWarps * 32, 3) scan_prep_kernel(const __grid_constant__ ScanParams sp) {
    __shared__ uint64_t list_all[kScanWarps][kSelectList];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t q = blockIdx.x * sp.p_qpc + warp;
    if (q >= sp.nq) return;  // whole warp
    const DevLevel& lv = sp.l1;
    const bool plain = !sp.filter_of || __ldg(sp.filter_of + q) == -1;
    // position of the Start that fills the heap
    const uint32_t fi = plain ? __ldg(sp.full_at + q) : kOffPath;
    const uint32_t kq = sp.q_k ? __ldg(sp.q_k + q) : sp.k;
    if (fi == kOffPath) {
        if (lane == 0) {
            sp.first_i[q] = kOffPath;
            sp.left[atomicAdd(sp.left_n, 1u)] = q;
        }
        return;
    }
    const int32_t* rows = sp.start_row + (size_t)q * sp.start_visits;
    const uint32_t* starts = sp.start_first + (size_t)q * sp.start_visits;
    DevCluster cl = lv.clusters[__ldg(starts)];
    const uint32_t* ord = sp.q_order + (size_t)q * sp.q_order_stride;
    const uint32_t cnt = __ldg(sp.q_order_count + q);
    const uint32_t* src = sp.start_dist + (size_t)__ldg(rows) * sp.start_stride;
    RegKeys rk;
    if (cl.n <= 32u * kRegKeys) rk.load(src, cl.n);  // in flight while the query is quantized
    // |q|^2 over the first checkpoint's dims
    uint32_t qn = 0;
    if constexpr (U8) {
        const uint32_t word = lane < sp.g1 ? __ldg(sp.qwords + (size_t)q * sp.nwords + lane) : 0u;
        qn = __reduce_add_sync(0xffffffffu, __dp4a(word, word, 0u));
    } else {
        const float x = lane < sp.cp1 ? __ldg(sp.queries + (size_t)q * lv.d + lane) : 0.0f;
        float sq = x * x;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        qn = __float_as_uint(sq);
    }
    // every later non-empty visit into its cluster's list; the visit that opens a chunk of
    // scan_chunk list entries also opens the bitmap work item of that chunk. Four visits a lane at a
    // time: each is a chain of three round trips (cluster, size, list slot).
    for (uint32_t i0 = fi + 1 + lane; i0 < cnt; i0 += 128) {
        uint32_t c[4], slot[4], n[4];
        bool on[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) c[u] = i0 + 32 * u < cnt ? __ldg(ord + i0 + 32 * u) : 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            n[u] = i0 + 32 * u < cnt ? lv.clusters[c[u]].n : 0u;
            on[u] = n[u] != 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) slot[u] = on[u] ? atomicAdd(sp.vl_count + c[u], 1u) : 0u;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const uint32_t i = i0 + 32 * u;
            if (i >= cnt) continue;
            if (!on[u]) {  // num_embeddings == 0 (searcher.hpp:662)
                sp.vinfo[(size_t)q * sp.q_order_stride + i] = 0u;
                continue;
            }
            sp.vl[(size_t)c[u] * sp.nq + slot[u]] = q * sp.q_order_stride + i;
            if (slot[u] % scan_chunk(n[u]) == 0) {
                const uint32_t it = atomicAdd(sp.n_items, 1u);
                sp.items[2 * it] = c[u];
                sp.items[2 * it + 1] = slot[u];
            }
        }
    }
    float* hd = sp.heap_d + (size_t)q * sp.k;
    uint32_t* hid = sp.heap_id + (size_t)q * sp.k;
    uint32_t have = 0, top = 0;
    for (uint32_t s = 0;;) {  // the Starts up to the one that fills the heap
        const uint32_t n = cl.n;
        const uint32_t m = kq - have < n ? kq - have : n;
        const uint32_t* ids = reinterpret_cast<const uint32_t*>(sp.arena + cl.ids_off);
        const uint32_t kth = n <= 32u * kRegKeys ? start_push<U8>(rk, n, m, ids, lv, hd + have, hid + have, list_all[warp], src)
                                                 : start_push<U8>(MemKeys{src}, n, m, ids, lv, hd + have, hid + have, list_all[warp], src);
        top = kth > top ? kth : top;
        have += m;
        if (sp.stats && lane == 0) {
            add_stat(sp, 0, (unsigned long long)n * lv.d * Raw<U8>::kElem);
            add_stat(sp, 3 + kStart, (unsigned long long)n * lv.d * Raw<U8>::kElem);
            add_stat(sp, 1, 1ull);
        }
        if (have >= kq) break;
        ++s;
        cl = lv.clusters[__ldg(starts + s)];
        src = sp.start_dist + (size_t)__ldg(rows + s) * sp.start_stride;
        if (cl.n <= 32u * kRegKeys) rk.load(src, cl.n);
    }
    if (lane == 0) {
        // heap top after the pushes: the largest of their last keys; the first checkpoint's bound at it
        const float tau0 = Raw<U8>::reported(top, lv);
        const uint32_t thr = Raw<U8>::thr(tau0, sp.cp1, lv, sp.ratios);
        const long long lim = (long long)thr - (long long)qn;
        if constexpr (U8)
            sp.lim[q] = lim > 0x7FFFFFFFll ? 0x7FFFFFFF : (int32_t)lim;
        else  // scan_bitmap_kernel's margin for the TF32 products
            sp.lim[q] = __float_as_int(nan_unless_finite(__uint_as_float(thr) - __uint_as_float(qn) * kTf32Keep + kTf32Tiny));
        sp.first_i[q] = fi;
    }
}

// ------------------------------------------------------------------------------------ bitmaps
// CTA = one work item: up to 64 visits of one cluster. A warp takes every fourth 32-vector block and
// loops over the item's queries, 16 at a time, with one mma per 8 vectors (U8, m16n8k16) or two
// (TF32, m16n8k8). Column n of tile t is vector 4 n + t of the block, so a lane loads four vectors'
// words with one 16-byte read, and its eight results of a query are the bits 8 gk .. 8 gk + 7 of that
// query's 32-bit word. The words go to the item's bitmaps in shared memory (sp.bm_tile; clusters too
// large for that write all words to global memory). Once the cluster is done the CTA knows every
// visit's candidates: most visits have none, and only the bitmaps of light visits are written out.
//
// An F32 vector is left out only when it surely reaches the bound. The TF32 operands are off by
// 2^-11 of each factor, so q.x by at most 2^-10 |q||x| <= 2^-11 (|q|^2 + |x|^2), which counts twice;
// the test allows 2^-9 (|q|^2 + |x|^2) for that and for the sums' own rounding, and what is not
// finite is a candidate. The replay computes the reference's exact first-step distance of every candidate.
//
// Pairs were computed one query at a time before, with dp4a (U8: 186 us for 310,000 visits of
// 1,000-vector clusters) or the chains in packed FP32 (2 x 16 operations a pair: 171 us for 300
// queries x 895 clusters of 223 vectors, 63 us for 1,000 x 16 of 316): both bound by issue slots.
__device__ __forceinline__ void mma_first(int (&c)[4], const uint32_t (&a)[2], uint32_t b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.s32.u8.u8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%0, %1, %2, %3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(b));
}
__device__ __forceinline__ void mma_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
template <bool U8>
__global__ void __launch_bounds__(kBitmapThreads) scan_bitmap_kernel(const __grid_constant__ ScanParams sp) {
    constexpr uint32_t QS = U8 ? 4 : kScanDims + 4;  // words per staged query: fragment rows hit distinct banks
    constexpr uint32_t kWarps = kBitmapThreads / 32;
    __shared__ __align__(16) uint32_t qd[kScanCQ * QS];
    __shared__ int32_t ql[kScanCQ];
    __shared__ uint32_t qe[kScanCQ];
    __shared__ uint32_t qcnt[kScanCQ];
    extern __shared__ uint32_t tile[];  // [kScanCQ][bm_words | 1]
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gq = lane >> 2, gk = lane & 3;  // fragment row / k-group of this lane
    const uint32_t ts = sp.bm_words | 1u;
    const DevLevel& lv = sp.l1;
    const uint32_t g1 = sp.g1;
    for (uint32_t it = blockIdx.x; it < sp.n_items[0]; it += gridDim.x) {
        const uint32_t c = sp.items[2 * it], first = sp.items[2 * it + 1];
        const uint32_t left = sp.vl_count[c] - first;
        const DevCluster cl = lv.clusters[c];
        const uint32_t n = cl.n, nb = (n + 31) >> 5;
        const uint32_t cq = scan_chunk(n), nqc = left < cq ? left : cq;
        if (threadIdx.x < nqc) {
            const uint32_t e = sp.vl[(size_t)c * sp.nq + first + threadIdx.x];
            qe[threadIdx.x] = e;
            ql[threadIdx.x] = sp.lim[e / sp.q_order_stride];
        }
        if (threadIdx.x < kScanCQ) qcnt[threadIdx.x] = 0;
        __syncthreads();
        for (uint32_t e = threadIdx.x; e < kScanCQ * (U8 ? 4 : kScanDims); e += kBitmapThreads) {
            const uint32_t j = e / (U8 ? 4 : kScanDims), g = e % (U8 ? 4 : kScanDims);
            uint32_t w = 0;
            if (j < nqc && g < g1) w = __ldg(sp.qwords + (size_t)(qe[j] / sp.q_order_stride) * sp.nwords + g);
            qd[j * QS + g] = U8 ? w : to_tf32(__uint_as_float(w));
        }
        __syncthreads();
        const uint32_t* vert = reinterpret_cast<const uint32_t*>(sp.arena + cl.vert_off);
        for (uint32_t blk = warp; blk < nb; blk += kWarps) {
            // words g = gk, gk + 4, ... of vectors 4 gq .. 4 gq + 3 of the block (inside n_pad; what
            // lies past n is masked), and |x|^2 of the vectors of this lane's results
            constexpr int G = U8 ? 1 : 4;
            uint4 x[G];
#pragma unroll
            for (int g = 0; g < G; ++g)
                x[g] = gk + 4 * g < g1
                           ? __ldg(reinterpret_cast<const uint4*>(vert + (size_t)(gk + 4 * g) * cl.n_pad + blk * 32) + gq)
                           : make_uint4(0u, 0u, 0u, 0u);
            uint32_t b[G][4];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                b[g][0] = x[g].x;
                b[g][1] = x[g].y;
                b[g][2] = x[g].z;
                b[g][3] = x[g].w;
            }
            uint32_t xn[2][4];  // [e][t]: vector 4 (2 gk + e) + t
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                uint32_t s;
                if constexpr (U8) {
                    s = __dp4a(b[0][t], b[0][t], 0u);
                    s += __shfl_xor_sync(0xffffffffu, s, 1);
                    s += __shfl_xor_sync(0xffffffffu, s, 2);
                } else {
                    float sf = 0.0f;
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const float xf = __uint_as_float(b[g][t]);
                        sf = fmaf(xf, xf, sf);
                        b[g][t] = to_tf32(xf);
                    }
                    sf += __shfl_xor_sync(0xffffffffu, sf, 1);
                    sf += __shfl_xor_sync(0xffffffffu, sf, 2);
                    s = __float_as_uint(nan_unless_finite(sf * kTf32Keep));
                }
                xn[0][t] = __shfl_sync(0xffffffffu, s, gk * 8);
                xn[1][t] = __shfl_sync(0xffffffffu, s, gk * 8 + 4);
            }
            const uint32_t valid = n - blk * 32 >= 32 ? 0xFFFFFFFFu : (1u << (n - blk * 32)) - 1u;
            for (uint32_t j0 = 0; j0 < nqc; j0 += 16) {
                const uint32_t* q0 = qd + (j0 + gq) * QS + gk;
                const uint32_t* q1 = q0 + 8 * QS;
                uint32_t w0 = 0, w1 = 0;  // this lane's bits of queries j0 + gq and j0 + gq + 8
                if constexpr (U8) {
                    const uint32_t a[2] = {q0[0], q1[0]};
                    const int32_t l0 = ql[j0 + gq], l1 = ql[j0 + gq + 8];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        int d[4] = {0, 0, 0, 0};
                        mma_first(d, a, b[0][t]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {  // |q - x|^2 - |q|^2 against lim
                            if ((int32_t)xn[e][t] - 2 * d[e] < l0) w0 |= 1u << (4 * e + t);
                            if ((int32_t)xn[e][t] - 2 * d[2 + e] < l1) w1 |= 1u << (4 * e + t);
                        }
                    }
                } else {
                    const uint32_t a0[4] = {q0[0], q1[0], q0[4], q1[4]}, a1[4] = {q0[8], q1[8], q0[12], q1[12]};
                    const float l0 = __int_as_float(ql[j0 + gq]), l1 = __int_as_float(ql[j0 + gq + 8]);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                        mma_first(d, a0, b[0][t], b[1][t]);
                        mma_first(d, a1, b[2][t], b[3][t]);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            if (!(fmaf(-2.0f, d[e], __uint_as_float(xn[e][t])) >= l0)) w0 |= 1u << (4 * e + t);
                            if (!(fmaf(-2.0f, d[2 + e], __uint_as_float(xn[e][t])) >= l1)) w1 |= 1u << (4 * e + t);
                        }
                    }
                }
                w0 <<= 8 * gk;
                w1 <<= 8 * gk;
                w0 |= __shfl_xor_sync(0xffffffffu, w0, 1);
                w1 |= __shfl_xor_sync(0xffffffffu, w1, 1);
                w0 |= __shfl_xor_sync(0xffffffffu, w0, 2);
                w1 |= __shfl_xor_sync(0xffffffffu, w1, 2);
                const uint32_t j = j0 + gq + 8 * gk;
                if (gk < 2 && j < nqc) {
                    const uint32_t word = (gk ? w1 : w0) & valid;
                    uint32_t* row = sp.bm_tile ? tile + j * ts : sp.bm + (size_t)qe[j] * sp.bm_words;
                    row[blk] = word;
                    if (word) atomicAdd(&qcnt[j], (uint32_t)__popc(word));
                }
            }
        }
        __syncthreads();
        // class of every visit of the item; a warmup can pass its first step only when fewer than
        // ceil(0.8 n) vectors reach the bound, and the candidates hold every vector below it
        const uint32_t needed = (uint32_t)ceilf(__fmul_rn(kSelectivity, (float)n));
        if (threadIdx.x < nqc) {
            const uint32_t cnt = qcnt[threadIdx.x];
            uint32_t info = cnt;
            if (sp.stats) add_stat(sp, 12, cnt);
            if (sp.cp1 < lv.dv && n - cnt < needed) {
                // columns are handed out in units of 32; none is asked for once they are used up, so
                // the counter stays far from its range
                info = kHeavyBit;
                const uint32_t cap = sp.hv_cap / 32;
                if (__ldcg(sp.hv_alloc) < cap) {
                    const uint32_t col = atomicAdd(sp.hv_alloc, nb);
                    const bool fits = col + nb <= cap;
                    if (fits) info |= col + 1;
                    for (uint32_t b = 0; b < nb && col + b < cap; ++b) {
                        sp.hv_blk[2 * (col + b)] = fits ? qe[threadIdx.x] : 0xFFFFFFFFu;
                        sp.hv_blk[2 * (col + b) + 1] = b;
                    }
                }
            }
            sp.vinfo[qe[threadIdx.x]] = info;
            qcnt[threadIdx.x] = info;
        }
        __syncthreads();
        if (sp.bm_tile) {
            for (uint32_t j = warp; j < nqc; j += kWarps) {
                const uint32_t info = qcnt[j];
                if (info == 0 || (info & kHeavyBit)) continue;
                for (uint32_t w = lane; w < nb; w += 32) sp.bm[(size_t)qe[j] * sp.bm_words + w] = tile[j * ts + w];
            }
        }
        __syncthreads();  // the next item overwrites the arrays
    }
}

// ------------------------------------------------------------------------------------ replay
// Per-warp shared memory: qw [nwords] | hd, hid [r_heap_cap] | area [r_area_bytes] (candidate
// offsets as u16, or the final sort) | sbits [bm_words] survivor bitmap of one cluster |
// sv_pos, sv_d [r_surv_cap] the survivors of a first warmup step and their distances.
struct ReplayWarp {
    uint32_t* qw;
    float* hd;
    uint32_t* hid;
    uint16_t* cand;
    uint64_t* sortbuf;
    uint32_t* sbits;
    uint32_t* sv_pos;
    uint32_t* sv_d;
};

// candidates a replay lane tests per memory round trip
template <bool U8>
constexpr int kCandPerLane = U8 ? 4 : 2;
constexpr int kFallPerLane = 4;  // vectors a replay lane carries through a full warmup step

// The vertical dims from cur0 on in 64-dim steps for a vector below every bound up to `cur` (the
// horizontal blocks included), tested after each step.
template <bool U8>
__device__ __forceinline__ bool scan_follow_vertical(const ScanParams& sp, const DevCluster& c, const uint32_t* qw,
                                                     uint32_t v, uint32_t cur0, uint32_t cur, float top, uint32_t& raw,
                                                     unsigned long long& vbytes) {
    const DevLevel& lv = sp.l1;
    const uint32_t* vert = reinterpret_cast<const uint32_t*>(sp.arena + c.vert_off);
    uint32_t cur_v = cur0;
    while (cur_v < lv.dv) {
        const uint32_t last = (cur_v + kHDim < lv.dv) ? cur_v + kHDim : lv.dv;
        vbytes += (last - cur_v) * Raw<U8>::kElem;
        const uint32_t g_end = Raw<U8>::word(last);
        for (uint32_t g0 = U8 ? cur_v >> 2 : cur_v; g0 < g_end; g0 += 8) {
            uint32_t x[8];
#pragma unroll
            for (int t = 0; t < 8; ++t) x[t] = g0 + t < g_end ? __ldg(vert + (size_t)(g0 + t) * c.n_pad + v) : 0u;
#pragma unroll
            for (int t = 0; t < 8; ++t)
                if (g0 + t < g_end) raw = Raw<U8>::step(qw[g0 + t], x[t], raw);
        }
        cur = (cur + kHDim < lv.d) ? cur + kHDim : lv.d;
        cur_v = last;
        if (!Raw<U8>::below(raw, Raw<U8>::thr(top, cur, lv, sp.ratios))) return false;
        if (cur == lv.d) break;
    }
    return true;
}

// 16-byte pieces of vector v's row in horizontal block b.
template <bool U8>
__device__ __forceinline__ const uint4* hblock_row(const ScanParams& sp, const DevCluster& c, uint32_t b, uint32_t v) {
    return reinterpret_cast<const uint4*>(sp.arena + c.hor_off) + ((size_t)b * c.n_pad + v) * (Raw<U8>::kHWords / 4);
}

// One survivor of the warmup bound at checkpoint cur0: the horizontal blocks, then the
// remaining vertical dims in 64-dim steps, tested after each against the bound of the heap top
// `top` fixed for the whole cluster (searcher.hpp:437-540). Returns whether it is still below
// the bound at the end; raw is its running distance.
template <bool U8>
__device__ __forceinline__ bool scan_follow(const ScanParams& sp, const DevCluster& c, const uint32_t* qw,
                                            uint32_t v, uint32_t cur0, float top, uint32_t& raw,
                                            unsigned long long& hbytes, unsigned long long& vbytes) {
    const DevLevel& lv = sp.l1;
    uint32_t cur = cur0;
    for (uint32_t b = 0; b < lv.n_hblocks; ++b) {
        raw = Raw<U8>::add(raw, hblock_sum<U8>(qw + Raw<U8>::hword(lv, b), hblock_row<U8>(sp, c, b, v)));
        hbytes += kHDim * Raw<U8>::kElem;
        cur += kHDim;
        if (!Raw<U8>::below(raw, Raw<U8>::thr(top, cur, lv, sp.ratios))) return false;
    }
    return scan_follow_vertical<U8>(sp, c, qw, v, cur0, cur, top, raw, vbytes);
}

// Positions of the set bits of one word per lane (word index w_rel of a group of 32 words),
// ascending, as offsets from the group's first vector into cand; returns their number.
__device__ __forceinline__ uint32_t scan_bits_to_offsets(uint32_t word, uint32_t w_rel, uint16_t* cand) {
    uint32_t total;
    uint32_t at = warp_exclusive_scan(__popc(word), total);
    while (word) {
        const uint32_t bit = __ffs(word) - 1;
        word &= word - 1;
        cand[at++] = (uint16_t)(w_rel * 32 + bit);
    }
    __syncwarp();
    return total;
}

// Whether a vector with full distance `full` may stay below bound `thr` at all d dims. F32 leaves
// room for another order of the sum: its d + 1 non-negative terms are each rounded at most d + 2
// times by 2^-24 in either order (2^-22 d is twice the difference that allows).
template <bool U8>
__device__ __forceinline__ bool may_stay_below(uint32_t full, uint32_t thr, uint32_t d) {
    if constexpr (U8) return full < thr;
    const float t = __uint_as_float(thr);
    return !(__uint_as_float(full) > t + t * ((float)(d + 16) * 2.384185791015625e-7f));
}

// A heavy visit needs the running distance of all its vectors at up to every warmup checkpoint and
// then a long survivor path for most of them. These values do not depend on the query's heap: row
// s < ncp of a vector's column in hv is its running distance at warmup checkpoint s, row ncp + b the
// sum of horizontal block b, and hv_full their sum over all dims. One query in eight has such a visit
// (1M x 1024 SQ8 tree) but the few with three of them set the time when their own CTA computed them
// (a walk ends after 10 us on average, the last after 77), so every 32-vector block of every
// heavy visit is split into units -- its vertical chain, and a few horizontal blocks each -- that all
// warps of the grid share. Replay of 777 queries 79 -> 48 us, of 10,000 137 -> 103, F32 2,000 queries
// on 200,000 x 768 225 -> 150, 300 exhaustive ones 170 -> 117.
// Units are claimed from a counter, so each is run by a warp that is on the GPU, and a walk that needs
// the values (heavy_ready) waits for units that are running; it gives up after a bounded number of
// polls and then runs its warmups itself.
// hv_full adds the units in any order: exact for U8; F32 readers allow for it (may_stay_below).
template <bool U8>
__device__ __forceinline__ void heavy_unit(const ScanParams& sp, uint32_t cb, uint32_t part) {
    const DevLevel& lv = sp.l1;
    const uint32_t lane = threadIdx.x & 31, nhb = lv.n_hblocks;
    const uint32_t e = sp.hv_blk[2 * cb], v = sp.hv_blk[2 * cb + 1] * 32 + lane;
    if (e == 0xFFFFFFFFu) return;
    const DevCluster c = lv.clusters[__ldg(sp.q_order + e)];
    if (v < c.n) {
        const uint32_t* qw = sp.qwords + (size_t)(e / sp.q_order_stride) * sp.nwords;
        uint32_t* out = sp.hv + ((size_t)cb << 5) + lane;
        uint32_t sum = 0;
        if (part == 0) {
            const uint32_t* col = reinterpret_cast<const uint32_t*>(sp.arena + c.vert_off) + v;
            const uint32_t groups = Raw<U8>::word(lv.dv);
            constexpr int NL = U8 ? 16 : 32;  // words in flight
            uint32_t s = 0, next = sp.cp1;
            for (uint32_t g0 = 0; g0 < groups; g0 += NL) {
                uint32_t x[NL];
#pragma unroll
                for (int t = 0; t < NL; ++t) x[t] = g0 + t < groups ? __ldg(col + (size_t)(g0 + t) * c.n_pad) : 0u;
#pragma unroll
                for (int t = 0; t < NL; ++t) {
                    if (g0 + t < groups) {
                        sum = Raw<U8>::step(__ldg(qw + g0 + t), x[t], sum);
                        if ((g0 + t + 1) * (U8 ? 4 : 1) >= next) {  // checkpoints: multiples of 16 dims, then d_v
                            out[(size_t)s * sp.hv_cap] = sum;
                            ++s;
                            next += c_scan_fetch[s < kNumFetchSizes ? s : kNumFetchSizes - 1];
                            if (next > lv.dv) next = lv.dv;
                        }
                    }
                }
            }
        } else {
            const uint32_t b0 = (part - 1) * kHeavyBlocks;
            out += (size_t)(sp.hv_ncp + b0) * sp.hv_cap;
            constexpr int NB = (int)kHeavyBlocks;
            if constexpr (U8) {
                uint4 x[NB][4];
#pragma unroll
                for (int k = 0; k < NB; ++k)
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        x[k][t] = b0 + k < nhb ? __ldg(hblock_row<U8>(sp, c, b0 + k, v) + t) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int k = 0; k < NB; ++k) {
                    if (b0 + k < nhb) {
                        const uint4* qh = reinterpret_cast<const uint4*>(qw + Raw<U8>::hword(lv, b0 + k));
                        uint32_t h = 0;
#pragma unroll
                        for (int t = 0; t < 4; ++t) h = sq16(__ldg(qh + t), x[k][t], h);
                        out[(size_t)k * sp.hv_cap] = h;
                        sum += h;
                    }
                }
            } else {
                for (uint32_t k = 0; k < NB && b0 + k < nhb; ++k) {
                    const uint32_t h = hblock_sum<U8>(qw + Raw<U8>::hword(lv, b0 + k), hblock_row<U8>(sp, c, b0 + k, v));
                    out[(size_t)k * sp.hv_cap] = h;
                    sum = Raw<U8>::add(sum, h);
                }
            }
        }
        uint32_t* full = sp.hv_full + ((size_t)cb << 5) + lane;
        if constexpr (U8) atomicAdd(full, sum);
        else atomicAdd(reinterpret_cast<float*>(full), __uint_as_float(sum));
    }
}

// Runs claimed units until none is left; returns their number.
template <bool U8>
__device__ __forceinline__ uint32_t heavy_units(const ScanParams& sp) {
    const uint32_t cap = sp.hv_cap / 32, got = sp.hv_alloc[0];
    const uint32_t blocks = got < cap ? got : cap;
    const uint32_t parts = 1 + (sp.l1.n_hblocks + kHeavyBlocks - 1) / kHeavyBlocks;
    const uint32_t total = blocks * parts;
    // units of a claim: a grid has up to 3,552 warps, so with a few units for each of them a claim of
    // four leaves warps idle, and with many the counter's atomics queue. Replay with claims of 1 and of 4:
    // 10,000 queries on the 1M x 1024 SQ8 tree 133 and 108 us, 300 exhaustive F32 ones 119 and 166,
    // 1,000 F32 ones on 316 clusters 37 and 53.
    const uint32_t chunk = total > 8192u ? 4u : 1u;
    for (;;) {
        uint32_t u = 0;
        if (total && (threadIdx.x & 31) == 0) u = atomicAdd(sp.hv_next, chunk);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= total) return total;
        const uint32_t end = u + chunk < total ? u + chunk : total;
        for (uint32_t x = u; x < end; ++x) heavy_unit<U8>(sp, x % blocks, x / blocks);
        __threadfence();  // every lane's values before the warp's count
        __syncwarp();
        if ((threadIdx.x & 31) == 0) atomicAdd(sp.hv_done, end - u);
    }
}

// Whether all `total` units are done, after a bounded wait.
__device__ __forceinline__ bool heavy_ready(const ScanParams& sp, uint32_t total) {
    uint32_t done = 0;
    for (uint32_t i = 0; i < kHeavyPolls; ++i) {
        done = *reinterpret_cast<volatile uint32_t*>(sp.hv_done);
        if (done >= total) break;
        __nanosleep(100);
    }
    __threadfence();
    return __all_sync(0xffffffffu, done >= total);
}

template <bool U8>
__global__ void __launch_bounds__(kScanWarps * 32, U8 ? 3 : 2) scan_replay_kernel(const __grid_constant__ ScanParams sp) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // Queries that start in the same cluster visit the same ones next: with one Start a query they run at
    // the same time, in neighbouring CTAs. (Batches with several Starts a query run in their order; no
    // difference was measured on indexes whose clusters L2 holds.)
    // warps past r_qpc own no query (no shared-memory region either) and only run heavy units
    const uint32_t units = heavy_units<U8>(sp);
    uint32_t q = warp < sp.r_qpc ? blockIdx.x + warp * gridDim.x : 0xFFFFFFFFu;
    if (sp.by_start) q = q < sp.nq && q < __ldg(sp.n_by_start) ? __ldg(sp.by_start + q) : 0xFFFFFFFFu;
    const uint32_t fi = q < sp.nq ? sp.first_i[q] : kOffPath;
    const DevLevel& lv = sp.l1;
    uint8_t* base = smem + (size_t)warp * sp.r_warp_bytes;
    ReplayWarp R;
    R.qw = reinterpret_cast<uint32_t*>(base);
    R.hd = reinterpret_cast<float*>(base + ((size_t)sp.nwords * 4 + 15) / 16 * 16);
    R.hid = reinterpret_cast<uint32_t*>(R.hd + sp.r_heap_cap);
    R.cand = reinterpret_cast<uint16_t*>(R.hid + sp.r_heap_cap);
    R.sortbuf = reinterpret_cast<uint64_t*>(R.cand);
    R.sbits = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(R.cand) + sp.r_area_bytes);
    R.sv_pos = R.sbits + (sp.bm_words + 3) / 4 * 4;
    R.sv_d = R.sv_pos + sp.r_surv_cap;
    const uint32_t stride = sp.q_order_stride;
    const uint32_t* ord = sp.q_order + (size_t)q * stride;
    const uint32_t* vis = sp.vinfo + (size_t)q * stride;
    const uint32_t kq = fi == kOffPath ? 0u : (sp.q_k ? __ldg(sp.q_k + q) : sp.k);
    const uint32_t cnt = fi == kOffPath ? 0u : __ldg(sp.q_order_count + q);
    float top = 0.0f;
    uint32_t slot = 0;
    if (fi == kOffPath) return;  // whole warp; there is no block-wide barrier
    for (uint32_t w = lane; w < sp.nwords; w += 32) R.qw[w] = __ldg(sp.qwords + (size_t)q * sp.nwords + w);
    for (uint32_t j = lane; j < kq; j += 32) {
        R.hd[j] = __ldg(sp.heap_d + (size_t)q * sp.k + j);
        R.hid[j] = __ldg(sp.heap_id + (size_t)q * sp.k + j);
    }
    __syncwarp();
    warp_heap_top(R.hd, kq, top, slot);
    uint32_t* scratch = sp.start_dist + (size_t)__ldg(sp.start_row + (size_t)q * sp.start_visits) * sp.start_stride;
    const uint32_t S = sp.r_surv_cap;
    unsigned long long b_warm = 0, b_h = 0, b_v = 0, merged = 0;
    unsigned long long n_surv = 0, n_fast = 0, n_full = 0;
    unsigned long long b_warm_l = 0;  // per lane: the first step of every visit
    uint32_t visits_l = 0, fast_l = 0;

    // Merges the warp's vectors that stayed below every bound (alive), in lane order
    // (MergeIntoHeap, searcher.hpp:542-566).
    auto merge = [&](const DevCluster& c, bool alive, uint32_t v, uint32_t raw) {
        const uint32_t idv = alive ? __ldg(reinterpret_cast<const uint32_t*>(sp.arena + c.ids_off) + v) : 0u;
        const float dd = Raw<U8>::reported(raw, lv);
        merged += __popc(__ballot_sync(0xffffffffu, alive));
        // the top only falls: a vector that is not below it once never is
        unsigned bal = __ballot_sync(0xffffffffu, alive && dd < top);
        while (bal) {
            const int l = __ffs(bal) - 1;
            const float ddl = __shfl_sync(0xffffffffu, dd, l);
            const uint32_t idl = __shfl_sync(0xffffffffu, idv, l);
            if (lane == 0) {
                R.hd[slot] = ddl;
                R.hid[slot] = idl;
            }
            __syncwarp();
            warp_heap_top(R.hd, kq, top, slot);
            bal &= bal - 1;
            bal &= __ballot_sync(0xffffffffu, dd < top);
        }
    };

    // Follows the lane's survivor (alive, v, raw) through Prune with the bound at `tp`, then merges.
    auto prune_merge = [&](const DevCluster& c, bool alive, uint32_t v, uint32_t raw, uint32_t cur, float tp) {
        if (alive) alive = scan_follow<U8>(sp, c, R.qw, v, cur, tp, raw, b_h, b_v);
        merge(c, alive, v, raw);
    };
    // A heavy visit on its values computed ahead; col: its first vector's column. A vector can only be
    // merged when its full distance is below the bound at all d dims: a visit without any changes
    // nothing. Its reads are batched, eight blocks' full distances and four steps of four blocks.
    auto heavy_visit = [&](const DevCluster& c, size_t col) {
        const uint32_t n = c.n, W = (n + 31) >> 5;
        const uint32_t* hv = sp.hv + col;
        const uint32_t* full = sp.hv_full + col;
        const float tp = top;  // the bound's heap top, fixed for the whole cluster
        const uint32_t thr_d = Raw<U8>::thr(tp, lv.d, lv, sp.ratios);
        uint32_t any = 0;
        for (uint32_t w0 = 0; w0 < W; w0 += 8) {
            uint32_t x[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = (w0 + u) * 32 + lane < n ? __ldcg(full + (w0 + u) * 32 + lane) : 0u;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                // statistics count the blocks of vectors that end up pruned too
                const unsigned may = __ballot_sync(0xffffffffu, (w0 + u) * 32 + lane < n &&
                                                                    (sp.stats || may_stay_below<U8>(x[u], thr_d, lv.d)));
                any |= may;
                if (lane == 0 && w0 + u < W) R.sbits[w0 + u] = may;
            }
        }
        if (!any) return;
        __syncwarp();
        const uint32_t* bmh = R.sbits;
        const uint32_t needed = (uint32_t)ceilf(__fmul_rn(kSelectivity, (float)n));
        uint32_t cur = 0, step = 0, n_pruned = 0;
        while (n_pruned < needed && cur < lv.dv) {  // Warmup (searcher.hpp:374-435), four steps at a time
            uint32_t last[4], thr[4], cnt[4];
            uint32_t at = cur;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                at += c_scan_fetch[step + g < (uint32_t)kNumFetchSizes ? step + g : kNumFetchSizes - 1];
                if (at > lv.dv) at = lv.dv;
                last[g] = at;
                thr[g] = Raw<U8>::thr(tp, at, lv, sp.ratios);
                cnt[g] = 0;
            }
            const uint32_t* row = hv + (size_t)step * sp.hv_cap;
            for (uint32_t v0 = 0; v0 < n; v0 += 128) {
                uint32_t x[4][4];
#pragma unroll
                for (int g = 0; g < 4; ++g)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const uint32_t v = v0 + 32 * u + lane;
                        x[g][u] = v < n && step + g < sp.hv_ncp ? __ldcg(row + (size_t)g * sp.hv_cap + v) : 0u;
                    }
#pragma unroll
                for (int g = 0; g < 4; ++g)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        cnt[g] += (v0 + 32 * u + lane < n && Raw<U8>::reached(x[g][u], thr[g])) ? 1u : 0u;
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (n_pruned < needed && cur < lv.dv) {
                    n_pruned = __reduce_add_sync(0xffffffffu, cnt[g]);
                    if (cur == 0) n_surv += n - n_pruned;
                    else b_warm += (unsigned long long)n * (last[g] - cur) * Raw<U8>::kElem;
                    cur = last[g];
                    ++step;
                }
            }
        }
        if (step == 1) ++n_fast;
        else ++n_full;
        // Prune (searcher.hpp:437-540) and merge of the mergeable vectors, 32 at a time in position
        // order; their horizontal sums are loaded six at a time, ahead of their tests
        constexpr int HB = 6;
        const uint32_t thr = Raw<U8>::thr(tp, cur, lv, sp.ratios);
        const uint32_t* erow = hv + (size_t)(step - 1) * sp.hv_cap;
        const uint32_t* brow = hv + (size_t)sp.hv_ncp * sp.hv_cap;
        for (uint32_t w0 = 0; w0 < W; w0 += 32) {
            const uint32_t total = scan_bits_to_offsets(w0 + lane < W ? bmh[w0 + lane] : 0u, lane, R.cand);
            for (uint32_t j0 = 0; j0 < total; j0 += 32) {
                bool alive = j0 + lane < total;
                const uint32_t v = alive ? w0 * 32 + R.cand[j0 + lane] : 0u;
                uint32_t raw = alive ? __ldcg(erow + v) : 0u;
                alive = alive && Raw<U8>::below(raw, thr);
                uint32_t cv = cur;
                for (uint32_t b0 = 0; b0 < lv.n_hblocks && __any_sync(0xffffffffu, alive); b0 += HB) {
                    uint32_t x[HB];
#pragma unroll
                    for (int u = 0; u < HB; ++u)
                        x[u] = (alive && b0 + u < lv.n_hblocks) ? __ldcg(brow + (size_t)(b0 + u) * sp.hv_cap + v) : 0u;
#pragma unroll
                    for (int u = 0; u < HB; ++u) {
                        if (alive && b0 + u < lv.n_hblocks) {
                            raw = Raw<U8>::add(raw, x[u]);
                            b_h += kHDim * Raw<U8>::kElem;
                            cv += kHDim;
                            alive = Raw<U8>::below(raw, Raw<U8>::thr(tp, cv, lv, sp.ratios));
                        }
                    }
                }
                if (alive) alive = scan_follow_vertical<U8>(sp, c, R.qw, v, cur, cv, tp, raw, b_v);
                merge(c, alive, v, raw);
            }
            __syncwarp();  // cand is rewritten by the next word group
        }
    };

    // Visits without a candidate end their warmup at the first step with no survivor (n >= 0.8 n
    // vectors reach the bound): only the others are walked. On the 1M x 1024 SQ8 tree a query has
    // one or two of them in 31 visits, and walking all of them was a chain of 31 record and bitmap
    // round trips.
    uint32_t info_next = 0;
    {
        const uint32_t il = ((fi + 1) & ~31u) + lane;
        if (il > fi && il < cnt) info_next = __ldg(vis + il);
    }
    for (uint32_t i0 = (fi + 1) & ~31u; i0 < cnt; i0 += 32) {
      const uint32_t il = i0 + lane;
      const bool in = il > fi && il < cnt;
      const uint32_t info_l = info_next;
      info_next = il + 32 < cnt ? __ldg(vis + il + 32) : 0u;  // in flight during these visits
      if (sp.stats && in) {
          const uint32_t n = lv.clusters[__ldg(ord + il)].n;
          visits_l += n ? 1u : 0u;
          b_warm_l += (unsigned long long)n * sp.cp1 * Raw<U8>::kElem;
          fast_l += (n && info_l == 0) ? 1u : 0u;
      }
      for (unsigned todo = __ballot_sync(0xffffffffu, info_l != 0); todo; todo &= todo - 1) {
        const uint32_t src = __ffs(todo) - 1, i = i0 + src;
        const uint32_t info = __shfl_sync(0xffffffffu, info_l, src);
        const DevCluster c = lv.clusters[__ldg(ord + i)];
        if ((info & kHeavyBit) && (info & ~kHeavyBit) && heavy_ready(sp, units)) {
            heavy_visit(c, (size_t)((info & ~kHeavyBit) - 1) << 5);
            continue;
        }
        const uint32_t n = c.n;
        const uint32_t* vert = reinterpret_cast<const uint32_t*>(sp.arena + c.vert_off);
        const uint32_t W = (n + 31) >> 5;
        const uint32_t needed = (uint32_t)ceilf(__fmul_rn(kSelectivity, (float)n));
        const uint32_t* bmp = sp.bm + ((size_t)q * stride + i) * sp.bm_words;
        // Warmup step 1 from the candidates: the exact first-checkpoint distance of each, and the
        // survivors under the current bound, in position order
        const uint32_t thr1 = Raw<U8>::thr(top, sp.cp1, lv, sp.ratios);
        uint32_t ns = 0, open = 0;  // below the bound; not reaching it (F32: not a number, too)
        const bool light = !(info & kHeavyBit);  // a heavy visit keeps no bitmap
        for (uint32_t w0 = 0; light && w0 < W; w0 += 32) {
            const uint32_t w = w0 + lane;
            const uint32_t word = w < W ? __ldg(bmp + w) : 0u;
            const uint32_t total = scan_bits_to_offsets(word, lane, R.cand);
            constexpr int CP = kCandPerLane<U8>;
            constexpr int GW = U8 ? 4 : (int)kScanDims;  // words of the first step at most
            for (uint32_t j0 = 0; j0 < total; j0 += 32 * CP) {
                uint32_t v[CP], x[CP][GW];
#pragma unroll
                for (int u = 0; u < CP; ++u) {
                    const uint32_t j = j0 + 32 * u + lane;
                    v[u] = j < total ? w0 * 32 + R.cand[j] : 0xFFFFFFFFu;
                    const bool in = v[u] != 0xFFFFFFFFu;
                    const uint32_t* col = vert + (in ? v[u] : 0u);
#pragma unroll
                    for (int g = 0; g < GW; ++g)
                        x[u][g] = (in && (uint32_t)g < sp.g1) ? __ldg(col + (size_t)g * c.n_pad) : 0u;
                }
#pragma unroll
                for (int u = 0; u < CP; ++u) {
                    uint32_t d1 = 0;
#pragma unroll
                    for (int g = 0; g < GW; ++g)
                        if ((uint32_t)g < sp.g1) d1 = Raw<U8>::step(R.qw[g], x[u][g], d1);
                    const bool in = v[u] != 0xFFFFFFFFu;
                    const bool s = in && Raw<U8>::below(d1, thr1);
                    const unsigned bal = __ballot_sync(0xffffffffu, s);
                    const uint32_t r = ns + __popc(bal & ((1u << lane) - 1u));
                    if (s && r < S) {
                        R.sv_pos[r] = v[u];
                        R.sv_d[r] = d1;
                    }
                    ns += __popc(bal);
                    if constexpr (U8) open = ns;
                    else open += __popc(__ballot_sync(0xffffffffu, in && !Raw<U8>::reached(d1, thr1)));
                }
            }
            __syncwarp();
        }
        const bool exits = sp.cp1 >= lv.dv || n - open >= needed;  // the warmup stops after step 1
        const float tp = top;  // the bound's heap top, fixed for the whole cluster
        n_surv += ns;
        if (light && exits && ns <= S) {
            ++n_fast;
            // Prune and MergeIntoHeap of the survivors, 32 at a time in position order
            for (uint32_t g0 = 0; g0 < ns; g0 += 32) {
                const uint32_t j = g0 + lane;
                const bool alive = j < ns;
                prune_merge(c, alive, alive ? R.sv_pos[j] : 0u, alive ? R.sv_d[j] : 0u, sp.cp1, tp);
            }
            continue;
        }
        // the warmup continues past its first step (or keeps more survivors than the list
        // holds): the whole Warmup (searcher.hpp:374-435) over every vector, the running
        // distances in the query's scratch row
        ++n_full;
        uint32_t cur = 0, step = 0, n_pruned = 0;
        while (n_pruned < needed && cur < lv.dv) {
            uint32_t last = cur + c_scan_fetch[step < kNumFetchSizes ? step : kNumFetchSizes - 1];
            if (last > lv.dv) last = lv.dv;
            const uint32_t thr = Raw<U8>::thr(top, last, lv, sp.ratios);
            const uint32_t g0 = U8 ? cur >> 2 : cur, g_end = Raw<U8>::word(last);
            uint32_t cntp = 0;
            for (uint32_t v0 = 0; v0 < n; v0 += 32 * kFallPerLane) {
                uint32_t acc[kFallPerLane];
#pragma unroll
                for (int u = 0; u < kFallPerLane; ++u) {
                    const uint32_t v = v0 + 32 * u + lane;
                    acc[u] = (v < n && cur > 0) ? scratch[v] : 0u;
                }
                for (uint32_t g = g0; g < g_end; g += 4) {
                    uint32_t xs[4][kFallPerLane];
#pragma unroll
                    for (int gg = 0; gg < 4; ++gg)
#pragma unroll
                        for (int u = 0; u < kFallPerLane; ++u) {
                            const uint32_t v = v0 + 32 * u + lane;
                            xs[gg][u] = (v < n && g + gg < g_end) ? __ldg(vert + (size_t)(g + gg) * c.n_pad + v) : 0u;
                        }
#pragma unroll
                    for (int gg = 0; gg < 4; ++gg) {
                        const uint32_t qv = g + gg < g_end ? R.qw[g + gg] : 0u;  // past the end: adds 0
#pragma unroll
                        for (int u = 0; u < kFallPerLane; ++u) acc[u] = Raw<U8>::step(qv, xs[gg][u], acc[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < kFallPerLane; ++u) {
                    const uint32_t v = v0 + 32 * u + lane;
                    if (v < n) {
                        scratch[v] = acc[u];
                        cntp += Raw<U8>::reached(acc[u], thr) ? 1u : 0u;
                    }
                }
            }
            n_pruned = __reduce_add_sync(0xffffffffu, cntp);
            if (cur > 0) b_warm += (unsigned long long)n * (last - cur) * Raw<U8>::kElem;
            else if (!light) n_surv += n - n_pruned;
            cur = last;
            ++step;
        }
        // Prune: the vectors below the bound at the warmup's last checkpoint, in position order
        const uint32_t thr = Raw<U8>::thr(top, cur, lv, sp.ratios);
        for (uint32_t v0 = 0; v0 < n; v0 += 32) {
            const uint32_t v = v0 + lane;
            const unsigned bal = __ballot_sync(0xffffffffu, v < n && Raw<U8>::below(scratch[v], thr));
            if (lane == 0) R.sbits[v0 >> 5] = bal;
        }
        __syncwarp();
        for (uint32_t w0 = 0; w0 < W; w0 += 32) {
            const uint32_t w = w0 + lane;
            const uint32_t total = scan_bits_to_offsets(w < W ? R.sbits[w] : 0u, lane, R.cand);
            for (uint32_t j0 = 0; j0 < total; j0 += 32) {
                const uint32_t j = j0 + lane;
                const bool alive = j < total;
                const uint32_t v = alive ? w0 * 32 + R.cand[j] : 0u;
                prune_merge(c, alive, v, alive ? scratch[v] : 0u, cur, tp);
            }
            __syncwarp();  // cand is rewritten by the next word group
        }
      }
    }
    // BuildResultSetFromHeap (searcher.hpp:568-585)
    const uint32_t N = next_pow2(kq);
    for (uint32_t j = lane; j < N; j += 32)
        R.sortbuf[j] = j < kq ? (((uint64_t)__float_as_uint(R.hd[j]) << 32) | R.hid[j]) : ~0ull;
    __syncwarp();
    warp_sort_u64(R.sortbuf, N);
    uint32_t hs = kq;
    if (__uint_as_float((uint32_t)(R.sortbuf[hs - 1] >> 32)) == FLT_MAX) --hs;
    uint32_t* oi = sp.out_ids + (size_t)q * sp.k;
    float* od = sp.out_dists + (size_t)q * sp.k;
    for (uint32_t j = lane; j < sp.k; j += 32) {
        if (j < hs) {
            const uint64_t e = R.sortbuf[j];
            oi[j] = (uint32_t)e;
            od[j] = __uint_as_float((uint32_t)(e >> 32));
        } else {
            oi[j] = 0xFFFFFFFFu;
            od[j] = __int_as_float(0x7f800000);
        }
    }
    if (lane == 0) sp.out_counts[q] = hs;
    if (sp.stats) {
        const unsigned long long h = __reduce_add_sync(0xffffffffu, (uint32_t)b_h);
        const unsigned long long vv = __reduce_add_sync(0xffffffffu, (uint32_t)b_v);
        const uint32_t visits = __reduce_add_sync(0xffffffffu, visits_l);
        n_fast += __reduce_add_sync(0xffffffffu, fast_l);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) b_warm_l += __shfl_xor_sync(0xffffffffu, b_warm_l, o);
        b_warm += b_warm_l;
        if (lane == 0) {
            add_stat(sp, 0, b_warm + h + vv);
            add_stat(sp, 3 + kWarmup, b_warm);
            add_stat(sp, 3 + kSurvivorH, h);
            add_stat(sp, 3 + kSurvivorV, vv);
            add_stat(sp, 1, visits);
            add_stat(sp, 2, merged);
            add_stat(sp, 13, n_surv);
            add_stat(sp, 14, n_fast);
            add_stat(sp, 15, n_full);
        }
    }
}

// ------------------------------------------------------------------------------------ launch
uint64_t scan_item_bound(uint32_t nq, uint32_t stride, uint32_t n1, uint32_t max_n) {
    return (uint64_t)nq * stride / scan_chunk(max_n) + n1 + 1;
}

// Shared memory of a bitmap work item's tile; 0: the bitmaps of clusters this large go straight
// to global memory.
size_t scan_bitmap_smem(uint32_t bm_words) {
    const size_t b = (size_t)kScanCQ * (bm_words | 1u) * 4;
    return b <= kBitmapTileMax ? b : 0;
}

uint32_t scan_queries_per_cta() { return kScanWarps; }

template <bool U8>
static cudaError_t launch_scan_t(const ScanParams& sp, cudaStream_t st, const cudaEvent_t* ev) {
    cudaError_t e;
    const uint32_t ctas = (sp.nq + sp.p_qpc - 1) / sp.p_qpc;
    scan_prep_kernel<U8><<<ctas, sp.p_qpc * 32, 0, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[0], st)) != cudaSuccess) return e;
    const size_t tile = scan_bitmap_smem(sp.bm_words);
    if (tile) {
        e = cudaFuncSetAttribute(scan_bitmap_kernel<U8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile);
        if (e != cudaSuccess) return e;
    }
    scan_bitmap_kernel<U8><<<sp.item_bound < 8192 ? sp.item_bound : 8192, kBitmapThreads, tile, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[1], st)) != cudaSuccess) return e;
    const size_t smem = (size_t)sp.r_qpc * sp.r_warp_bytes;
    e = cudaFuncSetAttribute(scan_replay_kernel<U8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    scan_replay_kernel<U8><<<(sp.nq + sp.r_qpc - 1) / sp.r_qpc, kScanWarps * 32, smem, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[2], st)) != cudaSuccess) return e;
    return cudaSuccess;
}

// ev (optional, 3 events): recorded after the prep kernel, the bitmaps and the replay.
cudaError_t launch_scan(const ScanParams& sp, cudaStream_t st, const cudaEvent_t* ev) {
    return sp.l1.is_u8 ? launch_scan_t<true>(sp, st, ev) : launch_scan_t<false>(sp, st, ev);
}

}  // namespace pdxg
