// Cluster-major scan of U8 levels: PDXearch (searcher.hpp:217-566) for a whole batch, with the
// first warmup step computed once per cluster for all the queries that visit it.
//
// Per query, PDXearch visits its clusters in order. The first non-empty one is a Start (full
// distances, the best k pushed); every later one runs Warmup: partial distances over the
// vertical dims in steps of 16, 16, 32, ... (DIMENSIONS_FETCHING_SIZES), testing after each step
// how many vectors reach the ADSampling bound thr(top) = top * ratio[dims] (as U8 raw distances)
// and stopping once ceil(0.8 n) do. On the IVF2 SQ8 workloads that exit comes after the first
// step almost always, so most of the scan is the first 16 dims of every vector of every visited
// cluster, one query at a time, each query re-reading the same clusters.
//
// The heap top only falls once the heap is full (MergeIntoHeap replaces the top with a smaller
// distance), and the bound is monotone in it. So the bound a query applies at any later cluster
// is at most tau0, its heap top right after the Start, and a vector below that later bound at
// the first checkpoint is below the bound at tau0. That set -- the candidates -- is computed
// cluster-major: every cluster's first-checkpoint rows are read once per group of 64 queries and
// each (query, cluster) pair gets a bitmap of its candidates. Then one warp per query replays
// PDXearch in visit order with its true heap top: the vectors below the bound are the
// candidates whose exact first-checkpoint distance is below it, so the warmup's count and its
// survivors are exact; where the warmup would not stop after the first step the warp runs the
// whole warmup itself. Survivors then follow Prune (searcher.hpp:437-540) one per lane and are
// merged in position order (searcher.hpp:542-566), as in the per-query kernel.
//
//   scan_prep_kernel   : warp per query -- quantized query words, the Start's pushes (the m
//                        smallest batched-Start distances, ties by position) and tau0's bound;
//                        every later visit appended to its cluster's list, with a work item per
//                        64 list entries; queries this path does not take go to a list for the
//                        per-query kernel
//   scan_bitmap_kernel : persistent CTAs over the items: candidate bitmaps with dp4a, exact
//                        |q - x|^2 = |q|^2 + |x|^2 - 2 q.x over the first checkpoint's dims; each
//                        visit is classed as empty (no candidate), light (its bitmap kept) or
//                        heavy (so many candidates that its warmup may pass the first step)
//   scan_replay_kernel : warp per query -- Warmup / Prune / MergeIntoHeap / result, over the
//                        visits that are not empty; the heavy visits of a CTA's queries are
//                        first computed by all its warps together
#include <cfloat>
#include <cstdint>
#include <cuda_runtime.h>

#include "pdxg_block.cuh"
#include "pdxg_common.cuh"

namespace pdxg {

constexpr uint32_t kScanCQ = 64;         // visits per bitmap work item
constexpr int kBitmapThreads = 256;
constexpr int kBitmapBPW = 4;            // 32-vector blocks a bitmap warp holds at once
constexpr int kScanWarps = 8;            // queries per prep / replay CTA
constexpr uint32_t kOffPath = 0xFFFFFFFFu;
constexpr uint32_t kHeavyBit = 0x80000000u;  // visit class: 0 empty, candidates of a light visit,
                                             // kHeavyBit a heavy one
constexpr uint32_t kHeavyList = 64;      // heavy visits a replay CTA computes ahead
constexpr uint32_t kBitmapTileMax = 64 * 1024;  // bytes of a work item's bitmaps in shared memory

// DIMENSIONS_FETCHING_SIZES (common.hpp:47-49)
__constant__ uint32_t c_scan_fetch[kNumFetchSizes] = {16, 16, 32, 32, 32, 32, 64, 64, 64, 64,
                                                     128, 128, 128, 128, 256, 256, 512, 1024, 2048, 16384};

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

__device__ __forceinline__ float reported_u8(uint32_t raw, const DevLevel& lv) {
    return __fmul_rn(__uint2float_rn(raw), lv.inv_scale_sq);
}

__device__ __forceinline__ void add_stat(const ScanParams& sp, int idx, unsigned long long v) {
    if (v) atomicAdd(sp.stats + idx, v);
}

// ------------------------------------------------------------------------------------ prep
constexpr int kRegKeys = 32;  // Start distances a prep lane keeps in registers (clusters <= 1024)

// The m-th smallest of the n keys key(v) (exact radix select, 8 bits a pass; hist: 256 words of
// this warp's shared memory).
template <class Key>
__device__ __forceinline__ uint32_t warp_radix_select(uint32_t n, uint32_t m, uint32_t* hist, Key key) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t prefix = 0, mask = 0, rem = m;
    for (int shift = 24; shift >= 0; shift -= 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) hist[lane * 8 + j] = 0;
        __syncwarp();
        key.for_each(n, [&](uint32_t, uint32_t k) {
            if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1u);
        });
        __syncwarp();
        uint32_t loc[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            loc[j] = hist[lane * 8 + j];
            sum += loc[j];
        }
        uint32_t tot;
        const uint32_t excl = warp_exclusive_scan(sum, tot);
        const unsigned own = __ballot_sync(0xffffffffu, excl < rem && rem <= excl + sum);
        const uint32_t owner = __ffs(own) - 1;
        uint32_t bin = 0, cum = excl;
        if (lane == owner) {
            int b = 0;
            for (; b < 7; ++b) {
                if (cum + loc[b] >= rem) break;
                cum += loc[b];
            }
            bin = lane * 8 + b;
        }
        bin = __shfl_sync(0xffffffffu, bin, owner);
        cum = __shfl_sync(0xffffffffu, cum, owner);
        prefix |= bin << shift;
        mask |= 0xFFu << shift;
        rem -= cum;
        __syncwarp();
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
// Returns the m-th key.
template <class Key>
__device__ __forceinline__ uint32_t start_push(const Key& key, uint32_t n, uint32_t m, uint32_t* hist,
                                               const uint32_t* ids, const DevLevel& lv, float* hd, uint32_t* hid) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t kth = warp_radix_select(n, m, hist, key);
    uint32_t pushed = 0;
    for (int pass = 0; pass < 2 && pushed < m; ++pass) {
        key.for_chunks(n, [&](uint32_t v0, uint32_t kv) {
            const uint32_t v = v0 + lane;
            const bool sel = pushed < m && v < n && (pass == 0 ? kv < kth : kv == kth);
            const unsigned b = __ballot_sync(0xffffffffu, sel);
            const uint32_t at = pushed + __popc(b & ((1u << lane) - 1u));
            if (sel && at < m) {
                hd[at] = reported_u8(kv, lv);
                hid[at] = __ldg(ids + v);
            }
            pushed += __popc(b);
        });
    }
    return kth;
}

// Dynamic shared memory: the warps' query rows (prep_qs set: kScanWarps x d floats), staged
// with one coalesced pass; without it the query is read from global memory.
__global__ void __launch_bounds__(kScanWarps * 32) scan_prep_kernel(const __grid_constant__ ScanParams sp) {
    __shared__ uint32_t hist_all[kScanWarps][256];
    extern __shared__ __align__(16) float qs_all[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t q = blockIdx.x * kScanWarps + warp;
    if (q >= sp.nq) return;  // whole warp
    uint32_t* hist = hist_all[warp];
    const DevLevel& lv = sp.l1;
    const bool plain = !sp.filter_of || __ldg(sp.filter_of + q) == -1;
    const int32_t row = plain ? __ldg(sp.start_row + q) : -1;
    const uint32_t kq = sp.q_k ? __ldg(sp.q_k + q) : sp.k;
    auto leave = [&]() {
        if (lane == 0) {
            sp.first_i[q] = kOffPath;
            sp.left[atomicAdd(sp.left_n, 1u)] = q;
        }
    };
    if (row < 0) {
        leave();
        return;
    }
    const uint32_t first = __ldg(sp.start_first + q);
    const DevCluster cl = lv.clusters[first];
    const uint32_t n = cl.n;
    const uint32_t m = kq < n ? kq : n;
    if (m < kq) {  // the heap is not full after the Start: the next cluster is a Start too
        leave();
        return;
    }
    // position of the Start cluster in the visit order
    const uint32_t* ord = sp.q_order + (size_t)q * sp.q_order_stride;
    const uint32_t cnt = __ldg(sp.q_order_count + q);
    uint32_t fi = kOffPath;
    for (uint32_t i0 = 0; i0 < cnt && fi == kOffPath; i0 += 32) {
        const uint32_t i = i0 + lane;
        const unsigned b = __ballot_sync(0xffffffffu, i < cnt && __ldg(ord + i) == first);
        if (b) fi = i0 + __ffs(b) - 1;
    }
    if (fi == kOffPath) {
        leave();
        return;
    }
    const uint32_t* src = sp.start_dist + (size_t)row * sp.start_stride;
    RegKeys rk;
    if (n <= 32u * kRegKeys) rk.load(src, n);  // in flight while the query is quantized
    // QuantizeEmbedding (scalar.hpp:76-94) in the scan's packed word layout; |q|^2 over the
    // first checkpoint's words
    const float* qf = sp.queries + (size_t)q * lv.d;
    if (sp.prep_qs) {
        float* qs = qs_all + (size_t)warp * sp.prep_qs_stride;
        for (uint32_t i0 = 0; i0 < lv.d; i0 += 128) {
            float t[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t i = i0 + 32 * u + lane;
                t[u] = i < lv.d ? __ldg(qf + i) : 0.0f;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t i = i0 + 32 * u + lane;
                if (i < lv.d) qs[i] = t[u];
            }
        }
        __syncwarp();
        qf = qs;
    }
    uint32_t* qw = sp.qwords + (size_t)q * sp.nwords;
    uint32_t qn = 0;
    for (uint32_t w = lane; w < sp.nwords; w += 32) {
        const uint32_t word = quantize_word(qf, lv, w);
        qw[w] = word;
        if (w < sp.g1) qn = __dp4a(word, word, qn);
    }
    qn = __reduce_add_sync(0xffffffffu, qn);
    // every later non-empty visit into its cluster's list; the visit that opens a chunk of
    // kScanCQ list entries also opens the bitmap work item of that chunk
    for (uint32_t i = fi + 1 + lane; i < cnt; i += 32) {
        const uint32_t c = __ldg(ord + i);
        if (lv.clusters[c].n == 0) {  // num_embeddings == 0 (searcher.hpp:662)
            sp.vinfo[(size_t)q * sp.q_order_stride + i] = 0u;
            continue;
        }
        const uint32_t slot = atomicAdd(sp.vl_count + c, 1u);
        sp.vl[(size_t)c * sp.nq + slot] = q * sp.q_order_stride + i;
        if (slot % kScanCQ == 0) {
            const uint32_t it = atomicAdd(sp.n_items, 1u);
            sp.items[2 * it] = c;
            sp.items[2 * it + 1] = slot / kScanCQ;
        }
    }
    const uint32_t* ids = reinterpret_cast<const uint32_t*>(sp.arena + cl.ids_off);
    float* hd = sp.heap_d + (size_t)q * sp.k;
    uint32_t* hid = sp.heap_id + (size_t)q * sp.k;
    const uint32_t kth = n <= 32u * kRegKeys ? start_push(rk, n, m, hist, ids, lv, hd, hid)
                                             : start_push(MemKeys{src}, n, m, hist, ids, lv, hd, hid);
    if (lane == 0) {
        // heap top after the pushes: the m-th key; the first checkpoint's bound at it
        const float tau0 = reported_u8(kth, lv);
        const long long lim = (long long)thr_u8(tau0, sp.cp1, lv, sp.ratios) - (long long)qn;
        sp.lim[q] = lim > 0x7FFFFFFFll ? 0x7FFFFFFF : (int32_t)lim;
        sp.first_i[q] = fi;
        if (sp.stats) {
            add_stat(sp, 0, (unsigned long long)n * lv.d);
            add_stat(sp, 3 + kStart, (unsigned long long)n * lv.d);
            add_stat(sp, 1, 1ull);
        }
    }
}

// ------------------------------------------------------------------------------------ bitmaps
// CTA = one work item: up to 64 visits of one cluster. Warp w holds the first-checkpoint words
// of vector blocks w, w + 8, ... (lane = vector) in registers with |x|^2, and loops over the
// item's queries: 4 dp4a give q.x, and the ballot of |x|^2 - 2 q.x < lim is the 32-bit word of
// that block in the query's bitmap. Lane j keeps the word of query j mod 32 and the 32 words go
// to the item's bitmaps in shared memory together (sp.bm_tile; clusters too large for that write
// all words to global memory). Once the cluster is done the CTA knows every visit's candidates:
// most visits have none, and only the bitmaps of light visits are written out.
__global__ void __launch_bounds__(kBitmapThreads) scan_bitmap_kernel(const __grid_constant__ ScanParams sp) {
    __shared__ uint4 qv[kScanCQ];
    __shared__ int32_t ql[kScanCQ];
    __shared__ uint32_t qe[kScanCQ];
    __shared__ uint32_t qcnt[kScanCQ];
    __shared__ uint32_t item;
    extern __shared__ uint32_t tile[];  // [kScanCQ][bm_words | 1]
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t ts = sp.bm_words | 1u;  // odd row stride: 32 rows of one column hit distinct banks
    constexpr uint32_t kWarps = kBitmapThreads / 32;
    const DevLevel& lv = sp.l1;
    const uint32_t g1 = sp.g1;
    for (;;) {
        if (threadIdx.x == 0) item = atomicAdd(sp.queue, 1u);
        __syncthreads();
        const uint32_t it = item;
        __syncthreads();
        if (it >= sp.n_items[0]) break;
        const uint32_t c = sp.items[2 * it], a = sp.items[2 * it + 1];
        const uint32_t L = sp.vl_count[c];
        const uint32_t nqc = (L - a * kScanCQ) < kScanCQ ? (L - a * kScanCQ) : kScanCQ;
        if (threadIdx.x < nqc) {
            const uint32_t e = sp.vl[(size_t)c * sp.nq + a * kScanCQ + threadIdx.x];
            const uint32_t q = e / sp.q_order_stride;
            const uint32_t* w = sp.qwords + (size_t)q * sp.nwords;
            qv[threadIdx.x] = make_uint4(__ldg(w), g1 > 1 ? __ldg(w + 1) : 0u, g1 > 2 ? __ldg(w + 2) : 0u,
                                         g1 > 3 ? __ldg(w + 3) : 0u);
            ql[threadIdx.x] = sp.lim[q];
            qe[threadIdx.x] = e;
            qcnt[threadIdx.x] = 0;
        }
        __syncthreads();
        const DevCluster cl = lv.clusters[c];
        const uint32_t n = cl.n;
        const uint32_t nb = (n + 31) >> 5;
        const uint32_t* vert = reinterpret_cast<const uint32_t*>(sp.arena + cl.vert_off);
        for (uint32_t b0 = warp; b0 < nb; b0 += kWarps * kBitmapBPW) {
            uint32_t x[kBitmapBPW][4], xn[kBitmapBPW], word[kBitmapBPW];
            bool valid[kBitmapBPW];
#pragma unroll
            for (int b = 0; b < kBitmapBPW; ++b) {
                const uint32_t blk = b0 + b * kWarps;
                const uint32_t v = blk * 32 + lane;
                valid[b] = blk < nb && v < n;
                xn[b] = 0;
                word[b] = 0;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    // rows past the cluster's vectors but inside n_pad hold padding: never read
                    x[b][g] = (valid[b] && (uint32_t)g < g1) ? __ldg(vert + (size_t)g * cl.n_pad + v) : 0u;
                    xn[b] = __dp4a(x[b][g], x[b][g], xn[b]);
                }
            }
            for (uint32_t j = 0; j < nqc; ++j) {
                const uint4 qq = qv[j];
                const int32_t lj = ql[j];
#pragma unroll
                for (int b = 0; b < kBitmapBPW; ++b) {
                    uint32_t dot = __dp4a(qq.x, x[b][0], 0u);
                    dot = __dp4a(qq.y, x[b][1], dot);
                    dot = __dp4a(qq.z, x[b][2], dot);
                    dot = __dp4a(qq.w, x[b][3], dot);
                    const int32_t val = (int32_t)xn[b] - 2 * (int32_t)dot;  // |q - x|^2 - |q|^2
                    const unsigned bal = __ballot_sync(0xffffffffu, valid[b] && val < lj);
                    if (lane == (j & 31)) word[b] = bal;
                }
                if ((j & 31) == 31 || j + 1 == nqc) {
                    const uint32_t jj = (j & ~31u) + lane;
                    if (jj <= j) {
                        uint32_t* row = sp.bm_tile ? tile + jj * ts : sp.bm + (size_t)qe[jj] * sp.bm_words;
                        uint32_t cnt = 0;
#pragma unroll
                        for (int b = 0; b < kBitmapBPW; ++b) {
                            const uint32_t blk = b0 + b * kWarps;
                            if (blk < nb) {
                                row[blk] = word[b];
                                cnt += __popc(word[b]);
                            }
                        }
                        if (cnt) atomicAdd(&qcnt[jj], cnt);
                    }
                }
            }
        }
        __syncthreads();
        // class of every visit of the item; a warmup can pass its first step only when fewer than
        // ceil(0.8 n) vectors reach the bound, and the candidates hold every vector below it
        const uint32_t needed = (uint32_t)ceilf(__fmul_rn(kSelectivity, (float)n));
        if (threadIdx.x < nqc) {
            const uint32_t cnt = qcnt[threadIdx.x];
            const uint32_t info = (sp.cp1 < lv.dv && n - cnt < needed) ? kHeavyBit : cnt;
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
        __syncthreads();
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

constexpr int kCandPerLane = 4;  // candidates a replay lane tests per memory round trip
constexpr int kFallPerLane = 4;  // vectors a replay lane carries through a full warmup step

__device__ __forceinline__ uint32_t sq16(const uint4& q, const uint4& x, uint32_t acc) {
    acc = sq4(q.x, x.x, acc);
    acc = sq4(q.y, x.y, acc);
    acc = sq4(q.z, x.z, acc);
    return sq4(q.w, x.w, acc);
}

// The vertical dims from cur0 on in 64-dim steps for a vector below every bound up to `cur` (the
// horizontal blocks included), tested after each step.
__device__ __forceinline__ bool scan_follow_vertical(const ScanParams& sp, const DevCluster& c, const uint32_t* qw,
                                                     uint32_t v, uint32_t cur0, uint32_t cur, float top, uint32_t& raw,
                                                     unsigned long long& vbytes) {
    const DevLevel& lv = sp.l1;
    const uint32_t* vert = reinterpret_cast<const uint32_t*>(sp.arena + c.vert_off);
    uint32_t cur_v = cur0;
    while (cur_v < lv.dv) {
        const uint32_t last = (cur_v + kHDim < lv.dv) ? cur_v + kHDim : lv.dv;
        vbytes += last - cur_v;
        for (uint32_t g = cur_v >> 2; g < ((last + 3) >> 2); ++g)
            raw = sq4(qw[g], __ldg(vert + (size_t)g * c.n_pad + v), raw);
        cur = (cur + kHDim < lv.d) ? cur + kHDim : lv.d;
        cur_v = last;
        if (!(raw < thr_u8(top, cur, lv, sp.ratios))) return false;
        if (cur == lv.d) break;
    }
    return true;
}

// One survivor of the warmup bound at checkpoint cur0: the horizontal blocks, then the
// remaining vertical dims in 64-dim steps, tested after each against the bound of the heap top
// `top` fixed for the whole cluster (searcher.hpp:437-540). Returns whether it is still below
// the bound at the end; raw is its running distance.
__device__ __forceinline__ bool scan_follow(const ScanParams& sp, const DevCluster& c, const uint32_t* qw,
                                            uint32_t v, uint32_t cur0, float top, uint32_t& raw,
                                            unsigned long long& hbytes, unsigned long long& vbytes) {
    const DevLevel& lv = sp.l1;
    const uint32_t nhb = lv.n_hblocks;
    uint32_t cur = cur0;
    if (nhb) {
        const uint4* row = reinterpret_cast<const uint4*>(sp.arena + c.hor_off) + (size_t)v * 4;
        const size_t bstride = (size_t)c.n_pad * 4;  // uint4 per block
        for (uint32_t b = 0; b < nhb; ++b) {
            uint4 x[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) x[t] = __ldg(row + b * bstride + t);
            const uint4* qh = reinterpret_cast<const uint4*>(qw + lv.qw_hoff + b * 16);
#pragma unroll
            for (int t = 0; t < 4; ++t) raw = sq16(qh[t], x[t], raw);
            hbytes += kHDim;
            cur += kHDim;
            if (!(raw < thr_u8(top, cur, lv, sp.ratios))) return false;
        }
    }
    return scan_follow_vertical(sp, c, qw, v, cur0, cur, top, raw, vbytes);
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

// Values of vector v of a heavy visit into column `out` (row stride sp.hv_cap): row s < ncp is the
// running distance at warmup checkpoint s, row ncp + b the sum of horizontal block b. They do not
// depend on the query's heap, so the loads of 64 vertical dims, then of three blocks, are in flight
// together (8 dims and two blocks: 152 against 108 us for the replay of a 777-query batch). Returns
// the full distance.
__device__ __forceinline__ uint32_t heavy_column(const ScanParams& sp, const DevCluster& c, const uint32_t* qw,
                                                 uint32_t v, uint32_t* out) {
    const DevLevel& lv = sp.l1;
    const uint32_t* col = reinterpret_cast<const uint32_t*>(sp.arena + c.vert_off) + v;
    const uint32_t groups = (lv.dv + 3) >> 2;
    uint32_t raw = 0, s = 0, next = sp.cp1;
    for (uint32_t g0 = 0; g0 < groups; g0 += 16) {
        uint32_t x[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) x[t] = g0 + t < groups ? __ldg(col + (size_t)(g0 + t) * c.n_pad) : 0u;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            if (g0 + t < groups) {
                raw = sq4(qw[g0 + t], x[t], raw);
                if ((g0 + t + 1) * 4 >= next) {  // checkpoints are multiples of 16 dims, the last is d_v
                    out[(size_t)s * sp.hv_cap] = raw;
                    ++s;
                    next += c_scan_fetch[s < kNumFetchSizes ? s : kNumFetchSizes - 1];
                    if (next > lv.dv) next = lv.dv;
                }
            }
        }
    }
    out += (size_t)sp.hv_ncp * sp.hv_cap;
    const uint4* row = reinterpret_cast<const uint4*>(sp.arena + c.hor_off) + (size_t)v * 4;
    const size_t bstride = (size_t)c.n_pad * 4;  // uint4 per block
    for (uint32_t b0 = 0; b0 < lv.n_hblocks; b0 += 3) {
        uint4 x[3][4];
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
            for (int t = 0; t < 4; ++t)
                x[u][t] = b0 + u < lv.n_hblocks ? __ldg(row + (b0 + u) * bstride + t) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            if (b0 + u < lv.n_hblocks) {
                const uint4* qh = reinterpret_cast<const uint4*>(qw + lv.qw_hoff + (b0 + u) * 16);
                uint32_t sum = 0;
#pragma unroll
                for (int t = 0; t < 4; ++t) sum = sq16(qh[t], x[u][t], sum);
                out[(size_t)(b0 + u) * sp.hv_cap] = sum;
                raw += sum;
            }
        }
    }
    return raw;
}

// A heavy visit needs the running distance of all its vectors at up to every warmup checkpoint and
// then a long survivor path for most of them. Done by the query's own warp at the visit's turn that
// is a chain of several hundred dependent loads: 1-2 % of the queries of a 777-query batch on the
// 1M x 1024 SQ8 tree took about 400 us there and set the kernel's time. Here the CTA's warps first
// share out the 32-vector blocks of its queries' heavy visits (HeavyList), and the replay reads the
// values; a visit that finds no room in the list or in sp.hv runs its warmup in the warp.
// A vector can only be merged when its full distance is below the bound at all d dims, at most
// that of the heap top after the Start: those vectors are marked in the visit's bitmap, and a
// visit without any changes nothing.
struct HeavyList {
    uint32_t n;
    uint32_t warp[kHeavyList], visit[kHeavyList];
    uint32_t base[kHeavyList];  // first column / 32 in sp.hv
    uint32_t end[kHeavyList];   // 32-vector blocks of the list up to and with this visit
    uint32_t thr0[kScanWarps];  // bound at all d dims of each warp's heap top after the Start
};

__global__ void __launch_bounds__(kScanWarps * 32, 3) scan_replay_kernel(const __grid_constant__ ScanParams sp) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ HeavyList HL;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // warps past r_qpc own no query (no shared-memory region either) and only share the heavy visits
    const uint32_t q = blockIdx.x * sp.r_qpc + warp;
    const uint32_t fi = warp < sp.r_qpc && q < sp.nq ? sp.first_i[q] : kOffPath;
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
    if (threadIdx.x == 0) HL.n = 0;
    __syncthreads();
    if (fi != kOffPath) {
        for (uint32_t w = lane; w < sp.nwords; w += 32) R.qw[w] = __ldg(sp.qwords + (size_t)q * sp.nwords + w);
        for (uint32_t j = lane; j < kq; j += 32) {
            R.hd[j] = __ldg(sp.heap_d + (size_t)q * sp.k + j);
            R.hid[j] = __ldg(sp.heap_id + (size_t)q * sp.k + j);
        }
        __syncwarp();
        warp_heap_top(R.hd, kq, top, slot);
        if (lane == 0) HL.thr0[warp] = thr_u8(top, lv.d, lv, sp.ratios);
        for (uint32_t i = fi + 1 + lane; i < cnt; i += 32) {
            if (!(__ldg(vis + i) & kHeavyBit) || HL.n >= kHeavyList) continue;
            // columns are handed out in units of 32; none is asked for once they are used up, so the
            // counter stays far from its range
            if (__ldcg(sp.hv_alloc) >= sp.hv_cap / 32) continue;
            const uint32_t nb = (lv.clusters[__ldg(ord + i)].n + 31) >> 5;
            const uint32_t col = atomicAdd(sp.hv_alloc, nb);
            if (col + nb > sp.hv_cap / 32) continue;
            const uint32_t at = atomicAdd(&HL.n, 1u);
            if (at >= kHeavyList) continue;
            HL.warp[at] = warp;
            HL.visit[at] = i;
            HL.base[at] = col;
            HL.end[at] = nb;
        }
    }
    __syncthreads();
    const uint32_t n_heavy = HL.n < kHeavyList ? HL.n : kHeavyList;
    if (n_heavy) {  // block-uniform
        if (threadIdx.x == 0)
            for (uint32_t j = 1; j < n_heavy; ++j) HL.end[j] += HL.end[j - 1];
        __syncthreads();
        uint32_t j = 0;
        for (uint32_t b = warp; b < HL.end[n_heavy - 1]; b += kScanWarps) {
            while (HL.end[j] <= b) ++j;
            const uint32_t blk = b - (j ? HL.end[j - 1] : 0u);
            const uint32_t hw = HL.warp[j];
            const uint32_t hq = blockIdx.x * sp.r_qpc + hw;
            const DevCluster c = lv.clusters[__ldg(sp.q_order + (size_t)hq * stride + HL.visit[j])];
            const uint32_t v = blk * 32 + lane;
            uint32_t full = 0xFFFFFFFFu;
            if (v < c.n)
                full = heavy_column(sp, c, reinterpret_cast<const uint32_t*>(smem + (size_t)hw * sp.r_warp_bytes), v,
                                    sp.hv + ((size_t)(HL.base[j] + blk) << 5) + lane);
            // statistics count the blocks of vectors that end up pruned too
            const unsigned may = __ballot_sync(0xffffffffu, v < c.n && (sp.stats || full < HL.thr0[hw]));
            if (lane == 0) sp.bm[((size_t)hq * stride + HL.visit[j]) * sp.bm_words + blk] = may;
        }
        __syncthreads();
    }
    if (fi == kOffPath) return;  // whole warp; no block-wide barrier follows
    uint4 q1 = make_uint4(0u, 0u, 0u, 0u);  // first checkpoint's query words (zero past g1)
    q1.x = R.qw[0];
    if (sp.g1 > 1) q1.y = R.qw[1];
    if (sp.g1 > 2) q1.z = R.qw[2];
    if (sp.g1 > 3) q1.w = R.qw[3];
    uint32_t* scratch = sp.start_dist + (size_t)__ldg(sp.start_row + q) * sp.start_stride;
    const uint32_t S = sp.r_surv_cap;
    unsigned long long b_warm = 0, b_h = 0, b_v = 0, merged = 0;
    unsigned long long n_cand = 0, n_surv = 0, n_fast = 0, n_full = 0;
    unsigned long long b_warm_l = 0;  // per lane: the first step of every visit
    uint32_t visits_l = 0, fast_l = 0;

    // Merges the warp's vectors that stayed below every bound (alive), in lane order
    // (MergeIntoHeap, searcher.hpp:542-566).
    auto merge = [&](const DevCluster& c, bool alive, uint32_t v, uint32_t raw) {
        const uint32_t idv = alive ? __ldg(reinterpret_cast<const uint32_t*>(sp.arena + c.ids_off) + v) : 0u;
        const float dd = reported_u8(raw, lv);
        unsigned bal = __ballot_sync(0xffffffffu, alive);
        merged += __popc(bal);
        while (bal) {
            const int l = __ffs(bal) - 1;
            bal &= bal - 1;
            const float ddl = __shfl_sync(0xffffffffu, dd, l);
            const uint32_t idl = __shfl_sync(0xffffffffu, idv, l);
            if (ddl < top) {
                if (lane == 0) {
                    R.hd[slot] = ddl;
                    R.hid[slot] = idl;
                }
                __syncwarp();
                warp_heap_top(R.hd, kq, top, slot);
            }
        }
    };

    // Follows the lane's survivor (alive, v, raw) through Prune with the bound at `tp`, then merges.
    auto prune_merge = [&](const DevCluster& c, bool alive, uint32_t v, uint32_t raw, uint32_t cur, float tp) {
        if (alive) alive = scan_follow(sp, c, R.qw, v, cur, tp, raw, b_h, b_v);
        merge(c, alive, v, raw);
    };
    // A heavy visit on its values computed ahead, hv pointing at its first vector's column.
    // bmh: its mergeable vectors.
    auto heavy_visit = [&](const DevCluster& c, const uint32_t* hv, const uint32_t* bmh) {
        const uint32_t n = c.n, W = (n + 31) >> 5;
        uint32_t any = 0;
        for (uint32_t w = lane; w < W; w += 32) any |= bmh[w];
        if (!__any_sync(0xffffffffu, any != 0)) return;
        const uint32_t needed = (uint32_t)ceilf(__fmul_rn(kSelectivity, (float)n));
        const float tp = top;  // the bound's heap top, fixed for the whole cluster
        uint32_t cur = 0, step = 0, n_pruned = 0;
        while (n_pruned < needed && cur < lv.dv) {  // Warmup (searcher.hpp:374-435)
            uint32_t last = cur + c_scan_fetch[step < kNumFetchSizes ? step : kNumFetchSizes - 1];
            if (last > lv.dv) last = lv.dv;
            const uint32_t thr = thr_u8(tp, last, lv, sp.ratios);
            const uint32_t* row = hv + (size_t)step * sp.hv_cap;
            uint32_t cntp = 0;
            for (uint32_t v0 = 0; v0 < n; v0 += 256) {
                uint32_t x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t v = v0 + 32 * u + lane;
                    x[u] = v < n ? row[v] : 0u;
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) cntp += (v0 + 32 * u + lane < n && x[u] >= thr) ? 1u : 0u;
            }
            n_pruned = __reduce_add_sync(0xffffffffu, cntp);
            if (cur == 0) n_surv += n - n_pruned;
            else b_warm += (unsigned long long)n * (last - cur);
            cur = last;
            ++step;
        }
        if (step == 1) ++n_fast;
        else ++n_full;
        // Prune (searcher.hpp:437-540) and merge of the mergeable vectors, 32 at a time in position
        // order; their horizontal sums are loaded kHeavyBlocks at a time, ahead of their tests
        constexpr int kHeavyBlocks = 6;
        const uint32_t thr = thr_u8(tp, cur, lv, sp.ratios);
        const uint32_t* erow = hv + (size_t)(step - 1) * sp.hv_cap;
        const uint32_t* brow = hv + (size_t)sp.hv_ncp * sp.hv_cap;
        for (uint32_t w0 = 0; w0 < W; w0 += 32) {
            const uint32_t total = scan_bits_to_offsets(w0 + lane < W ? bmh[w0 + lane] : 0u, lane, R.cand);
            for (uint32_t j0 = 0; j0 < total; j0 += 32) {
                bool alive = j0 + lane < total;
                const uint32_t v = alive ? w0 * 32 + R.cand[j0 + lane] : 0u;
                uint32_t raw = alive ? erow[v] : 0u;
                alive = alive && raw < thr;
                uint32_t cv = cur;
                for (uint32_t b0 = 0; b0 < lv.n_hblocks && __any_sync(0xffffffffu, alive); b0 += kHeavyBlocks) {
                    uint32_t x[kHeavyBlocks];
#pragma unroll
                    for (int u = 0; u < kHeavyBlocks; ++u)
                        x[u] = (alive && b0 + u < lv.n_hblocks) ? brow[(size_t)(b0 + u) * sp.hv_cap + v] : 0u;
#pragma unroll
                    for (int u = 0; u < kHeavyBlocks; ++u) {
                        if (alive && b0 + u < lv.n_hblocks) {
                            raw += x[u];
                            b_h += kHDim;
                            cv += kHDim;
                            alive = raw < thr_u8(tp, cv, lv, sp.ratios);
                        }
                    }
                }
                if (alive) alive = scan_follow_vertical(sp, c, R.qw, v, cur, cv, tp, raw, b_v);
                merge(c, alive, v, raw);
            }
            __syncwarp();  // cand is rewritten by the next word group
        }
    };

    // Visits without a candidate end their warmup at the first step with no survivor (n >= 0.8 n
    // vectors reach the bound): only the others are walked. On the 1M x 1024 SQ8 tree a query has
    // one or two of them in 31 visits, and walking all of them was a chain of 31 record and bitmap
    // round trips.
    for (uint32_t i0 = (fi + 1) & ~31u; i0 < cnt; i0 += 32) {
      const uint32_t il = i0 + lane;
      const bool in = il > fi && il < cnt;
      uint32_t info_l = in ? __ldg(vis + il) : 0u;
      if (sp.stats && in) {
          const uint32_t n = lv.clusters[__ldg(ord + il)].n;
          visits_l += n ? 1u : 0u;
          b_warm_l += (unsigned long long)n * sp.cp1;
          fast_l += (n && info_l == 0) ? 1u : 0u;
      }
      for (unsigned todo = __ballot_sync(0xffffffffu, info_l != 0); todo; todo &= todo - 1) {
        const uint32_t src = __ffs(todo) - 1, i = i0 + src;
        const uint32_t info = __shfl_sync(0xffffffffu, info_l, src);
        const DevCluster c = lv.clusters[__ldg(ord + i)];
        if (info & kHeavyBit) {
            uint32_t at = 0xFFFFFFFFu;
            for (uint32_t j = lane; j < n_heavy; j += 32)
                if (HL.warp[j] == warp && HL.visit[j] == i) at = j;
            at = __reduce_min_sync(0xffffffffu, at);
            if (at != 0xFFFFFFFFu) {
                heavy_visit(c, sp.hv + ((size_t)HL.base[at] << 5), sp.bm + ((size_t)q * stride + i) * sp.bm_words);
                continue;
            }
        }
        const uint32_t n = c.n;
        const uint32_t* vert = reinterpret_cast<const uint32_t*>(sp.arena + c.vert_off);
        const uint32_t W = (n + 31) >> 5;
        const uint32_t needed = (uint32_t)ceilf(__fmul_rn(kSelectivity, (float)n));
        const uint32_t* bmp = sp.bm + ((size_t)q * stride + i) * sp.bm_words;
        // Warmup step 1 from the candidates: the exact first-checkpoint distance of each, and the
        // survivors under the current bound, in position order
        const uint32_t thr1 = thr_u8(top, sp.cp1, lv, sp.ratios);
        uint32_t ns = 0;
        const bool light = !(info & kHeavyBit);  // a heavy visit keeps no bitmap
        for (uint32_t w0 = 0; light && w0 < W; w0 += 32) {
            const uint32_t w = w0 + lane;
            const uint32_t word = w < W ? __ldg(bmp + w) : 0u;
            const uint32_t total = scan_bits_to_offsets(word, lane, R.cand);
            n_cand += total;
            for (uint32_t j0 = 0; j0 < total; j0 += 32 * kCandPerLane) {
                uint32_t v[kCandPerLane];
                uint4 x[kCandPerLane];
#pragma unroll
                for (int u = 0; u < kCandPerLane; ++u) {
                    const uint32_t j = j0 + 32 * u + lane;
                    v[u] = j < total ? w0 * 32 + R.cand[j] : 0xFFFFFFFFu;
                    const bool in = v[u] != 0xFFFFFFFFu;
                    const uint32_t* col = vert + (in ? v[u] : 0u);
                    x[u].x = in ? __ldg(col) : 0u;
                    x[u].y = (in && sp.g1 > 1) ? __ldg(col + (size_t)c.n_pad) : 0u;
                    x[u].z = (in && sp.g1 > 2) ? __ldg(col + 2 * (size_t)c.n_pad) : 0u;
                    x[u].w = (in && sp.g1 > 3) ? __ldg(col + 3 * (size_t)c.n_pad) : 0u;
                }
#pragma unroll
                for (int u = 0; u < kCandPerLane; ++u) {
                    const uint32_t d1 = sq16(q1, x[u], 0u);
                    const bool s = v[u] != 0xFFFFFFFFu && d1 < thr1;
                    const unsigned bal = __ballot_sync(0xffffffffu, s);
                    const uint32_t r = ns + __popc(bal & ((1u << lane) - 1u));
                    if (s && r < S) {
                        R.sv_pos[r] = v[u];
                        R.sv_d[r] = d1;
                    }
                    ns += __popc(bal);
                }
            }
            __syncwarp();
        }
        const bool exits = sp.cp1 >= lv.dv || n - ns >= needed;  // the warmup stops after step 1
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
            const uint32_t thr = thr_u8(top, last, lv, sp.ratios);
            const uint32_t g0 = cur >> 2, g_end = (last + 3) >> 2;
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
                        const uint32_t qv = g + gg < g_end ? R.qw[g + gg] : 0u;
#pragma unroll
                        for (int u = 0; u < kFallPerLane; ++u) acc[u] = sq4(qv, xs[gg][u], acc[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < kFallPerLane; ++u) {
                    const uint32_t v = v0 + 32 * u + lane;
                    if (v < n) {
                        scratch[v] = acc[u];
                        cntp += acc[u] >= thr ? 1u : 0u;
                    }
                }
            }
            n_pruned = __reduce_add_sync(0xffffffffu, cntp);
            if (cur > 0) b_warm += (unsigned long long)n * (last - cur);
            cur = last;
            ++step;
        }
        // Prune: the vectors below the bound at the warmup's last checkpoint, in position order
        const uint32_t thr = thr_u8(top, cur, lv, sp.ratios);
        for (uint32_t v0 = 0; v0 < n; v0 += 32) {
            const uint32_t v = v0 + lane;
            const unsigned bal = __ballot_sync(0xffffffffu, v < n && scratch[v] < thr);
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
            add_stat(sp, 12, n_cand);
            add_stat(sp, 13, n_surv);
            add_stat(sp, 14, n_fast);
            add_stat(sp, 15, n_full);
        }
    }
}

// ------------------------------------------------------------------------------------ launch
uint64_t scan_item_bound(uint32_t nq, uint32_t stride, uint32_t n1) {
    return (uint64_t)nq * stride / kScanCQ + n1 + 1;
}

// Shared memory of a bitmap work item's tile; 0: the bitmaps of clusters this large go straight
// to global memory.
size_t scan_bitmap_smem(uint32_t bm_words) {
    const size_t b = (size_t)kScanCQ * (bm_words | 1u) * 4;
    return b <= kBitmapTileMax ? b : 0;
}

int scan_bitmap_occupancy(uint32_t bm_words) {
    int blocks = 0;
    const size_t tile = scan_bitmap_smem(bm_words);
    if (tile) cudaFuncSetAttribute(scan_bitmap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, scan_bitmap_kernel, kBitmapThreads, tile);
    return blocks;
}

uint32_t scan_queries_per_cta() { return kScanWarps; }

// ev (optional, 3 events): recorded after the prep kernel, the bitmaps and the replay.
cudaError_t launch_scan(const ScanParams& sp, int bitmap_grid, cudaStream_t st, const cudaEvent_t* ev) {
    cudaError_t e = cudaMemsetAsync(sp.vl_count, 0, sizeof(uint32_t) * sp.l1.nclusters, st);
    if (e != cudaSuccess) return e;
    // left_n, n_items, queue and hv_alloc are consecutive
    if ((e = cudaMemsetAsync(sp.left_n, 0, 4 * sizeof(uint32_t), st)) != cudaSuccess) return e;
    const uint32_t ctas = (sp.nq + kScanWarps - 1) / kScanWarps;
    const size_t prep_smem = sp.prep_qs ? (size_t)kScanWarps * sp.prep_qs_stride * 4 : 0;
    if (prep_smem) {
        e = cudaFuncSetAttribute(scan_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prep_smem);
        if (e != cudaSuccess) return e;
    }
    scan_prep_kernel<<<ctas, kScanWarps * 32, prep_smem, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[0], st)) != cudaSuccess) return e;
    const size_t tile = scan_bitmap_smem(sp.bm_words);
    if (tile) {
        e = cudaFuncSetAttribute(scan_bitmap_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile);
        if (e != cudaSuccess) return e;
    }
    scan_bitmap_kernel<<<bitmap_grid, kBitmapThreads, tile, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[1], st)) != cudaSuccess) return e;
    const size_t smem = (size_t)sp.r_qpc * sp.r_warp_bytes;
    e = cudaFuncSetAttribute(scan_replay_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    scan_replay_kernel<<<(sp.nq + sp.r_qpc - 1) / sp.r_qpc, kScanWarps * 32, smem, st>>>(sp);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if (ev && (e = cudaEventRecord(ev[2], st)) != cudaSuccess) return e;
    return cudaSuccess;
}

}  // namespace pdxg
