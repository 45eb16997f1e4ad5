// select.cu -- merge of the per-split shortlists (or of the threshold scan's
// candidate segments), exact re-rank, final top-k.
//
// Replaces the reference's cross-chunk host merge (mergeResBitonic,
// src/cuknnBitonic.cu:381-417; mergeResHeap, src/cuknnHeap.cu:26-62) and the
// final +||q||^2 pass (dot3, include/utils.h:485-491).  One warp per query:
// the `splits` sorted shortlists are merged pairwise by rank (ties: earlier
// split first, which is also lower index, so the reference's "earlier chunk
// wins" rule holds), then either
//   rerank = 1: every shortlisted candidate gets its exact distance
//               (direct difference, oracle convention), the shortlist is
//               re-sorted by (distance, index) and the first k are returned;
//   rerank = 0: the first k by GEMM-form key are returned with
//               distance = key + ||q||^2 (the reference's output contract).
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"
#include "kernels.h"

namespace knn {

namespace {
constexpr int kSelWarps = 4;

__host__ __device__ inline int pow2_at_least(int x)
{
    int p = 32;
    while (p < x) p <<= 1;
    return p;
}

// cur[0..kp) holds the query's shortlist sorted by (key, index) (sentinels at
// the end); cur has room for pow2_at_least(kp) words.  Writes the k results of
// query q (re-ranked by exact distance, or key + ||q||^2).
__device__ __forceinline__ void finish_query(uint64_t* cur, int kp, int k, int64_t q, int rerank,
                                             const float* __restrict__ corpus, int64_t ldc,
                                             const float* __restrict__ queries, int64_t ldq, int D,
                                             const float* __restrict__ qn, float* qv, float* out_dist,
                                             int32_t* out_idx, float* out_idx_f)
{
    const int lane = threadIdx.x & 31;
    if (rerank) {
        const int P = pow2_at_least(kp);
        const float* qrow = queries + q * ldq;
        for (int d = lane; d < D; d += 32) qv[d] = __ldg(qrow + d);
        __syncwarp();
        for (int j = lane; j < P; j += 32) {
            uint64_t w = j < kp ? cur[j] : kSentinel;
            if (w != kSentinel) {
                uint32_t n = unpack_idx(w);
                float dist = exact_dist_row(qv, corpus + (int64_t)n * ldc, D);
                w = pack_key(dist, n);
            }
            cur[j] = w;
        }
        __syncwarp();
        warp_sort_smem(cur, P);
        for (int j = lane; j < k; j += 32) {
            uint64_t w = cur[j];
            bool ok = w != kSentinel;
            float dv = ok ? unpack_key(w) : __int_as_float(0x7f800000);
            int32_t iv = ok ? (int32_t)unpack_idx(w) : -1;
            if (out_dist) out_dist[q * k + j] = dv;
            if (out_idx) out_idx[q * k + j] = iv;
            if (out_idx_f) out_idx_f[q * k + j] = (float)iv;
        }
    } else {
        const float qq = qn[q];
        for (int j = lane; j < k; j += 32) {
            uint64_t w = cur[j];
            bool ok = w != kSentinel;
            float dv = ok ? __fadd_rn(unpack_key(w), qq) : __int_as_float(0x7f800000);
            int32_t iv = ok ? (int32_t)unpack_idx(w) : -1;
            if (out_dist) out_dist[q * k + j] = dv;
            if (out_idx) out_idx[q * k + j] = iv;
            if (out_idx_f) out_idx_f[q * k + j] = (float)iv;
        }
    }
}
}  // namespace

__global__ void __launch_bounds__(kSelWarps * 32)
select_kernel(const uint64_t* __restrict__ part, int splits, int64_t Q, int kp, int k,
              const float* __restrict__ corpus, int64_t ldc, const float* __restrict__ queries,
              int64_t ldq, int D, int rerank, const float* __restrict__ qn,
              float* __restrict__ out_dist, int32_t* __restrict__ out_idx, float* __restrict__ out_idx_f,
              const SelectExtra ex)
{
    extern __shared__ __align__(16) unsigned char smem[];
    if (ex.skip_if_zero != nullptr && *ex.skip_if_zero == 0u) return;
    const int P = pow2_at_least(kp);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // per warp: cur[P], nxt[P], other[kp], query vector[D]
    size_t per_warp_words = (size_t)3 * P;
    uint64_t* cur = reinterpret_cast<uint64_t*>(smem) + warp * per_warp_words;
    uint64_t* nxt = cur + P;
    uint64_t* oth = nxt + P;
    float* qv = reinterpret_cast<float*>(reinterpret_cast<uint64_t*>(smem) + kSelWarps * per_warp_words) +
                (size_t)warp * ((D + 3) & ~3);

    const int64_t q = (int64_t)blockIdx.x * kSelWarps + warp;  // row of `part`
    if (q >= Q) return;
    if (ex.redo_in != nullptr && ex.redo_in[q / ex.qtile] == 0u) return;
    int64_t qout = q;  // query whose results this row holds
    int64_t rows = Q, row = q;
    if (ex.qcount != nullptr) {
        if (q >= (int64_t)*ex.qcount) return;
        qout = ex.qmap[q];
        const FixGroup g = q < ex.fix.g[0].rows ? ex.fix.g[0] : ex.fix.g[1];
        row = q < ex.fix.g[0].rows ? q : q - ex.fix.g[0].rows;
        rows = g.rows;
        part = g.part;
        splits = g.splits;
    }

    for (int j = lane; j < kp; j += 32) cur[j] = part[(size_t)row * kp + j];
    __syncwarp();
    for (int s = 1; s < splits; ++s) {
        const uint64_t* src = part + ((size_t)s * rows + row) * kp;
        for (int j = lane; j < kp; j += 32) oth[j] = src[j];
        __syncwarp();
        warp_merge_lists(cur, oth, nxt, kp);
        uint64_t* t = cur; cur = nxt; nxt = t;
        __syncwarp();
    }

    if (ex.thr_out != nullptr) {
        // threshold extraction: key of the thr_rank-th entry
        if (lane == 0) {
            const uint64_t w = cur[ex.thr_rank - 1];
            ex.thr_out[q] = w == kSentinel ? 0xFFFFFFFFu : (uint32_t)(w >> 32);
        }
        return;
    }
    if (ex.redo_out != nullptr && ex.need > 0 && cur[ex.need - 1] == kSentinel) {
        // fewer entries than required passed a seeded threshold: this query's tile is redone
        if (lane == 0) ex.redo_out[q / ex.qtile] = 1u;
        return;
    }
    finish_query(cur, kp, k, qout, rerank, corpus, ldc, queries, ldq, D, qn, qv, out_dist, out_idx, out_idx_f);
}

// ---------------------------------------------------------------- threshold-scan selection
namespace {
// candidate words a warp can hold in threshold mode (seeding passes)
constexpr int kCandThrMax = 1024;

// scan word (raw float bits of the key << 32 | index) -> ordered word (pack_key)
__device__ __forceinline__ uint64_t raw_to_ordered(uint64_t w)
{
    return pack_key(__uint_as_float((uint32_t)(w >> 32)), (uint32_t)w);
}

// number of words w[0..n) (shared memory) not above x, summed over the warp
// Radix-4 step of the rank search: the counts of values not above y0 < y1 < y2 in one
// pass (n <= 65,535, so two counts share a 32-bit reduction), and the 2-bit digit d of the
// rank-th smallest value: the number of thresholds with fewer than `rank` values not
// above them.  Half the dependent rounds of a bitwise search.
template <typename V, typename F>
__device__ __forceinline__ uint32_t radix4_digit(const uint64_t* w, int n, V y0, V y1, V y2, uint32_t rank, F val)
{
    const int lane = threadIdx.x & 31;
    uint32_t a = 0, b = 0;
    for (int e = lane; e < n; e += 32) {
        const V v = val(w[e]);
        a += (v <= y0 ? 1u : 0u) + (v <= y1 ? 0x10000u : 0u);
        b += v <= y2 ? 1u : 0u;
    }
    a = __reduce_add_sync(0xffffffffu, a);
    b = __reduce_add_sync(0xffffffffu, b);
    return ((a & 0xffffu) < rank ? 1u : 0u) + ((a >> 16) < rank ? 1u : 0u) + (b < rank ? 1u : 0u);
}

// Threshold mode with few keys: at most kThrRegs keys per lane, ranks up to kThrRankRegs.
constexpr int kThrRegs = 8;
constexpr int kThrRankRegs = 64;

// The ordered key of rank `rank` (1-based, ties counted) among the key halves of w[0..n),
// n <= 32 * kThrRegs, n >= rank: lane l holds w[l + 32 i], sorted in registers (Batcher's
// odd-even merge network for 8); each round the warp minimum of the lanes' heads is found, every
// lane whose head equals it drops its head, and the count of dropped keys decides the rank.
__device__ __forceinline__ uint32_t rank_in_registers(const uint64_t* w, int n, uint32_t rank)
{
    const int lane = threadIdx.x & 31;
    uint32_t k[kThrRegs];
#pragma unroll
    for (int i = 0; i < kThrRegs; ++i) k[i] = lane + 32 * i < n ? (uint32_t)(w[lane + 32 * i] >> 32) : 0xFFFFFFFFu;
    auto ce = [&](int a, int b) {
        const uint32_t lo = min(k[a], k[b]), hi = max(k[a], k[b]);
        k[a] = lo;
        k[b] = hi;
    };
    ce(0, 1); ce(2, 3); ce(4, 5); ce(6, 7);
    ce(0, 2); ce(1, 3); ce(4, 6); ce(5, 7);
    ce(1, 2); ce(5, 6);
    ce(0, 4); ce(1, 5); ce(2, 6); ce(3, 7);
    ce(2, 4); ce(3, 5);
    ce(1, 2); ce(3, 4); ce(5, 6);
    uint32_t removed = 0, x = 0xFFFFFFFFu;
    for (uint32_t it = 0; it < rank; ++it) {  // every round drops at least one key
        const uint32_t m = __reduce_min_sync(0xffffffffu, k[0]);
        const bool hit = k[0] == m;
        removed += (uint32_t)__popc(__ballot_sync(0xffffffffu, hit));
        if (removed >= rank) {  // warp-uniform
            x = m;
            break;
        }
        if (hit) {
#pragma unroll
            for (int i = 0; i < kThrRegs - 1; ++i) k[i] = k[i + 1];
            k[kThrRegs - 1] = 0xFFFFFFFFu;
        }
    }
    return x;
}

}  // namespace

// Threshold mode, one warp per query over the threshold scan's segments: the key of rank thr_rank.
__global__ void __launch_bounds__(kSelWarps * 32) select_threshold_kernel(const CandSelect c)
{
    extern __shared__ __align__(16) unsigned char smem[];
    if (c.skip_if != nullptr && *c.skip_if != 0u) return;
    if (c.skip_if_zero != nullptr && *c.skip_if_zero == 0u) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int buf_max = c.buf_words;
    uint64_t* buf = reinterpret_cast<uint64_t*>(smem) + (size_t)warp * buf_max;
    const int64_t q = (int64_t)blockIdx.x * kSelWarps + warp;
    if (q >= c.Q) return;

    // segments s = lane + 32 r: their counts, all loaded at once
    constexpr int kSegPerLane = kScanMaxSegs / 32;
    uint32_t n4[kSegPerLane];
    uint32_t stored = 0, found = 0;
    bool over = false;
#pragma unroll
    for (int r = 0; r < kSegPerLane; ++r) {
        const int s = lane + 32 * r;
        const uint32_t n = s < c.nseg ? __ldg(c.cnt + (size_t)s * c.Q + q) : 0u;
        found += n;
        over |= n > (uint32_t)c.cap;
        n4[r] = min(n, (uint32_t)c.cap);
        stored += n4[r];
    }
    const uint32_t total = __reduce_add_sync(0xffffffffu, stored);
    const uint32_t found_all = __reduce_add_sync(0xffffffffu, found);
    const bool overflow = __any_sync(0xffffffffu, over);

    if (overflow || found_all < (uint32_t)c.thr_rank || total > (uint32_t)buf_max) {
        if (lane == 0) c.thr_out[q] = c.thr_fallback ? c.thr_fallback[q] : __int_as_float(0x7f800000);
        return;
    }

    // gather: each lane copies its own segments (segment-major prefix over r, then lanes)
    uint32_t base = 0;
#pragma unroll
    for (int r = 0; r < kSegPerLane; ++r) {
        if (32 * r >= c.nseg) break;  // warp-uniform: no segments left
        uint32_t pre = n4[r];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += v;
        }
        const uint32_t tot_r = __shfl_sync(0xffffffffu, pre, 31);
        const uint32_t my = base + pre - n4[r];
        const uint64_t* src = c.cand + ((size_t)(lane + 32 * r) * c.Q + q) * c.cap;
        for (uint32_t i0 = 0; i0 < n4[r]; i0 += 8) {
            uint64_t v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = i0 + u < n4[r] ? __ldg(src + i0 + u) : 0ull;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (i0 + u < n4[r]) buf[my + i0 + u] = raw_to_ordered(v[u]);
        }
        base += tot_r;
    }
    __syncwarp();
    const int n = (int)total;

    // smallest key x with at least thr_rank keys not above it
    uint32_t x = 0;
    if (n <= 32 * kThrRegs && c.thr_rank <= kThrRankRegs) {
        // few keys, small rank: each lane sorts its keys in registers, then the warp takes
        // minima in rank order (each round removes the lanes' heads equal to the minimum)
        x = rank_in_registers(buf, n, (uint32_t)c.thr_rank);
    } else {
        // radix-4 search, two bits per round: x's digit at bits [b0, b0 + 2) is the number
        // of the thresholds x | d 2^b0 | (2^b0 - 1), d = 0, 1, 2, with fewer than thr_rank
        // keys not above them
        for (int b0 = 30; b0 >= 0; b0 -= 2) {
            const uint32_t low = (1u << b0) - 1u;
            const uint32_t d = radix4_digit(buf, n, x | low, x | (1u << b0) | low, x | (2u << b0) | low,
                                            (uint32_t)c.thr_rank, [](uint64_t v) { return (uint32_t)(v >> 32); });
            x |= d << b0;
        }
    }
    if (lane == 0) {
        const float key = ord2f(x);
        // strictly above the key of rank thr_rank: that key itself passes a "< T" test
        c.thr_out[q] = key < __int_as_float(0x7f800000) ? nextafterf(key, __int_as_float(0x7f800000)) : key;
    }
}

// ---------------------------------------------------------------- one block per query
// Result mode of the selection, a whole block on each query.  Bound by the latency of a query's
// chain of dependent steps (counts, gather, rank search, re-rank, sort) until every SM is full, by
// issue slots above.  One warp per query took 25 to 150 us for that chain whatever the number of
// queries (rank search two bits a round, a sort before and one after a re-rank staged through
// shared memory); measured against it: 32,768 x 1,024, 256 queries 124 -> 19 us, 100,003 x 43, k =
// 512, 777 queries 157 -> 56, 10,000 queries of 500,000 x 128 integers at k = 100 96 -> 87.  Here
//  * the kp smallest words are found exactly by a byte-wise histogram search that starts at the
//    highest bit in which the words differ (two or three rounds), so nothing is sorted before the
//    re-rank;
//  * eight lanes compute one candidate's distance, lane u the partial sum over d = u (mod 8) (the
//    oracle's order), all of a block's rows in flight at once, read from global memory in whole
//    32-byte sectors, nothing staged;
//  * the shortlist is then ordered once, by counting smaller words (up to kRankSortMax) or a
//    bitonic sort.
constexpr int kRankSortMax = 128;
constexpr int64_t kThrBlockQ = 1536;  // threshold mode: a warp per query above
// Up to a query an SM: 512 threads each, which shorten one query's chain of round trips (48 queries on
// 2,000,000 x 128: threshold from 7,813 keys 7.5 -> 4.9 us, selection 12.9 -> 11.8, the search 150 -> 145).
constexpr int64_t kSelFewQ = kSms;
constexpr int64_t kSelWideQ = 384;  // up to this many queries: 256 threads each, above 128

// The first k of `cur` (m packed words: key or distance above index) in ascending order to the
// outputs, distances plus qq; (+inf, -1) past m.
template <int kT, typename Args>
__device__ __forceinline__ void emit_sorted(const Args& c, int64_t q, uint64_t* cur, int m, bool add_qn, float qq)
{
    const int tid = threadIdx.x;
    auto put = [&](int j, uint64_t w) {
        const bool ok = w != kSentinel;
        const float dv = !ok ? __int_as_float(0x7f800000) : add_qn ? __fadd_rn(unpack_key(w), qq) : unpack_key(w);
        const int32_t iv = ok ? (int32_t)unpack_idx(w) : -1;
        if (c.out_dist) c.out_dist[q * c.k + j] = dv;
        if (c.out_idx) c.out_idx[q * c.k + j] = iv;
        if (c.out_idx_f) c.out_idx_f[q * c.k + j] = (float)iv;
    };
    if (m <= kRankSortMax) {
        // words are distinct (indices are): a word's place is the number of smaller words
        const ulonglong2* p2 = reinterpret_cast<const ulonglong2*>(cur);
        for (int j = tid; j < m; j += kT) {
            const uint64_t w = cur[j];
            int r = 0;
            for (int e = 0; e < m / 2; ++e) {
                const ulonglong2 x = p2[e];
                r += (x.x < w ? 1 : 0) + (x.y < w ? 1 : 0);
            }
            if (m & 1) r += cur[m - 1] < w ? 1 : 0;
            if (r < c.k) put(r, w);
        }
        for (int j = m + tid; j < c.k; j += kT) put(j, kSentinel);
        return;
    }
    const int P = pow2_at_least(m);
    for (int j = m + tid; j < P; j += kT) cur[j] = kSentinel;
    __syncthreads();
    for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = tid; i < (P >> 1); i += kT) {
                const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                const bool up = (lo & size) == 0;
                const uint64_t x = cur[lo], y = cur[hi];
                if ((x > y) == up) {
                    cur[lo] = y;
                    cur[hi] = x;
                }
            }
            // a warp's pairs stay within its own 64 words while strides are up to 32
            const int next = stride > 1 ? stride >> 1 : size;
            if (stride <= 32 && next <= 32) __syncwarp();
            else __syncthreads();
        }
    }
    for (int j = tid; j < c.k; j += kT) put(j, j < m ? cur[j] : kSentinel);
}

// Exact distances of the m rows named by list's words (direct difference, the oracle's order: eight
// partial sums over d mod 8, fixed tree), packed above their indices: eight lanes a row.  Bound by the
// round trips of a group's rows.  Rows of fewer than 128 columns: kB steps of eight columns of kR rows in
// flight, predicated (the selection of 777 queries, 512 rows of 43 columns each: 56 -> 44 us; 4,096 queries, 48
// rows of 96: 47.7 -> 42.4); longer ones sixteen steps at a time (predicated batches and batches of 32
// were slower there, by instructions and by registers: 256 columns 40 against 52 and 51 us).
template <int kT, int kR, int kB>
__device__ __forceinline__ void rerank_rows(uint64_t* list, int m, const float* __restrict__ corpus, int64_t ldc,
                                            const float* qv, int D)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = lane & 7, g = lane >> 3;
    for (int j0 = 4 * kR * warp; j0 < m; j0 += kT / 8 * kR) {
        uint32_t idx[kR];
        float p[kR], v[kR][kB];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const int j = j0 + 4 * r + g;
            idx[r] = j < m ? unpack_idx(list[j]) : 0u;
            const float* row = corpus + (int64_t)idx[r] * ldc + u;
            p[r] = 0.f;
#pragma unroll
            for (int t = 0; t < kB; ++t)
                if (8 * t + u < D) v[r][t] = __ldg(row + 8 * t);
        }
#pragma unroll
        for (int t = 0; t < kB; ++t)
            if (8 * t + u < D) {
                const float y = qv[8 * t + u];
#pragma unroll
                for (int r = 0; r < kR; ++r) {
                    const float x = __fsub_rn(y, v[r][t]);
                    p[r] = __fmaf_rn(x, x, p[r]);
                }
            }
        __syncwarp();
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            // ((p0 + p1) + (p2 + p3)) + ((p4 + p5) + (p6 + p7))
            float s = __fadd_rn(p[r], __shfl_xor_sync(0xffffffffu, p[r], 1));
            s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 2));
            s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 4));
            const int j = j0 + 4 * r + g;
            if (u == 0 && j < m) list[j] = pack_key(s, idx[r]);
        }
    }
}

template <int kT>
__device__ __forceinline__ void rerank_block(uint64_t* list, int m, const float* __restrict__ corpus, int64_t ldc,
                                             const float* qv, int D)
{
    if (D <= 32) return rerank_rows<kT, 4, 4>(list, m, corpus, ldc, qv, D);
    if (D <= 64) return rerank_rows<kT, 2, 8>(list, m, corpus, ldc, qv, D);
    if (D < 128) return rerank_rows<kT, 1, 16>(list, m, corpus, ldc, qv, D);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = lane & 7, g = lane >> 3;
    const int full = D >> 3;  // whole steps of eight columns
    for (int j0 = 4 * warp; j0 < m; j0 += kT / 8) {
        const int j = j0 + g;
        const uint32_t idx = j < m ? unpack_idx(list[j]) : 0u;
        const float* row = corpus + (int64_t)idx * ldc + u;
        float p = 0.f;
        int i = 0;
        for (; i + 16 <= full; i += 16) {
            float v[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) v[t] = __ldg(row + 8 * (i + t));
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const float x = __fsub_rn(qv[8 * (i + t) + u], v[t]);
                p = __fmaf_rn(x, x, p);
            }
        }
        for (; i < full; i += 4) {
            float v[4];
#pragma unroll
            for (int t = 0; t < 4; ++t) v[t] = i + t < full ? __ldg(row + 8 * (i + t)) : 0.f;
#pragma unroll
            for (int t = 0; t < 4; ++t)
                if (i + t < full) {
                    const float x = __fsub_rn(qv[8 * (i + t) + u], v[t]);
                    p = __fmaf_rn(x, x, p);
                }
        }
        if (8 * full + u < D) {
            const float x = __fsub_rn(qv[8 * full + u], __ldg(row + 8 * full));
            p = __fmaf_rn(x, x, p);
        }
        // ((p0 + p1) + (p2 + p3)) + ((p4 + p5) + (p6 + p7))
        p = __fadd_rn(p, __shfl_xor_sync(0xffffffffu, p, 1));
        p = __fadd_rn(p, __shfl_xor_sync(0xffffffffu, p, 2));
        p = __fadd_rn(p, __shfl_xor_sync(0xffffffffu, p, 4));
        if (u == 0 && j < m) list[j] = pack_key(p, idx);
    }
}

// The bin of a 256-bin histogram where the running count reaches rank: its digit, the rank within it
// and its count, by the calling warp.
__device__ __forceinline__ void find_bin(const uint32_t* hist, uint32_t rank, uint32_t& digit, uint32_t& within,
                                         uint32_t& count)
{
    const int lane = threadIdx.x & 31;
    uint32_t b[8], s = 0;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        b[u] = hist[8 * lane + u];
        s += b[u];
    }
    uint32_t inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    uint32_t run = inc - s;
    if (run < rank && inc >= rank) {
        bool found = false;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (!found && run + b[u] >= rank) {
                digit = (uint32_t)(8 * lane + u);
                within = rank - run;
                count = b[u];
                found = true;
            }
            run += b[u];
        }
    }
}

// Shortlists by split-FP16 keys where the shape's keys are FP32 ones otherwise (corpora below 16,384 rows, more than
// 128 columns or entries): the split's products are coarser than FP32's, so such a shortlist counts only if no row
// outside it can be nearer than its k-th (else: widen, or the CUDA-core fix-up).  split_key_error: what the key of a row
// within C of the origin can err by against a query of squared norm qq, both as FP32 sums,
//   2 |q| C (3 n + 4) 2^-22   products: n = D / 16 steps of three MMAs, two ulps of the accumulator a step (measured:
//                             half an ulp, by truncation; 1,024 uniform columns 5.9e-6 |q| |c| in all against
//                             4.7e-5 here); split residues
//   (C^2 + |q| C) 2^-22       the norm's and the key's own roundings
//   |q|^2 2^-17               ||q||^2 as summed here
//   D 1e-44                   squares in the subnormal range
// 10,000 x 300 uniform rows: 3e-3 in all, the 10th and 32nd neighbours 0.7 apart.
__device__ __forceinline__ float split_key_error(float qq, float C, int D)
{
    const float R = sqrtf(qq);
    return 2.f * R * C * (float)(3 * ((D + 15) / 16) + 4) * 0x1p-22f + (C * C + R * C) * 0x1p-22f + qq * 0x1p-17f +
           (float)D * 1e-44f;
}
// relative error of a re-ranked distance
__device__ __forceinline__ float dist_error(int D) { return (float)(D / 8 + 8) * 0x1p-24f; }

// Lower bound on the re-ranked distance of rows whose keys are `key` or more: one at a squared distance below S = key +
// ||q||^2 has |c| <= |q| + sqrt(S).  -inf when nothing is sure.
__device__ __forceinline__ float outside_bound(float key, float qq, int D)
{
    const float S = key + qq;
    const float b = (S - split_key_error(qq, sqrtf(qq) + sqrtf(fmaxf(S, 0.f)), D)) * (1.f - dist_error(D));
    return b > 0.f ? b : -__int_as_float(0x7f800000);  // (NaN: -inf)
}

// Whether k of the re-ranked list's distances lie below the bound.
template <int kT>
__device__ __forceinline__ bool list_holds(const uint64_t* list, int m, int k, float bound)
{
    int n = 0;
    for (int j0 = 0; j0 < m; j0 += kT) {
        const int j = j0 + (int)threadIdx.x;
        n += __syncthreads_count(j < m && unpack_key(list[j]) < bound);
    }
    return n >= k;
}

// kThr: threshold mode -- the next float above the key of rank thr_rank, or the fallback.  Blocks an SM:
// ten of 128 threads (47 registers; at 63 a million rows' 10,000 queries take 97 instead of 88 us), four
// of 256 (for the re-rank's loads in flight: 256 queries, 32 rows of 1,024 columns 18.9 -> 15.5 us).
template <int kT, bool kThr, bool kSmall = false>
__global__ void __launch_bounds__(kT, kT == 128 ? 10 : 1024 / kT) select_block_kernel(const CandSelect c)
{
    if (c.skip_if != nullptr && *c.skip_if != 0u) return;
    if (c.skip_if_zero != nullptr && *c.skip_if_zero == 0u) return;
    constexpr int kW = kT / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t* cur = reinterpret_cast<uint64_t*>(smem);               // shortlist [pow2_at_least(kp)]
    uint64_t* buf = kThr ? cur : cur + pow2_at_least(c.kp);           // candidates [buf_words]
    float* qv = reinterpret_cast<float*>(buf + c.buf_words);         // query [D]
    __shared__ uint32_t hist[256];
    __shared__ uint64_t wmin[kW], wmax[kW];
    __shared__ uint32_t wtot[kW], digit_s, rank_s, hit_s, m_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t q = blockIdx.x;

    if (!kThr && c.rerank)
        for (int d = tid; d < c.D; d += kT) qv[d] = __ldg(c.queries + q * c.ldq + d);
    // segment counts: thread t owns segments t, t + kT, ...
    constexpr int kSeg = kScanMaxSegs / kT;
    uint32_t n[kSeg], mine = 0;
    bool over = false;
#pragma unroll
    for (int r = 0; r < kSeg; ++r) {
        const int s = tid + kT * r;
        n[r] = s < c.nseg ? __ldg(c.cnt + (size_t)s * c.Q + q) : 0u;
        over |= n[r] > (uint32_t)c.cap;
        mine += n[r];
    }
    uint32_t pre = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, pre, o);
        if (lane >= o) pre += v;
    }
    if (lane == 31) wtot[warp] = pre;
    if (tid == 0) m_s = 0;
    const bool overflow = __syncthreads_or(over) != 0;
    uint32_t at = pre - mine, total = 0;
#pragma unroll
    for (int w = 0; w < kW; ++w) {
        const uint32_t t = wtot[w];
        if (w < warp) at += t;
        total += t;
    }
    if (kThr && (overflow || total < (uint32_t)c.thr_rank || total > (uint32_t)c.buf_words)) {
        if (tid == 0) c.thr_out[q] = c.thr_fallback ? c.thr_fallback[q] : __int_as_float(0x7f800000);
        return;
    }
    if (!kThr && (overflow || total < (uint32_t)c.need || total > (uint32_t)c.buf_words)) {
        if constexpr (kSmall) {
            // a query that is not finite has no split keys, and with them no results
            bool odd = false;
            for (int d = tid; d < c.D; d += kT) odd |= !(fabsf(__ldg(c.queries + q * c.ldq + d)) < __int_as_float(0x7f800000));
            if (!c.certify && __syncthreads_or(odd)) {
                emit_sorted<kT>(c, q, cur, 0, false, 0.f);
                return;
            }
        }
        if (tid == 0) {
            const uint32_t pos = atomicAdd(c.fail_cnt, 1u);
            c.fail_idx[pos] = (int32_t)q;
            c.fail_thr[pos] = 0xFFFFFFFFu;
        }
        return;
    }
    uint64_t lo = kSentinel, hi = 0;
#pragma unroll
    for (int r = 0; r < kSeg; ++r) {
        const uint64_t* src = c.cand + ((size_t)(tid + kT * r) * c.Q + q) * c.cap;
        for (uint32_t i0 = 0; i0 < n[r]; i0 += 8) {
            uint64_t v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = i0 + u < n[r] ? __ldg(src + i0 + u) : 0ull;
#pragma unroll
            for (int u = 0; u < 8; ++u)
                if (i0 + u < n[r]) {
                    const uint64_t w = raw_to_ordered(v[u]);
                    buf[at + i0 + u] = w;
                    lo = w < lo ? w : lo;
                    hi = w > hi ? w : hi;
                }
        }
        at += n[r];
    }
    const int nn = (int)total, kp = kThr ? c.thr_rank : c.kp;
    uint64_t W = hi;
    int m = nn;
    uint64_t* list = buf;
    if (nn > kp) {
        // W: the kp-th smallest word; words share the bits above the highest differing one
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const uint64_t a = __shfl_xor_sync(0xffffffffu, lo, o), b = __shfl_xor_sync(0xffffffffu, hi, o);
            lo = a < lo ? a : lo;
            hi = b > hi ? b : hi;
        }
        if (lane == 0) {
            wmin[warp] = lo;
            wmax[warp] = hi;
        }
        for (int b = tid; b < 256; b += kT) hist[b] = 0;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kW; ++w) {
            lo = wmin[w] < lo ? wmin[w] : lo;
            hi = wmax[w] > hi ? wmax[w] : hi;
        }
        int top = 64 - __clzll((long long)(lo ^ hi));  // bits [0, top) differ (nn > kp >= 1: words are distinct)
        uint64_t x = top >= 64 ? 0ull : (lo >> top) << top;
        uint32_t rank = (uint32_t)kp;                   // among the words that share x's bits [top, 64)
        for (;;) {
            const int sh = max(top - 8, 0);
            const uint64_t mask = top >= 64 ? 0ull : ~((1ull << top) - 1ull);
            for (int e = tid; e < nn; e += kT) {
                const uint64_t w = buf[e];
                if ((w & mask) == x) atomicAdd(&hist[(uint32_t)(w >> sh) & ((1u << (top - sh)) - 1u)], 1u);
            }
            __syncthreads();
            if (warp == 0) find_bin(hist, rank, digit_s, rank_s, hit_s);
            __syncthreads();
            x |= (uint64_t)digit_s << sh;
            rank = rank_s;
            top = sh;
            if (rank == hit_s || sh == 0) break;  // the bin ends exactly at rank kp
            for (int b = tid; b < 256; b += kT) hist[b] = 0;
            __syncthreads();
        }
        W = top > 0 ? x | ((1ull << top) - 1ull) : x;
        for (int e0 = 0; !kThr && e0 < nn; e0 += kT) {
            const int e = e0 + tid;
            const uint64_t w = e < nn ? buf[e] : kSentinel;
            const bool keep = e < nn && w <= W;
            const uint32_t bal = __ballot_sync(0xffffffffu, keep);
            uint32_t base = 0;
            if (lane == 0 && bal) base = atomicAdd(&m_s, (uint32_t)__popc(bal));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (keep) cur[base + __popc(bal & ((1u << lane) - 1u))] = w;
        }
        m = kp;
        list = cur;
    }
    if constexpr (kThr) {
        // the key of rank thr_rank: the largest word not above W (nn == kp: the largest of all)
        uint64_t best = 0;
        if (nn > kp) {
            for (int e = tid; e < nn; e += kT)
                if (buf[e] <= W && buf[e] > best) best = buf[e];
        } else {
            best = hi;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const uint64_t b = __shfl_xor_sync(0xffffffffu, best, o);
            best = b > best ? b : best;
        }
        __syncthreads();
        if (lane == 0) wmax[warp] = best;
        __syncthreads();
        if (tid == 0) {
#pragma unroll
            for (int w = 0; w < kW; ++w) best = wmax[w] > best ? wmax[w] : best;
            const float key = unpack_key(best);
            // strictly above the key of rank thr_rank: that key itself passes a "< T" test
            c.thr_out[q] = key < __int_as_float(0x7f800000) ? nextafterf(key, __int_as_float(0x7f800000)) : key;
        }
        return;
    }
    __syncthreads();

    // exact integer keys: the ranking by key is the ranking by distance, distance = key + ||q||^2
    bool exact = false;
    if (c.int_stats != nullptr && c.qn != nullptr) {
        const float mx = __uint_as_float(__ldg(c.int_stats + 1));
        exact = __ldg(c.int_stats) == 0u && (c.bf16_inexact == nullptr || __ldg(c.bf16_inexact) == 0u) &&
                2.0 * (double)c.D * (double)mx * (double)mx < 16777216.0;
    }
    const bool rr = c.rerank && !exact;
    float bound = 0.f;
    if (kSmall && c.certify) {
        // the largest key of the shortlist, and ||q||^2
        __shared__ uint32_t wkey[kW];
        __shared__ float wqq[kW];
        uint32_t key = 0;
        float qq = 0.f;
        for (int j = tid; j < m; j += kT) key = max(key, (uint32_t)(list[j] >> 32));
        for (int d = tid; d < c.D; d += kT) qq = __fmaf_rn(qv[d], qv[d], qq);
        key = __reduce_max_sync(0xffffffffu, key);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) qq += __shfl_xor_sync(0xffffffffu, qq, o);
        if (lane == 0) {
            wkey[warp] = key;
            wqq[warp] = qq;
        }
        __syncthreads();
        qq = 0.f;
#pragma unroll
        for (int w = 0; w < kW; ++w) {
            key = max(key, wkey[w]);
            qq += wqq[w];
        }
        bound = outside_bound(ord2f(key), qq, c.D);
    }
    if (rr) {
        rerank_block<kT>(list, m, c.corpus, c.ldc, qv, c.D);
        __syncthreads();
    }
    if (kSmall && c.certify) {
        if (!list_holds<kT>(list, m, c.k, bound)) {
            if (tid == 0) {
                const uint32_t pos = atomicAdd(c.fail_cnt, 1u);
                c.fail_idx[pos] = (int32_t)q;
                c.fail_thr[pos] = 0xFFFFFFFFu;
            }
            return;
        }
    }
    emit_sorted<kT>(c, q, list, m, !rr, rr ? 0.f : __ldg(c.qn + q));
}

// n keys of a dense row as ordered words into shared memory (padding and values that are not finite as
// +inf), eight 16-byte loads of a thread in flight; lo / hi / cnt: the thread's smallest and largest
// finite word, and how many.  Rows are padded to whole tiles, so the last 16 bytes may lie past n.
template <int kT>
__device__ __forceinline__ void load_ordered(const float* __restrict__ row, int n, uint32_t* ord, uint32_t& lo,
                                             uint32_t& hi, uint32_t& cnt)
{
    constexpr uint32_t kInf = 0xFF800000u;  // f2ord(+inf)
    for (int i0 = 4 * (int)threadIdx.x; i0 < n; i0 += 32 * kT) {
        float4 v[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int i = i0 + 4 * kT * b;
            if (i < n) v[b] = __ldg(reinterpret_cast<const float4*>(row + i));
        }
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int i = i0 + 4 * kT * b;
            if (i >= n) break;
            const float f[4] = {v[b].x, v[b].y, v[b].z, v[b].w};
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                o[e] = f[e] < __int_as_float(0x7f800000) && i + e < n ? f2ord(f[e]) : kInf;
                if (o[e] < kInf) {
                    lo = min(lo, o[e]);
                    hi = max(hi, o[e]);
                    ++cnt;
                }
            }
            *reinterpret_cast<uint4*>(ord + i) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
}

// ---------------------------------------------------------------- thresholds from dense keys
// One block per query: the keys, as ordered words, into shared memory.  Ranks up to kDenseRank: the
// rank-th smallest of 32 group minima (four threads each, or sixteen) bounds the key of that rank from above, so
// only the few keys up to it are collected and the rank among them counted.  Otherwise the key is
// found by a byte-wise histogram search from the highest bit in which the finite keys differ.
// Latency-bound for few queries (48 x 3,907 keys 6.3 us, 11.9 by histogram), by issue slots for many
// (10,000 x 1,954 keys 35 us against 60).
constexpr int kDenseRank = 24;
constexpr int kDenseList = 256;
template <int kDenseT>
__global__ void __launch_bounds__(kDenseT) dense_threshold_kernel(const float* __restrict__ keys, int64_t ldk, int n,
                                                                  int rank, float* __restrict__ thr_out,
                                                                  uint32_t* clear, const uint32_t* skip_if,
                                                                  const uint32_t* skip_if_zero)
{
    if (blockIdx.x == 0 && threadIdx.x == 0 && clear != nullptr) *clear = 0u;
    if (skip_if != nullptr && *skip_if != 0u) return;
    if (skip_if_zero != nullptr && *skip_if_zero == 0u) return;
    extern __shared__ __align__(16) uint32_t ord[];  // [n rounded up to 4]
    __shared__ uint32_t hist[256];
    __shared__ uint32_t wlo[kDenseT / 32], whi[kDenseT / 32], wcnt[kDenseT / 32], digit_s, rank_s, hit_s;
    __shared__ uint32_t gmin[32], list_n;
    __shared__ __align__(16) uint32_t list[kDenseList];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t q = blockIdx.x;
    if (tid == 0) list_n = 0;
    constexpr uint32_t kInf = 0xFF800000u;  // f2ord(+inf); NaN keys count as +inf
    const float* row = keys + q * ldk;
    uint32_t lo = 0xFFFFFFFFu, hi = 0u, cnt = 0;
    load_ordered<kDenseT>(row, n, ord, lo, hi, cnt);
    const uint32_t mine = lo;
    constexpr int kGroup = kDenseT / 32;  // threads a group
    uint32_t g = lo;
#pragma unroll
    for (int o = 1; o < kGroup; o <<= 1) g = min(g, __shfl_xor_sync(0xffffffffu, g, o));
    if ((lane & (kGroup - 1)) == 0) gmin[tid / kGroup] = g;
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
        wlo[warp] = lo;
        whi[warp] = hi;
        wcnt[warp] = cnt;
    }
    for (int b = tid; b < 256; b += kDenseT) hist[b] = 0;
    __syncthreads();
    cnt = 0;
#pragma unroll
    for (int w = 0; w < kDenseT / 32; ++w) {
        lo = min(lo, wlo[w]);
        hi = max(hi, whi[w]);
        cnt += wcnt[w];
    }
    if (cnt < (uint32_t)rank) {
        if (tid == 0) thr_out[q] = __int_as_float(0x7f800000);
        return;
    }
    if (rank <= kDenseRank) {
        // every warp ranks the 32 minima (ties by group), one per lane
        const uint32_t v = gmin[lane];
        int less = 0;
#pragma unroll
        for (int o = 0; o < 32; ++o) {
            const uint32_t w = __shfl_sync(0xffffffffu, v, o);
            less += w < v || (w == v && o < lane) ? 1 : 0;
        }
        const uint32_t at = __ballot_sync(0xffffffffu, less == rank - 1);
        const uint32_t U = __shfl_sync(0xffffffffu, v, __ffs((int)at) - 1);
        if (U < kInf) {  // at least `rank` keys are not above U
            if (mine <= U)
                for (int i = 4 * tid; i < n; i += 4 * kDenseT)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (ord[i + u] <= U) {
                            const uint32_t pos = atomicAdd(&list_n, 1u);
                            if (pos < kDenseList) list[pos] = ord[i + u];
                        }
            __syncthreads();
            const int m = (int)list_n;
            if (m <= kDenseList) {
                for (int j = tid; j < m; j += kDenseT) {
                    const uint32_t w = list[j];
                    int below = 0, same = 0;
                    for (int e = 0; e < m; ++e) {
                        below += list[e] < w ? 1 : 0;
                        same += list[e] == w ? 1 : 0;
                    }
                    // equal keys write the same word
                    if (below < rank && below + same >= rank) thr_out[q] = nextafterf(ord2f(w), __int_as_float(0x7f800000));
                }
                return;
            }
        }
    }
    int top = 32 - __clz((int)(lo ^ hi));  // bits [0, top) differ
    uint32_t x = top >= 32 ? 0u : (lo >> top) << top, r = (uint32_t)rank;
    while (top > 0) {
        const int sh = max(top - 8, 0);
        const uint32_t mask = top >= 32 ? 0u : ~((1u << top) - 1u);
        for (int i = 4 * tid; i < n; i += 4 * kDenseT) {
            const uint4 v = *reinterpret_cast<const uint4*>(ord + i);
            const uint32_t o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (o[u] < kInf && (o[u] & mask) == x) atomicAdd(&hist[(o[u] >> sh) & ((1u << (top - sh)) - 1u)], 1u);
        }
        __syncthreads();
        if (warp == 0) find_bin(hist, r, digit_s, rank_s, hit_s);
        __syncthreads();
        x |= digit_s << sh;
        r = rank_s;
        top = sh;
        if (top == 0 || (hit_s == 1u)) break;
        for (int b = tid; b < 256; b += kDenseT) hist[b] = 0;
        __syncthreads();
    }
    if (top > 0 && hit_s == 1u) {
        // a single key in the bin: it is the one
        const uint32_t mask = ~((1u << top) - 1u);
        for (int i = tid; i < n; i += kDenseT)
            if (ord[i] < kInf && (ord[i] & mask) == x) {
                const float key = ord2f(ord[i]);
                thr_out[q] = nextafterf(key, __int_as_float(0x7f800000));
            }
    } else if (tid == 0) {
        // strictly above the key of that rank: the key itself passes a "< T" test
        thr_out[q] = nextafterf(ord2f(x), __int_as_float(0x7f800000));
    }
}

// Many queries over few keys: a warp per query.  A block per query spends 21 of its 36 us for 10,000 queries x
// 1,954 keys on starting and joining blocks; here all warps are resident at once (17.5 us; 4,096 x 489 keys 5.2
// against 10.4; 2,048 x 3,907 12.1 against 13.7; 1,000 x 6,250 26 against 14: not there).  The rank-th
// smallest lane minimum bounds the wanted key; a second read collects the few keys up to it.  Fewer than
// rank lanes with finite keys, or more keys than the list holds (ties): the key is found by repeated minima.
constexpr int kDenseWarps = 8;
constexpr int kDenseWarpKeys = 4096;
constexpr int kDenseWarpList = 64;
__global__ void __launch_bounds__(32 * kDenseWarps) dense_threshold_warp_kernel(
    const float* __restrict__ keys, int64_t ldk, int n, int rank, int64_t Q, float* __restrict__ thr_out, uint32_t* clear,
    const uint32_t* skip_if, const uint32_t* skip_if_zero)
{
    if (blockIdx.x == 0 && threadIdx.x == 0 && clear != nullptr) *clear = 0u;
    if (skip_if != nullptr && *skip_if != 0u) return;
    if (skip_if_zero != nullptr && *skip_if_zero == 0u) return;
    __shared__ float lists[kDenseWarps][kDenseWarpList];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t q = (int64_t)blockIdx.x * kDenseWarps + warp;
    if (q >= Q) return;
    const float inf = __int_as_float(0x7f800000);
    const float* row = keys + q * ldk;
    float* list = lists[warp];
    float mine = inf;
    for (int i0 = 4 * lane; i0 - 4 * lane < n; i0 += 1024) {
        float4 v[8];
#pragma unroll
        for (int b = 0; b < 8; ++b)
            v[b] = i0 + 128 * b < n ? __ldg(reinterpret_cast<const float4*>(row + i0 + 128 * b)) : make_float4(inf, inf, inf, inf);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int i = i0 + 128 * b;
            // rows are padded to whole tiles, so the last 16 bytes may lie past n (minima ignore NaN)
            mine = fminf(mine, i < n ? v[b].x : inf);
            mine = fminf(mine, i + 1 < n ? v[b].y : inf);
            mine = fminf(mine, i + 2 < n ? v[b].z : inf);
            mine = fminf(mine, i + 3 < n ? v[b].w : inf);
        }
    }
    // the lanes' minima in order (ties by lane)
    int less = 0;
#pragma unroll
    for (int o = 0; o < 32; ++o) {
        const float w = __shfl_sync(0xffffffffu, mine, o);
        less += w < mine || (w == mine && o < lane) ? 1 : 0;
    }
    const float U = __shfl_sync(0xffffffffu, mine, __ffs((int)__ballot_sync(0xffffffffu, less == rank - 1)) - 1);
    int m = 0;
    if (U < inf) {
        for (int i0 = 4 * lane; i0 - 4 * lane < n; i0 += 128) {
            const float4 v = i0 < n ? __ldg(reinterpret_cast<const float4*>(row + i0)) : make_float4(inf, inf, inf, inf);
            const float f[4] = {v.x, v.y, v.z, v.w};
            if (!__any_sync(0xffffffffu, mine <= U && (f[0] <= U || f[1] <= U || f[2] <= U || f[3] <= U))) continue;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool in = i0 + e < n && f[e] <= U;
                const uint32_t bal = __ballot_sync(0xffffffffu, in);
                const int at = m + __popc(bal & ((1u << lane) - 1u));
                if (in && at < kDenseWarpList) list[at] = f[e];
                m += __popc(bal);
            }
        }
        __syncwarp();
        if (m <= kDenseWarpList) {
            for (int j = lane; j < m; j += 32) {
                const float w = list[j];
                int below = 0, same = 0;
                for (int e = 0; e < m; ++e) {
                    below += list[e] < w ? 1 : 0;
                    same += list[e] == w ? 1 : 0;
                }
                // equal keys write the same word
                if (below < rank && below + same >= rank) thr_out[q] = nextafterf(w, inf);
            }
            return;
        }
    }
    // the smallest keys one value after the other
    float last = -inf, T = inf;
    bool first = true;
    for (int left = rank; left > 0; first = false) {
        float best = inf;
        for (int i = lane; i < n; i += 32) {
            const float f = __ldg(row + i);
            if (f < best && (first || f > last)) best = f;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, o));
        if (!(best < inf)) break;  // fewer than rank finite keys
        uint32_t same = 0;
        for (int i = lane; i < n; i += 32) same += __ldg(row + i) == best ? 1u : 0u;
        left -= (int)__reduce_add_sync(0xffffffffu, same);
        last = best;
        if (left <= 0) T = nextafterf(best, inf);
    }
    if (lane == 0) thr_out[q] = T;
}

cudaError_t launch_dense_threshold(const float* keys, int64_t ldk, int n, int rank, int64_t Q, float* thr_out,
                                   uint32_t* clear, const uint32_t* skip_if, const uint32_t* skip_if_zero,
                                   cudaStream_t s)
{
    if (Q <= 0) return cudaSuccess;
    if (n < 1 || n > kDenseRows || rank < 1 || ldk % 4 != 0 || ldk < n) return cudaErrorInvalidValue;
    const size_t smem = (size_t)((n + 3) & ~3) * 4;
    if (Q > kThrBlockQ && n <= kDenseWarpKeys && rank <= kDenseRank)
        dense_threshold_warp_kernel<<<(unsigned)((Q + kDenseWarps - 1) / kDenseWarps), 32 * kDenseWarps, 0, s>>>(
            keys, ldk, n, rank, Q, thr_out, clear, skip_if, skip_if_zero);
    else if (Q <= kSelFewQ)
        dense_threshold_kernel<512><<<(unsigned)Q, 512, smem, s>>>(keys, ldk, n, rank, thr_out, clear, skip_if, skip_if_zero);
    else
        dense_threshold_kernel<128><<<(unsigned)Q, 128, smem, s>>>(keys, ldk, n, rank, thr_out, clear, skip_if, skip_if_zero);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- small corpora
// A block per query over the values of every row (SmallSelect), which sit in shared memory as ordered
// words.  For short shortlists the need-th smallest of the threads' minima (one value a thread, by a
// byte-wise histogram search) bounds the need-th smallest of all, and the few words up to it are
// collected and ranked by counting; otherwise the search runs over all the words, ties at the end by
// index (10,000 keys, 500 queries, shortlist 32: 21.5 us that way).  Direct mode
// computes the exact distances first, eight lanes a row, four rows a lane in flight: one launch serves
// the whole search, bound by the reads of the corpus from L2 (each block reads all of it).
// Direct mode's distances alone decide while every squared norm and distance stays below kDirectMost: then no
// norm and no key ||c||^2 - 2 q.c leaves the float range.  Otherwise the rows are ranked by their FP32 keys as
// everywhere else (small_keys), so that a row whose norm or key overflows is no result and one whose distance
// alone does is (+inf, its index).
constexpr int kSmallList = 256;
constexpr float kDirectMost = 1e37f;

// Every row's key as an ordered word (+inf where it is not below +inf), a thread a row, sixteen columns in flight: in
// the arithmetic of the CUDA-core kernel where the shape's keys are FP32 ones; otherwise from a product q.c whose
// partial sums do not overflow, as a tensor-core step adds its products.  Norms: the search's (cn), or here a
// compensated float sum (the FP64 pipe took ten times as long as the rest).  A query with infinite values has FP32
// keys, which those values decide, but no split keys.
static __device__ __noinline__ void small_keys(const SmallSelect& c, const float* qv, bool finite, uint32_t* ord)
{
    constexpr uint32_t kInf = 0xFF800000u;
    constexpr int kB = 16;
    const float inf = __int_as_float(0x7f800000);
    float big = 0.f;
    if (!c.fp32_keys)
        for (int d = 0; d < c.D; ++d) big = fmaxf(big, fabsf(qv[d]));
    // (a row with a norm lies below 2^64)
    const float down = big >= 0x1p32f ? 0x1p-80f : 1.f, up = big >= 0x1p32f ? 0x1p80f : 1.f;
    for (int i = threadIdx.x; i < c.n; i += blockDim.x) {
        const float* row = c.corpus + (int64_t)i * c.ldc;
        float dot = 0.f, n0 = 0.f, n1 = 0.f;
        if (!finite && c.cn != nullptr)
            for (int d = 0; d < c.D; ++d)
                if (!(fabsf(qv[d]) < inf)) dot = __fmaf_rn(qv[d], __ldg(row + d), dot);
        for (int d0 = 0; d0 < c.D && (finite || c.cn == nullptr); d0 += kB) {
            float v[kB];
#pragma unroll
            for (int e = 0; e < kB; ++e) v[e] = d0 + e < c.D ? __ldg(row + d0 + e) : 0.f;
#pragma unroll
            for (int e = 0; e < kB; ++e)
                if (d0 + e < c.D) {
                    dot = __fmaf_rn(qv[d0 + e] * down, v[e], dot);
                    if (c.cn == nullptr) {
                        // n0 + n1 += v^2: the square's residual and the sum's (TwoSum)
                        const float sq = __fmul_rn(v[e], v[e]), s = __fadd_rn(n0, sq), b = __fsub_rn(s, n0);
                        n1 += __fmaf_rn(v[e], v[e], -sq) + (__fsub_rn(n0, __fsub_rn(s, b)) + __fsub_rn(sq, b));
                        n0 = s;
                    }
                }
        }
        const float norm = c.cn != nullptr ? __ldg(c.cn + i) : n0 < inf ? __fadd_rn(n0, n1) : n0;
        const float key = __fmaf_rn(-2.0f, dot * up, norm);
        ord[i] = (c.fp32_keys || finite) && key < inf ? f2ord(key) : kInf;
    }
}

// The exact distances of cur[0..m) (a thread a row) over their keys.
static __device__ __noinline__ void small_rerank(const SmallSelect& c, const float* qv, uint64_t* cur, int m)
{
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const uint32_t i = unpack_idx(cur[j]);
        cur[j] = pack_key(exact_dist_row(qv, c.corpus + (int64_t)i * c.ldc, c.D), i);
    }
}

// A shortlist of split keys that is not certain to hold the k nearest (its re-ranked words cur[0..m), qq: ||q||^2):
// the exact distances of every row that its key does not rule out, as words over the keys, +inf for the others.
// A row at the k-th distance of the shortlist or nearer has |c| <= |q| + that distance, so its key lies below U.
// Eight lanes a row, each warp 32 rows in turn (10,000 x 300, 500 queries, every column offset by 20, which leaves a
// tenth of the rows: 245 us a search; by 80, which leaves all, 1,364.  Two rows a group, eight steps each: 253 and
// 1,201, but 1,549 instead of 1,273 for 1,400 queries of 16,000 x 2,048 that few rows remain possible for).  False,
// and nothing written, where squares may leave the float range or (give_up) a quarter of the rows and more remain.
template <int kT>
static __device__ __noinline__ bool widen(const SmallSelect& c, const float* qv, float qq, const uint64_t* cur, int m,
                                          bool give_up, uint32_t* ord)
{
    constexpr uint32_t kInf = 0xFF800000u;
    constexpr int kB = 16;  // steps of eight columns in flight
    __shared__ float kth_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, u = lane & 7, g = lane >> 3;
    for (int j = threadIdx.x; j < m; j += kT) {
        const uint64_t w = cur[j];
        int below = 0;
        for (int e = 0; e < m; ++e) below += cur[e] < w ? 1 : 0;
        if (below == c.k - 1) kth_s = unpack_key(w);
    }
    __syncthreads();
    const float kth = kth_s;
    if (!(qq < kDirectMost) || !(kth < kDirectMost)) return false;
    const float S = kth * (1.f + 2.f * dist_error(c.D)) + (float)c.D * 1e-44f;
    const uint32_t U = f2ord(S - qq + split_key_error(qq, sqrtf(qq) + sqrtf(S), c.D));
    if (give_up) {
        int rows = 0;
        for (int r0 = 0; r0 < c.n; r0 += kT) {
            const int r = r0 + (int)threadIdx.x;
            rows += __syncthreads_count(r < c.n && ord[r] <= U && ord[r] < kInf);
        }
        if (rows >= c.n / 4) return false;
    }
    for (int r0 = 32 * warp; r0 < c.n; r0 += kT) {
        const uint32_t o = r0 + lane < c.n ? ord[r0 + lane] : kInf;
        uint32_t todo = __ballot_sync(0xffffffffu, o <= U && o < kInf);
        if (r0 + lane < c.n && !((todo >> lane) & 1u)) ord[r0 + lane] = kInf;
        while (todo) {
            uint32_t t = todo;  // the group takes the g-th row left
            for (int i = 0; i < g; ++i) t &= t - 1u;
            const bool in = t != 0u;
            const int r = r0 + (in ? __ffs((int)t) - 1 : 0);
            const float* row = c.corpus + (int64_t)r * c.ldc + u;
            float p = 0.f;
            for (int d0 = 0; d0 < c.D; d0 += 8 * kB) {
                float v[kB];
#pragma unroll
                for (int i = 0; i < kB; ++i)
                    if (in && d0 + 8 * i + u < c.D) v[i] = __ldg(row + d0 + 8 * i);
#pragma unroll
                for (int i = 0; i < kB; ++i)
                    if (in && d0 + 8 * i + u < c.D) {
                        const float x = __fsub_rn(qv[d0 + 8 * i + u], v[i]);
                        p = __fmaf_rn(x, x, p);
                    }
            }
            __syncwarp();
            // ((p0 + p1) + (p2 + p3)) + ((p4 + p5) + (p6 + p7))
            p = __fadd_rn(p, __shfl_xor_sync(0xffffffffu, p, 1));
            p = __fadd_rn(p, __shfl_xor_sync(0xffffffffu, p, 2));
            p = __fadd_rn(p, __shfl_xor_sync(0xffffffffu, p, 4));
            if (u == 0 && in) ord[r] = p < __int_as_float(0x7f800000) ? f2ord(p) : kInf;
            for (int i = 0; i < 4; ++i) todo &= todo - 1u;
        }
    }
    return true;
}

// What the block shares while it picks words.
template <int kT>
struct SmallShared {
    uint32_t hist[256];
    uint32_t wlo[kT / 32], whi[kT / 32], wcnt[kT / 32], digit, rank, hit, m;
    float wqq[kT / 32];
    __align__(16) uint64_t list[kSmallList];
    float qq;  // direct mode: ||q||^2
};

// The extent of the words below +inf and their number: a thread's ...
struct WordExtent {
    uint32_t lo = 0xFFFFFFFFu, hi = 0u, cnt = 0, mine = 0;  // mine: the thread's smallest, all ones when it has none
};
template <int kT>
__device__ __forceinline__ WordExtent thread_extent(const uint32_t* ord, int n)
{
    constexpr uint32_t kInf = 0xFF800000u;
    WordExtent x;
    for (int i = 4 * (int)threadIdx.x; i < n; i += 4 * kT) {
        const uint4 v = *reinterpret_cast<const uint4*>(ord + i);
        const uint32_t o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (o[e] < kInf) {
                x.lo = min(x.lo, o[e]);
                x.hi = max(x.hi, o[e]);
                ++x.cnt;
            }
    }
    return x;
}
// ... and the block's (the words are visible to it afterwards).
template <int kT>
__device__ __forceinline__ void block_extent(SmallShared<kT>& S, WordExtent& x)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    x.mine = x.lo;
    x.lo = __reduce_min_sync(0xffffffffu, x.lo);
    x.hi = __reduce_max_sync(0xffffffffu, x.hi);
    x.cnt = __reduce_add_sync(0xffffffffu, x.cnt);
    if (lane == 0) {
        S.wlo[warp] = x.lo;
        S.whi[warp] = x.hi;
        S.wcnt[warp] = x.cnt;
    }
    __syncthreads();
    x.cnt = 0;
#pragma unroll
    for (int w = 0; w < kT / 32; ++w) {
        x.lo = min(x.lo, S.wlo[w]);
        x.hi = max(x.hi, S.whi[w]);
        x.cnt += S.wcnt[w];
    }
}

// The `need` smallest (word, index) pairs of ord[0..n) into cur, in no order; how many.  edge: no other word is smaller.
// S.hist and S.m are zero before and (S.hist) after.
template <int kT>
__device__ __forceinline__ int pick_words(SmallShared<kT>& S, const uint32_t* ord, int n, int need, const WordExtent& xt,
                                          uint64_t* cur, uint32_t& edge)
{
    constexpr uint32_t kInf = 0xFF800000u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t lo = xt.lo, hi = xt.hi, cnt = xt.cnt, mine = xt.mine;
    // keep the words not above W, and of those equal to W + 1 (when ties > 0) the first `ties`
    uint32_t W = kInf - 1u, ties = 0;
    edge = kInf;
    const int m = (int)min(cnt, (uint32_t)need);
    bool done = false;
    int top = 32 - __clz((int)(lo ^ hi));  // bits [0, top) differ
    uint32_t x = top >= 32 ? 0u : (lo >> top) << top, rank = (uint32_t)need, hit = cnt;
    if (cnt > (uint32_t)need && need <= kT / 2 && n >= 4 * kT) {
        // the need-th smallest thread minimum, or a bound on it at the end of a small bin
        int tp = top;
        uint32_t y = x, r = rank, h = kT;
        while (tp > 0 && h - r > 8u) {
            const int sh = max(tp - 8, 0);
            const uint32_t mask = tp >= 32 ? 0u : ~((1u << tp) - 1u);
            if (mine < kInf && (mine & mask) == y) atomicAdd(&S.hist[(mine >> sh) & ((1u << (tp - sh)) - 1u)], 1u);
            __syncthreads();
            if (tid == 0) S.hit = 0;
            __syncthreads();
            if (warp == 0) find_bin(S.hist, r, S.digit, S.rank, S.hit);
            __syncthreads();
            for (int b = tid; b < 256; b += kT) S.hist[b] = 0;
            __syncthreads();
            h = S.hit;
            if (h == 0) break;  // fewer than need threads hold finite words
            y |= S.digit << sh;
            r = S.rank;
            tp = sh;
        }
        if (h != 0) {
            const uint32_t U = tp > 0 ? y | ((1u << tp) - 1u) : y;
            if (mine <= U)
                for (int i = 4 * tid; i < n; i += 4 * kT)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (ord[i + e] <= U) {
                            const uint32_t pos = atomicAdd(&S.m, 1u);
                            if (pos < kSmallList) S.list[pos] = ((uint64_t)ord[i + e] << 32) | (uint32_t)(i + e);
                        }
            __syncthreads();
            const int found = (int)S.m;
            if (found <= kSmallList) {
                // words are distinct: a word's place is the number of smaller ones
                for (int j = tid; j < found; j += kT) {
                    const uint64_t w = S.list[j];
                    int below = 0;
                    for (int e = 0; e < found; ++e) below += S.list[e] < w ? 1 : 0;
                    if (below < m) cur[below] = w;
                }
                done = true;
            }
            __syncthreads();
            if (done) edge = (uint32_t)(cur[m - 1] >> 32);
            if (tid == 0) S.m = 0;
        }
        __syncthreads();
    }
    if (!done && cnt > (uint32_t)need) {
        while (top > 0 && rank != hit) {
            const int sh = max(top - 8, 0);
            const uint32_t mask = top >= 32 ? 0u : ~((1u << top) - 1u);
            for (int i = 4 * tid; i < n; i += 4 * kT) {
                const uint4 v = *reinterpret_cast<const uint4*>(ord + i);
                const uint32_t o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (o[e] < kInf && (o[e] & mask) == x) atomicAdd(&S.hist[(o[e] >> sh) & ((1u << (top - sh)) - 1u)], 1u);
            }
            __syncthreads();
            if (warp == 0) find_bin(S.hist, rank, S.digit, S.rank, S.hit);
            __syncthreads();
            x |= S.digit << sh;
            rank = S.rank;
            hit = S.hit;
            top = sh;
            for (int b = tid; b < 256; b += kT) S.hist[b] = 0;
            __syncthreads();
        }
        if (rank == hit) {
            W = top > 0 ? x | ((1u << top) - 1u) : x;
        } else {  // more words equal to x than are wanted
            W = x - 1u;
            ties = rank;
        }
        edge = W + 1u;
    }
    for (int e0 = 0; !done && e0 < n; e0 += kT) {
        const int e = e0 + tid;
        const uint32_t o = e < n ? ord[e] : kInf;
        const bool keep = o <= W && o < kInf;
        const uint32_t bal = __ballot_sync(0xffffffffu, keep);
        uint32_t base = 0;
        if (lane == 0 && bal) base = atomicAdd(&S.m, (uint32_t)__popc(bal));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (keep) cur[base + __popc(bal & ((1u << lane) - 1u))] = ((uint64_t)o << 32) | (uint32_t)e;
    }
    __syncthreads();
    if (ties > 0 && warp == 0) {
        uint32_t at = S.m, left = ties;
        for (int e0 = 0; e0 < n && left > 0; e0 += 32) {
            const int e = e0 + lane;
            const bool tie = e < n && ord[e] == W + 1u;
            const uint32_t bal = __ballot_sync(0xffffffffu, tie);
            const uint32_t pos = (uint32_t)__popc(bal & ((1u << lane) - 1u));
            if (tie && pos < left) cur[at + pos] = ((uint64_t)(W + 1u) << 32) | (uint32_t)e;
            const uint32_t took = min(left, (uint32_t)__popc(bal));
            at += took;
            left -= took;
        }
    }
    __syncthreads();
    return m;
}

// A second way to the results, for queries that the first is not certain of: `ord` becomes the exact distances of
// the rows that the shortlist cur[0..m) does not rule out (wide), or every row's FP32 key.
template <int kT>
static __device__ __noinline__ void pick_again(const SmallSelect& c, int64_t q, const float* qv, float qq, bool wide, int m,
                                               uint64_t* cur, uint32_t* ord, SmallShared<kT>& S)
{
    const float inf = __int_as_float(0x7f800000);
    bool odd = false;
    for (int d = threadIdx.x; d < c.D; d += kT) odd |= !(fabsf(qv[d]) < inf);
    const bool finite = __syncthreads_or(odd) == 0;
    if (qq != qq) {  // some value is NaN, and so is every key
        emit_sorted<kT>(c, q, cur, 0, false, 0.f);
        return;
    }
    wide = wide && widen<kT>(c, qv, qq, cur, m, c.fail_idx != nullptr, ord);
    if (!wide && c.fail_idx != nullptr) {
        if (threadIdx.x == 0) {
            const uint32_t pos = atomicAdd(c.fail_cnt, 1u);
            c.fail_idx[pos] = (int32_t)q;
            c.fail_thr[pos] = 0xFFFFFFFFu;
        }
        return;
    }
    if (!wide) {
        __syncthreads();
        small_keys(c, qv, finite, ord);
    }
    if (threadIdx.x == 0) S.m = 0;
    __syncthreads();
    WordExtent x = thread_extent<kT>(ord, c.n);
    block_extent<kT>(S, x);
    uint32_t edge;
    m = pick_words<kT>(S, ord, c.n, wide ? c.k : min(max(c.need, c.kp), c.n), x, cur, edge);
    if (!wide) {
        small_rerank(c, qv, cur, m);
        __syncthreads();
    }
    emit_sorted<kT>(c, q, cur, m, false, 0.f);
}

enum SmallMode { kSmallDense, kSmallCertified, kSmallDirect };
template <int kT, int kMode>
__global__ void __launch_bounds__(kT, kMode == kSmallCertified ? 1024 / kT : 0) select_small_kernel(const __grid_constant__ SmallSelect c)
{
    constexpr uint32_t kInf = 0xFF800000u;  // f2ord(+inf)
    extern __shared__ __align__(16) unsigned char smem[];
    const int n4 = (c.n + 3) & ~3;
    uint64_t* cur = reinterpret_cast<uint64_t*>(smem);                             // [pow2_at_least(need, kp)]
    uint32_t* ord = reinterpret_cast<uint32_t*>(cur + pow2_at_least(max(c.need, c.kp)));  // [n4]
    float* qv = reinterpret_cast<float*>(ord + n4);                                // [D]
    __shared__ SmallShared<kT> S;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t q = blockIdx.x;
    const int n = c.n;
    float qq = 0.f;  // the thread's share of ||q||^2, then all of it (certified mode)
    for (int d = tid; d < c.D; d += kT) {
        const float y = __ldg(c.queries + q * c.ldq + d);
        qv[d] = y;
        qq = __fmaf_rn(y, y, qq);
    }
    for (int b = tid; b < 256; b += kT) S.hist[b] = 0;
    if (tid == 0) S.m = 0;
    WordExtent x;
    bool over = false;  // direct mode: some distance overflows (one that is NaN has a row without a key)
    if constexpr (kMode == kSmallDirect) {
        __syncthreads();
        if (warp == 0) {
            float s = 0.f;
            for (int d = lane; d < c.D; d += 32) s = __fmaf_rn(qv[d], qv[d], s);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) S.qq = s;
        }
        constexpr int kR = 4;  // rows a lane has in flight
        const int u = lane & 7, g = lane >> 3, full = c.D >> 3;
        for (int r0 = 4 * kR * warp; r0 < n; r0 += kT / 8 * kR) {
            float p[kR];
            const float* row[kR];
#pragma unroll
            for (int t = 0; t < kR; ++t) {
                p[t] = 0.f;
                row[t] = c.corpus + (int64_t)min(r0 + 4 * t + g, n - 1) * c.ldc + u;
            }
            int i = 0;
            for (; i + 4 <= full; i += 4) {
                float v[kR][4];
#pragma unroll
                for (int t = 0; t < kR; ++t)
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[t][e] = __ldg(row[t] + 8 * (i + e));
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float y = qv[8 * (i + e) + u];
#pragma unroll
                    for (int t = 0; t < kR; ++t) {
                        const float x = __fsub_rn(y, v[t][e]);
                        p[t] = __fmaf_rn(x, x, p[t]);
                    }
                }
            }
            for (; 8 * i + u < c.D; ++i) {
                const float y = qv[8 * i + u];
#pragma unroll
                for (int t = 0; t < kR; ++t) {
                    const float x = __fsub_rn(y, __ldg(row[t] + 8 * i));
                    p[t] = __fmaf_rn(x, x, p[t]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int t = 0; t < kR; ++t) {
                // ((p0 + p1) + (p2 + p3)) + ((p4 + p5) + (p6 + p7))
                float s = __fadd_rn(p[t], __shfl_xor_sync(0xffffffffu, p[t], 1));
                s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 2));
                s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, 4));
                const int r = r0 + 4 * t + g;
                over |= s == __int_as_float(0x7f800000);
                if (u == 0 && r < n) ord[r] = s < __int_as_float(0x7f800000) ? f2ord(s) : kInf;
            }
        }
        for (int i = n + tid; i < n4; i += kT) ord[i] = kInf;
        over = __syncthreads_or(over) != 0;
        x = thread_extent<kT>(ord, n);
    } else {
        load_ordered<kT>(c.keys + q * c.ldk, n, ord, x.lo, x.hi, x.cnt);
    }
    if constexpr (kMode == kSmallCertified) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) qq += __shfl_xor_sync(0xffffffffu, qq, o);
        if (lane == 0) S.wqq[warp] = qq;
    }
    block_extent<kT>(S, x);
    if constexpr (kMode == kSmallDirect) {
        if (over || x.hi >= f2ord(kDirectMost) || !(S.qq < kDirectMost))
            return pick_again<kT>(c, q, qv, S.qq, false, 0, cur, ord, S);
    }
    uint32_t edge;
    const int m = pick_words<kT>(S, ord, n, c.need, x, cur, edge);
    if constexpr (kMode == kSmallCertified) {
        qq = 0.f;
#pragma unroll
        for (int w = 0; w < kT / 32; ++w) qq += S.wqq[w];
        rerank_block<kT>(cur, m, c.corpus, c.ldc, qv, c.D);
        __syncthreads();
        // every row with a key, or k results that no other row can precede
        const bool every = x.cnt <= (uint32_t)c.need;
        if (!(every ? qq < __int_as_float(0x7f800000) : list_holds<kT>(cur, m, c.k, outside_bound(ord2f(edge), qq, c.D))))
            return pick_again<kT>(c, q, qv, qq, !every, m, cur, ord, S);
    } else if constexpr (kMode == kSmallDense) {
        rerank_block<kT>(cur, m, c.corpus, c.ldc, qv, c.D);
        __syncthreads();
    }
    emit_sorted<kT>(c, q, cur, m, false, 0.f);
}

template <int kT, int kMode>
static cudaError_t run_select_small(const SmallSelect& c, size_t smem, cudaStream_t s)
{
    cudaError_t e = reserve_smem((const void*)select_small_kernel<kT, kMode>, smem);
    if (e != cudaSuccess) return e;
    select_small_kernel<kT, kMode><<<(unsigned)c.Q, kT, smem, s>>>(c);
    return cudaGetLastError();
}

cudaError_t launch_select_small(const SmallSelect& c, cudaStream_t s)
{
    if (c.Q <= 0) return cudaSuccess;
    if (c.n < 1 || c.n > kSmallRows || c.k < 1 || c.need < c.k || c.need > kMaxKpScan || c.D < 1 ||
        (c.keys && (c.ldk % 4 != 0 || c.ldk < c.n)) || (!c.keys && (c.kp < c.k || c.kp > kMaxKpScan)) ||
        (c.fail_idx && (!c.keys || !c.fp32_keys || !c.fail_cnt || !c.fail_thr)))
        return cudaErrorInvalidValue;
    const size_t smem = (size_t)pow2_at_least(std::max(c.need, c.kp)) * 8 + (size_t)((c.n + 3) & ~3) * 4 + (size_t)((c.D + 3) & ~3) * 4;
    if (c.keys && c.fp32_keys)
        return c.Q <= kSelWideQ ? run_select_small<512, kSmallCertified>(c, smem, s)
                                : run_select_small<256, kSmallCertified>(c, smem, s);
    if (c.keys)
        return c.Q <= kSelWideQ ? run_select_small<512, kSmallDense>(c, smem, s)
                                : run_select_small<256, kSmallDense>(c, smem, s);
    return c.Q <= kSms ? run_select_small<1024, kSmallDirect>(c, smem, s) : run_select_small<256, kSmallDirect>(c, smem, s);
}

size_t select_smem_bytes(int kp, int D, int rerank)
{
    int P = pow2_at_least(kp);
    return (size_t)kSelWarps * 3 * P * 8 + (rerank ? (size_t)kSelWarps * ((D + 3) & ~3) * 4 : 0);
}

cudaError_t launch_select(const uint64_t* part, int splits, int64_t Q, int kp, int k,
                          const float* corpus, int64_t ldc, const float* queries, int64_t ldq,
                          int D, int rerank, const float* qn, float* out_dist, int32_t* out_idx,
                          float* out_idx_f, cudaStream_t s, const SelectExtra& ex)
{
    if (Q <= 0) return cudaSuccess;
    size_t smem = select_smem_bytes(kp, D, rerank);
    cudaError_t e = reserve_smem((const void*)select_kernel, smem);
    if (e != cudaSuccess) return e;
    unsigned blocks = (unsigned)((Q + kSelWarps - 1) / kSelWarps);
    select_kernel<<<blocks, kSelWarps * 32, smem, s>>>(part, splits, Q, kp, k, corpus, ldc, queries, ldq, D,
                                                       rerank, qn, out_dist, out_idx, out_idx_f, ex);
    return cudaGetLastError();
}

// Merge of a corpus block's top-kb into the running top-k of every query (the
// reference's cross-block merge of its host-streamed corpus blocks,
// src/cuknnBitonic.cu:550-589, done on the device): both lists are sorted by
// (distance, index); block indices are shifted by the block's first row; the
// first min(k, have + kb) entries of the union in (distance, index) order go to
// the output list (and, as floats, to out_idx_f when given).  One thread per query.
__global__ void merge_topk_kernel(const float* __restrict__ run_d, const int32_t* __restrict__ run_i, int have,
                                  const float* __restrict__ blk_d, const int32_t* __restrict__ blk_i, int kb,
                                  int32_t offset, int64_t Q, int k, float* __restrict__ out_d,
                                  int32_t* __restrict__ out_i, float* __restrict__ out_idx_f)
{
    const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= Q) return;
    const float* rd = run_d + q * k;
    const int32_t* ri = run_i + q * k;
    const float* bd = blk_d + q * kb;
    const int32_t* bi = blk_i + q * kb;
    const int n = min(k, have + kb);
    int a = 0, b = 0;
    for (int j = 0; j < n; ++j) {
        bool take_a;
        if (a >= have) {
            take_a = false;
        } else if (b >= kb) {
            take_a = true;
        } else {
            const float da = rd[a], db = bd[b];
            const int32_t ia = ri[a], ib = bi[b] + offset;
            take_a = da < db || (da == db && ia < ib);
        }
        const float d = take_a ? rd[a] : bd[b];
        const int32_t i = take_a ? ri[a] : bi[b] + offset;
        a += take_a ? 1 : 0;
        b += take_a ? 0 : 1;
        out_d[q * k + j] = d;
        out_i[q * k + j] = i;
        if (out_idx_f) out_idx_f[q * k + j] = (float)i;
    }
}

cudaError_t launch_merge_topk(const float* run_d, const int32_t* run_i, int have, const float* blk_d,
                              const int32_t* blk_i, int kb, int32_t offset, int64_t Q, int k, float* out_d,
                              int32_t* out_i, float* out_idx_f, cudaStream_t s)
{
    if (Q <= 0) return cudaSuccess;
    if (k < 1 || kb < 0 || kb > k || have < 0 || have > k || (have > 0 && (!run_d || !run_i)) || !out_d || !out_i ||
        (kb > 0 && (!blk_d || !blk_i)))
        return cudaErrorInvalidValue;
    merge_topk_kernel<<<(unsigned)((Q + 127) / 128), 128, 0, s>>>(run_d, run_i, have, blk_d, blk_i, kb, offset, Q, k,
                                                                  out_d, out_i, out_idx_f);
    return cudaGetLastError();
}

cudaError_t launch_select_cand(const CandSelect& c_in, cudaStream_t s)
{
    if (c_in.Q <= 0) return cudaSuccess;
    CandSelect c = c_in;
    const bool thr = c.thr_out != nullptr;
    // threshold mode: a query stores at most nseg * cap words, often far fewer than the
    // buffer's limit at the coarse seeding levels; a smaller buffer lets more warps run
    if (thr)
        c.buf_words = (int)std::min<int64_t>(kCandThrMax, ((int64_t)c.nseg * c.cap + 31) / 32 * 32);
    else if (c.kp >= 1 && c.kp <= kMaxKpScan)
        c.buf_words = c.buf_words > 0 ? std::min(kCandMaxFew, std::max((c.buf_words + 31) / 32 * 32, pow2_at_least(c.kp)))
                                      : kCandMax;
    if (c.nseg < 1 || c.nseg > kScanMaxSegs || c.cap < 1 ||
        (!thr && (c.kp < 1 || c.kp > kMaxKpScan || c.k > c.kp || c.fail_idx == nullptr || c.fail_cnt == nullptr || c.fail_thr == nullptr ||
                  (!c.rerank && c.qn == nullptr) || (c.certify && !c.small) || (c.small && (!c.rerank || c.int_stats != nullptr)))) ||
        (thr && (c.thr_rank < 1 || c.thr_rank > kCandThrMax)))
        return cudaErrorInvalidValue;
    if (thr && c.Q <= kThrBlockQ) {
        // a block per query while warps would leave SMs idle: 62,500-row level of 2,000,000 x 128, 64 /
        // 777 / 2,048 queries 7.9 (256 threads) / 8.9 (128) / 11.5 against 17.8 / 10.0 / 9.7 us
        const size_t smem = (size_t)c.buf_words * 8;
        if (c.Q <= kSelFewQ)
            select_block_kernel<512, true><<<(unsigned)c.Q, 512, smem, s>>>(c);
        else if (c.Q <= kSelWideQ)
            select_block_kernel<256, true><<<(unsigned)c.Q, 256, smem, s>>>(c);
        else
            select_block_kernel<128, true><<<(unsigned)c.Q, 128, smem, s>>>(c);
    } else if (thr) {
        const size_t smem = (size_t)kSelWarps * c.buf_words * 8;
        cudaError_t e = reserve_smem((const void*)select_threshold_kernel, smem);
        if (e != cudaSuccess) return e;
        select_threshold_kernel<<<(unsigned)((c.Q + kSelWarps - 1) / kSelWarps), kSelWarps * 32, smem, s>>>(c);
    } else {
        // 256 threads shorten one query's chain, 128 fill the chip better once every SM has work:
        // selection of 256 / 777 queries 9.4 / 14.4 against 11.4 / 11.4 us (65,536 x 128, k = 16),
        // 31.9 / 64.0 against 50.0 / 55.5 us (100,003 x 43, k = 512, before the re-rank took two rows at a time)
        const size_t smem = ((size_t)pow2_at_least(c.kp) + c.buf_words) * 8 + (size_t)((c.D + 3) & ~3) * 4;
        const int t = c.Q <= kSelFewQ ? 512 : c.Q <= kSelWideQ ? 256 : 128;
        auto* kernel = c.small    ? (t == 512   ? select_block_kernel<512, false, true>
                                     : t == 256 ? select_block_kernel<256, false, true>
                                                : select_block_kernel<128, false, true>)
                       : t == 512 ? select_block_kernel<512, false>
                       : t == 256 ? select_block_kernel<256, false>
                                  : select_block_kernel<128, false>;
        cudaError_t e = reserve_smem((const void*)kernel, smem);
        if (e != cudaSuccess) return e;
        kernel<<<(unsigned)c.Q, t, smem, s>>>(c);
    }
    return cudaGetLastError();
}

}  // namespace knn
