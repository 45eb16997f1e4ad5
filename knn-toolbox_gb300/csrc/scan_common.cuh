// scan_common.cuh -- epilogue helpers shared by the threshold scans (scan_bf16.cu,
// scan_f16.cu, scan_tf32.cu): keys of a chunk of accumulator columns, its groups' minima,
// the append of the keys below the query's threshold to its segment, dense stores.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include "tc_ptx.cuh"

namespace knn {
namespace {

// Minimum of 8 keys (four min instructions).
__device__ __forceinline__ float min8(const float* k)
{
    return fminf(ptx::fmin3(ptx::fmin3(k[0], k[1], k[2]), ptx::fmin3(k[3], k[4], k[5]), k[6]), k[7]);
}

// Keys of a W-column chunk of scaled operands (E4M3, FP16 split), in place: ||c||^2 + m (s_c acc), with
// the corpus scales s_c at scl, m = -2 s_q.
template <int W>
__device__ __forceinline__ void chunk_scaled_keys(float (&v)[W], const float* nrm, const float* scl, float m)
{
    const float4* n4 = reinterpret_cast<const float4*>(nrm);
    const float4* s4 = reinterpret_cast<const float4*>(scl);
#pragma unroll
    for (int u = 0; u < W / 4; ++u) {
        const float4 c = n4[u], sc = s4[u];
        float t0, t1, t2, t3;
        ptx::mul2(t0, t1, v[4 * u], v[4 * u + 1], sc.x, sc.y);
        ptx::mul2(t2, t3, v[4 * u + 2], v[4 * u + 3], sc.z, sc.w);
        ptx::fma2(v[4 * u], v[4 * u + 1], t0, t1, m, c.x, c.y);
        ptx::fma2(v[4 * u + 2], v[4 * u + 3], t2, t3, m, c.z, c.w);
    }
}

// Keys of a W-column chunk of unscaled operands, in place: ||c||^2 - 2 acc.
template <int W>
__device__ __forceinline__ void chunk_norm_keys(float (&v)[W], const float* nrm)
{
    const float4* n4 = reinterpret_cast<const float4*>(nrm);
#pragma unroll
    for (int u = 0; u < W / 4; ++u) {
        const float4 c = n4[u];
        ptx::fma2(v[4 * u], v[4 * u + 1], v[4 * u], v[4 * u + 1], -2.0f, c.x, c.y);
        ptx::fma2(v[4 * u + 2], v[4 * u + 3], v[4 * u + 2], v[4 * u + 3], -2.0f, c.z, c.w);
    }
}

// Release of a norm slot by an epilogue warp, once its loads have returned.  Right after the loads in program order
// the arrival could overtake them, queued behind the appends of earlier tiles, and the slot be filled anew: beside
// queries that append whole tiles rows were lost (9,000 x 5 rows, nine tenths of the values zero: 20 of 3,000 queries).
// So the arrival's address depends on the vote over all lanes' keys (zero: 0, which the compiler does not know).
__device__ __forceinline__ void release_norms(uint32_t bar, uint32_t vote, uint32_t zero)
{
    if ((threadIdx.x & 31) == 0) ptx::mbar_arrive(bar + (vote & zero));
}
// ... of a dense pass, after the shuffles of its stores have used the keys.
__device__ __forceinline__ void release_norms(uint32_t bar)
{
    __syncwarp();
    if ((threadIdx.x & 31) == 0) ptx::mbar_arrive(bar);
}

// Keys of the columns at or past `rem` (rows past the corpus view in its last tile) set to +inf.
template <int W>
__device__ __forceinline__ void chunk_mask(float (&key)[W], int c0, int rem)
{
#pragma unroll
    for (int j = 0; j < W; ++j)
        if (c0 + j >= rem) key[j] = __int_as_float(0x7f800000);
}

// Minima of a chunk's 8-column groups.
template <int W>
__device__ __forceinline__ void chunk_minima(const float (&key)[W], float (&gm)[W / 8])
{
#pragma unroll
    for (int g = 0; g < W / 8; ++g) gm[g] = min8(key + 8 * g);
}
template <int N>
__device__ __forceinline__ float min_of(const float (&v)[N])
{
    float m = v[0];
#pragma unroll
    for (int i = 1; i + 1 < N; i += 2) m = ptx::fmin3(m, v[i], v[i + 1]);
    return N % 2 == 0 ? fminf(m, v[N - 1]) : m;
}

// Append the keys below T, in increasing corpus index, given the groups' minima.  Words hold the raw
// key bits above the index; the selection maps them to ordered keys.  A group with a single key below
// T (the usual case) stores its minimum at the position found from the mask of hits; more hits take
// the column walk.
template <int W>
__device__ __forceinline__ void chunk_append(const float (&key)[W], const float (&gm)[W / 8], float T, uint32_t base,
                                             uint64_t* out, uint32_t cap, uint32_t& cnt)
{
#pragma unroll
    for (int g = 0; g < W / 8; ++g) {
        if (gm[g] < T) {
            const float* kg = key + 8 * g;
            uint32_t hm = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (kg[j] < T) hm |= 1u << j;
            if ((hm & (hm - 1u)) == 0u) {
                if (cnt < cap)
                    out[cnt] = ((uint64_t)__float_as_uint(gm[g]) << 32) | (uint64_t)(base + (uint32_t)(8 * g + __ffs((int)hm) - 1));
                ++cnt;
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float k = kg[j];
                    const bool h = k < T;
                    if (h && cnt < cap)
                        out[cnt] = ((uint64_t)__float_as_uint(k) << 32) | (uint64_t)(base + (uint32_t)(8 * g + j));
                    cnt += h ? 1u : 0u;
                }
            }
        }
    }
}

// The warp's 32 x W keys (lane = row) to 32 rows of the dense key matrix: `base` is row 0's first
// column (16-byte aligned), `rows` the rows that exist.  Groups of W / 4 lanes first transpose their
// blocks of 16-byte words, so that a store instruction writes whole 4 W-byte rows: written by lane, its
// 32 words fell into 32 lines, and the stores of a 128-column tile took about 4,000 cycles of an SM.
template <int W>
__device__ __forceinline__ void chunk_store(float (&key)[W], float* base, int64_t ldk, int rows)
{
    constexpr int n = W / 4;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = n / 2; s > 0; s >>= 1) {
        const bool up = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < n; ++i) {
            if (i & s) continue;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float& a = key[4 * i + e];
                float& b = key[4 * (i | s) + e];
                const float got = __shfl_xor_sync(0xffffffffu, up ? a : b, s);
                if (up) a = got;
                else b = got;
            }
        }
    }
    const int g = lane & ~(n - 1), l = lane & (n - 1);
#pragma unroll
    for (int j = 0; j < n; ++j)
        if (g + j < rows)
            *reinterpret_cast<float4*>(base + (g + j) * ldk + 4 * l) =
                make_float4(key[4 * j], key[4 * j + 1], key[4 * j + 2], key[4 * j + 3]);
}

}  // namespace
}  // namespace knn
