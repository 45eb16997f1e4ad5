// prep.cu -- corpus/query preparation: row norms, BF16 / E4M3 copies and the FP16 hi/lo split.
//
// Replaces the reference's norm kernels crpdot2_* / dot4_* (include/utils.h:72-357,
// 516-766), which reduce x_d^2 in float with a warp-synchronous tree.  Here a
// row norm is the float rounding of a double sum taken in d order (exact for
// the integer-valued data of the 1M x 128 workload and within one rounding of
// exact otherwise); the same convention is used by the CPU oracle.
#include <algorithm>
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>
#include "common.cuh"
#include "kernels.h"

namespace knn {

__global__ void norms_kernel(const float* __restrict__ x, int64_t n, int64_t ld, int D,
                             float* __restrict__ out, int64_t n_pad)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    if (i >= n) {  // padding rows never enter a shortlist
        out[i] = __int_as_float(0x7f800000);
        return;
    }
    const float* r = x + i * ld;
    double acc = 0.0;
    int d = 0;
    for (; d + 4 <= D; d += 4) {
        float a = __ldg(r + d), b = __ldg(r + d + 1), c = __ldg(r + d + 2), e = __ldg(r + d + 3);
        acc = __fma_rn((double)a, (double)a, acc);
        acc = __fma_rn((double)b, (double)b, acc);
        acc = __fma_rn((double)c, (double)c, acc);
        acc = __fma_rn((double)e, (double)e, acc);
    }
    for (; d < D; ++d) {
        float a = __ldg(r + d);
        acc = __fma_rn((double)a, (double)a, acc);
    }
    out[i] = __double2float_rn(acc);
}

// Round a float to the nearest TF32 value (10 explicit mantissa bits, ties to
// even), returned as a float whose low 13 bits are zero.
__device__ __forceinline__ float tf32_rne(float x)
{
    uint32_t u = __float_as_uint(x);
    if ((u & 0x7f800000u) == 0x7f800000u) return x;  // inf / nan unchanged
    u += 0xfffu + ((u >> 13) & 1u);
    u &= 0xffffe000u;
    return __uint_as_float(u);
}

// BF16 copy of a row-major matrix, rows padded with zeros to dpb columns, and
// a global "not exactly representable" flag: *not_exact becomes 1 when some
// element differs from its BF16 rounding (inf/nan count as not exact).  One
// block per 128-row tile.
__global__ void bf16_tiles_kernel(const float* __restrict__ x, int64_t n, int64_t ld, int D, int dpb,
                                  __nv_bfloat16* __restrict__ out, uint32_t* __restrict__ not_exact)
{
    const int64_t r0 = (int64_t)blockIdx.x * 128;
    const int64_t rows = min((int64_t)128, n - r0);
    const int64_t total = rows * dpb;
    int bad = 0;
    for (int64_t i = threadIdx.x; i < total; i += blockDim.x) {
        const int64_t r = r0 + i / dpb;
        const int c = (int)(i % dpb);
        const float v = c < D ? __ldg(x + r * ld + c) : 0.f;
        const __nv_bfloat16 b = __float2bfloat16_rn(v);
        if (out) out[r * dpb + c] = b;
        bad |= !(__bfloat162float(b) == v);
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0 && bad) atomicOr(not_exact, 1u);
}

// hi = tf32(x), lo = tf32(x - hi); rows padded with zeros to dp columns.
// One block per 128-row tile, one warp per row at a time (eight rows in flight per block), each
// lane a float4 of columns: coalesced 16-byte loads and stores.  lo_flags[tile] = 1 when any lo
// in the tile is nonzero (the tensor-core kernels skip the correction products otherwise).
__global__ void __launch_bounds__(256) split_tf32_kernel(const float* __restrict__ x, int64_t n, int64_t ld, int D,
                                                          int dp, float* __restrict__ hi, float* __restrict__ lo,
                                                          uint32_t* __restrict__ lo_flags,
                                                          uint32_t* __restrict__ any_lo,
                                                          const uint32_t* __restrict__ skip_unless)
{
    // BF16-exact inputs are searched by the BF16 kernels: nothing to prepare
    if (skip_unless && *skip_unless == 0u) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t r0 = (int64_t)blockIdx.x * 128;
    // 16-byte loads when every row starts 16-byte aligned and holds whole float4s
    const bool vec = (ld % 4 == 0) && (D % 4 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15u) == 0);
    int any = 0;
    for (int rr = warp; rr < 128; rr += 8) {
        const int64_t r = r0 + rr;
        if (r >= n) break;  // warp-uniform
        const float* row = x + r * ld;
        float4* H = reinterpret_cast<float4*>(hi + r * dp);
        float4* L = reinterpret_cast<float4*>(lo + r * dp);
        for (int c = 4 * lane; c < dp; c += 128) {
            float v[4];
            if (vec) {
                float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < D) t = __ldg(reinterpret_cast<const float4*>(row + c));
                v[0] = t.x;
                v[1] = t.y;
                v[2] = t.z;
                v[3] = t.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = c + i < D ? __ldg(row + c + i) : 0.f;
            }
            float h[4], l[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                h[i] = tf32_rne(v[i]);
                l[i] = tf32_rne(__fsub_rn(v[i], h[i]));
                any |= (l[i] != 0.f);
            }
            H[c >> 2] = make_float4(h[0], h[1], h[2], h[3]);
            L[c >> 2] = make_float4(l[0], l[1], l[2], l[3]);
        }
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) {
        if (lo_flags) lo_flags[blockIdx.x] = any ? 1u : 0u;
        if (any && any_lo) atomicOr(any_lo, 1u);
    }
}

__global__ void gather_norms_kernel(const float* __restrict__ src, int64_t n, int64_t stride, float* __restrict__ out,
                                    int64_t n_pad, const uint32_t* __restrict__ skip_unless,
                                    const float* __restrict__ scales, float* __restrict__ out_scales)
{
    if (skip_unless && *skip_unless == 0u) return;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    out[i] = i < n ? src[i * stride] : __int_as_float(0x7f800000);
    if (out_scales) out_scales[i] = i < n ? scales[i * stride] : 0.f;
}

// Preparation of a row-major matrix in one coalesced read, one warp per kU rows: lane l holds
// columns 128 j + 4 l .. 128 j + 4 l + 3 of every 128-column chunk j < kChunks (float4 loads when
// rows are 16-byte aligned).  Per row, as requested (PrepJob):
//  * BF16 side: copy into bf[n][dpb] (zero padded) and the "not exactly representable" flag
//    (*not_exact |= 1); integrality and magnitude: int_stats[0] |= 1 when some value is not an
//    integer, int_stats[1] = max |x| as float bits; the norm as BF16 parts;
//  * E4M3 copy into f8[n][f8_bytes] (zero padded) with per-row absmax scales
//    (scale = max|x| / 448, codes = satfinite(x * 448 / max|x|));
//  * FP16 side: the split hi / lo [n][hp] with row scales and tile flags (split_pair2);
//  * row norms into norms[0..n_pad) (+inf for n <= i < n_pad): the float rounding of the double
//    sum of x_d^2 taken in d order (the convention of norms_kernel and the CPU oracle), certified
//    from a float-float sum -- see certified_norm -- and, for the rows that leaves open, from a
//    double sum over the warp, then the serial double loop.
// Adaptive jobs (done != null) write one side per warp batch: the BF16 side until the corpus is
// known not to be BF16-exact (*not_exact, read again every few batches), the FP16 side from then
// on; done[batch] says which, and a second, catch-up launch over the same matrix (run_if =
// not_exact) writes the FP16 side of the batches that came before.  So BF16-exact data cost no FP16
// copy and other data little of the BF16 one, in one read of the matrix.
// Bound by memory on integer rows (1,000,000 x 128: 128 us for 800 MB; 149 before the next batch's
// loads were issued ahead), by issue slots and memory about equally on FP32 rows (1,000,003 x 96,
// adaptive: 146 us + 6 of catch-up for 770 MB, where a BF16 pass and a split pass took 335 + 186;
// 32,768 x 1,024: 48 us for 268 MB, 154 + 97 as one thread a row and a split).
struct PrepArgs : PrepJob {
    int hp;
};
// One launch's jobs: blocks [0, first) take j[0], the rest j[1].  Corpus and queries of a search share one
// (32,768 and 256 rows of 1,024 columns: 49.8 + 3.7 us and the gap between them -> 51.4).
struct PrepPair {
    PrepArgs j[2];
    unsigned first;
};

// s + t = a + b exactly (Knuth's TwoSum; no contraction: explicit roundings)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& t)
{
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    t = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Norm of a row from the lanes' float-float partial sums (hi, lo).  The TwoSums are exact, so
// S_ff = hi + lo differs from the exact sum S only by the roundings of the lo additions and by
// residuals of squares below the float range (< 2^-149 each).  Every term folded into lo is at
// most 2^-24 of a partial sum: with m elements a lane, its TwoSum residuals (m, the sum of its two
// chains included) total at most m 2^-24 of its share of S, its square residuals 2^-24 of it, and
// the 31 tree TwoSums 2^-24 S each, so the terms total E <= (m + 32) 2^-24 S.  A lane's lo roundings
// (at most 2m + 2) err by at most 2^-24 of its share of E each and the 5 tree levels by 2 2^-24 E, so
// |S_ff - S| <= (2m + 12) 2^-24 E + D 2^-149 < c S + D 2^-149 with c = 2^-36 for m <= 12 (3 chunks
// of 128 columns) and 2^-34 for m <= 64 (16 chunks).  The double d-order sum differs from S by at
// most D 2^-52 S.  When [S_ff - B, S_ff + B] (B the sum of both bounds, S bounded by 1.01 (hi +
// |lo|)) lies strictly inside the rounding interval of f = fl(S_ff) -- half the spacing below f on
// one side, half the spacing above on the other (they differ at powers of two) -- the double sum
// rounds to f as well; otherwise the caller recomputes the row in double.
template <int kChunks>
__device__ __forceinline__ bool certified_norm(float hi, float lo, int D, float& f)
{
    static_assert(kChunks <= 16, "the bound covers 64 elements a lane");
    f = __fadd_rn(hi, lo);
    if (!(f >= 0x1p-100f && f <= 0x1p126f)) return false;  // also rejects nan
    const float r = __fadd_rn(__fsub_rn(hi, f), lo);        // S_ff - f: hi - f exact (Sterbenz)
    const float S = 1.01f * (hi + fabsf(lo));
    const float B = ((kChunks <= 3 ? 0x1p-36f : 0x1p-34f) + (float)D * 0x1p-52f) * S + 0x1p-137f;
    const float rr = fabsf(r) * 0.0001f;                      // rounding of r itself
    // the neighbours of a positive normal f are its bits -1 and +1
    const float h_dn = 0.5f * (f - __uint_as_float(__float_as_uint(f) - 1u));
    const float h_up = 0.5f * (__uint_as_float(__float_as_uint(f) + 1u) - f);
    return r + rr + B < h_up && r - rr - B > -h_dn;
}

// (h, l) += (oh, ol) as float-float: exact TwoSum of the high parts, the low parts and
// the residual added.  Symmetric: both partners of a butterfly step get the same values
// (the TwoSum residual is the exact error whatever the operand order).
__device__ __forceinline__ void ff_add(float& h, float& l, float oh, float ol)
{
    float s, t;
    two_sum(h, oh, s, t);
    h = s;
    l = __fadd_rn(__fadd_rn(l, ol), t);
}

// Sums of kU rows' float-float partials over the warp, transposed: the first log2(kU)
// levels halve the rows a lane holds (it keeps the rows of its half of the warp and
// receives its partner's partials of them), the remaining levels are a butterfly within
// groups of 32 / kU lanes.  Each row is still summed by a complete pairwise tree of depth
// 5 over the 32 lanes' partials (31 exact TwoSums, low parts added along paths of 5
// levels), so certified_norm's bound holds as for a plain 32-lane butterfly, at a quarter
// of the shuffles for four rows.  Lane l ends with row l / (32 / kU), identical across
// its group.
template <int kU>
__device__ __forceinline__ void ff_reduce_rows(const float (&hi)[kU], const float (&lo)[kU], int lane, float& h,
                                               float& l)
{
    static_assert(kU == 1 || kU == 2 || kU == 4, "1, 2 or 4 rows per warp");
    constexpr unsigned kAll = 0xffffffffu;
    if constexpr (kU == 4) {
        const bool up = (lane & 16) != 0;  // keeps rows 2, 3 (else 0, 1)
        float h0 = up ? hi[2] : hi[0], l0 = up ? lo[2] : lo[0];
        float h1 = up ? hi[3] : hi[1], l1 = up ? lo[3] : lo[1];
        const float s0h = up ? hi[0] : hi[2], s0l = up ? lo[0] : lo[2];
        const float s1h = up ? hi[1] : hi[3], s1l = up ? lo[1] : lo[3];
        ff_add(h0, l0, __shfl_xor_sync(kAll, s0h, 16), __shfl_xor_sync(kAll, s0l, 16));
        ff_add(h1, l1, __shfl_xor_sync(kAll, s1h, 16), __shfl_xor_sync(kAll, s1l, 16));
        const bool up3 = (lane & 8) != 0;  // keeps the second of the two
        h = up3 ? h1 : h0;
        l = up3 ? l1 : l0;
        const float sh = up3 ? h0 : h1, sl = up3 ? l0 : l1;
        ff_add(h, l, __shfl_xor_sync(kAll, sh, 8), __shfl_xor_sync(kAll, sl, 8));
    } else if constexpr (kU == 2) {
        const bool up = (lane & 16) != 0;  // keeps row 1 (else 0)
        h = up ? hi[1] : hi[0];
        l = up ? lo[1] : lo[0];
        const float sh = up ? hi[0] : hi[1], sl = up ? lo[0] : lo[1];
        ff_add(h, l, __shfl_xor_sync(kAll, sh, 16), __shfl_xor_sync(kAll, sl, 16));
    } else {
        h = hi[0];
        l = lo[0];
    }
    constexpr int kFirst = kU == 4 ? 4 : kU == 2 ? 8 : 16;
#pragma unroll
    for (int o = kFirst; o > 0; o >>= 1) ff_add(h, l, __shfl_xor_sync(kAll, h, o), __shfl_xor_sync(kAll, l, o));
}

// v[g] for a lane-dependent g < kU without indexing a register array
template <int kU>
__device__ __forceinline__ float pick_row(const float (&v)[kU], int g)
{
    float x = v[0];
#pragma unroll
    for (int u = 1; u < kU; ++u) x = g == u ? v[u] : x;
    return x;
}

// The norm f as three BF16 parts, then zeros: one 32-byte row of the operand that adds ||c||^2
// inside the BF16 scan's MMA.  n1 + n2 + n3 == f exactly for f = 0 and f >= 2^-100 (each
// remainder is exact by Sterbenz's lemma, a multiple of f's FP32 ulp, and the last one holds at
// most 8 significant bits, all within BF16's normal range); smaller norms are kept to within
// 2^-133, BF16's subnormal spacing.  Norms that are not finite in BF16 (past 3.39e38) keep n1
// alone (+inf).
__device__ __forceinline__ void store_norm_parts(__nv_bfloat16* dst, float f)
{
    const __nv_bfloat16 n1 = __float2bfloat16_rn(f);
    __nv_bfloat16 n2 = __float2bfloat16_rn(0.f), n3 = n2;
    if (isfinite(__bfloat162float(n1))) {
        const float r1 = __fsub_rn(f, __bfloat162float(n1));
        n2 = __float2bfloat16_rn(r1);
        n3 = __float2bfloat16_rn(__fsub_rn(r1, __bfloat162float(n2)));
    }
    uint4 w0;
    w0.x = (uint32_t)__bfloat16_as_ushort(n1) | ((uint32_t)__bfloat16_as_ushort(n2) << 16);
    w0.y = (uint32_t)__bfloat16_as_ushort(n3);
    w0.z = 0u;
    w0.w = 0u;
    static_assert(kNormParts * 2 == 2 * sizeof(uint4), "one row of norm parts is two 16-byte words");
    uint4* d = reinterpret_cast<uint4*>(dst);
    d[0] = w0;
    d[1] = make_uint4(0u, 0u, 0u, 0u);
}

// Packed pairs of floats (sm_100+: one instruction for two IEEE operations).
using F2 = uint64_t;
__device__ __forceinline__ F2 pk(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void upk(F2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Float-float sum (hi, lo) of the squares of a lane's m = 4 kChunks elements: two chains, one per
// half of the packed pairs, then their sum.  The chains accumulate the negated squares n = -fl(x^2)
// (x - y is then x + y throughout; every operation is symmetric under negation): with e = x^2 +
// n exact by fma and s + t = h + n by TwoSum, h = s, l += t - e.
template <int kChunks>
__device__ __forceinline__ void ff_squares(const float (&v)[kChunks][4], float& hi, float& lo)
{
    const F2 m1 = pk(-1.f, -1.f);
    F2 h = 0, l = 0;
#pragma unroll
    for (int j = 0; j < kChunks; ++j)
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            const F2 x = pk(v[j][i], v[j][i + 1]);
            const F2 n = mul2(x, mul2(x, m1));
            const F2 e = fma2(x, x, n);
            if (j == 0 && i == 0) {
                h = n;
                l = mul2(e, m1);
                continue;
            }
            // TwoSum: s = h + n, b = s - h, t = (h - (s - b)) + (n - b)
            const F2 s = add2(h, n);
            const F2 b = fma2(h, m1, s);
            const F2 t = add2(fma2(fma2(b, m1, s), m1, h), fma2(b, m1, n));
            h = s;
            l = add2(l, fma2(e, m1, t));
        }
    float h0, h1, l0, l1, t;
    upk(h, h0, h1);
    upk(l, l0, l1);
    two_sum(-h0, -h1, hi, t);
    lo = __fadd_rn(__fadd_rn(-l0, -l1), t);
}

__device__ __forceinline__ float fmax3(float a, float b, float c)
{
    float m;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}

// s x0, s x1 as hi + lo FP16 pairs, in packed arithmetic.  A value that is not finite leaves NaN in lo (inf - inf), so
// its keys are NaN and enter no segment.
__device__ __forceinline__ void split_pair2(float x0, float x1, F2 sc, uint32_t& hi, uint32_t& lo)
{
    float y0, y1, z0, z1;
    const F2 y = mul2(pk(x0, x1), sc);
    upk(y, y0, y1);
    const __half2 h = __floats2half2_rn(y0, y1);
    upk(fma2(pk(__low2float(h), __high2float(h)), pk(-1.f, -1.f), y), z0, z1);
    const __half2 l = __floats2half2_rn(z0, z1);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Squares of a lane's m = 4 kChunks elements summed in two parts, by extraction against a power of
// two sigma > (D + 1) max|x|^2 > S, the row's sum: with q_0 = sigma and q_i = fl(q_{i-1} + x_i^2),
// q stays in [sigma, 2 sigma], so d_i = q_i - q_{i-1} is exact and a multiple of 2^-23 sigma, and
// hi = sum of d_i is exact in whatever order it is formed (it stays below sigma).  What d_i
// leaves of the square, r_i = fl(x_i^2 - d_i), is at most 2^-24 sigma and off by at most 2^-48
// sigma (and 2^-149, squares below the float range); lo = sum of the r_i: a lane's two chains and
// their sum round at most m times by 2^-24 of at most m 2^-24 sigma, the tree's five levels together
// by 5 x 2^-24 of 32 m 2^-24 sigma.  So hi + lo is within 32 m (m + 6) 2^-48 sigma + D 2^-149 of S;
// the double d-order sum within D 2^-52 of it.  Returns the sum of those bounds (infinite for rows
// out of range, which rounds_to then leaves to the double sum).  4 packed instructions a pair, where
// a float-float sum takes 11.
template <int kChunks>
__device__ __forceinline__ float ex_squares(const float (&v)[kChunks][4], float mx, int D, float& hi, float& lo)
{
    static_assert(kChunks <= 2, "m <= 8");
    const float t = (float)(D + 1) * mx * mx;
    const bool in = mx >= 0x1p-50f && t < 0x1p124f;
    const float sigma = in ? __uint_as_float((__float_as_uint(t) & 0x7f800000u) + 0x00800000u) : 1.f;
    const F2 m1 = pk(-1.f, -1.f);
    F2 q = pk(sigma, sigma), l = 0;
#pragma unroll
    for (int j = 0; j < kChunks; ++j)
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
            const F2 x = pk(v[j][i], v[j][i + 1]);
            const F2 s = fma2(x, x, q);
            const F2 nd = fma2(s, m1, q);  // -d
            const F2 r = fma2(x, x, nd);
            l = j == 0 && i == 0 ? r : add2(l, r);
            q = s;
        }
    float q0, q1, l0, l1;
    upk(q, q0, q1);
    upk(l, l0, l1);
    hi = __fadd_rn(__fsub_rn(q0, sigma), __fsub_rn(q1, sigma));
    lo = __fadd_rn(l0, l1);
    constexpr float m = 4.f * kChunks;
    return in ? (32.f * m * (m + 6.f) * 0x1p-48f + (float)D * 0x1p-52f) * sigma + 0x1p-140f : __int_as_float(0x7f800000);
}

// f = fl(hi + lo); true when every value within `bound` of hi + lo rounds to f.
template <int kU>
__device__ __forceinline__ bool rounds_to(float hi, float lo, float bound, float& f)
{
    f = __fadd_rn(hi, lo);
    const float r = __fadd_rn(__fsub_rn(hi, f), lo);  // hi + lo - f; hi - f is exact (lo is small)
    const float e = bound + fabsf(r) * 0.0001f;        // and the rounding of r itself
    // the neighbours of a positive normal f are its bits -1 and +1
    const float h_dn = 0.5f * (f - __uint_as_float(__float_as_uint(f) - 1u));
    const float h_up = 0.5f * (__uint_as_float(__float_as_uint(f) + 1u) - f);
    return f >= 0x1p-100f && r + e < h_up && r - e > -h_dn;
}

// Sums of kU rows' float partials over the warp, transposed as in ff_reduce_rows.
template <int kU>
__device__ __forceinline__ float reduce_rows(const float (&x)[kU], int lane)
{
    constexpr unsigned kAll = 0xffffffffu;
    float h;
    if constexpr (kU == 4) {
        const bool up = (lane & 16) != 0;
        float h0 = up ? x[2] : x[0], h1 = up ? x[3] : x[1];
        h0 = __fadd_rn(h0, __shfl_xor_sync(kAll, up ? x[0] : x[2], 16));
        h1 = __fadd_rn(h1, __shfl_xor_sync(kAll, up ? x[1] : x[3], 16));
        const bool up3 = (lane & 8) != 0;
        h = __fadd_rn(up3 ? h1 : h0, __shfl_xor_sync(kAll, up3 ? h0 : h1, 8));
    } else if constexpr (kU == 2) {
        const bool up = (lane & 16) != 0;
        h = __fadd_rn(up ? x[1] : x[0], __shfl_xor_sync(kAll, up ? x[0] : x[1], 16));
    } else {
        h = x[0];
    }
    constexpr int kFirst = kU == 4 ? 4 : kU == 2 ? 8 : 16;
#pragma unroll
    for (int o = kFirst; o > 0; o >>= 1) h = __fadd_rn(h, __shfl_xor_sync(kAll, h, o));
    return h;
}

// The row's norm from a double sum over the warp, or the serial d-order sum where that leaves the
// float rounding open; the same value in every lane.  Reads the row again: passing the lane's
// elements would give them a home in local memory on the way that nearly every row takes.
static __device__ __noinline__ float double_norm(const float* row, int D)
{
    const int lane = threadIdx.x & 31;
    double t = 0.0;
    bool grid = true;  // multiples of 2^-10
    for (int d = lane; d < D; d += 32) {
        const float v = __ldg(row + d);
        const double x = (double)v;
        t = __fma_rn(x, x, t);
        grid &= rintf(v * 1024.f) == v * 1024.f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (!(t < __longlong_as_double(0x7ff0000000000000ll))) return (float)t;  // inf or nan in any order
    // multiples of 2^-20 that sum below 2^33: exact in any order (integers, whose norms lie halfway between two
    // floats every other time from 2^24 on, else all took the serial loop: 42,649 x 1,400 values 0..199, a host
    // search 2.3 -> 5.5 ms)
    if (__all_sync(0xffffffffu, grid) && t < 0x1p33) return __double2float_rn(t);
    // both sums err by their additions' roundings: (D + D / 32 + 6) 2^-53 of the sum in all
    const double B = (double)(2 * D + 8) * 1.01 * 0x1p-53 * t;
    const float a = __double2float_rn(t - B), b = __double2float_rn(t + B);
    if (a == b) return a;
    float f = 0.f;
    if (lane == 0) {
        double acc = 0.0;
        for (int d = 0; d < D; ++d) {
            const double x = (double)__ldg(row + d);
            acc = __fma_rn(x, x, acc);
        }
        f = __double2float_rn(acc);
    }
    return __shfl_sync(0xffffffffu, f, 0);
}

template <int kChunks, int kU, bool kVec>
__global__ void __launch_bounds__(256, kChunks <= 8 ? 3 : 2)
    prep_rows_kernel(const __grid_constant__ PrepPair pp)
{
    const bool second = blockIdx.x >= pp.first;
    const PrepArgs& p = pp.j[second ? 1 : 0];
    if (p.run_if != nullptr && *p.run_if == 0u) return;
    const unsigned block = blockIdx.x - (second ? pp.first : 0u), blocks = second ? gridDim.x - pp.first : pp.first;
    const int lane = threadIdx.x & 31;
    const int gw = (int)((block * blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)((blocks * blockDim.x) >> 5);
    const int n = (int)p.n;                   // the engine's corpora have fewer than 2^31 rows
    const int nb = (int)((p.n + kU - 1) / kU);  // batches of kU rows; warp w takes w, w + nw, ...
    const int D = p.D;
    const bool want_norms = p.norms != nullptr || p.np != nullptr;
    const bool check = p.bf != nullptr || p.not_exact != nullptr;
    uint32_t frac = 0, bad = 0;
    float mx_all = 0.f;
    bool inexact = false;  // adaptive: *not_exact seen set
    int it = 0;
    // this warp's batches in turn, 32 looked ahead at once (catch-up: those without their FP16 side)
    int64_t b0 = gw - (int64_t)32 * nw;
    uint32_t todo = 0;
    auto next = [&]() -> int {
        while (todo == 0u) {
            b0 += (int64_t)32 * nw;
            if (b0 >= nb) return -1;
            const int64_t lb = b0 + (int64_t)lane * nw;
            todo = __ballot_sync(0xffffffffu, lb < nb && !(p.catch_up && p.done[lb]));
        }
        const int batch = (int)b0 + (__ffs((int)todo) - 1) * nw;
        todo &= todo - 1u;
        return batch;
    };
    auto load = [&](int batch, float (&v)[kU][kChunks][4]) {
        const int m = min(kU, n - batch * kU);
        const float* src = p.x + (int64_t)batch * kU * p.ld + 4 * lane;
#pragma unroll
        for (int u = 0; u < kU; ++u) {
#pragma unroll
            for (int j = 0; j < kChunks; ++j) {
                const int c = 128 * j + 4 * lane;
                if constexpr (kVec) {
                    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (u < m && c < D) t = __ldg(reinterpret_cast<const float4*>(src + 128 * j));
                    v[u][j][0] = t.x;
                    v[u][j][1] = t.y;
                    v[u][j][2] = t.z;
                    v[u][j][3] = t.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) v[u][j][i] = (u < m && c + i < D) ? __ldg(src + 128 * j + i) : 0.f;
                }
            }
            src += p.ld;
        }
    };
    auto body = [&](int batch, const float (&v)[kU][kChunks][4]) {
        const int base = batch * kU;
        const int m = min(kU, n - base);  // rows of this batch
        bool bf = true, hf = p.hi != nullptr;
        if (p.catch_up) {
            bf = false;
        } else if (p.done != nullptr) {
            // one flag word for every warp of the grid: read it seldom
            if (!inexact && (it < 2 || (it & 3) == 3))
                inexact = __any_sync(0xffffffffu, *(volatile const uint32_t*)p.not_exact != 0u);
            bf = !inexact;
            hf = inexact;
            if (lane == 0) p.done[batch] = inexact ? 1 : 0;
        }
        // per row: max |x| (in every lane); rows past n hold zeros and change nothing
        float rmx[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            float mx = 0.f;
#pragma unroll
            for (int j = 0; j < kChunks; ++j) {
                mx = fmax3(mx, fabsf(v[u][j][0]), fabsf(v[u][j][1]));
                mx = fmax3(mx, fabsf(v[u][j][2]), fabsf(v[u][j][3]));
            }
            rmx[u] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
            mx_all = fmaxf(mx_all, rmx[u]);
        }
        bool all_int = false, exact = false;
        if (bf) {
            // integrality, by (x + 1.5 2^23) - 1.5 2^23 == x (integers of 2^22 and more count as
            // fractions: no use of the flag goes that far), and exactness in BF16: the low 16
            // bits are zero (and the value is no NaN, which the first test tells)
            const F2 big = pk(12582912.f, 12582912.f), nbig = pk(-12582912.f, -12582912.f);
            uint32_t rfrac = 0, rlow = 0;
            float mx = 0.f;
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                mx = fmaxf(mx, rmx[u]);
#pragma unroll
                for (int j = 0; j < kChunks; ++j)
#pragma unroll
                    for (int i = 0; i < 4; i += 2) {
                        float y0, y1;
                        upk(add2(add2(pk(v[u][j][i], v[u][j][i + 1]), big), nbig), y0, y1);
                        rfrac |= !(y0 == v[u][j][i]) | !(y1 == v[u][j][i + 1]);
                        rlow |= __float_as_uint(v[u][j][i]) | __float_as_uint(v[u][j][i + 1]);
                    }
            }
            rlow &= 0xffffu;
            if (rfrac && !rlow) {
                // fractions may hide a NaN whose low bits are zero
#pragma unroll
                for (int u = 0; u < kU; ++u)
#pragma unroll
                    for (int j = 0; j < kChunks; ++j)
#pragma unroll
                        for (int i = 0; i < 4; ++i) rlow |= !(v[u][j][i] == v[u][j][i]);
            }
            // bits: some fraction, some inexact value
            const uint32_t f2 = (rfrac ? 1u : 0u) | (rlow ? 2u : 0u);
            const uint32_t w2 = __reduce_or_sync(0xffffffffu, f2);
            frac |= w2 & 1u;
            all_int = (w2 & 1u) == 0u && (float)D * mx * mx < 16777216.f;
            exact = (w2 & 1u) == 0u && mx <= 4096.f;
            if (check && (w2 & 2u)) {
                if (p.done != nullptr) {
                    // the other warps' next batches should know
                    if (lane == 0) atomicOr(p.not_exact, 1u);
                    inexact = true;
                } else {
                    bad = 1u;
                }
            }
            if (p.bf != nullptr) {
                __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(p.bf) + (int64_t)base * p.dpb + 4 * lane;
#pragma unroll
                for (int u = 0; u < kU; ++u) {
#pragma unroll
                    for (int j = 0; j < kChunks; ++j) {
                        const __nv_bfloat162 w0 = __floats2bfloat162_rn(v[u][j][0], v[u][j][1]);
                        const __nv_bfloat162 w1 = __floats2bfloat162_rn(v[u][j][2], v[u][j][3]);
                        uint2 w;
                        w.x = *reinterpret_cast<const uint32_t*>(&w0);
                        w.y = *reinterpret_cast<const uint32_t*>(&w1);
                        if (u < m && 128 * j + 4 * lane < p.dpb) *reinterpret_cast<uint2*>(dst + 128 * j) = w;
                    }
                    dst += p.dpb;
                }
            }
        }
        if (p.f8 != nullptr) {
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                if (u >= m) break;  // warp-uniform
                const float mx = rmx[u];
                const float inv = mx > 0.f ? 448.f / mx : 0.f;
                uint32_t* dst = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(p.f8) + (int64_t)(base + u) * p.f8_bytes);
#pragma unroll
                for (int j = 0; j < kChunks; ++j) {
                    const int c = 128 * j + 4 * lane;
                    if (c < p.f8_bytes) {
                        const uint32_t a = __nv_cvt_float2_to_fp8x2(make_float2(v[u][j][0] * inv, v[u][j][1] * inv),
                                                                    __NV_SATFINITE, __NV_E4M3);
                        const uint32_t b = __nv_cvt_float2_to_fp8x2(make_float2(v[u][j][2] * inv, v[u][j][3] * inv),
                                                                    __NV_SATFINITE, __NV_E4M3);
                        dst[c >> 2] = a | (b << 16);
                    }
                }
                if (lane == 0) p.scales[base + u] = mx / 448.f;
            }
        }
        // lane l settles row g = l / (32 / kU) of the batch where the rows are settled together
        constexpr int kGroup = 32 / kU;
        const int g = lane / kGroup;
        const bool lead = lane % kGroup == 0 && g < m;
        if (hf) {
            const int64_t at = (int64_t)base * p.hp + 4 * lane;
            __half* H = static_cast<__half*>(p.hi) + at;
            __half* L = static_cast<__half*>(p.lo) + at;
            uint32_t any = 0;
            float inv[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const float sc = row_scale(rmx[u], inv[u]);
                const F2 sc2 = pk(sc, sc);
#pragma unroll
                for (int j = 0; j < kChunks; ++j) {
                    uint2 h, l;
                    split_pair2(v[u][j][0], v[u][j][1], sc2, h.x, l.x);
                    split_pair2(v[u][j][2], v[u][j][3], sc2, h.y, l.y);
                    any |= l.x | l.y;
                    if (u < m && 128 * j + 4 * lane < p.hp) {
                        *reinterpret_cast<uint2*>(H + 128 * j) = h;
                        *reinterpret_cast<uint2*>(L + 128 * j) = l;
                    }
                }
                H += p.hp;
                L += p.hp;
            }
            if (lead) p.rs[base + g] = pick_row(inv, g);
            // a batch lies in one tile: kU divides its rows
            if (__any_sync(0xffffffffu, (any & 0x7fff7fffu) != 0u) && lane == 0 && p.lo_flags)
                p.lo_flags[base / kTileRows] = 1u;
        }
        if (want_norms && !p.catch_up) {
            float f;
            if (all_int) {
                // integers whose squares sum below 2^24: every partial sum is an exact integer,
                // so any order gives the double sum's value
                float fr[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    fr[u] = 0.f;
#pragma unroll
                    for (int j = 0; j < kChunks; ++j)
#pragma unroll
                        for (int i = 0; i < 4; ++i) fr[u] = __fmaf_rn(v[u][j][i], v[u][j][i], fr[u]);
                }
                f = reduce_rows<kU>(fr, lane);
            } else {
                float hi[kU], lo[kU];
                bool ok;
                if constexpr (kChunks <= 2) {
                    float bound[kU];
#pragma unroll
                    for (int u = 0; u < kU; ++u) bound[u] = ex_squares<kChunks>(v[u], rmx[u], D, hi[u], lo[u]);
                    ok = rounds_to<kU>(reduce_rows<kU>(hi, lane), reduce_rows<kU>(lo, lane), pick_row(bound, g), f);
                } else {
#pragma unroll
                    for (int u = 0; u < kU; ++u) ff_squares<kChunks>(v[u], hi[u], lo[u]);
                    float h, l;
                    ff_reduce_rows<kU>(hi, lo, lane, h, l);
                    ok = certified_norm<kChunks>(h, l, D, f);
                }
                // integers up to 2^12: squares, high parts and low parts (below 2^24) are exact integers, so f is
                // the sum's rounding even where that is a tie
                ok |= exact;
                const uint32_t open = __ballot_sync(0xffffffffu, !ok);
                if (open != 0u) {
#pragma unroll
                    for (int u = 0; u < kU; ++u) {
                        if ((open >> (u * kGroup)) & 1u) {
                            const float fd = double_norm(p.x + (int64_t)(u < m ? base + u : 0) * p.ld, u < m ? D : 0);
                            if (g == u) f = fd;
                        }
                    }
                }
            }
            if (lead) {
                if (p.norms) p.norms[base + g] = f;
                if (bf && p.np) store_norm_parts(static_cast<__nv_bfloat16*>(p.np) + (int64_t)(base + g) * kNormParts, f);
            }
        }
        ++it;
    };
    if constexpr (kChunks <= 4) {
        // the next batch's loads are in flight while this one is processed
        float va[kU][kChunks][4], vb[kU][kChunks][4];
        int ba = next();
        if (ba >= 0) load(ba, va);
        while (ba >= 0) {
            const int bb = next();
            if (bb >= 0) load(bb, vb);
            body(ba, va);
            if (bb < 0) break;
            ba = next();
            if (ba >= 0) load(ba, va);
            body(bb, vb);
        }
    } else {
        for (int b = next(); b >= 0; b = next()) {
            float v[kU][kChunks][4];
            load(b, v);
            body(b, v);
        }
    }
    // padding rows past n
    for (int64_t i = p.n + (int64_t)block * blockDim.x + threadIdx.x; i < p.n_pad;
         i += (int64_t)blocks * blockDim.x) {
        if (p.norms && !p.catch_up) p.norms[i] = __int_as_float(0x7f800000);
        if (p.scales) p.scales[i] = 0.f;
        if (p.rs) p.rs[i] = 0.f;
    }
    // flags: one atomic per warp
    if (p.not_exact != nullptr && bad != 0u && lane == 0) atomicOr(p.not_exact, 1u);
    if (p.int_stats != nullptr && !p.catch_up) {
        if (frac != 0u && lane == 0) atomicOr(p.int_stats, 1u);
        if (lane == 0 && mx_all > 0.f) atomicMax(p.int_stats + 1, __float_as_uint(mx_all));
    }
}

int64_t prep_batches(int64_t n, int D) { return (n + (D <= 128 ? 3 : D <= 256 ? 1 : 0)) / (D <= 128 ? 4 : D <= 256 ? 2 : 1); }

// The job's kernel arguments; false when it is not one the kernel takes.
static bool prep_args(const PrepJob& job, PrepArgs* a)
{
    static_cast<PrepJob&>(*a) = job;
    const int D = job.D;
    a->n_pad = std::max(job.n, job.n_pad);
    // the kernel covers ceil(D / 128) chunks of 128 columns (or bytes)
    const int span = (D + 127) / 128 * 128;
    if (D < 1 || D > kPrepMaxD || job.n > 0x7fffffffLL || (job.f8 != nullptr && (job.scales == nullptr || job.f8_bytes % 128 != 0 ||
                                                         job.f8_bytes < D || job.f8_bytes > span)) ||
        (job.bf != nullptr && (job.dpb % 64 != 0 || job.dpb < D || job.dpb > span)) ||
        (job.hi != nullptr && (!job.lo || !job.rs)) || (job.done != nullptr && (!job.hi || !job.not_exact)) ||
        (job.catch_up && !job.done))
        return false;
    a->hp = split_pitch(D);
    return true;
}

// rows to cover: the padding too where it is written
static int64_t prep_rows(const PrepJob& job)
{
    return std::max(job.n, (job.norms || job.scales || job.rs) ? job.n_pad : job.n);
}

// 16-byte loads where every row starts 16-byte aligned and holds whole float4s
static bool prep_vec(const PrepJob& job)
{
    return job.ld % 4 == 0 && job.D % 4 == 0 && (reinterpret_cast<uintptr_t>(job.x) & 15u) == 0;
}

cudaError_t launch_prep(const PrepJob& job, cudaStream_t s, const PrepJob* second)
{
    // two jobs share a launch when they take the same kernel
    if (second != nullptr &&
        (second->D != job.D || prep_vec(*second) != prep_vec(job) || prep_rows(job) <= 0 || prep_rows(*second) <= 0)) {
        const cudaError_t e = launch_prep(job, s);
        return e != cudaSuccess ? e : launch_prep(*second, s);
    }
    const int64_t rows = prep_rows(job);
    if (rows <= 0) return cudaSuccess;
    PrepPair a;
    if (!prep_args(job, &a.j[0]) || !prep_args(second ? *second : job, &a.j[1])) return cudaErrorInvalidValue;
    const int D = job.D;
    // one wave of blocks (three an SM, two for the widest rows), each warp walking its share of the rows;
    // of two jobs each gets blocks by its rows
    const int64_t kBlocks = kSms * (D <= 1024 ? 3 : 2);
    const int64_t nb = prep_batches(rows, D), nb2 = second ? prep_batches(prep_rows(*second), D) : 0;
    const int64_t want = (nb + 7) / 8, want2 = (nb2 + 7) / 8;
    int64_t b1 = std::min(want, kBlocks), b2 = want2;
    if (b1 + b2 > kBlocks) {
        b2 = std::max<int64_t>(want2 ? 1 : 0, std::min(want2, (kBlocks * nb2 + (nb + nb2) / 2) / (nb + nb2)));
        b1 = std::max<int64_t>(1, std::min(want, kBlocks - b2));
    }
    a.first = (unsigned)b1;
    const unsigned blocks = (unsigned)(b1 + b2);
    auto go = [&](auto* wide, auto* scalar) { (prep_vec(job) ? wide : scalar)<<<blocks, 256, 0, s>>>(a); };
    if (D <= 128)
        go(prep_rows_kernel<1, 4, true>, prep_rows_kernel<1, 4, false>);
    else if (D <= 256)
        go(prep_rows_kernel<2, 2, true>, prep_rows_kernel<2, 2, false>);
    else if (D <= 384)
        go(prep_rows_kernel<3, 1, true>, prep_rows_kernel<3, 1, false>);
    else if (D <= 512)
        go(prep_rows_kernel<4, 1, true>, prep_rows_kernel<4, 1, false>);
    else if (D <= 1024)
        go(prep_rows_kernel<8, 1, true>, prep_rows_kernel<8, 1, false>);
    else
        go(prep_rows_kernel<16, 1, true>, prep_rows_kernel<16, 1, false>);
    return cudaGetLastError();
}

cudaError_t launch_row_norms(const float* x, int64_t n, int64_t ld, int D, float* norms, int64_t n_pad, cudaStream_t s)
{
    if (D > kPrepMaxD) return launch_norms(x, n, ld, D, norms, n_pad, s);
    PrepJob j;
    j.x = x;
    j.n = n;
    j.ld = ld;
    j.D = D;
    j.norms = norms;
    j.n_pad = n_pad;
    return launch_prep(j, s);
}

cudaError_t launch_gather_norms(const float* src, int64_t n, int64_t stride, float* out, int64_t n_pad,
                                cudaStream_t s, const uint32_t* skip_unless, const float* scales, float* out_scales)
{
    if (n_pad <= 0) return cudaSuccess;
    if ((scales == nullptr) != (out_scales == nullptr)) return cudaErrorInvalidValue;
    gather_norms_kernel<<<(unsigned)((n_pad + 255) / 256), 256, 0, s>>>(src, n, stride, out, n_pad, skip_unless,
                                                                         scales, out_scales);
    return cudaGetLastError();
}

cudaError_t launch_norms(const float* x, int64_t n, int64_t ld, int D, float* out, int64_t n_pad,
                         cudaStream_t s)
{
    if (n_pad <= 0) return cudaSuccess;
    int threads = 256;
    int64_t blocks = (n_pad + threads - 1) / threads;
    norms_kernel<<<(unsigned)blocks, threads, 0, s>>>(x, n, ld, D, out, n_pad);
    return cudaGetLastError();
}

cudaError_t launch_split_tf32(const float* x, int64_t n, int64_t ld, int D, int dp, float* hi, float* lo,
                         uint32_t* lo_flags, uint32_t* any_lo, const uint32_t* skip_unless, cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    if (dp % 4 != 0 || dp < D) return cudaErrorInvalidValue;  // rows of whole float4s
    const int64_t tiles = (n + 127) / 128;
    split_tf32_kernel<<<(unsigned)tiles, 256, 0, s>>>(x, n, ld, D, dp, hi, lo, lo_flags, any_lo, skip_unless);
    return cudaGetLastError();
}

cudaError_t launch_bf16(const float* x, int64_t n, int64_t ld, int D, int dpb, void* out, uint32_t* not_exact,
                        cudaStream_t s)
{
    if (n <= 0) return cudaSuccess;
    const int64_t tiles = (n + 127) / 128;
    bf16_tiles_kernel<<<(unsigned)tiles, 256, 0, s>>>(x, n, ld, D, dpb, static_cast<__nv_bfloat16*>(out), not_exact);
    return cudaGetLastError();
}

}  // namespace knn
