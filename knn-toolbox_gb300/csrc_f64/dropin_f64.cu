// dropin_f64.cu -- the double-precision library (libknngb300_double.so), the
// counterpart of the reference's libcuknn_double.a (Makefile:60-64: the same
// sources built with -D__DOUBLE__, knntype = double).  It exports the same C
// names with double arguments (include/cuknns.h with __DOUBLE__ defined) plus a
// status-returning device API (include/knn_gb300_f64.h).
//
// GB300's FP64 rate is a small fraction of its FP32 / tensor rate, so the
// double path does not scan the corpus in FP64.  Instead:
//   1. corpus and queries are rounded to FP32 and the float engine returns,
//      per query, the kp nearest rows by FP32 distance (kp > k);
//   2. those kp candidates are re-ranked by FP64 direct-difference distance
//      (sum over d, in d order, of (q_d - c_d)^2 with separate multiply and add)
//      and the first k kept;
//   3. a query is accepted only if no row outside its shortlist can belong to
//      its FP64 top-k: every outside row has an FP32 distance >= the shortlist's
//      largest, D32, and an FP64 distance >= D32 - E, where E bounds the error
//      of an FP32 distance of rounded data, E = (D/8 + 10) * 2^-24 *
//      (|q| + max|c|)^2 + 1e-5 * D32 (the last term covers the float engine's
//      own ranking tolerance) + 1e-44 D (subnormals), unbounded where norms can leave the float range;
//      accepted when the k-th FP64 distance < D32 - E, or when the shortlist holds every row;
//   4. any other query is searched again by an FP64 brute-force kernel.
// Results: the exact FP64 top-k ordered by (distance, index).
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>

#include <cuda_runtime.h>

#include "cuknns.h"
#include "knn_gb300.h"
#include "knn_gb300_f64.h"

namespace knn64 {

namespace {
thread_local std::string g_err;

int fail(int code, const char* fmt, ...)
{
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}

#define F64_CUDA(call)                                                                                            \
    do {                                                                                                          \
        cudaError_t e_ = (call);                                                                                  \
        if (e_ != cudaSuccess) return fail(KNNS_ERR_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_));       \
    } while (0)

struct Buf {
    void* p = nullptr;
    size_t cap = 0;
    int ensure(size_t bytes)
    {
        if (bytes <= cap) return KNNS_OK;
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        if (cudaMalloc(&p, bytes) != cudaSuccess) {
            (void)cudaGetLastError();
            return fail(KNNS_ERR_NOMEM, "cudaMalloc(%zu) failed", bytes);
        }
        cap = bytes;
        return KNNS_OK;
    }
};

struct Work {
    std::mutex mu;
    Buf c32, q32, cand_d, cand_i, dd, bound, ncand, cmax, fails, hc, hq, hd, hi;
};

std::mutex g_mu;
std::map<int, std::unique_ptr<Work>> g_work;

Work* work_for_device()
{
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_mu);
    auto& w = g_work[dev];
    if (!w) w.reset(new Work());
    return w.get();
}

constexpr int kSortMax = 512;    // shortlist entries one warp re-ranks
constexpr int64_t kMostBlocks = 152 * 8;  // eight an SM
constexpr int kBruteBuf = 2048;  // candidate buffer of the brute-force kernel

// x rounded to FP32 (to nearest, ties to even) in integer arithmetic, for zeros and magnitudes of FP32's
// normal range (ok): the conversion instruction runs on the FP64 pipe, which it kept the kernel below
// waiting on (32,768 x 128 values: 34 us, 13 without it, of which the bytes take 7).
__device__ __forceinline__ float to_f32(double x, bool& ok)
{
    const uint64_t u = (uint64_t)__double_as_longlong(x);
    const uint32_t hi = (uint32_t)(u >> 32), sign = hi & 0x80000000u;
    const bool zero = (u << 1) == 0ull;
    ok = zero || ((hi >> 20) & 0x7ffu) - 897u < 254u;
    // drop 29 fraction bits: half an ulp less one, plus one for an odd last bit; a carry moves into the
    // exponent (past the largest float: to infinity)
    const uint64_t r = (u & 0x7fffffffffffffffull) + 0x0fffffffull + ((u >> 29) & 1ull);
    return __uint_as_float(sign | (zero ? 0u : (uint32_t)(r >> 29) - (896u << 23)));
}

// FP32 copy of the rows (out[rows][D]) and, when mx is given, an upper bound on the largest row norm
// (as ordered bits in *mx): one warp a row, coalesced, kV values a lane in flight (4 for up to 128
// columns, 8 above).  The bound comes from an FP32 sum of squares (off by less than 2e-5 of itself for any
// D the engine takes), or from sqrt(D) max|x| where the squares come near the end of the float range.
template <int kV>
__global__ void __launch_bounds__(256) to_f32_kernel(const double* __restrict__ x, int64_t rows, int64_t ld, int D,
                                                     float* __restrict__ out, unsigned long long* __restrict__ mx)
{
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    float best = 0.f;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
        const double* row = x + r * ld;
        float* dst = out + r * D;
        float ss = 0.f, big = 0.f;
        bool lost = false;  // a value that is no float: not even its bound is known
        for (int c0 = 0; c0 < D; c0 += 32 * kV) {
            double v[kV];
#pragma unroll
            for (int i = 0; i < kV; ++i) v[i] = c0 + 32 * i + lane < D ? __ldg(row + c0 + 32 * i + lane) : 0.0;
            float f[kV];
            bool all = true;
#pragma unroll
            for (int i = 0; i < kV; ++i) {
                bool ok;
                f[i] = to_f32(v[i], ok);
                all &= ok;
            }
            // (a vote, so that the compiler leaves the instruction behind a branch)
            if (!__all_sync(0xffffffffu, all))
#pragma unroll
                for (int i = 0; i < kV; ++i) {
                    f[i] = (float)v[i];
                    lost |= f[i] != f[i] || (f[i] == 0.f && (__double_as_longlong(v[i]) << 1) != 0);
                }
#pragma unroll
            for (int i = 0; i < kV; ++i) {
                const int c = c0 + 32 * i + lane;
                if (c < D) dst[c] = f[i];
                ss = __fmaf_rn(f[i], f[i], ss);
                big = fmaxf(big, fabsf(f[i]));
            }
        }
        if (mx == nullptr) continue;
        lost |= !(big < __int_as_float(0x7f800000));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            ss += __shfl_xor_sync(0xffffffffu, ss, o);
            big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
        }
        // in float, rounded up (1e-6 covers the roundings; integer and float work only: a double
        // comparison a value made this kernel four times slower)
        float b = ss >= 1e-30f && ss < 1e38f ? sqrtf(ss) * (1.f + 3e-5f) : big * sqrtf((float)D) * (1.f + 1e-5f);
        if (__any_sync(0xffffffffu, lost)) b = __int_as_float(0x7f800000);
        best = fmaxf(best, b);
    }
    if (mx == nullptr) return;
    // one atomic a block
    __shared__ float wbest[8];
    if (lane == 0) wbest[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) best = fmaxf(best, wbest[w]);
        atomicMax(mx, (unsigned long long)__double_as_longlong((double)best));
    }
}

__device__ __forceinline__ double dist64(const double* __restrict__ q, const double* __restrict__ c, int D)
{
    double acc = 0.0;
    for (int d = 0; d < D; ++d) {
        const double t = __dsub_rn(q[d], c[d]);
        acc = __dadd_rn(acc, __dmul_rn(t, t));
    }
    return acc;
}

__device__ __forceinline__ bool pair_less(double a, int ia, double b, int ib) { return a < b || (a == b && ia < ib); }

// FP64 distances of the FP32 candidates that can still matter: an FP32 distance is within E of its
// FP64 one (see the file's head), so the k-th FP64 distance is at most the k-th FP32 one plus E and a
// candidate more than 2 E past that cannot be among the k.  Block (q, j): candidates 32 j .. 32 j + 31 of
// query q, a thread each, the next eight columns in flight; the sum runs in d order.  ncand[q]: how many.
// Bound by the FP64 pipe (three operations a column): a
// warp's operations take about 90 cycles each whatever runs beside it (blocks of 128 or of 16 threads, or
// two blocks an SM at most: 22, 25 and 20 us).  64 queries x 256 x 128: 19 us, 24.6 with blocks of two
// warps and no loads ahead, 197 as one warp a query over all candidates.
constexpr int kDistT = 32;
__device__ __forceinline__ double err_bound(const double* qv, int D, double d32, unsigned long long cmax_bits)
{
    const int lane = threadIdx.x & 31;
    double qq = 0.0;
    for (int d = lane; d < D; d += 32) qq = __dadd_rn(qq, __dmul_rn(qv[d], qv[d]));
    for (int o = 16; o > 0; o >>= 1) qq += __shfl_xor_sync(0xffffffffu, qq, o);
    const double s = sqrt(qq) + __longlong_as_double((long long)cmax_bits);
    // norms and products that can leave the float range: rows without an FP32 key are in no shortlist,
    // however near they are, so none proves anything
    if (!(s * s < 1e38)) return __longlong_as_double(0x7ff0000000000000ll);
    // (the last term: squares and sums rounded in the subnormal range)
    return ((double)D / 8.0 + 10.0) * 5.9604644775390625e-08 * s * s + 1e-5 * d32 + (double)D * 1e-44;
}

__global__ void __launch_bounds__(kDistT) dist64_kernel(const double* __restrict__ data, int64_t N, int64_t ldc,
                                                        const double* __restrict__ queries, int64_t ldq, int D,
                                                        const float* __restrict__ cd32, const int32_t* __restrict__ ci,
                                                        int kp, int k, const unsigned long long* __restrict__ cmax_bits,
                                                        double* __restrict__ dd, int32_t* __restrict__ ncand,
                                                        double* __restrict__ bound)
{
    const int64_t q = blockIdx.x;
    const double* qv = queries + q * ldq;
    const float* d32 = cd32 + q * kp;
    const double E = err_bound(qv, D, (double)d32[kp - 1], *cmax_bits);
    const double lim = (double)d32[k - 1] + 2.0 * E;
    const bool all = kp >= N || !(lim < __longlong_as_double(0x7ff0000000000000ll));
    const int j = blockIdx.y * kDistT + threadIdx.x;
    if (blockIdx.y == 0 && threadIdx.x == 0) bound[q] = (double)d32[kp - 1] - E;
    const bool in = j < kp;
    const bool want = in && (all || (double)d32[j] <= lim);
    // candidates come sorted by FP32 distance (missing ones last): the last wanted one counts them
    if (want && (j == kp - 1 || !(all || (double)d32[j + 1] <= lim))) ncand[q] = j + 1;
    if (!want) return;
    const int32_t n = ci[q * kp + j];
    double acc = 0.0;
    if (n < 0) {
        acc = __longlong_as_double(0x7ff0000000000000ll);
    } else {
        const double* c = data + (int64_t)n * ldc;
        int d = 0;
        double v[8];
        if (D >= 8)
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __ldg(c + i);
        for (; d + 8 <= D; d += 8) {
            double w[8], t[8];
            const bool more = d + 16 <= D;
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = more ? __ldg(c + d + 8 + i) : 0.0;
            // stage by stage: column by column each operation waited for the one before it
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] = __dsub_rn(__ldg(qv + d + i), v[i]);
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] = __dmul_rn(t[i], t[i]);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc = __dadd_rn(acc, t[i]);
                v[i] = w[i];
            }
        }
        for (; d < D; ++d) {
            const double t = __dsub_rn(__ldg(qv + d), __ldg(c + d));
            acc = __dadd_rn(acc, __dmul_rn(t, t));
        }
    }
    dd[q * kp + j] = acc;
}

// One block per query: its candidates in (distance, index) order by counting the smaller ones, the
// acceptance test, the k results or an entry in the failure list.
__global__ void __launch_bounds__(256) rerank64_kernel(int64_t N, const double* __restrict__ dd,
                                                       const int32_t* __restrict__ ci, const int32_t* __restrict__ ncand,
                                                       const double* __restrict__ bound, int kp, int k,
                                                       const double* __restrict__ queries, int64_t ldq, int D,
                                                       double* __restrict__ out_d, int32_t* __restrict__ out_i,
                                                       uint32_t* __restrict__ fails)
{
    // distances as their bits: not negative, so they order as integers (and a double comparison costs
    // what 32 integer ones do)
    __shared__ longlong2 sw[kSortMax];  // {distance bits, index}
    __shared__ int rank[kSortMax];
    __shared__ double kth;
    const int64_t q = blockIdx.x;
    const int m = ncand[q];
    bool gap = false;
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        const int32_t n = ci[q * kp + j];
        gap |= n < 0;
        sw[j] = make_longlong2(__double_as_longlong(dd[q * kp + j]), n >= 0 ? n : 0x7fffffff);
    }
    if (threadIdx.x == 0) kth = __longlong_as_double(0x7ff0000000000000ll);
    bool missing = __syncthreads_or(gap) != 0;
    if (missing && kp >= N) {
        // (a query that is not finite has no finite distance to look for)
        bool inf = false;
        for (int d = threadIdx.x; d < D; d += blockDim.x)
            inf |= !(fabs(queries[q * ldq + d]) < __longlong_as_double(0x7ff0000000000000ll));
        missing = __syncthreads_or(inf) == 0;
    }
    for (int j = threadIdx.x; j < m; j += blockDim.x) {
        int below = 0;
        const longlong2 w = sw[j];
        for (int e = 0; e < m; ++e) {
            const longlong2 x = sw[e];
            // equal pairs (missing candidates) by place
            below += x.x < w.x || (x.x == w.x && (x.y < w.y || (x.y == w.y && e < j))) ? 1 : 0;
        }
        rank[j] = below;
        if (below == k - 1) kth = __longlong_as_double(w.x);
    }
    __syncthreads();
    // the shortlist covers the corpus (a row whose norm or key overflowed FP32 is missing from it), or its
    // k-th FP64 distance stays below the smallest FP64 distance any row outside it can have
    if (!(kp >= N ? !missing : m >= k && kth < bound[q])) {
        if (threadIdx.x == 0) fails[1 + atomicAdd(fails, 1u)] = (uint32_t)q;
        return;
    }
    for (int j = threadIdx.x; j < m; j += blockDim.x)
        if (rank[j] < k) {
            out_d[q * k + rank[j]] = __longlong_as_double(sw[j].x);
            out_i[q * k + rank[j]] = (int32_t)sw[j].y;
        }
}

// One CTA per listed query: FP64 distances to every row, kept in a shared
// buffer below a shrinking threshold, sorted and trimmed to k when it fills.
__global__ void __launch_bounds__(256) brute64_kernel(const double* __restrict__ data, int64_t ldc, int64_t N,
                                                      const double* __restrict__ queries, int64_t ldq, int D, int k,
                                                      const uint32_t* __restrict__ fails, double* __restrict__ out_d,
                                                      int32_t* __restrict__ out_i)
{
    __shared__ double bd[kBruteBuf];
    __shared__ int bi[kBruteBuf];
    __shared__ int cnt;
    __shared__ double T;
    if (blockIdx.x >= fails[0]) return;
    const int64_t q = fails[1 + blockIdx.x];
    const double* qv = queries + q * ldq;
    if (threadIdx.x == 0) {
        cnt = 0;
        T = __longlong_as_double(0x7ff0000000000000ll);
    }
    __syncthreads();
    auto trim = [&]() {
        // sort the buffer (padded to kBruteBuf), keep the first k, threshold = k-th (if full)
        for (int j = cnt + threadIdx.x; j < kBruteBuf; j += blockDim.x) {
            bd[j] = __longlong_as_double(0x7ff0000000000000ll);
            bi[j] = 0x7fffffff;
        }
        __syncthreads();
        for (int size = 2; size <= kBruteBuf; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = threadIdx.x; i < kBruteBuf / 2; i += blockDim.x) {
                    const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
                    const bool up = (lo & size) == 0;
                    if (pair_less(bd[hi], bi[hi], bd[lo], bi[lo]) == up) {
                        const double td = bd[lo];
                        bd[lo] = bd[hi];
                        bd[hi] = td;
                        const int ti = bi[lo];
                        bi[lo] = bi[hi];
                        bi[hi] = ti;
                    }
                }
                __syncthreads();
            }
        if (threadIdx.x == 0) {
            cnt = min(cnt, k);
            if (cnt == k) T = bd[k - 1];
        }
        __syncthreads();
    };
    for (int64_t base = 0; base < N; base += blockDim.x) {
        if (cnt + (int)blockDim.x > kBruteBuf) trim();
        const int64_t n = base + threadIdx.x;
        if (n < N) {
            const double v = dist64(qv, data + n * ldc, D);
            // rows arrive in increasing index order: a later row never wins a tie
            if (v < T) {
                const int slot = atomicAdd(&cnt, 1);
                bd[slot] = v;
                bi[slot] = (int)n;
            }
        }
        __syncthreads();
    }
    trim();
    for (int j = threadIdx.x; j < k; j += blockDim.x) {
        out_d[q * k + j] = bd[j];
        out_i[q * k + j] = bi[j];
    }
}

int shortlist_len(int k, int64_t N) { return (int)std::min<int64_t>(N, std::min(kSortMax, std::max(k + 32, 2 * k))); }

int search_device(const double* corpus, int64_t N, int64_t ldc, const double* queries, int64_t Q, int64_t ldq, int D,
                  int k, double* dist, int32_t* idx, cudaStream_t s)
{
    if (N <= 0 || D <= 0 || k <= 0 || Q < 0 || ldc < D || ldq < D || !corpus || (Q > 0 && !queries))
        return fail(KNNS_ERR_INVALID, "invalid arguments");
    if (k > N) return fail(KNNS_ERR_INVALID, "k=%d exceeds the corpus size N=%lld", k, (long long)N);
    if (k > kSortMax) return fail(KNNS_ERR_UNSUPPORTED, "the double path returns at most %d neighbours", kSortMax);
    if (N > 0x7fffffffLL) return fail(KNNS_ERR_UNSUPPORTED, "corpus larger than 2^31-1 rows");
    if (Q == 0) return KNNS_OK;
    Work* W = work_for_device();
    std::lock_guard<std::mutex> lk(W->mu);
    const int kp = shortlist_len(k, N);
    int rc = W->c32.ensure((size_t)N * D * 4);
    if (!rc) rc = W->q32.ensure((size_t)Q * D * 4);
    if (!rc) rc = W->cand_d.ensure((size_t)Q * kp * 4);
    if (!rc) rc = W->cand_i.ensure((size_t)Q * kp * 4);
    if (!rc) rc = W->dd.ensure((size_t)Q * kp * 8);
    if (!rc) rc = W->bound.ensure((size_t)Q * 8);
    if (!rc) rc = W->ncand.ensure((size_t)Q * 4);
    if (!rc) rc = W->cmax.ensure(8);
    if (!rc) rc = W->fails.ensure((size_t)(Q + 1) * 4);
    if (rc) return rc;
    F64_CUDA(cudaMemsetAsync(W->cmax.p, 0, 8, s));
    F64_CUDA(cudaMemsetAsync(W->fails.p, 0, 4, s));
    auto blocks = [](int64_t rows) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((rows + 7) / 8, kMostBlocks)); };
    auto* to_f32_rows = D <= 128 ? to_f32_kernel<4> : to_f32_kernel<8>;
    to_f32_rows<<<blocks(N), 256, 0, s>>>(corpus, N, ldc, D, (float*)W->c32.p, (unsigned long long*)W->cmax.p);
    to_f32_rows<<<blocks(Q), 256, 0, s>>>(queries, Q, ldq, D, (float*)W->q32.p, nullptr);
    F64_CUDA(cudaGetLastError());
    // FP32 shortlist of kp rows per query, ordered by exact FP32 distance
    rc = knns_search_device((const float*)W->c32.p, N, D, (const float*)W->q32.p, Q, D, D, kp, (float*)W->cand_d.p,
                            (int32_t*)W->cand_i.p, nullptr, s);
    if (rc) return fail(rc, "float shortlist: %s", knns_last_error());
    const dim3 dgrid((unsigned)Q, (unsigned)((kp + kDistT - 1) / kDistT));
    dist64_kernel<<<dgrid, kDistT, 0, s>>>(
        corpus, N, ldc, queries, ldq, D, (const float*)W->cand_d.p, (const int32_t*)W->cand_i.p, kp, k,
        (const unsigned long long*)W->cmax.p, (double*)W->dd.p, (int32_t*)W->ncand.p, (double*)W->bound.p);
    rerank64_kernel<<<(unsigned)Q, 256, 0, s>>>(N, (const double*)W->dd.p, (const int32_t*)W->cand_i.p,
                                                (const int32_t*)W->ncand.p, (const double*)W->bound.p, kp, k, queries, ldq, D, dist, idx,
                                                (uint32_t*)W->fails.p);
    // queries whose shortlist could not be proven complete (the grid covers every query; the
    // CTAs past the failure count return at once)
    brute64_kernel<<<(unsigned)Q, 256, 0, s>>>(corpus, ldc, N, queries, ldq, D, k, (const uint32_t*)W->fails.p,
                                                dist, idx);
    F64_CUDA(cudaGetLastError());
    rc = knns_check_device(s);
    if (rc) return fail(rc, "%s", knns_last_error());
    return KNNS_OK;
}

int search_host(const double* query, const double* data, double* values, double* indices, int N, int Q, int D,
                int k, double* seconds)
{
    if (!query || !data || N <= 0 || Q < 0 || D <= 0 || k <= 0) return fail(KNNS_ERR_INVALID, "invalid arguments");
    Work* W = work_for_device();
    cudaStream_t s = nullptr;
    F64_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int rc;
    {
        std::lock_guard<std::mutex> lk(W->mu);
        rc = W->hc.ensure((size_t)N * D * 8);
        if (!rc) rc = W->hq.ensure((size_t)Q * D * 8 + 8);
        if (!rc) rc = W->hd.ensure((size_t)Q * k * 8 + 8);
        if (!rc) rc = W->hi.ensure((size_t)Q * k * 4 + 8);
    }
    std::unique_ptr<int32_t[]> ih(new int32_t[(size_t)Q * k + 1]);
    if (!rc) {
        cudaEventRecord(e0, s);
        cudaMemcpyAsync(W->hc.p, data, (size_t)N * D * 8, cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(W->hq.p, query, (size_t)Q * D * 8, cudaMemcpyHostToDevice, s);
        rc = search_device((const double*)W->hc.p, N, D, (const double*)W->hq.p, Q, D, D, k, (double*)W->hd.p,
                           (int32_t*)W->hi.p, s);
        if (!rc) {
            cudaMemcpyAsync(values, W->hd.p, (size_t)Q * k * 8, cudaMemcpyDeviceToHost, s);
            cudaMemcpyAsync(ih.get(), W->hi.p, (size_t)Q * k * 4, cudaMemcpyDeviceToHost, s);
            cudaEventRecord(e1, s);
            if (cudaStreamSynchronize(s) != cudaSuccess) rc = fail(KNNS_ERR_CUDA, "copy back failed");
        }
    }
    if (!rc) {
        for (int64_t i = 0; i < (int64_t)Q * k; ++i) indices[i] = (double)ih[i];
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (seconds) *seconds = ms / 1000.0;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaStreamDestroy(s);
    return rc;
}

}  // namespace
}  // namespace knn64

using namespace knn64;

extern "C" {

int knns_search_device_f64(const double* corpus, int64_t N, int64_t ldc, const double* queries, int64_t Q,
                           int64_t ldq, int D, int k, double* dist, int32_t* idx, void* stream)
{
    g_err.clear();
    return search_device(corpus, N, ldc, queries, Q, ldq, D, k, dist, idx, (cudaStream_t)stream);
}

int knns_search_host_f64(const double* corpus, int64_t N, const double* queries, int64_t Q, int D, int k,
                         double* dist, int32_t* idx)
{
    g_err.clear();
    if (N > 0x7fffffffLL || Q > 0x7fffffffLL) return fail(KNNS_ERR_UNSUPPORTED, "sizes beyond int");
    std::unique_ptr<double[]> fi(new double[(size_t)Q * k + 1]);
    double secs = 0;
    int rc = search_host(queries, corpus, dist, fi.get(), (int)N, (int)Q, D, k, &secs);
    if (!rc && idx)
        for (int64_t i = 0; i < Q * k; ++i) idx[i] = (int32_t)fi[i];
    return rc;
}

const char* knns_f64_last_error(void) { return g_err.c_str(); }

// include/cuknns.h:75 (src/cuknnBitonic.cu:422), knntype = double
double gpuknnsBitonic(double* query, double* data, double* values, double* indices, int objects, int numQueries,
                      int attributes, int k, int numStreams)
{
    (void)numStreams;
    g_err.clear();
    double secs = 0;
    if (search_host(query, data, values, indices, objects, numQueries, attributes, k, &secs)) return DBL_MAX;
    return secs;
}

// include/cuknns.h:83 (src/cuknnHeap.cu:394): same engine, same contract
double gpuknnsHeap(double* query, double* data, double* values, double* indices, int objects, int numQueries,
                   int attributes, int k, int numStreams)
{
    return gpuknnsBitonic(query, data, values, indices, objects, numQueries, attributes, k, numStreams);
}

// include/cuknns.h:85 (src/knnsplan.cu:25): the double engine has one configuration
void knnsplan(knnplan* plan, long int N, long int Q, long int D, long int k)
{
    if (!plan) return;
    plan->pt2Function = gpuknnsBitonic;
    plan->objects = (int)N;
    plan->numQueries = (int)Q;
    plan->dimentions = (int)D;
    plan->k = (int)k;
    plan->numStreams = 1;
}

// include/cuknns.h:87 (src/knnsexecute.cu:6)
void knnsexecute(knnplan plan, double* data, double* queries, double* KNNdist, double* KNNidx)
{
    const double t = plan.pt2Function(queries, data, KNNdist, KNNidx, plan.objects, plan.numQueries, plan.dimentions,
                                      plan.k, plan.numStreams);
    printf("Time Elapsed: %f\n", t);
}

}  // extern "C"
