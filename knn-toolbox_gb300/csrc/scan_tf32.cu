// scan_tf32.cu -- tensor-core 3xTF32 threshold scan for FP32 data of any width and
// shortlists of up to 512 entries.
//
// The scan on split keys (scan_f16.cu) with TF32 operands instead of FP16 ones, at half its rate:
// it serves the searches whose result depends on the keys' rounding -- shortlists without a margin
// over k (k close to 512, or to 128 beside the BF16 scan), and rerank = 0, which returns the keys.
//
// Keys: with x = hi + lo (hi = tf32(x), lo = tf32(x - hi)), q.c is accumulated in
// FP32 as qhi.chi + qhi.clo + qlo.chi by tcgen05.mma.kind::tf32; a correction
// product whose low part is zero for the whole corpus tile (or query tile) is
// skipped -- it would add exact zeros.
//
// Tile: 128 queries (MMA M, TMEM lanes) x 128 corpus rows (MMA N), K in chunks of
// 32 FP32 columns (one 128-byte swizzle row).  Both operands come from shared
// memory, so any D works and tensor memory holds only accumulators: four of 128
// columns.  A ring slot carries one K chunk of the query tile and of the corpus
// tile, high and low parts (4 x 16 KB).
// Warp roles (608 threads):
//   warp 0      producer: per tile and K chunk the query and corpus boxes (2-D TMA,
//               32 fp32 x 128 rows, 128-byte swizzle), low parts only where present;
//               per tile the corpus norms (1-D bulk copy);
//   warps 1, 18 MMA issuers, into accumulator t mod 4: of the even / odd tiles when a
//               tile takes at most half the ring, else warp 1 alone (see below);
//   warps 2..17 epilogue: thread = query (TMEM lane); warp 2 + 4p + j reads
//               columns [32p, 32p + 32) of lane quarter j, releases the
//               accumulator, forms the keys, appends those below the threshold.
// Every mbarrier wait is bounded; on timeout the kernel records an error code in
// the device error word and winds down without hanging the GPU.
#include <algorithm>
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>
#include "common.cuh"
#include "kernels.h"
#include "scan_common.cuh"
#include "tc_ptx.cuh"

namespace knn {

namespace {
constexpr int kTN = 128;                     // corpus rows per tile
constexpr int kParts = kScanParts;           // epilogue column parts (32 columns each)
constexpr int kEpi = 4 * kParts;             // epilogue warps
constexpr int kIss = 2;                      // MMA issuing threads
constexpr int kThreads = 32 * (1 + kIss + kEpi);
constexpr int kAcc = 4;                      // TMEM accumulators of 128 columns
constexpr int kNorm = 8;                     // tiles of corpus norms in flight
constexpr uint32_t kBox = 128u * 128u;       // one operand box: 128 rows x 32 fp32
constexpr uint32_t kSlot = 4u * kBox;        // query hi, query lo, corpus hi, corpus lo
constexpr int kMaxRing = 3;
constexpr uint32_t kCtrl = 512;
constexpr uint64_t kTimeout = 4000000000ull;
constexpr uint32_t kIdesc = ptx::idesc_tf32(kTileQ, kTN);

struct TSmem {
    unsigned char* ring;
    float* norms;       // [kNorm][kTN]
    uint64_t* full;     // [kMaxRing]
    uint64_t* empty;    // [kMaxRing]
    uint64_t* accf;     // [kAcc]
    uint64_t* acce;     // [kAcc]
    uint64_t* nfull;    // [kNorm]
    uint64_t* nempty;   // [kNorm]
    uint64_t* drain;
    uint32_t* tmem_holder;
    volatile int* abort;
    volatile uint32_t* slot_lo;  // [kMaxRing]: bit 0 query low part loaded, bit 1 corpus low part
};

__device__ __forceinline__ bool t_wait(const TscanArgs& a, const TSmem& s, uint64_t* bar, uint32_t parity, int code)
{
    if (ptx::mbar_try_wait(bar, parity)) return true;
    if (*s.abort) return false;
    if (ptx::mbar_wait(bar, parity, kTimeout)) return true;
    atomicCAS(a.err, 0, code);
    *s.abort = 1;
    return false;
}

template <bool kDense>
__global__ void __launch_bounds__(kThreads, 1) tscan_kernel(const __grid_constant__ TscanArgs a)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    // device-side path choice: the kernel runs only when *run_if != 0
    if (a.run_if != nullptr && *a.run_if == 0u) return;
    if ((ptx::smem_u32(sm) & 1023u) != 0u) {
        if (threadIdx.x == 0) atomicCAS(a.err, 0, kDevMisaligned);
        return;
    }
    const int R = a.ring;
    TSmem s;
    s.ring = sm;
    s.norms = reinterpret_cast<float*>(sm + (size_t)R * kSlot);
    uint64_t* bars = reinterpret_cast<uint64_t*>(s.norms + kNorm * kTN);
    s.full = bars;
    s.empty = bars + kMaxRing;
    s.accf = bars + 2 * kMaxRing;
    s.acce = s.accf + kAcc;
    s.nfull = s.acce + kAcc;
    s.nempty = s.nfull + kNorm;
    s.drain = s.nempty + kNorm;
    uint32_t* words = reinterpret_cast<uint32_t*>(s.drain + 1);
    s.tmem_holder = words;
    s.abort = reinterpret_cast<volatile int*>(words + 1);
    s.slot_lo = words + 2;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t q0 = (int64_t)blockIdx.x * kTileQ;
    const int split = a.split0 + (int)blockIdx.y;
    const int64_t n_begin = (int64_t)split * a.split_len;
    const int64_t n_end = min(a.N, n_begin + a.split_len);
    const int ntiles = n_end > n_begin ? (int)((n_end - n_begin + kTN - 1) / kTN) : 0;
    const int nch = a.dp / 32;

    if (tid == 0) {
        for (int i = 0; i < R; ++i) {
            ptx::mbar_init(&s.full[i], 1);
            ptx::mbar_init(&s.empty[i], 1);
        }
        for (int b = 0; b < kAcc; ++b) {
            ptx::mbar_init(&s.accf[b], 1);
            ptx::mbar_init(&s.acce[b], kEpi);
        }
        for (int b = 0; b < kNorm; ++b) {
            ptx::mbar_init(&s.nfull[b], 1);
            ptx::mbar_init(&s.nempty[b], kEpi);
        }
        ptx::mbar_init(s.drain, kIss);
        *s.abort = 0;
        ptx::fence_mbar_init();
        ptx::tma_prefetch_desc(&a.tm_qhi);
        ptx::tma_prefetch_desc(&a.tm_qlo);
        ptx::tma_prefetch_desc(&a.tm_chi);
        ptx::tma_prefetch_desc(&a.tm_clo);
    }
    if (warp == 1) {
        ptx::tmem_alloc(s.tmem_holder, 512);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *s.tmem_holder;

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (lane == 0) {
            const uint32_t qlo = a.qlo_flags ? __ldg(a.qlo_flags + blockIdx.x) : 1u;
            int it = 0;
            bool ok = true;
            for (int t = 0; t < ntiles && ok; ++t) {
                const int64_t n0 = n_begin + (int64_t)t * kTN;
                // view rows are whole 128-row tiles of the flags' corpus (main pass: split_len % 128 == 0)
                const uint32_t clo = a.clo_flags ? __ldg(a.clo_flags + n0 / kTN) : 1u;
                for (int c = 0; c < nch; ++c, ++it) {
                    const int st = it % R;
                    const uint32_t ph = (uint32_t)(it / R) & 1u;
                    if (!t_wait(a, s, &s.empty[st], ph ^ 1u, kDevTimeoutProducer)) { ok = false; break; }
                    unsigned char* dst = s.ring + (size_t)st * kSlot;
                    s.slot_lo[st] = (qlo ? 1u : 0u) | (clo ? 2u : 0u);  // published by the arrive below
                    ptx::mbar_arrive_expect_tx(&s.full[st], kBox * (2u + (qlo ? 1u : 0u) + (clo ? 1u : 0u)));
                    ptx::tma_load_2d(dst, &a.tm_qhi, &s.full[st], c * 32, (int)q0);
                    if (qlo) ptx::tma_load_2d(dst + kBox, &a.tm_qlo, &s.full[st], c * 32, (int)q0);
                    ptx::tma_load_2d(dst + 2 * kBox, &a.tm_chi, &s.full[st], c * 32, (int)n0);
                    if (clo) ptx::tma_load_2d(dst + 3 * kBox, &a.tm_clo, &s.full[st], c * 32, (int)n0);
                }
                if (!ok) break;
                const int ns = t % kNorm;
                if (!t_wait(a, s, &s.nempty[ns], ((uint32_t)(t / kNorm) & 1u) ^ 1u, kDevTimeoutProducer)) {
                    ok = false;
                    break;
                }
                // the norms are padded with +inf at least one tile past the view
                ptx::mbar_arrive_expect_tx(&s.nfull[ns], kTN * 4u);
                ptx::bulk_load(s.norms + ns * kTN, a.cn + n0, kTN * 4u, &s.nfull[ns]);
            }
            if (!ok) {
                // let copies already issued land before the CTA winds down
                const int first = it - R > 0 ? it - R : 0;
                for (int j = first; j < it; ++j) ptx::mbar_wait(&s.full[j % R], (uint32_t)(j / R) & 1u, kTimeout);
            }
        }
    } else if (warp == 1 || warp == 2 + kEpi) {
        // ------------------------------------------------------------ MMA issuers
        // Two issuers alternate tiles only when a tile's chunks fill at most half the ring: an
        // issuer's wait on a slot must never run two phases ahead of the slot's barrier, which
        // is guaranteed when the slot's previous use (R chunks back) is one of its own chunks
        // (or none).  With longer tiles a second issuer could wait on a slot whose previous
        // use, in the other issuer's tile, has not landed yet -- its parity would then read
        // as complete -- so warp 1 issues every tile in order and warp 18 only drains.
        const int nissue = 2 * nch <= R ? kIss : 1;
        if (lane == 0) {
            const int iss = warp == 1 ? 0 : 1;
            bool ok = true;
            for (int t = iss; t < ntiles && ok && iss < nissue; t += nissue) {
                const int b = t % kAcc;
                const uint32_t use = (uint32_t)(t / kAcc);
                if (!t_wait(a, s, &s.acce[b], (use & 1u) ^ 1u, kDevTimeoutMma)) { ok = false; break; }
                ptx::tc_fence_after();
                const uint32_t d_tmem = tmem + (uint32_t)b * kTN;
                int it = t * nch;
                for (int c = 0; c < nch; ++c, ++it) {
                    const int st = it % R;
                    const uint32_t ph = (uint32_t)(it / R) & 1u;
                    if (!t_wait(a, s, &s.full[st], ph, kDevTimeoutMma)) { ok = false; break; }
                    ptx::tc_fence_after();
                    const uint32_t lo = s.slot_lo[st];
                    const uint32_t base = ptx::smem_u32(s.ring + (size_t)st * kSlot);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        // K steps of 8 fp32 (32 bytes) within the 128-byte swizzle rows
                        const uint64_t qh = ptx::desc_sw128_kmajor(base + kk * 32);
                        const uint64_t ch = ptx::desc_sw128_kmajor(base + 2 * kBox + kk * 32);
                        ptx::mma_tf32_ss(d_tmem, qh, ch, kIdesc, (c | kk) != 0);
                        if (lo & 2u) ptx::mma_tf32_ss(d_tmem, qh, ptx::desc_sw128_kmajor(base + 3 * kBox + kk * 32), kIdesc, 1u);
                        if (lo & 1u) ptx::mma_tf32_ss(d_tmem, ptx::desc_sw128_kmajor(base + kBox + kk * 32), ch, kIdesc, 1u);
                    }
                    // the tile's last chunk: accumulator-ready first (the epilogue waits on it)
                    if (c == nch - 1) ptx::mma_commit(&s.accf[b]);
                    ptx::mma_commit(&s.empty[st]);
                }
                if (!ok) break;
            }
            // all MMAs issued by this thread retire before TMEM is released
            ptx::mma_commit(s.drain);
            ptx::mbar_wait(s.drain, 0, kTimeout);
        }
    } else {
        // ------------------------------------------------------------ epilogue
        const int ew = warp - 2;
        const int quad = warp & 3;  // TMEM lane quarter this warp may access
        const int part = ew >> 2;   // columns [32 part, 32 part + 32) of every tile
        const int row = quad * 32 + lane;
        const int64_t q = q0 + row;
        const bool valid = q < a.Q;
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        const float T = valid ? (a.thr ? __ldg(a.thr + q) : __int_as_float(0x7f800000)) : -__int_as_float(0x7f800000);
        const size_t seg = (size_t)split * kParts + part;
        uint64_t* out = kDense ? nullptr : a.cand + (seg * (size_t)a.Q + (size_t)(valid ? q : 0)) * (size_t)a.cap;
        // dense: this warp's rows
        float* krow = kDense ? a.keys + (q0 + quad * 32) * a.ldk : nullptr;
        const int krows = (int)min((int64_t)32, a.Q - (q0 + quad * 32));
        uint32_t cnt = 0;
        const uint32_t cap = (uint32_t)a.cap;
        for (int t = 0; t < ntiles; ++t) {
            const int b = t % kAcc;
            const uint32_t use = (uint32_t)(t / kAcc);
            const int ns = t % kNorm;
            // warp-uniform outcome: tcgen05.ld below is warp-collective
            const bool ok = t_wait(a, s, &s.accf[b], use & 1u, kDevTimeoutEpilogue) &&
                            t_wait(a, s, &s.nfull[ns], (uint32_t)(t / kNorm) & 1u, kDevTimeoutEpilogue);
            if (!__all_sync(0xffffffffu, ok)) break;
            ptx::tc_fence_after();
            float v[32];
            __syncwarp();
            ptx::tmem_ld32(tmem + (uint32_t)b * kTN + lane_base + (uint32_t)(32 * part), v);
            ptx::tmem_wait_ld_regs(v);
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s.acce[b]);
            const float* nrm = s.norms + ns * kTN + 32 * part;
            const uint32_t base = (uint32_t)(n_begin + (int64_t)t * kTN) + (uint32_t)(32 * part);
            chunk_norm_keys<32>(v, nrm);
            if constexpr (kDense) {
                chunk_store<32>(v, krow + base, a.ldk, krows);
            } else {
                float g[4];
                chunk_minima<32>(v, g);
                if (__any_sync(0xffffffffu, min_of(g) < T)) chunk_append<32>(v, g, T, base, out, cap, cnt);
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s.nempty[ns]);
        }
        if (!kDense && valid) a.cnt[seg * (size_t)a.Q + (size_t)q] = cnt;
    }

    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    if (warp == 1) {
        __syncwarp();
        ptx::tmem_dealloc(tmem, 512);
    }
}

// ---------------------------------------------------------------- queries in tensor memory
// Rows of at most 128 columns: the query tile's TF32 hi and lo parts sit in tensor memory (A
// from TMEM, tcgen05.mma kind::tf32 [d], [a], b-desc), so the ring carries only corpus chunks
// (high and low parts, 2 x 16 KB per slot) and each MMA reads one operand from shared memory:
// with both operands there, the MMA reads and the TMA fills together exceed the shared-memory
// bandwidth.  Tensor memory: A hi [0, dp), A lo [dp, 2 dp), two 128-column accumulators at
// 256 and 384.  Two MMA issuers, warps 1 and 18, take the even and the odd tiles, one
// accumulator each: the tensor pipe queues little work beyond the MMA being issued, so one
// thread's barrier waits and commits idle it.  Each has its own half of the ring: a slot's uses all
// belong to one issuer, which waits for each of them in order, so no wait can take an older phase of
// a slot's barrier for a newer one.  Keys, epilogue and segments are those of tscan_kernel, so
// the candidates are the same.
constexpr int kAccTA = 2;
constexpr uint32_t kAccColTA = 256;
constexpr uint32_t kSlotTA = 2u * kBox;  // corpus hi, corpus lo
constexpr int kMaxRingTA = 6;

struct TaSmem {
    unsigned char* ring;
    float* norms;       // [kNorm][kTN]
    uint64_t* full;     // [kMaxRingTA]
    uint64_t* empty;    // [kMaxRingTA]
    uint64_t* accf;     // [kAccTA]
    uint64_t* acce;     // [kAccTA]
    uint64_t* nfull;    // [kNorm]
    uint64_t* nempty;   // [kNorm]
    uint64_t* aready;
    uint64_t* drain;
    uint32_t* tmem_holder;
    volatile int* abort;
    volatile uint32_t* slot_lo;  // [kMaxRingTA]: 1 when the slot's corpus low part was loaded
    uint32_t* alo;               // 1 when some query of the tile has a low part
};

__device__ __forceinline__ bool ta_wait(const TscanArgs& a, const TaSmem& s, uint64_t* bar, uint32_t parity, int code)
{
    if (ptx::mbar_try_wait(bar, parity)) return true;
    if (*s.abort) return false;
    if (ptx::mbar_wait(bar, parity, kTimeout)) return true;
    atomicCAS(a.err, 0, code);
    *s.abort = 1;
    return false;
}

__device__ __forceinline__ float tf32_round(float x)
{
    uint32_t u = __float_as_uint(x);
    if ((u & 0x7f800000u) == 0x7f800000u) return x;
    u += 0xfffu + ((u >> 13) & 1u);
    u &= 0xffffe000u;
    return __uint_as_float(u);
}

template <bool kDense>
__global__ void __launch_bounds__(kThreads, 1) tscan_ta_kernel(const __grid_constant__ TscanArgs a)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    // device-side path choice: the kernel runs only when *run_if != 0
    if (a.run_if != nullptr && *a.run_if == 0u) return;
    if ((ptx::smem_u32(sm) & 1023u) != 0u) {
        if (threadIdx.x == 0) atomicCAS(a.err, 0, kDevMisaligned);
        return;
    }
    const int R = a.ring;
    TaSmem s;
    s.ring = sm;
    s.norms = reinterpret_cast<float*>(sm + (size_t)R * kSlotTA);
    uint64_t* bars = reinterpret_cast<uint64_t*>(s.norms + kNorm * kTN);
    s.full = bars;
    s.empty = bars + kMaxRingTA;
    s.accf = bars + 2 * kMaxRingTA;
    s.acce = s.accf + kAccTA;
    s.nfull = s.acce + kAccTA;
    s.nempty = s.nfull + kNorm;
    s.aready = s.nempty + kNorm;
    s.drain = s.aready + 1;
    uint32_t* words = reinterpret_cast<uint32_t*>(s.drain + 1);
    s.tmem_holder = words;
    s.abort = reinterpret_cast<volatile int*>(words + 1);
    s.alo = words + 2;
    s.slot_lo = words + 3;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t q0 = (int64_t)blockIdx.x * kTileQ;
    const int split = a.split0 + (int)blockIdx.y;
    const int64_t n_begin = (int64_t)split * a.split_len;
    const int64_t n_end = min(a.N, n_begin + a.split_len);
    const int ntiles = n_end > n_begin ? (int)((n_end - n_begin + kTN - 1) / kTN) : 0;
    const int nch = a.dp / 32;
    const int half = R / 2;  // an issuer's ring slots

    if (tid == 0) {
        for (int i = 0; i < R; ++i) {
            ptx::mbar_init(&s.full[i], 1);
            ptx::mbar_init(&s.empty[i], 1);
        }
        for (int b = 0; b < kAccTA; ++b) {
            ptx::mbar_init(&s.accf[b], 1);
            ptx::mbar_init(&s.acce[b], kEpi);
        }
        for (int b = 0; b < kNorm; ++b) {
            ptx::mbar_init(&s.nfull[b], 1);
            ptx::mbar_init(&s.nempty[b], kEpi);
        }
        ptx::mbar_init(s.aready, 4);
        ptx::mbar_init(s.drain, kIss);
        *s.abort = 0;
        *s.alo = 0;
        ptx::fence_mbar_init();
        ptx::tma_prefetch_desc(&a.tm_chi);
        ptx::tma_prefetch_desc(&a.tm_clo);
    }
    if (warp == 1) {
        ptx::tmem_alloc(s.tmem_holder, 512);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *s.tmem_holder;

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        if (lane == 0) {
            // slots and phases of the two halves
            int st[2] = {0, half};
            uint32_t ph[2] = {0, 0};
            int used[2] = {0, 0};
            bool ok = true;
            for (int t = 0; t < ntiles && ok; ++t) {
                const int64_t n0 = n_begin + (int64_t)t * kTN;
                const uint32_t clo = a.clo_flags ? __ldg(a.clo_flags + n0 / kTN) : 1u;
                const int h = t & 1;
                int x = h ? st[1] : st[0], u = h ? used[1] : used[0];
                uint32_t p = h ? ph[1] : ph[0];
                for (int c = 0; c < nch; ++c) {
                    if (!ta_wait(a, s, &s.empty[x], p ^ 1u, kDevTimeoutProducer)) { ok = false; break; }
                    unsigned char* dst = s.ring + (size_t)x * kSlotTA;
                    s.slot_lo[x] = clo;  // published by the arrive below
                    ptx::mbar_arrive_expect_tx(&s.full[x], kBox * (clo ? 2u : 1u));
                    ptx::tma_load_2d(dst, &a.tm_chi, &s.full[x], c * 32, (int)n0);
                    if (clo) ptx::tma_load_2d(dst + kBox, &a.tm_clo, &s.full[x], c * 32, (int)n0);
                    ++u;
                    if (++x == (h + 1) * half) {
                        x = h * half;
                        p ^= 1u;
                    }
                }
                if (h) st[1] = x, ph[1] = p, used[1] = u;
                else st[0] = x, ph[0] = p, used[0] = u;
                if (!ok) break;
                const int ns = t % kNorm;
                if (!ta_wait(a, s, &s.nempty[ns], ((uint32_t)(t / kNorm) & 1u) ^ 1u, kDevTimeoutProducer)) {
                    ok = false;
                    break;
                }
                // the norms are padded with +inf at least one tile past the view
                ptx::mbar_arrive_expect_tx(&s.nfull[ns], kTN * 4u);
                ptx::bulk_load(s.norms + ns * kTN, a.cn + n0, kTN * 4u, &s.nfull[ns]);
            }
            if (!ok) {
                // let copies already issued land before the CTA winds down
                for (int h = 0; h < 2; ++h) {
                    const int n = h ? used[1] : used[0];
                    for (int e = max(0, n - half); e < n; ++e)
                        ptx::mbar_wait(&s.full[h * half + e % half], (uint32_t)(e / half) & 1u, kTimeout);
                }
            }
        }
    } else if (warp == 1 || warp == 2 + kEpi) {
        // ------------------------------------------------------------ MMA issuers
        // issuer i takes the tiles t = i (mod 2), into accumulator i; each commit tracks only its own
        // MMAs.  Little stands between the accumulator's release and the tile's first MMA: slots and
        // descriptors advance by additions, and the tile's first chunk is looked at before (with the
        // K steps past the data left out: 100,003 x 43, 777 queries 60 -> 53 us).
        if (lane == 0) {
            const int iss = warp == 1 ? 0 : 1;
            bool ok = ta_wait(a, s, s.aready, 0, kDevTimeoutAload);
            ptx::tc_fence_after();
            const uint32_t alo = *s.alo;
            const uint64_t ring_desc = ptx::desc_sw128_kmajor(ptx::smem_u32(s.ring));  // (in 16-byte units)
            const uint32_t d_tmem = tmem + kAccColTA + (uint32_t)iss * kTN;
            int st = iss * half;
            uint32_t ph = 0, aph = 1;  // (accumulators start free)
            for (int t = iss; t < ntiles && ok; t += kIss, aph ^= 1u) {
                for (int c = 0; c < nch; ++c) {
                    if (!ta_wait(a, s, &s.full[st], ph, kDevTimeoutMma)) { ok = false; break; }
                    const uint32_t clo = s.slot_lo[st];
                    const uint64_t base = ring_desc + (uint64_t)((uint32_t)st * kSlotTA >> 4);
                    // K steps of 8 fp32 (32 bytes within the 128-byte swizzle rows); those past the last
                    // data column hold zeros on both sides: skipped
                    const int ks = min(4, (a.D - 32 * c + 7) >> 3);
                    if (c == 0 && !ta_wait(a, s, &s.acce[iss], aph, kDevTimeoutMma)) { ok = false; break; }
                    ptx::tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        if (kk >= ks) break;
                        const uint64_t ch = base + 2 * kk;
                        const uint32_t ahi = tmem + (uint32_t)(c * 32 + kk * 8);
                        ptx::mma_tf32_ts(d_tmem, ahi, ch, kIdesc, (c | kk) != 0);
                        if (clo) ptx::mma_tf32_ts(d_tmem, ahi, ch + (kBox >> 4), kIdesc, 1u);
                        if (alo) ptx::mma_tf32_ts(d_tmem, ahi + (uint32_t)a.dp, ch, kIdesc, 1u);
                    }
                    // the tile's last chunk: accumulator-ready first (the epilogue waits on it)
                    if (c == nch - 1) ptx::mma_commit(&s.accf[iss]);
                    ptx::mma_commit(&s.empty[st]);
                    if (++st == (iss + 1) * half) {
                        st = iss * half;
                        ph ^= 1u;
                    }
                }
            }
            // all MMAs issued by this thread retire before TMEM is released
            ptx::mma_commit(s.drain);
            ptx::mbar_wait(s.drain, 0, kTimeout);
        }
    } else if (warp < 2 + kEpi) {
        // ------------------------------------------------------------ epilogue
        const int ew = warp - 2;
        const int quad = warp & 3;  // TMEM lane quarter this warp may access
        const int part = ew >> 2;   // columns [32 part, 32 part + 32) of every tile
        const int row = quad * 32 + lane;
        const int64_t q = q0 + row;
        const bool valid = q < a.Q;
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        if (part == 0) {
            // A operand: this lane's query as TF32 hi / lo parts into TMEM
            const float* qrow = a.queries + (valid ? q : 0) * a.ldq;
            uint32_t any_lo = 0;
            for (int c = 0; c < nch; ++c) {
                float hi[32], lo[32];
#pragma unroll
                for (int u = 0; u < 32; ++u) {
                    const int d = c * 32 + u;
                    const float x = (valid && d < a.D) ? __ldg(qrow + d) : 0.f;
                    hi[u] = tf32_round(x);
                    lo[u] = tf32_round(__fsub_rn(x, hi[u]));
                    any_lo |= (lo[u] != 0.f) ? 1u : 0u;
                }
                __syncwarp();
                ptx::tmem_st32(tmem + lane_base + (uint32_t)(c * 32), hi);
                ptx::tmem_st32(tmem + lane_base + (uint32_t)(a.dp + c * 32), lo);
            }
            ptx::tmem_wait_st();
            if (__any_sync(0xffffffffu, any_lo != 0u) && lane == 0) atomicOr(s.alo, 1u);
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(s.aready);
        }
        const float T = valid ? (a.thr ? __ldg(a.thr + q) : __int_as_float(0x7f800000)) : -__int_as_float(0x7f800000);
        const size_t seg = (size_t)split * kParts + part;
        uint64_t* out = kDense ? nullptr : a.cand + (seg * (size_t)a.Q + (size_t)(valid ? q : 0)) * (size_t)a.cap;
        // dense: this warp's rows
        float* krow = kDense ? a.keys + (q0 + quad * 32) * a.ldk : nullptr;
        const int krows = (int)min((int64_t)32, a.Q - (q0 + quad * 32));
        uint32_t cnt = 0;
        const uint32_t cap = (uint32_t)a.cap;
        const uint32_t accf = ptx::smem_u32(s.accf), acce = ptx::smem_u32(s.acce);
        const uint32_t nfull = ptx::smem_u32(s.nfull), nempty = ptx::smem_u32(s.nempty);
        const uint32_t c0 = 32u * (uint32_t)part, tb = tmem + kAccColTA + lane_base + c0;
        uint32_t b = 0, ph = 0, ns = 0, nph = 0, nb = (uint32_t)n_begin + c0;
        for (int t = 0; t < ntiles; ++t, nb += kTN) {
            // warp-uniform outcome: tcgen05.ld below is warp-collective
            bool ok = ptx::mbar_try_wait(accf + 8u * b, ph) && ptx::mbar_try_wait(nfull + 8u * ns, nph);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = ta_wait(a, s, &s.accf[b], ph, kDevTimeoutEpilogue) && ta_wait(a, s, &s.nfull[ns], nph, kDevTimeoutEpilogue);
                if (!__all_sync(0xffffffffu, ok)) break;
            }
            ptx::tc_fence_after();
            float v[32];
            __syncwarp();
            ptx::tmem_ld32(tb + b * kTN, v);
            ptx::tmem_wait_ld_regs(v);
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(acce + 8u * b);
            if (++b == kAccTA) {
                b = 0;
                ph ^= 1u;
            }
            chunk_norm_keys<32>(v, s.norms + ns * kTN + c0);
            if constexpr (kDense) {
                chunk_store<32>(v, krow + nb, a.ldk, krows);
                release_norms(nempty + 8u * ns);
            } else {
                float g[4];
                chunk_minima<32>(v, g);
                const uint32_t hot = __ballot_sync(0xffffffffu, min_of(g) < T);
                release_norms(nempty + 8u * ns, hot, a.zero);
                if (hot) chunk_append<32>(v, g, T, nb, out, cap, cnt);
            }
            if (++ns == kNorm) {
                ns = 0;
                nph ^= 1u;
            }
        }
        if (!kDense && valid) a.cnt[seg * (size_t)a.Q + (size_t)q] = cnt;
    }

    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    if (warp == 1) {
        __syncwarp();
        ptx::tmem_dealloc(tmem, 512);
    }
}
}  // namespace

size_t tscan_smem_bytes(int ring, bool tmem_a)
{
    return (size_t)ring * (tmem_a ? kSlotTA : kSlot) + (size_t)kNorm * kTN * 4 + kCtrl;
}

int tscan_ring(bool tmem_a)
{
    int r = tmem_a ? kMaxRingTA : kMaxRing;
    while (r > 2 && tscan_smem_bytes(r, tmem_a) > kScanSmemLimit) --r;
    return r;
}

cudaError_t launch_tscan(const TscanArgs& a, int splits, cudaStream_t st)
{
    const bool ta = a.tmem_a != 0;
    if (a.dp < 32 || a.dp % 32 != 0 || a.split_len % kTN != 0 || (!a.keys && a.cap < 1) || splits < 1 || a.split0 < 0 ||
        a.ring < 2 || a.ring > (ta ? kMaxRingTA : kMaxRing) || (ta && (a.dp > 128 || !a.queries || a.D > a.dp)))
        return cudaErrorInvalidValue;
    const size_t smem = tscan_smem_bytes(a.ring, ta);
    if (smem > kScanSmemLimit) return cudaErrorInvalidValue;
    if (a.Q <= 0) return cudaSuccess;
    auto* kernel = a.keys ? (ta ? tscan_ta_kernel<true> : tscan_kernel<true>)
                          : (ta ? tscan_ta_kernel<false> : tscan_kernel<false>);
    cudaError_t e = reserve_smem((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((a.Q + kTileQ - 1) / kTileQ), (unsigned)splits);
    kernel<<<grid, kThreads, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace knn
