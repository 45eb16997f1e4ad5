// scan_f16.cu -- tensor-core threshold scan for FP32 data of any width and shortlists of up to
// 512 entries, on keys from split FP16 operands.
//
// The exact form's distance stage for data that are not exact in BF16, for rows wider than 128
// and for k above 128: the reference's pdist_NT SGEMM (include/utils.h:957-985) followed by its
// selections (bitonic_shared, src/cuknnBitonic.cu:45-254, up to k = 512; the heap of
// src/cuknnHeap.cu:146-291 for large k), restructured as the BF16 threshold scan is
// (scan_bf16.cu): every key ||c||^2 - 2 q.c strictly below the query's seeded threshold is
// appended to the query's candidate segment, and the selection (select.cu) takes the shortlist from the
// segments and re-ranks it by exact distance.
//
// Keys: every row x is scaled by a power of two s that puts max |x| into [2^14, 2^15), then
// split as s x = hi + lo, hi = fp16(s x), lo = fp16(s x - hi): 11 + 11 significant bits, what the
// 3xTF32 split this replaces held (components 2^-17 and more below the row's largest keep
// 2^-39 of that largest), at half the bytes and on an MMA kind with twice TF32's rate.
// q.c = (qhi.chi + qhi.clo + qlo.chi) / (s_q s_c), the products exact in FP32 and accumulated in
// FP32 by tcgen05.mma.kind::f16; the epilogue multiplies the row's 1 / s_c (exact) and adds the
// norm in one fma with -2 / s_q.  A correction product whose low part is zero for the whole
// corpus tile (or query tile) is skipped -- it would add exact zeros.
//
// Both kernels are bound by the tensor pipe (3 x 2 N Q D FLOPs).  Main pass against the 3xTF32 one
// (same box): 1,000,003 x 96, 2,000 queries 726 us against 1,356 (1,620 TFLOP/s executed, at the card's
// power limit); 65,536 x 128, 1,024 queries 39 against 74; 32,768 x 1,024, 256 queries 48 against 92.  Key error against
// FP64 relative to ||c||^2 + ||q||^2, rms: uniform D = 128 6.4e-7 against 9.8e-7, D = 1,024 5.9e-6
// against 8.2e-6, Gaussian D = 96 1.1e-7 against 1.8e-7, mixture D = 96 2.9e-7 against 4.6e-7.
//
// Warp roles (640 threads):
//   warp 0      producer: per tile and K chunk of 64 columns (one 128-byte swizzle row) the
//               corpus boxes (2-D TMA), low parts only where present;
//   warps 1, 18 MMA issuers;
//   warps 2..17 epilogue: thread = query (TMEM lane); warp 2 + 4p + j reads part p of the tile's
//               columns in lane quarter j, releases the accumulator, forms the keys, appends
//               those below the threshold (dense passes: stores every key in the query's row);
//   warp 19     per tile the norms and row scales: bulk copies, or a gather for a strided view.
// Every mbarrier wait is bounded; on timeout the kernel records an error code in the device
// error word and winds down without hanging the GPU.
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
constexpr int kParts = kScanParts;           // epilogue column parts
constexpr int kEpi = 4 * kParts;             // epilogue warps
constexpr int kIss = 2;                      // MMA issuing warps
constexpr int kThreads = 32 * (2 + kIss + kEpi);
constexpr int kCols = 64;                    // FP16 columns per K chunk (128-byte swizzle rows)
constexpr uint32_t kBox = 128u * 128u;       // one operand box: 128 rows x 64 FP16
constexpr uint32_t kCtrl = 512;
constexpr uint64_t kTimeout = 4000000000ull;

struct FSmem {
    unsigned char* ring;
    float* norms;       // [slots][tile rows] norms, then as many row scales
    uint64_t* full;
    uint64_t* empty;
    uint64_t* accf;
    uint64_t* acce;
    uint64_t* nfull;
    uint64_t* nempty;
    uint64_t* aready;
    uint64_t* drain;
    uint32_t* tmem_holder;
    volatile int* abort;
    uint32_t* alo;               // 1 when some query of the tile has a low part
    volatile uint32_t* slot_lo;  // per ring slot: bit 0 corpus low part loaded, bit 1 query low part
};

__device__ __forceinline__ bool f_wait(const FscanArgs& a, const FSmem& s, uint64_t* bar, uint32_t parity, int code)
{
    if (ptx::mbar_try_wait(bar, parity)) return true;
    if (*s.abort) return false;
    if (ptx::mbar_wait(bar, parity, kTimeout)) return true;
    atomicCAS(a.err, 0, code);
    *s.abort = 1;
    return false;
}

// K steps of 16 columns that hold data in chunk c of rows of D columns (the rest are zeros)
__device__ __forceinline__ int chunk_steps(int D, int c) { return min(4, (D - c * kCols + 15) >> 4); }

// The norm warp: norms and row scales of every tile into their ring (kSlots tiles of kRows, the
// scales after all norms), +inf and 0 past the view.  Views of the whole corpus are contiguous and
// padded at least one tile past their end; strided ones (the seeding samples) are gathered.
template <int kRows, int kSlots>
__device__ __forceinline__ void load_norms(const FscanArgs& a, const FSmem& s, int64_t n_begin, int ntiles)
{
    const int lane = threadIdx.x & 31;
    for (int t = 0; t < ntiles; ++t) {
        const int ns = t % kSlots;
        const int64_t n0 = n_begin + (int64_t)t * kRows;
        const bool ok = f_wait(a, s, &s.nempty[ns], ((uint32_t)(t / kSlots) & 1u) ^ 1u, kDevTimeoutProducer);
        if (!__all_sync(0xffffffffu, ok)) return;
        float* nrm = s.norms + ns * kRows;
        float* scl = s.norms + (kSlots + ns) * kRows;
        if (a.stride == 1) {
            if (lane == 0) {
                ptx::mbar_arrive_expect_tx(&s.nfull[ns], 2u * kRows * 4u);
                ptx::bulk_load(nrm, a.cn + n0, kRows * 4u, &s.nfull[ns]);
                ptx::bulk_load(scl, a.cs + n0, kRows * 4u, &s.nfull[ns]);
            }
        } else {
#pragma unroll
            for (int i = lane; i < kRows; i += 32) {
                const bool in = n0 + i < a.N;
                nrm[i] = in ? __ldg(a.cn + (n0 + i) * a.stride) : __int_as_float(0x7f800000);
                scl[i] = in ? __ldg(a.cs + (n0 + i) * a.stride) : 0.f;
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s.nfull[ns]);
        }
    }
}

// ---------------------------------------------------------------- queries in tensor memory
// Rows of at most 256 columns.  The query tile's hi and lo parts sit in tensor memory (A from
// TMEM, two FP16 per column: hi [0, 32 nch), lo [32 nch, 64 nch)), so the ring carries only corpus
// chunks (hi and lo, 2 x 16 KB a slot) and each MMA reads one operand from shared memory: with
// both there, MMA reads and TMA fills together exceed its bandwidth.  Tile 128 queries x 128
// corpus rows; three 128-column accumulators at 128, 256, 384 for up to 128 columns, two at 256,
// 384 above.  Two MMA issuers take the even and the odd tiles (the tensor pipe queues little work
// beyond the MMA being issued, so one thread's barrier waits and commits idle it), each with its
// own half of the ring: a slot's uses all belong to one issuer, which waits for each of them in
// order, so no wait can take an older phase of a slot's barrier for a newer one.
constexpr int kTN = 128;
constexpr int kRingHalf = 3;
constexpr int kRingTA = 2 * kRingHalf;
constexpr int kMaxAcc = 3;
constexpr int kNorm = 8;                     // tiles of corpus norms and scales in flight
constexpr uint32_t kSlotTA = 2u * kBox;      // corpus hi, corpus lo

template <bool kDense>
__global__ void __launch_bounds__(kThreads, 1) fscan_ta_kernel(const __grid_constant__ FscanArgs a)
{
    constexpr uint32_t kIdesc = ptx::idesc_f16(kTileQ, kTN);
    extern __shared__ __align__(1024) unsigned char sm[];
    // device-side path choice: the kernel runs only when *run_if != 0
    if (a.run_if != nullptr && *a.run_if == 0u) return;
    if ((ptx::smem_u32(sm) & 1023u) != 0u) {
        if (threadIdx.x == 0) atomicCAS(a.err, 0, kDevMisaligned);
        return;
    }
    FSmem s;
    s.ring = sm;
    s.norms = reinterpret_cast<float*>(sm + (size_t)kRingTA * kSlotTA);
    uint64_t* bars = reinterpret_cast<uint64_t*>(s.norms + 2 * kNorm * kTN);
    s.full = bars;
    s.empty = s.full + kRingTA;
    s.accf = s.empty + kRingTA;
    s.acce = s.accf + kMaxAcc;
    s.nfull = s.acce + kMaxAcc;
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
    const int nch = (a.D + kCols - 1) / kCols;
    const int nacc = nch <= 2 ? 3 : 2;
    const uint32_t acc_col = nch <= 2 ? 128u : 256u;

    if (tid == 0) {
        for (int i = 0; i < kRingTA; ++i) {
            ptx::mbar_init(&s.full[i], 1);
            ptx::mbar_init(&s.empty[i], 1);
        }
        for (int b = 0; b < kMaxAcc; ++b) {
            ptx::mbar_init(&s.accf[b], 1);
            ptx::mbar_init(&s.acce[b], kEpi);
        }
        for (int b = 0; b < kNorm; ++b) {
            ptx::mbar_init(&s.nfull[b], 1);
            ptx::mbar_init(&s.nempty[b], kEpi);
        }
        ptx::mbar_init(s.aready, kEpi);
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
            int it[2] = {0, 0};  // chunks loaded into each issuer's half of the ring
            bool ok = true;
            for (int t = 0; t < ntiles && ok; ++t) {
                const int64_t n0 = n_begin + (int64_t)t * kTN;
                const uint32_t clo = a.clo_flags ? __ldg(a.clo_flags + n0 / kTN) : 1u;
                const int h = t & 1;
                int i = h ? it[1] : it[0];
                for (int c = 0; c < nch; ++c, ++i) {
                    const int st = h * kRingHalf + i % kRingHalf;
                    const uint32_t ph = (uint32_t)(i / kRingHalf) & 1u;
                    if (!f_wait(a, s, &s.empty[st], ph ^ 1u, kDevTimeoutProducer)) { ok = false; break; }
                    unsigned char* dst = s.ring + (size_t)st * kSlotTA;
                    s.slot_lo[st] = clo;  // published by the arrive below
                    ptx::mbar_arrive_expect_tx(&s.full[st], kBox * (clo ? 2u : 1u));
                    ptx::tma_load_2d(dst, &a.tm_chi, &s.full[st], c * kCols, (int)n0);
                    if (clo) ptx::tma_load_2d(dst + kBox, &a.tm_clo, &s.full[st], c * kCols, (int)n0);
                }
                if (h) it[1] = i;
                else it[0] = i;
            }
            if (!ok) {
                // let copies already issued land before the CTA winds down
                for (int h = 0; h < 2; ++h) {
                    const int n = h ? it[1] : it[0];
                    for (int j = max(0, n - kRingHalf); j < n; ++j)
                        ptx::mbar_wait(&s.full[h * kRingHalf + j % kRingHalf], (uint32_t)(j / kRingHalf) & 1u, kTimeout);
                }
            }
        }
    } else if (warp == 3 + kEpi) {
        load_norms<kTN, kNorm>(a, s, n_begin, ntiles);
    } else if (warp == 1 || warp == 2 + kEpi) {
        // ------------------------------------------------------------ MMA issuers
        if (lane == 0) {
            const int iss = warp == 1 ? 0 : 1;
            bool ok = f_wait(a, s, s.aready, 0, kDevTimeoutAload);
            ptx::tc_fence_after();
            const uint32_t alo = *s.alo;
            const uint32_t lo_col = 32u * (uint32_t)nch;
            // Little may stand between an accumulator's release and the tile's first MMA: slots, phases
            // and accumulators advance by additions, and the tile's first chunk (a slot of the issuer's
            // own, long full) is looked at before the accumulator (with divisions by the number of
            // accumulators here and in the epilogue the pass over 1,000,003 x 96 with 2,000 queries took
            // 760 us, 726 so, at the card's power limit).
            const uint64_t ring_desc = ptx::desc_sw128_kmajor(ptx::smem_u32(s.ring));  // (in 16-byte units)
            int st = iss * kRingHalf;
            uint32_t ph = 0, b = (uint32_t)iss, aph = 1;  // (accumulators start free)
            for (int t = iss; t < ntiles && ok; t += kIss) {
                const uint32_t d_tmem = tmem + acc_col + b * kTN;
                for (int c = 0; c < nch; ++c) {
                    if (!f_wait(a, s, &s.full[st], ph, kDevTimeoutMma)) { ok = false; break; }
                    const uint32_t clo = s.slot_lo[st];
                    const uint64_t base = ring_desc + (uint64_t)((uint32_t)st * kSlotTA >> 4);
                    const int ks = chunk_steps(a.D, c);
                    if (c == 0 && !f_wait(a, s, &s.acce[b], aph, kDevTimeoutMma)) { ok = false; break; }
                    ptx::tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        if (kk >= ks) break;
                        // K steps of 16 FP16 (32 bytes, 8 TMEM columns)
                        const uint64_t ch = base + 2 * kk;
                        const uint32_t ahi = tmem + (uint32_t)(c * 32 + kk * 8);
                        ptx::mma_f16_ts(d_tmem, ahi, ch, kIdesc, (c | kk) != 0);
                        if (clo) ptx::mma_f16_ts(d_tmem, ahi, ch + (kBox >> 4), kIdesc, 1u);
                        if (alo) ptx::mma_f16_ts(d_tmem, ahi + lo_col, ch, kIdesc, 1u);
                    }
                    // the tile's last chunk: accumulator-ready first (the epilogue waits on it)
                    if (c == nch - 1) ptx::mma_commit(&s.accf[b]);
                    ptx::mma_commit(&s.empty[st]);
                    if (++st == (iss + 1) * kRingHalf) {
                        st = iss * kRingHalf;
                        ph ^= 1u;
                    }
                }
                if ((b += kIss) >= (uint32_t)nacc) {
                    b -= (uint32_t)nacc;
                    aph ^= 1u;
                }
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
        {
            // A operand: this lane's query, hi then lo chunks of 64 columns (32 TMEM columns each),
            // dealt over the four parts' warps; columns past the row are zeros
            uint32_t any_lo = 0;
            for (int j = part; j < 2 * nch; j += kParts) {
                const int c = j >= nch ? j - nch : j;
                const uint4* src = reinterpret_cast<const uint4*>(
                    (j >= nch ? a.qlo : a.qhi) + (valid ? q : 0) * (int64_t)a.hp + c * kCols);
                float v[32];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    uint4 w = make_uint4(0u, 0u, 0u, 0u);
                    if (valid && c * kCols + 8 * u < a.hp) w = __ldg(src + u);
                    v[4 * u] = __uint_as_float(w.x);
                    v[4 * u + 1] = __uint_as_float(w.y);
                    v[4 * u + 2] = __uint_as_float(w.z);
                    v[4 * u + 3] = __uint_as_float(w.w);
                    if (j >= nch) any_lo |= (w.x | w.y | w.z | w.w) & 0x7fff7fffu;
                }
                __syncwarp();
                ptx::tmem_st32(tmem + lane_base + (uint32_t)(j * 32), v);
            }
            ptx::tmem_wait_st();
            if (__any_sync(0xffffffffu, any_lo != 0u) && lane == 0) atomicOr(s.alo, 1u);
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(s.aready);
        }
        const float T = valid ? (a.thr ? __ldg(a.thr + q) : __int_as_float(0x7f800000)) : -__int_as_float(0x7f800000);
        const float m = valid ? -2.0f * __ldg(a.qs + q) : 0.f;
        const size_t seg = (size_t)split * kParts + part;
        uint64_t* out = kDense ? nullptr : a.cand + (seg * (size_t)a.Q + (size_t)(valid ? q : 0)) * (size_t)a.cap;
        // dense: this warp's rows
        float* krow = kDense ? a.keys + (q0 + quad * 32) * a.ldk : nullptr;
        const int krows = (int)min((int64_t)32, a.Q - (q0 + quad * 32));
        uint32_t cnt = 0;
        const uint32_t cap = (uint32_t)a.cap;
        // Every warp takes every tile: barrier addresses, phases and the tile's row stay in registers,
        // and one vote decides whether the tile holds anything to append.
        const uint32_t accf = ptx::smem_u32(s.accf), acce = ptx::smem_u32(s.acce);
        const uint32_t nfull = ptx::smem_u32(s.nfull), nempty = ptx::smem_u32(s.nempty);
        const uint32_t c0 = 32u * (uint32_t)part, tb = tmem + acc_col + lane_base + c0;
        uint32_t b = 0, ph = 0, ns = 0, nph = 0, nb = (uint32_t)n_begin + c0;
        for (int t = 0; t < ntiles; ++t, nb += kTN) {
            // warp-uniform outcome: tcgen05.ld below is warp-collective
            bool ok = ptx::mbar_try_wait(accf + 8u * b, ph) && ptx::mbar_try_wait(nfull + 8u * ns, nph);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = f_wait(a, s, &s.accf[b], ph, kDevTimeoutEpilogue) && f_wait(a, s, &s.nfull[ns], nph, kDevTimeoutEpilogue);
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
            if (++b == (uint32_t)nacc) {
                b = 0;
                ph ^= 1u;
            }
            const float* nrm = s.norms + ns * kTN + c0;
            chunk_scaled_keys<32>(v, nrm, nrm + kNorm * kTN, m);
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

// ---------------------------------------------------------------- both operands in shared memory
// Rows wider than 256 columns: tensor memory cannot hold the queries beside the accumulators, so
// a ring slot carries one K chunk of the query tile and of the corpus tile, hi and lo parts.  Tile
// 128 queries x 256 corpus rows (two accumulators of 256 columns): a chunk's 12 MMAs of 128 cycles
// read 12 KB and its slot fills 96 KB, 160 bytes of shared memory per MMA cycle against 217 for
// 128-row tiles.  One issuer takes every tile in order (slots are refilled within a tile); its
// waits hide behind the 128-cycle MMAs already issued.
// Dense passes whose tiles would leave more than half of the SMs idle take tiles of 128 rows (256 queries on
// 8,192 of 32,768 x 1,024 rows: 64 CTAs of one tile 24 us, 128 CTAs 16).
constexpr int kWN = 256;
constexpr int kWNarrow = 128;
constexpr int kRingW = 2;                    // tiles of 256 rows; 3 of 128
constexpr int kMaxRingW = 3;
constexpr int kAccW = 2;
constexpr int kNormW = 4;
// query hi, query lo, corpus hi (2 boxes, or 1), corpus lo
constexpr uint32_t slot_w(int rows) { return (2u + 2u * (uint32_t)(rows / 128)) * kBox; }

// Append of a chunk by the mask of its 8-column groups that hold a key below T: the two chunks of a
// 256-row tile leave no registers for the groups' minima (47 us a pass over 32,768 x 1,024 with 256
// queries; 51 and 49 with them, spilled).
// Words hold the raw key bits above the index; the selection maps them to
// ordered keys.  A lane whose group holds a single key below T (the usual case
// where a warp appends at all) stores the group's minimum at the key's position
// found from the mask of hits; more hits take the column walk.
template <int W>
__device__ __forceinline__ void masked_append(const float (&key)[W], uint32_t gm, float T, uint32_t base,
                                             uint64_t* out, uint32_t cap, uint32_t& cnt)
{
    constexpr int G = 8;
#pragma unroll
    for (int g = 0; g < W / G; ++g) {
        if ((gm >> g) & 1u) {
            const float* kg = key + G * g;
            uint32_t hm = 0;
#pragma unroll
            for (int j = 0; j < G; ++j) hm |= (kg[j] < T ? 1u : 0u) << j;
            if ((hm & (hm - 1u)) == 0u) {
                const float k = min8(kg);
                if (cnt < cap)
                    out[cnt] = ((uint64_t)__float_as_uint(k) << 32) |
                               (uint64_t)(base + (uint32_t)(G * g + __ffs((int)hm) - 1));
                ++cnt;
            } else {
#pragma unroll
                for (int j = 0; j < G; ++j) {
                    const float k = kg[j];
                    const bool h = k < T;
                    if (h && cnt < cap)
                        out[cnt] = ((uint64_t)__float_as_uint(k) << 32) | (uint64_t)(base + (uint32_t)(G * g + j));
                    cnt += h ? 1u : 0u;
                }
            }
        }
    }
}
template <int W>
__device__ __forceinline__ uint32_t masked_keys(float (&v)[W], const float* nrm, const float* scl, float m, float T)
{
    chunk_scaled_keys<W>(v, nrm, scl, m);
    uint32_t gm = 0;
#pragma unroll
    for (int g = 0; g < W / 8; ++g) gm |= (min8(v + 8 * g) < T ? 1u : 0u) << g;
    return gm;
}

template <bool kDense, int kW>
__global__ void __launch_bounds__(kThreads, 1) fscan_wide_kernel(const __grid_constant__ FscanArgs a)
{
    constexpr uint32_t kIdesc = ptx::idesc_f16(kTileQ, kW);
    constexpr int kBoxes = kW / 128;         // 128-row boxes of a corpus operand
    constexpr int kRing = kW == kWN ? kRingW : kMaxRingW;
    constexpr uint32_t kSlotW = slot_w(kW);
    constexpr int kPart = kW / kParts;       // columns of a tile an epilogue warp takes
    extern __shared__ __align__(1024) unsigned char sm[];
    if (a.run_if != nullptr && *a.run_if == 0u) return;
    if ((ptx::smem_u32(sm) & 1023u) != 0u) {
        if (threadIdx.x == 0) atomicCAS(a.err, 0, kDevMisaligned);
        return;
    }
    FSmem s;
    s.ring = sm;
    s.norms = reinterpret_cast<float*>(sm + (size_t)kRing * kSlotW);
    uint64_t* bars = reinterpret_cast<uint64_t*>(s.norms + 2 * kNormW * kW);
    s.full = bars;
    s.empty = s.full + kRing;
    s.accf = s.empty + kRing;
    s.acce = s.accf + kAccW;
    s.nfull = s.acce + kAccW;
    s.nempty = s.nfull + kNormW;
    s.drain = s.nempty + kNormW;
    s.aready = s.drain;
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
    const int ntiles = n_end > n_begin ? (int)((n_end - n_begin + kW - 1) / kW) : 0;
    const int nch = (a.D + kCols - 1) / kCols;

    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) {
            ptx::mbar_init(&s.full[i], 1);
            ptx::mbar_init(&s.empty[i], 1);
        }
        for (int b = 0; b < kAccW; ++b) {
            ptx::mbar_init(&s.accf[b], 1);
            ptx::mbar_init(&s.acce[b], kEpi);
        }
        for (int b = 0; b < kNormW; ++b) {
            ptx::mbar_init(&s.nfull[b], 1);
            ptx::mbar_init(&s.nempty[b], kEpi);
        }
        ptx::mbar_init(s.drain, 1);
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
                const int64_t n0 = n_begin + (int64_t)t * kW;
                // flags of the tile's 128-row boxes (allocated past the last row's tile)
                const uint32_t clo =
                    a.clo_flags ? __ldg(a.clo_flags + n0 / 128) | __ldg(a.clo_flags + n0 / 128 + kBoxes - 1) : 1u;
                for (int c = 0; c < nch; ++c, ++it) {
                    const int st = it % kRing;
                    const uint32_t ph = (uint32_t)(it / kRing) & 1u;
                    if (!f_wait(a, s, &s.empty[st], ph ^ 1u, kDevTimeoutProducer)) { ok = false; break; }
                    unsigned char* dst = s.ring + (size_t)st * kSlotW;
                    s.slot_lo[st] = (clo ? 1u : 0u) | (qlo ? 2u : 0u);  // published by the arrive below
                    ptx::mbar_arrive_expect_tx(&s.full[st], kBox * (1u + kBoxes + (qlo ? 1u : 0u) + (clo ? (uint32_t)kBoxes : 0u)));
                    ptx::tma_load_2d(dst, &a.tm_qhi, &s.full[st], c * kCols, (int)q0);
                    ptx::tma_load_2d(dst + 2 * kBox, &a.tm_chi, &s.full[st], c * kCols, (int)n0);
                    if (qlo) ptx::tma_load_2d(dst + kBox, &a.tm_qlo, &s.full[st], c * kCols, (int)q0);
                    if (clo) ptx::tma_load_2d(dst + (2 + kBoxes) * kBox, &a.tm_clo, &s.full[st], c * kCols, (int)n0);
                }
            }
            if (!ok) {
                // let copies already issued land before the CTA winds down
                for (int j = max(0, it - kRing); j < it; ++j)
                    ptx::mbar_wait(&s.full[j % kRing], (uint32_t)(j / kRing) & 1u, kTimeout);
            }
        }
    } else if (warp == 3 + kEpi) {
        load_norms<kW, kNormW>(a, s, n_begin, ntiles);
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            bool ok = true;
            int it = 0;
            for (int t = 0; t < ntiles && ok; ++t) {
                const int b = t % kAccW;
                const uint32_t use = (uint32_t)(t / kAccW);
                if (!f_wait(a, s, &s.acce[b], (use & 1u) ^ 1u, kDevTimeoutMma)) { ok = false; break; }
                ptx::tc_fence_after();
                const uint32_t d_tmem = tmem + (uint32_t)b * kW;
                for (int c = 0; c < nch; ++c, ++it) {
                    const int st = it % kRing;
                    if (!f_wait(a, s, &s.full[st], (uint32_t)(it / kRing) & 1u, kDevTimeoutMma)) { ok = false; break; }
                    ptx::tc_fence_after();
                    const uint32_t lo = s.slot_lo[st];
                    const uint32_t base = ptx::smem_u32(s.ring + (size_t)st * kSlotW);
                    const int ks = chunk_steps(a.D, c);
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        if (kk >= ks) break;
                        const uint64_t qh = ptx::desc_sw128_kmajor(base + kk * 32);
                        const uint64_t ch = ptx::desc_sw128_kmajor(base + 2 * kBox + kk * 32);
                        ptx::mma_f16_ss(d_tmem, qh, ch, kIdesc, (c | kk) != 0);
                        if (lo & 1u) ptx::mma_f16_ss(d_tmem, qh, ptx::desc_sw128_kmajor(base + (2 + kBoxes) * kBox + kk * 32), kIdesc, 1u);
                        if (lo & 2u) ptx::mma_f16_ss(d_tmem, ptx::desc_sw128_kmajor(base + kBox + kk * 32), ch, kIdesc, 1u);
                    }
                    if (c == nch - 1) ptx::mma_commit(&s.accf[b]);
                    ptx::mma_commit(&s.empty[st]);
                }
                if (!ok) break;
            }
            // all MMAs issued by this thread retire before TMEM is released
            ptx::mma_commit(s.drain);
            ptx::mbar_wait(s.drain, 0, kTimeout);
        }
    } else if (warp < 2 + kEpi) {
        // ------------------------------------------------------------ epilogue
        const int ew = warp - 2;
        const int quad = warp & 3;
        const int part = ew >> 2;   // columns [kPart part, kPart part + kPart) of every tile
        const int row = quad * 32 + lane;
        const int64_t q = q0 + row;
        const bool valid = q < a.Q;
        const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
        const float T = valid ? (a.thr ? __ldg(a.thr + q) : __int_as_float(0x7f800000)) : -__int_as_float(0x7f800000);
        const float m = valid ? -2.0f * __ldg(a.qs + q) : 0.f;
        const size_t seg = (size_t)split * kParts + part;
        uint64_t* out = kDense ? nullptr : a.cand + (seg * (size_t)a.Q + (size_t)(valid ? q : 0)) * (size_t)a.cap;
        // dense: this warp's rows
        float* krow = kDense ? a.keys + (q0 + quad * 32) * a.ldk : nullptr;
        const int krows = (int)min((int64_t)32, a.Q - (q0 + quad * 32));
        uint32_t cnt = 0;
        const uint32_t cap = (uint32_t)a.cap;
        for (int t = 0; t < ntiles; ++t) {
            const int b = t % kAccW;
            const uint32_t use = (uint32_t)(t / kAccW);
            const int ns = t % kNormW;
            const bool ok = f_wait(a, s, &s.accf[b], use & 1u, kDevTimeoutEpilogue) &&
                            f_wait(a, s, &s.nfull[ns], (uint32_t)(t / kNormW) & 1u, kDevTimeoutEpilogue);
            if (!__all_sync(0xffffffffu, ok)) break;
            ptx::tc_fence_after();
            const uint32_t tb = tmem + (uint32_t)b * kW + lane_base + (uint32_t)(kPart * part);
            float v[32], w[32];
            __syncwarp();
            ptx::tmem_ld32(tb, v);
            if constexpr (kPart == 64) ptx::tmem_ld32(tb + 32, w);
            ptx::tmem_wait_ld_regs(v);
            if constexpr (kPart == 64) ptx::tie_regs(w);
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(&s.acce[b]);
            const float* nrm = s.norms + ns * kW + kPart * part;
            const uint32_t base = (uint32_t)(n_begin + (int64_t)t * kW) + (uint32_t)(kPart * part);
            const uint32_t g = masked_keys<32>(v, nrm, nrm + kNormW * kW, m, T);
            if constexpr (kDense) {
                chunk_store<32>(v, krow + n_begin + (int64_t)t * kW + kPart * part, a.ldk, krows);
            } else if (__any_sync(0xffffffffu, g != 0u)) {
                masked_append<32>(v, g, T, base, out, cap, cnt);
            }
            if constexpr (kPart == 64) {
                const uint32_t h = masked_keys<32>(w, nrm + 32, nrm + kNormW * kW + 32, m, T);
                if constexpr (kDense) {
                    chunk_store<32>(w, krow + n_begin + (int64_t)t * kW + kPart * part + 32, a.ldk, krows);
                } else if (__any_sync(0xffffffffu, h != 0u)) {
                    masked_append<32>(w, h, T, base + 32u, out, cap, cnt);
                }
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

constexpr size_t kSmemTA = (size_t)kRingTA * kSlotTA + 2 * kNorm * kTN * 4 + kCtrl;
constexpr size_t smem_w(int rows)
{
    return (size_t)(rows == kWN ? kRingW : kMaxRingW) * slot_w(rows) + 2 * kNormW * rows * 4 + kCtrl;
}
static_assert(kSmemTA <= kScanSmemLimit && smem_w(kWN) <= kScanSmemLimit && smem_w(kWNarrow) <= kScanSmemLimit,
              "shared memory of the FP16-split scan");
}  // namespace

int fscan_tile_rows(int D) { return D <= kFscanTmemD ? kTN : kWN; }
int fscan_dense_rows(int D, int64_t Q, int64_t n, int sms)
{
    if (D <= kFscanTmemD) return kTN;
    return 2 * ((Q + kTileQ - 1) / kTileQ) * ((n + kWN - 1) / kWN) <= sms ? kWNarrow : kWN;
}
int fscan_part_cols(int D) { return fscan_tile_rows(D) / kParts; }
int fscan_ring(int D) { return D <= kFscanTmemD ? kRingTA : kRingW; }

cudaError_t launch_fscan(const FscanArgs& a, int splits, cudaStream_t st)
{
    const bool ta = a.D <= kFscanTmemD;
    const int tn = a.keys ? a.dense_rows : fscan_tile_rows(a.D);
    if (a.keys && (ta ? tn != kTN : tn != kWN && tn != kWNarrow)) return cudaErrorInvalidValue;
    if (a.D < 1 || a.hp < a.D || a.hp % 8 != 0 || a.split_len % tn != 0 || (!a.keys && a.cap < 1) || a.stride < 1 || splits < 1 || a.split0 < 0 ||
        !a.cn || !a.cs || !a.qs || (ta && (!a.qhi || !a.qlo)))
        return cudaErrorInvalidValue;
    if (a.Q <= 0) return cudaSuccess;
    const size_t smem = ta ? kSmemTA : smem_w(tn);
    auto* kernel = !a.keys ? (ta ? fscan_ta_kernel<false> : fscan_wide_kernel<false, kWN>)
                   : ta    ? fscan_ta_kernel<true>
                   : tn == kWN ? fscan_wide_kernel<true, kWN> : fscan_wide_kernel<true, kWNarrow>;
    cudaError_t e = reserve_smem((const void*)kernel, smem);
    if (e != cudaSuccess) return e;
    dim3 grid((unsigned)((a.Q + kTileQ - 1) / kTileQ), (unsigned)splits);
    kernel<<<grid, kThreads, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace knn
