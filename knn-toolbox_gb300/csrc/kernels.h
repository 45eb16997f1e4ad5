// kernels.h -- launchers of the engine's CUDA kernels (internal interface).
#pragma once

#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace knn {

constexpr int kSms = 152;  // SMs of the chip that fixed grids and query counts are for (Engine::sms: the device's)

// Tile geometry shared by host and device.
constexpr int kTileQ = 128;       // queries per CTA (tensor-core M, TMEM lanes)
constexpr int kTileN = 128;       // corpus rows per tile (tensor-core N)
constexpr int kChunkK = 32;       // fp32 elements per 128-byte swizzle row
constexpr int kMaxDpTC = 128;     // A hi + lo must fit next to two accumulators in TMEM
constexpr int kMaxKpTC = 128;     // shortlist entries per query held in shared memory
constexpr int kSimtTileN = 64;

// error codes written by kernels into the device error word
enum DeviceError : int {
    kDevOk = 0,
    kDevTimeoutProducer = 1,
    kDevTimeoutMma = 2,
    kDevTimeoutEpilogue = 3,
    kDevTimeoutAload = 4,
    kDevMisaligned = 5,
};

// Raises a kernel's dynamic shared memory limit on the current device to `bytes`.  It is never lowered: engines of
// other threads (a server's slots) launch the same kernels, and a search with a smaller size set the limit between
// another's setting it and its launch.
cudaError_t reserve_smem(const void* kernel, size_t bytes);

cudaError_t launch_norms(const float* x, int64_t n, int64_t ld, int D, float* out, int64_t n_pad,
                         cudaStream_t s);
constexpr int kTileRows = 128;
__host__ __device__ constexpr int split_pitch(int D) { return (D + 7) & ~7; }  // rows of whole 16-byte words
// TF32 hi/lo split into [n][dp] arrays; lo_flags[tile of 128 rows] = any lo != 0 (may be null);
// *any_lo (zeroed by the caller, may be null) becomes 1 when some tile has a low part.  When
// skip_unless is given and *skip_unless == 0 at run time, the kernel does nothing.
cudaError_t launch_split_tf32(const float* x, int64_t n, int64_t ld, int D, int dp, float* hi, float* lo,
                         uint32_t* lo_flags, uint32_t* any_lo, const uint32_t* skip_unless, cudaStream_t s);
// BF16 copy into [n][dpb] (out may be null: check only); *not_exact |= 1 when some element
// is not exactly representable in BF16.
cudaError_t launch_bf16(const float* x, int64_t n, int64_t ld, int D, int dpb, void* out, uint32_t* not_exact,
                        cudaStream_t s);

// One pass over a row-major matrix (prep_rows_kernel); every output is optional.
constexpr int kPrepMaxD = 2048;
constexpr int kNormParts = 16;
struct PrepJob {
    const float* x = nullptr;
    int64_t n = 0, ld = 0;
    int D = 0;
    // norms[0..n_pad): the float rounding of the double sum of squares in column order, +inf padding
    float* norms = nullptr;
    int64_t n_pad = 0;
    // BF16 side: copy [n][dpb]; *not_exact |= 1 when some element is not exactly representable;
    // int_stats (2 words, zeroed by the caller): [0] |= 1 when some value is not an integer, [1] =
    // max |x| as float bits; np: norm parts [n][kNormParts] BF16, (n1, n2, n3, 0, ...) with n1 + n2 +
    // n3 equal to the row's FP32 norm
    void* bf = nullptr;
    int dpb = 0;
    uint32_t* not_exact = nullptr;
    uint32_t* int_stats = nullptr;
    void* np = nullptr;
    // E4M3 copy [n][f8_bytes] (f8_bytes a multiple of 128, zero padded) with per-row absmax scales
    // (row = scale * codes; scales[n..n_pad) = 0)
    void* f8 = nullptr;
    int f8_bytes = 0;
    float* scales = nullptr;
    // FP16 side: hi = fp16(s x), lo = fp16(s x - hi), s the power of two that puts the row's largest
    // |x| into [2^14, 2^15); hi / lo are [n][split_pitch(D)] FP16, zero padded, rs[0..n_pad) the
    // reciprocals 1 / s (0 for n <= i < n_pad).  lo_flags[tile of 128 rows] (zeroed by the caller) becomes 1 when
    // some lo is nonzero
    void* hi = nullptr;
    void* lo = nullptr;
    float* rs = nullptr;
    uint32_t* lo_flags = nullptr;
    // adaptive: the BF16 or the FP16 side per batch of rows, by *not_exact (see prep_rows_kernel);
    // done: one byte per batch (prep_batches of them), 1 when the FP16 side was written.  catch_up:
    // the FP16 side of the batches whose done byte is 0, nothing else.
    uint8_t* done = nullptr;
    bool catch_up = false;
    const uint32_t* run_if = nullptr;  // the launch does nothing when *run_if == 0 at run time
};
int64_t prep_batches(int64_t n, int D);
// second: a job of the same kind and row width to share the launch with (its own launch otherwise)
cudaError_t launch_prep(const PrepJob& job, cudaStream_t s, const PrepJob* second = nullptr);
// norms of rows of any width
cudaError_t launch_row_norms(const float* x, int64_t n, int64_t ld, int D, float* norms, int64_t n_pad, cudaStream_t s);

// Fix-up launches: compacted rows (row r is query qmap[r], present while r < *qcount) in two groups
// that one 1-D grid covers, the first rows on enough corpus splits to fill the GPU, the rest (rare) on
// a few.  Blocks of rows past the count return at once.  thr: one word per row, all ones.
struct FixGroup {
    int64_t rows = 0, split_len = 0;
    int tiles = 0, splits = 0;  // query tiles, corpus splits
    uint64_t* part = nullptr;   // [splits][rows][kp]
};
struct FixGroups {
    FixGroup g[2];
    int blocks() const { return g[0].tiles * g[0].splits + g[1].tiles * g[1].splits; }
};

#ifdef __CUDACC__
struct FixBlock {
    FixGroup g;
    int tile, split;  // within the group
    int64_t row0;     // the group's first compacted row
};
__device__ __forceinline__ FixBlock fix_block(const FixGroups& f, int b)
{
    const int na = f.g[0].tiles * f.g[0].splits;
    const bool second = b >= na;
    const FixGroup g = second ? f.g[1] : f.g[0];
    const int i = second ? b - na : b;
    // a split's tiles after one another: later splits of a tile start from the thresholds that earlier ones have
    // published (216,570 x 4 rows of three values, 9,806 queries, all failing: fix-up 2.74 ms with a tile's splits
    // side by side, 1.93 so)
    return {g, i % g.tiles, i / g.tiles, second ? f.g[0].rows : 0};
}
#endif

// CUDA-core FP32 fused distance + shortlist.  qpb in {32, 128}.
size_t simt_smem_bytes(int qpb, int kp);
// tile_redo (optional): a CTA runs only when tile_redo[blockIdx.x] != 0.
// fix (optional, with qmap and qcount): a fix-up launch; Q, split_len, splits and part are the groups'.
cudaError_t launch_simt(const float* corpus, int64_t N, int64_t ldc, const float* cn,
                        const float* queries, int64_t Q, int64_t ldq, int D, int kp, int qpb,
                        int64_t split_len, int splits, uint64_t* part, uint32_t* thr_g, cudaStream_t s,
                        const uint32_t* tile_redo = nullptr, const int32_t* qmap = nullptr,
                        const uint32_t* qcount = nullptr, const FixGroups* fix = nullptr);

// Tensor-core 3xTF32 fused distance + shortlist (tcgen05, TMA, TMEM).
struct TcArgs {
    CUtensorMap tm_hi;        // corpus hi  [N][dp] fp32, box {32, 128}, 128B swizzle
    CUtensorMap tm_lo;        // corpus lo
    CUtensorMap tm_bf;        // corpus bf16 [N][dpb], box {64, 128}, 128B swizzle
    const float* cn;          // [>= roundup(N,128)] corpus norms, +inf padding
    const float* queries;     // [Q][ldq]
    int64_t Q;
    int64_t ldq;
    int64_t N;
    int64_t split_len;        // corpus rows per split, multiple of kTileN
    uint64_t* part;           // [splits][Q][kp]
    uint32_t* thr_g;          // [Q] shared per-query threshold (order-mapped key), or null
    const uint32_t* lo_flags; // [ceil(N/128)] 1 when the corpus tile has a nonzero TF32 low part, or null
    const uint32_t* corpus_any_lo;  // 1 when any corpus tile has a low part (null: assume so)
    const uint32_t* not_exact;      // 0 when corpus and queries are BF16-exact (null: TF32 path only)
    const uint32_t* tile_redo;      // optional: a CTA runs only when tile_redo[blockIdx.x] != 0
    // optional (qcount non-null): a fix-up launch of the groups in fix; Q, split_len and part are the
    // groups', thr_g rows are the compacted ones
    const int32_t* qmap;
    const uint32_t* qcount;
    FixGroups fix;
    float* dump;              // optional: raw dot tile of CTA (0,0), tile 0, [128][128]
    int* err;                 // device error word
    int D;
    int dp;                   // D rounded up to kChunkK
    int dpb;                  // D rounded up to 64 (BF16 boxes)
    int kp;
    int stages;
    uint64_t timeout_ns;      // bound of every barrier wait (0: 4 s)
    int test_stall;           // test hook: the producer issues no copy, so the waits run out
};
size_t tc_smem_bytes(int kp, int stages);
int tc_max_stages(int kp);
// Launches the BF16 (bf16 = true) or TF32 variant; each returns at once unless
// *a.not_exact selects it (BF16: inputs exact in BF16; TF32: otherwise).
cudaError_t launch_tc(const TcArgs& a, int splits, bool bf16, cudaStream_t s);

// Tensor-core BF16 threshold scan (csrc/scan_bf16.cu): 128 queries x 256-row
// corpus tiles; every key strictly below the query's threshold is appended to
// the query's segment cand[(split*kScanParts + part)][q][0..cap) (part = the
// tile's 64-column quarter; in increasing corpus index), as (raw float bits of
// the key) << 32 | index; cnt[(split*kScanParts + part)][q] = keys found (may
// exceed cap: overflow).
constexpr int kScanTileN = 256;
constexpr int kScanParts = 4;
constexpr int kScanMaxRing = 8;
constexpr size_t kScanSmemLimit = 232448;
// Row width of the scan's operands in 16-bit units (dpb below): D rounded up to
// 64 for BF16 keys; for E4M3 keys the row's bytes (D rounded up to 128) / 2,
// so both key types share one tile geometry per 128-byte K box.
struct ScanArgs {
    CUtensorMap tm_c;          // corpus [N][dpb] 16-bit units (view), box {64, scan_box_rows(dpb)}, 128B swizzle
    CUtensorMap tm_np;         // BF16 keys: norm parts of the view [N][kNormParts] BF16, box {16, tile rows},
                               // 32B swizzle (E4M3 keys: unused)
    const void* qbf;           // queries [Q][dpb] 16-bit units (BF16, or E4M3 bytes)
    const float* cn;           // fp8: [>= N + scan_tile_rows(dpb)] corpus norms of the view, +inf padding
    const float* cs;           // fp8: corpus row scales of the view (same padding, 0 there)
    const float* qs;           // fp8: query row scales [Q]
    const float* thr;          // [Q] thresholds (null: +inf, every key collected)
    const uint32_t* skip_if;   // optional: the kernel returns at once when *skip_if != 0
    uint64_t* cand;            // [splits*kScanParts][Q][cap]
    uint32_t* cnt;             // [splits*kScanParts][Q]
    float* keys;               // dense pass (else null): every key, to keys[q * ldk + row] (rows past the
    int64_t ldk;               // view: +inf); cand, cnt, cap, thr unused; ldk a multiple of the tile rows
    int* err;                  // device error word
    int64_t Q;
    int64_t N;
    int64_t split_len;         // multiple of scan_tile_rows(dpb)
    int cap;
    int dpb;                   // row width in 16-bit units, multiple of 64, <= 256
    int ksteps;                // MMA K steps holding data (32 bytes each): ceil(D / 16) BF16, ceil(D / 32) E4M3
    int bps;                   // K-boxes per ring slot (divides dpb/64)
    int ring;                  // ring slots
    int fp8;                   // keys from E4M3 operands with per-row scales
    int split0;                // first split of this launch (grid row y is split split0 + y)
    uint32_t zero;             // 0 (release_norms)
    int accs;                  // TMEM accumulators: 2 (tiles of 224 / 192 rows) or 4 (tiles of 96)
};
// corpus rows per tile (MMA N): with 2 accumulators 224 for dpb <= 128, 192 for dpb <= 256;
// with 4 accumulators 96
int scan_tile_rows(int dpb, int accs);
// rows of the corpus tensor map's box (one whole tile)
int scan_box_rows(int dpb, int accs);
// most columns of one tile that a single candidate segment (epilogue part) collects
int scan_part_cols(int dpb, int accs);
size_t scan_smem_bytes(int dpb, int bps, int ring, bool fp8, int accs);
// Ring geometry for dpb (want_bps = 0: automatic).  Returns 0 on success.
int scan_plan(int dpb, int want_bps, int* bps, int* ring, bool fp8, int accs);
cudaError_t launch_scan(const ScanArgs& a, int splits, cudaStream_t s);

// Tensor-core 3xTF32 threshold scan (csrc/scan_tf32.cu): 128 queries x 128-row corpus
// tiles, K in chunks of 32 FP32 columns, both operands from shared memory (any D, a
// multiple of 32 after padding); the candidate segments are those of the BF16 scan
// (kScanParts per split, 32 columns of every tile each).
struct TscanArgs {
    CUtensorMap tm_qhi, tm_qlo;   // queries hi / lo [Q][dp] fp32, box {32, 128}, 128B swizzle
    CUtensorMap tm_chi, tm_clo;   // corpus hi / lo view [N][dp] fp32, same boxes
    const float* cn;              // [>= N + 128] corpus norms of the view, +inf padding
    const float* thr;             // [Q] thresholds (null: +inf, every key collected)
    const uint32_t* qlo_flags;    // [query tiles] 1 when the tile has a nonzero low part (null: all)
    const uint32_t* clo_flags;    // [128-row tiles of the view] same for the corpus (null: all)
    uint64_t* cand;               // [splits*kScanParts][Q][cap]
    uint32_t* cnt;                // [splits*kScanParts][Q]
    float* keys;                  // dense pass, as ScanArgs
    int64_t ldk;
    int* err;                     // device error word
    int64_t Q;
    int64_t N;
    int64_t split_len;            // multiple of 128
    int cap;
    int dp;                       // D rounded up to 32
    int split0;                   // first split of this launch
    int ring;                     // ring slots (tscan_ring())
    const uint32_t* run_if;       // optional: the kernel returns at once when *run_if == 0
    // dp <= 128: the queries' TF32 hi / lo parts in tensor memory, split by the kernel from the
    // FP32 queries (tm_qhi, tm_qlo, qlo_flags unused); the ring carries corpus chunks only
    uint32_t zero;                // 0 (release_norms)
    int tmem_a;
    const float* queries;         // [Q][ldq] fp32 (tmem_a)
    int64_t ldq;
    int D;
};
size_t tscan_smem_bytes(int ring, bool tmem_a);
int tscan_ring(bool tmem_a);
cudaError_t launch_tscan(const TscanArgs& a, int splits, cudaStream_t s);

// Tensor-core FP16-split threshold scan (csrc/scan_f16.cu): 128 queries x fscan_tile_rows(D)-row
// corpus tiles, K in chunks of 64 FP16 columns; the candidate segments are those of the BF16 scan
// (kScanParts per split, fscan_part_cols(D) columns of every tile each).  Operands as launch_prep
// writes them (FP16 side).
constexpr int kFscanTmemD = 256;  // widest rows whose queries sit in tensor memory
struct FscanArgs {
    CUtensorMap tm_qhi, tm_qlo;   // D > kFscanTmemD: queries hi / lo [Q][hp] fp16, box {64, 128}, 128B swizzle
    CUtensorMap tm_chi, tm_clo;   // corpus hi / lo view [N][hp] fp16, box {64, tile rows}, 128B swizzle
    const uint16_t* qhi;          // queries hi / lo [Q][hp] fp16 (D <= kFscanTmemD)
    const uint16_t* qlo;
    const float* qs;              // [Q] query row scales
    const float* cn;              // corpus norms, every stride-th one the view's; stride 1: [>= N + tile
    const float* cs;              // rows] with +inf padding; row scales likewise, 0 padding
    int64_t stride;
    const float* thr;             // [Q] thresholds (null: +inf, every key collected)
    const uint32_t* qlo_flags;    // D > kFscanTmemD: [query tiles] 1 when the tile has a low part (null: all)
    const uint32_t* clo_flags;    // [128-row tiles of the view, + 1] same for the corpus (null: all)
    uint64_t* cand;               // [splits*kScanParts][Q][cap]
    uint32_t* cnt;                // [splits*kScanParts][Q]
    float* keys;                  // dense pass, as ScanArgs
    int64_t ldk;
    int* err;                     // device error word
    int64_t Q;
    int64_t N;
    int64_t split_len;            // multiple of the tile rows
    int cap;
    int D;
    int hp;                       // row pitch of the queries' copies
    int dense_rows;               // dense pass: corpus rows per tile (fscan_dense_rows)
    int split0;                   // first split of this launch
    uint32_t zero;                // 0 (release_norms)
    const uint32_t* run_if;       // optional: the kernel returns at once when *run_if == 0
};
int fscan_tile_rows(int D);
// tile rows of a dense pass over n rows
int fscan_dense_rows(int D, int64_t Q, int64_t n, int sms);
int fscan_part_cols(int D);
int fscan_ring(int D);
cudaError_t launch_fscan(const FscanArgs& a, int splits, cudaStream_t st);

// Merge of the per-split shortlists, optional exact re-rank, final top-k.
// Extra modes (all optional):
//  * thr_out: instead of results, write the order-mapped key of the merged
//    shortlist's entry thr_rank (1-based; all ones when missing) per query;
//  * redo_out / need: when the merged shortlist holds fewer than `need` real
//    entries, set redo_out[q / qtile] = 1 and write no result for q;
//  * redo_in: process only queries whose tile has redo_in[q / qtile] != 0.
//  * skip_if_zero: the kernel does nothing when *skip_if_zero == 0 (device-side path choice);
//  * qmap / qcount / fix: the rows of a fix-up launch: row r is query qmap[r], present when
//    r < *qcount; results go to that query's row.
struct SelectExtra {
    uint32_t* thr_out = nullptr;
    int thr_rank = 0;
    uint32_t* redo_out = nullptr;
    int need = 0;
    const uint32_t* redo_in = nullptr;
    int qtile = 128;
    const uint32_t* skip_if_zero = nullptr;
    const int32_t* qmap = nullptr;
    const uint32_t* qcount = nullptr;
    FixGroups fix;
};
size_t select_smem_bytes(int kp, int D, int rerank);
cudaError_t launch_select(const uint64_t* part, int splits, int64_t Q, int kp, int k,
                          const float* corpus, int64_t ldc, const float* queries, int64_t ldq,
                          int D, int rerank, const float* qn, float* out_dist, int32_t* out_idx,
                          float* out_idx_f, cudaStream_t s, const SelectExtra& ex = SelectExtra());

// Seeding from a dense pass's keys: thr_out[q] = the next float above the key of rank `rank`
// (1-based) of keys[q * ldk .. + n), n <= kDenseRows; +inf when fewer keys are finite.  *clear
// becomes 0 whatever the gates (skip_if / skip_if_zero as CandSelect) say.
constexpr int kDenseRows = 8192;
cudaError_t launch_dense_threshold(const float* keys, int64_t ldk, int n, int rank, int64_t Q, float* thr_out,
                                   uint32_t* clear, const uint32_t* skip_if, const uint32_t* skip_if_zero,
                                   cudaStream_t s);

// Small corpora, no thresholds: per query, the `need` smallest of n values and the k results.
//  * keys given: a dense pass's keys (row q at keys + q * ldk); the `need` smallest (key, index) pairs
//    are re-ranked by exact distance.  With fp32_keys (shapes whose keys are FP32 ones but for this path) a
//    shortlist that may miss one of the k nearest, the split keys' errors considered, is replaced by every row
//    that they do not rule out -- or, where fail_idx is given and those are most rows, the query gets no result but
//    a place there (count in *fail_cnt; fail_thr as CandSelect);
//  * keys null: the exact distances themselves, computed by the kernel (need = k).  Where squares leave the
//    float range: the kp smallest (key, index) pairs re-ranked as above, the keys in FP32 arithmetic, by the
//    kernel too (of a query that is not finite: only with fp32_keys).
// n <= kSmallRows.  Rows whose key is not below +inf are never results; missing results are (+inf, -1).
constexpr int kSmallRows = 16384;
struct SmallSelect {
    const float* keys = nullptr;
    int64_t ldk = 0;
    int n = 0, need = 0, k = 0, kp = 0;
    bool fp32_keys = false;
    const float* cn = nullptr;  // [n] row norms (optional)
    int32_t* fail_idx = nullptr;
    uint32_t* fail_cnt = nullptr;
    uint32_t* fail_thr = nullptr;
    int64_t Q = 0;
    const float* corpus = nullptr;
    int64_t ldc = 0;
    const float* queries = nullptr;
    int64_t ldq = 0;
    int D = 0;
    float* out_dist = nullptr;
    int32_t* out_idx = nullptr;
    float* out_idx_f = nullptr;
};
cudaError_t launch_select_small(const SmallSelect& c, cudaStream_t s);

// Selection over the threshold scan's candidate segments (one warp per query).
// The candidates of query q are the first min(cnt, cap) words of its nseg
// segments; total = sum of cnt (the number of keys below the threshold).
//  * thr_out (threshold mode): thr_out[q] = the next float above the key of
//    rank thr_rank (1-based) when total >= thr_rank, no segment overflowed and
//    total <= its buffer; otherwise thr_out[q] = thr_fallback[q] (+inf if null);
//  * result mode: the kp smallest (key, index) words form the shortlist, then
//    re-rank / output as launch_select.  A query whose candidates cannot be
//    trusted (overflow, total < need, total > buf_words) is appended to
//    fail_idx (count in *fail_cnt) and gets no result.
constexpr int kCandMax = 2048;
constexpr int kCandMaxFew = 6144;  // for a plan's own buffer size, of few queries
constexpr int kMaxKpScan = 512;  // longest shortlist the threshold scan's selection keeps
constexpr int kScanMaxSegs = 512;  // candidate segments per query (splits x kScanParts)
struct CandSelect {
    const uint64_t* cand = nullptr;
    const uint32_t* cnt = nullptr;
    int nseg = 0;
    int cap = 0;
    int64_t Q = 0;
    const uint32_t* skip_if = nullptr;       // the kernel does nothing when *skip_if != 0
    const uint32_t* skip_if_zero = nullptr;  // the kernel does nothing when *skip_if_zero == 0
    float* thr_out = nullptr;
    int thr_rank = 0;
    const float* thr_fallback = nullptr;
    int kp = 0;
    int k = 0;
    int need = 0;
    int rerank = 1;
    const float* corpus = nullptr;
    int64_t ldc = 0;
    const float* queries = nullptr;
    int64_t ldq = 0;
    int D = 0;
    const float* qn = nullptr;
    float* out_dist = nullptr;
    int32_t* out_idx = nullptr;
    float* out_idx_f = nullptr;
    int32_t* fail_idx = nullptr;
    uint32_t* fail_cnt = nullptr;
    uint32_t* fail_thr = nullptr;  // all ones at every failed query's place (the fix-up's thresholds)
    // corpora below 16,384 rows, re-ranked: certify -- a query also fails when its shortlist may miss a row (as
    // SmallSelect::fp32_keys); else a query that is not finite does not fail but has no results
    bool small = false, certify = false;
    // exact-key test (optional): keys and distances are exact integers when every corpus and
    // query value is an integer, 2 * D * max|x|^2 < 2^24 and the BF16 copies are exact; the
    // re-rank is then skipped (distance = key + qn[q], the same value it would compute)
    const uint32_t* int_stats = nullptr;  // [0] not-integer flag, [1] max|x| bits (corpus and queries)
    const uint32_t* bf16_inexact = nullptr;
    // per-warp candidate buffer (words): result mode takes it as the caller's bound on one
    // query's stored candidates (0 = kCandMax; a query above it fails over to the fix-up);
    // threshold mode sets it from nseg * cap
    int buf_words = 0;
};
cudaError_t launch_select_cand(const CandSelect& c, cudaStream_t s);

// Running top-k (have entries, row pitch k) merged with a block's top-kb (pitch kb,
// indices + offset) into out (pitch k, min(k, have + kb) entries); out_idx_f optional.
cudaError_t launch_merge_topk(const float* run_d, const int32_t* run_i, int have, const float* blk_d,
                              const int32_t* blk_i, int kb, int32_t offset, int64_t Q, int k, float* out_d,
                              int32_t* out_i, float* out_idx_f, cudaStream_t s);

// out[i] = src[i * stride] for i < n, +inf for n <= i < n_pad (norms of padding rows), the
// norms of a strided corpus sample; nothing when skip_unless is given and *skip_unless == 0.
// With scales / out_scales the row scales of the sample are gathered too (padding 0).
cudaError_t launch_gather_norms(const float* src, int64_t n, int64_t stride, float* out, int64_t n_pad,
                                cudaStream_t s, const uint32_t* skip_unless = nullptr,
                                const float* scales = nullptr, float* out_scales = nullptr);

}  // namespace knn
