// Workspace layout and launch geometry shared by the scan, select and finish kernels.
#pragma once

#include "jf_common.cuh"

namespace jf {

constexpr int kScanWarps = 4;         // consumer warps per scan CTA; each owns whole pages
constexpr int kHeadsPad = 8;          // query heads of one KV head, padded to the MMA N
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kMinusBig = -1.0e30f; // finite stand-in for "no score seen yet"
#ifdef __CUDACC__
// A softmax reference point in the base-2 domain, as the scan's exp2(fma(s, log2(e), -ref)) uses it.  Every
// factor between two reference points and every weight of a selected entry is formed from this rounded
// product (not contracted into an fma), so that its rounding -- 2^-24 of it, 1e-6 of a weight at scores of
// 50 -- cancels between W, o_old and the normaliser.
__device__ __forceinline__ float ref_log2(float m) { return __fmul_rn(m, kLog2e); }
#endif

struct ModeInfo {
  int k_bits, v_bits, group_size, ng, k_row, v_row;
};
__host__ __device__ inline ModeInfo mode_info(int mode) {
  if (mode == JF_MODE_K4V4) return ModeInfo{4, 4, 128, 1, 64, 64};
  return ModeInfo{3, 2, 64, 2, 48, 32};
}

// The scan puts the query heads of one KV head on the eight columns of an MMA.  A GQA group of
// 16 (the reference's limit, jetfire_vllm/adapter/release_policy.py:31-34) is handled as two
// "virtual" KV heads of eight query heads each that read the same cache rows: every kernel sees
// H_kv << shift heads of G >> shift query heads and indexes the cache with (head >> shift).
struct HeadGeom { int H_kv, G, shift; };
__host__ __device__ inline HeadGeom head_geom(int H_q, int H_kv) {
  const int G = H_q / H_kv;
  const int shift = (G > kHeadsPad) ? 1 : 0;
  return HeadGeom{H_kv << shift, G >> shift, shift};
}

// Query heads of a KV head up to which both scans use the other four of the eight columns too (kNarrow: scan_k3v2_kernel
// repeats the heads there, scan_k4v4_kernel has a tile's second page there).
constexpr int kNarrowGroup = 4;
static_assert(kNarrowGroup <= kHeadsPad / 2, "columns 4-7 are free");
// Resident scan CTAs per SM (set by registers / shared memory of the kernel variant); G: query heads per (virtual) KV head.
__host__ __device__ inline int scan_ctas_per_sm(int mode, int q_dtype, int G) {
  return (mode == JF_MODE_K3V2 && q_dtype == JF_DTYPE_FP16 && G > kNarrowGroup) ? 3 : 4;
}

// ---- how the scan's work is cut -----------------------------------------------------------
// The unit of work is two 16-token pages of a sequence.  A launch has B * splits CTAs per KV head.
// `splits`: as many as fill one wave of resident CTAs, or two waves where that leaves fewer of them idle
// -- a CTA costs about eight units besides its own (start, merge: 3-4 us) -- with at least one unit per
// warp.  (K4V4, 16 sequences x 8 KV heads x 131072 positions: four splits fill 86 % of a wave, nine 97 %
// of two, 511 -> 478 us.)  Two waves only where the workspace has room for their partials (`most_waves`):
// what a call requires is the one wave's, which does not shrink as the row grows.
constexpr int kSliceOverhead = 8;
inline int scan_units(int max_S) { return ((max_S + JF_BLOCK_SIZE - 1) / JF_BLOCK_SIZE + 1) / 2; }
inline int scan_split_cap(int units) { return units < 8 ? 1 : units > 4 * 512 ? 512 : units / 4; }
inline int scan_splits(int mode, int q_dtype, int B, int H_kv, int G, int max_S, int most_waves) {
  const int units = scan_units(max_S), cap = scan_split_cap(units);
  const int pairs = B * H_kv, wave = num_sms() * scan_ctas_per_sm(mode, q_dtype, G);
  int best = 1;
  int64_t best_cost = INT64_MAX;
  for (int w = 1; w <= most_waves; ++w) {
    int s = w * wave / pairs;
    if (s > cap) s = cap;
    if (s < 1) s = 1;
    const int64_t waves = (static_cast<int64_t>(pairs) * s + wave - 1) / wave;
    const int64_t cost = waves * ((units + s - 1) / s + kSliceOverhead);
    if (cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

// A long ragged K3V2 batch shares the B * splits CTAs of a KV head out among its sequences in proportion
// to their lengths: with the same number for each, the short ones' CTAs left a third of the GPU idle
// (8 sequences of 5k-32k: 38.8 -> 34.0 us).  The lengths are only known on the device, so scan, select
// and finish work the shares out from them, each for itself and to the same result.  That costs a CTA
// about a microsecond, the work of two or three units, and gains a fraction of the scan: taken from
// kShareMin units a CTA on.  (Shares whatever the length: 1.3 us lost on a 2k row of one sequence, 3.6 us
// on three rows of 3-6k.)  Where all sequences have the units of the longest possible row -- a full
// batch -- the shares are equal again.  K4V4 keeps equal shares: its CTA has no registers left for the
// other case, which cost the scan of a full batch 2-5 %.
constexpr int kShareMin = 24;
struct SliceGeom {
  int splits, units;          // CTAs per sequence; units of a row of max_S positions
  int units_per_split;        // ceil(units / splits)
  int even;                   // every sequence has `splits` CTAs, whatever its length
};
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t slice_units(int len) { return len > 0 ? static_cast<uint32_t>((((len + 15) >> 4) + 1) >> 1) : 0u; }
// Length of sequence `lane` of the 32 from b0 on (0 past B), clamped to the row.
__device__ __forceinline__ int slice_len(const int32_t* seq_lens, int B, int max_S, int b0, int lane) {
  return b0 + lane < B ? max(min(seq_lens[b0 + lane], max_S), 0) : 0;
}
// Whole warp: total units and non-empty sequences, and whether every sequence has the units of max_S.
// `my_len`: slice_len of the first 32 sequences.
struct SliceSums { uint32_t total, live; bool equal; };
__device__ __forceinline__ SliceSums slice_sums(const SliceGeom& g, const int32_t* seq_lens, int B, int max_S, int lane, int my_len) {
  SliceSums r{0u, 0u, true};
  for (int b0 = 0; b0 < B; b0 += 32) {
    const uint32_t u = slice_units(b0 == 0 ? my_len : slice_len(seq_lens, B, max_S, b0, lane));
    if (__any_sync(0xFFFFFFFFu, b0 + lane < B && u != static_cast<uint32_t>(g.units))) r.equal = false;
    r.total += u;
    r.live += u > 0u ? 1u : 0u;
  }
  if (!r.equal) {
    r.total = __reduce_add_sync(0xFFFFFFFFu, r.total);
    r.live = __reduce_add_sync(0xFFFFFFFFu, r.live);
  }
  return r;
}
// CTAs of a sequence of `units` units: one, and its share of the rest (so that they add up to no more than
// there are); never more than units.
__device__ __forceinline__ uint32_t slice_count(const SliceGeom& g, const SliceSums& s, int B, uint32_t units) {
  if (units == 0u) return 0u;
  return min(1u + units * (static_cast<uint32_t>(B * g.splits) - s.live) / s.total, units);
}
// Whole warp: where the partials of (KV head, sequence) lie -- the first one's index and how many.  (The
// partial of CTA i of a KV head is number hkv * B * splits + i.)
__device__ __forceinline__ void slice_partials(const SliceGeom& g, const int32_t* seq_lens, int B, int max_S, int hkv, int b, int lane,
                                               int& first, int& count) {
  first = (hkv * B + b) * g.splits;
  count = g.splits;
  if (g.even) return;
  const int my_len = slice_len(seq_lens, B, max_S, 0, lane);
  const SliceSums s = slice_sums(g, seq_lens, B, max_S, lane, my_len);
  if (s.equal) return;
  uint32_t before = 0u, mine = 0u;
  for (int b0 = 0; b0 <= b; b0 += 32) {
    const uint32_t n = slice_count(g, s, B, slice_units(b0 == 0 ? my_len : slice_len(seq_lens, B, max_S, b0, lane)));
    before += __reduce_add_sync(0xFFFFFFFFu, b0 + lane < b ? n : 0u);
    mine = __shfl_sync(0xFFFFFFFFu, n, b & 31);
  }
  first = hkv * B * g.splits + static_cast<int>(before);
  count = static_cast<int>(mine);
}
#endif

// Which select kernel a call takes -- decided from the arguments alone, so that the scan (which
// then leaves the maxima of groups of pages: K3V2 pairs of pages, K4V4 pages) and the select
// kernel (which then takes its threshold from them and never stages the row) agree.
//   narrow: more rows than multiprocessors -> two blocks share one, and a staged chunk is 16384
//           positions; otherwise a row has a multiprocessor to itself and a chunk of 32768;
//   lean:   the row does not fit one staged chunk, there are enough groups for the K-th largest group
//           maximum to be a tight bound, and the score rows are whole pages that 16-byte loads can read.
// Rows of one chunk stay with the kernel that stages them.  Scan + select, staged / from maxima, us, top-k
// 256 (64 where there are too few groups for that):
//   128 rows   K4V4 16384 29.2 / 29.6, 32768 41.3 / 41.7, 40960 50.4 / 48.1;  K3V2 8192 22.9 / 23.3,
//              16384 31.4 / 30.5, 32768 52.1 / 49.8, 40960 62.7 / 56.7
//    32 rows   K4V4 32768 24.0 / 23.7, 40960 29.3 / 25.8;  K3V2 32768 26.0 / 26.0, 40960 31.5 / 28.0
//   256 rows   (8 KV heads x 8 sequences) K4V4 16384 44.3 / 44.2, 20480 53.0 / 50.0;  K3V2 12288 39.5 / 39.5,
//              16384 49.1 / 47.8, 20480 64.1 / 54.7
// so the line is right for K4V4 and within 2 % up to there, and K3V2 would gain up to 5 % from half of it on.
// The maxima cost the scan 0.4 % (K3V2, whose warps form them anyway) and 4-5 % (K4V4).
constexpr int kStagedTopK = 2048;   // widest top-k of the kernel that stages the row
struct SelectPlan { bool narrow, lean, supported; };
inline SelectPlan select_plan(const jf_decode_args* a, const float* scores) {
  int sort_n = 512;
  while (sort_n < 2 * a->top_k) sort_n <<= 1;
  SelectPlan pl;
  pl.narrow = a->B * a->H_q > num_sms() && sort_n <= 1024;
  const int groups = (a->max_S + 15) / 16 / (a->mode == JF_MODE_K3V2 ? 2 : 1);
  const bool readable = (a->max_S & 15) == 0 && (reinterpret_cast<uintptr_t>(scores) & 15) == 0;
  pl.lean = readable && a->max_S > 32 * (pl.narrow ? 512 : 1024) && groups >= 4 * a->top_k;
  // A top-k above kStagedTopK has no room for its sort buffer beside a staged row: such calls
  // always take the kernel that stages nothing (with few groups its histogram tier gives way to
  // the exact radix tier over the row in L2).  pl.supported is false if they cannot.
  pl.supported = a->top_k <= kStagedTopK || readable;
  if (a->top_k > kStagedTopK) { pl.lean = readable; pl.narrow = false; }
  return pl;
}

struct Workspace {
  int32_t* status;   // status record: 64-bit tag, then the error code (see report_status)
  float* part_o;     // [H_kv][B * splits][8][128], see SliceGeom
  float* part_m;     // [H_kv][B * splits][8]
  float* part_l;     // [H_kv][B * splits][8]
  float* part_smax;  // [H_kv][B * splits][2]  largest K group scale seen (per group)
  float* pmax;       // [B][H_q][page_max_stride] largest approximate score of every pair of 16-token pages (K3V2) / every page (K4V4)
  float* scores;     // [B][H_q][max_S] approximate scores
  uint64_t bytes;
};

__host__ __device__ inline uint64_t align_up(uint64_t x, uint64_t a) { return (x + a - 1) / a * a; }
// entries per row of the page maxima, rounded up to whole float4s: K3V2 one per pair of 16-token
// pages, K4V4 one per page
__host__ __device__ inline int page_max_stride(int mode, int max_S) {
  const int group = (mode == JF_MODE_K3V2) ? 2 * JF_BLOCK_SIZE : JF_BLOCK_SIZE;
  return (((max_S + group - 1) / group) + 3) & ~3;
}

// With room for `partials` partials of the scan (CTAs).
inline Workspace carve_workspace(void* base, int mode, int B, int H_q, int max_S, uint64_t partials) {
  uint64_t off = 0;
  uint8_t* p = static_cast<uint8_t*>(base);
  Workspace w{};
  w.status = reinterpret_cast<int32_t*>(p + off);   off = align_up(off + 256, 256);
  w.part_o = reinterpret_cast<float*>(p + off);     off = align_up(off + partials * kHeadsPad * JF_HEAD_DIM * 4, 256);
  w.part_m = reinterpret_cast<float*>(p + off);     off = align_up(off + partials * kHeadsPad * 4, 256);
  w.part_l = reinterpret_cast<float*>(p + off);     off = align_up(off + partials * kHeadsPad * 4, 256);
  w.part_smax = reinterpret_cast<float*>(p + off);  off = align_up(off + partials * 2 * 4, 256);
  w.pmax = reinterpret_cast<float*>(p + off);
  off = align_up(off + static_cast<uint64_t>(B) * H_q * page_max_stride(mode, max_S) * 4, 256);
  w.scores = reinterpret_cast<float*>(p + off);
  off = align_up(off + static_cast<uint64_t>(B) * H_q * max_S * 4, 256);
  w.bytes = off;
  return w;
}
// Least partials a call needs room for (one wave, the query type with more CTAs, so one workspace serves
// both), and the most any call of up to these sizes makes use of (neither shrinks as B or max_S grows but
// for the remainder of a wave in the first).
inline uint64_t partials_needed(int mode, int B, int H_q, int H_kv, int max_S) {
  const HeadGeom hg = head_geom(H_q, H_kv);
  return static_cast<uint64_t>(B) * hg.H_kv * scan_splits(mode, JF_DTYPE_BF16, B, hg.H_kv, hg.G, max_S, 1);
}
inline uint64_t partials_useful(int mode, int B, int H_q, int H_kv, int max_S) {
  const uint64_t pairs = static_cast<uint64_t>(B) * head_geom(H_q, H_kv).H_kv, capped = pairs * scan_split_cap(scan_units(max_S));
  const uint64_t waves = 2ull * num_sms() * scan_ctas_per_sm(mode, JF_DTYPE_BF16, 1), most = capped < waves ? capped : waves;
  return most > pairs ? most : pairs;
}
// CTAs per sequence and KV head of a call (the same for its scan, select and finish), and its workspace.
inline int call_splits(const jf_decode_args* a) {
  const HeadGeom hg = head_geom(a->H_q, a->H_kv);
  const int two = scan_splits(a->mode, a->q_dtype, a->B, hg.H_kv, hg.G, a->max_S, 2);
  const uint64_t partials = static_cast<uint64_t>(a->B) * hg.H_kv * two;
  if (carve_workspace(nullptr, a->mode, a->B, a->H_q, a->max_S, partials).bytes <= a->workspace_bytes) return two;
  return scan_splits(a->mode, a->q_dtype, a->B, hg.H_kv, hg.G, a->max_S, 1);
}
inline Workspace call_workspace(const jf_decode_args* a, int splits) {
  return carve_workspace(a->workspace, a->mode, a->B, a->H_q, a->max_S,
                         static_cast<uint64_t>(a->B) * head_geom(a->H_q, a->H_kv).H_kv * splits);
}

// Status record at the start of the workspace.  A kernel whose bounded wait ran out writes
// the code and then the tag; a record without the tag reads as "no error", so a workspace
// needs no initialisation and no launch has to clear it.  jf_decode_status reads the record
// and clears it.
constexpr unsigned long long kStatusTag = 0x4A46535441545553ull;  // "JFSTATUS"
// Word 4 of the record: written by every scan -- this value if it left page maxima, 0 if not --
// and checked by the select kernel that works from them, so that a select whose arguments do not
// match the scan's reports JF_ERR_STATE (and selects nothing) instead of reading stale maxima.
constexpr int32_t kPageMaxTag = 0x504D4158;  // "PMAX"
// Word 8: how the wait of the step's end went, for its other blocks (adapter_step.cu); cleared by every scan
// that reads K.
constexpr int kWaitWord = 8;
constexpr int32_t kWaitDone = 1, kWaitRanOut = 2;
#ifdef __CUDACC__
__device__ __forceinline__ void report_status(int32_t* status, int code) {
  status[2] = code;
  __threadfence();
  *reinterpret_cast<unsigned long long*>(status) = kStatusTag;
}
#endif

jf_status_t validate_decode_args(const jf_decode_args* a);
// the cut of a call's work (`splits`: call_splits)
SliceGeom slice_geom(const jf_decode_args* a, int splits);
// device address of the library's built-in scratch array on the current device (decode_static.cu)
jf_status_t static_scratch_address(void** out);

}  // namespace jf
