// Pieces shared by the per-mode scan kernels: parameters, ring-slot geometry, the CTA-level
// merge of the four warps' partials.
#pragma once

#include "decode_common.cuh"

namespace jf {

template <int MODE> struct Tile;
template <> struct Tile<JF_MODE_K3V2> {
  // A warp's ring is made of slots of two pages; a page is [K | V | K scales | V scales].
  static constexpr int kKRow = 48, kVRow = 32, kNG = 2;
  static constexpr int kKPage = 768, kVPage = 512, kSPage = 64;   // bytes per page and array
  static constexpr int kVOff = 768, kKsOff = 1280, kVsRel = 64;   // page-relative; V scales from the K scales
  static constexpr int kPageTx = 1408;    // bytes per page
  static constexpr int kSlotBytes = 2 * kPageTx;
  static constexpr int kSlots = 4;        // two-page slots per warp: eight pages in flight
};
template <> struct Tile<JF_MODE_K4V4> {
  // A warp's ring is made of two-page slots: [K page A | K page B | V page A | V page B |
  // K scales A, B | V scales A, B].  Two pages whose blocks are neighbours in the cache are
  // fetched as one 32-row tensor copy per tensor and one 64-byte copy per scale array; the
  // tiles are written by swizzled tensor copies and sit on 1024-byte boundaries.
  static constexpr int kKRow = 64, kVRow = 64, kNG = 1;
  static constexpr int kPageBytes = 1024;                 // K (or V) data of one page
  static constexpr int kVOff = 2048;                      // V page, from the K page of the same half
  static constexpr int kScaleOff = 4096;                  // K scales of half 0, from the slot base
  static constexpr int kVsOff = 64;                       // V scales, from the K scales of the same half
  static constexpr int kSlotBytes = 4608;
  static constexpr int kPageTx = 2112;                    // bytes that land per page
  static constexpr int kSlots = 2;                        // two-page slots per warp (4 CTAs = 16 warps per SM)
};

struct ScanParams {
  const void* q;
  const uint8_t* k_data;
  const uint16_t* k_scales;
  const uint8_t* v_data;
  const uint16_t* v_scales;
  const int64_t* block_table;
  const int32_t* seq_lens;
  float* scores;
  float* pmax;          // K3V2: largest score of every pair of pages, [B][H_q][np_stride] (see the select kernel)
  float* part_o;
  float* part_m;
  float* part_l;
  float* part_smax;
  int32_t* status;
  int64_t num_slots;
  int B, H_q, H_kv, G, max_S, max_blocks;
  float attn_scale;
  int q_dtype;
  bool fill_tail;       // the scores past a sequence's end are set to -inf
  int kv_shift;         // cache head = KV head >> kv_shift (see head_geom)
  int np_stride;        // entries per row of pmax
  SliceGeom geom;       // how the work is cut
  // K4V4: work is cut into two-page tiles (see scan_k4v4_kernel)
  int n_tiles, tiles_per_split, tiles_per_warp, ref_chunk;
  int tile_base[9];
};

// Grid (splits, sequences, KV heads), or (1, KV heads, sequences) with one CTA per pair: there are so many pairs
// then that they take about a wave or more, and with the sequences slowest blocks of one length follow one
// another, the short ones of falling lengths at the end (128 sequences of 700 and less x 8 KV heads, K4V4: 18
// us, 23 with the KV heads slowest, in no order slower).  With more CTAs a pair it is the other way round
// (16 ragged sequences of 65536 x 8, K4V4: 198 us, 204 with the sequences slowest).
struct ScanBlock { int b, hkv; };
__device__ __forceinline__ ScanBlock scan_block(const ScanParams& p) {
  const bool one = p.geom.splits == 1;
  return ScanBlock{static_cast<int>(one ? blockIdx.z : blockIdx.y), static_cast<int>(one ? blockIdx.y : blockIdx.z)};
}
inline dim3 scan_grid(const ScanParams& p) {
  return p.geom.splits == 1 ? dim3(1, p.H_kv, p.B) : dim3(p.geom.splits, p.B, p.H_kv);
}

// The positions [lo, hi) of `heads` score rows from `row` on: -inf, by the whole block, 16 bytes a store between the unaligned
// ends.  (With stores of four bytes a scan's own CTAs, 128 threads each, took 109 us where they now take 72: see kTailKernelBytes.)
__device__ __forceinline__ void fill_neg_inf(float* row, int max_S, int heads, int lo, int hi) {
  const int tid = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x), n = max(hi - lo, 0);
  row += lo;
  for (int h = 0; h < heads; ++h, row += max_S) {
    const int head = min(static_cast<int>(-(reinterpret_cast<uintptr_t>(row) >> 2) & 3), n), quads = (n - head) >> 2;
    float4* body = reinterpret_cast<float4*>(row + head);
    for (int i = tid; i < quads; i += nt) body[i] = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
    const int edge = tid < head ? tid : 4 * quads + tid;   // up to three elements before the quads, up to three after
    if (edge < n && (tid < head || edge >= head + 4 * quads)) row[edge] = -INFINITY;
  }
}
// Scores past the end of the block's sequence.  The sequence's CTAs of the KV head share the positions out, each for all query
// heads.  (In a kernel of its own this was a launch, of the two-stage call order's seven.)
__device__ __forceinline__ void fill_score_tail(const ScanParams& p, const ScanBlock& blk) {
  const int len = max(min(p.seq_lens[blk.b], p.max_S), 0), rest = p.max_S - len, parts = gridDim.x;
  const int per = (rest + parts - 1) / parts, lo = len + static_cast<int>(blockIdx.x) * per;
  fill_neg_inf(p.scores + (static_cast<int64_t>(blk.b) * p.H_q + blk.hkv * p.G) * p.max_S, p.max_S, p.G, lo, min(lo + per, p.max_S));
}

// This CTA's slice: units [lo, hi) of sequence b, whose length is len.  CTA x of sequence y of a KV head is its
// number y * splits + x; with equal shares that is slice x of sequence y.  Whole warp, the same for all lanes.
struct ScanSlice { int b, len, lo, hi; };
template <bool kShares>
__device__ __forceinline__ ScanSlice scan_slice(const ScanParams& p, int y, int lane) {
  const SliceGeom& g = p.geom;
  ScanSlice r;
  r.b = y;
  r.lo = blockIdx.x * g.units_per_split;
  r.hi = r.lo + g.units_per_split;   // (the sequence may end before)
  if (!kShares) {
    r.len = min(p.seq_lens[r.b], p.max_S);
    return r;
  }
  // the one load that everything waits for: a sequence's length per lane
  const int my_len = slice_len(p.seq_lens, p.B, p.max_S, 0, lane);
  const SliceSums s = slice_sums(g, p.seq_lens, p.B, p.max_S, lane, my_len);
  if (!s.equal) {
    uint32_t i = y * g.splits + blockIdx.x;   // CTAs left before this one
    r.b = r.lo = r.hi = 0;
    for (int b0 = 0; b0 < p.B; b0 += 32) {
      const uint32_t units = slice_units(b0 == 0 ? my_len : slice_len(p.seq_lens, p.B, p.max_S, b0, lane));
      const uint32_t n = slice_count(g, s, p.B, units);
      uint32_t incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += t;
      }
      const uint32_t hit = __ballot_sync(0xFFFFFFFFu, i < incl);
      if (hit) {
        const int l = __ffs(hit) - 1;
        const uint32_t k = i - incl + n;   // slice k of n, on the lane of the sequence
        const uint32_t lo = k * units / max(n, 1u), hi = (k + 1) * units / max(n, 1u);
        r.b = b0 + l;
        r.lo = __shfl_sync(0xFFFFFFFFu, static_cast<int>(lo), l);
        r.hi = __shfl_sync(0xFFFFFFFFu, static_cast<int>(hi), l);
        break;
      }
      i -= __shfl_sync(0xFFFFFFFFu, incl, 31);
    }
  }
  r.len = __shfl_sync(0xFFFFFFFFu, my_len, r.b & 31);
  if (r.b >= 32) r.len = max(min(p.seq_lens[r.b], p.max_S), 0);
  return r;
}

// Pairs of floats for the packed fp32 instructions (two results per issue slot).
__device__ __forceinline__ uint64_t pair_f32(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpair_f32(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

constexpr int kBtChunk = 16;              // block-table entries fetched per load (one per lane of a half-warp)

// Bytes of shared memory the merge needs (per-warp output tiles + statistics).
constexpr int kMergeBytes = (kScanWarps * kHeadsPad * JF_HEAD_DIM + 3 * kScanWarps * kHeadsPad) * 4;

// CTA-level merge, fixed summation order (bit-reproducible, no atomics).  Before the call
// every warp has written its un-permuted output tile to sm_o[warp][head][d] for the heads of the
// group; only these are merged and stored (with all eight, those of a group of four cost a scan
// of one wave 0.5 us: 1 x 32768 x 32 / 8 heads 11.2 -> 10.7).  l0/l1 are the lane's partial softmax
// sums for heads 2*tig and 2*tig+1, m_ref0/1 its reference points, smax0/1 the largest K group
// scales it saw.
__device__ __forceinline__ void cta_merge_store(const ScanParams& p, uint8_t* smem, float l0, float l1,
                                                float m_ref0, float m_ref1, float smax0, float smax1) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tig = lane & 3;
  float* sm_o = reinterpret_cast<float*>(smem);               // [4 warps][8][128]
  float* sm_m = sm_o + kScanWarps * kHeadsPad * JF_HEAD_DIM;  // [4][8]
  float* sm_l = sm_m + kScanWarps * kHeadsPad;                // [4][8]
  float* sm_s = sm_l + kScanWarps * kHeadsPad;                // [4][2]
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    l0 += __shfl_xor_sync(0xFFFFFFFFu, l0, o);
    l1 += __shfl_xor_sync(0xFFFFFFFFu, l1, o);
  }
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    smax0 = fmaxf(smax0, __shfl_xor_sync(0xFFFFFFFFu, smax0, o));
    smax1 = fmaxf(smax1, __shfl_xor_sync(0xFFFFFFFFu, smax1, o));
  }
  if (g == 0) {
    sm_m[warp * 8 + 2 * tig] = m_ref0; sm_m[warp * 8 + 2 * tig + 1] = m_ref1;
    sm_l[warp * 8 + 2 * tig] = l0;     sm_l[warp * 8 + 2 * tig + 1] = l1;
  }
  if (lane == 0) { sm_s[warp * 2] = smax0; sm_s[warp * 2 + 1] = smax1; }
  __syncthreads();
  const ScanBlock blk = scan_block(p);
  const int64_t pidx = (static_cast<int64_t>(blk.hkv) * p.B + blk.b) * gridDim.x + blockIdx.x;
  float* po = p.part_o + pidx * (kHeadsPad * JF_HEAD_DIM);
  for (int i = threadIdx.x; i < p.G * JF_HEAD_DIM; i += blockDim.x) {
    const int h = i >> 7;
    float M = kMinusBig;
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w) M = fmaxf(M, sm_m[w * 8 + h]);
    float acc = 0.f;
#pragma unroll
    for (int w = 0; w < kScanWarps; ++w)
      acc = fmaf(sm_o[w * (kHeadsPad * JF_HEAD_DIM) + i], ex2(ref_log2(sm_m[w * 8 + h]) - ref_log2(M)), acc);
    po[i] = acc;
  }
  if (threadIdx.x < p.G) {
    const int h = threadIdx.x;
    float M = kMinusBig;
    for (int w = 0; w < kScanWarps; ++w) M = fmaxf(M, sm_m[w * 8 + h]);
    float L = 0.f;
    for (int w = 0; w < kScanWarps; ++w) L += sm_l[w * 8 + h] * ex2(ref_log2(sm_m[w * 8 + h]) - ref_log2(M));
    p.part_m[pidx * kHeadsPad + h] = M;
    p.part_l[pidx * kHeadsPad + h] = L;
  }
  if (threadIdx.x < 2) {
    float s = 0.f;
    for (int w = 0; w < kScanWarps; ++w) s = fmaxf(s, sm_s[w * 2 + threadIdx.x]);
    p.part_smax[pidx * 2 + threadIdx.x] = s;
  }
}

// parts: 0 = scores and output partials, 1 = scores and softmax sums only, 2 = output partials from
// stored scores; int8p: the reference's batch > 1 weight rounding
jf_status_t launch_scan_k4v4(ScanParams sp, bool int8p, int parts, dim3 grid, cudaStream_t stream);

}  // namespace jf
