// Finish stage shared by the fused select+finish kernel and the stand-alone finish kernel:
// merge the scan's split partials (log-sum-exp) into o_hat and the softmax statistics, and
// compute the approximate contribution of the selected set from the scan's own scores,
//   W = sum_{i in T} p_i,   o_old_unnorm[d] = sum_{i in T} (p_i * vscale_i,g(d)) * vcode_i,d
// (jetfire_vllm/csrc/int2_softmax_v.cu:738-788; V4: csrc/int4_softmax_v.cu:599-817), as the
// reference's Stage B does with the scores of its Stage A: what the later merge subtracts
// is exactly what the approximate pass added for these positions.
//
// Every summation order is fixed (no floating-point atomics) and does not depend on the block
// size: a block of NT threads plays the 1024 thread-items and the 32 warps of the widest
// block one after the other, so every kernel that runs this code gives the same bits.
//
// The selected set's sum runs on the tensor cores like the scan's P.V: sixteen entries are a "page",
// the masked code fields of their packed V rows go to mma.sync.m16n8k16 as subnormal fp16 numbers
// without arithmetic, the weights (times the V group scale, rounded to fp16 as the scan rounds its P
// operand) are the other operand -- one column of it; the codes' offset leaves through a
// sum-of-weights tile.
//
// What bounds it: latency -- one row per block, a chain of phases.  So there are two barriers for any
// top-k: the V words are read where they lie (the candidates' rows in shared memory, or the cache)
// instead of being brought into order first, a warp's groups accumulate in the MMA's registers, and the
// merge of the scan's partials is apart, for the caller to place where it waits for memory anyway.
#pragma once

#include "decode_common.cuh"

namespace jf {

constexpr int kSelThreads = 1024;                        // widest block; the unit of the fixed orders below
constexpr int kSelWarps = kSelThreads / 32;
constexpr int kSplitGroups = 16;                         // split partials are summed in 16 strided groups, a warp each

struct TailParams {
  const float* scores;
  const float* part_o;
  const float* part_m;
  const float* part_l;
  const uint8_t* v_data;
  const uint16_t* v_scales;
  float* o_hat;
  float* o_old;
  float* W;
  float* softmax_m;
  float* softmax_inv_z;
  int64_t num_slots;
  int H_q, H_kv, G, max_S, B, top_k;
  SliceGeom geom;   // where the scan's partials lie (slice_partials)
  int kv_shift;   // cache head = KV head >> kv_shift (see head_geom)
};

template <int MODE>
struct TailSmem {
  static constexpr int VW = (MODE == JF_MODE_K3V2) ? 8 : 16;    // 32-bit words per packed V row
  static constexpr int kParts = (MODE == JF_MODE_K3V2) ? 2 : 4; // channel ranges (64 / 32 channels), one per warp item
  static constexpr int kRows = kSelWarps / kParts;              // warps of the widest block per range
  float red[kRows][JF_HEAD_DIM];
  float sum[JF_MAX_TOP_K / 32];                                 // weights' sums of 32 entries each
  int32_t ref[JF_MAX_TOP_K];                                    // entry -> its V row: candidate, or slot
  uint16_t w[JF_MAX_TOP_K * ((MODE == JF_MODE_K3V2) ? 2 : 1)];  // weight * V scale as fp16 (K3V2: per group)
};

// The scan's partials of a row merged over the splits, unnormalised: sixteen partial sums per channel.
struct alignas(16) SplitSums {
  float o[kSplitGroups][JF_HEAD_DIM];
  float z[kSplitGroups];
};
// Warp w < 16 sums splits w, w + 16, ...: four channels a lane (a 512-byte row per load), the weight worked
// out by every lane from a broadcast load; two splits are in flight.
__device__ __forceinline__ void merge_splits(const TailParams& p, SplitSums& out, int64_t pbase, int splits, int hi, float M) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp >= kSplitGroups) return;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  float Z = 0.f;
#pragma unroll 1
  for (int s = warp; s < splits; s += 2 * kSplitGroups) {
    const bool two = s + kSplitGroups < splits;
    const int64_t e0 = (pbase + s) * kHeadsPad + hi, e1 = two ? e0 + kSplitGroups * kHeadsPad : e0;
    const float m0 = p.part_m[e0], m1 = p.part_m[e1], l0 = p.part_l[e0], l1 = p.part_l[e1];
    const float4 a = reinterpret_cast<const float4*>(p.part_o + e0 * JF_HEAD_DIM)[lane];
    const float4 c = reinterpret_cast<const float4*>(p.part_o + e1 * JF_HEAD_DIM)[lane];
    const float w0 = ex2(ref_log2(m0) - ref_log2(M)), w1 = two ? ex2(ref_log2(m1) - ref_log2(M)) : 0.f;
    Z = fmaf(l0, w0, Z);
    o.x = fmaf(a.x, w0, o.x); o.y = fmaf(a.y, w0, o.y); o.z = fmaf(a.z, w0, o.z); o.w = fmaf(a.w, w0, o.w);
    Z = fmaf(l1, w1, Z);
    o.x = fmaf(c.x, w1, o.x); o.y = fmaf(c.y, w1, o.y); o.z = fmaf(c.z, w1, o.z); o.w = fmaf(c.w, w1, o.w);
  }
  reinterpret_cast<float4*>(out.o[warp])[lane] = o;
  if (lane == 0) out.z[warp] = Z;
}

// What the fused kernel already holds in shared memory per candidate (null pointers in the
// stand-alone kernel): slot, scan score, V scales, packed V row.  The values are the ones
// the stand-alone kernel reads from global memory, so both give the same bits.
struct TailPrefetch {
  const int32_t* slot;
  const float* score;
  const uint32_t* vsc;    // K3: both group scales; K4: the aligned pair of scales that holds this slot's
  const uint32_t* vrows;
};

__device__ __forceinline__ uint32_t f16_bits_sat(float x) { return pack_f16x2_sat(x, 0.f) & 0xFFFFu; }

// Rounds in flight where a warp may have many and reads them from global memory (`many`: the stand-alone kernel, and the block of
// top-k above 512).  K4V4 gains by it, K3V2, with twice the arithmetic an entry, loses.  Four / one, us: the finish of 256 rows, top-k
// 2048, 40.3 / 47.2 (K3V2 51.8 / 43.1), of 512 12.9 / 14.1 (16.2 / 14.7); scan + select of 256 rows of 32768, top-k 4096, 344 / 354 (386 / 383).
__host__ __device__ constexpr int tail_rounds(int mode, bool many) { return mode == JF_MODE_K4V4 && many ? 4 : 1; }

// PPW channel ranges (part0 ...) of the selected set's weighted V sum, by one warp: groups of sixteen
// entries g0, g0 + step, ... of `top_k`.  `row(e)` = address of entry e's packed V row.
template <int MODE, int PPW, int kRounds, typename RowFn>
__device__ __forceinline__ void tail_part(const TailSmem<MODE>& sm, float* red, int part0, int g0, int step, int top_k, RowFn row) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  constexpr int NT_ = (MODE == JF_MODE_K3V2) ? 4 : 2;   // output tiles per part, and one for the sum of weights
  float t[PPW][NT_ + 1][4];
#pragma unroll
  for (int k = 0; k < PPW; ++k)
#pragma unroll
    for (int i = 0; i <= NT_; ++i) t[k][i][0] = t[k][i][1] = t[k][i][2] = t[k][i][3] = 0.f;
  // entries of the k-slots 2tig, 2tig+1, 2tig+8, 2tig+9, as in the scan's V path of the mode
  const int e_a = (MODE == JF_MODE_K3V2) ? tig : ((2 * tig >> 2) & 1) | (((2 * tig >> 1) & 1) << 2) | ((2 * tig & 1) << 1);
  const int e_b = (MODE == JF_MODE_K3V2) ? tig + 4
                                         : (((2 * tig + 1) >> 2) & 1) | ((((2 * tig + 1) >> 1) & 1) << 2) | (((2 * tig + 1) & 1) << 1);
#pragma unroll kRounds
  for (int grp = g0; 16 * grp < top_k; grp += step) {
    const int e0 = 16 * grp;   // entries past top_k have a place in the arrays and weigh nothing
    const uint8_t *ra = row(e0 + e_a), *rb = row(e0 + e_b), *rc = row(e0 + e_a + 8), *rd = row(e0 + e_b + 8);
    if (MODE == JF_MODE_K3V2) {
      uint32_t wa = 0u, wb = 0u, wc = 0u, wd = 0u;   // {group 0, group 1} weights
      if (g == 0) {   // the one column of the weight operand
        const uint32_t* w = reinterpret_cast<const uint32_t*>(sm.w) + e0;
        wa = w[e_a]; wb = w[e_b]; wc = w[e_a + 8]; wd = w[e_b + 8];
      }
#pragma unroll
      for (int k = 0; k < PPW; ++k) {
        const int part = part0 + k, at = 16 * part + 2 * g;
        const uint32_t Ha = *reinterpret_cast<const uint16_t*>(ra + at), Hb = *reinterpret_cast<const uint16_t*>(rb + at);
        const uint32_t Hc = *reinterpret_cast<const uint16_t*>(rc + at), Hd = *reinterpret_cast<const uint16_t*>(rd + at);
        const uint32_t sel = part ? 0x7632u : 0x5410u;
        const uint32_t b0 = prmt(wa, wb, sel), b1 = prmt(wc, wd, sel);
        const uint32_t XA = Ha | (Hb << 16), XB = Hc | (Hd << 16);
        const uint32_t XA2 = XA >> 10, XB2 = XB >> 10;
        constexpr uint32_t m0 = 0x00030003u;
        mma_f16_16816(t[k][0], XA & m0, XA & (m0 << 2), XB & m0, XB & (m0 << 2), b0, b1);
        mma_f16_16816(t[k][1], XA & (m0 << 4), XA & (m0 << 6), XB & (m0 << 4), XB & (m0 << 6), b0, b1);
        mma_f16_16816(t[k][2 % NT_], XA & (m0 << 8), XA2 & m0, XB & (m0 << 8), XB2 & m0, b0, b1);
        mma_f16_16816(t[k][3 % NT_], XA2 & (m0 << 2), XA2 & (m0 << 4), XB2 & (m0 << 2), XB2 & (m0 << 4), b0, b1);
        mma_f16_16816(t[k][NT_], 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, b0, b1);
      }
    } else {
      uint32_t b0 = 0u, b1 = 0u;
      if (g == 0) {
        b0 = sm.w[e0 + e_a] | (static_cast<uint32_t>(sm.w[e0 + e_b]) << 16);
        b1 = sm.w[e0 + e_a + 8] | (static_cast<uint32_t>(sm.w[e0 + e_b + 8]) << 16);
      }
#pragma unroll
      for (int k = 0; k < PPW; ++k) {
        const int wi = (part0 + k) & 1, bp = (part0 + k) >> 1, at = 8 * g + 4 * wi;   // channels 16g + 8wi ..
        const uint32_t wa = *reinterpret_cast<const uint32_t*>(ra + at), wb = *reinterpret_cast<const uint32_t*>(rb + at);
        const uint32_t wc = *reinterpret_cast<const uint32_t*>(rc + at), wd = *reinterpret_cast<const uint32_t*>(rd + at);
        const uint32_t sel = bp ? 0x7632u : 0x5410u;
        const uint32_t XA = prmt(wa, wb, sel), XB = prmt(wc, wd, sel);
        const uint32_t XA2 = XA >> 8, XB2 = XB >> 8;
        constexpr uint32_t m0 = 0x000F000Fu;
        mma_f16_16816(t[k][0], XA & m0, XA & (m0 << 4), XB & m0, XB & (m0 << 4), b0, b1);
        mma_f16_16816(t[k][1], XA2 & m0, XA2 & (m0 << 4), XB2 & m0, XB2 & (m0 << 4), b0, b1);
        mma_f16_16816(t[k][NT_], 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, 0x3C003C00u, b0, b1);
      }
    }
  }
  if (tig != 0) return;
#pragma unroll
  for (int k = 0; k < PPW; ++k) {
    const int part = part0 + k;
    const float* sums = t[k][NT_];
    if (MODE == JF_MODE_K3V2) {   // column 0: rows g (fields 2ml) and g + 8 (fields 2ml + 1)
#pragma unroll
      for (int ml = 0; ml < NT_; ++ml) {
        const int fa = 2 * ml, fb = 2 * ml + 1;
        // bit position of field f in its 16-bit half (after the shift by 10 for f >= 5) and its channel
        const int pa = fa <= 4 ? 2 * fa : 2 * fa - 10, pb = fb <= 4 ? 2 * fb : 2 * fb - 10;
        const int da = 64 * part + 8 * g + 4 * (fa >> 2) + 3 - (fa & 3), db = 64 * part + 8 * g + 4 * (fb >> 2) + 3 - (fb & 3);
        red[da] = fmaf(t[k][ml][0], 16777216.0f / static_cast<float>(1 << pa), -2.0f * sums[0]);
        red[db] = fmaf(t[k][ml][2], 16777216.0f / static_cast<float>(1 << pb), -2.0f * sums[2]);
      }
    } else {   // low nibble -> row g (odd channel), high nibble -> row g + 8 (even channel)
      const int wi = part & 1, bp = part >> 1;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int dlo = 16 * g + 8 * wi + 4 * bp + 2 * e + 1;
        red[dlo] = fmaf(t[k][e][0], 16777216.0f, -8.0f * sums[0]);
        red[dlo - 1] = fmaf(t[k][e][2], 1048576.0f, -8.0f * sums[2]);
      }
    }
  }
}

// `src(kk, pos, cidx)` yields the kk-th selected entry (rank order): its position and its
// index in the prefetched arrays; false if there is no such entry.  PRE: the prefetched arrays are there.
// M = max over the splits of the scan's reference points.  n = sequence length.  `splits` = the merged
// partials, written before the block's last barrier or by the same threads as here.
template <int MODE, int NT, bool PRE, int kRounds, typename Src>
__device__ __forceinline__ void finish_tail(const TailParams& p, TailSmem<MODE>& sm, const TailPrefetch& pf,
                                            const SplitSums& splits, float M, int n, int b, int h, const int64_t* bt, Src src) {
  constexpr int VW = TailSmem<MODE>::VW, kRows = TailSmem<MODE>::kRows;
  constexpr int kW = NT / 32;                 // warps of this block
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hkv = h / p.G;
  const int64_t bh = static_cast<int64_t>(b) * p.H_q + h;
  const ModeInfo mi = mode_info(MODE);
  const uint8_t* v_rows = p.v_data + static_cast<int64_t>(hkv >> p.kv_shift) * p.num_slots * mi.v_row;
  const uint16_t* v_sc = p.v_scales + static_cast<int64_t>(hkv >> p.kv_shift) * p.num_slots * mi.ng;
  const float* srow = p.scores + bh * p.max_S;

  // ---- selected set: weights from the scan's scores, 32 entries per warp and step ----
#pragma unroll kRounds
  for (int k0 = 32 * warp; k0 < p.top_k; k0 += NT) {
    const int kk = k0 + lane;
    int ref = 0;
    float w = 0.f, vs0 = 0.f, vs1 = 0.f;
    int pos = -1, cidx = 0;
    if (kk < p.top_k && n > 0 && src(kk, pos, cidx) && pos >= 0 && pos < n) {
      float approx;
      uint32_t sw = 0u;
      int64_t slot = -1;
      if (PRE) {
        slot = pf.slot[cidx];
        approx = pf.score[cidx];
        sw = pf.vsc[cidx];
        if (MODE == JF_MODE_K4V4) sw = (slot & 1) ? (sw >> 16) : (sw & 0xFFFFu);  // the pair that holds the scale
        ref = cidx;
      } else {
        const int64_t blk = bt[pos >> 4];
        approx = srow[pos];  // independent of the block-table lookup
        if (blk >= 0 && blk < (p.num_slots >> 4)) {
          slot = blk * 16 + (pos & 15);
          ref = static_cast<int>(slot);
          if (MODE == JF_MODE_K3V2) sw = __ldg(reinterpret_cast<const uint32_t*>(v_sc + slot * 2));
          else sw = __ldg(v_sc + slot);
        }
      }
      if (slot >= 0) {
        w = ex2(__fmaf_rn(approx, kLog2e, -ref_log2(M)));
        vs0 = __uint_as_float(sw << 16);
        vs1 = __uint_as_float(sw & 0xFFFF0000u);
      }
    }
    sm.ref[kk] = ref;     // the arrays hold a whole number of 32 entries: the last group's padding weighs nothing
    if (MODE == JF_MODE_K3V2)
      reinterpret_cast<uint32_t*>(sm.w)[kk] = pack_f16x2_sat(w * vs0, w * vs1);
    else
      sm.w[kk] = static_cast<uint16_t>(f16_bits_sat(w * vs0));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xFFFFFFFFu, w, o);
    if (lane == 0) sm.sum[k0 >> 5] = w;
  }
  __syncthreads();
  const int groups = (p.top_k + 15) / 16;
  {
    constexpr int PPW = kSelWarps / kW;   // ranges per warp: two in a block of 512 threads
    const int r = warp % kRows, part0 = (warp / kRows) * PPW;
    if (r < groups) {
      if (PRE)
        tail_part<MODE, PPW, kRounds>(sm, sm.red[r], part0, r, kRows, p.top_k,
                             [&](int e) { return reinterpret_cast<const uint8_t*>(pf.vrows + sm.ref[e] * VW); });
      else
        tail_part<MODE, PPW, kRounds>(sm, sm.red[r], part0, r, kRows, p.top_k,
                             [&](int e) { return v_rows + static_cast<int64_t>(sm.ref[e]) * (4 * VW); });
    }
  }
  __syncthreads();
  if (tid < JF_HEAD_DIM) {
    // the normaliser and the sum of weights pairwise: a running sum would round once per term at its full size
    float acc_old = 0.f, o[kSplitGroups], z[kSplitGroups];
#pragma unroll
    for (int r = 0; r < kRows; ++r)
      if (r < groups) acc_old += sm.red[r][tid];
#pragma unroll
    for (int gI = 0; gI < kSplitGroups; ++gI) { o[gI] = splits.o[gI][tid]; z[gI] = splits.z[gI]; }
#pragma unroll
    for (int d = kSplitGroups / 2; d > 0; d >>= 1)
#pragma unroll
      for (int gI = 0; gI < d; ++gI) { o[gI] += o[gI + d]; z[gI] += z[gI + d]; }
    const float Z = z[0];
    const bool live = (Z > 0.f) && (n > 0);
    const float inv_z = live ? (1.0f / Z) : 0.f;
    p.o_hat[bh * JF_HEAD_DIM + tid] = o[0] * inv_z;
    p.o_old[bh * JF_HEAD_DIM + tid] = acc_old * inv_z;
    float ws = 0.f;
    if (warp == 0) {
#pragma unroll 1
      for (int i = lane; 32 * i < p.top_k; i += 32) ws += sm.sum[i];
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) ws += __shfl_xor_sync(0xFFFFFFFFu, ws, d);
    }
    if (tid == 0) {
      p.W[bh] = ws * inv_z;
      if (p.softmax_m) p.softmax_m[bh] = live ? M : 0.f;
      if (p.softmax_inv_z) p.softmax_inv_z[bh] = inv_z;
    }
  }
}

// Shared by both kernels: the merged reference point M = max over the splits, block-wide.
// `red` = a float of shared memory per warp.  Ends with a barrier.  NT: threads of the block.
template <int NT>
__device__ __forceinline__ float block_max_of_splits(const float* part_m, int64_t pbase, int hi, int splits, float* red) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float M = kMinusBig;
#pragma unroll 1
  for (int s = tid; s < splits; s += NT) M = fmaxf(M, part_m[(pbase + s) * kHeadsPad + hi]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, o));
  if (lane == 0) red[warp] = M;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) M = fmaxf(M, red[w]);
  return M;
}

struct Workspace;
TailParams make_tail_params(const jf_decode_args* a, const Workspace& ws, int splits);
jf_status_t launch_select(const jf_decode_args* a, cudaStream_t stream, bool fused);

}  // namespace jf
