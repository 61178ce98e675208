// Quantise-on-append: fp16/bf16 K/V rows -> INT2/3/4 packed rows + bf16 group scales,
// scattered into the paged cache by slot.
//
// Arithmetic is the torch reference's (jetfire_vllm/kernels/intN_pack.py:81-98):
//   amax over the group -> fp32 amax / qmax (IEEE) clamped to 1e-8 -> bf16 (RNE)
//   q = clamp(rint(x / float(scale_bf16)), -qmax, qmax)   (IEEE divide, half-even)
// and the wire format is :172-222 (INT4 nibbles, INT2 MSB-first quads, INT3 24-bit
// groups split over three byte planes).  Negative slots are skipped
// (jetfire_vllm/kernels/fused_quant_write.py:150-152).
//
// Half a warp owns a (token, kv-head) row of K and the same row of V: lane l (0..15) holds
// elements 8l..8l+7 of each (one 16-byte load), which are one INT3 group, one INT4 word or one
// INT2 half-word of the packed row.  The halves of a warp take consecutive tokens of one head,
// so that what they store is contiguous in the cache; the slot is looked up once for both sides.
//
// What bounds it: instruction issue, until the arithmetic got small enough for memory to matter.
// The two divisions are not executed.  The inputs have at most 11 significant bits and a scale has
// 8, so a quotient that is not exactly on a rounding boundary k + 1/2 is at least 2^-12 (relative)
// away from it: rounding the approximate quotient to a multiple of 2^-14 first (its error is
// 2^-21) puts exact ties exactly on the tie and leaves everything else on its side of the
// boundary.  One fma against 768 does that rounding (floats there are 2^-14 apart), one add
// against 1.5 * 2^23 rounds half-even to the integer: two instructions per element instead of
// sixteen.  The scale goes the same way (approximate quotient rounded to 16 significant bits,
// then to bf16's 8).  Both identities hold for every input of the two types (enumerated in
// tests/test_append_rounding.py); groups with a NaN, an infinity or values past 2^125 take the divisions.
// Measured on a B200, 32768 tokens x 8 KV heads, INT3 K + INT2 V (157 MB): 71.0 us with the divisions'
// predecessor, 31.1 us = 5.1 TB/s with this form; 95 warp instructions per two rows of a side (256
// before), 74 % of the issue slots, DRAM at 51 % of its peak.  The copies alone take 26 us.
//
// Mirror rows: the reference keeps every appended row in full precision in host memory
// (jetfire_vllm/adapter/cache_store.py:311-323) and fills it with a device-to-host copy, a
// host synchronisation and an index_copy_ per append (:746-756), or through pinned staging
// and a host callback under CUDA graphs (:616-640).  Here the kernel that packs a row also
// stores its 256 raw bytes -- already in the half-warp's registers as sixteen 16-byte pieces
// -- straight into the mirror through a device-visible pointer (mapped pinned host memory),
// one coalesced 256-byte write per row, so an append is one launch with no host step.  The
// store's record of filled slots (:686-759) is written by the same launch.
#include <algorithm>

#include "jf_common.cuh"

namespace jf {

constexpr int kRowsPerHalf = 2;    // rows of K (and of V) a half-warp loads before it processes any
constexpr int kWarpsPerCta = 4;
// Batches of rows a block goes through (it loads one while it works on the one before): as many as leave 1.8 rounds
// of the six blocks that a multiprocessor holds, up to five; from there on as many (up to 8) as leave four rounds.  One batch a
// block up to four rounds, and four rounds then, was 15 % slower in the middle: 6500 x 8 rows 9.1 -> 8.1 us, 9000 12.4 ->
// 11.0, 12000 15.8 -> 13.8, 16000 17.8 -> 17.0; 3001 (4.3 us), 24000 (24.2) and 32768 (31.4) as before.  (A block with n
// batches takes 1.2 + 1.7 n us of a round: one wave of 0.85 with 3 batches 6.2 us, with 6 batches 11.8, 10 batches 18.2.)
constexpr int kMaxBatches = 8, kBlocksResident = 6, kBlocksPerSm = 4 * kBlocksResident;
inline int pack_batches(int64_t units, int sms) {
  const int64_t round = static_cast<int64_t>(sms) * kBlocksResident, want = (5 * units + round * 9 / 2) / (round * 9);
  const int64_t most = std::min<int64_t>(std::max<int64_t>(5, units / (static_cast<int64_t>(sms) * kBlocksPerSm)), kMaxBatches);
  return static_cast<int>(std::max<int64_t>(1, std::min(want, most)));
}
constexpr int kTokensPerBatch = kWarpsPerCta * 2 * kRowsPerHalf;   // of a block

struct PackSide {
  const void* x;
  int64_t stride_t, stride_h;
  uint8_t* data;
  uint16_t* scales;
  int nbits;
  uint16_t* mirror;   // (H_kv, num_slots, 128) 16-bit rows, device-visible; may be null
};

template <int DT> __device__ __forceinline__ uint32_t absmax2(uint32_t a, uint32_t b) {   // of two packed pairs; NaN wins, signs are left over
  uint32_t d;
  if (DT == JF_DTYPE_BF16) asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  else asm("max.NaN.xorsign.abs.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// acc * 2^S + b as an integer multiply-add (the FMA pipe has twice the throughput of the logic pipe)
template <int S> __device__ __forceinline__ uint32_t shl_add(uint32_t acc, uint32_t b) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(acc), "n"(1 << S), "r"(b));
  return d;
}

// Two 16-bit elements of a word as floats.
template <int DT> __device__ __forceinline__ void unpack2(uint32_t w, float& lo, float& hi) {
  if (DT == JF_DTYPE_BF16) {
    lo = __uint_as_float(w << 16);
    hi = __uint_as_float(w & 0xFFFF0000u);
  } else {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    lo = f.x;
    hi = f.y;
  }
}

__device__ __forceinline__ uint64_t pair_f32(float lo, float hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}

// What the lanes of a half-warp need per row and side, besides the raw elements.
struct RowQuant {
  uint32_t scale_hi;   // the group's scale, bf16 bits in the high half
  uint32_t c[8];       // bits of the floats 1.5 * 2^23 + q
};

// Largest magnitude of the lane's group: packed pairs, NaN wins, the sign bits are left over.
template <int DT, int GS> __device__ __forceinline__ uint32_t group_absmax(uint4 raw) {
  uint32_t m = absmax2<DT>(absmax2<DT>(raw.x, raw.y), absmax2<DT>(raw.z, raw.w));
#pragma unroll
  for (int o = 1; o < GS / 8; o <<= 1) m = absmax2<DT>(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  return absmax2<DT>(m, prmt(m, m, 0x1032u)) & 0x7FFF7FFFu;
}

// The quick form (see the head of the file): `m` = group_absmax, finite and below 2^125.
template <int DT, int QMAX>
__device__ __forceinline__ void quantise_quick(uint4 raw, uint32_t m, RowQuant& r) {
  float amax, dup;
  unpack2<DT>(m, dup, amax);
  float y = amax * (1.0f / static_cast<float>(QMAX));
  // to 16 significant bits first, where the quotient can be a tie of the rounding to bf16: nine bits
  // times 3 or 7 do not fit the eight of a bf16 input, and a division by 1 is exact
  if (DT == JF_DTYPE_FP16 && QMAX > 1) y = __uint_as_float((__float_as_uint(y) + 0x80u) & 0xFFFFFF00u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r.scale_hi) : "f"(fmaxf(y, 1e-8f)), "f"(0.0f));
  float rs;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rs) : "f"(__uint_as_float(r.scale_hi)));
  const uint64_t rs2 = pair_f32(rs, rs), c768 = pair_f32(768.0f, 768.0f);
  const uint64_t magic = pair_f32(12582912.0f - 768.0f, 12582912.0f - 768.0f);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo, hi;
    unpack2<DT>(w[i], lo, hi);
    uint64_t v = pair_f32(lo, hi);
    asm("fma.rn.f32x2 %0, %0, %1, %2;" : "+l"(v) : "l"(rs2), "l"(c768));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(magic));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(r.c[2 * i]), "=r"(r.c[2 * i + 1]) : "l"(v));
  }
}

// Any input: the divisions themselves (out of line: rare).
__device__ __noinline__ uint32_t code_by_division(float x, float sf, float qmax) {
  return __float_as_uint(fminf(fmaxf(rintf(__fdiv_rn(x, sf)), -qmax), qmax) + 12582912.0f);
}
// Every lane of the warp calls this (shuffles).
template <int DT, int QMAX, int GS>
__device__ __forceinline__ void quantise_by_division(uint4 raw, RowQuant& r) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
  float f[8], amax = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) unpack2<DT>(w[i], f[2 * i], f[2 * i + 1]);
#pragma unroll
  for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(f[i]));
#pragma unroll
  for (int o = 1; o < GS / 8; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  const float scale = fmaxf(__fdiv_rn(amax, static_cast<float>(QMAX)), 1e-8f);
  r.scale_hi = static_cast<uint32_t>(__bfloat16_as_ushort(__float2bfloat16_rn(scale))) << 16;
  const float sf = __uint_as_float(r.scale_hi);
#pragma unroll
  for (int i = 0; i < 8; ++i) r.c[i] = code_by_division(f[i], sf, static_cast<float>(QMAX));
}

// Codes to their places by one multiply-add each, most significant first; the constant parts of the
// floats' bits and the code offset leave together at the end (all modulo 2^32).
template <int NBITS, int GS>
__device__ __forceinline__ void store_row(const RowQuant& r, uint8_t* __restrict__ out_row, uint16_t* __restrict__ scale_row,
                                          int sub, bool live) {
  constexpr uint32_t kOne = 0x4B400000u - (1u << (NBITS - 1));
  const uint32_t(&c)[8] = r.c;
  uint32_t word;
  if (NBITS == 4) {        // byte B = (code 2B << 4) | code 2B+1
    word = c[6];
    word = shl_add<4>(word, c[7]); word = shl_add<4>(word, c[4]); word = shl_add<4>(word, c[5]);
    word = shl_add<4>(word, c[2]); word = shl_add<4>(word, c[3]); word = shl_add<4>(word, c[0]);
    word = shl_add<4>(word, c[1]);
    word -= kOne * 0x11111111u;
    if (live) reinterpret_cast<uint32_t*>(out_row)[sub] = word;
  } else if (NBITS == 2) { // byte B = four codes, first in the top bits
    word = c[4];
    word = shl_add<2>(word, c[5]); word = shl_add<2>(word, c[6]); word = shl_add<2>(word, c[7]);
    word = shl_add<2>(word, c[0]); word = shl_add<2>(word, c[1]); word = shl_add<2>(word, c[2]);
    word = shl_add<2>(word, c[3]);
    word -= kOne * 0x5555u;
    if (live) reinterpret_cast<uint16_t*>(out_row)[sub] = static_cast<uint16_t>(word);
  } else {                 // eight codes -> 24 bits MSB-first, byte p of group i at out_row[16 p + i]
    word = c[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) word = shl_add<3>(word, c[i]);
    word -= kOne * 011111111u;   // 1 + 8 + 64 + ...
    // four neighbouring lanes transpose their bytes, so that each holds a word of one byte plane
    // (plane 0 the most significant byte) and a row takes one store instead of three
    word = prmt(word, __shfl_xor_sync(0xFFFFFFFFu, word, 1), (sub & 1) ? 0x3715u : 0x6240u);
    word = prmt(word, __shfl_xor_sync(0xFFFFFFFFu, word, 2), (sub & 2) ? 0x3276u : 0x5410u);
    // lane j of four now holds byte j of the four words, low lane first: byte 2 is plane 0
    const int j = sub & 3;
    if (live && j < 3) *reinterpret_cast<uint32_t*>(out_row + 16 * (2 - j) + (sub & 12)) = word;
  }
  // scales: one per group, written by the group's first lane
  const uint16_t sb = static_cast<uint16_t>(r.scale_hi >> 16);
  if (GS == 64) { if (live && (sub & 7) == 0) scale_row[sub >> 3] = sb; }
  else { if (live && sub == 0) scale_row[0] = sb; }
}

// One row of one side.  RowT: type of a row's index in the cache (32 bits where they reach: one
// multiply-add per address instead of three).  `m` = group_absmax; `quick`: the whole warp may
// take the quick form.
template <int DT, int NBITS, int GS, bool kStore, typename RowT>
__device__ __forceinline__ void pack_row(const PackSide& s, uint4 raw, uint32_t m, bool quick, RowT row, int sub, bool live) {
  constexpr int QMAX = (1 << (NBITS - 1)) - 1;
  const uint64_t o = row;
  if (kStore && s.mirror != nullptr && live) reinterpret_cast<uint4*>(s.mirror + o * JF_HEAD_DIM)[sub] = raw;
  RowQuant r;
  if (quick) quantise_quick<DT, QMAX>(raw, m, r);
  else quantise_by_division<DT, QMAX, GS>(raw, r);
  store_row<NBITS, GS>(r, s.data + o * (16 * NBITS), s.scales + o * (128 / GS), sub, live);
}
// NB: code width of the side, 0 = taken from the arguments at run time.
template <int DT, int NB, int GS, bool kStore, typename RowT>
__device__ __forceinline__ void pack_side(const PackSide& s, uint4 raw, uint32_t m, bool quick, RowT row, int sub, bool live) {
  if (NB == 2 || (NB == 0 && s.nbits == 2)) pack_row<DT, 2, GS, kStore, RowT>(s, raw, m, quick, row, sub, live);
  else if (NB == 3 || (NB == 0 && s.nbits == 3)) pack_row<DT, 3, GS, kStore, RowT>(s, raw, m, quick, row, sub, live);
  else pack_row<DT, 4, GS, kStore, RowT>(s, raw, m, quick, row, sub, live);
}

// Block (head, run of tokens); a warp takes every kWarpsPerCta-th batch of consecutive tokens of the
// run, every other token per half, and loads a batch while it works on the one before.
// KB / VB: code widths, 0 = from the arguments; VB = -1: no V side.  kStore: the rows also go to the
// mirrors and the record of filled slots (where given).
template <int DT, int GS, int KB, int VB, bool kStore, typename RowT>
__global__ void __launch_bounds__(kWarpsPerCta * 32)
pack_append_kernel(const PackSide k, const PackSide v, const int64_t* __restrict__ slots, int64_t T, int64_t num_slots,
                   int batches, uint8_t* __restrict__ filled) {
  constexpr int R = kRowsPerHalf;
  const int lane = threadIdx.x & 31, half = lane >> 4, sub = lane & 15;
  const int h = blockIdx.x;
  int64_t t = (static_cast<int64_t>(blockIdx.z) * gridDim.y + blockIdx.y) * (static_cast<int64_t>(batches) * kTokensPerBatch) +
              (threadIdx.x >> 5) * (2 * R) + half;
  pdl_wait();
  pdl_trigger();   // the next kernel may start its prologue; it waits for this grid before reading
  if (t - half >= T) return;
  const uint16_t* kx = reinterpret_cast<const uint16_t*>(k.x) + h * k.stride_h + 8 * sub;
  const uint16_t* vx = reinterpret_cast<const uint16_t*>(v.x) + h * v.stride_h + 8 * sub;
  const RowT head_row = static_cast<RowT>(h) * static_cast<RowT>(num_slots);
  struct Batch {
    uint4 k[R], v[R];
    int64_t slot[R];
  };
  // tokens past the end read the last one and count as skipped; rows of skipped tokens are read
  // too: the load does not wait for the slot
  auto load = [&](int64_t t0, Batch& b) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int64_t ti = t0 + 2 * i, tc = ti < T ? ti : T - 1;
      b.slot[i] = ti < T ? slots[tc] : -1;
      b.k[i] = __ldg(reinterpret_cast<const uint4*>(kx + tc * k.stride_t));
      if (VB >= 0) b.v[i] = __ldg(reinterpret_cast<const uint4*>(vx + tc * v.stride_t));
    }
  };
  Batch nxt;
  load(t, nxt);
  for (int it = 0; it < batches; ++it) {
    const Batch cur = nxt;
    t += kTokensPerBatch;
    const bool more = it + 1 < batches && t - half < T;
    if (more) load(t, nxt);
    // one test for all the rows at hand: NaNs, infinities and magnitudes of 2^125 and more (only
    // bf16 has finite ones; the reciprocal of such a scale would be subnormal) take the divisions
    uint32_t km[R], vm[R], top = 0u;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      km[i] = group_absmax<DT, GS>(cur.k[i]);
      vm[i] = (VB >= 0) ? group_absmax<DT, GS>(cur.v[i]) : 0u;
      top = max(top, max(km[i], vm[i]));
    }
    constexpr uint32_t kTop = (DT == JF_DTYPE_BF16) ? 0x7E000000u : 0x7C000000u;   // bits of 2^125 / infinity in the high half
    const bool quick = !__any_sync(0xFFFFFFFFu, top >= kTop);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      // the two halves of a warp may disagree here; every lane runs the arithmetic (full-mask
      // shuffles), only live rows are stored
      const bool live = static_cast<uint64_t>(cur.slot[i]) < static_cast<uint64_t>(num_slots);   // never write outside the cache
      const RowT o = head_row + static_cast<RowT>(cur.slot[i]);   // not used when not live
      if (kStore && filled != nullptr && h == 0 && live && sub == 0) filled[cur.slot[i]] = 1;
      pack_side<DT, KB, GS, kStore, RowT>(k, cur.k[i], km[i], quick, o, sub, live);
      if (VB >= 0) pack_side<DT, VB < 0 ? 0 : VB, GS, kStore, RowT>(v, cur.v[i], vm[i], quick, o, sub, live);
    }
    if (!more) break;
  }
}

static jf_status_t check_side(const void* x, int64_t st, int64_t sh, const void* data, const void* scales, int nbits) {
  if (!x || !data || !scales) return JF_ERR_ARG;
  if (nbits < 2 || nbits > 4) return JF_ERR_UNSUPPORTED;
  if (!aligned(x, 16) || (st % 8) != 0 || (sh % 8) != 0) return JF_ERR_ARG;
  if (!aligned(data, 16) || !aligned(scales, 4)) return JF_ERR_ARG;
  return JF_OK;
}

template <int DT, int GS, bool kStore>
static cudaError_t launch_typed(const PackSide& k, const PackSide* v, dim3 grid, int64_t T, const int64_t* slots,
                                int64_t num_slots, int batches, uint8_t* filled, cudaStream_t stream) {
  const dim3 block(kWarpsPerCta * 32);
#define JF_LAUNCH(KB, VB, ROW, V) \
  launch_pdl(pack_append_kernel<DT, GS, KB, VB, kStore, ROW>, grid, block, 0, stream, k, V, slots, T, num_slots, batches, filled)
  if (!v) return JF_LAUNCH(0, -1, uint64_t, k);
  // the two modes of the decode path get kernels of their own, for caches of fewer than 2^31 rows
  const bool narrow = static_cast<uint64_t>(num_slots) * grid.x <= 0x7FFFFFFFull;
  if (narrow && GS == 64 && k.nbits == 3 && v->nbits == 2) return JF_LAUNCH(3, 2, uint32_t, *v);
  if (narrow && GS == 128 && k.nbits == 4 && v->nbits == 4) return JF_LAUNCH(4, 4, uint32_t, *v);
  return JF_LAUNCH(0, 0, uint64_t, *v);
#undef JF_LAUNCH
}

static jf_status_t launch_pack(const PackSide& k, const PackSide* v, int dtype, int64_t T, int H,
                               const int64_t* slots, int64_t num_slots, int gs, cudaStream_t stream, uint8_t* filled = nullptr) {
  if (T < 0 || H <= 0 || num_slots <= 0 || !slots) return JF_ERR_ARG;
  if (gs != 64 && gs != 128) return JF_ERR_UNSUPPORTED;
  if (dtype != JF_DTYPE_BF16 && dtype != JF_DTYPE_FP16) return JF_ERR_UNSUPPORTED;
  if (T == 0) return JF_OK;
  const int64_t units = (T + kTokensPerBatch - 1) / kTokensPerBatch;
  const int batches = pack_batches(units * H, num_sms());
  const int64_t ctas = (units + batches - 1) / batches;
  const int64_t gz = (ctas + 65534) / 65535;       // the y and z extents of a grid end at 65535
  if (gz > 65535) return JF_ERR_UNSUPPORTED;
  const dim3 grid(static_cast<unsigned>(H), static_cast<unsigned>((ctas + gz - 1) / gz), static_cast<unsigned>(gz));
  const bool store = k.mirror != nullptr || filled != nullptr;
  cudaError_t e;
#define JF_LAUNCH(DT, GS) (store ? launch_typed<DT, GS, true>(k, v, grid, T, slots, num_slots, batches, filled, stream) \
                                 : launch_typed<DT, GS, false>(k, v, grid, T, slots, num_slots, batches, filled, stream))
  if (dtype == JF_DTYPE_BF16) e = gs == 64 ? JF_LAUNCH(JF_DTYPE_BF16, 64) : JF_LAUNCH(JF_DTYPE_BF16, 128);
  else e = gs == 64 ? JF_LAUNCH(JF_DTYPE_FP16, 64) : JF_LAUNCH(JF_DTYPE_FP16, 128);
#undef JF_LAUNCH
  JF_CUDA_TRY(e);
  return JF_OK;
}

}  // namespace jf

extern "C" jf_status_t jf_pack_append(const void* x_tok, int32_t dtype, int64_t T, int32_t H_kv,
                                      int64_t stride_t, int64_t stride_h, const int64_t* slots,
                                      uint8_t* out_data, void* out_scales, int64_t num_slots,
                                      int32_t nbits, int32_t group_size, jf_stream_t stream) {
  jf_status_t st = jf::check_side(x_tok, stride_t, stride_h, out_data, out_scales, nbits);
  if (st != JF_OK) return st;
  jf::PackSide k{x_tok, stride_t, stride_h, out_data, static_cast<uint16_t*>(out_scales), nbits, nullptr};
  return jf::launch_pack(k, nullptr, dtype, T, H_kv, slots, num_slots, group_size,
                         static_cast<cudaStream_t>(stream));
}

extern "C" jf_status_t jf_pack_append_kv(const void* key_tok, const void* value_tok, int32_t dtype,
                                         int64_t T, int32_t H_kv, int64_t k_stride_t, int64_t k_stride_h,
                                         int64_t v_stride_t, int64_t v_stride_h, const int64_t* slots,
                                         uint8_t* k_data, void* k_scales, uint8_t* v_data, void* v_scales,
                                         int64_t num_slots, int32_t k_bits, int32_t v_bits,
                                         int32_t group_size, jf_stream_t stream) {
  jf_status_t st = jf::check_side(key_tok, k_stride_t, k_stride_h, k_data, k_scales, k_bits);
  if (st != JF_OK) return st;
  st = jf::check_side(value_tok, v_stride_t, v_stride_h, v_data, v_scales, v_bits);
  if (st != JF_OK) return st;
  jf::PackSide k{key_tok, k_stride_t, k_stride_h, k_data, static_cast<uint16_t*>(k_scales), k_bits, nullptr};
  jf::PackSide v{value_tok, v_stride_t, v_stride_h, v_data, static_cast<uint16_t*>(v_scales), v_bits, nullptr};
  return jf::launch_pack(k, &v, dtype, T, H_kv, slots, num_slots, group_size,
                         static_cast<cudaStream_t>(stream));
}

extern "C" jf_status_t jf_pack_append_kv_mirror(const void* key_tok, const void* value_tok, int32_t dtype,
                                                int64_t T, int32_t H_kv, int64_t k_stride_t, int64_t k_stride_h,
                                                int64_t v_stride_t, int64_t v_stride_h, const int64_t* slots,
                                                uint8_t* k_data, void* k_scales, uint8_t* v_data, void* v_scales,
                                                int64_t num_slots, int32_t k_bits, int32_t v_bits,
                                                int32_t group_size, void* k_mirror, void* v_mirror,
                                                jf_stream_t stream) {
  jf_status_t st = jf::check_side(key_tok, k_stride_t, k_stride_h, k_data, k_scales, k_bits);
  if (st != JF_OK) return st;
  st = jf::check_side(value_tok, v_stride_t, v_stride_h, v_data, v_scales, v_bits);
  if (st != JF_OK) return st;
  if (!k_mirror || !v_mirror || !jf::aligned(k_mirror, 16) || !jf::aligned(v_mirror, 16)) return JF_ERR_ARG;
  jf::PackSide k{key_tok, k_stride_t, k_stride_h, k_data, static_cast<uint16_t*>(k_scales), k_bits,
                 static_cast<uint16_t*>(k_mirror)};
  jf::PackSide v{value_tok, v_stride_t, v_stride_h, v_data, static_cast<uint16_t*>(v_scales), v_bits,
                 static_cast<uint16_t*>(v_mirror)};
  return jf::launch_pack(k, &v, dtype, T, H_kv, slots, num_slots, group_size,
                         static_cast<cudaStream_t>(stream));
}

extern "C" jf_status_t jf_store_append(const void* key_tok, const void* value_tok, int32_t dtype, int64_t T, int32_t H_kv,
                                       int64_t k_stride_t, int64_t k_stride_h, int64_t v_stride_t, int64_t v_stride_h,
                                       const int64_t* slots, uint8_t* k_data, void* k_scales, uint8_t* v_data,
                                       void* v_scales, int64_t num_slots, int32_t k_bits, int32_t v_bits,
                                       int32_t group_size, void* k_mirror, void* v_mirror, uint8_t* filled,
                                       jf_stream_t stream) {
  jf_status_t st = jf::check_side(key_tok, k_stride_t, k_stride_h, k_data, k_scales, k_bits);
  if (st != JF_OK) return st;
  st = jf::check_side(value_tok, v_stride_t, v_stride_h, v_data, v_scales, v_bits);
  if (st != JF_OK) return st;
  if ((k_mirror == nullptr) != (v_mirror == nullptr) || !jf::aligned(k_mirror, 16) || !jf::aligned(v_mirror, 16)) return JF_ERR_ARG;
  jf::PackSide k{key_tok, k_stride_t, k_stride_h, k_data, static_cast<uint16_t*>(k_scales), k_bits,
                 static_cast<uint16_t*>(k_mirror)};
  jf::PackSide v{value_tok, v_stride_t, v_stride_h, v_data, static_cast<uint16_t*>(v_scales), v_bits,
                 static_cast<uint16_t*>(v_mirror)};
  return jf::launch_pack(k, &v, dtype, T, H_kv, slots, num_slots, group_size, static_cast<cudaStream_t>(stream), filled);
}
