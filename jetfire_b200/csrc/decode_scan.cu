// Fused low-bit decode-attention scan for sm_100a.
//
// One pass over the packed KV cache computes, for all query heads of a KV head at once
// (so every packed byte is read from HBM once per step):
//   approximate scores  s = attn_scale * sum_g  scale_g * (q . codes_g)       -> scratch
//   online softmax      p = exp(s - m_ref)                                   (registers)
//   output partial      O += (p * vscale) . vcodes                           (registers)
// Replaces the reference's Stage A score kernels (jetfire_vllm/csrc/int3_qk_scores.cu:
// 103-312, csrc/int8tc_qk_scores.cu:133-488) and Stage B softmax.V kernels
// (csrc/int2_softmax_v.cu:101-144, 601-789; csrc/int8tc_softmax_v_fused.cu:1017-1401),
// which materialise scores and weights in HBM and read V once per *query* head.
//
// Data movement: a 16-token page of the cache is contiguous per tensor (768 B of INT3 K,
// 512 B of INT2 V, 64 + 64 B of bf16 scales for K3V2); a warp fetches two pages at a time with
// asynchronous 16-byte copies, half a warp per page, into its own ring of four two-page slots in
// shared memory, and reads them back with ldmatrix.  A page is exactly one MMA M tile.
// Block-table entries are fetched sixteen at a time, a chunk ahead of their use, and parked in
// shared memory together with what the copies need, so that the loop never waits for a global
// load and the warp-uniform work per page stays small.
//
// What bounds it: the issue of instructions, not memory and not a warp's dependent chain (the keys of the next
// round gone through beside the softmax and P.V of the last: no difference).  A page is 278 warp instructions (352
// with bulk copies, 280 before the codes sat at two bit positions).  On a scheduler of a B200 a logic or integer
// instruction takes two cycles of its pipe, packed 16-bit arithmetic two of the other, and an mma.sync.m16n8k16 -- 8.6 cycles
// alone -- does not run under them: beside a dozen others it adds 3.5 to 7 cycles, so that the 18 of a page are about a
// fifth of its ~ 550.  Of the 62.4 us of a layer of 4 sequences x 8 KV heads x 65536 positions (0.46 of the copy peak;
// 74.4 with bulk copies) the expansion of the K codes takes 10, of the V codes 4, the copies 8 and the score stores 2.
// (The same work as 128-token tiles on tcgen05, the expanded codes in tensor memory: 74 us.  A token a thread is 320
// instructions a page with its stores to tensor memory, and those that turn V over run at a quarter of the rate.)
//
// Compute: tokens sit on the MMA M axis and the (<= 8) query heads on N = 8.  Packed codes
// are expanded in registers straight into the A fragments of mma.sync.m16n8k16 (the
// dequantised tile never goes through shared memory).  A masked 2-/3-/4-bit field, read as a
// 16-bit float, is a subnormal number code * 2^pos * 2^-24 (fp16) or * 2^-133 (bf16): V fields go
// to the tensor core as they are (one AND per two codes), K fields take one bf16x2 fma that
// applies offset, group scale and the reference's bf16 rounding together.  The power-of-two
// factors are undone on the other operand (K: folded into Q) or on the output row (V); the V
// group scale is folded into P, the V codes' offset leaves through a sum(P) tile at the end.
//
// Narrow groups (at most four query heads per KV head, kNarrow): the eight columns would be half empty, so columns 4-7 repeat
// the heads.  In P.V the two halves carry the weights of the two V groups: half the conversions and transposes and one sum
// tile.  In the scores they carry the two bf16 terms of an fp16 query: half the MMAs, and four CTAs a multiprocessor instead
// of three.  32 / 8 heads: bf16 16 falling lengths up to 16384 51.4 -> 49.3 us, 1 x 32768 11.85 -> 11.35; fp16 4 x 32768
// 39.6 -> 35.3, 1 x 3000 6.6 -> 5.6.
#include "decode_scan.cuh"

namespace jf {

namespace {

// Bit position at which code x (0..7) of an INT3 group is picked up (see the unpack in the
// kernel): the 3-bit field has to sit inside the 7-bit bf16 mantissa.  Two positions, so that a
// (token, group) takes two offset constants.
__device__ __forceinline__ constexpr int k3_pos(int x) { return (x & 1) ? 0 : 3; }
// bit position of 2-bit field f (0..7, bit offset 2f of a 16-bit half row word)
__device__ __forceinline__ constexpr int v2_pos(int f) { return f <= 4 ? 2 * f : 2 * f - 10; }
// head-dim index inside the 8-wide chunk for field f: bytes are little-endian in the
// 16-bit load, codes MSB-first inside a byte
__device__ __forceinline__ constexpr int v2_dlocal(int f) { return 4 * (f >> 2) + 3 - (f & 3); }


// Dequantised K in the reference's rounding, times a power of two, in ONE bf16x2 fma per two
// codes.  The masked 3-bit field, read as bf16, is the subnormal f * 2^POS * 2^-133 (exponent
// bits zero).  With S = scale * 2^100 and C = -4 * 2^POS * 2^-133 * S = -scale * 2^(POS - 31)
// (both exact: powers of two times the scale),
//   fma(field, S, C) = bf16_rn((f - 4) * scale * 2^(POS - 33)) = 2^(POS - 33) * bf16_rn((f - 4) * scale):
// the fma rounds once, and a power of two commutes with the rounding -- which is
// jetfire_vllm/csrc/int3_qk_scores.cu:94-99.  The factor 2^(POS - 33) is undone by the query
// operand.  (An 8-bit scale times a 3-bit integer needs at most 10 bits: exact before rounding.)
struct K3Scale {
  uint32_t S;       // scale * 2^100, both halves
  uint32_t C0, C3;  // -scale * 2^(POS - 31) for POS = 0 and 3, both halves
};
__device__ __forceinline__ K3Scale k3_scale(uint32_t scale2) {
  K3Scale k;
  k.S = mul_bf16x2(scale2, 0x71807180u);    // 2^100
  k.C0 = mul_bf16x2(scale2, 0xB000B000u);   // -2^-31
  k.C3 = mul_bf16x2(scale2, 0xB180B180u);   // -2^-28
  return k;
}
template <int POS>
__device__ __forceinline__ uint32_t k3_field(uint32_t v, const K3Scale& k) {
  constexpr uint32_t m = (7u << POS) | (7u << (POS + 16));
  return fma_bf16x2(v & m, k.S, POS == 0 ? k.C0 : k.C3);
}
// One 32-bit word of each byte plane (4 INT3 groups = 32 channels of one row) -> 16 bf16x2
// registers R[pair][code]: pair p holds groups (2p, 2p+1) in its (low, high) halves.
__device__ __forceinline__ void k3_unpack_row(uint32_t P0, uint32_t P1, uint32_t P2, const K3Scale& k,
                                              uint32_t (&R)[2][8]) {
#pragma unroll
  for (int pr = 0; pr < 2; ++pr) {
    const uint32_t sel = pr ? 0x7362u : 0x5140u;
    const uint32_t lo = prmt(P2, P1, sel);  // halves: bits 15..0 of the two 24-bit groups
    const uint32_t hi = prmt(P1, P0, sel);  // halves: bits 23..8
    const uint32_t w5 = lo >> 6, w3 = hi >> 4, w1 = hi >> 10;   // codes 5, 4 | 3, 2 | 1, 0 at bits 0 and 3
    R[pr][7] = k3_field<0>(lo, k);
    R[pr][6] = k3_field<3>(lo, k);
    R[pr][5] = k3_field<0>(w5, k);
    R[pr][4] = k3_field<3>(w5, k);
    R[pr][3] = k3_field<0>(w3, k);
    R[pr][2] = k3_field<3>(w3, k);
    R[pr][1] = k3_field<0>(w1, k);
    R[pr][0] = k3_field<3>(w1, k);
  }
}

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the fp16 form without ordering against other asm statements (the compiler interleaves the pages)
__device__ __forceinline__ void mma_f16_nv(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                           uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// A V field as an fp16 operand without arithmetic: the masked 2-bit field, read as fp16, is the
// subnormal code * 2^POS * 2^-24.  The codes' offset of 2 is not removed per element: one extra
// MMA per page and group against a row of ones collects sum(P), and the epilogue forms
// 2^(24 - POS) * acc - 2 * sum(P).
template <int POS>
__device__ __forceinline__ uint32_t v2_field(uint32_t v) {
  constexpr uint32_t m = (3u << POS) | (3u << (POS + 16));
  return v & m;
}
constexpr uint32_t kOnesF16x2 = 0x3C003C00u;

// Shared-memory matrix loads: four 8 x 8 matrices of 16-bit elements, one row of 16 bytes per lane.
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <int OFF>
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(addr), "n"(OFF) : "memory");
  return v;
}
// base + index * SIZE in one multiply-add
template <int SIZE>
__device__ __forceinline__ const uint8_t* page_ptr(const void* base, uint32_t index) {
  uint64_t d;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(index), "n"(SIZE), "l"(base));
  return reinterpret_cast<const uint8_t*>(d);
}
// largest magnitudes of two packed bf16 pairs (NaN wins, sign bits are left over)
__device__ __forceinline__ uint32_t absmax_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// Per-warp state that lives across pages.
template <int QT>
struct K3State {
  uint32_t qf[QT][8][2];   // query fragments (B operand of the K MMA)
  float oacc[9][4];        // output accumulators, O^T fragments; tile 8: sum of the P operand, rows 0-7 V group 0, rows 8-15 group 1
  float m_ref0, m_ref1;    // softmax reference points of heads 2tig, 2tig+1
  uint64_t l2;             // softmax sums of the two heads
  uint32_t smax2;          // largest K group scales seen (bf16 pair: group 0, group 1; sign bits are noise)
  uint32_t ks_sel;         // PRMT selector: this lane's K group scale into both halves
  uint32_t vs_sel;         // narrow: PRMT selector of this lane's V group scale, as a float
};

// Scores of one page: token g of the lane in acc[0..1] (heads 2tig, 2tig+1), token g + 8 in acc[2..3].
template <int QT>
__device__ __forceinline__ void k3_scores(const K3State<QT>& st, float (&acc)[4], uint32_t p0a, uint32_t p0b, uint32_t p1a,
                                          uint32_t p1b, uint32_t p2a, uint32_t p2b, uint32_t ksa, uint32_t ksb) {
  uint32_t R0[2][8], R1[2][8];
  k3_unpack_row(p0a, p1a, p2a, k3_scale(prmt(ksa, ksa, st.ks_sel)), R0);
  k3_unpack_row(p0b, p1b, p2b, k3_scale(prmt(ksb, ksb, st.ks_sel)), R1);
  acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
#pragma unroll
  for (int t = 0; t < QT; ++t)
#pragma unroll
    for (int x = 0; x < 8; ++x)
      mma_bf16_16816(acc, R0[0][x], R1[0][x], R0[1][x], R1[1][x], st.qf[t][x][0], st.qf[t][x][1]);
}

// The P operand of one page: weights p[0..1] of token g, p[2..3] of token g + 8 (heads 2tig, 2tig+1) times
// the V scales, as {tokens 2tig, 2tig+1 | 2tig+8, 2tig+9} of head g, for channel half 0 then 1.
__device__ __forceinline__ void k3_weights(uint32_t (&B)[4], const float (&p)[4], uint32_t vsa, uint32_t vsb) {
#pragma unroll
  for (int qh = 0; qh < 2; ++qh) {
    const float va = __uint_as_float(qh ? (vsa & 0xFFFF0000u) : (vsa << 16)), vb = __uint_as_float(qh ? (vsb & 0xFFFF0000u) : (vsb << 16));
    float w[4];
    unpair_f32(mul2(pair_f32(p[0], p[1]), pair_f32(va, va)), w[0], w[1]);
    unpair_f32(mul2(pair_f32(p[2], p[3]), pair_f32(vb, vb)), w[2], w[3]);
    B[2 * qh] = movmatrix_trans(pack_f16x2_sat(w[0], w[1]));
    B[2 * qh + 1] = movmatrix_trans(pack_f16x2_sat(w[2], w[3]));
  }
}
// Narrow: the lane's columns belong to one V group, `vs_sel` picks its scale; B = {tokens 0-7, tokens 8-15}.
__device__ __forceinline__ void k3_weights_narrow(uint32_t (&B)[4], const float (&p)[4], uint32_t vsa, uint32_t vsb, uint32_t vs_sel) {
  const float va = __uint_as_float(prmt(vsa, 0u, vs_sel)), vb = __uint_as_float(prmt(vsb, 0u, vs_sel));
  float w[4];
  unpair_f32(mul2(pair_f32(p[0], p[1]), pair_f32(va, va)), w[0], w[1]);
  unpair_f32(mul2(pair_f32(p[2], p[3]), pair_f32(vb, vb)), w[2], w[3]);
  B[0] = movmatrix_trans(pack_f16x2_sat(w[0], w[1]));
  B[1] = movmatrix_trans(pack_f16x2_sat(w[2], w[3]));
}
// One page's (P * vscale).V into the output accumulators.  X = the page's V words, transposed so that a
// register holds two tokens' halves: {tokens 0-7, tokens 8-15} of channel half 0, then of half 1.
template <bool kNarrow>
__device__ __forceinline__ void k3_values(float (&oacc)[9][4], const uint32_t (&B)[4], const uint32_t (&X)[4]) {
#pragma unroll
  for (int qh = 0; qh < 2; ++qh) {
    const uint32_t B0 = B[kNarrow ? 0 : 2 * qh], B1 = B[kNarrow ? 1 : 2 * qh + 1], XA = X[2 * qh], XB = X[2 * qh + 1];
    const uint32_t XA2 = XA >> 10, XB2 = XB >> 10;
    // fields 2ml -> output row g, 2ml+1 -> output row g+8
    mma_f16_nv(oacc[qh * 4 + 0], v2_field<0>(XA), v2_field<2>(XA), v2_field<0>(XB), v2_field<2>(XB), B0, B1);
    mma_f16_nv(oacc[qh * 4 + 1], v2_field<4>(XA), v2_field<6>(XA), v2_field<4>(XB), v2_field<6>(XB), B0, B1);
    mma_f16_nv(oacc[qh * 4 + 2], v2_field<8>(XA), v2_field<0>(XA2), v2_field<8>(XB), v2_field<0>(XB2), B0, B1);
    mma_f16_nv(oacc[qh * 4 + 3], v2_field<2>(XA2), v2_field<4>(XA2), v2_field<2>(XB2), v2_field<4>(XB2), B0, B1);
    if (!kNarrow) mma_f16_nv(oacc[8], qh ? 0u : kOnesF16x2, qh ? kOnesF16x2 : 0u, qh ? 0u : kOnesF16x2, qh ? kOnesF16x2 : 0u, B0, B1);
  }
  if (kNarrow) mma_f16_nv(oacc[8], kOnesF16x2, kOnesF16x2, kOnesF16x2, kOnesF16x2, B[0], B[1]);
}

// One round: two 16-token pages (A and B, one ring slot at shared-memory address `sb`).  Rows of the
// pages are MMA rows in order; a lane holds tokens g and g + 8 of both.  ldmatrix does what used to be
// fourteen scalar loads and four joins per page: untransposed it hands each lane its word of a K byte
// plane, transposed it pairs two tokens' V halves in one register.
// kMasked: only the first `live_a` / `live_b` tokens count (the last page of a sequence; an absent second page,
// a page whose block id was invalid: none); the common instance carries none of that logic.
// kParts: 0 = scores and output partials; 1 = scores and softmax sums only (no V);
// 2 = output partials from scores read back from memory (no K).
// kNarrow: the group has at most four query heads, and columns 4-7 repeat them: with the other V group's weights in P.V, with
// the second term of an fp16 query (kSplitQ) in the scores.
template <int QT, bool kMasked, int kParts, bool kNarrow, bool kSplitQ>
__device__ __forceinline__ void k3v2_round(K3State<QT>& st, uint32_t sb, const uint32_t (&off)[4], int g, int live_a, int live_b,
                                           float attn, float* row0, float* row1, uint32_t at, bool st0, bool st1,
                                           float* pm_row, uint32_t pm_at, bool pm_store, int lane) {
  using T = Tile<JF_MODE_K3V2>;
  constexpr bool kDoK = kParts != 2, kDoV = kParts != 1;
  // the lane's scores: two rows of the warp's, at the same byte offset (32 bits: one register for both)
  float* const sp0 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(row0) + at);
  float* const sp1 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(row1) + at);
  // the K side's shared-memory reads are issued up front
  uint32_t ka[4], kb[4], kc[4];   // planes 0, 1 of page A; of page B; plane 2 of both: {tokens 0-7, 8-15} each
  uint32_t ksa0 = 0u, ksa1 = 0u, ksb0 = 0u, ksb1 = 0u, vsa0 = 0u, vsa1 = 0u, vsb0 = 0u, vsb1 = 0u;
  uint32_t xa[4], xb[4];
  const uint32_t sc = sb + off[3];
  if (kDoK) {
    ldsm_x4(ka, sb + off[0]);
    ldsm_x4(kc, sb + off[1]);
    ldsm_x4(kb, sb + off[0] + T::kPageTx);
    ksa0 = lds32<0>(sc); ksa1 = lds32<32>(sc); ksb0 = lds32<T::kPageTx>(sc); ksb1 = lds32<T::kPageTx + 32>(sc);
  }
  const bool la = !kMasked || g < live_a, ha = !kMasked || g + 8 < live_a;
  const bool lb = !kMasked || g < live_b, hb = !kMasked || g + 8 < live_b;
  if (kMasked) {   // what an absent page's half of the slot holds need not even be finite
    if (!la) ksa0 = 0u;
    if (!ha) ksa1 = 0u;
    if (!lb) ksb0 = 0u;
    if (!hb) ksb1 = 0u;
  }

  // ---------------- scores ----------------
  float sA[4] = {0.f, 0.f, 0.f, 0.f}, sB[4] = {0.f, 0.f, 0.f, 0.f};
  if (kDoK) {
    st.smax2 = absmax_bf16x2(st.smax2, absmax_bf16x2(absmax_bf16x2(ksa0, ksa1), absmax_bf16x2(ksb0, ksb1)));
    k3_scores<QT>(st, sA, ka[0], ka[1], ka[2], ka[3], kc[0], kc[1], ksa0, ksa1);
    k3_scores<QT>(st, sB, kb[0], kb[1], kb[2], kb[3], kc[2], kc[3], ksb0, ksb1);
    if (kSplitQ) {   // the two terms of a score lie four columns apart
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sA[i] += __shfl_xor_sync(0xFFFFFFFFu, sA[i], 2);
        sB[i] += __shfl_xor_sync(0xFFFFFFFFu, sB[i], 2);
      }
    }
    const uint64_t attn2 = pair_f32(attn, attn);
    unpair_f32(mul2(pair_f32(sA[0], sA[1]), attn2), sA[0], sA[1]);
    unpair_f32(mul2(pair_f32(sA[2], sA[3]), attn2), sA[2], sA[3]);
    unpair_f32(mul2(pair_f32(sB[0], sB[1]), attn2), sB[0], sB[1]);
    unpair_f32(mul2(pair_f32(sB[2], sB[3]), attn2), sB[2], sB[3]);
  } else {
    // the scores an earlier scan stored (heads past the group stay at 0: their columns are dropped)
    if (st0) {
      if (la) sA[0] = sp0[0];
      if (ha) sA[2] = sp0[8];
      if (lb) sB[0] = sp0[16];
      if (hb) sB[2] = sp0[24];
    }
    if (st1) {
      if (la) sA[1] = sp1[0];
      if (ha) sA[3] = sp1[8];
      if (lb) sB[1] = sp1[16];
      if (hb) sB[3] = sp1[24];
    }
  }
  if (kMasked) {
    if (!la) sA[0] = sA[1] = -INFINITY;
    if (!ha) sA[2] = sA[3] = -INFINITY;
    if (!lb) sB[0] = sB[1] = -INFINITY;
    if (!hb) sB[2] = sB[3] = -INFINITY;
  }
  if (kDoK) {
    if (st0) {
      if (la) sp0[0] = sA[0];
      if (ha) sp0[8] = sA[2];
      if (lb) sp0[16] = sB[0];
      if (hb) sp0[24] = sB[2];
    }
    if (st1) {
      if (la) sp1[0] = sA[1];
      if (ha) sp1[8] = sA[3];
      if (lb) sp1[16] = sB[1];
      if (hb) sp1[24] = sB[3];
    }
  }

  // the V side, requested ahead of the softmax (with the K side it would not fit the registers)
  if (kDoV) {
    ldsm_x4_trans(xa, sb + off[2]);
    ldsm_x4_trans(xb, sb + off[2] + T::kPageTx);
    vsa0 = lds32<T::kVsRel>(sc); vsa1 = lds32<T::kVsRel + 32>(sc);
    vsb0 = lds32<T::kVsRel + T::kPageTx>(sc); vsb1 = lds32<T::kVsRel + T::kPageTx + 32>(sc);
    if (kMasked) {
      if (!la) vsa0 = 0u;
      if (!ha) vsa1 = 0u;
      if (!lb) vsb0 = 0u;
      if (!hb) vsb1 = 0u;
    }
  }

  // ---------------- online softmax over both pages ----------------
  // The reference point may lag the true maximum by less than 4 (exp stays below e^4, the fp16 P
  // operand cannot overflow); the exact maximum is only taken when a score runs ahead of it.
  float mx0 = fmaxf(fmaxf(sA[0], sA[2]), fmaxf(sB[0], sB[2])), mx1 = fmaxf(fmaxf(sA[1], sA[3]), fmaxf(sB[1], sB[3]));
  if (kDoK) {
    // largest score of the round's pages per head, for the select kernel's threshold: the halves of the
    // warp trade one head for the other (each lane sends one value and keeps one), then reduce over lane
    // bits 3 and 2
    const bool up = (lane & 16) != 0;
    float v = fmaxf(up ? mx1 : mx0, __shfl_xor_sync(0xFFFFFFFFu, up ? mx0 : mx1, 16));
    v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, 8));
    v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, 4));
    if (pm_store) *reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(pm_row) + pm_at) = v;
  }
  if (__any_sync(0xFFFFFFFFu, mx0 > st.m_ref0 + 4.0f || mx1 > st.m_ref1 + 4.0f)) {
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      mx0 = fmaxf(mx0, __shfl_xor_sync(0xFFFFFFFFu, mx0, o));
      mx1 = fmaxf(mx1, __shfl_xor_sync(0xFFFFFFFFu, mx1, o));
    }
    const float n0 = fmaxf(st.m_ref0, mx0), n1 = fmaxf(st.m_ref1, mx1);
    const float f0 = ex2(ref_log2(st.m_ref0) - ref_log2(n0)), f1 = ex2(ref_log2(st.m_ref1) - ref_log2(n1));
    st.l2 = mul2(st.l2, pair_f32(f0, f1));
    if (kDoV) {
#pragma unroll
      for (int i = 0; i < 9; ++i) { st.oacc[i][0] *= f0; st.oacc[i][1] *= f1; st.oacc[i][2] *= f0; st.oacc[i][3] *= f1; }
    }
    st.m_ref0 = n0; st.m_ref1 = n1;
  }
  const uint64_t c2 = pair_f32(kLog2e, kLog2e), mb2 = pair_f32(-ref_log2(st.m_ref0), -ref_log2(st.m_ref1));
  float pA[4], pB[4];
  unpair_f32(fma2(pair_f32(sA[0], sA[1]), c2, mb2), pA[0], pA[1]);
  unpair_f32(fma2(pair_f32(sA[2], sA[3]), c2, mb2), pA[2], pA[3]);
  unpair_f32(fma2(pair_f32(sB[0], sB[1]), c2, mb2), pB[0], pB[1]);
  unpair_f32(fma2(pair_f32(sB[2], sB[3]), c2, mb2), pB[2], pB[3]);
#pragma unroll
  for (int i = 0; i < 4; ++i) { pA[i] = ex2(pA[i]); pB[i] = ex2(pB[i]); }
  st.l2 = add2(st.l2, add2(add2(pair_f32(pA[0], pA[1]), pair_f32(pA[2], pA[3])), add2(pair_f32(pB[0], pB[1]), pair_f32(pB[2], pB[3]))));

  // ---------------- (P * vscale).V ----------------
  if (kDoV) {
    uint32_t BA[4], BB[4];
    if (kNarrow) {
      k3_weights_narrow(BA, pA, vsa0, vsa1, st.vs_sel);
      k3_weights_narrow(BB, pB, vsb0, vsb1, st.vs_sel);
    } else {
      k3_weights(BA, pA, vsa0, vsa1);
      k3_weights(BB, pB, vsb0, vsb1);
    }
    k3_values<kNarrow>(st.oacc, BA, xa);
    k3_values<kNarrow>(st.oacc, BB, xb);
  }
}

}  // namespace

// ------------------------------------------------------------------------------------
// K3V2
// ------------------------------------------------------------------------------------
template <int DT, int kParts, bool kShares, bool kNarrow>
__global__ void __launch_bounds__(kScanWarps * 32, (DT == JF_DTYPE_FP16 && !kNarrow) ? 3 : 4)
scan_k3v2_kernel(const ScanParams p) {
  using T = Tile<JF_MODE_K3V2>;
  constexpr int kQTerms = (DT == JF_DTYPE_FP16 && !kNarrow) ? 2 : 1;
  constexpr bool kSplitQ = DT == JF_DTYPE_FP16 && kNarrow;
  constexpr bool kDoK = kParts != 2, kDoV = kParts != 1;
  extern __shared__ __align__(128) uint8_t smem[];
  // the warp index is the same for all lanes; routing it through a shuffle tells the
  // compiler so, and lets slot addresses live in uniform registers
  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int g = lane >> 2, tig = lane & 3;
  const ScanBlock blk = scan_block(p);
  const int hkv = blk.hkv;

  const uint32_t smem_base = smem_u32(smem);
  constexpr int kRingBytes = kScanWarps * T::kSlots * T::kSlotBytes;
  constexpr int kPagesInFlight = 2 * T::kSlots;
  const uint32_t slots0 = smem_base + warp * (T::kSlots * T::kSlotBytes);
  // parked per page: its index in the cache (over all KV heads) and how many of its 16 tokens are live (see bt_entry)
  int2* bt_s = reinterpret_cast<int2*>(smem + kRingBytes) + warp * (2 * kBtChunk);

  pdl_wait();  // nothing above reads global memory

  const ScanSlice slice = scan_slice<kShares>(p, blk.b, lane);
  const int b = slice.b, len = slice.len, n_pages = (len + 15) >> 4;
  // Warp w owns a contiguous quarter of the split's pages, so its block-table entries are
  // contiguous too: sixteen lanes fetch sixteen entries with one load, a whole chunk ahead of
  // its use, and park them in shared memory.  (A load issued while megabytes of page copies are
  // queued in the memory system takes microseconds; fetched one entry at a time, a page or two
  // ahead, those loads stalled the loop.)
  const int per_warp = 2 * ((slice.hi - slice.lo + kScanWarps - 1) / kScanWarps);   // whole units: pairs of pages
  const int pg_first = 2 * slice.lo + warp * per_warp;
  const int my_n = max(0, min(min(pg_first + per_warp, 2 * slice.hi), n_pages) - pg_first);
  const int64_t* bt_w = p.block_table + static_cast<int64_t>(b) * p.max_blocks + pg_first;
  const int bt_avail = p.max_blocks - pg_first;   // entries of the row from this warp's first page on
  auto bt_load = [&](int chunk) -> int64_t {   // lanes 0..15: entry 16 * chunk + lane (never read when out of range)
    const int e = chunk * kBtChunk + lane;
    return (lane < kBtChunk && e < bt_avail) ? bt_w[e] : -1;
  };
  int64_t bt_pend = bt_load(0);
  const int64_t n_blocks_phys = p.num_slots >> 4;

  const uint32_t head_page0 = static_cast<uint32_t>(hkv >> p.kv_shift) * static_cast<uint32_t>(n_blocks_phys);
  const int last_pg = (len & 15) ? (n_pages - 1) : -1;   // the only page that can be partial
  // entry e of this warp (page pg_first + e) from its block id, worked out by sixteen lanes at
  // once when a chunk arrives: the sequence's last page may be partial; entries past the warp's range count -1.
  // An invalid block id counts no live token, and its tokens score -inf.  Who stores that is a matter of registers: behind
  // the round (the entry then counts -1 less its tokens, and fetches nothing) 4 x 65536 x 64 heads takes 62.0 us, from
  // here 63.9 (62.7 without either); an fp16 query of a wide group spills there, 8 falling lengths up to 32761 33.35 us,
  // from here 32.3 (32.8).
  constexpr bool kStoreHere = kQTerms == 2;
  auto bt_entry = [&](int64_t blk64, int e) -> int2 {
    const int pg = pg_first + e;
    const bool bad = blk64 < 0 || blk64 >= n_blocks_phys;
    const int tokens = pg == last_pg ? len - pg * 16 : 16, valid = e >= my_n ? -1 : !bad ? tokens : kStoreHere ? 0 : -1 - tokens;
    if (kDoK && kStoreHere && valid == 0) {
      float* row = p.scores + (static_cast<int64_t>(b) * p.H_q + hkv * p.G) * p.max_S + pg * 16;
#pragma unroll 1
      for (int h = 0; h < p.G; ++h, row += p.max_S)
#pragma unroll 1
        for (int i = 0; i < tokens; ++i) row[i] = -INFINITY;
    }
    return make_int2(static_cast<int>(head_page0 + (bad ? 0u : static_cast<uint32_t>(blk64))), valid);
  };
  // The copies of a slot's one or two pages, 16 bytes a lane: each half of the warp fetches a page
  // (lanes of an absent one stay out), seven instructions and four address multiply-adds per round.
  // (Bulk copies issued by one elected lane cost the warp 30 instructions more per page.)  Completion
  // is counted per thread and round (commit groups); a round without copies commits an empty group, so
  // that the count stays right.
  const int half = lane >> 4, l16 = lane & 15;
  const uint32_t dst = slots0 + half * T::kPageTx + 16 * l16;
  const uint32_t lane16 = 16 * l16;
  auto refill = [&](uint32_t slot_off, int e0) {   // pages e0, e0 + 1 of the warp; uniform
    const int2 ent = bt_s[(e0 + half) & (2 * kBtChunk - 1)];
    if (ent.y >= 0) {
      const uint32_t page = static_cast<uint32_t>(ent.x), d = dst + slot_off;
      if (kDoK) {
        const uint8_t* src = page_ptr<T::kKPage>(p.k_data, page) + lane16;
        cp_async_16_off<0>(d, src);
        cp_async_16_off<256>(d, src);
        cp_async_16_off<512>(d, src);
      }
      if (kDoV) {
        const uint8_t* src = page_ptr<T::kVPage>(p.v_data, page) + lane16;
        cp_async_16_off<0>(d + T::kVOff, src);
        cp_async_16_off<256>(d + T::kVOff, src);
      }
      // lanes 0-3 of a half: the K scales, 4-7: the V scales (next to them in the slot)
      if (kDoK && l16 < 4) cp_async_16_off<0>(d + T::kKsOff, page_ptr<T::kSPage>(p.k_scales, page) + lane16);
      if (kDoV && (l16 & 12) == 4) cp_async_16_off<0>(d + T::kKsOff, page_ptr<T::kSPage>(p.v_scales, page) + (lane16 - 64));
    }
  };
  const int4* ent_s = reinterpret_cast<const int4*>(bt_s);   // entries of a round's two pages (16 rounds resident)

  // prologue: chunk 0 to shared memory, chunk 1 requested, the ring filled
  if (lane < kBtChunk) bt_s[lane] = bt_entry(bt_pend, lane);
  int bt_stored = 0;   // chunks 0..bt_stored are in shared memory; chunk bt_stored + 1 is in bt_pend
  bt_pend = bt_load(1);
  __syncwarp();
#pragma unroll
  for (int sl = 0; sl < T::kSlots; ++sl) {
    if (2 * sl < my_n) refill(sl * T::kSlotBytes, 2 * sl);
    cp_async_commit();
  }

  // ---- query fragments: B operand of the K MMA, scaled by 2^(33 - pos) of the code it meets.
  //      Lane (head n = g, tig) covers channels 32 tig + 8 j + x (group j, code x); k-step x
  //      pairs groups (0,1) in b0 and (2,3) in b1.  A bf16 query is used as is; an fp16 query
  //      (11-bit significand) is split exactly into two bf16 terms, hi + lo. ----
  K3State<kQTerms> st;
  if (kDoK) {
    const int col = kNarrow ? (g & 3) : g, h = hkv * p.G + col;
    const bool live = col < p.G;
    const int64_t qbase = (static_cast<int64_t>(b) * p.H_q + h) * JF_HEAD_DIM;
    // this lane's 32 channels are contiguous: four 16-byte loads
    uint32_t qraw[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (live) v = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.q) + qbase + 32 * tig) + i);
      qraw[4 * i] = v.x; qraw[4 * i + 1] = v.y; qraw[4 * i + 2] = v.z; qraw[4 * i + 3] = v.w;
    }
    auto qval = [&](int d) {  // channel 32 tig + d of this lane's head
      const uint32_t w = qraw[d >> 1];
      return Elem<DT>::to_f32(static_cast<uint16_t>((d & 1) ? (w >> 16) : (w & 0xFFFFu)));
    };
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const float sc = 8589934592.0f / static_cast<float>(1 << k3_pos(x));   // 2^(33 - POS), see k3_field
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int d0 = 16 * half + x;  // group j = 2 * half
        const float a = qval(d0) * sc, c = qval(d0 + 8) * sc;
        const uint32_t hi2 = pack_bf16x2(a, c);
        st.qf[0][x][half] = hi2;
        if (kQTerms == 2) {
          const float ra = a - __uint_as_float(hi2 << 16), rc = c - __uint_as_float(hi2 & 0xFFFF0000u);
          st.qf[kQTerms - 1][x][half] = pack_bf16x2(ra, rc);
        }
        if (kSplitQ && g >= 4) st.qf[0][x][half] = pack_bf16x2(a - __uint_as_float(hi2 << 16), c - __uint_as_float(hi2 & 0xFFFF0000u));
      }
    }
  }
  st.ks_sel = (tig >> 1) ? 0x3232u : 0x1010u;
  st.vs_sel = (tig >> 1) ? 0x3244u : 0x1044u;
#pragma unroll
  for (int i = 0; i < 9; ++i) { st.oacc[i][0] = st.oacc[i][1] = st.oacc[i][2] = st.oacc[i][3] = 0.f; }
  st.m_ref0 = kMinusBig; st.m_ref1 = kMinusBig; st.l2 = 0ull;
  st.smax2 = 0u;

  // this lane's offsets in a slot: the matrix rows it names (row r of matrix m = lane >> 3) and its scales
  const int mr = (lane & 7) + 8 * ((lane >> 3) & 1), mh = lane >> 4;
  const uint32_t off[4] = {
      static_cast<uint32_t>(mr * T::kKRow + 16 * mh),                      // K planes 0 and 1 of page A (B: + kPageTx)
      static_cast<uint32_t>(mr * T::kKRow + 32 + T::kPageTx * mh),         // K plane 2 of pages A and B
      static_cast<uint32_t>(T::kVOff + mr * T::kVRow + 16 * mh),           // V halves of page A (B: + kPageTx)
      static_cast<uint32_t>(T::kKsOff + g * 4)};                           // scales of token g
  // scores: byte offsets from the rows of the KV head's first two query heads (eight rows of at most
  // 2^18 positions: 32 bits reach)
  float* const row0 = p.scores + (static_cast<int64_t>(b) * p.H_q + hkv * p.G) * p.max_S;
  float* const row1 = row0 + p.max_S;
  const int head0 = kNarrow ? 2 * (tig & 1) : 2 * tig;   // of the lane's columns 2tig, 2tig + 1
  uint32_t at = 4u * (head0 * static_cast<uint32_t>(p.max_S) + g + 16u * pg_first);
  // (narrow: the lanes of columns 4-7 read scores, but the others write them)
  const bool mine = !kNarrow || !kDoK || tig < 2;
  const bool st0 = mine && head0 < p.G, st1 = mine && head0 + 1 < p.G;
  // Page-pair maxima (pages 2m, 2m+1; a warp's range starts at an even page): after the round's
  // butterfly the lanes with bits 2 and 3 clear hold them -- lane bit 4 clear: head 2tig, set: 2tig+1.
  const int pm_head = 2 * tig + (lane >> 4);
  const bool want_pm = kDoK && p.pmax != nullptr;   // the same for the whole grid
  const bool pm_store = want_pm && (lane & 12) == 0 && pm_head < p.G;
  float* const pm_row = p.pmax + (static_cast<int64_t>(b) * p.H_q + hkv * p.G) * p.np_stride;
  uint32_t pm_at = 4u * (pm_head * static_cast<uint32_t>(p.np_stride) + (pg_first >> 1));
  const float attn = p.attn_scale;

  // A round takes one slot: two pages (one at the end of the range).
  uint32_t slot_off = 0u;
  for (int it = 0; it < my_n; it += 2) {
    cp_async_wait_group<T::kSlots - 1>();   // this lane's copies of the round have landed ...
    __syncwarp();                           // ... and every other lane's
    const uint32_t sb = slots0 + slot_off;
    const int4 ent = ent_s[(it >> 1) & (kBtChunk - 1)];   // the round's parked entries are still resident
    if (ent.y + ent.w == 32)
      k3v2_round<kQTerms, false, kParts, kNarrow, kSplitQ>(st, sb, off, g, 16, 16, attn, row0, row1, at, st0, st1, pm_row, pm_at, pm_store, lane);
    else {
      k3v2_round<kQTerms, true, kParts, kNarrow, kSplitQ>(st, sb, off, g, ent.y, ent.w, attn, row0, row1, at, st0, st1, pm_row, pm_at, pm_store,
                                        lane);
      if (kDoK && !kStoreHere && min(ent.y, ent.w) < -1) {
        const int na = -1 - ent.y, nb = -1 - ent.w;
        float* const s0 = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(row0) + at);
        for (int h = 0; h < 2; ++h) {
          float* const s = s0 + (h ? p.max_S : 0);
          if (!(h ? st1 : st0)) continue;
          if (g < na) s[0] = -INFINITY;
          if (g + 8 < na) s[8] = -INFINITY;
          if (g < nb) s[16] = -INFINITY;
          if (g + 8 < nb) s[24] = -INFINITY;
        }
      }
    }
    at += 128u;
    pm_at += 4u;
    __syncwarp();
    if (((it + kPagesInFlight + 1) >> 4) > bt_stored) {   // the refill below reads entries up to it + kPagesInFlight + 1
      ++bt_stored;
      if (lane < kBtChunk) bt_s[(bt_stored & 1) * kBtChunk + lane] = bt_entry(bt_pend, bt_stored * kBtChunk + lane);
      bt_pend = bt_load(bt_stored + 1);
      __syncwarp();
    }
    const int e0 = it + kPagesInFlight;   // first page to fetch into the slot just freed
    if (e0 < my_n) refill(slot_off, e0);
    cp_async_commit();
    slot_off = (slot_off == (T::kSlots - 1) * T::kSlotBytes) ? 0u : slot_off + T::kSlotBytes;
  }

  if (kDoK && p.fill_tail) fill_score_tail(p, blk);
  pdl_trigger();  // the next kernel may start its prologue; it waits for this grid before reading
  if (kDoK && threadIdx.x == 0 && (blockIdx.x | blockIdx.y | blockIdx.z) == 0) {
    p.status[4] = want_pm ? kPageMaxTag : 0;
    p.status[kWaitWord] = 0;
  }

  // ---------------- CTA merge: 4 warps -> one partial ----------------
  __syncthreads();  // every warp is done with its slots; smem is reused below
  {
    float* wo = reinterpret_cast<float*>(smem) + warp * (kHeadsPad * JF_HEAD_DIM);
#pragma unroll
    for (int mt = 0; mt < 8; ++mt) {
      const int qh = mt >> 2, ml = mt & 3;
      const int fa = 2 * ml, fb = 2 * ml + 1;
      const int da = 64 * qh + 8 * g + v2_dlocal(fa), db = 64 * qh + 8 * g + v2_dlocal(fb);
      // 2^(24 - POS) * sum(P * field) - 2 * sum(P): the codes' offset leaves here (see v2_field)
      const float ua = 16777216.0f / static_cast<float>(1 << v2_pos(fa)), ub = 16777216.0f / static_cast<float>(1 << v2_pos(fb));
      if (kNarrow && (tig >> 1) != qh) continue;   // the columns of the other group
      const float* sum = st.oacc[8] + (kNarrow ? 0 : 2 * qh);
      wo[head0 * JF_HEAD_DIM + da] = fmaf(st.oacc[mt][0], ua, -2.0f * sum[0]);
      wo[(head0 + 1) * JF_HEAD_DIM + da] = fmaf(st.oacc[mt][1], ua, -2.0f * sum[1]);
      wo[head0 * JF_HEAD_DIM + db] = fmaf(st.oacc[mt][2], ub, -2.0f * sum[0]);
      wo[(head0 + 1) * JF_HEAD_DIM + db] = fmaf(st.oacc[mt][3], ub, -2.0f * sum[1]);
    }
  }
  float l0, l1;
  unpair_f32(st.l2, l0, l1);
  cta_merge_store(p, smem, l0, l1, st.m_ref0, st.m_ref1, __uint_as_float((st.smax2 & 0x7FFFu) << 16),
                  __uint_as_float(st.smax2 & 0x7FFF0000u));
}

// ------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------
jf_status_t validate_decode_args(const jf_decode_args* a) {
  if (!a) return JF_ERR_ARG;
  if (a->mode != JF_MODE_K3V2 && a->mode != JF_MODE_K4V4) return JF_ERR_UNSUPPORTED;
  if (a->q_dtype != JF_DTYPE_BF16 && a->q_dtype != JF_DTYPE_FP16) return JF_ERR_UNSUPPORTED;
  if (a->B <= 0 || a->H_q <= 0 || a->H_kv <= 0 || a->max_S <= 0) return JF_ERR_ARG;
  if (a->H_q % a->H_kv != 0) return JF_ERR_ARG;
  const int G = a->H_q / a->H_kv;
  if (G > kHeadsPad && G != JF_MAX_GROUP) return JF_ERR_UNSUPPORTED;   // 1..8, or 16 as two halves
  if (a->block_size != JF_BLOCK_SIZE) return JF_ERR_UNSUPPORTED;
  if (a->max_S > 262144) return JF_ERR_UNSUPPORTED;
  if (a->top_k < 1 || a->top_k > JF_MAX_TOP_K) return JF_ERR_UNSUPPORTED;
  if (a->max_blocks < (a->max_S + 15) / 16) return JF_ERR_ARG;
  if (a->num_slots <= 0 || (a->num_slots % 16) != 0) return JF_ERR_ARG;
  // the scan kernels carry a page's first cache row (over all KV heads) as a 32-bit integer
  if (static_cast<uint64_t>(a->H_kv) * static_cast<uint64_t>(a->num_slots) > 0x7FFFFFFFull) return JF_ERR_UNSUPPORTED;
  if (a->scan_parts < JF_SCAN_ALL || a->scan_parts > JF_SCAN_V_ONLY) return JF_ERR_ARG;
  if (a->stage_b != JF_STAGE_B_FP32 && a->stage_b != JF_STAGE_B_INT8P) return JF_ERR_ARG;
  if (a->stage_b == JF_STAGE_B_INT8P && a->mode != JF_MODE_K4V4) return JF_ERR_UNSUPPORTED;
  const bool need_k = a->scan_parts != JF_SCAN_V_ONLY, need_v = a->scan_parts != JF_SCAN_K_ONLY;
  if (!a->block_table || !a->seq_lens) return JF_ERR_ARG;
  if (need_k && (!a->q || !a->k_data || !a->k_scales)) return JF_ERR_ARG;
  if (need_v && (!a->v_data || !a->v_scales)) return JF_ERR_ARG;
  if (!need_k && !a->scores) return JF_ERR_ARG;   // the scores are this call's input
  if (!aligned(a->k_data, 16) || !aligned(a->v_data, 16) || !aligned(a->k_scales, 16) || !aligned(a->v_scales, 16))
    return JF_ERR_ARG;
  if (!a->workspace || !aligned(a->workspace, 256)) return JF_ERR_WORKSPACE;
  if (a->workspace_bytes < jf_decode_workspace_bytes(a->mode, a->B, a->H_q, a->H_kv, a->max_S, a->top_k))
    return JF_ERR_WORKSPACE;
  return JF_OK;
}

SliceGeom slice_geom(const jf_decode_args* a, int splits) {
  SliceGeom g{};
  g.splits = splits;
  g.units = scan_units(a->max_S);
  g.units_per_split = (g.units + g.splits - 1) / g.splits;
  g.even = a->mode != JF_MODE_K3V2 || a->B == 1 || g.units_per_split < kShareMin;
  return g;
}

template <int DT, int kParts, bool kShares, bool kNarrow>
jf_status_t launch_k3v2_variant(const ScanParams& sp, dim3 grid, cudaStream_t stream) {
  using T = Tile<JF_MODE_K3V2>;
  const size_t smem = kScanWarps * T::kSlots * T::kSlotBytes + kScanWarps * 2 * kBtChunk * 8;  // ring, block-table chunks
  static_assert(kScanWarps * T::kSlots * T::kSlotBytes >= kMergeBytes, "merge buffer");
  JF_ENSURE_SMEM((scan_k3v2_kernel<DT, kParts, kShares, kNarrow>), smem);
  JF_CUDA_TRY(launch_pdl(scan_k3v2_kernel<DT, kParts, kShares, kNarrow>, grid, dim3(kScanWarps * 32), smem, stream, sp));
  JF_CUDA_TRY(cudaGetLastError());
  return JF_OK;
}
template <int DT, int kParts>
jf_status_t launch_k3v2(const ScanParams& sp, dim3 grid, cudaStream_t stream) {
  if (sp.G <= kNarrowGroup)
    return sp.geom.even ? launch_k3v2_variant<DT, kParts, false, true>(sp, grid, stream) : launch_k3v2_variant<DT, kParts, true, true>(sp, grid, stream);
  return sp.geom.even ? launch_k3v2_variant<DT, kParts, false, false>(sp, grid, stream) : launch_k3v2_variant<DT, kParts, true, false>(sp, grid, stream);
}

// Bytes of the scores from which on their tails have a kernel of their own.  Below, the scan's CTAs fill them and a
// launch is saved; of a gigabyte of tails, or half of one in few CTAs, they make less of the memory.  Scan and tails, in the scan / apart, us:
//   K3V2  128 sequences of 300 x 32 rows of 16384 (268 MB) 74.1 / 65.0;  8 of 200 x 32 of 131072 (134 MB) 30.3 / 69 with a block a row;
//         64 of 200 x 32 of 65536 (537 MB) 107.5 / 90.7;  32 x 32 of 131072 (537 MB) 113.8 / 87.6;  64 x 64 of 65536 (1.07 GB) 209 / 166
//   K4V4  81.2 / 71.0;  30.7 / 65;  120.5 / 91.8;  114.8 / 91.0;  229 / 167
// (With blocks of kTailPositions; one block a row, as before, 98, 98 and 170.)  The line lies above the case where the tails are
// short after all: a call of full rows pays the launch, 2 us.
constexpr int64_t kTailKernelBytes = 512ll << 20;
constexpr int kTailPositions = 32768;   // of a block
__global__ void __launch_bounds__(256) fill_score_tail_kernel(float* scores, const int32_t* seq_lens, int H_q, int max_S) {
  pdl_wait();
  pdl_trigger();   // the next kernel may start its prologue; it waits for this grid before reading
  const int bh = blockIdx.x, len = max(min(seq_lens[bh / H_q], max_S), 0), lo = blockIdx.y * kTailPositions;
  fill_neg_inf(scores + static_cast<int64_t>(bh) * max_S, max_S, 1, max(len, lo), min(lo + kTailPositions, max_S));
}

}  // namespace jf

extern "C" uint64_t jf_decode_workspace_bytes(int32_t mode, int32_t B, int32_t H_q, int32_t H_kv,
                                              int32_t max_S, int32_t top_k) {
  if (B <= 0 || H_q <= 0 || H_kv <= 0 || max_S <= 0 || top_k <= 0) return 0;
  return jf::carve_workspace(nullptr, mode, B, H_q, max_S, jf::partials_needed(mode, B, H_q, H_kv, max_S)).bytes;
}

extern "C" uint64_t jf_decode_workspace_useful_bytes(int32_t mode, int32_t B, int32_t H_q, int32_t H_kv,
                                                     int32_t max_S, int32_t top_k) {
  if (B <= 0 || H_q <= 0 || H_kv <= 0 || max_S <= 0 || top_k <= 0) return 0;
  const uint64_t most = jf::carve_workspace(nullptr, mode, B, H_q, max_S, jf::partials_useful(mode, B, H_q, H_kv, max_S)).bytes;
  const uint64_t least = jf_decode_workspace_bytes(mode, B, H_q, H_kv, max_S, top_k);
  return most > least ? most : least;
}

extern "C" jf_status_t jf_decode_scan(const jf_decode_args* a, jf_stream_t stream_) {
  using namespace jf;
  jf_status_t st = validate_decode_args(a);
  if (st != JF_OK) return st;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int splits = call_splits(a);
  Workspace ws = call_workspace(a, splits);
  ScanParams sp{};
  sp.q = a->q;
  sp.k_data = a->k_data;  sp.k_scales = static_cast<const uint16_t*>(a->k_scales);
  sp.v_data = a->v_data;  sp.v_scales = static_cast<const uint16_t*>(a->v_scales);
  sp.block_table = a->block_table;  sp.seq_lens = a->seq_lens;
  sp.scores = a->scores ? a->scores : ws.scores;
  // the maxima of groups of pages, if the select kernel of this call will work from them
  const SelectPlan plan = select_plan(a, sp.scores);
  if (!plan.supported) return JF_ERR_UNSUPPORTED;
  sp.pmax = plan.lean ? ws.pmax : nullptr;
  sp.np_stride = page_max_stride(a->mode, a->max_S);
  sp.part_o = ws.part_o; sp.part_m = ws.part_m; sp.part_l = ws.part_l; sp.part_smax = ws.part_smax;
  sp.status = ws.status;
  sp.num_slots = a->num_slots;
  const HeadGeom hg = head_geom(a->H_q, a->H_kv);
  sp.B = a->B; sp.H_q = a->H_q; sp.H_kv = hg.H_kv; sp.G = hg.G; sp.kv_shift = hg.shift;
  sp.max_S = a->max_S; sp.max_blocks = a->max_blocks;
  sp.geom = slice_geom(a, splits);
  sp.attn_scale = a->attn_scale;
  const bool seen = a->scores != nullptr && a->scan_parts != JF_SCAN_V_ONLY;   // scores the caller sees
  const bool apart = static_cast<int64_t>(a->B) * a->H_q * a->max_S * 4 >= kTailKernelBytes;
  sp.fill_tail = seen && !apart;
  sp.q_dtype = a->q_dtype;
  const dim3 grid = scan_grid(sp);
  if (a->mode == JF_MODE_K3V2) {
    // the query's type only matters where the query is read
    const int dt = a->scan_parts == JF_SCAN_V_ONLY ? JF_DTYPE_BF16 : a->q_dtype;
    if (dt == JF_DTYPE_BF16) {
      if (a->scan_parts == JF_SCAN_ALL) st = launch_k3v2<JF_DTYPE_BF16, 0>(sp, grid, stream);
      else if (a->scan_parts == JF_SCAN_K_ONLY) st = launch_k3v2<JF_DTYPE_BF16, 1>(sp, grid, stream);
      else st = launch_k3v2<JF_DTYPE_BF16, 2>(sp, grid, stream);
    } else {
      if (a->scan_parts == JF_SCAN_ALL) st = launch_k3v2<JF_DTYPE_FP16, 0>(sp, grid, stream);
      else st = launch_k3v2<JF_DTYPE_FP16, 1>(sp, grid, stream);
    }
  } else {
    st = launch_scan_k4v4(sp, a->stage_b == JF_STAGE_B_INT8P, a->scan_parts, grid, stream);
  }
  if (st == JF_OK && seen && apart)
    JF_CUDA_TRY(launch_pdl(fill_score_tail_kernel, dim3(a->B * a->H_q, (a->max_S + kTailPositions - 1) / kTailPositions),
                           dim3(256), 0, stream, a->scores, a->seq_lens, a->H_q, a->max_S));
  return st;
}
