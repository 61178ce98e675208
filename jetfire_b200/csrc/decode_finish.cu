// finish (stand-alone): the finish stage for a selected list that is already in memory --
// the phase-by-phase API; the fused entry point runs the same code inside the select kernel.
//
// merge_correct: out = dtype(o_hat + W * float(o_new) - o_old_unnorm)
// (jetfire_vllm/csrc/blend.cu:202-226).  The normaliser stays the approximate softmax's:
// this is mass substitution, not a re-normalised merge.
#include <cstring>

#include "finish_tail.cuh"

namespace jf {

namespace {

struct FinishParams {
  const int64_t* block_table;
  const int32_t* seq_lens;
  const int64_t* topk_idx;
  int max_blocks;
};

// One CTA per (query head, batch element), two per multiprocessor: a row is a chain of round trips to L2
// (selected positions, block ids, scales, V rows), which the other row's work covers.  512 rows of 65536
// positions 21.1 -> 15.0 us, 4096 rows of 1024 127 -> 76 against one block of 1024 threads, 32 rows 5.1 -> 5.2.
// The next kernel is not let in ahead of the end: in the two-stage order that gains nothing, and its blocks took the places of this
// one's where finish follows finish (256 rows, top-k 512: 14.7 us, 12.4 without).
constexpr int kFinishThreads = 512;
template <int MODE>
__global__ void __launch_bounds__(kFinishThreads, 2)
decode_finish_kernel(const FinishParams p, const TailParams tp) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  TailSmem<MODE>& tsm = *reinterpret_cast<TailSmem<MODE>*>(smem_raw);
  __shared__ float sm_m[kFinishThreads / 32];
  __shared__ SplitSums splits;
  const int h = blockIdx.x, b = blockIdx.y;
  const int hkv = h / tp.G, hi = h - hkv * tp.G;
  const int64_t bh = static_cast<int64_t>(b) * tp.H_q + h;
  pdl_wait();
  // the thread's first selected position: on its way while the partials are merged
  const int64_t* sel = p.topk_idx + bh * tp.top_k;
  const int first = threadIdx.x;
  const int64_t first_sel = first < tp.top_k ? sel[first] : -1;
  int pbase, n_splits;   // by every warp for itself
  slice_partials(tp.geom, p.seq_lens, tp.B, tp.max_S, hkv, b, threadIdx.x & 31, pbase, n_splits);
  const int n = min(p.seq_lens[b], tp.max_S);
  const float M = block_max_of_splits<kFinishThreads>(tp.part_m, pbase, hi, n_splits, sm_m);
  merge_splits(tp, splits, pbase, n_splits, hi, M);
  finish_tail<MODE, kFinishThreads, false, tail_rounds(MODE, true)>(tp, tsm, TailPrefetch{}, splits, M, n, b, h,
                                        p.block_table + static_cast<int64_t>(b) * p.max_blocks, [&](int kk, int& pos, int& cidx) {
                                          const int64_t v = kk == first ? first_sel : sel[kk];
                                          if (v < 0 || v >= n) return false;
                                          pos = static_cast<int>(v);
                                          cidx = -1;
                                          return true;
                                        });
}

// Exact row maximum and 1 / sum exp(s - max) of a stored score row, as the reference's
// statistics-emitting select computes them (jetfire_vllm/csrc/int8tc_qk_scores.cu:1790-1800):
// an empty or all -inf row gives m = 0, and a non-positive sum gives 1/Z = 0.
// One CTA per (query head, batch element); sums in a fixed order.
// What bounds it: latency.  A row of up to kStatsHeld positions is read once, all its loads in flight, and stays in
// registers between the two reductions; longer rows are read a second time for their rest.
constexpr int kStatsThreads = 512, kStatsPer = 16, kStatsHeld = kStatsThreads * kStatsPer;
__global__ void __launch_bounds__(kStatsThreads)
softmax_stats_kernel(const float* __restrict__ scores, const int32_t* __restrict__ seq_lens, float* __restrict__ out_m,
                     float* __restrict__ out_inv_z, int H_q, int max_S) {
  constexpr int kW = kStatsThreads / 32;
  __shared__ float red[kW], red_z[kW];
  const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  pdl_wait();
  pdl_trigger();   // the next kernel may start its prologue; it waits for this grid before reading
  const int n = max(0, min(seq_lens[b], max_S));
  const float* row = scores + (static_cast<int64_t>(b) * H_q + h) * max_S;
  float v[kStatsPer], m = -INFINITY;
#pragma unroll
  for (int k = 0; k < kStatsPer; ++k) {
    const int i = tid + k * kStatsThreads;
    v[k] = i < n ? row[i] : -INFINITY;
  }
#pragma unroll
  for (int k = 0; k < kStatsPer; ++k) m = fmaxf(m, v[k]);
  for (int i = tid + kStatsHeld; i < n; i += kStatsThreads) m = fmaxf(m, row[i]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if (lane == 0) red[warp] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kW; ++w) m = fmaxf(m, red[w]);
  if (!isfinite(m)) m = 0.f;
  float z = 0.f;
#pragma unroll
  for (int k = 0; k < kStatsPer; ++k) z += tid + k * kStatsThreads < n ? __expf(v[k] - m) : 0.f;
  for (int i = tid + kStatsHeld; i < n; i += kStatsThreads) z += __expf(row[i] - m);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) z += __shfl_xor_sync(0xFFFFFFFFu, z, o);
  if (lane == 0) red_z[warp] = z;
  __syncthreads();
  if (tid == 0) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kW; ++w) t += red_z[w];
    out_m[static_cast<int64_t>(b) * H_q + h] = m;
    out_inv_z[static_cast<int64_t>(b) * H_q + h] = t > 0.f ? 1.0f / t : 0.f;
  }
}

template <int DT>
__global__ void merge_correct_kernel(const float* __restrict__ o_hat, const float* __restrict__ o_old,
                                     const float* __restrict__ W, const uint16_t* __restrict__ o_new,
                                     uint16_t* __restrict__ out, int total) {
  pdl_wait();
  pdl_trigger();  // the next kernel may start its prologue; it waits for this grid before reading
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const float w = W[i / JF_HEAD_DIM];
  const float v = o_hat[i] + w * Elem<DT>::to_f32(o_new[i]) - o_old[i];
  out[i] = Elem<DT>::from_f32(v);
}

}  // namespace

}  // namespace jf

extern "C" jf_status_t jf_decode_finish(const jf_decode_args* a, jf_stream_t stream_) {
  using namespace jf;
  jf_status_t st = validate_decode_args(a);
  if (st != JF_OK) return st;
  if (!a->topk_idx || !a->o_hat || !a->o_old_unnorm || !a->W) return JF_ERR_ARG;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int splits = call_splits(a);
  Workspace ws = call_workspace(a, splits);
  FinishParams fp{};
  fp.block_table = a->block_table; fp.seq_lens = a->seq_lens; fp.topk_idx = a->topk_idx;
  fp.max_blocks = a->max_blocks;
  const TailParams tp = make_tail_params(a, ws, splits);
  dim3 grid(a->H_q, a->B);
  if (a->mode == JF_MODE_K3V2) {
    JF_ENSURE_SMEM((decode_finish_kernel<JF_MODE_K3V2>), sizeof(TailSmem<JF_MODE_K3V2>));
    JF_CUDA_TRY(launch_pdl(decode_finish_kernel<JF_MODE_K3V2>, grid, dim3(kFinishThreads), sizeof(TailSmem<JF_MODE_K3V2>), stream, fp, tp));
  } else {
    JF_ENSURE_SMEM((decode_finish_kernel<JF_MODE_K4V4>), sizeof(TailSmem<JF_MODE_K4V4>));
    JF_CUDA_TRY(launch_pdl(decode_finish_kernel<JF_MODE_K4V4>, grid, dim3(kFinishThreads), sizeof(TailSmem<JF_MODE_K4V4>), stream, fp, tp));
  }
  JF_CUDA_TRY(cudaGetLastError());
  return JF_OK;
}

extern "C" jf_status_t jf_softmax_stats(const float* scores, const int32_t* seq_lens, float* softmax_m,
                                        float* softmax_inv_z, int32_t B, int32_t H_q, int32_t max_S,
                                        jf_stream_t stream_) {
  using namespace jf;
  if (!scores || !seq_lens || !softmax_m || !softmax_inv_z || B <= 0 || H_q <= 0 || max_S <= 0) return JF_ERR_ARG;
  JF_CUDA_TRY(launch_pdl(softmax_stats_kernel, dim3(H_q, B), dim3(kStatsThreads), 0, static_cast<cudaStream_t>(stream_), scores,
                         seq_lens, softmax_m, softmax_inv_z, static_cast<int>(H_q), static_cast<int>(max_S)));
  return JF_OK;
}

// scan, then select + finish in one kernel
extern "C" jf_status_t jf_decode_fused(const jf_decode_args* a, jf_stream_t stream) {
  if (a && a->scan_parts != JF_SCAN_ALL) return JF_ERR_ARG;   // the fused step needs both halves
  jf_status_t st = jf_decode_scan(a, stream);
  if (st != JF_OK) return st;
  return jf::launch_select(a, static_cast<cudaStream_t>(stream), true);
}

// select + finish in one kernel, after a scan that ran on its own (the second half of jf_decode_fused)
extern "C" jf_status_t jf_select_finish(const jf_decode_args* a, jf_stream_t stream) {
  if (a && a->scan_parts == JF_SCAN_K_ONLY) return JF_ERR_ARG;   // the finish stage needs the V side
  return jf::launch_select(a, static_cast<cudaStream_t>(stream), true);
}

extern "C" jf_status_t jf_decode_status(const jf_decode_args* a, jf_stream_t stream_) {
  using namespace jf;
  if (!a) return JF_ERR_ARG;
  // no workspace: the calls went through jf_decode_fused_static, whose record is in the built-in array
  void* record = a->workspace;
  if (!record) {
    const jf_status_t st = static_scratch_address(&record);
    if (st != JF_OK) return st;
  }
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  struct { unsigned long long tag; int32_t code; int32_t pad; } host{};
  JF_CUDA_TRY(cudaMemcpyAsync(&host, record, sizeof(host), cudaMemcpyDeviceToHost, stream));
  JF_CUDA_TRY(cudaStreamSynchronize(stream));
  if (host.tag != kStatusTag || host.code == 0) return JF_OK;
  JF_CUDA_TRY(cudaMemsetAsync(record, 0, sizeof(host), stream));
  JF_CUDA_TRY(cudaStreamSynchronize(stream));
  return static_cast<jf_status_t>(host.code);
}

// The same reading on a host copy of the record's first 16 bytes, for callers that bring the
// record over with a copy of their own in the stream (no synchronisation here, nothing cleared).
extern "C" jf_status_t jf_decode_status_of_copy(const void* record_copy) {
  if (!record_copy) return JF_ERR_ARG;
  struct { unsigned long long tag; int32_t code; int32_t pad; } host{};
  memcpy(&host, record_copy, sizeof(host));
  if (host.tag != jf::kStatusTag || host.code == 0) return JF_OK;
  return static_cast<jf_status_t>(host.code);
}

extern "C" jf_status_t jf_merge_correct(const float* o_hat, const float* o_old_unnorm, const float* W,
                                        const void* o_new, void* out, int32_t dtype, int32_t B,
                                        int32_t H_q, jf_stream_t stream_) {
  using namespace jf;
  if (!o_hat || !o_old_unnorm || !W || !o_new || !out || B <= 0 || H_q <= 0) return JF_ERR_ARG;
  cudaStream_t stream = static_cast<cudaStream_t>(stream_);
  const int total = B * H_q * JF_HEAD_DIM;
  const int threads = 256, blocks = (total + threads - 1) / threads;
  if (dtype == JF_DTYPE_BF16)
    JF_CUDA_TRY(launch_pdl(merge_correct_kernel<JF_DTYPE_BF16>, dim3(blocks), dim3(threads), 0, stream, o_hat,
                           o_old_unnorm, W, static_cast<const uint16_t*>(o_new), static_cast<uint16_t*>(out), total));
  else if (dtype == JF_DTYPE_FP16)
    JF_CUDA_TRY(launch_pdl(merge_correct_kernel<JF_DTYPE_FP16>, dim3(blocks), dim3(threads), 0, stream, o_hat,
                           o_old_unnorm, W, static_cast<const uint16_t*>(o_new), static_cast<uint16_t*>(out), total));
  else
    return JF_ERR_UNSUPPORTED;
  return JF_OK;
}
