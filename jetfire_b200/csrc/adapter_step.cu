// The two ends of a stream-ordered decode step of the serving adapter, one kernel each.
//
// Between them lies jf_decode_fused.  The reference's graph-mode decode surrounds its kernels with
// copies, stream memory operations and host functions (jetfire_vllm/adapter/decode_path.py:2253-2492);
// as separate launches these were eleven nodes per layer (three input copies, two downloads, the
// trigger, the wait, the merge, the status download, an event), each with its launch on the host and
// its gap on the device: 170 us of host time a layer, around kernels of 21.
//
// begin  copies the step's inputs to the addresses the kept argument block names -- the query to the
//        device and to the host's copy (mapped pinned memory, posted writes), the block table with its
//        conversion to 64 bits, the lengths -- and clears the completion word.  Bound by launch latency.
// end    raises the trigger word (everything the correction reads has been written by earlier kernels
//        of the stream), waits for the completion word (bounded), merges the correction into the
//        caller's output and hands a recorded error over to the host.  Bound by the host's work.
// The selected slots need no copy: the select kernel writes them to mapped memory itself.
#include "decode_common.cuh"

namespace jf {
namespace {

struct BeginParams {
  const uint4* q;            // rows of 16 B pieces
  int64_t q_stride;          // between sequences, in pieces
  uint4* q_dev;
  uint4* q_host;
  const void* bt;
  int64_t bt_stride;
  int64_t* bt_dev;
  const void* lens;
  int32_t* lens_dev;
  volatile long long* done;
  int B, q_row, width, bt_dev_stride;   // q_row: pieces per sequence
  bool bt_i32, lens_i32;
};

__global__ void __launch_bounds__(256) step_begin_kernel(const BeginParams p) {
  pdl_wait();
  pdl_trigger();   // the next kernel may start its prologue; it waits for this grid before reading
  const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (t0 == 0) *p.done = 0;
  for (int i = t0; i < p.B * p.q_row; i += stride) {
    const int b = i / p.q_row, c = i - b * p.q_row;
    const uint4 v = p.q[b * p.q_stride + c];
    p.q_dev[i] = v;
    p.q_host[i] = v;
  }
  for (int i = t0; i < p.B * p.width; i += stride) {
    const int b = i / p.width, c = i - b * p.width;
    const int64_t at = b * p.bt_stride + c;
    p.bt_dev[static_cast<int64_t>(b) * p.bt_dev_stride + c] =
        p.bt_i32 ? static_cast<int64_t>(static_cast<const int32_t*>(p.bt)[at]) : static_cast<const int64_t*>(p.bt)[at];
  }
  for (int i = t0; i < p.B; i += stride)
    p.lens_dev[i] = p.lens_i32 ? static_cast<const int32_t*>(p.lens)[i] : static_cast<int32_t>(static_cast<const int64_t*>(p.lens)[i]);
}

struct EndParams {
  const float4* o_hat;
  const float4* o_old;
  const float* W;
  const uint2* o_new;        // four 16-bit channels each; mapped host memory or device memory
  uint16_t* out;
  int64_t out_stride;        // between sequences, in elements
  volatile long long* done;
  volatile long long* trigger;   // may be null: the correction was started by an earlier kernel
  int32_t* status;
  uint4* status_host;
  unsigned long long budget_ns;
  int rows, H_q;             // rows = B * H_q
};

constexpr int kEndThreads = 512;   // 16 rows of 32 four-channel pieces at a time
constexpr int kEndRows = 2;        // so often per block: 32 rows are one block, which needs no word from another (1.3 us)

template <int DT>
__global__ void __launch_bounds__(kEndThreads) step_end_kernel(const EndParams p) {
  pdl_wait();      // the kernels that wrote the slots, the query copy and the attention parts are complete
  pdl_trigger();
  // again, and late: a worker of a run that was given up may have set it since the step began (ahead of the loads,
  // so that the fence before the trigger does not wait a trip over the host link for it)
  if (threadIdx.x == 0 && blockIdx.x == 0 && p.trigger != nullptr) *p.done = 0;
  const int row0 = blockIdx.x * (kEndRows * kEndThreads / 32) + (threadIdx.x >> 5), piece = threadIdx.x & 31;
  // what the merge needs besides the correction, while that is on its way
  float4 a[kEndRows], o[kEndRows];
  float w[kEndRows];
#pragma unroll
  for (int k = 0; k < kEndRows; ++k) {
    const int row = row0 + k * (kEndThreads / 32);
    a[k] = o[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    w[k] = 0.f;
    if (row < p.rows) {
      a[k] = p.o_hat[row * 32 + piece];
      o[k] = p.o_old[row * 32 + piece];
      w[k] = p.W[row];
    }
  }
  if (threadIdx.x == 0) {
    volatile int32_t* const verdict = p.status + kWaitWord;
    const unsigned long long t0 = global_ns();
    if (blockIdx.x == 0) {
      // One block waits and decides for the grid: with a budget of its own each, the blocks could differ
      // around the limit, and those of a later wave would start it afresh.
      if (p.trigger != nullptr) {
        __threadfence_system();   // what the correction reads is on the host before the trigger is
        *p.trigger = 1;
      }
      bool ok = false;
      for (unsigned long long polls = 0; polls < (1ull << 32); ++polls) {
        if (*p.done != 0) { ok = true; break; }
        if (global_ns() - t0 > p.budget_ns) break;
        __nanosleep(polls < 64 ? 50 : 400);
      }
      __threadfence_system();     // what the host wrote before the word is read after it, by every block
      *verdict = ok ? kWaitDone : kWaitRanOut;
      if (!ok) report_status(p.status, JF_ERR_TIMEOUT);
      // an error that a kernel of the stream recorded is handed over: the host's copy keeps it until the host
      // has seen it, the record is free again (layers share the workspace, one of them reports)
      volatile int32_t* s = p.status;
      if (*reinterpret_cast<volatile unsigned long long*>(s) == kStatusTag) {
        *p.status_host = make_uint4(s[0], s[1], s[2], s[3]);
        s[0] = s[1] = 0;
      }
    } else {
      // block 0 started with this one or before it and gives up within the budget
      for (unsigned long long polls = 0; polls < (1ull << 32); ++polls) {
        if (*verdict != 0 || global_ns() - t0 > p.budget_ns + 1000000000ull) break;
        __nanosleep(20);
      }
      __threadfence_system();
    }
  }
  __syncthreads();
  uint32_t n0[kEndRows], n1[kEndRows];
#pragma unroll
  for (int k = 0; k < kEndRows; ++k) {
    const int row = row0 + k * (kEndThreads / 32);
    n0[k] = n1[k] = 0u;
    if (row < p.rows) {
      const volatile uint32_t* nw = reinterpret_cast<const volatile uint32_t*>(p.o_new + row * 32 + piece);
      n0[k] = nw[0];
      n1[k] = nw[1];
    }
  }
#pragma unroll
  for (int k = 0; k < kEndRows; ++k) {
    const int row = row0 + k * (kEndThreads / 32);
    if (row >= p.rows) break;
    const float n[4] = {Elem<DT>::to_f32(static_cast<uint16_t>(n0[k] & 0xFFFFu)), Elem<DT>::to_f32(static_cast<uint16_t>(n0[k] >> 16)),
                        Elem<DT>::to_f32(static_cast<uint16_t>(n1[k] & 0xFFFFu)), Elem<DT>::to_f32(static_cast<uint16_t>(n1[k] >> 16))};
    const float h[4] = {a[k].x, a[k].y, a[k].z, a[k].w}, old[4] = {o[k].x, o[k].y, o[k].z, o[k].w};
    uint16_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) r[i] = Elem<DT>::from_f32(h[i] + w[k] * n[i] - old[i]);
    const int b = row / p.H_q, hq = row - b * p.H_q;
    uint2* dst = reinterpret_cast<uint2*>(p.out + b * p.out_stride + hq * JF_HEAD_DIM) + piece;
    *dst = make_uint2(r[0] | (static_cast<uint32_t>(r[1]) << 16), r[2] | (static_cast<uint32_t>(r[3]) << 16));
  }
}

}  // namespace
}  // namespace jf

extern "C" jf_status_t jf_step_begin(const void* q, int64_t q_stride, void* q_dev, void* q_host_dev, const void* block_table,
                                     int32_t bt_is_i32, int64_t bt_stride, int32_t width, int64_t* bt_dev,
                                     int32_t bt_dev_stride, const void* seq_lens, int32_t lens_are_i32, int32_t* lens_dev,
                                     int64_t* done_dev, int32_t B, int32_t H_q, jf_stream_t stream) {
  using namespace jf;
  if (!q || !q_dev || !q_host_dev || !block_table || !bt_dev || !seq_lens || !lens_dev || !done_dev) return JF_ERR_ARG;
  if (B <= 0 || H_q <= 0 || width < 0 || width > bt_dev_stride || (q_stride & 7)) return JF_ERR_ARG;
  if (!aligned(q, 16) || !aligned(q_dev, 16) || !aligned(q_host_dev, 16)) return JF_ERR_ARG;
  if (static_cast<int64_t>(B) * H_q * 16 > 0x7FFFFFFF || static_cast<int64_t>(B) * width > 0x7FFFFFFF) return JF_ERR_UNSUPPORTED;
  BeginParams p{static_cast<const uint4*>(q), q_stride / 8, static_cast<uint4*>(q_dev), static_cast<uint4*>(q_host_dev),
                block_table, bt_stride, bt_dev, seq_lens, lens_dev, reinterpret_cast<volatile long long*>(done_dev),
                B, H_q * 16, width, bt_dev_stride, bt_is_i32 != 0, lens_are_i32 != 0};
  const int items = B * (H_q * 16 > width ? H_q * 16 : width), blocks = (items + 255) / 256, most = 2 * num_sms();
  JF_CUDA_TRY(launch_pdl(step_begin_kernel, dim3(blocks < most ? blocks : most), dim3(256), 0, static_cast<cudaStream_t>(stream), p));
  return JF_OK;
}

extern "C" jf_status_t jf_step_end(const float* o_hat, const float* o_old_unnorm, const float* W, const void* o_new, void* out,
                                   int64_t out_stride, int32_t dtype, int32_t B, int32_t H_q, int64_t* done_dev,
                                   int64_t* trigger_dev, int32_t timeout_ms, void* status_record, void* status_host_dev,
                                   jf_stream_t stream) {
  using namespace jf;
  if (!o_hat || !o_old_unnorm || !W || !o_new || !out || !done_dev || !status_record || !status_host_dev) return JF_ERR_ARG;
  if (B <= 0 || H_q <= 0 || timeout_ms <= 0 || timeout_ms > 60000) return JF_ERR_ARG;
  if (!aligned(o_hat, 16) || !aligned(o_old_unnorm, 16) || !aligned(o_new, 8) || !aligned(out, 8) || (out_stride & 3) ||
      !aligned(status_record, 16) || !aligned(status_host_dev, 16))
    return JF_ERR_ARG;
  if (dtype != JF_DTYPE_BF16 && dtype != JF_DTYPE_FP16) return JF_ERR_UNSUPPORTED;
  if (static_cast<int64_t>(B) * H_q > (1 << 25)) return JF_ERR_UNSUPPORTED;
  EndParams p{reinterpret_cast<const float4*>(o_hat), reinterpret_cast<const float4*>(o_old_unnorm), W,
              static_cast<const uint2*>(o_new), static_cast<uint16_t*>(out), out_stride,
              reinterpret_cast<volatile long long*>(done_dev), reinterpret_cast<volatile long long*>(trigger_dev),
              static_cast<int32_t*>(status_record), static_cast<uint4*>(status_host_dev),
              static_cast<unsigned long long>(timeout_ms) * 1000000ull, B * H_q, H_q};
  constexpr int per_block = kEndRows * kEndThreads / 32;
  const dim3 grid((B * H_q + per_block - 1) / per_block);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  JF_CUDA_TRY(dtype == JF_DTYPE_BF16 ? launch_pdl(step_end_kernel<JF_DTYPE_BF16>, grid, dim3(kEndThreads), 0, s, p)
                                     : launch_pdl(step_end_kernel<JF_DTYPE_FP16>, grid, dim3(kEndThreads), 0, s, p));
  return JF_OK;
}
