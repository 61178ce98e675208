// Python module `jetfire_b200._host`: the tensor-taking half of jetfire_b200/ops.py in native code.
//
// The operator surface takes torch tensors, checks them as the reference's TORCH_CHECKs do
// (jetfire_vllm/csrc/*.cu, *.cpp) and hands plain pointers to the C ABI.  In Python those checks
// and the ctypes conversions cost more than the kernels of a small call: 18 us for an append of
// eight tokens whose kernel takes 1.6, 58 us for the one-shot attention op whose kernels take 21.
// The same checks here take about a microsecond; what is left is the launches.
//
// Functions take positional arguments only (METH_FASTCALL) and return the C ABI's status, or a
// tuple that starts with it; ops.py turns a status into its exception.  Argument errors raise
// RuntimeError from here.  Launches run with the interpreter lock released: a full launch queue
// blocks only the calling thread.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty_like.h>
#include <ATen/ops/empty.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "../../include/jetfire_b200.h"

namespace {

struct ArgError {};   // a Python exception is set

[[noreturn]] void fail(const char* name, const char* what) {
  PyErr_Format(PyExc_RuntimeError, "%s: %s", name, what);
  throw ArgError();
}
inline void require(bool ok, const char* name, const char* what) {
  if (!ok) fail(name, what);
}

const at::Tensor& tensor(PyObject* o, const char* name, const char* what) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_RuntimeError, "%s: %s must be a tensor", name, what);
    throw ArgError();
  }
  return THPVariable_Unpack(o);
}
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw ArgError();
  return v;
}
int32_t int32(PyObject* o) {
  const int64_t v = integer(o);
  if (v < INT32_MIN || v > INT32_MAX) {
    PyErr_SetString(PyExc_OverflowError, "argument does not fit 32 bits");
    throw ArgError();
  }
  return static_cast<int32_t>(v);
}
// What int(x) and float(x) take, where the op's Python form converted its arguments with them.
struct Owned {
  PyObject* o;
  explicit Owned(PyObject* p) : o(p) { if (!o) throw ArgError(); }
  ~Owned() { Py_DECREF(o); }
};
int32_t as_int32(PyObject* o) {
  if (PyLong_CheckExact(o)) return int32(o);
  return int32(Owned(PyNumber_Long(o)).o);
}
double real(PyObject* o) {
  if (PyFloat_CheckExact(o)) return PyFloat_AS_DOUBLE(o);
  return PyFloat_AS_DOUBLE(Owned(PyNumber_Float(o)).o);
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw ArgError();
  return v != 0;
}
const char* text(PyObject* o) {
  const char* s = PyUnicode_AsUTF8(o);
  if (!s) throw ArgError();
  return s;
}
int dtype_id(const at::Tensor& t) {
  if (t.scalar_type() == at::kBFloat16) return JF_DTYPE_BF16;
  if (t.scalar_type() == at::kHalf) return JF_DTYPE_FP16;
  PyErr_Format(PyExc_RuntimeError, "expected bfloat16 or float16, got %s", c10::toString(t.scalar_type()));
  throw ArgError();
}
// Addresses are taken with the interpreter lock held: a tensor without storage (a fake, functional or batched
// one) throws here.  `out_ptr`: of memory that is written (a lazily copied tensor gets its own first).
inline const void* ptr(const at::Tensor& t) { return t.const_data_ptr(); }
inline void* out_ptr(const at::Tensor& t) { return t.mutable_data_ptr(); }
inline uint8_t* out_bytes(const at::Tensor& t) { return static_cast<uint8_t*>(out_ptr(t)); }
inline jf_stream_t current_stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// The contiguous form of a tensor, kept alive in `keep` when it is a copy.
inline const at::Tensor& contiguous(const at::Tensor& t, at::Tensor& keep) {
  if (t.is_contiguous()) return t;
  keep = t.contiguous();
  return keep;
}

// `f` must not throw: it runs without the interpreter lock.
template <typename F> jf_status_t unlocked(F&& f) {
  jf_status_t st;
  Py_BEGIN_ALLOW_THREADS
  st = f();
  Py_END_ALLOW_THREADS
  return st;
}

// Runs a function body; Python errors and C++ exceptions become a raised exception.
template <typename F> PyObject* guarded(F&& body) {
  HANDLE_TH_ERRORS
  try {
    return body();
  } catch (const ArgError&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

void expect_args(Py_ssize_t n, Py_ssize_t want, const char* name) {
  if (n != want) {
    PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, got %zd", name, want, n);
    throw ArgError();
  }
}

// ---- quantise-on-append -----------------------------------------------------------------

void check_side(const at::Tensor& x, const at::Tensor& data, const at::Tensor& scale, int nbits, int64_t group, const char* name) {
  require(x.is_cuda() && data.is_cuda() && scale.is_cuda(), name, "tensors must be CUDA");
  require(x.dim() == 3 && x.size(2) == JF_HEAD_DIM, name, "x_tok must be (T, H_kv, 128)");
  require(x.stride(2) == 1, name, "x_tok innermost dim must be contiguous");
  require(data.scalar_type() == at::kByte && data.is_contiguous(), name, "out_data must be contiguous uint8");
  require(scale.scalar_type() == at::kBFloat16 && scale.is_contiguous(), name, "out_scale must be contiguous bf16");
  require(group == 64 || group == 128, name, "group_size must be 64 or 128");
  const int64_t h = x.size(1);
  if (!(data.dim() == 3 && data.size(0) == h && data.size(2) == 16 * nbits)) {
    PyErr_Format(PyExc_RuntimeError, "%s: out_data must be (H_kv, num_slots, %d)", name, 16 * nbits);
    throw ArgError();
  }
  if (!(scale.dim() >= 2 && scale.size(0) == h && scale.size(1) == data.size(1) &&
        scale.numel() == h * data.size(1) * (JF_HEAD_DIM / group))) {
    PyErr_Format(PyExc_RuntimeError, "%s: out_scale must be (H_kv, num_slots, %d)", name, static_cast<int>(JF_HEAD_DIM / group));
    throw ArgError();
  }
}
void check_slots(const at::Tensor& slots, int64_t T, const char* name) {
  require(slots.is_cuda() && slots.scalar_type() == at::kLong && slots.dim() == 1 && slots.size(0) == T, name,
          "slot_idx must be (T,) int64 CUDA");
}

// quant_write(name, x_tok, slot_idx, out_data, out_scale, group_size, nbits)
PyObject* quant_write(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 7, "quant_write");
    const char* name = text(a[0]);
    const at::Tensor &x = tensor(a[1], name, "x_tok"), &slots_in = tensor(a[2], name, "slot_idx"),
                     &data = tensor(a[3], name, "out_data"), &scale = tensor(a[4], name, "out_scale");
    const int64_t group = integer(a[5]);
    const int nbits = int32(a[6]);
    check_side(x, data, scale, nbits, group, name);
    check_slots(slots_in, x.size(0), name);
    at::Tensor keep;
    const at::Tensor& slots = contiguous(slots_in, keep);
    const int dt = dtype_id(x);
    const jf_stream_t st = current_stream();
    const void* xp = ptr(x);
    const int64_t T = x.size(0), st_t = x.stride(0), st_h = x.stride(1), num_slots = data.size(1);
    const auto h = static_cast<int32_t>(x.size(1));
    const auto* sl = static_cast<const int64_t*>(ptr(slots));
    uint8_t* dp = out_bytes(data);
    void* sp = out_ptr(scale);
    return PyLong_FromLong(unlocked([&] {
      return jf_pack_append(xp, dt, T, h, st_t, st_h, sl, dp, sp, num_slots, nbits, static_cast<int32_t>(group), st);
    }));
  });
}

void check_mirror(const at::Tensor& m, const at::Tensor& key, const at::Tensor& k_data, const char* name) {
  require(m.is_cuda() && m.is_contiguous() && m.scalar_type() == key.scalar_type() && m.dim() == 3 && m.size(0) == k_data.size(0) &&
              m.size(1) == k_data.size(1) && m.size(2) == JF_HEAD_DIM,
          name, "mirror must be a contiguous device-visible (H_kv, num_slots, 128) tensor of the tokens' dtype");
}

// quant_write_kv(name, key, value, slot_idx, k_data, k_scales, v_data, v_scales, group_size, k_bits, v_bits,
//                k_mirror | None, v_mirror | None, filled | None)
PyObject* quant_write_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 14, "quant_write_kv");
    const char* name = text(a[0]);
    const at::Tensor &key = tensor(a[1], name, "key_tok"), &value = tensor(a[2], name, "value_tok"),
                     &slots_in = tensor(a[3], name, "slot_idx"), &kd = tensor(a[4], name, "k_data"),
                     &ks = tensor(a[5], name, "k_scales"), &vd = tensor(a[6], name, "v_data"), &vs = tensor(a[7], name, "v_scales");
    const int64_t group = integer(a[8]);
    const int kb = int32(a[9]), vb = int32(a[10]);
    check_side(key, kd, ks, kb, group, name);
    check_side(value, vd, vs, vb, group, name);
    require(key.sizes() == value.sizes() && key.scalar_type() == value.scalar_type(), name, "key/value shape or dtype mismatch");
    require(kd.size(1) == vd.size(1), name, "K and V caches differ in num_slots");
    check_slots(slots_in, key.size(0), name);
    const bool mirrored = a[11] != Py_None;
    void *km = nullptr, *vm = nullptr;
    if (mirrored) {
      const at::Tensor &k_mirror = tensor(a[11], name, "k_mirror_dev"), &v_mirror = tensor(a[12], name, "v_mirror_dev");
      check_mirror(k_mirror, key, kd, name);
      check_mirror(v_mirror, key, kd, name);
      km = out_ptr(k_mirror);
      vm = out_ptr(v_mirror);
    }
    uint8_t* filled = nullptr;
    if (a[13] != Py_None) {
      const at::Tensor& f = tensor(a[13], name, "filled");
      require(f.is_cuda() && f.is_contiguous() && f.element_size() == 1 && f.numel() >= kd.size(1), name,
              "filled must hold a byte per slot");
      filled = out_bytes(f);
    }
    at::Tensor keep;
    const at::Tensor& slots = contiguous(slots_in, keep);
    const int dt = dtype_id(key);
    const jf_stream_t st = current_stream();
    const auto* sl = static_cast<const int64_t*>(ptr(slots));
    const auto h = static_cast<int32_t>(key.size(1));
    const int64_t T = key.size(0), num_slots = kd.size(1), k_t = key.stride(0), k_h = key.stride(1), v_t = value.stride(0),
                  v_h = value.stride(1);
    const void *kp = ptr(key), *vp = ptr(value);
    uint8_t *kdp = out_bytes(kd), *vdp = out_bytes(vd);
    void *ksp = out_ptr(ks), *vsp = out_ptr(vs);
    return PyLong_FromLong(unlocked([&] {
      if (mirrored || filled)
        return jf_store_append(kp, vp, dt, T, h, k_t, k_h, v_t, v_h, sl, kdp, ksp, vdp, vsp, num_slots, kb, vb,
                               static_cast<int32_t>(group), km, vm, filled, st);
      return jf_pack_append_kv(kp, vp, dt, T, h, k_t, k_h, v_t, v_h, sl, kdp, ksp, vdp, vsp, num_slots, kb, vb,
                               static_cast<int32_t>(group), st);
    }));
  });
}

// ---- decode attention -------------------------------------------------------------------

struct ModeShape { int k_bits, v_bits, groups; };
ModeShape mode_shape(int mode, const char* name) {
  require(mode == JF_MODE_K3V2 || mode == JF_MODE_K4V4, name, "unknown mode");
  return mode == JF_MODE_K3V2 ? ModeShape{3, 2, 2} : ModeShape{4, 4, 1};
}

inline bool capturing_now() { return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None; }

// Scratch per (device, stream): grows as needed, one block per pair, bounded in number (the blocks go
// back to the caching allocator when the table is cleared, which is safe in the order of the stream).
// A call that is being captured gets a block of its own from the graph's pool, as any temporary of the
// capture does: the graph keeps its address, and the table's block may be replaced or given back.
at::Tensor workspace(uint64_t bytes, c10::Device device) {
  static std::mutex mu;
  static auto* table = new std::map<std::pair<int, void*>, at::Tensor>();   // never destroyed: outlives the CUDA context at exit
  constexpr size_t kMaxEntries = 64;
  const int index = device.has_index() ? device.index() : c10::cuda::current_device();
  auto fresh = [&] {
    return at::detail::empty_cuda({static_cast<int64_t>(bytes) + 256}, at::kByte, c10::Device(c10::kCUDA, index), c10::nullopt);
  };
  if (capturing_now()) return fresh();
  const std::pair<int, void*> key(index, current_stream());
  std::lock_guard<std::mutex> lock(mu);
  auto it = table->find(key);
  if (it != table->end() && static_cast<uint64_t>(it->second.numel()) >= bytes) return it->second;
  if (it == table->end() && table->size() >= kMaxEntries) table->clear();
  at::Tensor t = fresh();
  (*table)[key] = t;
  return t;
}

// What a decode call is made of: the argument block and the tensors whose addresses it holds.
struct Decode {
  jf_decode_args a{};
  at::Tensor keep[7];   // contiguous copies, workspace
  int64_t B = 0, H_q = 0;
  c10::Device device{c10::kCUDA, 0};

  void common(int mode, const at::Tensor& block_table, const at::Tensor& seq_lens, int64_t max_S, int64_t h_q, int64_t h_kv,
              int64_t block_size, int64_t top_k, double scale, const char* name) {
    require(block_table.is_cuda() && seq_lens.is_cuda(), name, "block_table / seq_lens must be CUDA");
    device = block_table.device();
    require(seq_lens.dim() == 1, name, "seq_lens must be (B,) int32");
    B = seq_lens.size(0);
    H_q = h_q;
    require(block_table.scalar_type() == at::kLong && block_table.dim() == 2 && block_table.size(0) == B, name,
            "block_table must be (B, max_blocks) int64");
    require(seq_lens.scalar_type() == at::kInt, name, "seq_lens must be (B,) int32");
    a.mode = mode;
    a.q_dtype = JF_DTYPE_BF16;
    a.B = static_cast<int32_t>(B); a.H_q = static_cast<int32_t>(h_q); a.H_kv = static_cast<int32_t>(h_kv);
    a.max_S = static_cast<int32_t>(max_S); a.block_size = static_cast<int32_t>(block_size); a.top_k = static_cast<int32_t>(top_k);
    a.max_blocks = static_cast<int32_t>(block_table.size(1));
    a.attn_scale = static_cast<float>(scale);
    a.block_table = static_cast<const int64_t*>(ptr(contiguous(block_table, keep[0])));
    a.seq_lens = static_cast<const int32_t*>(ptr(contiguous(seq_lens, keep[1])));
  }
  void side(const at::Tensor& data, const at::Tensor& scales, int bits, int groups, bool k_side, const char* name) {
    require(data.is_cuda() && scales.is_cuda(), name, "cache tensors must be CUDA");
    require(data.scalar_type() == at::kByte && scales.scalar_type() == at::kBFloat16, name, "packed data must be uint8, scales bf16");
    require(data.is_contiguous() && scales.is_contiguous(), name, "cache tensors must be contiguous");
    if (!(data.dim() == 3 && data.size(0) == a.H_kv && data.size(2) == 16 * bits)) {
      PyErr_Format(PyExc_RuntimeError, "%s: %s must be (H_kv, num_slots, %d)", name, k_side ? "k_data" : "v_data", 16 * bits);
      throw ArgError();
    }
    require(a.num_slots == 0 || a.num_slots == data.size(1), name, "K and V caches differ in num_slots");
    a.num_slots = data.size(1);
    if (scales.numel() != a.H_kv * a.num_slots * groups) {
      PyErr_Format(PyExc_RuntimeError, "%s: scales must hold %d group(s) per slot", name, groups);
      throw ArgError();
    }
    if (k_side) { a.k_data = static_cast<const uint8_t*>(ptr(data)); a.k_scales = ptr(scales); }
    else { a.v_data = static_cast<const uint8_t*>(ptr(data)); a.v_scales = ptr(scales); }
  }
  void query(const at::Tensor& q, const char* name) {
    require(q.is_cuda(), name, "q must be CUDA");
    require(q.dim() == 3 && q.size(0) == B && q.size(1) == H_q && q.size(2) == JF_HEAD_DIM, name, "q must be (B, H_q, 128)");
    a.q_dtype = dtype_id(q);
    a.q = ptr(contiguous(q, keep[2]));
  }
  void scratch(PyObject* given, const char* name) {
    const uint64_t bytes = jf_decode_workspace_useful_bytes(a.mode, a.B, a.H_q, a.H_kv, a.max_S, a.top_k);
    require(bytes > 0, name, "bad shape");
    keep[3] = given && given != Py_None ? tensor(given, name, "workspace") : workspace(bytes, device);
    const auto base = reinterpret_cast<uintptr_t>(out_ptr(keep[3])), at = (base + 255) / 256 * 256;
    a.workspace = reinterpret_cast<void*>(at);
    a.workspace_bytes = static_cast<uint64_t>(keep[3].numel()) * keep[3].element_size() - (at - base);
  }
  at::Tensor f32(at::IntArrayRef shape) { return at::detail::empty_cuda(shape, at::kFloat, device, c10::nullopt); }
  at::Tensor i64(at::IntArrayRef shape) { return at::detail::empty_cuda(shape, at::kLong, device, c10::nullopt); }
};

PyObject* tuple_of(jf_status_t st, std::initializer_list<at::Tensor> tensors) {
  PyObject* r = PyTuple_New(1 + static_cast<Py_ssize_t>(tensors.size()));
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, PyLong_FromLong(st));
  Py_ssize_t i = 1;
  for (const at::Tensor& t : tensors) PyTuple_SET_ITEM(r, i++, THPVariable_Wrap(t));   // None for an undefined tensor
  return r;
}

// fused_attn(name, mode, q, k_data, k_scales, v_data, v_scales, block_table, seq_lens, max_S, H_q, H_kv, block_size,
//            top_k, attn_scale, workspace | None, want_scores, stage_b)
//   -> (status, o_hat, topk_slots, o_old_unnorm, W, topk_idx, softmax_m, softmax_inv_z, scores | None)
PyObject* fused_attn(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 18, "fused_attn");
    const char* name = text(p[0]);
    const int mode = int32(p[1]);
    const ModeShape m = mode_shape(mode, name);
    Decode d;
    d.common(mode, tensor(p[7], name, "block_table"), tensor(p[8], name, "seq_lens"), int32(p[9]), int32(p[10]), int32(p[11]),
             as_int32(p[12]), int32(p[13]), real(p[14]), name);
    d.query(tensor(p[2], name, "q"), name);
    d.side(tensor(p[3], name, "k_data"), tensor(p[4], name, "k_scales"), m.k_bits, m.groups, true, name);
    d.side(tensor(p[5], name, "v_data"), tensor(p[6], name, "v_scales"), m.v_bits, m.groups, false, name);
    d.scratch(p[15], name);
    d.a.stage_b = int32(p[17]);
    const int64_t B = d.B, H = d.H_q, K = d.a.top_k;
    at::Tensor o_hat = d.f32({B, H, JF_HEAD_DIM}), o_old = d.f32({B, H, JF_HEAD_DIM}), W = d.f32({B, H}), sm = d.f32({B, H}),
               inv = d.f32({B, H}), slots = d.i64({B, H, K}), idx = d.i64({B, H, K}), scores;
    if (truth(p[16])) scores = d.f32({B, H, d.a.max_S});
    d.a.o_hat = static_cast<float*>(out_ptr(o_hat)); d.a.o_old_unnorm = static_cast<float*>(out_ptr(o_old));
    d.a.W = static_cast<float*>(out_ptr(W)); d.a.softmax_m = static_cast<float*>(out_ptr(sm)); d.a.softmax_inv_z = static_cast<float*>(out_ptr(inv));
    d.a.topk_slots = static_cast<int64_t*>(out_ptr(slots)); d.a.topk_idx = static_cast<int64_t*>(out_ptr(idx));
    if (scores.defined()) d.a.scores = static_cast<float*>(out_ptr(scores));
    const jf_stream_t st = current_stream();
    const jf_status_t r = unlocked([&] { return jf_decode_fused(&d.a, st); });
    return tuple_of(r, {o_hat, slots, o_old, W, idx, sm, inv, scores});
  });
}

// stage_a(name, mode, q, k_data, k_scales, block_table, seq_lens, max_S, H_q, H_kv, block_size, attn_scale, top_k, stats)
//   -> (status, scores, topk_idx, topk_slots[, softmax_m, softmax_inv_z])
PyObject* stage_a(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 14, "stage_a");
    const char* name = text(p[0]);
    const int mode = int32(p[1]);
    const ModeShape m = mode_shape(mode, name);
    require(as_int32(p[10]) == JF_BLOCK_SIZE, name, "block_size must be 16");
    Decode d;
    d.common(mode, tensor(p[5], name, "block_table"), tensor(p[6], name, "seq_lens"), as_int32(p[7]), as_int32(p[8]), as_int32(p[9]),
             JF_BLOCK_SIZE, as_int32(p[12]), real(p[11]), name);
    d.query(tensor(p[2], name, "q"), name);
    d.side(tensor(p[3], name, "k_data"), tensor(p[4], name, "k_scales"), m.k_bits, m.groups, true, name);
    d.scratch(nullptr, name);
    d.a.scan_parts = JF_SCAN_K_ONLY;
    const bool stats = truth(p[13]);
    const int64_t B = d.B, H = d.H_q, K = d.a.top_k;
    at::Tensor scores = d.f32({B, H, d.a.max_S}), slots = d.i64({B, H, K}), idx = d.i64({B, H, K}), sm, inv;
    if (stats) { sm = d.f32({B, H}); inv = d.f32({B, H}); }
    d.a.scores = static_cast<float*>(out_ptr(scores));
    d.a.topk_slots = static_cast<int64_t*>(out_ptr(slots)); d.a.topk_idx = static_cast<int64_t*>(out_ptr(idx));
    const jf_stream_t st = current_stream();
    float *smp = stats ? static_cast<float*>(out_ptr(sm)) : nullptr, *invp = stats ? static_cast<float*>(out_ptr(inv)) : nullptr;
    const jf_status_t r = unlocked([&] {
      jf_status_t s = jf_decode_scan(&d.a, st);
      if (s == JF_OK) s = jf_topk_select(&d.a, st);
      if (s == JF_OK && stats)
        s = jf_softmax_stats(d.a.scores, d.a.seq_lens, smp, invp, d.a.B, d.a.H_q, d.a.max_S, st);
      return s;
    });
    return stats ? tuple_of(r, {scores, idx, slots, sm, inv}) : tuple_of(r, {scores, idx, slots});
  });
}

// stage_b(name, mode, stage_b, scores, v_data, v_scales, block_table, seq_lens, topk_idx, max_S, H_q, H_kv, block_size,
//         top_k, (o_hat, o_old_unnorm, W) | None) -> (status, o_hat, o_old_unnorm, W)
PyObject* stage_b(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 15, "stage_b");
    const char* name = text(p[0]);
    const int mode = int32(p[1]);
    const ModeShape m = mode_shape(mode, name);
    require(as_int32(p[12]) == JF_BLOCK_SIZE, name, "block_size must be 16");
    const at::Tensor &scores_in = tensor(p[3], name, "scores"), &idx_in = tensor(p[8], name, "topk_idx");
    require(scores_in.is_cuda() && scores_in.scalar_type() == at::kFloat && scores_in.dim() == 3, name, "scores must be f32 (B,H_q,max_S)");
    const int64_t K = as_int32(p[13]);
    require(idx_in.is_cuda() && idx_in.scalar_type() == at::kLong && idx_in.dim() == 3 && idx_in.size(2) == K, name,
            "topk_idx must be int64 (B,H_q,top_k)");
    Decode d;
    d.common(mode, tensor(p[6], name, "block_table"), tensor(p[7], name, "seq_lens"), as_int32(p[9]), as_int32(p[10]), as_int32(p[11]),
             JF_BLOCK_SIZE, K, 1.0, name);
    d.side(tensor(p[4], name, "v_data"), tensor(p[5], name, "v_scales"), m.v_bits, m.groups, false, name);
    const int64_t B = d.B, H = d.H_q;
    require(scores_in.size(0) == B && scores_in.size(1) == H && scores_in.size(2) == d.a.max_S, name,
            "scores must be contiguous f32 (B, H_q, max_S)");
    require(idx_in.size(0) == B && idx_in.size(1) == H, name, "topk_idx must be contiguous int64 (B, H_q, k)");
    d.scratch(nullptr, name);
    d.a.scan_parts = JF_SCAN_V_ONLY;
    d.a.stage_b = int32(p[2]);
    // inputs here: the argument block's type has them writable
    d.a.scores = static_cast<float*>(const_cast<void*>(ptr(contiguous(scores_in, d.keep[4]))));
    d.a.topk_idx = static_cast<int64_t*>(const_cast<void*>(ptr(contiguous(idx_in, d.keep[5]))));
    at::Tensor out[3];
    if (p[14] != Py_None) {
      const int64_t want[3] = {B * H * JF_HEAD_DIM, B * H * JF_HEAD_DIM, B * H};
      for (int i = 0; i < 3; ++i) {
        out[i] = tensor(PyTuple_GetItem(p[14], i), name, "output");
        const bool shape = out[i].dim() == (i < 2 ? 3 : 2) && out[i].size(0) == B && out[i].size(1) == H && out[i].numel() == want[i];
        require(out[i].is_cuda() && out[i].scalar_type() == at::kFloat && out[i].is_contiguous() && shape, name,
                "outputs must be contiguous f32 of shapes (B,H_q,128), (B,H_q,128), (B,H_q)");
      }
    } else {
      out[0] = d.f32({B, H, JF_HEAD_DIM});
      out[1] = d.f32({B, H, JF_HEAD_DIM});
      out[2] = d.f32({B, H});
    }
    d.a.o_hat = static_cast<float*>(out_ptr(out[0])); d.a.o_old_unnorm = static_cast<float*>(out_ptr(out[1]));
    d.a.W = static_cast<float*>(out_ptr(out[2]));
    const jf_stream_t st = current_stream();
    const jf_status_t r = unlocked([&] {
      const jf_status_t s = jf_decode_scan(&d.a, st);
      return s == JF_OK ? jf_decode_finish(&d.a, st) : s;
    });
    return tuple_of(r, {out[0], out[1], out[2]});
  });
}

// decode(which, address of a jf_decode_args) -> status: the phases of a kept call (ops.DecodeCall)
PyObject* decode(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 2, "decode");
    const int which = int32(p[0]);
    const auto* a = reinterpret_cast<const jf_decode_args*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLong(p[1])));
    const jf_stream_t st = current_stream();
    return PyLong_FromLong(unlocked([&] {
      switch (which) {
        case 0: return jf_decode_fused(a, st);
        case 1: return jf_decode_scan(a, st);
        case 2: return jf_topk_select(a, st);
        case 3: return jf_decode_finish(a, st);
        case 4: return jf_select_finish(a, st);
        default: return static_cast<jf_status_t>(JF_ERR_ARG);
      }
    }));
  });
}

// get_workspace(nbytes, tensor or None whose device counts) -> uint8 tensor
PyObject* get_workspace(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 2, "get_workspace");
    return THPVariable_Wrap(workspace(static_cast<uint64_t>(integer(p[0])), c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(integer(p[1])))));
  });
}

// ---- correction merge -------------------------------------------------------------------

// blend(name, o_hat, o_old_unnorm, W, o_new, out) -> status
PyObject* blend(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    expect_args(n, 6, "blend");
    const char* name = text(p[0]);
    const at::Tensor &o_hat = tensor(p[1], name, "o_hat"), &o_old = tensor(p[2], name, "o_old_unnorm"), &W = tensor(p[3], name, "W"),
                     &o_new = tensor(p[4], name, "o_new"), &out = tensor(p[5], name, "out");
    require(o_hat.is_cuda() && o_old.is_cuda() && W.is_cuda() && o_new.is_cuda() && out.is_cuda(), name, "all tensors must be CUDA");
    require(o_hat.scalar_type() == at::kFloat && o_old.scalar_type() == at::kFloat && W.scalar_type() == at::kFloat, name,
            "o_hat, o_old_unnorm, W must be float32");
    require(o_new.scalar_type() == out.scalar_type(), name, "o_new and out dtypes differ");
    require(o_hat.dim() == 3 && o_old.dim() == 3 && o_new.dim() == 3 && out.dim() == 3 && W.dim() == 2, name,
            "tensors must be 3D (W 2D)");
    require(out.is_contiguous(), name, "out must be contiguous");
    const auto shape = o_hat.sizes();
    require(o_old.sizes() == shape && o_new.sizes() == shape && out.sizes() == shape && W.size(0) == shape[0] && W.size(1) == shape[1] &&
                shape[2] == JF_HEAD_DIM,
            name, "shape mismatch");
    at::Tensor keep[4];
    const auto* a = static_cast<const float*>(ptr(contiguous(o_hat, keep[0])));
    const auto* b = static_cast<const float*>(ptr(contiguous(o_old, keep[1])));
    const auto* w = static_cast<const float*>(ptr(contiguous(W, keep[2])));
    const void* nw = ptr(contiguous(o_new, keep[3]));
    const int dt = dtype_id(out);
    const jf_stream_t st = current_stream();
    void* op = out_ptr(out);
    const auto B = static_cast<int32_t>(shape[0]), H = static_cast<int32_t>(shape[1]);
    return PyLong_FromLong(unlocked([&] { return jf_merge_correct(a, b, w, nw, op, dt, B, H, st); }));
  });
}

// ---- the adapter's decode step ----------------------------------------------------------

// Everything of a kept step that does not change from call to call.
struct Step {
  const jf_decode_args* a;
  at::Tensor q, block_table, seq_lens;      // device buffers the argument block names
  at::Tensor keep[8];                       // mapped views and outputs whose addresses follow
  void *q_dev, *q_host_dev, *o_new_dev, *status_host_dev;
  int64_t* bt_dev;
  int32_t *lens_dev, bt_dev_stride;
  void* status_host;
  int64_t *done_dev, *trigger_dev;
  int64_t ctx;                              // submit context of the host correction
  int64_t H_q;
  int32_t timeout_ms;
  // rows [cut, rows) of the correction on the GPU, when cut < rows
  const void *k_mirror = nullptr, *v_mirror = nullptr, *slots = nullptr;
  int32_t slots_i32 = 0;
  int64_t cut = 0, rows = 0;
};
constexpr const char* kStepName = "jetfire_b200._host.Step";
void step_free(PyObject* o) { delete static_cast<Step*>(PyCapsule_GetPointer(o, kStepName)); }

// step_create(address of the jf_decode_args, q, block_table, seq_lens, q_host_dev, o_new_dev, words_dev (int64: trigger at
//   0, completion at 8), status_host (CPU), status_host_dev, submit context, timeout_ms,
//   (k_mirror_dev, v_mirror_dev, slots_dev, cut) | None) -> capsule
PyObject* step_create(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    const char* name = "decode_step";
    expect_args(n, 12, "step_create");
    auto* s = new Step();
    PyObject* cap = PyCapsule_New(s, kStepName, step_free);
    if (!cap) { delete s; return nullptr; }
    try {
      s->a = reinterpret_cast<const jf_decode_args*>(static_cast<uintptr_t>(PyLong_AsUnsignedLongLong(p[0])));
      s->q = tensor(p[1], name, "q"); s->block_table = tensor(p[2], name, "block_table"); s->seq_lens = tensor(p[3], name, "seq_lens");
      for (int i = 0; i < 5; ++i) s->keep[i] = tensor(p[4 + i], name, "step buffer");
      s->q_host_dev = out_ptr(s->keep[0]); s->o_new_dev = out_ptr(s->keep[1]);
      auto* words = static_cast<int64_t*>(out_ptr(s->keep[2]));
      s->trigger_dev = words; s->done_dev = words + 8;
      s->status_host = out_ptr(s->keep[3]); s->status_host_dev = out_ptr(s->keep[4]);
      s->q_dev = out_ptr(s->q); s->bt_dev = static_cast<int64_t*>(out_ptr(s->block_table));
      s->lens_dev = static_cast<int32_t*>(out_ptr(s->seq_lens)); s->bt_dev_stride = static_cast<int32_t>(s->block_table.size(1));
      s->ctx = integer(p[9]);
      s->timeout_ms = int32(p[10]);
      s->H_q = s->q.size(1);
      s->rows = s->cut = s->q.size(0) * s->H_q;
      if (p[11] != Py_None) {
        for (int i = 0; i < 3; ++i) s->keep[5 + i] = tensor(PyTuple_GetItem(p[11], i), name, "correction buffer");
        s->k_mirror = ptr(s->keep[5]); s->v_mirror = ptr(s->keep[6]); s->slots = ptr(s->keep[7]);
        s->slots_i32 = s->keep[7].scalar_type() == at::kInt;
        s->cut = integer(PyTuple_GetItem(p[11], 3));
      }
    } catch (...) {
      Py_DECREF(cap);
      throw;
    }
    return cap;
  });
}

// step_run(capsule, query, block_table, seq_lens, output) -> (status, 1 if the stream is capturing, merged output that
//   still has to be copied into `output` | None).  Nothing here waits on the host.
PyObject* step_run(PyObject*, PyObject* const* p, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    const char* name = "decode_step";
    expect_args(n, 5, "step_run");
    auto* s = static_cast<Step*>(PyCapsule_GetPointer(p[0], kStepName));
    if (!s) return nullptr;
    const int64_t B = s->q.size(0), H = s->H_q, row = H * JF_HEAD_DIM;
    const jf_stream_t st = current_stream();
    const bool capturing = capturing_now();
    at::Tensor q = tensor(p[1], name, "query"), bt = tensor(p[2], name, "block_table"), lens = tensor(p[3], name, "seq_lens"),
               out = tensor(p[4], name, "output");
    require(q.is_cuda(), name, "query must be CUDA");
    require(q.scalar_type() == s->q.scalar_type(), name, "query dtype mismatch");
    require(q.dim() >= 2 && q.size(0) >= B && q.numel() == q.size(0) * row, name, "query must be (B, H_q, 128)");
    require(out.dim() >= 2 && out.size(0) >= B && out.numel() == out.size(0) * row, name, "output must be (B, H_q * 128)");
    // rows of H_q * 128 elements, whatever the leading dimensions are called
    auto rows_ok = [&](const at::Tensor& t, int64_t mult, uintptr_t align) {
      const bool two = t.dim() == 2 && t.size(1) == row && t.stride(1) == 1;
      const bool three = t.dim() == 3 && t.size(1) == H && t.size(2) == JF_HEAD_DIM && t.stride(2) == 1 && t.stride(1) == JF_HEAD_DIM;
      return (two || three) && t.stride(0) % mult == 0 && reinterpret_cast<uintptr_t>(ptr(t)) % align == 0;
    };
    // an output in place has the step's device and type; any other form is what a copy takes
    const bool same = out.is_cuda() && out.scalar_type() == s->q.scalar_type();
    require(same || !out.narrow(0, 0, B).is_contiguous(), name, "output must be a CUDA tensor of the query's dtype");
    require(bt.dim() == 2 && (bt.size(0) >= B || bt.size(0) == 1) && lens.dim() <= 1 && lens.numel() >= B, name,
            "block_table / seq_lens shape mismatch");
    jf_status_t r = JF_OK;
    if (!capturing) {   // an error of an earlier run, as far as it has arrived
      r = jf_decode_status_of_copy(s->status_host);
      if (r == JF_OK) r = jf_submit_ctx_status(s->ctx);
      else std::memset(s->status_host, 0, JF_STATUS_RECORD_BYTES);   // reported once; the next call runs
    }
    // forms that the kernels do not address go through a copy
    if (!rows_ok(q, 8, 16)) q = at::empty({B, row}, s->q.options()).copy_(q.narrow(0, 0, B).reshape({B, row}));
    if (!bt.is_cuda()) bt = bt.to(s->q.device());
    if ((bt.scalar_type() != at::kLong && bt.scalar_type() != at::kInt) || bt.stride(1) != 1) bt = bt.to(at::kLong).contiguous();
    if (!lens.is_cuda()) lens = lens.to(s->q.device());
    if (lens.dim() == 0) lens = lens.reshape({1});
    if ((lens.scalar_type() != at::kLong && lens.scalar_type() != at::kInt) || lens.stride(0) != 1) lens = lens.to(at::kInt).contiguous();
    const int64_t width = std::min<int64_t>(bt.size(1), s->block_table.size(1));
    at::Tensor merged;
    if (!same || !rows_ok(out, 4, 8)) merged = at::empty_like(s->q);
    const at::Tensor& dst = merged.defined() ? merged : out;
    const int64_t dst_stride = merged.defined() ? row : dst.stride(0);
    const int dt = dtype_id(s->q);
    if (r == JF_OK) {
      const void *qp = ptr(q), *btp = ptr(bt), *lp = ptr(lens);
      void* op = out_ptr(dst);
      const int64_t q_stride = q.stride(0), bt_stride = bt.size(0) < B ? 0 : bt.stride(0);   // one row for all: broadcast
      const int32_t bt_i32 = bt.scalar_type() == at::kInt, lens_i32 = lens.scalar_type() == at::kInt;
      r = unlocked([&] {
        jf_status_t e = jf_step_begin(qp, q_stride, s->q_dev, s->q_host_dev, btp, bt_i32, bt_stride, static_cast<int32_t>(width), s->bt_dev,
                                      s->bt_dev_stride, lp, lens_i32, s->lens_dev, s->done_dev, static_cast<int32_t>(B),
                                      static_cast<int32_t>(H), st);
        if (e == JF_OK) e = jf_decode_fused(s->a, st);
        int64_t* trigger = s->trigger_dev;
        if (e == JF_OK && s->cut < s->rows) {   // the GPU's rows, while the workers do theirs
          e = jf_stream_signal_host(st, s->done_dev, s->trigger_dev);
          trigger = nullptr;
          if (e == JF_OK)
            e = jf_gpu_topk_attn_rows(s->q_dev, s->k_mirror, s->v_mirror, s->slots, s->slots_i32, s->o_new_dev, dt, s->a->B, s->a->H_q,
                                      s->a->H_kv, s->a->num_slots, s->a->top_k, s->a->attn_scale, s->cut, s->rows, st);
        }
        if (e == JF_OK)
          e = jf_step_end(s->a->o_hat, s->a->o_old_unnorm, s->a->W, s->o_new_dev, op, dst_stride, dt, s->a->B, s->a->H_q,
                          s->done_dev, trigger, s->timeout_ms, s->a->workspace, s->status_host_dev, st);
        return e;
      });
    }
    PyObject* res = PyTuple_New(3);
    if (!res) return nullptr;
    PyTuple_SET_ITEM(res, 0, PyLong_FromLong(r));
    PyTuple_SET_ITEM(res, 1, PyLong_FromLong(capturing));
    PyTuple_SET_ITEM(res, 2, THPVariable_Wrap(merged));
    return res;
  });
}

#define JF_METHOD(f) {#f, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(f)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    JF_METHOD(quant_write), JF_METHOD(quant_write_kv), JF_METHOD(fused_attn), JF_METHOD(stage_a), JF_METHOD(stage_b),
    JF_METHOD(decode), JF_METHOD(get_workspace), JF_METHOD(blend), JF_METHOD(step_create), JF_METHOD(step_run),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "tensor-taking half of jetfire_b200.ops", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
  PyObject* m = PyModule_Create(&kModule);
  if (m && PyModule_AddStringConstant(m, "built_for", JF_TORCH_STAMP) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
