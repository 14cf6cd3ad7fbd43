// Host path of the Python entry points: argument checks, output allocation and the C-ABI call, as a
// CPython extension over torch's C++ tensors.
//
// An eager decode step of one layer is one or two launches of a few microseconds each; written in Python
// (shape and stride look-ups, torch.cuda.device, current_stream, a ctypes call with two dozen
// conversions) the host side of two calls took 41 us at batch 1, four times the kernels.  The
// same checks on at::Tensor cost tens of nanoseconds each, so the launches are what is left.
//
// The extension holds no product code of its own: it resolves the C-ABI functions of
// include/nvllm_b200.h from the library that the ctypes loader opened (bind), raises what the
// Python code raised (AssertionError for layout, RuntimeError for device and dtype, NvllmError for
// an argument the library refused), and never touches the device except through those functions,
// torch's allocator, and one event per staged decode step.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <limits>
#include <memory>
#include <string>
#include <vector>

#include "../../include/nvllm_b200.h"

namespace {

struct PyErrorSet {};  // thrown once a Python exception has been set

[[noreturn]] void raise(PyObject* type, const std::string& msg) {
  PyErr_SetString(type, msg.c_str());
  throw PyErrorSet{};
}
inline void require(bool cond, const char* what) {
  if (__builtin_expect(!cond, 0)) raise(PyExc_AssertionError, what);
}

struct Api {
  decltype(&nvllm_store_kvcache) store_kvcache;
  decltype(&nvllm_decode_paged) decode_paged;
  decltype(&nvllm_decode_step) decode_step;
  decltype(&nvllm_decode_workspace_bytes) decode_workspace_bytes;
  decltype(&nvllm_prefill_varlen) prefill_varlen;
  decltype(&nvllm_attention_decode) attention_decode;
  decltype(&nvllm_attention_prefill) attention_prefill;
  decltype(&nvllm_qk_norm_rope_store) qk_norm_rope_store;
  decltype(&nvllm_sample_tokens) sample_tokens;
  decltype(&nvllm_sample_candidates) sample_candidates;
  decltype(&nvllm_decode_step_inputs_pinned) decode_step_inputs_pinned;
} api;
PyObject* g_check = nullptr;  // _lib.check: raises NvllmError for a negative code

struct Names {
  PyObject *num_heads, *head_dim, *scale, *num_kv_heads, *k_cache, *v_cache, *is_prefill, *cu_seqlens_q, *cu_seqlens_k,
      *max_seqlen_q, *max_seqlen_k, *slot_mapping, *context_lens, *block_tables, *last_token, *num_tokens, *temperature,
      *block_table;
} names;

// ---- arguments -----------------------------------------------------------------------------

const at::Tensor& tensor(PyObject* o, const char* name) {
  if (__builtin_expect(!THPVariable_Check(o), 0)) raise(PyExc_TypeError, std::string(name) + " must be a torch.Tensor");
  return THPVariable_Unpack(o);
}
const at::Tensor* maybe_tensor(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor(o, name); }

void require_cuda_bf16(const char* name, const at::Tensor& t) {
  if (__builtin_expect(!t.is_cuda(), 0))
    raise(PyExc_RuntimeError, std::string(name) + " must be a CUDA tensor (nano_vllm_b200 has no CPU path)");
  if (__builtin_expect(t.scalar_type() != at::kBFloat16, 0))
    raise(PyExc_RuntimeError, std::string(name) + " must be bfloat16, got " + std::string(c10::toString(t.scalar_type())));
}
void require_i32(const char* name, const at::Tensor& t) {
  if (__builtin_expect(!t.is_cuda() || t.scalar_type() != at::kInt || (t.dim() > 0 && t.stride(-1) != 1), 0))
    raise(PyExc_RuntimeError, std::string(name) + " must be a CUDA int32 tensor with unit inner stride");
}
void require_dim(const char* name, const at::Tensor& t, int64_t dim) {
  if (__builtin_expect(t.dim() != dim, 0))
    raise(PyExc_ValueError, std::string(name) + " must have " + std::to_string(dim) + " dimensions, got " + std::to_string(t.dim()));
}
int64_t as_i64(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyErrorSet{};
  return v;
}
int32_t as_i32(PyObject* o) {
  const long long v = as_i64(o);
  if (v < std::numeric_limits<int32_t>::min() || v > std::numeric_limits<int32_t>::max())
    raise(PyExc_OverflowError, "Python integer out of bounds for int32");
  return static_cast<int32_t>(v);
}
uint64_t as_u64(PyObject* o) {  // modulo 2^64, as `x & 0xFFFFFFFFFFFFFFFF`
  PyObject* n = PyNumber_Index(o);
  if (!n) throw PyErrorSet{};
  const unsigned long long v = PyLong_AsUnsignedLongLongMask(n);
  Py_DECREF(n);
  if (v == static_cast<unsigned long long>(-1) && PyErr_Occurred()) throw PyErrorSet{};
  return v;
}
double as_double(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyErrorSet{};
  return v;
}
void check(int64_t code) {
  if (__builtin_expect(code >= 0, 1)) return;
  PyObject* r = PyObject_CallFunction(g_check, "L", static_cast<long long>(code));
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "nvllm call failed");
  throw PyErrorSet{};
}
// What may wait for the device runs without the interpreter lock, as a ctypes call or a torch operation does: a
// launch waits while the device's queue is full and an allocation may wait for all that is in front of it,
// which other threads of the program may have to finish.
template <class F>
auto unlocked(F&& f) {
  struct Unlock {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlock() { PyEval_RestoreThread(state); }
  } unlock;
  return f();
}
template <class F>
void launch(F&& f) {
  check(unlocked(f));
}
at::Tensor new_tensor(at::IntArrayRef sizes, const at::TensorOptions& options) {
  return unlocked([&] { return at::empty(sizes, options); });
}
template <class T>
T* ptr(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }
void* stream_of(const at::Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
// Rows of row_elems in a cache plane.  None of an empty one: the library refuses the shape that says so.
int64_t rows_in(const at::Tensor& t, int64_t row_elems) { return row_elems > 0 ? t.numel() / row_elems : 0; }
PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

// ---- decode scratch ---------------------------------------------------------------------
// One buffer per device, grown on demand and zero-filled when it is made: its head holds the
// arrival counters of the decode kernel, which must start at zero and which every completed
// call leaves at zero.  Outgrown buffers are kept alive because CUDA graphs captured earlier
// still hold their addresses.
std::vector<at::Tensor> g_workspaces, g_retired;

void workspace(const at::Tensor& like, int64_t nbytes, void** p, int64_t* size) {
  *p = nullptr;
  *size = 0;
  if (nbytes == 0) return;
  const size_t dev = static_cast<size_t>(like.device().index());
  if (g_workspaces.size() <= dev) g_workspaces.resize(dev + 1);
  auto enough = [&] { return g_workspaces[dev].defined() && g_workspaces[dev].numel() >= nbytes; };
  if (!enough()) {
    at::Tensor fresh = unlocked([&] { return at::zeros({std::max<int64_t>(nbytes, 1 << 20)}, like.options().dtype(at::kByte)); });
    if (!enough()) {  // not grown by another thread meanwhile
      if (g_workspaces[dev].defined()) g_retired.push_back(g_workspaces[dev]);
      g_workspaces[dev] = std::move(fresh);
    }
  }
  const at::Tensor& ws = g_workspaces[dev];
  *p = ws.data_ptr();
  *size = ws.numel();
}

// Zeroes the current device's buffers, outgrown ones too (after a launch whose waits ran out), and waits for that.
PyObject* clear_workspaces(PyObject* const*) {
  const c10::DeviceIndex dev = c10::cuda::current_device();
  std::vector<at::Tensor> all = g_workspaces;
  all.insert(all.end(), g_retired.begin(), g_retired.end());
  for (const at::Tensor& ws : all)
    if (ws.defined() && ws.device().index() == dev) ws.zero_();
  const c10::cuda::CUDAStream st = c10::cuda::getCurrentCUDAStream(dev);
  unlocked([&] { st.synchronize(); });
  Py_RETURN_NONE;
}

// ---- the operations -----------------------------------------------------------------------

// Rows of [n, heads, d] with unit inner stride and d between heads.
struct Rows {
  void* p;
  int64_t n, stride;
};

void check_store(const Rows& k, int64_t row, const at::Tensor& k_cache, const at::Tensor& v_cache, const at::Tensor& slot_mapping) {
  require(k_cache.dim() > 1 && k_cache.stride(1) == row && v_cache.dim() > 1 && v_cache.stride(1) == row,
          "k_cache.stride(1) == D and v_cache.stride(1) == D");
  require(slot_mapping.numel() == k.n, "slot_mapping.numel() == N");
  require_cuda_bf16("k_cache", k_cache);
  require_cuda_bf16("v_cache", v_cache);
  require_i32("slot_mapping", slot_mapping);
}

void store(const Rows& k, const Rows& v, int64_t row, const at::Tensor& k_cache, const at::Tensor& v_cache,
           const at::Tensor& slot_mapping) {
  check_store(k, row, k_cache, v_cache, slot_mapping);
  launch([&] {
    return api.store_kvcache(k.p, k.stride, v.p, v.stride, k_cache.data_ptr(), v_cache.data_ptr(), ptr<int32_t>(slot_mapping),
                             k.n, static_cast<int32_t>(row), rows_in(k_cache, row), stream_of(k_cache));
  });
}

struct Step {  // the new tokens' rows, for a call that stores as well
  Rows k, v;
  const int32_t* slots;
  bool one_launch;  // decode_step's rules; otherwise store_kvcache's, in a launch of its own
};

void decode(const Rows& q, int64_t hq, int64_t d, const at::Tensor& k_cache, const at::Tensor& v_cache,
            const at::Tensor& context_lens, const at::Tensor& block_tables, double scale, const Rows& out, const Step* step) {
  require_cuda_bf16("k_cache", k_cache);
  require_cuda_bf16("v_cache", v_cache);
  require_i32("context_lens", context_lens);
  require_i32("block_tables", block_tables);
  require(k_cache.is_contiguous() && v_cache.is_contiguous(), "k_cache.is_contiguous() and v_cache.is_contiguous()");
  require(block_tables.dim() == 2 && block_tables.size(0) == q.n && context_lens.numel() == q.n,
          "block_tables.dim() == 2 and block_tables.shape[0] == B and context_lens.numel() == B");
  if (q.n == 0) return;
  const int64_t hkv = k_cache.size(-2);
  const int32_t width = static_cast<int32_t>(block_tables.size(1));
  const int64_t num_blocks = rows_in(k_cache, NVLLM_BLOCK_SIZE * hkv * d);
  const int64_t need = api.decode_workspace_bytes(static_cast<int32_t>(q.n), width, static_cast<int32_t>(hq),
                                                  static_cast<int32_t>(hkv), static_cast<int32_t>(d));
  check(need);
  void* ws;
  int64_t ws_size;
  workspace(k_cache, need, &ws, &ws_size);
  const int32_t B = static_cast<int32_t>(q.n), HQ = static_cast<int32_t>(hq), HKV = static_cast<int32_t>(hkv),
                D = static_cast<int32_t>(d);
  void* st = stream_of(k_cache);
  if (step && !step->one_launch)
    launch([&] {
      return api.attention_decode(q.p, q.stride, step->k.p, step->k.stride, step->v.p, step->v.stride, step->slots, step->k.n,
                                  k_cache.data_ptr(), v_cache.data_ptr(), ptr<int32_t>(context_lens),
                                  ptr<int32_t>(block_tables), block_tables.stride(0), width, out.p, out.stride, B, HQ, HKV, D,
                                  static_cast<float>(scale), num_blocks, ws, ws_size, st);
    });
  else if (step)
    launch([&] {
      return api.decode_step(q.p, q.stride, step->k.p, step->k.stride, step->v.p, step->v.stride, step->slots,
                             k_cache.data_ptr(), v_cache.data_ptr(), ptr<int32_t>(context_lens), ptr<int32_t>(block_tables),
                             block_tables.stride(0), width, out.p, out.stride, B, HQ, HKV, D, static_cast<float>(scale),
                             num_blocks, ws, ws_size, st);
    });
  else
    launch([&] {
      return api.decode_paged(q.p, q.stride, k_cache.data_ptr(), v_cache.data_ptr(), ptr<int32_t>(context_lens),
                              ptr<int32_t>(block_tables), block_tables.stride(0), width, out.p, out.stride, B, HQ, HKV, D,
                              static_cast<float>(scale), num_blocks, ws, ws_size, st);
    });
}

// K/V of a prefill: packed rows, or the cache planes with a block table.
struct KV {
  Rows k, v;  // n = packed rows (0 with a table)
  int64_t hkv;
  const at::Tensor* block_tables;
  int64_t num_blocks;
};

KV paged_kv(const at::Tensor& k, const at::Tensor& v, const at::Tensor& block_tables) {
  require_i32("block_tables", block_tables);
  require(k.is_contiguous() && v.is_contiguous() && k.dim() == 4 && k.size(1) == NVLLM_BLOCK_SIZE,
          "k and v must be contiguous cache planes [blocks, 256, Hkv, D]");
  return {{k.data_ptr(), 0, k.stride(1)}, {v.data_ptr(), 0, k.stride(1)}, k.size(2), &block_tables, k.size(0)};
}

void prefill(const Rows& q, int64_t hq, int64_t d, const KV& kv, const at::Tensor& cu_q, const at::Tensor& cu_k, int64_t max_q,
             int64_t max_k, double scale, const Rows& out, void* stream, const Step* step = nullptr,
             const at::Tensor* k_cache = nullptr, const at::Tensor* v_cache = nullptr) {
  require_i32("cu_seqlens_q", cu_q);
  require_i32("cu_seqlens_k", cu_k);
  const int64_t batch = cu_q.numel() - 1;
  require(cu_k.numel() == batch + 1, "cu_seqlens_k.numel() == batch + 1");
  const at::Tensor* bt = kv.block_tables;
  if (bt)
    require(bt->dim() == 2 && bt->size(0) == batch, "block_tables.dim() == 2 and block_tables.shape[0] == batch");
  if (step) {
    launch([&] {
      return api.attention_prefill(q.p, q.stride, step->k.p, step->k.stride, step->v.p, step->v.stride, step->slots,
                                   k_cache->data_ptr(), v_cache->data_ptr(), bt ? ptr<int32_t>(*bt) : nullptr,
                                   bt ? bt->stride(0) : 0, bt ? static_cast<int32_t>(bt->size(1)) : 0, out.p, out.stride,
                                   ptr<int32_t>(cu_q), ptr<int32_t>(cu_k), q.n, step->k.n, static_cast<int32_t>(batch),
                                   static_cast<int32_t>(max_q), static_cast<int32_t>(max_k), static_cast<int32_t>(hq),
                                   static_cast<int32_t>(kv.hkv), static_cast<int32_t>(d), static_cast<float>(scale),
                                   rows_in(*k_cache, NVLLM_BLOCK_SIZE * kv.hkv * d), stream);
    });
    return;
  }
  if (q.n == 0 || batch == 0) return;
  launch([&] {
    return api.prefill_varlen(q.p, q.stride, kv.k.p, kv.k.stride, kv.v.p, kv.v.stride, bt ? ptr<int32_t>(*bt) : nullptr,
                              bt ? bt->stride(0) : 0, bt ? static_cast<int32_t>(bt->size(1)) : 0, out.p, out.stride,
                              ptr<int32_t>(cu_q), ptr<int32_t>(cu_k), q.n, kv.k.n, static_cast<int32_t>(batch),
                              static_cast<int32_t>(max_q), static_cast<int32_t>(max_k), static_cast<int32_t>(hq),
                              static_cast<int32_t>(kv.hkv), static_cast<int32_t>(d), static_cast<float>(scale), kv.num_blocks,
                              stream);
  });
}

// [n, heads, d] argument of a functional entry point.
Rows rows3(const at::Tensor& t, const char* what) {
  require(t.stride(-1) == 1 && t.stride(1) == t.size(2), what);
  return {t.data_ptr(), t.size(0), t.stride(0)};
}

at::Tensor output_for(PyObject* out, const at::Tensor& q, Rows* rows) {
  at::Tensor o = out == Py_None ? new_tensor(q.sizes(), q.options()) : tensor(out, "out");
  require(o.dim() == 3 && o.stride(-1) == 1 && o.stride(1) == q.size(2), "out.stride(-1) == 1 and out.stride(1) == D");
  *rows = {o.data_ptr(), o.size(0), o.stride(0)};
  return o;
}

// Activation of the layer: q.view(-1, heads, d) without the view where the layout is a plain one.
Rows activation(const at::Tensor& t, int64_t heads, int64_t d, at::Tensor* keep) {
  if (t.dim() == 2 && t.size(1) == heads * d && t.stride(1) == 1) return {t.data_ptr(), t.size(0), t.stride(0)};
  if (t.dim() == 3 && t.size(1) == heads && t.size(2) == d && t.stride(2) == 1 && t.stride(1) == d)
    return {t.data_ptr(), t.size(0), t.stride(0)};
  *keep = t.view({-1, heads, d});
  return rows3(*keep, "activation rows must have unit inner stride");
}

PyObject* store_kvcache(PyObject* const* a) {
  const at::Tensor &key = tensor(a[0], "key"), &value = tensor(a[1], "value"), &k_cache = tensor(a[2], "k_cache"),
                   &v_cache = tensor(a[3], "v_cache"), &slots = tensor(a[4], "slot_mapping");
  require_dim("key", key, 3);
  const Rows k = rows3(key, "key.stride(-1) == 1 and key.stride(1) == head_dim");
  require(value.dim() == 3 && value.stride(-1) == 1 && value.stride(1) == key.size(2),
          "value.stride(-1) == 1 and value.stride(1) == head_dim");
  require_cuda_bf16("key", key);
  require_cuda_bf16("value", value);
  const c10::cuda::CUDAGuard guard(key.device());
  store(k, {value.data_ptr(), value.size(0), value.stride(0)}, key.size(1) * key.size(2), k_cache, v_cache, slots);
  Py_RETURN_NONE;
}

PyObject* decode_paged(PyObject* const* a) {  // q, k_cache, v_cache, context_lens, block_tables, scale, out
  const at::Tensor& q = tensor(a[0], "q");
  require_dim("q", q, 3);
  require_cuda_bf16("q", q);
  const Rows qr = rows3(q, "q.stride(-1) == 1 and q.stride(1) == D");
  const c10::cuda::CUDAGuard guard(q.device());
  Rows o;
  at::Tensor out = output_for(a[6], q, &o);
  decode(qr, q.size(1), q.size(2), tensor(a[1], "k_cache"), tensor(a[2], "v_cache"), tensor(a[3], "context_lens"),
         tensor(a[4], "block_tables"), as_double(a[5]), o, nullptr);
  return wrap(std::move(out));
}

PyObject* decode_step(PyObject* const* a) {
  // q, key, value, k_cache, v_cache, slot_mapping, context_lens, block_tables, scale, out
  const at::Tensor &q = tensor(a[0], "q"), &key = tensor(a[1], "key"), &value = tensor(a[2], "value"),
                   &k_cache = tensor(a[3], "k_cache"), &slots = tensor(a[5], "slot_mapping");
  require_dim("q", q, 3);
  require_cuda_bf16("q", q);
  require_cuda_bf16("key", key);
  require_cuda_bf16("value", value);
  require_i32("slot_mapping", slots);
  const Rows qr = rows3(q, "q.stride(-1) == 1 and q.stride(1) == D");
  const int64_t B = q.size(0), D = q.size(2), hkv = k_cache.dim() >= 2 ? k_cache.size(-2) : 0;
  for (const at::Tensor* t : {&key, &value})
    require(t->dim() == 3 && t->size(0) == B && t->size(1) == hkv && t->size(2) == D,
            "key.shape == (B, Hkv, D) and value.shape == (B, Hkv, D)");
  const Step step = {rows3(key, "key.stride(-1) == 1 and key.stride(1) == D"),
                     rows3(value, "value.stride(-1) == 1 and value.stride(1) == D"), ptr<int32_t>(slots), true};
  require(slots.numel() == B, "slot_mapping.numel() == B");
  const c10::cuda::CUDAGuard guard(q.device());
  Rows o;
  at::Tensor out = output_for(a[9], q, &o);
  decode(qr, q.size(1), D, k_cache, tensor(a[4], "v_cache"), tensor(a[6], "context_lens"), tensor(a[7], "block_tables"),
         as_double(a[8]), o, &step);
  return wrap(std::move(out));
}

PyObject* prefill_varlen(PyObject* const* a) {
  // q, k, v, cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, scale, block_tables, out
  const at::Tensor &q = tensor(a[0], "q"), &k = tensor(a[1], "k"), &v = tensor(a[2], "v");
  require_dim("q", q, 3);
  require_cuda_bf16("q", q);
  require_cuda_bf16("k", k);
  require_cuda_bf16("v", v);
  const Rows qr = rows3(q, "q.stride(-1) == 1 and q.stride(1) == D");
  const at::Tensor* bt = maybe_tensor(a[8], "block_tables");
  KV kv;
  if (bt) {
    kv = paged_kv(k, v, *bt);
  } else {
    require(k.dim() == 3 && v.dim() == 3 && k.stride(-1) == 1 && v.stride(-1) == 1 && k.stride(1) == q.size(2) &&
                v.stride(1) == q.size(2),
            "k.dim() == 3, unit inner stride, D between heads");
    kv = {{k.data_ptr(), k.size(0), k.stride(0)}, {v.data_ptr(), v.size(0), v.stride(0)}, k.size(1), nullptr, 0};
  }
  const c10::cuda::CUDAGuard guard(q.device());
  Rows o;
  at::Tensor out = output_for(a[9], q, &o);
  prefill(qr, q.size(1), q.size(2), kv, tensor(a[3], "cu_seqlens_q"), tensor(a[4], "cu_seqlens_k"), as_i64(a[5]), as_i64(a[6]),
          as_double(a[7]), o, stream_of(q));
  return wrap(std::move(out));
}

struct Ref {  // owned reference
  PyObject* o;
  explicit Ref(PyObject* p) : o(p) {
    if (!p) throw PyErrorSet{};
  }
  ~Ref() { Py_DECREF(o); }
  Ref(const Ref&) = delete;
};
int64_t attr_i64(PyObject* o, PyObject* name) {
  Ref r(PyObject_GetAttr(o, name));
  return as_i64(r.o);
}

// Attention.forward: layer, context, q, k, v, kv_stored
PyObject* attention_forward(PyObject* const* a) {
  PyObject *layer = a[0], *ctx = a[1];
  const int64_t hq = attr_i64(layer, names.num_heads), hkv = attr_i64(layer, names.num_kv_heads),
                d = attr_i64(layer, names.head_dim);
  double scale;
  {
    Ref s(PyObject_GetAttr(layer, names.scale));
    scale = as_double(s.o);
  }
  Ref kc(PyObject_GetAttr(layer, names.k_cache)), vc(PyObject_GetAttr(layer, names.v_cache));
  const at::Tensor &k_cache = tensor(kc.o, "k_cache"), &v_cache = tensor(vc.o, "v_cache");
  const at::Tensor &q = tensor(a[2], "q"), &k = tensor(a[3], "k"), &v = tensor(a[4], "v");
  at::Tensor keep[3];
  const Rows qr = activation(q, hq, d, &keep[0]), kr = activation(k, hkv, d, &keep[1]), vr = activation(v, hkv, d, &keep[2]);
  const int kv_stored = PyObject_IsTrue(a[5]);
  if (kv_stored < 0) throw PyErrorSet{};
  int prefill_phase;
  {
    Ref p(PyObject_GetAttr(ctx, names.is_prefill));
    prefill_phase = PyObject_IsTrue(p.o);
    if (prefill_phase < 0) throw PyErrorSet{};
  }
  Ref bt(PyObject_GetAttr(ctx, names.block_tables));
  const bool do_store = k_cache.numel() && v_cache.numel() && !kv_stored;
  if (do_store || prefill_phase) {
    require_cuda_bf16("k", k);
    require_cuda_bf16("v", v);
  }
  require_cuda_bf16("q", q);
  const c10::cuda::CUDAGuard guard(q.device());
  Ref slots(PyObject_GetAttr(ctx, names.slot_mapping));
  Step step{};
  const Step* with_store = nullptr;
  if (do_store) {
    const at::Tensor& sm = tensor(slots.o, "slot_mapping");
    const int64_t block = NVLLM_BLOCK_SIZE * hkv * d;
    if (qr.n > 0 && block > 0 && k_cache.numel() % block == 0) {
      check_store(kr, hkv * d, k_cache, v_cache, sm);
      step = {kr, vr, ptr<int32_t>(sm), false};
      with_store = &step;
    } else {
      store(kr, vr, hkv * d, k_cache, v_cache, sm);
    }
  }
  at::Tensor out = new_tensor({qr.n, hq * d}, q.options());
  const Rows o = {out.data_ptr(), qr.n, hq * d};
  if (prefill_phase) {
    Ref cq(PyObject_GetAttr(ctx, names.cu_seqlens_q)), ck(PyObject_GetAttr(ctx, names.cu_seqlens_k));
    const int64_t mq = attr_i64(ctx, names.max_seqlen_q), mk = attr_i64(ctx, names.max_seqlen_k);
    const at::Tensor* table = maybe_tensor(bt.o, "block_tables");
    // prefix cache: every key is read through the table
    const KV kv = table ? paged_kv(k_cache, v_cache, *table) : KV{kr, vr, hkv, nullptr, 0};
    prefill(qr, hq, d, kv, tensor(cq.o, "cu_seqlens_q"), tensor(ck.o, "cu_seqlens_k"), mq, mk, scale, o, stream_of(q), with_store,
            &k_cache, &v_cache);
  } else {
    Ref lens(PyObject_GetAttr(ctx, names.context_lens));
    decode(qr, hq, d, k_cache, v_cache, tensor(lens.o, "context_lens"), tensor(bt.o, "block_tables"), scale, o, with_store);
  }
  return wrap(std::move(out));
}

PyObject* qk_norm_rope_store(PyObject* const* a) {
  // qkv, positions, q_weight, k_weight, cos_sin_cache, eps, slot_mapping, k_cache, v_cache, hq, hkv, d
  const at::Tensor &qkv = tensor(a[0], "qkv"), &positions = tensor(a[1], "positions"), &cs = tensor(a[4], "cos_sin_cache");
  const at::Tensor *qw = maybe_tensor(a[2], "q_weight"), *kw = maybe_tensor(a[3], "k_weight"),
                   *slots = maybe_tensor(a[6], "slot_mapping");
  const int64_t hq = as_i64(a[9]), hkv = as_i64(a[10]), d = as_i64(a[11]);
  require_cuda_bf16("qkv", qkv);
  require(qkv.dim() == 2 && qkv.stride(-1) == 1, "qkv.dim() == 2 and qkv.stride(-1) == 1");
  require(qkv.size(1) == (hq + 2 * hkv) * d, "qkv.shape[1] == (num_q_heads + 2 * num_kv_heads) * head_dim");
  require(positions.is_cuda() && positions.scalar_type() == at::kLong && positions.numel() == qkv.size(0),
          "positions must be a CUDA int64 tensor, one per token");
  require(cs.is_cuda() && cs.scalar_type() == at::kFloat && cs.is_contiguous(), "cos_sin_cache must be contiguous CUDA float32");
  if (d <= 0 || cs.numel() % d) raise(PyExc_RuntimeError, "cos_sin_cache does not divide into rows of head_dim");
  for (const at::Tensor* w : {qw, kw})
    if (w) {
      require_cuda_bf16("norm weight", *w);
      require(w->numel() == d && w->is_contiguous(), "a norm weight has head_dim contiguous elements");
    }
  void *kc = nullptr, *vc = nullptr;
  int64_t num_slots = 0;
  const int32_t* sm = nullptr;
  if (slots) {
    const at::Tensor &k_cache = tensor(a[7], "k_cache"), &v_cache = tensor(a[8], "v_cache");
    if (k_cache.numel() > 0 && v_cache.numel() > 0) {
      require_i32("slot_mapping", *slots);
      require_cuda_bf16("k_cache", k_cache);
      require_cuda_bf16("v_cache", v_cache);
      require(k_cache.is_contiguous() && v_cache.is_contiguous() && slots->numel() == qkv.size(0),
              "contiguous caches and one slot per token");
      kc = k_cache.data_ptr();
      vc = v_cache.data_ptr();
      num_slots = rows_in(k_cache, hkv * d);
      sm = ptr<int32_t>(*slots);
    }
  }
  const float eps = static_cast<float>(as_double(a[5]));
  const c10::cuda::CUDAGuard guard(qkv.device());
  launch([&] {
    return api.qk_norm_rope_store(qkv.data_ptr(), qkv.stride(0), ptr<int64_t>(positions), qw ? qw->data_ptr() : nullptr,
                                  kw ? kw->data_ptr() : nullptr, ptr<float>(cs), cs.numel() / d, eps, sm, kc, vc, num_slots,
                                  qkv.size(0), static_cast<int32_t>(hq), static_cast<int32_t>(hkv), static_cast<int32_t>(d),
                                  stream_of(qkv));
  });
  Py_RETURN_NONE;
}

// logits, temperatures, noise, seed, step, out [, vocab_offset]
PyObject* sample(PyObject* const* a, bool candidates) {
  const at::Tensor &logits = tensor(a[0], "logits"), &temps = tensor(a[1], "temperatures");
  const at::Tensor* noise = maybe_tensor(a[2], "noise");
  require(logits.is_cuda() && logits.dim() == 2 && logits.stride(-1) == 1, "logits must be a 2-D CUDA tensor with unit inner stride");
  const bool fp32 = logits.scalar_type() == at::kFloat;
  if (!fp32 && logits.scalar_type() != at::kBFloat16)
    raise(PyExc_AssertionError, "logits must be bf16 or fp32, got " + std::string(c10::toString(logits.scalar_type())));
  const int64_t B = logits.size(0), V = logits.size(1);
  require(temps.is_cuda() && temps.scalar_type() == at::kFloat && temps.numel() == B && temps.is_contiguous(),
          "temperatures must be contiguous CUDA float32, one per row");
  if (noise)
    require(noise->is_cuda() && noise->scalar_type() == at::kFloat && noise->sizes() == logits.sizes() && noise->stride(-1) == 1,
            "noise must be CUDA float32 of the logits' shape");
  const c10::cuda::CUDAGuard guard(logits.device());
  at::Tensor out = a[5] == Py_None ? new_tensor({B}, logits.options().dtype(at::kLong)) : tensor(a[5], "out");
  require(out.is_cuda() && out.scalar_type() == at::kLong && out.numel() == B && out.is_contiguous(),
          "out must be contiguous CUDA int64, one per row");
  const float* nz = noise ? ptr<float>(*noise) : nullptr;
  const int64_t nzs = noise ? noise->stride(0) : 0;
  const uint64_t seed = as_u64(a[3]), step = as_u64(a[4]);
  const int64_t offset = candidates ? as_i64(a[6]) : 0;
  if (candidates)
    launch([&] {
      return api.sample_candidates(logits.data_ptr(), fp32, logits.stride(0), ptr<float>(temps), nz, nzs, seed, step, offset,
                                   ptr<int64_t>(out), static_cast<int32_t>(B), static_cast<int32_t>(V), stream_of(logits));
    });
  else
    launch([&] {
      return api.sample_tokens(logits.data_ptr(), fp32, logits.stride(0), ptr<float>(temps), nz, nzs, seed, step,
                               ptr<int64_t>(out), static_cast<int32_t>(B), static_cast<int32_t>(V), stream_of(logits));
    });
  return wrap(std::move(out));
}
PyObject* sample_tokens(PyObject* const* a) { return sample(a, false); }
PyObject* sample_candidates(PyObject* const* a) { return sample(a, true); }

// ---- decode-step inputs ---------------------------------------------------------------------

struct Sections {  // byte offsets of the staging block (decode_inputs.layout)
  int64_t tokens, lens, temperatures, offsets, blocks;
  explicit Sections(int64_t n) : tokens(0), lens(8 * n), temperatures(12 * n), offsets(16 * n), blocks(16 * n + 4 * (n + 1)) {}
};

// Packs the sequences of a step into `buf`, in one pass over them: 40 us of list comprehensions at
// batch 256 became attribute look-ups and stores.
void pack_into(PyObject* seqs_obj, unsigned char* buf, int64_t size, bool with_temperatures, PyObject* temps_obj, int64_t* end,
               int64_t* widest, int64_t* count) {
  Ref seqs(PySequence_Fast(seqs_obj, "seqs must be a sequence"));
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seqs.o);
  const Sections off(n);
  auto too_small = [&](int64_t need) {
    raise(PyExc_ValueError, "staging block of " + std::to_string(size) + " bytes too small for " + std::to_string(n) +
                                " sequences (" + std::to_string(need) + " bytes or more)");
  };
  if (off.blocks > size) too_small(off.blocks);
  auto put = [&](int64_t at, auto v) { std::memcpy(buf + at, &v, sizeof(v)); };
  int64_t total = 0, wide = 0;
  put(off.offsets, static_cast<int32_t>(0));
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* s = PySequence_Fast_GET_ITEM(seqs.o, i);
    put(off.tokens + 8 * i, attr_i64(s, names.last_token));
    {
      Ref len(PyObject_GetAttr(s, names.num_tokens));
      put(off.lens + 4 * i, as_i32(len.o));
    }
    if (with_temperatures && temps_obj == Py_None) {
      Ref t(PyObject_GetAttr(s, names.temperature));
      put(off.temperatures + 4 * i, static_cast<float>(as_double(t.o)));
    }
    Ref table(PyObject_GetAttr(s, names.block_table));
    Ref blocks(PySequence_Fast(table.o, "block_table must be a sequence"));
    const Py_ssize_t m = PySequence_Fast_GET_SIZE(blocks.o);
    if (off.blocks + 4 * (total + m) > size) too_small(off.blocks + 4 * (total + m));
    for (Py_ssize_t j = 0; j < m; ++j) put(off.blocks + 4 * (total + j), as_i32(PySequence_Fast_GET_ITEM(blocks.o, j)));
    total += m;
    wide = std::max<int64_t>(wide, m);
    put(off.offsets + 4 * (i + 1), static_cast<int32_t>(total));
  }
  if (temps_obj != Py_None) {
    Ref temps(PySequence_Fast(temps_obj, "temperatures must be a sequence"));
    if (PySequence_Fast_GET_SIZE(temps.o) != n) raise(PyExc_ValueError, "one temperature per sequence");
    for (Py_ssize_t i = 0; i < n; ++i)
      put(off.temperatures + 4 * i, static_cast<float>(as_double(PySequence_Fast_GET_ITEM(temps.o, i))));
  }
  *end = off.blocks + 4 * total;
  *widest = wide;
  *count = n;
}

PyObject* pack(PyObject* const* a) {  // seqs, buf, with_temperatures, temperatures
  const int with = PyObject_IsTrue(a[2]);
  if (with < 0) throw PyErrorSet{};
  Py_buffer view;
  if (PyObject_GetBuffer(a[1], &view, PyBUF_WRITABLE | PyBUF_SIMPLE) != 0) throw PyErrorSet{};
  int64_t end, widest, n;
  try {
    pack_into(a[0], static_cast<unsigned char*>(view.buf), view.len, with, a[3], &end, &widest, &n);
  } catch (...) {
    PyBuffer_Release(&view);
    throw;
  }
  PyBuffer_Release(&view);
  return Py_BuildValue("LL", static_cast<long long>(end), static_cast<long long>(widest));
}

// Two pinned host blocks used in turn, each guarded by the event of the launch that last read it,
// so that packing a step never overwrites bytes that a launch still in flight is reading.
struct Stager {
  at::Tensor host[2], temperatures;
  cudaEvent_t read[2] = {nullptr, nullptr};
  bool used[2] = {false, false};
  int turn = 0;
  int64_t max_bs, width;
  // A launch that is still pending reads its block, which goes back to the pinned allocator with this object.
  ~Stager() {
    for (int t = 0; t < 2; ++t) {
      if (!read[t]) continue;
      if (used[t] && cudaEventQuery(read[t]) == cudaErrorNotReady) {
        Py_BEGIN_ALLOW_THREADS
        cudaEventSynchronize(read[t]);
        Py_END_ALLOW_THREADS
      }
      cudaEventDestroy(read[t]);
    }
    (void)cudaGetLastError();
  }
};
constexpr const char* kStagerName = "nano_vllm_b200.stager";

void cuda_check(cudaError_t e) {
  if (e != cudaSuccess) raise(PyExc_RuntimeError, std::string("CUDA error: ") + cudaGetErrorString(e));
}

// Returns when the launch that last read block t is done.  Other threads run while it is still pending, and what
// they did meanwhile is looked at again: one of them may have staged from the same block.
void wait_until_read(const Stager& s, int t) {
  while (s.used[t]) {
    cudaError_t e = cudaEventQuery(s.read[t]);
    if (e == cudaSuccess) return;
    if (e == cudaErrorNotReady) {
      (void)cudaGetLastError();
      Py_BEGIN_ALLOW_THREADS
      e = cudaEventSynchronize(s.read[t]);
      Py_END_ALLOW_THREADS
    }
    cuda_check(e);
  }
}

PyObject* make_stager(PyObject* const* a) {  // host block 0, host block 1, device temperatures, max_bs, table_width
  auto s = std::make_unique<Stager>();
  s->host[0] = tensor(a[0], "host block");
  s->host[1] = tensor(a[1], "host block");
  s->temperatures = tensor(a[2], "temperatures");
  s->max_bs = as_i64(a[3]);
  s->width = as_i64(a[4]);
  const c10::cuda::CUDAGuard guard(s->temperatures.device());
  for (cudaEvent_t& e : s->read) cuda_check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  PyObject* c = PyCapsule_New(s.get(), kStagerName, [](PyObject* o) {
    delete static_cast<Stager*>(PyCapsule_GetPointer(o, kStagerName));
  });
  if (!c) throw PyErrorSet{};
  s.release();
  return c;
}

PyObject* stage(PyObject* const* a) {
  // stager, seqs, graph_bs, with_temperatures, temperatures, input_ids, positions, slot_mapping, context_lens, block_tables
  auto* s = static_cast<Stager*>(PyCapsule_GetPointer(a[0], kStagerName));
  if (!s) throw PyErrorSet{};
  const int64_t graph_bs = as_i64(a[2]);
  const int with = PyObject_IsTrue(a[3]);
  if (with < 0) throw PyErrorSet{};
  const Py_ssize_t n0 = PySequence_Size(a[1]);
  if (n0 < 0) throw PyErrorSet{};
  require(0 < n0 && n0 <= graph_bs && graph_bs <= s->max_bs, "0 < n <= graph_bs <= self.max_bs");
  const int t = s->turn;
  s->turn ^= 1;
  wait_until_read(*s, t);
  int64_t end, widest, n;
  pack_into(a[1], ptr<unsigned char>(s->host[t]), s->host[t].numel(), with, a[4], &end, &widest, &n);
  const at::Tensor &ids = tensor(a[5], "input_ids"), &pos = tensor(a[6], "positions"), &slots = tensor(a[7], "slot_mapping"),
                   &lens = tensor(a[8], "context_lens"), &bt = tensor(a[9], "block_tables");
  require(bt.dim() == 2 && bt.size(1) == s->width && widest <= s->width,
          "bt.shape[1] == self.table_width and widest <= self.table_width");
  const Sections off(n);
  const bool temps = with || a[4] != Py_None;
  const c10::cuda::CUDAGuard guard(s->temperatures.device());
  void* st = stream_of(s->temperatures);
  launch([&] {
    return api.decode_step_inputs_pinned(s->host[t].data_ptr(), off.tokens, off.lens, off.offsets, off.blocks,
                                         off.temperatures, temps ? ptr<float>(s->temperatures) : nullptr,
                                         static_cast<int32_t>(n), static_cast<int32_t>(graph_bs),
                                         static_cast<int32_t>(widest), static_cast<int32_t>(s->width), ptr<int64_t>(ids),
                                         ptr<int64_t>(pos), ptr<int32_t>(slots), ptr<int32_t>(lens), ptr<int32_t>(bt),
                                         bt.stride(0), st);
  });
  cuda_check(cudaEventRecord(s->read[t], static_cast<cudaStream_t>(st)));
  s->used[t] = true;
  return wrap(s->temperatures.narrow(0, 0, n));
}

// ---- module ------------------------------------------------------------------------------------

PyObject* bind(PyObject* const* a) {  // library path, check
  const char* path = PyUnicode_AsUTF8(a[0]);
  if (!path) throw PyErrorSet{};
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);  // the handle the ctypes loader already holds
  if (!lib) raise(PyExc_ImportError, dlerror());
#define RESOLVE(name)                                                            \
  api.name = reinterpret_cast<decltype(api.name)>(dlsym(lib, "nvllm_" #name));   \
  if (!api.name) raise(PyExc_ImportError, "nvllm_" #name " is missing from the library")
  RESOLVE(store_kvcache);
  RESOLVE(decode_paged);
  RESOLVE(decode_step);
  RESOLVE(decode_workspace_bytes);
  RESOLVE(prefill_varlen);
  RESOLVE(attention_decode);
  RESOLVE(attention_prefill);
  RESOLVE(qk_norm_rope_store);
  RESOLVE(sample_tokens);
  RESOLVE(sample_candidates);
  RESOLVE(decode_step_inputs_pinned);
#undef RESOLVE
  Py_INCREF(a[1]);
  Py_XSETREF(g_check, a[1]);
#define NAME(x) \
  if (!names.x) names.x = PyUnicode_InternFromString(#x)
  NAME(num_heads); NAME(head_dim); NAME(scale); NAME(num_kv_heads); NAME(k_cache); NAME(v_cache); NAME(is_prefill);
  NAME(cu_seqlens_q); NAME(cu_seqlens_k); NAME(max_seqlen_q); NAME(max_seqlen_k); NAME(slot_mapping); NAME(context_lens);
  NAME(block_tables); NAME(last_token); NAME(num_tokens); NAME(temperature); NAME(block_table);
#undef NAME
  Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject* const*), int NARGS>
PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != NARGS) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", NARGS, nargs);
    return nullptr;
  }
  try {
    return F(args);
  } catch (const PyErrorSet&) {
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    if (type) PyErr_SetString(type, e.what());
    Py_XDECREF(type);
    Py_XDECREF(torch);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

#define METHOD(name, nargs) \
  {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&call<name, nargs>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    METHOD(bind, 2),
    METHOD(clear_workspaces, 0),
    METHOD(store_kvcache, 5),
    METHOD(decode_paged, 7),
    METHOD(decode_step, 10),
    METHOD(prefill_varlen, 10),
    METHOD(attention_forward, 6),
    METHOD(qk_norm_rope_store, 12),
    METHOD(sample_tokens, 6),
    METHOD(sample_candidates, 7),
    METHOD(pack, 4),
    METHOD(make_stager, 5),
    METHOD(stage, 10),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Host path of nano_vllm_b200's entry points.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host() { return PyModule_Create(&module); }
