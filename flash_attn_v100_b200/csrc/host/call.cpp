// The host side of a call of the attention operators in one native step: checks, output, scratch and stream, then the C entry point.
//
// What bounds a small call is the host: a decode of four short sequences runs 6 us on the GPU, and its call took 17.9 us in Python and
// ctypes, 5.9 here (a pass among others 17.95 -> 8.2 us, packed prefill of three short prompts 21.2 -> 16.4).  Every function here takes the arguments of its operator in ops.py and returns the result, or None where the call is anything
// but the plain case (another tensor type, a shape or type that does not fit, no scratch for this stream yet, a mode or transform that is active): ops.py then
// goes on as it would without this module, which is where every refusal and its message come from.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <climits>

#include "../../../include/fa_b200.h"

namespace {

struct Entries {
  decltype(&fa_last_error) last_error;
  decltype(&fa_decode_workspace_bytes) workspace_bytes;
  decltype(&fa_paged_decode_gqa_f16) paged, paged_bf16, paged_out_bf16;
  decltype(&fa_decode_gqa_f16) decode, decode_bf16;
  decltype(&fa_decode_varlen_f16) contig;
  decltype(&fa_decode_sliding_window_gqa_f16) window;
  decltype(&fa_decode_int8_kv_cache_gqa) int8_kv;
  decltype(&fa_decode_int8_gqa) int8_qk;
  decltype(&fa_prefill_dense_f16) dense, dense_bf16;
  decltype(&fa_prefill_varlen_zeroed) varlen;
};
Entries g;
PyObject* g_workspaces = nullptr;      // ops._workspaces: (device, stream) -> uint8 tensor

// Arguments of a call, looked at once.  `ok` turns false where the call is not the plain case.
struct Call {
  bool ok = true;
  int dev = -1;

  explicit Call(bool enough) : ok(enough && g_workspaces != nullptr) {
    if (at::impl::torch_function_mode_enabled() || c10::impl::TorchDispatchModeTLS::any_modes_set()) ok = false;
  }
  // A contiguous tensor with that type and number of dimensions on the current CUDA device, with memory of its own.
  const at::Tensor* tensor(PyObject* o, at::ScalarType type, int64_t dims) {
    if (!ok || !THPVariable_CheckExact(o)) {
      ok = false;
      return nullptr;
    }
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.defined() || !t.is_cuda()) {
      ok = false;
      return nullptr;
    }
    if (dev < 0) dev = c10::cuda::current_device();
    const auto ks = t.key_set();
    ok = t.has_storage() && t.get_device() == dev && t.scalar_type() == type && t.dim() == dims && t.is_contiguous() &&
         !ks.has(c10::DispatchKey::Functionalize) && !ks.has(c10::DispatchKey::FuncTorchBatched) && !ks.has(c10::DispatchKey::FuncTorchGradWrapper) &&
         !ks.has(c10::DispatchKey::Python);
    return ok ? &t : nullptr;
  }
  int integer(PyObject* o) {
    if (!ok || !PyLong_CheckExact(o)) {
      ok = false;
      return 0;
    }
    int overflow = 0;
    const long v = PyLong_AsLongAndOverflow(o, &overflow);
    if (overflow != 0 || v < INT_MIN || v > INT_MAX) ok = false;
    return (int)v;
  }
  int flag(PyObject* o) {
    if (o == Py_True) return 1;
    if (o == Py_False) return 0;
    return integer(o) != 0;
  }
  void need(bool cond) { ok = ok && cond; }
  void heads(int64_t hq, int64_t hkv) { need(hkv > 0 && hq >= hkv && hq % hkv == 0); }
  static bool fits(const at::Tensor* t) { return t->numel() > 0 && t->numel() <= (int64_t)INT_MAX * 64; }
};

cudaStream_t stream_of(int dev) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(); }

// Scratch of this stream, or null (none yet, or too small).  The dictionary keeps every buffer that a launch has had alive.
void* workspace(int dev, cudaStream_t s, int B, int HQ, int HKV, int D, size_t* bytes) {
  const size_t need = g.workspace_bytes(B, HQ, HKV, D);
  if (need == 0) return nullptr;
  PyObject* key = Py_BuildValue("(iK)", dev, (unsigned long long)reinterpret_cast<uintptr_t>(s));
  if (key == nullptr) return nullptr;
  PyObject* ws = PyDict_GetItemWithError(g_workspaces, key);      // borrowed
  Py_DECREF(key);
  if (ws == nullptr || !THPVariable_Check(ws)) {
    PyErr_Clear();
    return nullptr;
  }
  const at::Tensor& t = THPVariable_Unpack(ws);
  *bytes = (size_t)t.numel();
  return *bytes >= need ? t.data_ptr() : nullptr;
}

PyObject* result(int rc, const at::Tensor& out) {
  if (rc != 0) {
    const char* why = g.last_error();
    PyErr_SetString(PyExc_RuntimeError, why != nullptr && why[0] != 0 ? why : "a call of the attention library failed");
    return nullptr;
  }
  return THPVariable_Wrap(out);
}

#define FA_LAUNCH(...)          \
  do {                          \
    Py_BEGIN_ALLOW_THREADS      \
    rc = (__VA_ARGS__);         \
    Py_END_ALLOW_THREADS        \
  } while (0)

// What the decodes share: q [B, HQ, 1, D] against k, v of one shape, the output, the scratch.
struct Decode {
  const at::Tensor *q, *k, *v;
  int B, HQ, HKV, N, D;
  at::Tensor out;
  void* ws = nullptr;
  size_t ws_bytes = 0;
  cudaStream_t s = nullptr;

  Decode(Call& c, PyObject* const* a, at::ScalarType q_type, at::ScalarType kv_type) {
    q = c.tensor(a[0], q_type, 4);
    k = c.tensor(a[1], kv_type, 4);
    v = c.tensor(a[2], kv_type, 4);
    if (!c.ok) return;
    c.need(q->size(2) == 1 && k->sizes() == v->sizes() && q->size(3) == k->size(3) && q->size(3) <= 256 && Call::fits(q) && Call::fits(k));
    c.need(k->size(0) <= INT_MAX && k->size(2) <= INT_MAX);
    c.heads(q->size(1), k->size(1));
    if (!c.ok) return;
    B = (int)q->size(0); HQ = (int)q->size(1); HKV = (int)k->size(1); N = (int)k->size(2); D = (int)q->size(3);
  }
  // Last of the checks: output and scratch.
  bool ready(Call& c, at::ScalarType out_type) {
    if (!c.ok) return false;
    s = stream_of(c.dev);
    ws = workspace(c.dev, s, B, HQ, HKV, D, &ws_bytes);
    if (ws == nullptr) return false;
    out = at::empty({B, HQ, 1, D}, q->options().dtype(out_type));
    return true;
  }
  bool same_batch() const { return q->size(0) == k->size(0); }
};

// (q, k_cache, v_cache, block_table, seq_lens, max_num_blocks, bfloat16 elements, bfloat16 result)
PyObject* paged(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 8);
  if (!c.ok) Py_RETURN_NONE;
  const int bf = c.flag(a[6]), out_bf = c.flag(a[7]);
  const at::ScalarType type = bf ? at::kBFloat16 : at::kHalf;
  Decode d(c, a, type, type);
  const at::Tensor *table = c.tensor(a[3], at::kInt, 2), *lens = c.tensor(a[4], at::kInt, 1);
  const int width = c.integer(a[5]);
  if (!c.ok) Py_RETURN_NONE;
  c.need(d.N == 16 && table->size(0) == d.B && lens->size(0) == d.B && width > 0);
  const int64_t used = std::min<int64_t>(width, table->size(1));
  c.need((int64_t)(d.B - 1) * width + used <= table->numel());
  if (!d.ready(c, bf || out_bf ? at::kBFloat16 : at::kHalf)) Py_RETURN_NONE;
  int rc;
  FA_LAUNCH((bf ? g.paged_bf16 : (out_bf ? g.paged_out_bf16 : g.paged))(
      d.q->data_ptr(), d.k->data_ptr(), d.v->data_ptr(), d.out.data_ptr(), table->data_ptr<int32_t>(), lens->data_ptr<int32_t>(), d.B, d.HQ, d.HKV, d.D,
      d.k->size(0), width, used * 16, d.ws, d.ws_bytes, d.s));
  return result(rc, d.out);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, causal, cache_len, bfloat16 elements)
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 6);
  if (!c.ok) Py_RETURN_NONE;
  const int bf = c.flag(a[5]), causal = c.flag(a[3]), len = c.integer(a[4]);
  const at::ScalarType type = bf ? at::kBFloat16 : at::kHalf;
  Decode d(c, a, type, type);
  if (!c.ok) Py_RETURN_NONE;
  c.need(d.same_batch() && len >= 0 && len < d.N);
  if (!d.ready(c, type)) Py_RETURN_NONE;
  int rc;
  FA_LAUNCH((bf ? g.decode_bf16 : g.decode)(d.q->data_ptr(), d.k->data_ptr(), d.v->data_ptr(), d.out.data_ptr(), d.B, d.HQ, d.HKV, d.N, d.D, causal, len,
                                            d.ws, d.ws_bytes, d.s));
  return result(rc, d.out);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, cache_lens, causal)
PyObject* contig(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 5);
  if (!c.ok) Py_RETURN_NONE;
  Decode d(c, a, at::kHalf, at::kHalf);
  const at::Tensor* lens = c.tensor(a[3], at::kInt, 1);
  const int causal = c.flag(a[4]);
  if (!c.ok) Py_RETURN_NONE;
  c.need(d.same_batch() && lens->size(0) == d.B);
  if (!d.ready(c, at::kHalf)) Py_RETURN_NONE;
  int rc;
  FA_LAUNCH(g.contig(d.q->data_ptr(), d.k->data_ptr(), d.v->data_ptr(), d.out.data_ptr(), lens->data_ptr<int32_t>(), d.B, d.HQ, d.HKV, d.N, d.D, causal, d.ws,
                     d.ws_bytes, d.s));
  return result(rc, d.out);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, cache_len, window_size, sink_size)
PyObject* window(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 6);
  if (!c.ok) Py_RETURN_NONE;
  const int len = c.integer(a[3]), size = c.integer(a[4]), sink = c.integer(a[5]);
  Decode d(c, a, at::kHalf, at::kHalf);
  if (!c.ok) Py_RETURN_NONE;
  c.need(d.same_batch());
  if (!d.ready(c, at::kHalf)) Py_RETURN_NONE;
  int rc;
  FA_LAUNCH(g.window(d.q->data_ptr(), d.k->data_ptr(), d.v->data_ptr(), d.out.data_ptr(), d.B, d.HQ, d.HKV, d.N, d.D, len, size, sink, d.ws, d.ws_bytes, d.s));
  return result(rc, d.out);
  END_HANDLE_TH_ERRORS
}

bool scales_fit(const Decode& d, const at::Tensor* t) { return t->size(0) == d.B && t->size(1) == d.HKV && t->size(2) == d.N; }

// (q, k, v, k_scale, v_scale, cache_len)
PyObject* int8_kv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 6);
  if (!c.ok) Py_RETURN_NONE;
  const int len = c.integer(a[5]);
  Decode d(c, a, at::kHalf, at::kChar);
  const at::Tensor *ks = c.tensor(a[3], at::kHalf, 3), *vs = c.tensor(a[4], at::kHalf, 3);
  if (!c.ok) Py_RETURN_NONE;
  c.need(d.same_batch() && scales_fit(d, ks) && scales_fit(d, vs));
  if (!d.ready(c, at::kHalf)) Py_RETURN_NONE;
  int rc;
  FA_LAUNCH(g.int8_kv(d.q->data_ptr(), d.k->data_ptr(), d.v->data_ptr(), ks->data_ptr(), vs->data_ptr(), d.out.data_ptr(), d.B, d.HQ, d.HKV, d.N, d.D, len, d.ws,
                      d.ws_bytes, d.s));
  return result(rc, d.out);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, q_scale, k_scale, cache_len)
PyObject* int8_qk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 6);
  if (!c.ok) Py_RETURN_NONE;
  const int len = c.integer(a[5]);
  Decode d(c, a, at::kHalf, at::kHalf);
  const at::Tensor *qs = c.tensor(a[3], at::kFloat, 2), *ks = c.tensor(a[4], at::kFloat, 3);
  if (!c.ok) Py_RETURN_NONE;
  c.need(d.same_batch() && qs->size(0) == d.B && qs->size(1) == d.HQ && scales_fit(d, ks) && len >= 0 && len < d.N);
  if (!d.ready(c, at::kHalf)) Py_RETURN_NONE;
  int rc;
  FA_LAUNCH(g.int8_qk(d.q->data_ptr(), d.k->data_ptr(), d.v->data_ptr(), d.out.data_ptr(), qs->data_ptr<float>(), ks->data_ptr<float>(), d.B, d.HQ, d.HKV, d.N,
                      d.D, len, nullptr, d.ws, d.ws_bytes, d.s));
  return result(rc, d.out);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, causal, bfloat16 elements)
PyObject* dense(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 5);
  if (!c.ok) Py_RETURN_NONE;
  const int causal = c.flag(a[3]), bf = c.flag(a[4]);
  const at::ScalarType type = bf ? at::kBFloat16 : at::kHalf;
  const at::Tensor *q = c.tensor(a[0], type, 4), *k = c.tensor(a[1], type, 4), *v = c.tensor(a[2], type, 4);
  if (!c.ok) Py_RETURN_NONE;
  c.need(k->sizes() == v->sizes() && q->size(0) == k->size(0) && q->size(2) == k->size(2) && q->size(3) == k->size(3) && q->size(3) <= 256 &&
         q->size(0) <= INT_MAX && q->size(2) <= INT_MAX && Call::fits(q) && Call::fits(k));
  c.heads(q->size(1), k->size(1));
  if (!c.ok) Py_RETURN_NONE;
  const at::Tensor out = at::empty(q->sizes(), q->options());
  const cudaStream_t s = stream_of(c.dev);
  int rc;
  FA_LAUNCH((bf ? g.dense_bf16 : g.dense)(q->data_ptr(), k->data_ptr(), v->data_ptr(), out.data_ptr(), (int)q->size(0), (int)q->size(1), (int)k->size(1),
                                          (int)q->size(2), (int)q->size(3), causal, s));
  return result(rc, out);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, cu_seqlens, max_seqlen, causal, bfloat16 elements, bfloat16 result)
PyObject* varlen(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  Call c(n == 8);
  if (!c.ok) Py_RETURN_NONE;
  const int longest = c.integer(a[4]), causal = c.flag(a[5]), bf = c.flag(a[6]), out_bf = c.flag(a[7]);
  const at::ScalarType type = bf ? at::kBFloat16 : at::kHalf;
  const at::Tensor *q = c.tensor(a[0], type, 3), *k = c.tensor(a[1], type, 3), *v = c.tensor(a[2], type, 3), *cu = c.tensor(a[3], at::kInt, 1);
  if (!c.ok) Py_RETURN_NONE;
  c.need(k->sizes() == v->sizes() && q->size(0) == k->size(0) && q->size(2) == k->size(2) && q->size(2) <= 256 && q->size(2) % 8 == 0 && longest > 0 &&
         cu->size(0) > 1 && cu->size(0) <= INT_MAX && Call::fits(q) && Call::fits(k));
  c.heads(q->size(1), k->size(1));
  if (!c.ok) Py_RETURN_NONE;
  const at::Tensor out = at::empty(q->sizes(), q->options().dtype(bf || out_bf ? at::kBFloat16 : at::kHalf));
  const cudaStream_t s = stream_of(c.dev);
  const int batch = (int)cu->size(0) - 1, HQ = (int)q->size(1), D = (int)q->size(2);
  int rc;
  FA_LAUNCH(g.varlen(q->data_ptr(), k->data_ptr(), v->data_ptr(), out.data_ptr(), cu->data_ptr<int32_t>(), batch, q->size(0), HQ, (int)k->size(1), D, longest,
                     causal, bf, out_bf, s));
  return result(rc, out);
  END_HANDLE_TH_ERRORS
}

// bind(entry addresses by name, ops._workspaces)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyDict_Check(a[0]) || !PyDict_Check(a[1])) {
    PyErr_SetString(PyExc_TypeError, "bind takes two dictionaries");
    return nullptr;
  }
  bool ok = true;
  auto get = [&](const char* name, auto& fn) {
    PyObject* v = PyDict_GetItemString(a[0], name);
    void* p = v != nullptr ? PyLong_AsVoidPtr(v) : nullptr;
    ok = ok && p != nullptr;
    fn = reinterpret_cast<std::remove_reference_t<decltype(fn)>>(p);
  };
  get("fa_last_error", g.last_error);
  get("fa_decode_workspace_bytes", g.workspace_bytes);
  get("fa_paged_decode_gqa_f16", g.paged);
  get("fa_paged_decode_gqa_bf16", g.paged_bf16);
  get("fa_paged_decode_gqa_f16_out_bf16", g.paged_out_bf16);
  get("fa_decode_gqa_f16", g.decode);
  get("fa_decode_gqa_bf16", g.decode_bf16);
  get("fa_decode_varlen_f16", g.contig);
  get("fa_decode_sliding_window_gqa_f16", g.window);
  get("fa_decode_int8_kv_cache_gqa", g.int8_kv);
  get("fa_decode_int8_gqa", g.int8_qk);
  get("fa_prefill_dense_f16", g.dense);
  get("fa_prefill_dense_bf16", g.dense_bf16);
  get("fa_prefill_varlen_zeroed", g.varlen);
  if (!ok) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "an entry point is missing");
    return nullptr;
  }
  Py_INCREF(a[1]);
  Py_XSETREF(g_workspaces, a[1]);
  Py_RETURN_NONE;
}

#define FA_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {FA_METHOD(bind),   FA_METHOD(paged),   FA_METHOD(decode), FA_METHOD(contig), FA_METHOD(window),
                           FA_METHOD(int8_kv), FA_METHOD(int8_qk), FA_METHOD(dense),  FA_METHOD(varlen), {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_call", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__call(void) {
  PyObject* m = PyModule_Create(&g_module);
  if (m != nullptr && (PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) != 0 || PyModule_AddStringConstant(m, "built_for", FA_BUILT_FOR) != 0)) Py_CLEAR(m);
  return m;
}
