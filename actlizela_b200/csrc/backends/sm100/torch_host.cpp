// Native host path of the Python entry points: argument checks, output allocation and the C-ABI call of one pass in
// one extension function.  The Python wrappers keep the full checks and their messages: a function here returns None
// for anything it does not take (another device current, an ill-formed operand, a failure record to report, a library
// selected by the environment other than the one bound), and the wrapper then goes its own way, which raises or runs.
//
// Why native: a small pass is host bound.  The wrappers spent 9-30 us per call (attribute reads, device guards, ctypes)
// against 2-10 us of kernel time; these functions take 3-5 us including the launch.
//
// Holds no state but the bound addresses and which devices are configured; outputs and scratch come from torch's caching
// allocator per call, on the caller's current stream, so calls from several threads, on several streams and under
// stream capture behave like the wrappers.
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

namespace {
using at::Tensor;
using P = const void*;
using LL = long long;

struct Entries {
  int (*select)(int, int, int, int, int);
  LL (*workspace_bytes)(int, int, int, int, int);
  int (*forward)(P, P, P, P, P, const float*, void*, float*, void*, LL, int, int, int, int, int, int, void*);
  LL (*varlen_workspace_bytes)(LL, int, int, int);
  int (*varlen_host)(P, P, P, P, P, const float*, void*, float*, void*, LL, const int*, int, int, int, int, void*);
  int (*varlen_device)(P, P, P, P, P, const float*, void*, float*, void*, LL, const int*, int, LL, int, int, int, void*);
  LL (*projections_workspace_bytes)(int, int, int, int, int);
  int (*projections)(P, LL, P, P, const float*, const float*, const float*, void*, float*, void*, LL, int, int, int, int, int, void*);
  int (*last_failure)(int*);
  int (*prepare_inputs)(P, LL, P, P, const float*, const float*, void*, void*, void*, float*, void*, LL, int, int, void*);
  int (*decode_step)(P, P, P, P, P, float*, void*, int, int, int, int, void*);
  int (*verify_step)(P, P, P, P, P, const float*, void*, float*, int, int, int, int, int, void*);
  int (*commit_step)(P, P, const float*, const int*, float*, int, int, int, int, int, void*);
  int (*rmsnorm_gated)(P, P, P, void*, LL, void*);
  int (*out_proj)(P, P, void*, int, int, int, void*);
};
constexpr int kEntries = sizeof(Entries) / sizeof(void*);
constexpr int kDevices = 64;
Entries g_entries;
bool g_bound = false;
bool g_has_override = false;
std::string g_override;
bool g_configured[kDevices] = {};

// -------------------------------------------------------------------------------------------------- operand checks
// One call's operands: `ok` turns false at the first that the call does not take.
struct Operands {
  bool ok = true;
  int device = -1;
  const Tensor* take(PyObject* o, at::ScalarType dtype, int64_t ndim, bool aligned = true) {
    return take(o, dtype, dtype, ndim, aligned);
  }
  const Tensor* take(PyObject* o, at::ScalarType dtype, at::ScalarType other, int64_t ndim, bool aligned = true) {
    if (!ok || !THPVariable_Check(o)) return fail();
    const Tensor& t = THPVariable_Unpack(o);
    const auto type = t.scalar_type();
    if (!t.is_cuda() || (type != dtype && type != other) || (ndim >= 0 && t.dim() != ndim) || t.requires_grad() ||
        !t.is_contiguous() || (aligned && (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15)))
      return fail();
    const int at = t.get_device();
    if (device < 0) device = at;
    else if (device != at) return fail();
    return &t;
  }
  const Tensor* fail() {
    ok = false;
    return nullptr;
  }
  void require(bool condition) { ok = ok && condition; }
};
bool shape_is(const Tensor& t, std::initializer_list<int64_t> shape) { return t.sizes().equals(at::IntArrayRef(shape.begin(), shape.size())); }

// the bound library is the selected one, the operands' device is current (and configured, where kernels need that) and
// no earlier launch left a failure record
bool ready(const Operands& x, bool configured) {
  if (!x.ok || !g_bound || x.device < 0 || x.device >= kDevices || x.device != c10::cuda::current_device()) return false;
  if (configured && !g_configured[x.device]) return false;
  const char* selected = std::getenv("ACTLIZE_LA_SM100_LIBRARY");
  if ((selected != nullptr) != g_has_override || (selected && g_override != selected)) return false;
  if (configured) {
    int record[4];
    if (g_entries.last_failure(record) || record[0]) return false;
  }
  return true;
}
void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream(device).stream(); }
Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, int device) {
  return at::detail::empty_cuda(shape, dtype, c10::Device(c10::kCUDA, device), c10::nullopt);
}
const float* floats(const Tensor* t) { return t ? static_cast<const float*>(t->const_data_ptr()) : nullptr; }
bool is_fp32(const Tensor& t) { return t.scalar_type() == at::kFloat; }
PyObject* none() { Py_RETURN_NONE; }
PyObject* failed(int code) {
  PyErr_Format(PyExc_RuntimeError, "cuda_sm100 native call failed with CUDA error code %d", code);
  return nullptr;
}
PyObject* pair(const Tensor& a, const Tensor* b) {
  PyObject* tuple = PyTuple_New(2);
  if (!tuple) return nullptr;
  PyTuple_SET_ITEM(tuple, 0, THPVariable_Wrap(a));
  if (b) PyTuple_SET_ITEM(tuple, 1, THPVariable_Wrap(*b));
  else {
    Py_INCREF(Py_None);
    PyTuple_SET_ITEM(tuple, 1, Py_None);
  }
  return tuple;
}
bool truth(PyObject* o, bool& ok) {
  const int value = PyObject_IsTrue(o);
  if (value < 0) {
    PyErr_Clear();
    ok = false;
  }
  return value > 0;
}
int small_int(PyObject* o, bool& ok) {
  if (!PyLong_CheckExact(o)) {
    ok = false;
    return 0;
  }
  const long value = PyLong_AsLong(o);
  if (value < 1 || value > (1 << 24)) {
    PyErr_Clear();
    ok = false;
  }
  return int(value);
}
bool fits(std::initializer_list<int64_t> sizes) {
  for (int64_t s : sizes)
    if (s < 1 || s > INT32_MAX) return false;
  return true;
}

#define GDN_ENTRY(name, count)                                                     \
  PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t nargs) {             \
    HANDLE_TH_ERRORS                                                               \
    if (nargs != (count)) return none();                                           \
    Operands x;
#define GDN_END END_HANDLE_TH_ERRORS }

// forward(q, k, v, g, beta, initial_state | None, output_final_state)
GDN_ENTRY(forward, 7)
  const Tensor *q = x.take(args[0], at::kBFloat16, 4), *k = x.take(args[1], at::kBFloat16, 4), *v = x.take(args[2], at::kBFloat16, 4);
  const Tensor *g = x.take(args[3], at::kFloat, at::kBFloat16, 3, false), *beta = x.take(args[4], at::kBFloat16, 3, false);
  const Tensor* initial = args[5] == Py_None ? nullptr : x.take(args[5], at::kFloat, 4, false);
  const bool want = truth(args[6], x.ok);
  if (!x.ok) return none();
  const int64_t b = q->size(0), t = q->size(1), hk = q->size(2), hv = v->size(2);
  x.require(fits({b, t, hk, hv}) && q->size(3) == 128 && hv % hk == 0 && k->sizes() == q->sizes() && shape_is(*v, {b, t, hv, 128}) &&
            shape_is(*g, {b, t, hv}) && shape_is(*beta, {b, t, hv}) && (!initial || shape_is(*initial, {b, hv, 128, 128})));
  if (!ready(x, true)) return none();
  const int fp32 = is_fp32(*g), config = g_entries.select(b, t, hk, hv, fp32);
  const LL need = config < 0 ? -1 : g_entries.workspace_bytes(b, t, hk, hv, config);
  if (need < 0) return none();
  Tensor out = empty(v->sizes(), at::kBFloat16, x.device), final_state;
  if (want) final_state = empty({b, hv, 128, 128}, at::kFloat, x.device);
  const Tensor scratch = empty({need}, at::kByte, x.device);
  const int rc = g_entries.forward(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), g->const_data_ptr(), beta->const_data_ptr(),
                                   floats(initial), out.mutable_data_ptr(), want ? static_cast<float*>(final_state.mutable_data_ptr()) : nullptr,
                                   scratch.mutable_data_ptr(), need, b, t, hk, hv, fp32, config, stream_of(x.device));
  return rc ? failed(rc) : pair(out, want ? &final_state : nullptr);
GDN_END

// varlen(q, k, v, g, beta, cu_seqlens, initial_states | None, output_final_state)
GDN_ENTRY(varlen, 8)
  const Tensor *q = x.take(args[0], at::kBFloat16, 4), *k = x.take(args[1], at::kBFloat16, 4), *v = x.take(args[2], at::kBFloat16, 4);
  const Tensor *g = x.take(args[3], at::kFloat, at::kBFloat16, 3, false), *beta = x.take(args[4], at::kBFloat16, 3, false);
  const Tensor *offsets = nullptr, *initial = args[6] == Py_None ? nullptr : x.take(args[6], at::kFloat, 4, false);
  std::vector<int> host;
  if (THPVariable_Check(args[5])) {
    offsets = x.take(args[5], at::kInt, 1, false);
  } else if (PyList_CheckExact(args[5]) || PyTuple_CheckExact(args[5])) {
    const Py_ssize_t count = PySequence_Fast_GET_SIZE(args[5]);
    host.reserve(count);
    for (Py_ssize_t i = 0; i < count && x.ok; ++i) {
      PyObject* item = PySequence_Fast_GET_ITEM(args[5], i);
      const long at = PyLong_CheckExact(item) ? PyLong_AsLong(item) : -1;
      x.require(at >= (host.empty() ? 0 : host.back()) && at <= INT32_MAX);
      host.push_back(int(at));
    }
    if (PyErr_Occurred()) PyErr_Clear();
  } else {
    x.fail();
  }
  const bool want = truth(args[7], x.ok);
  if (!x.ok) return none();
  const int64_t t = q->size(1), hk = q->size(2), hv = v->size(2), n = (offsets ? offsets->numel() : int64_t(host.size())) - 1;
  x.require(fits({n, t, hk, hv}) && q->size(0) == 1 && q->size(3) == 128 && hv % hk == 0 && k->sizes() == q->sizes() &&
            shape_is(*v, {1, t, hv, 128}) && shape_is(*g, {1, t, hv}) && shape_is(*beta, {1, t, hv}) &&
            (!initial || shape_is(*initial, {n, hv, 128, 128})) && (offsets || (host.front() == 0 && host.back() == t)));
  if (!ready(x, true)) return none();
  const LL need = g_entries.varlen_workspace_bytes(t, n, hk, hv);
  if (need < 0) return none();
  const int fp32 = is_fp32(*g);
  Tensor out = empty(v->sizes(), at::kBFloat16, x.device), final_states;
  if (want) final_states = empty({n, hv, 128, 128}, at::kFloat, x.device);
  const Tensor scratch = empty({need}, at::kByte, x.device);
  float* states = want ? static_cast<float*>(final_states.mutable_data_ptr()) : nullptr;
  const int rc = offsets
      ? g_entries.varlen_device(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), g->const_data_ptr(), beta->const_data_ptr(),
                                floats(initial), out.mutable_data_ptr(), states, scratch.mutable_data_ptr(), need,
                                static_cast<const int*>(offsets->const_data_ptr()), n, t, hk, hv, fp32, stream_of(x.device))
      : g_entries.varlen_host(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), g->const_data_ptr(), beta->const_data_ptr(),
                              floats(initial), out.mutable_data_ptr(), states, scratch.mutable_data_ptr(), need, host.data(), n, hk, hv, fp32,
                              stream_of(x.device));
  return rc ? failed(rc) : pair(out, want ? &final_states : nullptr);
GDN_END

// projections(mixed, a, b, a_log, dt_bias, key_heads, value_heads, initial_state | None, output_final_state)
GDN_ENTRY(projections, 9)
  const Tensor *mixed = x.take(args[0], at::kBFloat16, 3), *a = x.take(args[1], at::kBFloat16, 3), *b = x.take(args[2], at::kBFloat16, 3);
  const Tensor *a_log = x.take(args[3], at::kFloat, 1), *dt_bias = x.take(args[4], at::kFloat, 1);
  const Tensor* initial = args[7] == Py_None ? nullptr : x.take(args[7], at::kFloat, 4);
  const int64_t hk = small_int(args[5], x.ok), hv = small_int(args[6], x.ok);
  const bool want = truth(args[8], x.ok);
  if (!x.ok) return none();
  const int64_t bsz = mixed->size(0), t = mixed->size(1);
  x.require(fits({bsz, t}) && hv % hk == 0 && mixed->size(2) == (2 * hk + hv) * 128 && shape_is(*a, {bsz, t, hv}) && shape_is(*b, {bsz, t, hv}) &&
            shape_is(*a_log, {hv}) && shape_is(*dt_bias, {hv}) && (!initial || shape_is(*initial, {bsz, hv, 128, 128})));
  if (!ready(x, true)) return none();
  const int config = g_entries.select(bsz, t, hk, hv, 1);
  const LL need = config < 0 ? -1 : g_entries.projections_workspace_bytes(bsz, t, hk, hv, config);
  if (need < 0) return none();
  Tensor out = empty({bsz, t, hv, 128}, at::kBFloat16, x.device), final_state;
  if (want) final_state = empty({bsz, hv, 128, 128}, at::kFloat, x.device);
  const Tensor scratch = empty({need}, at::kByte, x.device);
  const int rc = g_entries.projections(mixed->const_data_ptr(), mixed->size(2), a->const_data_ptr(), b->const_data_ptr(), floats(a_log),
                                       floats(dt_bias), floats(initial), out.mutable_data_ptr(),
                                       want ? static_cast<float*>(final_state.mutable_data_ptr()) : nullptr, scratch.mutable_data_ptr(), need,
                                       bsz, t, hk, hv, config, stream_of(x.device));
  return rc ? failed(rc) : pair(out, want ? &final_state : nullptr);
GDN_END

// prepare_inputs(mixed, a, b, a_log, dt_bias, key_heads, value_heads)
GDN_ENTRY(prepare_inputs, 7)
  const Tensor *mixed = x.take(args[0], at::kBFloat16, 2), *a = x.take(args[1], at::kBFloat16, 2), *b = x.take(args[2], at::kBFloat16, 2);
  const Tensor *a_log = x.take(args[3], at::kFloat, 1), *dt_bias = x.take(args[4], at::kFloat, 1);
  const int64_t hk = small_int(args[5], x.ok), hv = small_int(args[6], x.ok);
  if (!x.ok) return none();
  const int64_t n = mixed->size(0);
  x.require(fits({n}) && hv % hk == 0 && mixed->size(1) == (2 * hk + hv) * 128 && shape_is(*a, {n, hv}) && shape_is(*b, {n, hv}) &&
            shape_is(*a_log, {hv}) && shape_is(*dt_bias, {hv}));
  if (!ready(x, false)) return none();
  const Tensor out[5] = {empty({n, hk, 128}, at::kBFloat16, x.device), empty({n, hk, 128}, at::kBFloat16, x.device),
                         empty({n, hv, 128}, at::kBFloat16, x.device), empty({n, hv}, at::kFloat, x.device),
                         empty({n, hv}, at::kBFloat16, x.device)};
  const int rc = g_entries.prepare_inputs(mixed->const_data_ptr(), mixed->size(1), a->const_data_ptr(), b->const_data_ptr(), floats(a_log),
                                          floats(dt_bias), out[0].mutable_data_ptr(), out[1].mutable_data_ptr(), out[2].mutable_data_ptr(),
                                          static_cast<float*>(out[3].mutable_data_ptr()), out[4].mutable_data_ptr(), n, hk, hv,
                                          stream_of(x.device));
  if (rc) return failed(rc);
  PyObject* tuple = PyTuple_New(5);
  for (int i = 0; tuple && i < 5; ++i) PyTuple_SET_ITEM(tuple, i, THPVariable_Wrap(out[i]));
  return tuple;
GDN_END

// decode_step(q, k, v, g, beta, state)
GDN_ENTRY(decode_step, 6)
  const Tensor *q = x.take(args[0], at::kBFloat16, 3), *k = x.take(args[1], at::kBFloat16, 3), *v = x.take(args[2], at::kBFloat16, 3);
  const Tensor *g = x.take(args[3], at::kFloat, at::kBFloat16, 2), *beta = x.take(args[4], at::kBFloat16, 2);
  const Tensor* state = x.take(args[5], at::kFloat, 4);
  if (!x.ok) return none();
  const int64_t b = q->size(0), hk = q->size(1), hv = v->size(1);
  x.require(fits({b, hk, hv}) && hv % hk == 0 && q->size(2) == 128 && k->sizes() == q->sizes() && shape_is(*v, {b, hv, 128}) &&
            shape_is(*g, {b, hv}) && shape_is(*beta, {b, hv}) && shape_is(*state, {b, hv, 128, 128}));
  if (!ready(x, false)) return none();
  Tensor out = empty(v->sizes(), at::kBFloat16, x.device);
  const int rc = g_entries.decode_step(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), g->const_data_ptr(), beta->const_data_ptr(),
                                       static_cast<float*>(state->mutable_data_ptr()), out.mutable_data_ptr(), b, hk, hv, is_fp32(*g),
                                       stream_of(x.device));
  return rc ? failed(rc) : THPVariable_Wrap(out);
GDN_END

// verify_step(q, k, v, g, beta, state)
GDN_ENTRY(verify_step, 6)
  const Tensor *q = x.take(args[0], at::kBFloat16, 4), *k = x.take(args[1], at::kBFloat16, 4), *v = x.take(args[2], at::kBFloat16, 4);
  const Tensor *g = x.take(args[3], at::kFloat, at::kBFloat16, 3), *beta = x.take(args[4], at::kBFloat16, 3);
  const Tensor* state = x.take(args[5], at::kFloat, 4);
  if (!x.ok) return none();
  const int64_t b = k->size(0), w = k->size(1), hk = k->size(2), hv = g->size(2);
  x.require(fits({b, w, hk, hv}) && w <= 64 && hv % hk == 0 && k->size(3) == 128 && q->sizes() == k->sizes() && shape_is(*v, {b, w, hv, 128}) &&
            shape_is(*g, {b, w, hv}) && shape_is(*beta, {b, w, hv}) && shape_is(*state, {b, hv, 128, 128}));
  if (!ready(x, false)) return none();
  Tensor out = empty(v->sizes(), at::kBFloat16, x.device), delta = empty(v->sizes(), at::kFloat, x.device);
  const int rc = g_entries.verify_step(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), g->const_data_ptr(), beta->const_data_ptr(),
                                       floats(state), out.mutable_data_ptr(), static_cast<float*>(delta.mutable_data_ptr()), b, w, hk, hv,
                                       is_fp32(*g), stream_of(x.device));
  return rc ? failed(rc) : pair(out, &delta);
GDN_END

// commit_step(k, g, delta, counts, state): the state itself, updated
GDN_ENTRY(commit_step, 5)
  const Tensor *k = x.take(args[0], at::kBFloat16, 4), *g = x.take(args[1], at::kFloat, at::kBFloat16, 3);
  const Tensor *delta = x.take(args[2], at::kFloat, 4), *counts = x.take(args[3], at::kInt, 1), *state = x.take(args[4], at::kFloat, 4);
  if (!x.ok) return none();
  const int64_t b = k->size(0), w = k->size(1), hk = k->size(2), hv = g->size(2);
  x.require(fits({b, w, hk, hv}) && w <= 64 && hv % hk == 0 && k->size(3) == 128 && shape_is(*g, {b, w, hv}) &&
            shape_is(*delta, {b, w, hv, 128}) && shape_is(*counts, {b}) && shape_is(*state, {b, hv, 128, 128}));
  if (!ready(x, false)) return none();
  const int rc = g_entries.commit_step(k->const_data_ptr(), g->const_data_ptr(), floats(delta), static_cast<const int*>(counts->const_data_ptr()),
                                       static_cast<float*>(state->mutable_data_ptr()), b, w, hk, hv, is_fp32(*g), stream_of(x.device));
  if (rc) return failed(rc);
  Py_INCREF(args[4]);
  return args[4];
GDN_END

// rmsnorm_gated(y, z, weight)
GDN_ENTRY(rmsnorm_gated, 3)
  const Tensor *y = x.take(args[0], at::kBFloat16, -1), *z = x.take(args[1], at::kBFloat16, -1), *weight = x.take(args[2], at::kBFloat16, 1);
  if (!x.ok) return none();
  x.require(y->dim() >= 1 && y->numel() > 0 && y->size(-1) == 128 && z->sizes() == y->sizes() && shape_is(*weight, {128}));
  if (!ready(x, false)) return none();
  Tensor out = empty(y->sizes(), at::kBFloat16, x.device);
  const int rc = g_entries.rmsnorm_gated(y->const_data_ptr(), z->const_data_ptr(), weight->const_data_ptr(), out.mutable_data_ptr(),
                                         y->numel() / 128, stream_of(x.device));
  return rc ? failed(rc) : THPVariable_Wrap(out);
GDN_END

// out_proj_gemm(a, w)
GDN_ENTRY(out_proj_gemm, 2)
  const Tensor *a = x.take(args[0], at::kBFloat16, 2), *w = x.take(args[1], at::kBFloat16, 2);
  if (!x.ok) return none();
  const int64_t m = a->size(0), k = a->size(1), n = w->size(0);
  x.require(fits({m, n, k}) && k % 8 == 0 && n % 8 == 0 && w->size(1) == k);
  if (!ready(x, true)) return none();
  Tensor out = empty({m, n}, at::kBFloat16, x.device);
  const int rc = g_entries.out_proj(a->const_data_ptr(), w->const_data_ptr(), out.mutable_data_ptr(), m, n, k, stream_of(x.device));
  return rc ? failed(rc) : THPVariable_Wrap(out);
GDN_END

// bind(addresses in the order of Entries, override | None)
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 2 || !PyTuple_Check(args[0]) || PyTuple_GET_SIZE(args[0]) != kEntries) {
    PyErr_SetString(PyExc_ValueError, "bind expects the entry addresses and the library override");
    return nullptr;
  }
  void* addresses[kEntries];
  for (int i = 0; i < kEntries; ++i) {
    addresses[i] = PyLong_AsVoidPtr(PyTuple_GET_ITEM(args[0], i));
    if (!addresses[i]) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "null entry address");
      return nullptr;
    }
  }
  g_has_override = args[1] != Py_None;
  if (g_has_override) {
    const char* text = PyUnicode_AsUTF8(args[1]);
    if (!text) return nullptr;
    g_override = text;
  }
  std::memcpy(&g_entries, addresses, sizeof(addresses));
  std::memset(g_configured, 0, sizeof(g_configured));
  g_bound = true;
  return none();
}
// configured(device index): the bound library's one-time set-up has run there, on a device of the policy's kind
PyObject* configured(PyObject*, PyObject* arg) {
  const long device = PyLong_AsLong(arg);
  if (device < 0 || device >= kDevices) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "device index out of range");
    return nullptr;
  }
  g_configured[device] = true;
  return none();
}

#define GDN_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(name)), METH_FASTCALL, nullptr}
PyMethodDef g_methods[] = {GDN_METHOD(forward), GDN_METHOD(varlen), GDN_METHOD(projections), GDN_METHOD(prepare_inputs),
                           GDN_METHOD(decode_step), GDN_METHOD(verify_step), GDN_METHOD(commit_step), GDN_METHOD(rmsnorm_gated),
                           GDN_METHOD(out_proj_gemm), GDN_METHOD(bind), {"configured", configured, METH_O, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "actlize_la_sm100_host", nullptr, -1, g_methods};
}  // namespace

PyMODINIT_FUNC PyInit_actlize_la_sm100_host(void) { return PyModule_Create(&g_module); }
