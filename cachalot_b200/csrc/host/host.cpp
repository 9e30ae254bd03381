// Native call path of the operators in ops.py (CPython extension module cachalot_b200._host).
//
// A decode step is a few hundred operator calls of 5-25 us of GPU work each, and the Python form of a call (dtype and
// layout conversions that change nothing, four or five tensor allocations, stream lookup, a ctypes call with up to
// thirty arguments) costs 20-35 us of host time: for small calls the host was the limit (fp8_linear [4096,8192]:
// 27 us per call around 13 us of GPU work).  Each function here is the same call for the plain case - CUDA tensors of
// the current device in the dtype and layout the kernels take - and returns None for everything else, also for every
// argument error: the caller then runs the general form, which converts or raises.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <initializer_list>

#include "../../../include/cachalot_b200.h"

namespace {

using at::ScalarType;

// The entry points of the C ABI, as the addresses _lib.py found in the library it loaded (by default the one beside this
// module, else CACHALOT_B200_LIB): this module links no library of its own, so both ways of a call end in the same one.
#define ENTRIES(X) \
  X(cachalot_bf16_gemv_f32) X(cachalot_fp8_linear) X(cachalot_group_rows) X(cachalot_group_rows_scratch_ints) \
  X(cachalot_last_error) X(cachalot_moe_decode) X(cachalot_moe_decode_workspace_bytes) X(cachalot_moe_layer_decode) \
  X(cachalot_moe_layer_decode_workspace_bytes) X(cachalot_moe_prefill) X(cachalot_moe_prefill_experts_workspace_bytes) X(cachalot_route_topk) \
  X(cachalot_router_logits) X(cachalot_shared_expert) X(cachalot_shared_expert_workspace_bytes)
struct Lib {
#define X(name) decltype(&::name) name = nullptr;
  ENTRIES(X)
#undef X
} lib;
bool bound = false;

// () -> names of the entry points
PyObject* entries(PyObject*, PyObject* const*, Py_ssize_t) {
#define X(name) #name,
  const char* const all[] = {ENTRIES(X)};
#undef X
  PyObject* out = PyList_New(0);
  for (const char* n : all) {
    PyObject* s = out ? PyUnicode_FromString(n) : nullptr;
    if (!s || PyList_Append(out, s) < 0) Py_CLEAR(out);
    Py_XDECREF(s);
  }
  return out;
}
// ({name: address}) -> None
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  if (n_args != 1 || !PyDict_Check(a[0])) return PyErr_Format(PyExc_TypeError, "bind takes a dict of addresses");
  Lib l;
  void* p;
#define X(name)                                                                                              \
  p = PyDict_GetItemString(a[0], #name) ? PyLong_AsVoidPtr(PyDict_GetItemString(a[0], #name)) : nullptr;     \
  if (!p) return PyErr_Occurred() ? nullptr : PyErr_Format(PyExc_ValueError, "no address for " #name);       \
  l.name = reinterpret_cast<decltype(l.name)>(p);
  ENTRIES(X)
#undef X
  lib = l, bound = true;
  Py_RETURN_NONE;
}

const at::Tensor* tensor_of(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// a contiguous tensor of this type on the current device?
bool plain(const at::Tensor* t, ScalarType dt, int device) {
  return t && t->is_cuda() && t->scalar_type() == dt && t->get_device() == device && t->is_contiguous();
}
bool plain_bytes(const at::Tensor* t, int device) {  // uint8 or one of the float8 types
  return t && t->is_cuda() && t->element_size() == 1 && t->get_device() == device && t->is_contiguous();
}
bool none_or_plain(PyObject* o, ScalarType dt, int device) { return o == Py_None || plain(tensor_of(o), dt, device); }
void* ptr_or_null(PyObject* o) { return o == Py_None ? nullptr : tensor_of(o)->data_ptr(); }

at::Tensor empty(std::initializer_list<int64_t> shape, ScalarType dt, int device) {
  return at::detail::empty_cuda(at::IntArrayRef(shape.begin(), shape.size()), dt, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt);
}
// Scratch of one call: from the caching allocator each time (about 0.5 us), so it is ordered with the stream it is used
// on and needs no pool of its own.  Its blocks are 512-byte aligned.
at::Tensor scratch(size_t bytes, int device) { return empty({(int64_t)(bytes < 256 ? 256 : bytes)}, ScalarType::Byte, device); }
size_t up256(size_t v) { return (v + 255) / 256 * 256; }

int current_device() { return (int)c10::cuda::current_device(); }
cachalot_stream_t current_stream(int device) {
  return reinterpret_cast<cachalot_stream_t>(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream());
}

// the exception a return code of the C ABI stands for (as _lib.check)
PyObject* raise(int rc) {
  PyObject* type = rc == CACHALOT_EUNSUPPORTED ? PyExc_NotImplementedError : rc == CACHALOT_ECUDA ? PyExc_RuntimeError : PyExc_ValueError;
  PyErr_SetString(type, lib.cachalot_last_error());
  return nullptr;
}

// Launches without the interpreter's lock, as ctypes makes them: a call that fills the launch queue (a launch per token, or
// calls far ahead of the GPU) waits in the driver, and other Python threads run meanwhile.
template <typename F>
int unlocked(F&& launch) {
  struct Unlock {
    PyThreadState* state = PyEval_SaveThread();
    ~Unlock() { PyEval_RestoreThread(state); }
  } u;
  return launch();
}
#define UNLOCKED(call) unlocked([&] { return call; })

// numeric arguments
struct Args {
  PyObject* const* a;
  bool bad = false;
  int i(int n) {
    const long v = PyLong_AsLong(a[n]);
    if (v == -1 && PyErr_Occurred()) PyErr_Clear(), bad = true;
    if (v != (int)v) bad = true;
    return (int)v;
  }
  double f(int n) {
    const double v = PyFloat_AsDouble(a[n]);
    if (v == -1.0 && PyErr_Occurred()) PyErr_Clear(), bad = true;
    return v;
  }
};

const cachalot_bank_desc* desc_of(PyObject* o) {  // the address of the bank's descriptor
  void* p = PyLong_AsVoidPtr(o);
  if (!p) PyErr_Clear();
  return static_cast<const cachalot_bank_desc*>(p);
}
bool plain_bank(const at::Tensor* slab, const cachalot_bank_desc* d, int device) {
  return d && plain(slab, ScalarType::Byte, device) && slab->dim() == 2 && slab->size(0) == d->n_slots && slab->size(1) == d->record_bytes;
}

#define PLAIN_OR_NONE(cond) \
  do {                      \
    if (!(cond)) Py_RETURN_NONE; \
  } while (0)

ScalarType out_type(int dt) { return dt == CACHALOT_F32 ? ScalarType::Float : ScalarType::BFloat16; }

// Weight scales of an FP8 matrix [n, k]: uint8 (E8M0, blocks of 32) or float32; the block size, 0 if they do not fit.
int fp8_block(const at::Tensor* s, int64_t n, int64_t k, int device, int* rule) {
  if (plain(s, ScalarType::Byte, device)) *rule = CACHALOT_SCALE_E8M0;
  else if (plain(s, ScalarType::Float, device)) *rule = CACHALOT_SCALE_F32;
  else return 0;
  if (s->dim() != 2 || s->size(1) <= 0) return 0;
  const int64_t block = *rule == CACHALOT_SCALE_E8M0 ? 32 : k / s->size(1);
  if ((block != 32 && block != 128) || k % block || s->size(0) != (n + block - 1) / block || s->size(1) != k / block) return 0;
  return (int)block;
}

// (x, weight, weight_scales, out dtype) -> y
PyObject* fp8_linear(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  PLAIN_OR_NONE(bound && n_args == 4);
  Args p{a};
  const int dev = current_device(), odt = (int)p.i(3);
  const at::Tensor *x = tensor_of(a[0]), *w = tensor_of(a[1]), *s = tensor_of(a[2]);
  PLAIN_OR_NONE(!p.bad && odt >= CACHALOT_BF16 && plain(x, ScalarType::BFloat16, dev) && plain_bytes(w, dev) && w->dim() == 2);
  PLAIN_OR_NONE((x->dim() == 1 || x->dim() == 2) && x->size(-1) == w->size(1));
  const int64_t n = w->size(0), k = w->size(1), rows = x->dim() == 2 ? x->size(0) : 1;
  int rule = 0;
  const int block = fp8_block(s, n, k, dev, &rule);
  PLAIN_OR_NONE(block && rows > 0 && rows < (1 << 30) && n > 0);
  const size_t codes_bytes = up256((size_t)rows * k);
  const at::Tensor ws = scratch(codes_bytes + (size_t)rows * (k / block) * 4, dev);
  at::Tensor y = x->dim() == 1 ? empty({n}, out_type(odt), dev) : empty({rows, n}, out_type(odt), dev);
  uint8_t* codes = static_cast<uint8_t*>(ws.data_ptr());
  const int rc = UNLOCKED(lib.cachalot_fp8_linear(x->data_ptr(), (int)rows, (int)k, block, rule, codes,
                                                  reinterpret_cast<float*>(codes + codes_bytes), static_cast<const uint8_t*>(w->data_ptr()),
                                                  s->data_ptr(), (int)n, y.data_ptr(), odt, current_stream(dev)));
  if (rc) return raise(rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// (x f32, weight bf16) -> y f32
PyObject* bf16_gemv_f32(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  PLAIN_OR_NONE(bound && n_args == 2);
  const int dev = current_device();
  const at::Tensor *x = tensor_of(a[0]), *w = tensor_of(a[1]);
  PLAIN_OR_NONE(plain(x, ScalarType::Float, dev) && plain(w, ScalarType::BFloat16, dev) && w->dim() == 2 && (x->dim() == 1 || x->dim() == 2));
  const int64_t n = w->size(0), k = w->size(1), rows = x->dim() == 2 ? x->size(0) : 1;
  PLAIN_OR_NONE(x->size(-1) == k && k % 64 == 0 && rows > 0 && n > 0);
  at::Tensor y = x->dim() == 1 ? empty({n}, ScalarType::Float, dev) : empty({rows, n}, ScalarType::Float, dev);
  const cachalot_stream_t st = current_stream(dev);
  for (int64_t r = 0; r < rows; r += 8) {
    const int rc = UNLOCKED(lib.cachalot_bf16_gemv_f32(static_cast<const float*>(x->data_ptr()) + r * k, (int)(rows - r < 8 ? rows - r : 8),
                                                       w->data_ptr(), (int)n, (int)k, static_cast<float*>(y.data_ptr()) + r * n, st));
    if (rc) return raise(rc);
  }
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

struct Shared {  // the shared expert's matrices
  const at::Tensor *w1, *s1, *w3, *s3, *w2, *s2;
  int64_t hidden, inter;
  int block, rule;
};
bool shared_from(PyObject* const* a, int64_t hidden, int dev, Shared* m) {  // w1, s1, w3 | None, s3 | None, w2, s2
  m->w1 = tensor_of(a[0]), m->s1 = tensor_of(a[1]), m->w2 = tensor_of(a[4]), m->s2 = tensor_of(a[5]);
  m->w3 = a[2] == Py_None ? nullptr : tensor_of(a[2]), m->s3 = a[3] == Py_None ? nullptr : tensor_of(a[3]);
  if (!plain_bytes(m->w1, dev) || !plain_bytes(m->w2, dev) || m->w1->dim() != 2 || m->w2->dim() != 2) return false;
  if (a[2] != Py_None && (!plain_bytes(m->w3, dev) || m->w3->dim() != 2)) return false;
  m->hidden = hidden, m->inter = m->w2->size(1);
  const int64_t rows1 = m->w3 ? m->inter : 2 * m->inter;
  if (m->w2->size(0) != hidden || m->w1->size(1) != hidden || m->w1->size(0) != rows1) return false;
  int r1 = 0, r3 = 0;
  m->block = fp8_block(m->s2, hidden, m->inter, dev, &m->rule);
  if (!m->block || fp8_block(m->s1, rows1, hidden, dev, &r1) != m->block || r1 != m->rule || hidden % m->block || m->inter % m->block) return false;
  if (!m->w3) return true;
  return m->w3->size(0) == m->inter && m->w3->size(1) == hidden && fp8_block(m->s3, m->inter, hidden, dev, &r3) == m->block && r3 == m->rule;
}
int run_shared(const void* x, int64_t rows, const Shared& m, double limit, const float* addend, void* out, int dev) {
  const size_t need = lib.cachalot_shared_expert_workspace_bytes((int)rows, (int)m.hidden, (int)m.inter, m.block);
  const at::Tensor ws = scratch(need, dev);
  return UNLOCKED(lib.cachalot_shared_expert(x, (int)rows, (int)m.hidden, (int)m.inter, static_cast<const uint8_t*>(m.w1->data_ptr()), m.s1->data_ptr(),
                                m.w3 ? static_cast<const uint8_t*>(m.w3->data_ptr()) : nullptr, m.w3 ? m.s3->data_ptr() : nullptr,
                                static_cast<const uint8_t*>(m.w2->data_ptr()), m.s2->data_ptr(), m.rule, m.block, (float)limit, addend,
                                ws.data_ptr(), (size_t)ws.numel(), out, current_stream(dev)));
}

// (x, w1, s1, w3 | None, s3 | None, w2, s2, limit) -> y bf16, in x's shape
PyObject* shared_expert(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  PLAIN_OR_NONE(bound && n_args == 8);
  Args p{a};
  const int dev = current_device();
  const at::Tensor* x = tensor_of(a[0]);
  const double limit = p.f(7);
  PLAIN_OR_NONE(!p.bad && plain(x, ScalarType::BFloat16, dev) && (x->dim() == 1 || x->dim() == 2));
  const int64_t rows = x->dim() == 2 ? x->size(0) : 1;
  Shared m;
  PLAIN_OR_NONE(rows > 0 && rows < (1 << 30) && shared_from(a + 1, x->size(-1), dev, &m));
  at::Tensor y = x->dim() == 1 ? empty({m.hidden}, ScalarType::BFloat16, dev) : empty({rows, m.hidden}, ScalarType::BFloat16, dev);
  const int rc = run_shared(x->data_ptr(), rows, m, limit, nullptr, y.data_ptr(), dev);
  if (rc) return raise(rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// (x [rows, H], slots [rows, k], gate weights [rows, k], slab, descriptor, limit, numerics, out dtype, status | None) -> out [rows, H]
PyObject* moe_forward(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  PLAIN_OR_NONE(bound && n_args == 9);
  Args p{a};
  const int dev = current_device(), num = (int)p.i(6), odt = (int)p.i(7);
  const double limit = p.f(5);
  const at::Tensor *x = tensor_of(a[0]), *slots = tensor_of(a[1]), *gw = tensor_of(a[2]), *slab = tensor_of(a[3]);
  const cachalot_bank_desc* d = desc_of(a[4]);
  PLAIN_OR_NONE(!p.bad && odt >= CACHALOT_BF16 && plain_bank(slab, d, dev) && none_or_plain(a[8], ScalarType::Int, dev));
  PLAIN_OR_NONE(plain(x, ScalarType::BFloat16, dev) && plain(slots, ScalarType::Int, dev) && plain(gw, ScalarType::Float, dev));
  PLAIN_OR_NONE(x->dim() == 2 && slots->dim() == 2 && gw->dim() == 2 && x->size(1) == d->hidden);
  const int64_t rows = x->size(0), k = slots->size(1);
  PLAIN_OR_NONE(rows > 0 && rows < (1 << 30) && slots->size(0) == rows && gw->size(0) == rows && gw->size(1) == k && k > 0 && k < 1024);
  at::Tensor out = empty({rows, d->hidden}, out_type(odt), dev);
  const at::Tensor ws = scratch(lib.cachalot_moe_decode_workspace_bytes(d, (int)rows, (int)k), dev);
  int* status = static_cast<int*>(ptr_or_null(a[8]));
  const int rc = UNLOCKED(lib.cachalot_moe_decode(slab->data_ptr(), d, x->data_ptr(), static_cast<const int32_t*>(slots->data_ptr()),
                                     static_cast<const float*>(gw->data_ptr()), (int)rows, (int)k, (float)limit, num, ws.data_ptr(),
                                     (size_t)ws.numel(), out.data_ptr(), odt, status, current_stream(dev)));
  if (rc) return raise(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

struct LayerCall {  // what a one-token layer takes besides x and the logits
  const at::Tensor *slab, *table;
  const cachalot_bank_desc* d;
  const float* bias;
  int layer, experts, topk, mode, norm, weights_bf16, numerics, odt;
  double temp, scale, limit;
  int* status;
};
int run_layer(const LayerCall& c, const void* x, const float* logits, void* out, int32_t* idx, float* w, int dev) {
  const at::Tensor ws = scratch(lib.cachalot_moe_layer_decode_workspace_bytes(c.d, c.topk), dev);
  return UNLOCKED(lib.cachalot_moe_layer_decode(c.slab->data_ptr(), c.d, x, logits, c.bias, static_cast<const int32_t*>(c.table->data_ptr()), c.layer,
                                   c.experts, c.topk, c.mode, (float)c.temp, (float)c.scale, c.norm, c.weights_bf16, (float)c.limit, c.numerics,
                                   ws.data_ptr(), (size_t)ws.numel(), out, c.odt, idx, w, c.status, current_stream(dev)));
}
bool table_fits(const at::Tensor* t, int layer, int64_t experts, int dev) {
  return plain(t, ScalarType::Int, dev) && t->dim() == 2 && t->size(1) == experts && layer >= 0 && layer < t->size(0);
}

// (x [H], logits [E], slab, descriptor, table, layer, topk, bias | None, mode, gate_temp, route_scale, norm, weights_bf16, limit, numerics,
//  out dtype, out | None, status | None, want_routing) -> out, or (out, indices, weights)
PyObject* layer_decode(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  PLAIN_OR_NONE(bound && n_args == 19);
  Args p{a};
  const int dev = current_device();
  const at::Tensor *x = tensor_of(a[0]), *logits = tensor_of(a[1]);
  LayerCall c;
  c.slab = tensor_of(a[2]), c.d = desc_of(a[3]), c.table = tensor_of(a[4]);
  c.layer = (int)p.i(5), c.topk = (int)p.i(6), c.mode = (int)p.i(8), c.temp = p.f(9), c.scale = p.f(10), c.norm = (int)p.i(11);
  c.weights_bf16 = (int)p.i(12), c.limit = p.f(13), c.numerics = (int)p.i(14), c.odt = (int)p.i(15);
  const bool want = p.i(18) != 0;
  PLAIN_OR_NONE(!p.bad && c.odt >= CACHALOT_BF16 && plain_bank(c.slab, c.d, dev));
  PLAIN_OR_NONE(plain(x, ScalarType::BFloat16, dev) && x->dim() == 1 && x->numel() == c.d->hidden);
  PLAIN_OR_NONE(plain(logits, ScalarType::Float, dev) && logits->dim() == 1);
  const int64_t e = logits->numel();
  PLAIN_OR_NONE(e <= 1024 && c.topk >= 1 && c.topk <= e && table_fits(c.table, c.layer, e, dev));
  PLAIN_OR_NONE(none_or_plain(a[7], ScalarType::Float, dev) && none_or_plain(a[17], ScalarType::Int, dev));
  PLAIN_OR_NONE(a[7] == Py_None || (tensor_of(a[7])->dim() == 1 && tensor_of(a[7])->numel() == e));
  PLAIN_OR_NONE(none_or_plain(a[16], out_type(c.odt), dev) && (a[16] == Py_None || tensor_of(a[16])->numel() == c.d->hidden));
  c.experts = (int)e, c.bias = static_cast<const float*>(ptr_or_null(a[7])), c.status = static_cast<int*>(ptr_or_null(a[17]));
  at::Tensor out = a[16] == Py_None ? empty({c.d->hidden}, out_type(c.odt), dev) : *tensor_of(a[16]);
  at::Tensor idx, w;
  if (want) idx = empty({c.topk}, ScalarType::Int, dev), w = empty({c.topk}, ScalarType::Float, dev);
  const int rc = run_layer(c, x->data_ptr(), static_cast<const float*>(logits->data_ptr()), out.data_ptr(),
                           want ? static_cast<int32_t*>(idx.data_ptr()) : nullptr, want ? static_cast<float*>(w.data_ptr()) : nullptr, dev);
  if (rc) return raise(rc);
  if (!want) return THPVariable_Wrap(std::move(out));
  return Py_BuildValue("(NNN)", THPVariable_Wrap(std::move(out)), THPVariable_Wrap(std::move(idx)), THPVariable_Wrap(std::move(w)));
  END_HANDLE_TH_ERRORS
}

// (x [T, H], expert_ids [T, k], weights [T, k], slab, descriptor, table, layer, experts, limit, mxfp4_act, status | None) -> out f32 [T, H]
PyObject* prefill_grouped(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  PLAIN_OR_NONE(bound && n_args == 11);
  Args p{a};
  const int dev = current_device(), layer = (int)p.i(6), mx = (int)p.i(9);
  const int64_t e = p.i(7);
  const double limit = p.f(8);
  const at::Tensor *x = tensor_of(a[0]), *ids = tensor_of(a[1]), *w = tensor_of(a[2]), *slab = tensor_of(a[3]), *table = tensor_of(a[5]);
  const cachalot_bank_desc* d = desc_of(a[4]);
  PLAIN_OR_NONE(!p.bad && plain_bank(slab, d, dev) && e > 0 && e <= 8192 && table_fits(table, layer, e, dev) && none_or_plain(a[10], ScalarType::Int, dev));
  PLAIN_OR_NONE(plain(x, ScalarType::BFloat16, dev) && plain(ids, ScalarType::Int, dev) && plain(w, ScalarType::Float, dev));
  PLAIN_OR_NONE(x->dim() == 2 && ids->dim() == 2 && w->dim() == 2 && x->size(1) == d->hidden);
  const int64_t t = ids->size(0), k = ids->size(1);
  PLAIN_OR_NONE(t > 0 && k > 0 && t * k < (1 << 30) && x->size(0) == t && w->size(0) == t && w->size(1) == k);
  const size_t perm = up256((size_t)t * k * 4), offs = up256((size_t)(e + 1) * 4);
  const size_t counts = up256(lib.cachalot_group_rows_scratch_ints((int)t, (int)k, (int)e) * 4);
  const size_t need = lib.cachalot_moe_prefill_experts_workspace_bytes(d, (int)t, (int)k, (int)e, mx);
  const at::Tensor ws = scratch(perm + offs + counts + need, dev);
  at::Tensor out = empty({t, d->hidden}, ScalarType::Float, dev);
  uint8_t* b = static_cast<uint8_t*>(ws.data_ptr());
  int32_t *pm = reinterpret_cast<int32_t*>(b), *of = reinterpret_cast<int32_t*>(b + perm), *ct = reinterpret_cast<int32_t*>(b + perm + offs);
  int* status = static_cast<int*>(ptr_or_null(a[10]));
  const cachalot_stream_t st = current_stream(dev);
  int rc = UNLOCKED(lib.cachalot_group_rows(static_cast<const int32_t*>(ids->data_ptr()), (int)t, (int)k, (int)e, pm, of, ct, status, st));
  if (!rc)
    rc = UNLOCKED(lib.cachalot_moe_prefill(slab->data_ptr(), d, x->data_ptr(), pm, of,
                              static_cast<const int32_t*>(table->data_ptr()) + (size_t)layer * e,
                              static_cast<const float*>(w->data_ptr()), (int)t, (int)k, (int)e, (float)limit, mx, b + perm + offs + counts,
                              (size_t)ws.numel() - perm - offs - counts, static_cast<float*>(out.data_ptr()), status, st));
  if (rc) return raise(rc);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// (x [H], gate_w [E, H], bias [E], slab, descriptor, table, layer, topk, gate_temp, route_scale, norm, limit, numerics, scores, status | None,
//  w1, s1, w3 | None, s3 | None, w2, s2) -> (out bf16 [H], indices, weights, scores | None)
PyObject* moe_block(PyObject*, PyObject* const* a, Py_ssize_t n_args) {
  HANDLE_TH_ERRORS
  PLAIN_OR_NONE(bound && n_args == 21);
  Args p{a};
  const int dev = current_device();
  const at::Tensor *x = tensor_of(a[0]), *gate = tensor_of(a[1]), *bias = tensor_of(a[2]);
  LayerCall c;
  c.slab = tensor_of(a[3]), c.d = desc_of(a[4]), c.table = tensor_of(a[5]);
  c.layer = (int)p.i(6), c.topk = (int)p.i(7), c.mode = CACHALOT_ROUTER_SQRT_SOFTPLUS, c.temp = p.f(8), c.scale = p.f(9), c.norm = (int)p.i(10);
  c.weights_bf16 = 0, c.limit = p.f(11), c.numerics = (int)p.i(12), c.odt = CACHALOT_F32;
  const bool want_scores = p.i(13) != 0;
  PLAIN_OR_NONE(!p.bad && plain_bank(c.slab, c.d, dev) && plain(x, ScalarType::BFloat16, dev) && x->dim() == 1 && x->numel() == c.d->hidden);
  const bool gate_bf16 = plain(gate, ScalarType::BFloat16, dev);
  PLAIN_OR_NONE((gate_bf16 || plain(gate, ScalarType::Float, dev)) && gate->dim() == 2 && gate->size(1) == c.d->hidden);
  const int64_t e = gate->size(0), h = c.d->hidden;
  PLAIN_OR_NONE(plain(bias, ScalarType::Float, dev) && bias->dim() == 1 && bias->numel() == e && none_or_plain(a[14], ScalarType::Int, dev));
  PLAIN_OR_NONE(e <= 1024 && c.topk >= 1 && c.topk <= e && table_fits(c.table, c.layer, e, dev));
  Shared m;
  PLAIN_OR_NONE(shared_from(a + 15, h, dev, &m));
  c.experts = (int)e, c.bias = static_cast<const float*>(bias->data_ptr()), c.status = static_cast<int*>(ptr_or_null(a[14]));
  const size_t lb = up256((size_t)e * 4), rb = up256((size_t)h * 4);
  const at::Tensor tmp = scratch(lb + rb + 512, dev);  // logits, routed sum, slots (unused)
  uint8_t* t = static_cast<uint8_t*>(tmp.data_ptr());
  float *logits = reinterpret_cast<float*>(t), *routed = reinterpret_cast<float*>(t + lb);
  at::Tensor out = empty({h}, ScalarType::BFloat16, dev), idx = empty({c.topk}, ScalarType::Int, dev), w = empty({c.topk}, ScalarType::Float, dev);
  at::Tensor sc;
  if (want_scores) sc = empty({e}, ScalarType::Float, dev);
  int32_t* ip = static_cast<int32_t*>(idx.data_ptr());
  float* wp = static_cast<float*>(w.data_ptr());
  const cachalot_stream_t st = current_stream(dev);
  int rc = UNLOCKED(lib.cachalot_router_logits(x->data_ptr(), gate->data_ptr(), gate_bf16 ? CACHALOT_BF16 : CACHALOT_F32, 1, (int)e, (int)h,
                                               logits, st));
  if (!rc && want_scores)
    rc = UNLOCKED(lib.cachalot_route_topk(logits, c.bias, nullptr, 0, 1, (int)e, c.topk, c.mode, (float)c.temp, (float)c.scale, c.norm, 0,
                                          ip, wp, nullptr, static_cast<float*>(sc.data_ptr()), st));
  if (!rc) rc = run_layer(c, x->data_ptr(), logits, routed, ip, wp, dev);
  if (!rc) rc = run_shared(x->data_ptr(), 1, m, c.limit, routed, out.data_ptr(), dev);
  if (rc) return raise(rc);
  PyObject* so = want_scores ? THPVariable_Wrap(std::move(sc)) : Py_NewRef(Py_None);
  return Py_BuildValue("(NNNN)", THPVariable_Wrap(std::move(out)), THPVariable_Wrap(std::move(idx)), THPVariable_Wrap(std::move(w)), so);
  END_HANDLE_TH_ERRORS
}

#define FAST(name) {#name, (PyCFunction)(void (*)(void))name, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {FAST(entries), FAST(bind), FAST(fp8_linear), FAST(bf16_gemv_f32), FAST(shared_expert), FAST(moe_forward), FAST(layer_decode),
                         FAST(prefill_grouped), FAST(moe_block), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native call path of the operators (see host.cpp).", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
