// The entry points that a decode step calls, for Python callers: descriptors and tensors are read and the C ABI is called without
// going through ctypes.  Semantics are those of the ctypes structures (qw38_b200/_lib.py): integers are taken modulo the field's
// width, tensors by data_ptr() and numel() at every call, nothing is kept between calls.
//
// Bound: host time.  A decode call of one token spends 4.2 us in the C entry and the driver.  Building and comparing structures
// in Python took 3.0 us more, this 1.4 (5120 x 5120 with a residual: 8.9 us per call in a loop, now 6.7; a pack 2.0 and 0.9).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <cstdint>

#include "../../include/q4k_b200.h"

namespace {

struct Names {
  PyObject *codes, *scales, *sums, *n, *k, *m, *padded_k, *layout, *quantizer, *codes_bytes, *scales_bytes, *weight, *input, *output, *residual,
      *epilogue, *activation_policy, *data_ptr, *numel, *dim, *size, *cuda_stream, *element_size;
} names;

struct Entries {
  decltype(&q4k_decode_mmv) decode_mmv;
  decltype(&q4k_decode_mmv_ranges) decode_mmv_ranges;
  decltype(&q4k_pack_q8_bf16) pack_q8_bf16;
  decltype(&q4k_pack_q8_f32) pack_q8_f32;
  decltype(&q4k_q8_project) q8_project;
  decltype(&q4k_q8_mlp) q8_mlp;
  decltype(&q4k_prefill_project) prefill_project;
  decltype(&q4k_prefill_paired_swiglu) prefill_paired_swiglu;
  decltype(&q4k_decode_mmv_paired) decode_mmv_paired;
} entries;
PyObject *get_device, *get_stream, *zero;

// A reference that is dropped at the end of its scope.
struct Ref {
  PyObject* p;
  explicit Ref(PyObject* o) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(Ref const&) = delete;
  Ref& operator=(Ref const&) = delete;
  explicit operator bool() const { return p != nullptr; }
};

// Python integer or anything with __index__ (shapes read through numpy), modulo 2^64 as ctypes takes it.  False: an exception is set.
bool as_u64(PyObject* o, uint64_t* to) {
  if (!o) return false;
  *to = PyLong_AsUnsignedLongLongMask(o);
  return !(*to == ~0ull && PyErr_Occurred());
}
bool attr(PyObject* o, PyObject* name, uint64_t* to) {
  Ref const v(PyObject_GetAttr(o, name));
  return as_u64(v.p, to);
}
bool call(PyObject* o, PyObject* name, uint64_t* to) {
  Ref const v(PyObject_CallMethodNoArgs(o, name));
  return as_u64(v.p, to);
}
template <class T> bool pointer(PyObject* tensor, T** to) {  // null for None
  uint64_t v = 0;
  if (tensor != Py_None && !call(tensor, names.data_ptr, &v)) return false;
  *to = reinterpret_cast<T*>(v);
  return true;
}
template <class T> bool tensor(PyObject* o, T** p, uint64_t* len) { return pointer(o, p) && call(o, names.numel, len); }
// A tensor or None.
template <class T> bool optional(PyObject* o, T** p, uint64_t* len) {
  *p = nullptr;
  *len = 0;
  return o == Py_None || tensor(o, p, len);
}

bool read_weight(PyObject* o, q4k_weight* w) {
  Ref const codes(PyObject_GetAttr(o, names.codes)), scales(PyObject_GetAttr(o, names.scales)), cb(PyObject_GetAttr(o, names.codes_bytes)),
      sb(PyObject_GetAttr(o, names.scales_bytes));
  uint64_t layout = 0, quantizer = 0, n = 0, k = 0;
  if (!codes || !scales || !cb || !sb || !attr(o, names.layout, &layout) || !attr(o, names.quantizer, &quantizer) || !attr(o, names.n, &n) ||
      !attr(o, names.k, &k) || !pointer(codes.p, &w->codes) || !pointer(scales.p, &w->scales))
    return false;
  w->layout = uint16_t(layout);
  w->quantizer = uint16_t(quantizer);
  w->n = uint32_t(n);
  w->k = uint32_t(k);
  w->padded_n = uint32_t((n + 7) / 8 * 8);
  w->padded_k = uint32_t((k + 255) / 256 * 256);
  return (cb.p == Py_None ? call(codes.p, names.numel, &w->codes_bytes) : as_u64(cb.p, &w->codes_bytes)) &&
         (sb.p == Py_None ? call(scales.p, names.numel, &w->scales_bytes) : as_u64(sb.p, &w->scales_bytes));
}

bool read_q8(PyObject* o, q4k_q8_input* x) {
  Ref const codes(PyObject_GetAttr(o, names.codes)), scales(PyObject_GetAttr(o, names.scales)), sums(PyObject_GetAttr(o, names.sums));
  uint64_t m = 0, k = 0, pk = 0;
  if (!codes || !scales || !sums || !tensor(codes.p, &x->codes, &x->codes_len) || !tensor(scales.p, &x->scales, &x->scales_len) ||
      !tensor(sums.p, &x->sums, &x->sums_len) || !attr(o, names.m, &m) || !attr(o, names.k, &k) || !attr(o, names.padded_k, &pk))
    return false;
  x->m = uint32_t(m);
  x->k = uint32_t(k);
  x->padded_k = uint32_t(pk);
  return true;
}

bool read_desc(PyObject* o, q4k_decode_desc* d) {
  Ref const weight(PyObject_GetAttr(o, names.weight)), input(PyObject_GetAttr(o, names.input)), output(PyObject_GetAttr(o, names.output)),
      residual(PyObject_GetAttr(o, names.residual));
  uint64_t dim = 0, rows = 1, epilogue = 0, policy = 0;
  if (!weight || !input || !output || !residual || !read_weight(weight.p, &d->weight) || !tensor(input.p, &d->input, &d->input_len) ||
      !optional(output.p, &d->output, &d->output_len) || !optional(residual.p, &d->residual, &d->residual_len) ||
      !call(input.p, names.dim, &dim) || !attr(o, names.epilogue, &epilogue) || !attr(o, names.activation_policy, &policy))
    return false;
  if (dim == 2) {
    Ref const v(PyObject_CallMethodOneArg(input.p, names.size, zero));
    if (!as_u64(v.p, &rows)) return false;
  }
  d->m = uint32_t(rows);
  d->epilogue = uint8_t(epilogue);
  d->activation_policy = uint8_t(policy);
  return true;
}

// The given stream's handle, or the current one's.
bool read_stream(PyObject* o, void** to) {
  uint64_t v = 0;
  if (o == Py_None) {
    Ref const device(PyObject_CallNoArgs(get_device));
    if (!device) return false;
    Ref const raw(PyObject_CallOneArg(get_stream, device.p));
    if (!as_u64(raw.p, &v)) return false;
  } else if (!attr(o, names.cuda_stream, &v)) {
    return false;
  }
  *to = reinterpret_cast<void*>(v);
  return true;
}

// The entry without the interpreter lock: a launch may wait for room in the driver's queue.
template <class F> int unlocked(F const& entry) {
  int st = 0;
  Py_BEGIN_ALLOW_THREADS
  st = entry();
  Py_END_ALLOW_THREADS
  return st;
}

bool arguments(Py_ssize_t got, Py_ssize_t want, const char* name) {
  if (got == want) return true;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments, not %zd", name, want, got);
  return false;
}

// (desc, workspace, failure, stream) -> status
PyObject* one_desc(PyObject* const* a, Py_ssize_t n, const char* name, decltype(&q4k_decode_mmv) entry) {
  q4k_decode_desc d{};
  void *workspace = nullptr, *stream = nullptr;
  uint64_t bytes = 0;
  int* failure = nullptr;
  if (!arguments(n, 4, name) || !read_desc(a[0], &d) || !tensor(a[1], &workspace, &bytes) || !pointer(a[2], &failure) ||
      !read_stream(a[3], &stream))
    return nullptr;
  return PyLong_FromLong(unlocked([&] { return entry(&d, workspace, bytes, failure, stream); }));
}
PyObject* decode_mmv(PyObject*, PyObject* const* a, Py_ssize_t n) { return one_desc(a, n, "decode_mmv", entries.decode_mmv); }
PyObject* prefill_project(PyObject*, PyObject* const* a, Py_ssize_t n) { return one_desc(a, n, "prefill_project", entries.prefill_project); }

// (first desc, second desc, workspace, failure, stream) -> status
PyObject* decode_mmv_paired(PyObject*, PyObject* const* a, Py_ssize_t n) {
  q4k_decode_desc d[2] = {};
  void *workspace = nullptr, *stream = nullptr;
  uint64_t bytes = 0;
  int* failure = nullptr;
  if (!arguments(n, 5, "decode_mmv_paired") || !read_desc(a[0], &d[0]) || !read_desc(a[1], &d[1]) || !tensor(a[2], &workspace, &bytes) ||
      !pointer(a[3], &failure) || !read_stream(a[4], &stream))
    return nullptr;
  if (!entries.decode_mmv_paired) return PyErr_Format(PyExc_RuntimeError, "decode_mmv_paired is not bound");
  return PyLong_FromLong(unlocked([&] { return entries.decode_mmv_paired(&d[0], &d[1], workspace, bytes, failure, stream); }));
}

// (gate, up, normalized, swiglu, tokens, workspace, failure, stream) -> status
PyObject* prefill_paired_swiglu(PyObject*, PyObject* const* a, Py_ssize_t n) {
  q4k_weight w[2] = {};
  uint16_t *normalized = nullptr, *swiglu = nullptr;
  void *workspace = nullptr, *stream = nullptr;
  uint64_t m = 0, bytes = 0;
  int* failure = nullptr;
  if (!arguments(n, 8, "prefill_paired_swiglu") || !read_weight(a[0], &w[0]) || !read_weight(a[1], &w[1]) || !pointer(a[2], &normalized) ||
      !pointer(a[3], &swiglu) || !as_u64(a[4], &m) || !tensor(a[5], &workspace, &bytes) || !pointer(a[6], &failure) || !read_stream(a[7], &stream))
    return nullptr;
  return PyLong_FromLong(
      unlocked([&] { return entries.prefill_paired_swiglu(&w[0], &w[1], normalized, swiglu, uint32_t(m), workspace, bytes, failure, stream); }));
}

// (sequence of descs, workspace, failure, stream) -> status
PyObject* decode_mmv_ranges(PyObject*, PyObject* const* a, Py_ssize_t n) {
  q4k_decode_desc d[3] = {};
  void *workspace = nullptr, *stream = nullptr;
  uint64_t bytes = 0;
  int* failure = nullptr;
  if (!arguments(n, 4, "decode_mmv_ranges")) return nullptr;
  // A copy that holds its items: reading a descriptor runs Python code, during which a caller's list may change.
  Ref const list(PySequence_Tuple(a[0]));
  if (!list) return nullptr;
  Py_ssize_t const count = PyTuple_GET_SIZE(list.p);
  for (Py_ssize_t i = 0; i < count && i < 3; ++i)  // the entry refuses any other count before it looks at them
    if (!read_desc(PyTuple_GET_ITEM(list.p, i), &d[i])) return nullptr;
  if (!tensor(a[1], &workspace, &bytes) || !pointer(a[2], &failure) || !read_stream(a[3], &stream)) return nullptr;
  return PyLong_FromLong(unlocked([&] { return entries.decode_mmv_ranges(d, uint32_t(count), workspace, bytes, failure, stream); }));
}

// (rows, is fp32, Q8Input, failure, stream) -> status
PyObject* pack_q8(PyObject*, PyObject* const* a, Py_ssize_t n) {
  q4k_q8_input x{};
  void *rows = nullptr, *stream = nullptr;
  uint64_t len = 0;
  int* failure = nullptr;
  if (!arguments(n, 5, "pack_q8") || !tensor(a[0], &rows, &len) || !read_q8(a[2], &x) || !pointer(a[3], &failure) || !read_stream(a[4], &stream))
    return nullptr;
  bool const fp32 = a[1] == Py_True;
  return PyLong_FromLong(unlocked([&] {
    return fp32 ? entries.pack_q8_f32(static_cast<const float*>(rows), len, x, failure, stream)
                : entries.pack_q8_bf16(static_cast<const uint16_t*>(rows), len, x, failure, stream);
  }));
}

// (weight, Q8Input, out, residual or None, stream) -> status
PyObject* q8_project(PyObject*, PyObject* const* a, Py_ssize_t n) {
  q4k_weight w{};
  q4k_q8_input x{};
  float *out = nullptr, *residual = nullptr;
  void* stream = nullptr;
  uint64_t out_len = 0, residual_len = 0;
  if (!arguments(n, 5, "q8_project") || !read_weight(a[0], &w) || !read_q8(a[1], &x) || !tensor(a[2], &out, &out_len) ||
      !optional(a[3], &residual, &residual_len) || !read_stream(a[4], &stream))
    return nullptr;
  return PyLong_FromLong(unlocked([&] { return entries.q8_project(&w, x, out, out_len, residual, residual_len, stream); }));
}

// (gate, up, down, residual, gamma, eps, out, m, workspace, pending failure or None, stream) -> (status, submitted)
PyObject* q8_mlp(PyObject*, PyObject* const* a, Py_ssize_t n) {
  q4k_weight w[3] = {};
  float *residual = nullptr, *out = nullptr;
  uint16_t* gamma = nullptr;
  int *pending = nullptr, submitted = 0;
  void *workspace = nullptr, *stream = nullptr;
  uint64_t m = 0, count = 0, element = 0, ignored = 0;
  if (!arguments(n, 11, "q8_mlp")) return nullptr;
  for (int i = 0; i < 3; ++i)
    if (!read_weight(a[i], &w[i])) return nullptr;
  double const eps = PyFloat_AsDouble(a[5]);
  if (eps == -1.0 && PyErr_Occurred()) return nullptr;
  if (!pointer(a[3], &residual) || !pointer(a[4], &gamma) || !pointer(a[6], &out) || !as_u64(a[7], &m) || !tensor(a[8], &workspace, &count) ||
      !call(a[8], names.element_size, &element) || !optional(a[9], &pending, &ignored) || !read_stream(a[10], &stream))
    return nullptr;
  int const st = unlocked([&] {
    return entries.q8_mlp(&w[0], &w[1], &w[2], residual, gamma, float(eps), out, uint32_t(m), workspace, count * element, stream, &submitted, pending);
  });
  return Py_BuildValue("ii", st, submitted);
}

// (addresses of the entries in the order above, torch's device and raw-stream lookups); without the last entry that one stays
// as it is
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 10 && !arguments(n, 11, "bind")) return nullptr;
  uint64_t p[9];
  p[8] = reinterpret_cast<uint64_t>(entries.decode_mmv_paired);
  for (int i = 0; i < n - 2; ++i)
    if (!as_u64(a[i], &p[i])) return nullptr;
  entries = {reinterpret_cast<decltype(entries.decode_mmv)>(p[0]),   reinterpret_cast<decltype(entries.decode_mmv_ranges)>(p[1]),
             reinterpret_cast<decltype(entries.pack_q8_bf16)>(p[2]), reinterpret_cast<decltype(entries.pack_q8_f32)>(p[3]),
             reinterpret_cast<decltype(entries.q8_project)>(p[4]),   reinterpret_cast<decltype(entries.q8_mlp)>(p[5]),
             reinterpret_cast<decltype(entries.prefill_project)>(p[6]),
             reinterpret_cast<decltype(entries.prefill_paired_swiglu)>(p[7]),
             reinterpret_cast<decltype(entries.decode_mmv_paired)>(p[8])};
  Py_INCREF(a[n - 2]);
  Py_INCREF(a[n - 1]);
  Py_XSETREF(get_device, a[n - 2]);
  Py_XSETREF(get_stream, a[n - 1]);
  Py_RETURN_NONE;
}

PyCFunction fast(PyObject* (*f)(PyObject*, PyObject* const*, Py_ssize_t)) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)); }
PyMethodDef methods[] = {{"bind", fast(bind), METH_FASTCALL, nullptr},
                         {"decode_mmv", fast(decode_mmv), METH_FASTCALL, nullptr},
                         {"decode_mmv_paired", fast(decode_mmv_paired), METH_FASTCALL, nullptr},
                         {"decode_mmv_ranges", fast(decode_mmv_ranges), METH_FASTCALL, nullptr},
                         {"pack_q8", fast(pack_q8), METH_FASTCALL, nullptr},
                         {"q8_project", fast(q8_project), METH_FASTCALL, nullptr},
                         {"q8_mlp", fast(q8_mlp), METH_FASTCALL, nullptr},
                         {"prefill_project", fast(prefill_project), METH_FASTCALL, nullptr},
                         {"prefill_paired_swiglu", fast(prefill_paired_swiglu), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_q4k_entries", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__q4k_entries() {
  struct { PyObject** to; const char* text; } const all[] = {
      {&names.codes, "codes"}, {&names.scales, "scales"}, {&names.sums, "sums"}, {&names.n, "n"}, {&names.k, "k"}, {&names.m, "m"},
      {&names.padded_k, "padded_k"}, {&names.layout, "layout"}, {&names.quantizer, "quantizer"}, {&names.codes_bytes, "codes_bytes"},
      {&names.scales_bytes, "scales_bytes"}, {&names.weight, "weight"}, {&names.input, "input"}, {&names.output, "output"},
      {&names.residual, "residual"}, {&names.epilogue, "epilogue"}, {&names.activation_policy, "activation_policy"},
      {&names.data_ptr, "data_ptr"}, {&names.numel, "numel"}, {&names.dim, "dim"}, {&names.size, "size"}, {&names.cuda_stream, "cuda_stream"},
      {&names.element_size, "element_size"}};
  for (auto const& e : all)
    if (!(*e.to = PyUnicode_InternFromString(e.text))) return nullptr;
  if (!(zero = PyLong_FromLong(0))) return nullptr;
  PyObject* const m = PyModule_Create(&module);
  // What it was built against, for the loader to compare with its own structures.
  PyObject* const sizes = m ? Py_BuildValue("(nnn)", Py_ssize_t(sizeof(q4k_weight)), Py_ssize_t(sizeof(q4k_q8_input)), Py_ssize_t(sizeof(q4k_decode_desc))) : nullptr;
  if (!sizes || PyModule_AddObject(m, "struct_sizes", sizes) < 0) {  // (takes the reference when it succeeds)
    Py_XDECREF(sizes);
    Py_XDECREF(m);
    return nullptr;
  }
  return m;
}
