// CPython entry of the launchers: `launch(name, dtype, *args)` and the fused chains' calls without ctypes.
//
// What bounds a small call is the host: a launch through ctypes cost 6.0 us of Python (symbol name built and looked up,
// every argument boxed and converted), three times the 2 us that the CUDA runtime needs to enqueue a kernel; through the
// typed stubs below it costs 0.4 us.  One stub per launcher is generated from its prototype in mp_kernels.h, so the
// arguments are converted to exactly the C types that the launcher declares and passed by a plain C call.
//
// The usual argument types are converted here (torch tensors, ints, floats, None, ctypes arrays and pointers, a Stream);
// a call with anything else goes to the ctypes path given to `setup`, which accepts or rejects it as before.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <vector>

#include "../../include/mp_jit.h"
#include "../../include/mp_kernels.h"

namespace {

// Objects handed over once by `setup` (borrowed for the life of the process).
PyObject* g_dtypes[3] = {nullptr, nullptr, nullptr};   // torch.float16 / float32 / float64
PyTypeObject* g_tensor = nullptr;                      // torch.Tensor
PyObject* g_data_ptr = nullptr;                        // torch.Tensor.data_ptr, called as a function
PyTypeObject* g_array = nullptr;                       // ctypes.Array
PyTypeObject* g_void_p = nullptr;                      // ctypes.c_void_p
PyTypeObject* g_context = nullptr;                     // StreamContext
PyTypeObject* g_stream = nullptr;                      // Stream
PyObject* g_fallback = nullptr;                        // the ctypes path of launch()
PyObject* g_ctx_name = nullptr;                        // "ctx"
PyObject* g_table = nullptr;                           // name -> index into kLaunchers

// ------------------------------ argument conversion: false = not a type handled here ------------------------------
bool from_buffer(PyObject* o, void* dst, size_t n) {
  Py_buffer b;
  if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) { PyErr_Clear(); return false; }
  const bool ok = static_cast<size_t>(b.len) >= n;
  if (ok) memcpy(dst, b.buf, n);
  PyBuffer_Release(&b);
  return ok;
}

bool to_pointer(PyObject* o, void** out) {
  if (o == Py_None) { *out = nullptr; return true; }
  if (Py_TYPE(o) == g_tensor || PyType_IsSubtype(Py_TYPE(o), g_tensor)) {
    PyObject* v = PyObject_CallOneArg(g_data_ptr, o);
    if (v == nullptr) { PyErr_Clear(); return false; }
    *out = PyLong_AsVoidPtr(v);
    Py_DECREF(v);
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
  }
  if (PyLong_CheckExact(o)) {
    *out = PyLong_AsVoidPtr(o);
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
  }
  if (Py_TYPE(o) == g_void_p) return from_buffer(o, out, sizeof(void*));   // the pointer it holds
  if (PyType_IsSubtype(Py_TYPE(o), g_array)) {                             // the address of its elements
    Py_buffer b;
    if (PyObject_GetBuffer(o, &b, PyBUF_SIMPLE) != 0) { PyErr_Clear(); return false; }
    *out = b.buf;
    PyBuffer_Release(&b);   // the caller's argument keeps the elements alive
    return true;
  }
  return false;
}

template <typename P> struct Convert;
template <typename E> struct Convert<E*> {
  static bool get(PyObject* o, E** out) {
    void* p;
    if (!to_pointer(o, &p)) return false;
    *out = static_cast<E*>(p);
    return true;
  }
};
template <> struct Convert<double> {
  static bool get(PyObject* o, double* out) {
    if (PyFloat_CheckExact(o)) { *out = PyFloat_AS_DOUBLE(o); return true; }
    if (!PyLong_CheckExact(o)) return false;
    *out = PyLong_AsDouble(o);
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
  }
};
template <> struct Convert<len_t> {
  static bool get(PyObject* o, len_t* out) {
    if (!PyLong_Check(o)) return false;
    *out = PyLong_AsUnsignedLongMask(o);
    if (PyErr_Occurred()) { PyErr_Clear(); return false; }
    return true;
  }
};
template <> struct Convert<StreamContext> {
  static bool get(PyObject* o, StreamContext* out) {
    if (Py_TYPE(o) == g_context) return from_buffer(o, out, sizeof(*out));
    if (Py_TYPE(o) != g_stream && !PyType_IsSubtype(Py_TYPE(o), g_stream)) return false;
    PyObject* c = PyObject_GetAttr(o, g_ctx_name);
    if (c == nullptr) { PyErr_Clear(); return false; }
    const bool ok = from_buffer(c, out, sizeof(*out));
    Py_DECREF(c);
    return ok;
  }
};

// ------------------------------ one stub per launcher ------------------------------
typedef bool (*StubFn)(PyObject* const* args, Py_ssize_t nargs);

template <typename... A> struct Args;
template <> struct Args<> {
  template <typename F, typename... Done>
  static bool call(F f, PyObject* const*, Done... done) {
    Py_BEGIN_ALLOW_THREADS   // as ctypes does: a launch may wait for room in the stream's queue
    f(done...);
    Py_END_ALLOW_THREADS
    return true;
  }
};
template <typename H, typename... T> struct Args<H, T...> {
  template <typename F, typename... Done>
  static bool call(F f, PyObject* const* args, Done... done) {
    H v;
    return Convert<H>::get(*args, &v) && Args<T...>::call(f, args + 1, done..., v);
  }
};
template <auto F> struct Stub;
template <typename... A, void (*F)(A...)> struct Stub<F> {
  static bool run(PyObject* const* args, Py_ssize_t nargs) { return nargs == sizeof...(A) && Args<A...>::call(F, args); }
};

struct Launcher { const char* name; StubFn fn[3]; };
#define MP_ENTRY(n) {#n, {Stub<&launch_##n##_r16>::run, Stub<&launch_##n##_r32>::run, Stub<&launch_##n##_r64>::run}}
const Launcher kLaunchers[] = {
    MP_ENTRY(reduce_ij_i), MP_ENTRY(reduce_ij_j), MP_ENTRY(broadcast_i_ij), MP_ENTRY(broadcast_j_ij), MP_ENTRY(dilate_reverse),
    MP_ENTRY(subtraction), MP_ENTRY(relu_reverse), MP_ENTRY(dilate), MP_ENTRY(translate), MP_ENTRY(permutate_ij_ji), MP_ENTRY(negate),
    MP_ENTRY(hadamard_reverse), MP_ENTRY(inner_product_ij_jk_ik), MP_ENTRY(hadamard), MP_ENTRY(fill), MP_ENTRY(relu), MP_ENTRY(addition),
    MP_ENTRY(copy), MP_ENTRY(sequence), MP_ENTRY(stepwise), MP_ENTRY(selu), MP_ENTRY(selu_reverse), MP_ENTRY(softmax_ij_j),
    MP_ENTRY(softmax_ij_j_reverse), MP_ENTRY(rmsnorm_ij_j), MP_ENTRY(rmsnorm_ij_j_reverse), MP_ENTRY(sgd), MP_ENTRY(adam),
    MP_ENTRY(inner_product_ij_kj_ik), MP_ENTRY(inner_product_ji_jk_ik), MP_ENTRY(linear_ij_jk_ik), MP_ENTRY(linear_ij_jk_ik_ik),
    MP_ENTRY(ssd_scan), MP_ENTRY(ssd_scan_reverse), MP_ENTRY(ssd_scan_raw), MP_ENTRY(ssd_scan_reverse_raw), MP_ENTRY(embedding),
    MP_ENTRY(embedding_reverse), MP_ENTRY(causal_conv1d_silu), MP_ENTRY(causal_conv1d_silu_reverse), MP_ENTRY(causal_conv1d_silu_segments),
    MP_ENTRY(causal_conv1d_silu_segments_reverse), MP_ENTRY(causal_conv1d_silu_segments_reverse_skip), MP_ENTRY(softplus_bias),
    MP_ENTRY(softplus_bias_reverse), MP_ENTRY(ssd_gate), MP_ENTRY(ssd_gate_reverse), MP_ENTRY(ssd_gate_rmsnorm),
    MP_ENTRY(ssd_gate_rmsnorm_reverse), MP_ENTRY(head_scale_accumulate), MP_ENTRY(cross_entropy), MP_ENTRY(neg_exp), MP_ENTRY(mse_loss_i_i),
    MP_ENTRY(bce_loss_i_i), MP_ENTRY(momentum), MP_ENTRY(permutate), MP_ENTRY(inner_product_bij_bjk_bik), MP_ENTRY(inner_product_bij_bkj_bik),
    MP_ENTRY(inner_product_bji_bjk_bik),
};

PyObject* py_launch(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  if (nargs >= 3 && kwnames == nullptr && PyUnicode_CheckExact(args[0])) {
    PyObject* idx = PyDict_GetItemWithError(g_table, args[0]);
    if (idx != nullptr) {
      for (int d = 0; d < 3; ++d)
        if (args[1] == g_dtypes[d]) {
          if (kLaunchers[PyLong_AsLong(idx)].fn[d](args + 2, nargs - 2)) Py_RETURN_NONE;
          break;
        }
    } else if (PyErr_Occurred()) {
      return nullptr;
    }
  }
  return PyObject_Vectorcall(g_fallback, args, nargs, kwnames);
}

// An operand of a chain: something with a `data_ptr` method (an AttributeError is raised for anything else), or None where there may be
// no tensor.  The kernels write through these pointers, so nothing else stands for an address here.
bool chain_pointer(PyObject* o, bool optional, void** out) {
  if (o == Py_None && optional) { *out = nullptr; return true; }
  const bool tensor = Py_TYPE(o) == g_tensor || PyType_IsSubtype(Py_TYPE(o), g_tensor);
  PyObject* v = tensor ? PyObject_CallOneArg(g_data_ptr, o) : PyObject_CallMethod(o, "data_ptr", nullptr);
  if (v == nullptr) return false;
  *out = PyLong_AsVoidPtr(v);
  Py_DECREF(v);
  return PyErr_Occurred() == nullptr;
}

bool chain_pointers(PyObject* seq, bool optional, std::vector<void*>& out) {
  PyObject* fast = PySequence_Fast(seq, "a list of tensors is expected");
  if (fast == nullptr) return false;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
  out.resize(static_cast<size_t>(n));
  bool ok = true;
  for (Py_ssize_t i = 0; ok && i < n; ++i) ok = chain_pointer(PySequence_Fast_GET_ITEM(fast, i), optional, &out[static_cast<size_t>(i)]);
  Py_DECREF(fast);
  return ok;
}

// The scalar arguments: handle of the compiled chain, element count, stream context.
bool chain_scalars(PyObject* handle, PyObject* count, PyObject* stream, void** h, len_t* n, StreamContext* ctx) {
  if (handle == Py_None) { PyErr_SetString(PyExc_ValueError, "the chain is closed"); return false; }
  if (to_pointer(handle, h) && Convert<len_t>::get(count, n) && Convert<StreamContext>::get(stream, ctx)) return true;
  PyErr_SetString(PyExc_TypeError, "(handle, ..., element count, StreamContext) expected");
  return false;
}

// chain_forward(handle, leaves, out, n, stream)
PyObject* py_chain_forward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  void *handle, *out;
  std::vector<void*> leaves;
  len_t n;
  StreamContext ctx;
  if (nargs != 5) { PyErr_SetString(PyExc_TypeError, "chain_forward: 5 arguments"); return nullptr; }
  if (!chain_scalars(args[0], args[3], args[4], &handle, &n, &ctx) || !chain_pointers(args[1], false, leaves) || !chain_pointer(args[2], false, &out))
    return nullptr;
  Py_BEGIN_ALLOW_THREADS
  mpJitForward(handle, leaves.data(), out, n, ctx);
  Py_END_ALLOW_THREADS
  Py_RETURN_NONE;
}

// chain_reverse(handle, leaves, g_out, g_leaves, alpha, n, stream)
PyObject* py_chain_reverse(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  void *handle, *gout;
  std::vector<void*> leaves, grads;
  double alpha;
  len_t n;
  StreamContext ctx;
  if (nargs != 7) { PyErr_SetString(PyExc_TypeError, "chain_reverse: 7 arguments"); return nullptr; }
  if (!chain_scalars(args[0], args[5], args[6], &handle, &n, &ctx) || !chain_pointers(args[1], true, leaves) || !chain_pointer(args[2], true, &gout) ||
      !chain_pointers(args[3], true, grads))
    return nullptr;
  if (!Convert<double>::get(args[4], &alpha)) { PyErr_SetString(PyExc_TypeError, "chain_reverse: alpha is a float"); return nullptr; }
  Py_BEGIN_ALLOW_THREADS
  mpJitReverse(handle, leaves.data(), gout, grads.data(), alpha, n, ctx);
  Py_END_ALLOW_THREADS
  Py_RETURN_NONE;
}

// setup(dtypes, Tensor, ctypes.Array, ctypes.c_void_p, StreamContext, Stream, fallback)
PyObject* py_setup(PyObject*, PyObject* args) {
  PyObject *d16, *d32, *d64, *tensor, *array, *void_p, *context, *stream, *fallback;
  if (!PyArg_ParseTuple(args, "(OOO)OOOOOO", &d16, &d32, &d64, &tensor, &array, &void_p, &context, &stream, &fallback)) return nullptr;
  PyObject* data_ptr = PyObject_GetAttrString(tensor, "data_ptr");
  if (data_ptr == nullptr) return nullptr;
  PyObject* keep[] = {d16, d32, d64, tensor, array, void_p, context, stream, fallback};
  for (PyObject* o : keep) Py_INCREF(o);
  g_dtypes[0] = d16; g_dtypes[1] = d32; g_dtypes[2] = d64;
  g_tensor = reinterpret_cast<PyTypeObject*>(tensor);
  g_data_ptr = data_ptr;
  g_array = reinterpret_cast<PyTypeObject*>(array);
  g_void_p = reinterpret_cast<PyTypeObject*>(void_p);
  g_context = reinterpret_cast<PyTypeObject*>(context);
  g_stream = reinterpret_cast<PyTypeObject*>(stream);
  g_fallback = fallback;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"setup", py_setup, METH_VARARGS, "Objects of the Python side that the conversions compare with."},
    {"launch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_launch)), METH_FASTCALL | METH_KEYWORDS,
     "launch(name, dtype, *args): call launch_<name>_<suffix>(*args); tensors become device pointers.\n"
     "The last argument must be a Stream or a StreamContext."},
    {"chain_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_chain_forward)), METH_FASTCALL, "mpJitForward"},
    {"chain_reverse", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_chain_reverse)), METH_FASTCALL, "mpJitReverse"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "mp_launch", "Native call path of the launchers.", -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_mp_launch(void) {
  g_ctx_name = PyUnicode_InternFromString("ctx");
  g_table = PyDict_New();
  if (g_ctx_name == nullptr || g_table == nullptr) return nullptr;
  for (size_t i = 0; i < sizeof(kLaunchers) / sizeof(kLaunchers[0]); ++i) {
    PyObject* v = PyLong_FromSize_t(i);
    if (v == nullptr || PyDict_SetItemString(g_table, kLaunchers[i].name, v) != 0) return nullptr;
    Py_DECREF(v);
  }
  return PyModule_Create(&kModule);
}
