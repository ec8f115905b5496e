// The calls that issue collectives, as a CPython extension: a Communicator of mccs_b200/client.py
// holds one CommCalls object and hands its methods out as its own.
//
// A collective on a small message costs the GPU a few microseconds; written in Python over ctypes
// its call alone cost four to five (keyword handling 0.3, looking up the current stream 1.3, the capture
// check 0.3, argument objects and the ctypes call 1.5), which n ranks driven by one thread pay n
// times. Here a call in a group takes 0.9, posting the request included: the tensors are read through
// torch's C++ interface, one dictionary look-up each for operator and variant, and the C call with the
// interpreter lock released.
//
// The C API's functions arrive as addresses (`bind`), so that this module always talks to the
// libmccs.so the package has loaded.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/TensorSubclassLikeUtils.h>
#include <c10/core/GradMode.h>
#include <c10/core/InferenceMode.h>
#ifdef MCCS_TORCH_CUDA
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#endif
#include <cuda.h>
#include <dlfcn.h>
#include <stdint.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/headeronly/version.h>

#include "../include/mccs.h"
#include "../include/mccs_noalloc.h"

namespace {

decltype(&mccsAllReduceEx) g_all_reduce;
decltype(&mccsAllGatherEx) g_all_gather;
decltype(&mccsReduceScatterEx) g_reduce_scatter;
decltype(&mccsCommSelfCopy) g_self_copy;
decltype(&mccsCommTakesAnyMemory) g_takes_any_memory;
decltype(&mccsMemInfo) g_mem_info;
decltype(&mccsGroupStart) g_group_start;
decltype(&mccsGroupEnd) g_group_end;

// Owned for the life of the process.
PyObject* g_dtypes;           // torch.dtype -> mccsDataType_t
PyObject* g_ops;              // operator name -> mccsRedOp_t
PyObject* g_algos;            // variant name -> mccsAlgo_t
PyObject* g_error;            // MccsError(code, what)
PyObject* g_buffer_type;      // Buffer
PyObject* g_capturing;        // () -> is the current stream of the current device capturing; None without CUDA
PyObject *s_lower, *s_cuda_stream, *s_ptr;

// The driver calls of the capture check, when libcuda is there.
decltype(&cuStreamIsCapturing) g_is_capturing;
decltype(&cuCtxGetDevice) g_ctx_device;

struct Calls {
  PyObject_HEAD
  mccsComm_t comm;
  int device;
  int cuda;     // the daemon's backend is CUDA
  int any_memory;   // mccsCommTakesAnyMemory
};

const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// torch's current stream on a device and its current device. A torch without CUDA has neither (and no CUDA
// tensors): the daemon's host backend needs none, a GPU's wants the stream named.
#ifdef MCCS_TORCH_CUDA
uint64_t current_stream(int device) { return (uint64_t)c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }
int current_device() { return (int)c10::cuda::current_device(); }
#else
uint64_t current_stream(int) { throw std::runtime_error("this torch is built without CUDA: a collective on a GPU needs stream="); }
int current_device() { return -1; }
#endif

// mccsDataType_t of a tensor, if there is one.
bool known_type(const at::Tensor& t, int* out) {
  switch (t.scalar_type()) {
    case at::kChar: *out = mccsInt8; return true;
    case at::kByte: *out = mccsUint8; return true;
    case at::kInt: *out = mccsInt32; return true;
    case at::kUInt32: *out = mccsUint32; return true;
    case at::kLong: *out = mccsInt64; return true;
    case at::kUInt64: *out = mccsUint64; return true;
    case at::kHalf: *out = mccsFloat16; return true;
    case at::kFloat: *out = mccsFloat32; return true;
    case at::kDouble: *out = mccsFloat64; return true;
    case at::kBFloat16: *out = mccsBfloat16; return true;
    default: return false;
  }
}

// The same; KeyError with the type, as the dictionary raises it, when there is none.
bool type_code(const at::Tensor& t, PyObject* of, int* out) {
  if (known_type(t, out)) return true;
  PyObject* d = PyObject_GetAttrString(of, "dtype");
  if (d) {
    PyErr_SetObject(PyExc_KeyError, d);
    Py_DECREF(d);
  }
  return false;
}

bool to_u64(PyObject* o, uint64_t* out) {   // steals nothing
  PyObject* i = PyNumber_Index(o);
  if (!i) {
    PyErr_Clear();
    i = PyNumber_Long(o);
    if (!i) return false;
  }
  *out = (uint64_t)PyLong_AsUnsignedLongLongMask(i);
  Py_DECREF(i);
  return !PyErr_Occurred();
}

// Address of a tensor, a Buffer or a raw pointer.
bool address(PyObject* o, uint64_t* out) {
  if (const at::Tensor* t = tensor(o)) { *out = (uint64_t)t->data_ptr(); return true; }
  if (PyObject_TypeCheck(o, (PyTypeObject*)g_buffer_type)) {
    PyObject* p = PyObject_GetAttr(o, s_ptr);
    if (!p) return false;
    const bool ok = to_u64(p, out);
    Py_DECREF(p);
    return ok;
  }
  return to_u64(o, out);
}

// dict[key] as an int; KeyError as Python's own subscription raises it.
bool lookup(PyObject* dict, PyObject* key, int* out) {
  PyObject* v = PyDict_GetItemWithError(dict, key);
  if (!v) {
    if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, key);
    return false;
  }
  *out = (int)PyLong_AsLong(v);
  return !(*out == -1 && PyErr_Occurred());
}

bool op_code(PyObject* op, int* out) {
  if (PyObject* v = PyDict_GetItemWithError(g_ops, op)) {
    *out = (int)PyLong_AsLong(v);
    return true;
  }
  if (PyErr_Occurred()) return false;
  PyObject* low = PyObject_CallMethodNoArgs(op, s_lower);
  if (!low) return false;
  const bool ok = lookup(g_ops, low, out);
  Py_DECREF(low);
  return ok;
}

PyObject* raise(int code, const char* what) {
  PyObject* e = PyObject_CallFunction(g_error, "is", code, what);
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  return nullptr;
}

// The stream a call goes to, and the refusal of graph capture: a collective takes its barrier
// epoch and its ticket from the daemon at the call, so a graph that captured one would replay
// stale values.
bool resolve_stream(Calls* self, PyObject* stream, uint64_t* out) {
  *out = 0;
  if (self->cuda) {
#ifdef MCCS_TORCH_CUDA
    const uint64_t current = current_stream(self->device);
#else
    const uint64_t current = stream && stream != Py_None ? 0 : current_stream(self->device);
#endif
    bool capturing = false, known = false;
    CUdevice now = -1;
    if (g_is_capturing && g_ctx_device && g_ctx_device(&now) == CUDA_SUCCESS && (int)now == self->device) {
      CUstreamCaptureStatus st = CU_STREAM_CAPTURE_STATUS_NONE;
      known = g_is_capturing((CUstream)current, &st) == CUDA_SUCCESS;
      capturing = known && st != CU_STREAM_CAPTURE_STATUS_NONE;
    }
    if (!known) {   // another device is current, or the question was refused: as torch answers it
      PyObject* c = PyObject_CallNoArgs(g_capturing);
      if (!c) PyErr_Clear();   // no usable CUDA runtime in this process: nothing can be capturing
      else { capturing = PyObject_IsTrue(c) == 1; Py_DECREF(c); }
    }
    if (capturing) { raise(mccsUnsupported, "a collective inside CUDA graph capture"); return false; }
    *out = current;
  }
  if (stream && stream != Py_None) {
    if (PyLong_Check(stream)) { *out = (uint64_t)PyLong_AsUnsignedLongLongMask(stream); return !PyErr_Occurred(); }
    PyObject* h = PyObject_GetAttr(stream, s_cuda_stream);
    if (!h) return false;
    const bool ok = to_u64(h, out);
    Py_DECREF(h);
    return ok;
  }
  return true;
}

// Arguments of a METH_FASTCALL | METH_KEYWORDS method by name; `npos` of them may be positional.
bool take(const char* fn, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames, const char* const* names, int npos, int nrequired,
          int total, PyObject** out) {
  if (nargs > npos) {
    PyErr_Format(PyExc_TypeError, "%s() takes at most %d positional arguments (%zd given)", fn, npos, nargs);
    return false;
  }
  for (Py_ssize_t i = 0; i < nargs; i++) out[i] = args[i];
  const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  for (Py_ssize_t k = 0; k < nkw; k++) {
    PyObject* name = PyTuple_GET_ITEM(kwnames, k);
    int at = -1;
    for (int i = 0; i < total && at < 0; i++)
      if (PyUnicode_CompareWithASCIIString(name, names[i]) == 0) at = i;
    if (at < 0) { PyErr_Format(PyExc_TypeError, "%s() got an unexpected keyword argument '%U'", fn, name); return false; }
    if (out[at]) { PyErr_Format(PyExc_TypeError, "%s() got multiple values for argument '%U'", fn, name); return false; }
    out[at] = args[nargs + k];
  }
  for (int i = 0; i < nrequired; i++)
    if (!out[i]) { PyErr_Format(PyExc_TypeError, "%s() missing required argument '%s'", fn, names[i]); return false; }
  return true;
}

bool given(PyObject* o) { return o && o != Py_None; }

// all_reduce and reduce_scatter: `from_send`: whether send (else recv) names type and count.
PyObject* reducing(Calls* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames, const char* fn, const char* what, bool scatter) {
  static const char* const names[] = {"send", "recv", "count", "dtype", "op", "scale", "algo", "stream"};
  PyObject* a[8] = {nullptr};
  if (!take(fn, args, nargs, kwnames, names, 2, scatter ? 2 : 1, 8, a)) return nullptr;
  PyObject* recv = given(a[1]) || scatter ? a[1] : a[0];
  PyObject* shape = scatter ? recv : a[0];
  uint64_t send_va, recv_va, count = 0;
  int dtype = 0, op = mccsSum, algo = mccsAlgoAuto;
  bool have_count = given(a[2]), have_dtype = given(a[3]);
  if (have_count && !to_u64(a[2], &count)) return nullptr;
  if (have_dtype && !lookup(g_dtypes, a[3], &dtype)) return nullptr;
  if (const at::Tensor* t = tensor(shape)) {
    if (!have_count) count = (uint64_t)t->numel();
    if (!have_dtype && !type_code(*t, shape, &dtype)) return nullptr;
  } else if (!have_count || !have_dtype) {
    PyErr_SetString(PyExc_ValueError, "dtype and count are needed for raw pointers");
    return nullptr;
  }
  float scale = 1.0f;
  if (a[5]) {
    const double d = PyFloat_AsDouble(a[5]);
    if (d == -1.0 && PyErr_Occurred()) return nullptr;
    scale = (float)d;
  }
  if (a[4] && !op_code(a[4], &op)) return nullptr;
  if (a[6] && !lookup(g_algos, a[6], &algo)) return nullptr;
  if (!address(a[0], &send_va)) return nullptr;
  if (recv == a[0]) recv_va = send_va;
  else if (!address(recv, &recv_va)) return nullptr;
  uint64_t stream;
  if (!resolve_stream(self, a[7], &stream)) return nullptr;
  mccsResult_t rc;
  const mccsComm_t comm = self->comm;
  Py_BEGIN_ALLOW_THREADS
  rc = (scatter ? g_reduce_scatter : g_all_reduce)(comm, (const void*)send_va, (void*)recv_va, (size_t)count, (mccsDataType_t)dtype, (mccsRedOp_t)op,
                                                   scale, (mccsAlgo_t)algo, (mccsStream_t)stream);
  Py_END_ALLOW_THREADS
  if (rc != mccsSuccess) return raise(rc, what);
  Py_RETURN_NONE;
}

PyObject* all_reduce(PyObject* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  return reducing((Calls*)self, args, nargs, kwnames, "all_reduce", "mccsAllReduce", false);
}

PyObject* reduce_scatter(PyObject* self, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  return reducing((Calls*)self, args, nargs, kwnames, "reduce_scatter", "mccsReduceScatter", true);
}

PyObject* all_gather(PyObject* self_, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  static const char* const names[] = {"send", "recv", "nbytes", "algo", "stream"};
  Calls* self = (Calls*)self_;
  PyObject* a[5] = {nullptr};
  if (!take("all_gather", args, nargs, kwnames, names, 2, 2, 5, a)) return nullptr;
  uint64_t nbytes = 0, send_va, recv_va, stream;
  if (given(a[2])) {
    if (!to_u64(a[2], &nbytes)) return nullptr;
  } else if (const at::Tensor* t = tensor(a[0])) {
    nbytes = (uint64_t)t->numel() * (uint64_t)t->element_size();
  } else {
    PyErr_SetString(PyExc_ValueError, "nbytes is needed for raw pointers");
    return nullptr;
  }
  int algo = mccsAlgoAuto;
  if (a[3] && !lookup(g_algos, a[3], &algo)) return nullptr;
  if (!address(a[0], &send_va) || !address(a[1], &recv_va)) return nullptr;
  if (!resolve_stream(self, a[4], &stream)) return nullptr;
  mccsResult_t rc;
  const mccsComm_t comm = self->comm;
  Py_BEGIN_ALLOW_THREADS
  rc = g_all_gather(comm, (const void*)send_va, (void*)recv_va, (size_t)nbytes, (mccsAlgo_t)algo, (mccsStream_t)stream);
  Py_END_ALLOW_THREADS
  if (rc != mccsSuccess) return raise(rc, "mccsAllGather");
  Py_RETURN_NONE;
}

// Whether the bytes behind a tensor are its values: no conjugation, sign or zero that torch applies
// when it reads them, no wrapper or mode that has to see the operation.
bool plain_bytes(const at::Tensor& t) {
  return !t.is_conj() && !t.is_neg() && !t._is_zerotensor() && !t.is_quantized() && !at::isTensorSubclassLike(t);
}

// Whether writing `out` from `in` concerns autograd beyond the version of `out`: what copy_ records, or
// refuses, is left to copy_.
bool autograd_takes_part(const at::Tensor& in, const at::Tensor& out) {
  return (at::GradMode::is_enabled() && (in.requires_grad() || out.requires_grad())) || in._fw_grad(0).defined() || out._fw_grad(0).defined() ||
         (out.is_inference() && !c10::InferenceMode::is_enabled());
}

// self_copy(send, recv, stream) -> bool. Any collective of a communicator of one rank whose tensors
// are plain memory of its GPU: one copy kernel on them where they are. False when that does not apply
// (more ranks, other devices, other layouts, differing types, values that are not the bytes, ranges that
// overlap in part, another stream than the current one) and the caller has to stage.
PyObject* self_copy(PyObject* self_, PyObject* const* args, Py_ssize_t nargs) {
  Calls* self = (Calls*)self_;
  if (nargs != 3) { PyErr_SetString(PyExc_TypeError, "self_copy(send, recv, stream)"); return nullptr; }
  const at::Tensor* in = self->any_memory ? tensor(args[0]) : nullptr;
  const at::Tensor* out = in ? tensor(args[1]) : nullptr;
  if (!out || !in->is_cuda() || !out->is_cuda() || in->get_device() != self->device || out->get_device() != self->device ||
      in->scalar_type() != out->scalar_type() || in->numel() != out->numel() || in->numel() == 0 || !plain_bytes(*in) || !plain_bytes(*out) ||
      !in->is_contiguous() || !out->is_contiguous())
    Py_RETURN_FALSE;
  const void* const from = in->data_ptr();
  void* const to = out->data_ptr();
  const size_t bytes = (size_t)in->numel() * (size_t)in->element_size();
  if (from != to && (from < to ? (const char*)to - (const char*)from : (const char*)from - (const char*)to) < (ptrdiff_t)bytes) Py_RETURN_FALSE;
  uint64_t stream;
  if (!resolve_stream(self, args[2], &stream)) return nullptr;
  // Memory of the service is named as such: the request then keeps it from being freed while it waits.
  int dtype;
  const bool service = g_mem_info(from, nullptr, nullptr, nullptr) == mccsSuccess && g_mem_info(to, nullptr, nullptr, nullptr) == mccsSuccess;
  if (service ? !known_type(*in, &dtype) : autograd_takes_part(*in, *out)) Py_RETURN_FALSE;
  // The tensors belong to the current stream's order, whichever stream the collective is given: the staged
  // form copies there.
  if (!service && stream != current_stream(self->device)) Py_RETURN_FALSE;
  mccsResult_t rc;
  const mccsComm_t comm = self->comm;
  Py_BEGIN_ALLOW_THREADS
  rc = service ? g_all_gather(comm, from, to, bytes, mccsAlgoAuto, (mccsStream_t)stream) : g_self_copy(comm, from, to, bytes, (mccsStream_t)stream);
  Py_END_ALLOW_THREADS
  if (rc == mccsUnsupported && !service) Py_RETURN_FALSE;
  if (rc == mccsSuccess && !service && !out->is_inference()) torch::autograd::impl::bump_version(*out);   // as copy_ does
  if (rc != mccsSuccess) return raise(rc, service ? "mccsAllGather" : "mccsCommSelfCopy");
  Py_RETURN_TRUE;
}

PyObject* attach(PyObject* self_, PyObject* args) {
  Calls* self = (Calls*)self_;
  unsigned long long h = 0;
  if (!PyArg_ParseTuple(args, "Kii", &h, &self->device, &self->cuda)) return nullptr;
  self->comm = (mccsComm_t)h;
  self->any_memory = self->comm ? g_takes_any_memory(self->comm) : 0;
  Py_RETURN_NONE;
}

// A tensor without storage throws when it is asked for its address: a Python error, not the end of
// the process.
template <typename... Args> PyObject* caught(PyObject* (*fn)(Args...), Args... args) {
  try {
    return fn(args...);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  } catch (...) {
    PyErr_SetString(PyExc_RuntimeError, "unknown C++ exception");
  }
  return nullptr;
}
template <PyObject* (*fn)(PyObject*, PyObject* const*, Py_ssize_t, PyObject*)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n, PyObject* kw) { return caught(fn, self, args, n, kw); }
template <PyObject* (*fn)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* args, Py_ssize_t n) { return caught(fn, self, args, n); }

PyMethodDef calls_methods[] = {
    {"all_reduce", (PyCFunction)(void (*)(void))(_PyCFunctionFastWithKeywords)guarded<all_reduce>, METH_FASTCALL | METH_KEYWORDS,
     "all_reduce(send, recv=None, *, count=None, dtype=None, op='sum', scale=1.0, algo='auto', stream=None)\n"
     "AllReduce ``count`` elements; in place when ``recv`` is None."},
    {"all_gather", (PyCFunction)(void (*)(void))(_PyCFunctionFastWithKeywords)guarded<all_gather>, METH_FASTCALL | METH_KEYWORDS,
     "all_gather(send, recv, *, nbytes=None, algo='auto', stream=None)\n"
     "AllGather ``nbytes`` per rank into ``recv`` (``nranks * nbytes`` bytes)."},
    {"reduce_scatter", (PyCFunction)(void (*)(void))(_PyCFunctionFastWithKeywords)guarded<reduce_scatter>, METH_FASTCALL | METH_KEYWORDS,
     "reduce_scatter(send, recv, *, count=None, dtype=None, op='sum', scale=1.0, algo='auto', stream=None)\n"
     "ReduceScatter: ``send`` holds ``nranks * count`` elements, ``recv`` receives the reduction of block ``rank``\n"
     "(``count`` elements). In place when ``recv`` is the rank's own block of ``send``. The reference has no such call."},
    {"self_copy", (PyCFunction)(void (*)(void))(_PyCFunctionFast)guarded<self_copy>, METH_FASTCALL,
     "self_copy(send, recv, stream) -> bool: a one-rank collective on ordinary CUDA tensors, in place of staging"},
    {"_attach", attach, METH_VARARGS, "_attach(handle, device, is_cuda): the communicator the calls go to (handle 0: none)"},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject calls_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* module_group_start(PyObject*, PyObject*) {
  const mccsResult_t rc = g_group_start();
  if (rc != mccsSuccess) return raise(rc, "mccsGroupStart");
  Py_RETURN_NONE;
}

// group_end(quiet): `quiet` when an exception is on its way out of the block already.
PyObject* module_group_end(PyObject*, PyObject* quiet) {
  mccsResult_t rc;
  Py_BEGIN_ALLOW_THREADS
  rc = g_group_end();
  Py_END_ALLOW_THREADS
  if (rc != mccsSuccess && quiet != Py_True) return raise(rc, "mccsGroupEnd");
  Py_RETURN_NONE;
}

// local_all_reduce(address of mccsLocalAllReduceNoAlloc, inputs, outputs, stream) -> its return value,
// or None when the tensors' device is not the current one (the caller makes it so and comes back).
PyObject* local_all_reduce(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 4) { PyErr_SetString(PyExc_TypeError, "local_all_reduce(function, inputs, outputs, stream)"); return nullptr; }
  const auto fn = (decltype(&mccsLocalAllReduceNoAlloc))PyLong_AsUnsignedLongLong(args[0]);
  if (PyErr_Occurred()) return nullptr;
  PyObject* seq[2] = {PySequence_Fast(args[1], "inputs"), nullptr};
  if (seq[0]) seq[1] = PySequence_Fast(args[2], "outputs");
  if (!seq[1]) { Py_XDECREF(seq[0]); return nullptr; }
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq[0]);
  const char* bad = nullptr;
  void* at[2][MCCS_NOALLOC_MAX_RANKS];
  int dtype = 0, device = -1;
  int64_t count = 0;
  if (n == 0) bad = "no tensors";
  else if (n != PySequence_Fast_GET_SIZE(seq[1]) || n > MCCS_NOALLOC_MAX_RANKS) bad = "need as many outputs as inputs, at most 8";
  const at::Tensor* first = nullptr;
  for (int side = 0; side < 2 && !bad; side++)
    for (Py_ssize_t i = 0; i < n && !bad; i++) {
      const at::Tensor* t = tensor(PySequence_Fast_GET_ITEM(seq[side], i));
      if (!first) first = t;
      if (!t || !t->is_cuda() || t->get_device() != first->get_device() || t->scalar_type() != first->scalar_type() || t->numel() != first->numel() ||
          !t->is_contiguous())
        bad = "tensors must be contiguous CUDA tensors of one device, dtype and size";
      else
        at[side][i] = t->data_ptr();
    }
  if (!bad) {
    device = (int)first->get_device();
    count = first->numel();
    switch (first->scalar_type()) {
      case at::kFloat: dtype = mccsFloat32; break;
      case at::kHalf: dtype = mccsFloat16; break;
      case at::kBFloat16: dtype = mccsBfloat16; break;
      default: bad = "float32, float16 or bfloat16 only";
    }
  }
  Py_DECREF(seq[0]);
  Py_DECREF(seq[1]);
  if (bad) { PyErr_SetString(PyExc_ValueError, bad); return nullptr; }
  // (The runtime's device: a thread that has not used CUDA yet has one, but no context of the driver's.)
  if (current_device() != device) Py_RETURN_NONE;
  uint64_t stream = 0;
  if (args[3] == Py_None) {
    stream = current_stream(device);
  } else {
    PyObject* h = PyObject_GetAttr(args[3], s_cuda_stream);
    const bool ok = h && to_u64(h, &stream);
    Py_XDECREF(h);
    if (!ok) return nullptr;
  }
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(at[0], at[1], (int)n, (size_t)count, dtype, (void*)stream);
  Py_END_ALLOW_THREADS
  return PyLong_FromLong(rc);
}

// bind(functions, Buffer, dtypes, ops, algos, MccsError, capturing)
PyObject* module_bind(PyObject*, PyObject* args) {
  unsigned long long ar, ag, rs, gs, ge, sc, am, mi;
  PyObject *buffer, *dtypes, *ops, *algos, *error, *capturing;
  if (!PyArg_ParseTuple(args, "(KKKKKKKK)OO!O!O!OO", &ar, &ag, &rs, &gs, &ge, &sc, &am, &mi, &buffer, &PyDict_Type, &dtypes, &PyDict_Type, &ops,
                        &PyDict_Type, &algos, &error, &capturing))
    return nullptr;
  g_all_reduce = (decltype(g_all_reduce))ar;
  g_all_gather = (decltype(g_all_gather))ag;
  g_reduce_scatter = (decltype(g_reduce_scatter))rs;
  g_group_start = (decltype(g_group_start))gs;
  g_group_end = (decltype(g_group_end))ge;
  g_self_copy = (decltype(g_self_copy))sc;
  g_takes_any_memory = (decltype(g_takes_any_memory))am;
  g_mem_info = (decltype(g_mem_info))mi;
  g_buffer_type = Py_NewRef(buffer);
  g_dtypes = Py_NewRef(dtypes);
  g_ops = Py_NewRef(ops);
  g_algos = Py_NewRef(algos);
  g_error = Py_NewRef(error);
  g_capturing = Py_NewRef(capturing);
  if (void* lib = dlopen("libcuda.so.1", RTLD_NOW | RTLD_LOCAL)) {
    g_is_capturing = (decltype(g_is_capturing))dlsym(lib, "cuStreamIsCapturing");
    g_ctx_device = (decltype(g_ctx_device))dlsym(lib, "cuCtxGetDevice");
  }
  Py_RETURN_NONE;
}

PyMethodDef module_methods[] = {{"bind", module_bind, METH_VARARGS, nullptr},
                                {"group_start", module_group_start, METH_NOARGS, nullptr},
                                {"group_end", module_group_end, METH_O, nullptr},
                                {"local_all_reduce", (PyCFunction)(void (*)(void))(_PyCFunctionFast)guarded<local_all_reduce>, METH_FASTCALL, nullptr},
                                {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_calls", "Collective calls of mccs_b200.", -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls(void) {
  calls_type.tp_name = "mccs_b200._calls.CommCalls";
  calls_type.tp_basicsize = sizeof(Calls);
  calls_type.tp_flags = Py_TPFLAGS_DEFAULT;
  calls_type.tp_methods = calls_methods;
  calls_type.tp_new = PyType_GenericNew;
  if (PyType_Ready(&calls_type) < 0) return nullptr;
  s_lower = PyUnicode_InternFromString("lower");
  s_cuda_stream = PyUnicode_InternFromString("cuda_stream");
  s_ptr = PyUnicode_InternFromString("ptr");
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  PyModule_AddObject(m, "CommCalls", Py_NewRef((PyObject*)&calls_type));
  PyModule_AddStringConstant(m, "built_for", TORCH_VERSION);   // it reads tensors through this version's C++ interface
  return m;
}
