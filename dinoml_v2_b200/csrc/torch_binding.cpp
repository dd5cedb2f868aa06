// CPython entry points for the tensor-level wrappers in kernels.py and Session.run_torch: argument checks, output allocation,
// the current stream and the C-ABI call in one native function.
//
// What bounds a decode-sized call is the host: the interpreted path (tensor attributes, shape tuples, torch.empty, the stream
// object, ctypes argument conversion) took 14.5 us per gemm_rcr call, 4.2 us of it inside the library, while the kernel of a
// [4096 x 4096] weight takes 5 us.  Here the same steps read the tensor's C++ object directly.
//
// Every function returns None when the arguments are not the plain case (a wrong type, shape, device or layout, a mapping that
// is not a dict): the Python wrapper then runs its own checks, which raise the documented errors.  A launch that fails returns
// the library's code as an int.  The interpreter lock is released around the library call, as ctypes does.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <climits>
#include <cstring>
#include <memory>
#include <vector>

#include "../../include/dinoml_b200_gguf.h"
#include "../../include/dinoml_b200_runtime.h"

namespace {

struct QTypeInfo { const char* name; int value, block, bytes; };
constexpr QTypeInfo kQTypes[] = {{"Q4_K", 12, 256, 144}, {"Q6_K", 14, 256, 210}, {"Q8_0", 8, 32, 34},  {"Q5_K", 13, 256, 176}, {"Q4_0", 2, 32, 18},
                                 {"Q2_K", 10, 256, 84},  {"Q3_K", 11, 256, 110}, {"MXFP4", 39, 32, 17}, {"NVFP4", 40, 64, 36}};

// A qtype as kernels.py takes it: a name in any case, a ggml enum value or a QType (its `value`).
const QTypeInfo* qtype_of(PyObject* o) {
  if (PyUnicode_Check(o)) {
    Py_ssize_t len = 0;
    const char* s = PyUnicode_AsUTF8AndSize(o, &len);
    if (s == nullptr) { PyErr_Clear(); return nullptr; }
    for (const QTypeInfo& q : kQTypes) {
      if (size_t(len) != std::strlen(q.name)) continue;
      bool same = true;
      for (Py_ssize_t i = 0; i < len && same; ++i) same = ((s[i] >= 'a' && s[i] <= 'z') ? s[i] - 32 : s[i]) == q.name[i];
      if (same) return &q;
    }
    return nullptr;
  }
  long value = -1;
  if (PyLong_CheckExact(o)) {
    value = PyLong_AsLong(o);
  } else {
    PyObject* v = PyObject_GetAttrString(o, "value");
    if (v == nullptr) { PyErr_Clear(); return nullptr; }
    if (PyLong_CheckExact(v)) value = PyLong_AsLong(v);
    Py_DECREF(v);
  }
  if (PyErr_Occurred()) PyErr_Clear();
  for (const QTypeInfo& q : kQTypes) if (q.value == value) return &q;
  return nullptr;
}

int dino_dtype(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return DINO_DTYPE_FLOAT16;
    case at::kFloat: return DINO_DTYPE_FLOAT32;
    case at::kBFloat16: return DINO_DTYPE_BFLOAT16;
    default: return 0;
  }
}

const at::Tensor* cuda_tensor(PyObject* o) {            // a contiguous CUDA tensor, or null
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() ? &t : nullptr;
}

// "auto" -> 0, an int -> itself; anything else (a family name, a tuning configuration) is left to variant_code() in Python.
bool variant_of(PyObject* o, int* out) {
  if (PyLong_CheckExact(o)) { *out = int(PyLong_AsLong(o)); return true; }
  if (PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, "auto") == 0) { *out = DINOML_B200_GGUF_VARIANT_AUTO; return true; }
  return false;
}

bool stream_of(PyObject* o, void** out) {
  if (o == Py_None) { *out = c10::cuda::getCurrentCUDAStream().stream(); return true; }
  PyObject* v = PyObject_GetAttrString(o, "cuda_stream");
  if (v == nullptr) { PyErr_Clear(); return false; }
  *out = PyLong_AsVoidPtr(v);
  Py_DECREF(v);
  if (PyErr_Occurred()) { PyErr_Clear(); return false; }
  return true;
}

template <typename F> PyObject* guarded(F f) {
  try {
    return f();
  } catch (const c10::OutOfMemoryError& e) {
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch != nullptr ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    if (type != nullptr) PyErr_SetString(type, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// [..., columns] in the dtype and on the device of `a`.
at::Tensor empty_like_rows(const at::Tensor& a, int64_t columns) {
  c10::SmallVector<int64_t, 8> shape(a.sizes().begin(), a.sizes().end());
  shape.back() = columns;
  return at::empty(shape, a.options().requires_grad(false));
}

// linear(a, b, qtype, bias, variant, out, stream) and gated(a, b01, qtype, bias01, variant, out, stream, activation)
PyObject* gemm(PyObject* const* args, bool gated, int activation) {
  const at::Tensor *a = cuda_tensor(args[0]), *b = cuda_tensor(args[1]);
  const QTypeInfo* q = qtype_of(args[2]);
  int variant = 0;
  void* stream = nullptr;
  if (a == nullptr || b == nullptr || q == nullptr || !variant_of(args[4], &variant) || a->dim() < 1) Py_RETURN_NONE;
  const int dtype = dino_dtype(a->scalar_type());
  const int64_t k = a->size(-1);
  if (dtype == 0 || k <= 0 || k % q->block || b->scalar_type() != at::kByte || b->dim() != 2 || b->size(1) != k / q->block * q->bytes) Py_RETURN_NONE;
  const int64_t m = a->numel() / k, rows = b->size(0), n = gated ? rows / 2 : rows;
  if (m > INT_MAX || rows > INT_MAX || k > INT_MAX || (gated && rows % 16)) Py_RETURN_NONE;
  const at::Tensor *bias = nullptr, *given = nullptr;
  if (args[3] != Py_None) {
    bias = cuda_tensor(args[3]);
    if (bias == nullptr || bias->scalar_type() != a->scalar_type() || bias->numel() != rows) Py_RETURN_NONE;
  }
  if (args[5] != Py_None && (given = cuda_tensor(args[5])) == nullptr) Py_RETURN_NONE;
  if (!stream_of(args[6], &stream)) Py_RETURN_NONE;
  const at::Tensor made = given != nullptr ? at::Tensor() : empty_like_rows(*a, n);
  const void* bias_ptr = bias != nullptr ? bias->const_data_ptr() : nullptr;
  const void *ap = a->const_data_ptr(), *bp = b->const_data_ptr();
  void* out = (given != nullptr ? *given : made).mutable_data_ptr();
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS
  rc = gated ? dinoml_b200_gguf_dual_gemm_rcr_bias(ap, bp, bias_ptr, out, nullptr, 0, q->value, dtype, int(m), int(n), int(k), activation, variant, stream)
             : dinoml_b200_gguf_gemm_rcr(ap, bp, bias_ptr, out, q->value, dtype, int(m), int(n), int(k), variant, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) return PyLong_FromLong(rc);
  if (given != nullptr) { Py_INCREF(args[5]); return args[5]; }
  return THPVariable_Wrap(made);
}

PyObject* py_linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 7) { PyErr_SetString(PyExc_TypeError, "linear takes 7 arguments"); return nullptr; }
  return guarded([&] { return gemm(args, false, 0); });
}

PyObject* py_gated(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 8) { PyErr_SetString(PyExc_TypeError, "gated takes 8 arguments"); return nullptr; }
  if (!PyUnicode_Check(args[7])) Py_RETURN_NONE;
  const int activation = PyUnicode_CompareWithASCIIString(args[7], "silu") == 0 ? 1 : PyUnicode_CompareWithASCIIString(args[7], "fast_gelu") == 0 ? 2 : 0;
  if (activation == 0) Py_RETURN_NONE;
  return guarded([&] { return gemm(args, true, activation); });
}

// dequantize(blocks, qtype, n_per_row, dtype name, out, stream)
PyObject* py_dequantize(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 6) { PyErr_SetString(PyExc_TypeError, "dequantize takes 6 arguments"); return nullptr; }
  return guarded([&]() -> PyObject* {
    const at::Tensor *blocks = cuda_tensor(args[0]), *given = nullptr;
    const QTypeInfo* q = qtype_of(args[1]);
    void* stream = nullptr;
    if (blocks == nullptr || q == nullptr || !PyLong_CheckExact(args[2]) || !PyUnicode_Check(args[3])) Py_RETURN_NONE;
    const int64_t k = PyLong_AsLongLong(args[2]);
    if (PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
    int code = -1;
    at::ScalarType type = at::kFloat;
    if (PyUnicode_CompareWithASCIIString(args[3], "float32") == 0) code = 0;
    else if (PyUnicode_CompareWithASCIIString(args[3], "float16") == 0) { code = 1; type = at::kHalf; }
    else if (PyUnicode_CompareWithASCIIString(args[3], "bfloat16") == 0) { code = 2; type = at::kBFloat16; }
    if (code < 0 || k <= 0 || k % q->block || blocks->scalar_type() != at::kByte || blocks->dim() != 2 || blocks->size(1) != k / q->block * q->bytes) Py_RETURN_NONE;
    if (args[4] != Py_None && (given = cuda_tensor(args[4])) == nullptr) Py_RETURN_NONE;
    if (!stream_of(args[5], &stream)) Py_RETURN_NONE;
    const int64_t rows = blocks->size(0);
    const at::Tensor made = given != nullptr ? at::Tensor() : at::empty({rows, k}, blocks->options().dtype(type));
    const void* in = blocks->const_data_ptr();
    void* out = (given != nullptr ? *given : made).mutable_data_ptr();
    int rc = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = libgguf_cuda_dequantize_rows_on_stream(in, q->value, rows, k, code, out, stream);
    Py_END_ALLOW_THREADS
    if (rc != 0) return PyLong_FromLong(rc);
    if (given != nullptr) { Py_INCREF(args[4]); return args[4]; }
    return THPVariable_Wrap(made);
  });
}

// ---- sessions.  A Runner carries what Session.run_torch needs of the artifact: the names and dtypes of its inputs and outputs,
// the output shapes as a walk over the nodes (a node's result is its input's shape with `columns` as the last dimension), and the
// run entry of the library the artifact loaded (an artifact may carry its own copy).
struct Runner {
  int (*run)(DinoSession*, const DinoTensor*, size_t, DinoTensor*, size_t) = nullptr;
  DinoSession* session = nullptr;
  struct Port { PyObject* name; int tensor; at::ScalarType type; };
  std::vector<Port> inputs, outputs;
  struct Node { int from, to; int64_t columns; };
  std::vector<Node> nodes;
  int tensors = 0;
  ~Runner() {
    for (Port& p : inputs) Py_XDECREF(p.name);
    for (Port& p : outputs) Py_XDECREF(p.name);
  }
};
constexpr const char* kRunnerName = "dinoml_b200.Runner";

bool scalar_type_of(const char* name, at::ScalarType* out) {
  if (std::strcmp(name, "float16") == 0) *out = at::kHalf;
  else if (std::strcmp(name, "bfloat16") == 0) *out = at::kBFloat16;
  else if (std::strcmp(name, "float32") == 0) *out = at::kFloat;
  else return false;
  return true;
}

// make_runner(run entry address, session address, tensors, [(name, tensor, dtype)...] inputs, outputs, [(from, to, columns)...])
PyObject* py_make_runner(PyObject*, PyObject* args) {
  unsigned long long run = 0, session = 0;
  int tensors = 0;
  PyObject *ins = nullptr, *outs = nullptr, *nodes = nullptr;
  if (!PyArg_ParseTuple(args, "KKiO!O!O!", &run, &session, &tensors, &PyList_Type, &ins, &PyList_Type, &outs, &PyList_Type, &nodes)) return nullptr;
  auto r = std::make_unique<Runner>();
  r->run = reinterpret_cast<decltype(r->run)>(uintptr_t(run));
  r->session = reinterpret_cast<DinoSession*>(uintptr_t(session));
  r->tensors = tensors;
  for (int side = 0; side < 2; ++side) {
    PyObject* list = side == 0 ? ins : outs;
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
      Runner::Port p{nullptr, 0, at::kFloat};
      const char* dtype = nullptr;
      if (!PyArg_ParseTuple(PyList_GET_ITEM(list, i), "Uis", &p.name, &p.tensor, &dtype)) return nullptr;
      if (p.tensor < 0 || p.tensor >= tensors || !scalar_type_of(dtype, &p.type)) { PyErr_SetString(PyExc_ValueError, "bad port"); return nullptr; }
      Py_INCREF(p.name);
      PyUnicode_InternInPlace(&p.name);
      (side == 0 ? r->inputs : r->outputs).push_back(p);
    }
  }
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(nodes); ++i) {
    int from = 0, to = 0;
    long long columns = 0;
    if (!PyArg_ParseTuple(PyList_GET_ITEM(nodes, i), "iiL", &from, &to, &columns)) return nullptr;
    if (from < 0 || from >= tensors || to < 0 || to >= tensors) { PyErr_SetString(PyExc_ValueError, "bad node"); return nullptr; }
    r->nodes.push_back({from, to, columns});
  }
  return PyCapsule_New(r.release(), kRunnerName, [](PyObject* c) { delete static_cast<Runner*>(PyCapsule_GetPointer(c, kRunnerName)); });
}

DinoTensor describe(const at::Tensor& t, int dtype) {
  DinoTensor d;
  std::memset(&d, 0, sizeof(d));
  d.data = t.numel() != 0 ? const_cast<void*>(t.const_data_ptr()) : nullptr;
  d.shape = t.sizes().data();
  d.ndim = size_t(t.dim());
  d.dtype = decltype(d.dtype)(dtype);
  d.nbytes = size_t(t.numel()) * t.element_size();
  d.device_type = decltype(d.device_type)(DINO_DEVICE_CUDA);
  d.flags = 1;
  return d;
}

// run_torch(runner, inputs dict, outputs dict or None) -> outputs dict, None (not the plain case) or an error code
PyObject* py_run_torch(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  if (nargs != 3) { PyErr_SetString(PyExc_TypeError, "run_torch takes 3 arguments"); return nullptr; }
  Runner* r = static_cast<Runner*>(PyCapsule_GetPointer(args[0], kRunnerName));
  if (r == nullptr) return nullptr;
  if (!PyDict_CheckExact(args[1]) || (args[2] != Py_None && !PyDict_CheckExact(args[2]))) Py_RETURN_NONE;
  return guarded([&]() -> PyObject* {
    c10::SmallVector<DinoTensor, 8> ins, outs;
    std::vector<at::Tensor> made;
    auto port = [](PyObject* dict, const Runner::Port& p) -> const at::Tensor* {
      PyObject* o = PyDict_GetItemWithError(dict, p.name);
      if (o == nullptr) { PyErr_Clear(); return nullptr; }
      if (!THPVariable_Check(o)) return nullptr;
      const at::Tensor& t = THPVariable_Unpack(o);
      return t.defined() && t.is_cuda() && t.layout() == at::kStrided && dino_dtype(t.scalar_type()) != 0 && t.numel() != 0 ? &t : nullptr;
    };
    const at::Tensor* first = nullptr;
    c10::SmallVector<c10::SmallVector<int64_t, 4>, 8> shapes;
    if (args[2] == Py_None) shapes.resize(size_t(r->tensors));
    for (const Runner::Port& p : r->inputs) {
      const at::Tensor* t = port(args[1], p);
      if (t == nullptr) Py_RETURN_NONE;
      if (first == nullptr) first = t;
      ins.push_back(describe(*t, dino_dtype(t->scalar_type())));
      if (args[2] == Py_None) shapes[size_t(p.tensor)].assign(t->sizes().begin(), t->sizes().end());
    }
    if (first == nullptr) Py_RETURN_NONE;
    PyObject* result = nullptr;
    if (args[2] == Py_None) {
      for (const Runner::Node& n : r->nodes) {
        if (shapes[size_t(n.from)].empty()) Py_RETURN_NONE;
        shapes[size_t(n.to)] = shapes[size_t(n.from)];
        shapes[size_t(n.to)].back() = n.columns;
      }
      made.reserve(r->outputs.size());
      for (const Runner::Port& p : r->outputs) {
        made.push_back(at::empty(shapes[size_t(p.tensor)], first->options().dtype(p.type).requires_grad(false)));
        outs.push_back(describe(made.back(), dino_dtype(p.type)));
      }
    } else {
      for (const Runner::Port& p : r->outputs) {
        const at::Tensor* t = port(args[2], p);
        if (t == nullptr) Py_RETURN_NONE;
        outs.push_back(describe(*t, dino_dtype(t->scalar_type())));
      }
    }
    int rc = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = r->run(r->session, ins.data(), ins.size(), outs.data(), outs.size());
    Py_END_ALLOW_THREADS
    if (rc != 0) return PyLong_FromLong(rc);
    if (args[2] != Py_None) return PyDict_Copy(args[2]);
    result = PyDict_New();
    if (result == nullptr) return nullptr;
    for (size_t i = 0; i < made.size(); ++i) {
      PyObject* t = THPVariable_Wrap(made[i]);
      if (t == nullptr || PyDict_SetItem(result, r->outputs[i].name, t) != 0) { Py_XDECREF(t); Py_DECREF(result); return nullptr; }
      Py_DECREF(t);
    }
    return result;
  });
}

PyMethodDef kMethods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_linear)), METH_FASTCALL, nullptr},
    {"gated", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_gated)), METH_FASTCALL, nullptr},
    {"dequantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_dequantize)), METH_FASTCALL, nullptr},
    {"make_runner", py_make_runner, METH_VARARGS, nullptr},
    {"run_torch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_run_torch)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_torch_binding", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_binding(void) { return PyModule_Create(&kModule); }
