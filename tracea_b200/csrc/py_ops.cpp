// CPython module behind tracea_b200.ops: turns torch tensors into the C ABI's tensor views and calls the library, without
// building a ctypes object per view.
//
// Why it exists: a small convolution is 5-10 us of GPU time, and through ctypes the calling thread spent 21-32 us per call
// on the GPU machines measured, most of it on the shape / stride arrays of five views.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include "../../include/tracea_b200.h"

namespace {

struct PyError {};   // a Python exception has been set

constexpr int kMaxRank = 8;
struct View {
  uint64_t shape[kMaxRank];
  int64_t stride[kMaxRank];
  TraceaTensorView v;
};

// `order`: dimension d of the view is dimension order[d] of the tensor (nullptr: the same).
void fill(View& o, const at::Tensor& t, const int* order = nullptr) {
  TraceaDType dt;
  switch (t.scalar_type()) {
    case at::kFloat: dt = TRACEA_DTYPE_FLOAT32; break;
    case at::kHalf: dt = TRACEA_DTYPE_FLOAT16; break;
    case at::kBFloat16: dt = TRACEA_DTYPE_BFLOAT16; break;
    case at::kInt: dt = TRACEA_DTYPE_INT32; break;
    case at::kChar: dt = TRACEA_DTYPE_INT8; break;
    default:
      PyErr_Format(PyExc_TypeError, "unsupported dtype %s", c10::toString(t.scalar_type()));
      throw PyError{};
  }
  const int64_t rank = t.dim();
  if (rank > kMaxRank) {
    PyErr_Format(PyExc_ValueError, "tensors of more than %d dimensions are not supported", kMaxRank);
    throw PyError{};
  }
  for (int64_t d = 0; d < rank; ++d) {
    const int64_t s = order != nullptr ? order[d] : d;
    o.shape[d] = static_cast<uint64_t>(t.size(s));
    o.stride[d] = t.stride(s);
  }
  o.v.ptr = t.data_ptr();
  o.v.rank = static_cast<uint32_t>(rank);
  o.v.shape = o.shape;
  o.v.stride = o.stride;
  o.v.dtype = dt;
  o.v.device_id = t.is_cuda() ? static_cast<int32_t>(t.get_device()) : -1;
}

const at::Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "%s must be a torch.Tensor, not %s", name, Py_TYPE(o)->tp_name);
    throw PyError{};
  }
  return THPVariable_Unpack(o);
}
const at::Tensor* optional_tensor(PyObject* o, const char* name) { return o == Py_None ? nullptr : &tensor_arg(o, name); }

long int_arg(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred() != nullptr) throw PyError{};
  return v;
}

// Raises tracea_b200.ffi.TraceaError(status, last error text, entry).
[[noreturn]] void raise_status(TraceaStatus st, const char* entry) {
  char text[1024];
  const int32_t n = tracea_get_last_error(reinterpret_cast<uint8_t*>(text), sizeof(text));
  PyObject* mod = PyImport_ImportModule("tracea_b200.ffi");
  PyObject* cls = mod != nullptr ? PyObject_GetAttrString(mod, "TraceaError") : nullptr;
  PyObject* msg = cls != nullptr ? PyUnicode_DecodeUTF8(text, n > 0 ? n : 0, "replace") : nullptr;
  PyObject* exc = msg != nullptr ? PyObject_CallFunction(cls, "iOs", static_cast<int>(st), msg, entry) : nullptr;
  if (exc != nullptr) PyErr_SetObject(cls, exc);
  Py_XDECREF(exc);
  Py_XDECREF(msg);
  Py_XDECREF(cls);
  Py_XDECREF(mod);
  throw PyError{};
}

void* stream_of(const at::Tensor& t) {
  return t.is_cuda() ? static_cast<void*>(c10::cuda::getCurrentCUDAStream(t.get_device()).stream()) : nullptr;
}

// The library call itself, without the GIL: it may allocate, and on host tensors it copies and waits.
template <typename F>
TraceaStatus without_gil(F&& f) {
  PyThreadState* save = PyEval_SaveThread();
  const TraceaStatus st = f();
  PyEval_RestoreThread(save);
  return st;
}

const TraceaTensorView* opt(const at::Tensor* t, View& v, const int* order = nullptr) {
  if (t == nullptr) return nullptr;
  fill(v, *t, order);
  return &v.v;
}

constexpr int kChannelsLast[4] = {0, 3, 1, 2};   // logical NCHW of dimensions (N, H, W, C); KCRS of (K, R, S, C)

template <typename Body>
PyObject* guarded(Body&& body) {
  HANDLE_TH_ERRORS
  try {
    return body();
  } catch (const PyError&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

bool arg_count(Py_ssize_t got, Py_ssize_t want, const char* name) {
  if (got == want) return true;
  PyErr_Format(PyExc_TypeError, "%s takes %zd arguments (%zd given)", name, want, got);
  return false;
}

// conv2d(x, w, bias, residual, out, channels-last dimensions, epilogue kind, stride_h, stride_w, pad_h, pad_w, dil_h, dil_w,
// groups) -> out
PyObject* py_conv2d(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arg_count(n, 14, "conv2d")) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor &x = tensor_arg(a[0], "x"), &w = tensor_arg(a[1], "w"), &out = tensor_arg(a[4], "out");
    const at::Tensor *bias = optional_tensor(a[2], "bias"), *res = optional_tensor(a[3], "residual");
    const int* order = PyObject_IsTrue(a[5]) ? kChannelsLast : nullptr;
    if (order != nullptr && (x.dim() != 4 || w.dim() != 4 || out.dim() != 4 || (res != nullptr && res->dim() != 4))) {
      PyErr_SetString(PyExc_ValueError, "x, w, residual and out must have four dimensions");
      throw PyError{};
    }
    TraceaConv2dParams p;
    p.epilogue = static_cast<TraceaEpilogueKind>(int_arg(a[6]));
    p.stride_h = static_cast<uint32_t>(int_arg(a[7]));
    p.stride_w = static_cast<uint32_t>(int_arg(a[8]));
    p.padding_h = static_cast<uint32_t>(int_arg(a[9]));
    p.padding_w = static_cast<uint32_t>(int_arg(a[10]));
    p.dilation_h = static_cast<uint32_t>(int_arg(a[11]));
    p.dilation_w = static_cast<uint32_t>(int_arg(a[12]));
    p.groups = static_cast<uint32_t>(int_arg(a[13]));
    p.stream = stream_of(x);
    View vx, vw, vb, vr, vo;
    fill(vx, x, order);
    fill(vw, w, order);
    const TraceaTensorView* pb = opt(bias, vb);
    const TraceaTensorView* pr = opt(res, vr, order);
    fill(vo, out, order);
    const TraceaStatus st = without_gil([&] { return tracea_conv2d(vx.v, vw.v, pb, pr, &vo.v, p); });
    if (st != TRACEA_SUCCESS) raise_status(st, "tracea_conv2d");
    Py_INCREF(a[4]);
    return a[4];
  });
}

// gemm(x, w, bias, residual, out, epilogue kind) -> out
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arg_count(n, 6, "gemm")) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor &x = tensor_arg(a[0], "x"), &w = tensor_arg(a[1], "w"), &out = tensor_arg(a[4], "out");
    const at::Tensor *bias = optional_tensor(a[2], "bias"), *res = optional_tensor(a[3], "residual");
    TraceaGemmParams p;
    p.epilogue = static_cast<TraceaEpilogueKind>(int_arg(a[5]));
    p.stream = stream_of(x);
    View vx, vw, vb, vr, vo;
    fill(vx, x);
    fill(vw, w);
    const TraceaTensorView* pb = opt(bias, vb);
    const TraceaTensorView* pr = opt(res, vr);
    fill(vo, out);
    const TraceaStatus st = without_gil([&] { return tracea_gemm(vx.v, vw.v, pb, pr, &vo.v, p); });
    if (st != TRACEA_SUCCESS) raise_status(st, "tracea_gemm");
    Py_INCREF(a[4]);
    return a[4];
  });
}

// conv_transpose2d(x, w, bias, residual, out, epilogue kind, stride_h, stride_w, pad_h, pad_w, opad_h, opad_w, dil_h, dil_w)
// -> out
PyObject* py_conv_transpose2d(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (!arg_count(n, 14, "conv_transpose2d")) return nullptr;
  return guarded([&]() -> PyObject* {
    const at::Tensor &x = tensor_arg(a[0], "x"), &w = tensor_arg(a[1], "w"), &out = tensor_arg(a[4], "out");
    const at::Tensor *bias = optional_tensor(a[2], "bias"), *res = optional_tensor(a[3], "residual");
    TraceaConvTranspose2dParams p;
    p.epilogue = static_cast<TraceaEpilogueKind>(int_arg(a[5]));
    p.stride_h = static_cast<uint32_t>(int_arg(a[6]));
    p.stride_w = static_cast<uint32_t>(int_arg(a[7]));
    p.padding_h = static_cast<uint32_t>(int_arg(a[8]));
    p.padding_w = static_cast<uint32_t>(int_arg(a[9]));
    p.output_padding_h = static_cast<uint32_t>(int_arg(a[10]));
    p.output_padding_w = static_cast<uint32_t>(int_arg(a[11]));
    p.dilation_h = static_cast<uint32_t>(int_arg(a[12]));
    p.dilation_w = static_cast<uint32_t>(int_arg(a[13]));
    p.groups = 1;
    p.stream = stream_of(x);
    View vx, vw, vb, vr, vo;
    fill(vx, x);
    fill(vw, w);
    const TraceaTensorView* pb = opt(bias, vb);
    const TraceaTensorView* pr = opt(res, vr);
    fill(vo, out);
    const TraceaStatus st = without_gil([&] { return tracea_conv_transpose2d(vx.v, vw.v, pb, pr, &vo.v, p); });
    if (st != TRACEA_SUCCESS) raise_status(st, "tracea_conv_transpose2d");
    Py_INCREF(a[4]);
    return a[4];
  });
}

PyMethodDef kMethods[] = {
    {"conv2d", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_conv2d)), METH_FASTCALL, nullptr},
    {"gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_gemm)), METH_FASTCALL, nullptr},
    {"conv_transpose2d", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_conv_transpose2d)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_ops_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__ops_native() {
  PyObject* m = PyModule_Create(&kModule);
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) {   // what it was compiled against
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
