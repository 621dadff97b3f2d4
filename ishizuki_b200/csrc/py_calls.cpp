// The per-call half of the Python interface: one C function per entry point that a decode loop
// calls, from the tensors it is handed to the C ABI and back to a tensor.
//
// What bounds a call on a small matrix is the host: over ctypes a product cost 17 us (the current
// stream's Python object 3.6, the output tensor 2.4, reshaping and pointer objects 2, argument
// conversion 1.4, the kernel launch itself 2.2) around a kernel of 5. Here the same steps are C++
// on the tensor's own fields: the launch is more than half of what is left.
//
// Everything else (creating projections, files, groups) stays on ctypes in interface.py.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/ishizuki_cuda.h"

namespace {

PyObject *g_error = nullptr;  // interface.IshizukiError

void *handle_of(PyObject *o) { return PyLong_AsVoidPtr(o); }
void *stream_of(const at::Tensor &t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

PyObject *raise(ishi_status s, const ishi_ctx *ctx) {
  PyObject *e = PyObject_CallFunction(g_error, "is", (int)s, ishi_last_error(ctx));
  if (e) {
    PyErr_SetObject(g_error, e);
    Py_DECREF(e);
  }
  return nullptr;
}

// the C call without the interpreter lock: a launch may wait for room in the stream's queue
template <class F>
ishi_status unlocked(F &&f) {
  PyThreadState *save = PyEval_SaveThread();
  const ishi_status s = f();
  PyEval_RestoreThread(save);
  return s;
}

at::Tensor new_tensor(at::IntArrayRef shape, at::ScalarType type, const at::Tensor &like) {
  return at::detail::empty_cuda(shape, type, like.device(), std::nullopt);
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return ISHI_DT_F16;
    case at::kBFloat16: return ISHI_DT_BF16;
    case at::kFloat: return ISHI_DT_F32;
    default: return -1;
  }
}

// a torch dtype the decoders write
bool output_type(PyObject *o, at::ScalarType *t) {
  if (THPDtype_Check(o) && dtype_code(*t = reinterpret_cast<THPDtype *>(o)->scalar_type) >= 0) return true;
  PyErr_SetObject(PyExc_KeyError, o);
  return false;
}

bool arity(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, got);
  return got == want;
}

bool is_tensor(PyObject *o) {
  if (THPVariable_Check(o)) return true;
  PyErr_SetString(PyExc_TypeError, "a torch tensor is expected");
  return false;
}

// [rows, width] of a tensor whose last axis is the width, contiguous
struct Rows {
  at::Tensor t;
  int64_t rows = 0, width = 0;
  explicit Rows(const at::Tensor &x) : t(x.is_contiguous() ? x : x.contiguous()) {
    width = x.size(-1);
    rows = width > 0 ? x.numel() / width : 0;
  }
};

at::DimVector with_width(const at::Tensor &x, int64_t width) {
  at::DimVector shape(x.sizes().begin(), x.sizes().end());
  shape.back() = width;
  return shape;
}

bool half_rows(const at::Tensor &x) {
  if (x.scalar_type() == at::kHalf && x.is_cuda() && x.dim() > 0) return true;
  PyErr_SetString(PyExc_TypeError, "activations must be fp16 CUDA tensors");
  return false;
}

// linear(ctx, projection, x, output width, route, crossover, rotated, transposed, out or None)
PyObject *linear(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 9) || !is_tensor(a[2])) return nullptr;
  auto *ctx = static_cast<ishi_ctx *>(handle_of(a[0]));
  auto *p = static_cast<ishi_projection *>(handle_of(a[1]));
  const at::Tensor &x = THPVariable_Unpack(a[2]);
  if (!half_rows(x)) return nullptr;
  const int64_t width = PyLong_AsLongLong(a[3]);
  const int route = (int)PyLong_AsLong(a[4]), crossover = (int)PyLong_AsLong(a[5]);
  const int rotated = PyObject_IsTrue(a[6]), transposed = PyObject_IsTrue(a[7]);
  if (PyErr_Occurred()) return nullptr;
  ishi_status s = ishi_ctx_set_route(ctx, route, crossover);
  if (s != ISHI_OK) return raise(s, ctx);
  const Rows h(x);
  at::Tensor y;
  if (a[8] != Py_None) {
    if (!is_tensor(a[8])) return nullptr;
    y = THPVariable_Unpack(a[8]);
  } else if (transposed) {
    y = new_tensor({width, h.rows}, at::kHalf, x);
  } else {
    y = new_tensor(with_width(x, width), at::kHalf, x);
  }
  const int64_t ldy = a[8] != Py_None ? y.stride(0) : transposed ? h.rows : width;
  const void *xp = h.t.data_ptr();
  void *yp = y.data_ptr(), *st = stream_of(x);
  s = unlocked([&] {
    return rotated ? ishi_projection_apply_rotated(p, xp, (int)h.rows, yp, ldy, 0, st)
                   : ishi_projection_apply(p, xp, (int)h.rows, yp, ldy, transposed ? ISHI_OUT_TRANSPOSED : 0, st);
  });
  if (s != ISHI_OK) return raise(s, ctx);
  if (a[8] != Py_None) return Py_NewRef(a[8]);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// argmax(ctx, projection, x, route, crossover)
PyObject *argmax(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 5) || !is_tensor(a[2])) return nullptr;
  auto *ctx = static_cast<ishi_ctx *>(handle_of(a[0]));
  auto *p = static_cast<ishi_projection *>(handle_of(a[1]));
  const at::Tensor &x = THPVariable_Unpack(a[2]);
  if (!half_rows(x)) return nullptr;
  const int route = (int)PyLong_AsLong(a[3]), crossover = (int)PyLong_AsLong(a[4]);
  if (PyErr_Occurred()) return nullptr;
  ishi_status s = ishi_ctx_set_route(ctx, route, crossover);
  if (s != ISHI_OK) return raise(s, ctx);
  const Rows h(x);
  at::Tensor out = new_tensor({h.rows}, at::kInt, x);
  s = unlocked([&] { return ishi_projection_apply_argmax(p, h.t.data_ptr(), (int)h.rows, static_cast<int32_t *>(out.data_ptr()), stream_of(x)); });
  if (s != ISHI_OK) return raise(s, ctx);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// rms_norm(ctx, x, weight, eps)
PyObject *rms_norm(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 4) || !is_tensor(a[1]) || !is_tensor(a[2])) return nullptr;
  auto *ctx = static_cast<ishi_ctx *>(handle_of(a[0]));
  const at::Tensor &x = THPVariable_Unpack(a[1]);
  const at::Tensor w = THPVariable_Unpack(a[2]).contiguous();
  const float eps = (float)PyFloat_AsDouble(a[3]);
  if (PyErr_Occurred()) return nullptr;
  const int xd = dtype_code(x.scalar_type()), wd = dtype_code(w.scalar_type());
  if (xd < 0 || wd < 0) {
    PyErr_SetString(PyExc_KeyError, "fp16, bf16 and fp32 tensors are taken");
    return nullptr;
  }
  const Rows h(x);
  at::Tensor y = new_tensor(x.sizes(), at::kHalf, x);
  const ishi_status s = unlocked([&] {
    return ishi_rms_norm(ctx, h.t.data_ptr(), xd, h.rows, h.width, w.data_ptr(), wd, eps, y.data_ptr(), stream_of(x));
  });
  if (s != ISHI_OK) return raise(s, ctx);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// gather(ctx, ids, blocks, type, bytes of a row, input width, dtype): None when declined
PyObject *gather(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 7) || !is_tensor(a[1]) || !is_tensor(a[2])) return nullptr;
  auto *ctx = static_cast<ishi_ctx *>(handle_of(a[0]));
  at::Tensor ids = THPVariable_Unpack(a[1]);
  const at::Tensor &blocks = THPVariable_Unpack(a[2]);
  const int type = (int)PyLong_AsLong(a[3]);
  const int64_t per_row = PyLong_AsLongLong(a[4]), width = PyLong_AsLongLong(a[5]);
  if (PyErr_Occurred()) return nullptr;
  if (per_row == 0) {  // an input width of 0: the division below would end the process
    PyErr_SetString(PyExc_ZeroDivisionError, "a table row of no bytes");
    return nullptr;
  }
  at::ScalarType st;
  if (!output_type(a[6], &st)) return nullptr;
  ids = ids.to(at::kInt).contiguous();
  at::Tensor out = new_tensor({ids.numel(), width}, st, blocks);
  const ishi_status s = unlocked([&] {
    return ishi_ggml_gather(ctx, static_cast<const int32_t *>(ids.data_ptr()), ids.numel(), blocks.data_ptr(), blocks.numel(), type,
                            blocks.numel() / per_row, width, out.data_ptr(), dtype_code(st), stream_of(blocks));
  });
  if (s == ISHI_E_SHAPE || s == ISHI_E_UNSUPPORTED) Py_RETURN_NONE;
  if (s != ISHI_OK) return raise(s, ctx);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// dequantize(ctx, blocks, type, blocks' count, shape, dtype): None when declined
PyObject *dequantize(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 6) || !is_tensor(a[1])) return nullptr;
  auto *ctx = static_cast<ishi_ctx *>(handle_of(a[0]));
  const at::Tensor &blocks = THPVariable_Unpack(a[1]);
  const int type = (int)PyLong_AsLong(a[2]);
  const int64_t count = PyLong_AsLongLong(a[3]);
  at::DimVector shape;
  PyObject *dims = PySequence_Fast(a[4], "a shape is expected");
  if (!dims) return nullptr;
  for (Py_ssize_t i = 0; i < PySequence_Fast_GET_SIZE(dims); ++i) shape.push_back(PyLong_AsLongLong(PySequence_Fast_GET_ITEM(dims, i)));
  Py_DECREF(dims);
  if (PyErr_Occurred()) return nullptr;
  at::ScalarType st;
  if (!output_type(a[5], &st)) return nullptr;
  at::Tensor out = new_tensor(shape, st, blocks);
  const ishi_status s = unlocked([&] {
    return ishi_ggml_dequantize(ctx, type, blocks.data_ptr(), count, out.data_ptr(), dtype_code(st), stream_of(blocks));
  });
  if (s == ISHI_E_SHAPE || s == ISHI_E_UNSUPPORTED) Py_RETURN_NONE;
  if (s != ISHI_OK) return raise(s, ctx);
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// exl3_apply(ctx, trellis, input scales, output scales, codebook, x)
PyObject *exl3_apply(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arity(n, 6) || !is_tensor(a[1]) || !is_tensor(a[5])) return nullptr;
  auto *ctx = static_cast<ishi_ctx *>(handle_of(a[0]));
  const at::Tensor &trellis = THPVariable_Unpack(a[1]);
  ishi_exl3_desc d;
  d.trellis_dev = static_cast<const int16_t *>(trellis.data_ptr());
  d.k = trellis.size(0) * 16;
  d.n = trellis.size(1) * 16;
  d.words_per_tile = (int32_t)trellis.size(2);
  d.codebook = (int32_t)PyLong_AsLong(a[4]);
  d.input_scales_dev = a[2] == Py_None ? nullptr : THPVariable_Unpack(a[2]).data_ptr();
  d.output_scales_dev = a[3] == Py_None ? nullptr : THPVariable_Unpack(a[3]).data_ptr();
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor &x = THPVariable_Unpack(a[5]);
  if (x.dim() == 0 || x.size(-1) != d.k) {
    PyErr_Format(PyExc_RuntimeError, "activations of width %lld against an EXL3 weight of input width %lld",
                 x.dim() ? (long long)x.size(-1) : 0ll, (long long)d.k);
    return nullptr;
  }
  const Rows h(x.scalar_type() == at::kHalf ? x : x.to(at::kHalf));
  at::Tensor y = new_tensor(with_width(x, d.n), at::kHalf, x);
  const ishi_status s = unlocked([&] { return ishi_exl3_apply(ctx, &d, h.t.data_ptr(), (int)h.rows, y.data_ptr(), stream_of(x)); });
  if (s != ISHI_OK) return raise(s, ctx);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// device_of(tensor): its device's index, without the Python device object
PyObject *device_of(PyObject *, PyObject *t) {
  if (!is_tensor(t)) return nullptr;
  return PyLong_FromLong(THPVariable_Unpack(t).device().index());
}

// current_stream(device): the raw stream the device's work goes to
PyObject *current_stream(PyObject *, PyObject *device) {
  HANDLE_TH_ERRORS
  const long d = PyLong_AsLong(device);
  if (PyErr_Occurred()) return nullptr;
  return PyLong_FromVoidPtr(c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)d).stream());
  END_HANDLE_TH_ERRORS
}

// set_error(class): what a failing status is raised as, class(status, message)
PyObject *set_error(PyObject *, PyObject *cls) {
  Py_XSETREF(g_error, Py_NewRef(cls));
  Py_RETURN_NONE;
}

#define ISHI_FAST(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(name)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {ISHI_FAST(linear),
                          ISHI_FAST(argmax),
                          ISHI_FAST(rms_norm),
                          ISHI_FAST(gather),
                          ISHI_FAST(dequantize),
                          ISHI_FAST(exl3_apply),
                          {"device_of", device_of, METH_O, nullptr},
                          {"current_stream", current_stream, METH_O, nullptr},
                          {"set_error", set_error, METH_O, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() { return PyModule_Create(&kModule); }
