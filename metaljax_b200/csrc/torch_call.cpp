// The product's call from Python, natively: torch tensors in, one call of the C ABI, the result
// tensor out. A decode-sized product runs for a few microseconds on the device, and five DLPack
// capsules, their ctypes conversions and a tensor allocation through Python took 25 of them per call
// on the host (one row of 4096x4096: 25.0 us a call before, 5.4 us now, the kernel's own time); here the views are read from the tensors' own sizes and strides. Everything is
// validated where it was: by the C ABI. What is not an ordinary CUDA tensor (a subclass, a tensor
// that requires a gradient, an empty one, host memory) is declined -- None -- and takes the ctypes way, whose
// errors it keeps.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/qmm.h"

namespace {

typedef int (*QuantizedMatmul)(const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, qmm_tensor*, int,
                               int, int, int, void*);

// Entry points of the library that is loaded (ctypes hands their addresses over: one library per
// process, whichever file it was loaded from).
QuantizedMatmul g_quantized_matmul = nullptr;

bool dtype_of(at::ScalarType t, qmm_dtype* d) {
  d->lanes = 1;
  switch (t) {
    case at::kBFloat16: d->code = 4; d->bits = 16; return true;
    case at::kHalf: d->code = 2; d->bits = 16; return true;
    case at::kFloat: d->code = 2; d->bits = 32; return true;
    case at::kByte: d->code = 1; d->bits = 8; return true;
    case at::kUInt32: d->code = 1; d->bits = 32; return true;
    case at::kInt: d->code = 0; d->bits = 32; return true;
    default: return false;
  }
}

// The tensor behind a Python object, or NULL where the ctypes way has to decide.
const at::Tensor* plain_tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || t.requires_grad() || t.is_neg() || t.is_conj() || t.numel() == 0)
    return nullptr;
  return &t;
}

bool view_of(const at::Tensor& t, qmm_tensor* v) {
  if (!dtype_of(t.scalar_type(), &v->dtype)) return false;
  v->data = const_cast<void*>(t.const_data_ptr());
  v->device = {2, static_cast<int32_t>(t.get_device())};
  v->ndim = static_cast<int32_t>(t.dim());
  v->shape = const_cast<int64_t*>(t.sizes().data());
  v->strides = const_cast<int64_t*>(t.strides().data());
  v->byte_offset = 0;
  return true;
}

// The packed words: uint32, or int32 of the same bits.
bool words_of(const at::Tensor& t, qmm_tensor* v) {
  if (!view_of(t, v)) return false;
  if (t.scalar_type() == at::kInt) v->dtype.code = 1;
  return v->dtype.code == 1 && v->dtype.bits == 32;
}

// quantized_matmul(x, w, scales, biases | None, transpose, group_size, bits, mode, out | None, dtype | None)
// -> the result, a status code, or None (declined)
PyObject* quantized_matmul(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 10 || !g_quantized_matmul) Py_RETURN_NONE;
  const at::Tensor *x = plain_tensor(a[0]), *w = plain_tensor(a[1]), *s = plain_tensor(a[2]);
  const at::Tensor* b = a[3] == Py_None ? nullptr : plain_tensor(a[3]);
  if (!x || !w || !s || (!b && a[3] != Py_None) || x->dim() < 2 || w->dim() < 2) Py_RETURN_NONE;
  const int transpose = PyObject_IsTrue(a[4]);
  const long gs = PyLong_AsLong(a[5]), bits = PyLong_AsLong(a[6]), mode = PyLong_AsLong(a[7]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const int64_t lead = x->dim() - 2, m = x->size(-2), k = x->size(-1), cols = w->size(-2);
  at::Tensor y, xc;
  try {
    if (a[8] != Py_None) {
      const at::Tensor* out = plain_tensor(a[8]);
      if (!out || !out->is_contiguous() || out->dim() != x->dim() || out->size(-1) != cols || out->size(-2) != m) Py_RETURN_NONE;
      for (int64_t d = 0; d < lead; ++d)
        if (out->size(d) != x->size(d)) Py_RETURN_NONE;
      y = *out;
    } else {
      at::ScalarType dt = x->scalar_type();
      if (a[9] != Py_None) {
        if (!THPDtype_Check(a[9])) Py_RETURN_NONE;
        dt = reinterpret_cast<THPDtype*>(a[9])->scalar_type;
      }
      c10::SmallVector<int64_t, 5> shape(x->sizes().begin(), x->sizes().end());
      shape[lead + 1] = cols;
      y = at::detail::empty_cuda(shape, dt, x->device(), std::nullopt);
    }
    xc = x->is_contiguous() ? *x : x->contiguous();
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
  qmm_tensor vx, vw, vs, vb, vy;
  if (!view_of(xc, &vx) || !words_of(*w, &vw) || !view_of(*s, &vs) || (b && !view_of(*b, &vb)) || !view_of(y, &vy)) Py_RETURN_NONE;
  int64_t xs[3], ys[3];
  if (lead > 0) {                          // one weight per batch of x, or a shared one: then the batches are more rows
    const int64_t batches = x->numel() / (m * k);
    const bool shared = w->dim() != 3;
    vx.ndim = vy.ndim = shared ? 2 : 3;
    xs[0] = ys[0] = shared ? batches * m : batches;
    xs[1] = shared ? k : m;
    ys[1] = shared ? cols : m;
    xs[2] = k;
    ys[2] = cols;
    vx.shape = xs;
    vy.shape = ys;
    vx.strides = vy.strides = nullptr;
  }
  const int rc = g_quantized_matmul(&vx, &vw, &vs, b ? &vb : nullptr, &vy, transpose, static_cast<int>(gs), static_cast<int>(bits),
                                    static_cast<int>(mode), c10::cuda::getCurrentCUDAStream(x->get_device()).stream());
  if (rc) return PyLong_FromLong(rc);
  if (a[8] != Py_None) {
    Py_INCREF(a[8]);
    return a[8];
  }
  return THPVariable_Wrap(std::move(y));
}

// bind(address of qmm_quantized_matmul)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 1) {
    PyErr_SetString(PyExc_TypeError, "bind takes the entry points' addresses");
    return nullptr;
  }
  g_quantized_matmul = reinterpret_cast<QuantizedMatmul>(PyLong_AsVoidPtr(a[0]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(bind)), METH_FASTCALL, nullptr},
    {"quantized_matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(quantized_matmul)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
