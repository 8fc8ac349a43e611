// The product's call from Python, natively: torch tensors in, one call of the C ABI, the result
// tensor out. A decode-sized product runs for a few microseconds on the device, and five DLPack
// capsules, their ctypes conversions and a tensor allocation through Python took 25 of them per call
// on the host (one row of 4096x4096: 25.0 us a call before, 5.4 us now, the kernel's own time); here the views are read from the tensors' own sizes and strides. Everything is
// validated where it was: by the C ABI. What is not an ordinary CUDA tensor (a subclass, a tensor
// that requires a gradient, an empty one, host memory) is declined -- None -- and takes the ctypes way, whose
// errors it keeps. So is a call in which torch throws (a tensor without storage inside vmap, memory that runs out): no C++
// exception leaves an entry, and the ctypes way meets the same cause and raises it as torch's own error.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <vector>

#include "../../include/qmm.h"

namespace {

typedef int (*QuantizedMatmul)(const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, qmm_tensor*, int,
                               int, int, int, void*);

typedef int (*SiluMul)(const void*, const void*, void*, int64_t, int, void*);
typedef int (*GatedMatmul)(const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, const qmm_tensor*, qmm_tensor*, int, int, int,
                           void*);
typedef int (*GatedPays)(const qmm_problem*);
typedef int (*PackLayer)(const void*, uint32_t*, const void*, const void*, int, int, void*, void*, int, int64_t, int64_t, int64_t, int, uint64_t*, uint32_t*, void*);
typedef int64_t (*MoeWorkspace)(const qmm_moe_block*);
typedef int (*MoeExperts)(const qmm_moe_block*, void*);

// Entry points of the library that is loaded (ctypes hands their addresses over: one library per
// process, whichever file it was loaded from).
QuantizedMatmul g_quantized_matmul = nullptr;
SiluMul g_silu_mul = nullptr;
GatedMatmul g_gated_matmul = nullptr;
GatedPays g_gated_pays = nullptr;
PackLayer g_pack_layer = nullptr;
MoeWorkspace g_moe_workspace = nullptr;
MoeExperts g_moe_experts = nullptr;

constexpr int kDeclined = -1;         // (the library's codes are not negative)

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

// Runs f without the interpreter's lock, as ctypes and torch's own bindings do: a full launch queue makes an enqueue wait for the
// device, which may be waiting for another thread of Python (a host callback in the stream), and a copy or an allocation may wait too.
// What f throws is thrown again with the lock held.
template <typename F>
auto unlocked(F&& f) -> decltype(f()) {
  PyThreadState* state = PyEval_SaveThread();
  try {
    auto result = f();
    PyEval_RestoreThread(state);
    return result;
  } catch (const std::exception&) {
    PyEval_RestoreThread(state);
    throw;
  }
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
  at::Tensor y;
  at::ScalarType dt = x->scalar_type();
  if (a[8] != Py_None) {
    const at::Tensor* out = plain_tensor(a[8]);
    if (!out || !out->is_contiguous() || out->dim() != x->dim() || out->size(-1) != cols || out->size(-2) != m) Py_RETURN_NONE;
    for (int64_t d = 0; d < lead; ++d)
      if (out->size(d) != x->size(d)) Py_RETURN_NONE;
    y = *out;
  } else if (a[9] != Py_None) {
    if (!THPDtype_Check(a[9])) Py_RETURN_NONE;
    dt = reinterpret_cast<THPDtype*>(a[9])->scalar_type;
  }
  const int rc = unlocked([&]() -> int {
    if (!y.defined()) {
      c10::SmallVector<int64_t, 5> shape(x->sizes().begin(), x->sizes().end());
      shape[lead + 1] = cols;
      y = at::detail::empty_cuda(shape, dt, x->device(), std::nullopt);
    }
    const at::Tensor xc = x->is_contiguous() ? *x : x->contiguous();
    qmm_tensor vx, vw, vs, vb, vy;
    if (!view_of(xc, &vx) || !words_of(*w, &vw) || !view_of(*s, &vs) || (b && !view_of(*b, &vb)) || !view_of(y, &vy)) return kDeclined;
    int64_t xs[3], ys[3];
    if (lead > 0) {                        // one weight per batch of x, or a shared one: then the batches are more rows
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
    return g_quantized_matmul(&vx, &vw, &vs, b ? &vb : nullptr, &vy, transpose, static_cast<int>(gs), static_cast<int>(bits),
                              static_cast<int>(mode), c10::cuda::getCurrentCUDAStream(x->get_device()).stream());
  });
  if (rc == kDeclined) Py_RETURN_NONE;
  if (rc) return PyLong_FromLong(rc);
  if (a[8] != Py_None) {
    Py_INCREF(a[8]);
    return a[8];
  }
  return THPVariable_Wrap(std::move(y));
}

int elem_of(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return QMM_BF16;
    case at::kHalf: return QMM_F16;
    case at::kFloat: return QMM_F32;
    case at::kByte: return QMM_U8;
    default: return -1;
  }
}

// moe_experts(x, indices, weights, (w, scales, biases | None) x 3: gate, up, down, group_size, bits, mode)
// -> the result, a status code, or None (declined: what is not the plain block takes the step by step way)
PyObject* moe_experts(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 15 || !g_moe_experts) Py_RETURN_NONE;
  const at::Tensor *x = plain_tensor(a[0]), *idx = plain_tensor(a[1]), *wts = plain_tensor(a[2]);
  if (!x || !idx || !wts || x->dim() != 2 || idx->dim() != 2 || !x->is_contiguous() || !idx->is_contiguous()) Py_RETURN_NONE;
  if (reinterpret_cast<uintptr_t>(x->const_data_ptr()) % 16) Py_RETURN_NONE;      // (the steps gather its rows into memory of their own)
  const long gs = PyLong_AsLong(a[12]), bits = PyLong_AsLong(a[13]), mode = PyLong_AsLong(a[14]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if ((bits != 4 && bits != 8) || gs < 32 || wts->numel() != idx->numel() || idx->size(0) != x->size(0)) Py_RETURN_NONE;
  qmm_moe_block b = {};
  b.struct_size = sizeof(b);
  b.mode = static_cast<int32_t>(mode); b.bits = static_cast<int32_t>(bits); b.group_size = static_cast<int32_t>(gs);
  b.x_dtype = elem_of(x->scalar_type());
  if (b.x_dtype != QMM_BF16 && b.x_dtype != QMM_F16) Py_RETURN_NONE;
  if (idx->scalar_type() != at::kLong && idx->scalar_type() != at::kInt) Py_RETURN_NONE;
  b.index_bytes = idx->scalar_type() == at::kLong ? 8 : 4;
  b.tokens = x->size(0); b.d = x->size(1); b.k = static_cast<int32_t>(idx->size(1));
  qmm_moe_weight* ws[3] = {&b.w1, &b.w3, &b.w2};
  for (int i = 0; i < 3; ++i) {
    const at::Tensor *w = plain_tensor(a[3 + 3 * i]), *s = plain_tensor(a[4 + 3 * i]);
    const at::Tensor* z = a[5 + 3 * i] == Py_None ? nullptr : plain_tensor(a[5 + 3 * i]);
    if (!w || !s || (!z && a[5 + 3 * i] != Py_None) || w->dim() != 3 || s->dim() != 3 || !w->is_contiguous() || !s->is_contiguous() || (z && !z->is_contiguous()))
      Py_RETURN_NONE;
    if ((w->scalar_type() != at::kUInt32 && w->scalar_type() != at::kInt) || w->device() != x->device() || s->device() != x->device()) Py_RETURN_NONE;
    if (i == 0) {
      b.experts = static_cast<int32_t>(w->size(0));
      b.ffn = w->size(1);
      b.table_dtype = elem_of(s->scalar_type());
    }
    const int64_t rows = i < 2 ? b.ffn : b.d, k = i < 2 ? b.d : b.ffn;
    if (w->size(0) != b.experts || w->size(1) != rows || w->size(2) * 32 != k * bits || k % gs || s->size(0) != b.experts || s->size(1) != rows || s->size(2) != k / gs ||
        elem_of(s->scalar_type()) != b.table_dtype || (z && (z->sizes() != s->sizes() || z->scalar_type() != s->scalar_type() || z->device() != x->device())))
      Py_RETURN_NONE;
    *ws[i] = {w->const_data_ptr(), s->const_data_ptr(), z ? z->const_data_ptr() : nullptr};
  }
  if (idx->device() != x->device() || wts->device() != x->device()) Py_RETURN_NONE;
  const int64_t need = g_moe_workspace(&b);
  if (need < 0) Py_RETURN_NONE;
  at::Tensor y;
  const int rc = unlocked([&]() -> int {
    const at::Tensor w32 = wts->scalar_type() == at::kFloat && wts->is_contiguous() ? *wts : wts->to(at::kFloat).contiguous();
    y = at::detail::empty_cuda({b.tokens, b.d}, x->scalar_type(), x->device(), std::nullopt);
    const at::Tensor work = at::detail::empty_cuda({need}, at::kByte, x->device(), std::nullopt);
    b.x = x->const_data_ptr(); b.indices = idx->const_data_ptr(); b.weights = w32.const_data_ptr<float>();
    b.out = y.data_ptr(); b.workspace = work.data_ptr(); b.workspace_bytes = need;
    return g_moe_experts(&b, c10::cuda::getCurrentCUDAStream(x->get_device()).stream());
  });
  if (rc) return PyLong_FromLong(rc);
  return THPVariable_Wrap(std::move(y));
}

// A stored int4 Dense layer with consecutive groups (qmm._pack_dense): pack_layer(packed, scale, zero | None, K, N, wide, source)
// -> (words, scales, biases, digest, flags, group size, whether the tables are the scales' type), a status code, or None (declined). The tables are made
// before what they hold is known, as nearly every layer's are: one entry per stored group (the widest group size that divides it), biases in float32
// where there are zero points (a product of a scale and an integer seldom fits the scale's type; 8 times the scale does). `wide`, `source`: the tables' type is
// float32, or the scales', whatever they hold.
PyObject* pack_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 7 || !g_pack_layer) Py_RETURN_NONE;
  const at::Tensor *packed = plain_tensor(a[0]), *scale = plain_tensor(a[1]);
  const at::Tensor* zero = a[2] == Py_None ? nullptr : plain_tensor(a[2]);
  const int64_t k = PyLong_AsLongLong(a[3]), cols = PyLong_AsLongLong(a[4]);
  const int wide = PyObject_IsTrue(a[5]), source = PyObject_IsTrue(a[6]);
  if (PyErr_Occurred()) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (!packed || !scale || (!zero && a[2] != Py_None)) Py_RETURN_NONE;
  for (const at::Tensor* t : {packed, scale, zero ? zero : scale})
    if (t->dim() != 2 || !t->is_contiguous() || t->device() != packed->device()) Py_RETURN_NONE;
  const int64_t g = scale->size(0);
  if (packed->scalar_type() != at::kChar || packed->size(0) != k || packed->size(1) != (cols + 1) / 2 || scale->size(1) != cols || (zero && zero->sizes() != scale->sizes())) Py_RETURN_NONE;
  if (k >= (1LL << 24) || cols >= (1LL << 30) || k % g || k / g % 32) Py_RETURN_NONE;
  const at::ScalarType st = scale->scalar_type(), zt = zero ? zero->scalar_type() : at::kByte;
  const int scale_type = elem_of(st), zero_type = zt == at::kChar ? QMM_I8 : elem_of(zt);
  if (scale_type < 0 || st == at::kByte || zero_type < 0) Py_RETURN_NONE;
  const int64_t stored = k / g;
  const int group = stored % 128 == 0 ? 128 : stored % 64 == 0 ? 64 : 32;
  const int narrow = st != at::kFloat && !wide && (!zero || source);
  at::Tensor words, scales, biases;
  uint64_t digest = 0;
  uint32_t flags = 0;
  const int rc = unlocked([&]() -> int {
    const c10::cuda::CUDAGuard on(packed->device());
    const at::ScalarType table = narrow ? st : at::kFloat;
    words = at::detail::empty_cuda({cols, k / 8}, at::kUInt32, packed->device(), std::nullopt);
    scales = at::detail::empty_cuda({cols, k / group}, table, packed->device(), std::nullopt);
    biases = at::detail::empty_cuda({cols, k / group}, table, packed->device(), std::nullopt);
    return g_pack_layer(packed->const_data_ptr(), static_cast<uint32_t*>(words.data_ptr()), scale->const_data_ptr(), zero ? zero->const_data_ptr() : nullptr, scale_type,
                        zero ? zero_type : 0, scales.data_ptr(), biases.data_ptr(), narrow, g, cols, k, group, &digest, &flags,
                        c10::cuda::getCurrentCUDAStream(packed->get_device()).stream());
  });
  if (rc) return PyLong_FromLong(rc);
  return Py_BuildValue("(NNNKIiO)", THPVariable_Wrap(std::move(words)), THPVariable_Wrap(std::move(scales)), THPVariable_Wrap(std::move(biases)),
                       static_cast<unsigned long long>(digest), static_cast<unsigned int>(flags), group, narrow ? Py_True : Py_False);
}

// What is left of a program when all of it is products of two-dimensional activations and gates between them:
// run_steps(arguments, steps, returns, values): the program's values are numbered, its arguments first; `returns` are numbers; a step is
//   (x, result, w, scales, biases | None, group_size, bits, mode, dtype)    result = x . deq(w)^T as dtype
//   (gate, result, up)                                                      result = silu(gate) * up
// -> the list of the returned values, a status code, or None (declined: nothing has been launched unless torch threw). Everything is looked at before the
// first launch. A feed-forward of three products (4 rows, 2048 x 5632) took 42 us a call through a Python call each (products 6.1, the gate 8.5), 25 in one, and 17.5 with
// its gate and the two products before it as one launch; its kernels take 10.
struct Step {
  int x, result, up;                   // up < 0: a product
  const at::Tensor *w, *scales, *biases;
  int group_size, bits, mode;
  at::ScalarType dtype;
  int gate_from, up_from;              // a gate whose two products nothing else reads: their steps, left for it to make (else < 0)
  bool left;                           // a product that is left for its gate
};

PyObject* run_steps(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4 || !g_quantized_matmul || !g_silu_mul || !PyList_CheckExact(a[0]) || !PyList_CheckExact(a[1]) || !PyList_CheckExact(a[2])) Py_RETURN_NONE;
  const Py_ssize_t nargs = PyList_GET_SIZE(a[0]), nsteps = PyList_GET_SIZE(a[1]), nret = PyList_GET_SIZE(a[2]);
  const long count = PyLong_AsLong(a[3]);
  if (count < nargs || count > nargs + nsteps) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  // (shapes are known beforehand: x is [M, K] and a product [M, N])
  std::vector<const at::Tensor*> given(count, nullptr);
  std::vector<std::array<int64_t, 2>> shapes(count);
  std::vector<at::ScalarType> types(count);
  std::vector<char> known(count, 0);
  std::vector<Step> steps(nsteps);
  int device = -1;
  auto argument = [&](int i) -> bool {             // a value that a step reads
    if (i < 0 || i >= count) return false;
    if (known[i]) return true;
    if (i >= nargs) return false;
    const at::Tensor* t = plain_tensor(PyList_GET_ITEM(a[0], i));
    if (!t || t->dim() != 2 || !t->is_contiguous() || (device >= 0 && t->get_device() != device)) return false;
    given[i] = t;
    device = static_cast<int>(t->get_device());
    shapes[i] = {t->size(0), t->size(1)};
    types[i] = t->scalar_type();
    return known[i] = 1;
  };
  for (Py_ssize_t i = 0; i < nsteps; ++i) {
    PyObject* tuple = PyList_GET_ITEM(a[1], i);
    if (!PyTuple_CheckExact(tuple)) Py_RETURN_NONE;
    const Py_ssize_t size = PyTuple_GET_SIZE(tuple);
    if (size != 3 && size != 9) Py_RETURN_NONE;
    auto number = [&](int at) -> long { return PyLong_AsLong(PyTuple_GET_ITEM(tuple, at)); };
    Step& s = steps[i];
    s.x = static_cast<int>(number(0));
    s.result = static_cast<int>(number(1));
    s.up = s.gate_from = s.up_from = -1;
    s.left = false;
    bool fine = argument(s.x) && s.result >= nargs && s.result < count && !known[s.result];
    if (fine && size == 3) {
      s.up = static_cast<int>(number(2));
      fine = argument(s.up) && shapes[s.up] == shapes[s.x] && types[s.up] == types[s.x] && (types[s.x] == at::kBFloat16 || types[s.x] == at::kHalf) &&
             shapes[s.x][0] * shapes[s.x][1] % 8 == 0;
      for (int v : {s.x, s.up}) fine = fine && (!given[v] || reinterpret_cast<uintptr_t>(given[v]->const_data_ptr()) % 16 == 0);
      if (fine) {
        shapes[s.result] = shapes[s.x];
        types[s.result] = types[s.x];
      }
    } else if (fine) {
      s.w = plain_tensor(PyTuple_GET_ITEM(tuple, 2));
      s.scales = plain_tensor(PyTuple_GET_ITEM(tuple, 3));
      PyObject* b = PyTuple_GET_ITEM(tuple, 4);
      s.biases = b == Py_None ? nullptr : plain_tensor(b);
      s.group_size = static_cast<int>(number(5));
      s.bits = static_cast<int>(number(6));
      s.mode = static_cast<int>(number(7));
      PyObject* dtype = PyTuple_GET_ITEM(tuple, 8);
      fine = s.w && s.scales && (s.biases || b == Py_None) && s.w->dim() == 2 && s.w->get_device() == device && THPDtype_Check(dtype);
      if (fine) {
        s.dtype = reinterpret_cast<THPDtype*>(dtype)->scalar_type;
        shapes[s.result] = {shapes[s.x][0], s.w->size(0)};
        types[s.result] = s.dtype;
      }
    }
    if (PyErr_Occurred()) PyErr_Clear(), fine = false;
    if (!fine) Py_RETURN_NONE;
    known[s.result] = 1;
  }
  std::vector<int> returns(nret);
  for (Py_ssize_t i = 0; i < nret; ++i) {
    const long v = PyLong_AsLong(PyList_GET_ITEM(a[2], i));
    if (v < 0 || v >= count || (v >= nargs && !known[v])) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    returns[i] = static_cast<int>(v);
  }
  if (device < 0) Py_RETURN_NONE;
  // A gate of two products of one x that nothing else reads, where the library's one launch for the three is the faster.
  std::vector<int> readers(count, 0), maker(count, -1);
  for (Py_ssize_t i = 0; i < nsteps; ++i) {
    ++readers[steps[i].x];
    if (steps[i].up >= 0) ++readers[steps[i].up];
    maker[steps[i].result] = static_cast<int>(i);
  }
  for (int v : returns) ++readers[v];
  for (Step& s : steps) {
    if (s.up < 0 || s.x == s.up || !g_gated_matmul || !g_gated_pays || maker[s.x] < 0 || maker[s.up] < 0 || readers[s.x] != 1 || readers[s.up] != 1) continue;
    Step &g = steps[maker[s.x]], &u = steps[maker[s.up]];
    if (g.up >= 0 || u.up >= 0 || g.x != u.x || g.scales->scalar_type() != u.scales->scalar_type() || g.group_size != u.group_size || g.bits != u.bits || g.mode != u.mode || g.dtype != u.dtype || g.dtype != types[g.x])
      continue;
    qmm_problem p = {};
    p.struct_size = sizeof(p);
    p.mode = g.mode;
    p.bits = g.bits;
    p.group_size = g.group_size;
    p.x_dtype = p.y_dtype = elem_of(g.dtype);
    p.table_dtype = elem_of(g.scales->scalar_type());
    p.batch = 1;
    p.M = shapes[g.x][0];
    p.K = shapes[g.x][1];
    p.N = shapes[s.x][1];
    if (p.M < 2 || p.M > 16 || p.x_dtype < 0 || p.table_dtype < 0 || g_gated_pays(&p) != 1) continue;
    s.gate_from = maker[s.x];
    s.up_from = maker[s.up];
    g.left = u.left = true;
  }
  std::vector<at::Tensor> made(count);
  const int rc = unlocked([&]() -> int {
    void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    const at::Device on(at::kCUDA, static_cast<c10::DeviceIndex>(device));
    auto value = [&](int i) -> const at::Tensor& { return given[i] ? *given[i] : made[i]; };
    auto result = [&](const Step& s) -> at::Tensor& {
      at::Tensor& y = made[s.result];
      y = at::detail::empty_cuda({shapes[s.result][0], shapes[s.result][1]}, types[s.result], on, std::nullopt);
      return y;
    };
    struct Weight {
      qmm_tensor w, scales, biases;
      bool of(const Step& s) { return words_of(*s.w, &w) && view_of(*s.scales, &scales) && (!s.biases || view_of(*s.biases, &biases)); }
      const qmm_tensor* b(const Step& s) const { return s.biases ? &biases : nullptr; }
    };
    auto product = [&](const Step& s) -> int {
      qmm_tensor vx, vy;
      Weight weight;
      if (!view_of(value(s.x), &vx) || !weight.of(s) || !view_of(result(s), &vy)) return kDeclined;
      return g_quantized_matmul(&vx, &weight.w, &weight.scales, weight.b(s), &vy, 1, s.group_size, s.bits, s.mode, stream);
    };
    for (const Step& s : steps) {
      if (s.left) continue;
      int rc;
      if (s.up < 0) {
        if ((rc = product(s))) return rc;
        continue;
      }
      at::Tensor& y = result(s);
      if (s.gate_from >= 0) {
        const Step &g = steps[s.gate_from], &u = steps[s.up_from];
        qmm_tensor vx, vy;
        Weight gate, up;
        if (!view_of(value(g.x), &vx) || !gate.of(g) || !up.of(u) || !view_of(y, &vy)) return kDeclined;
        rc = g_gated_matmul(&vx, &gate.w, &gate.scales, gate.b(g), &up.w, &up.scales, up.b(u), &vy, g.group_size, g.bits, g.mode, stream);
        if (rc == 0) continue;
        if (rc != QMM_ERR_UNSUPPORTED) return rc;
        if ((rc = product(g)) || (rc = product(u))) return rc;
      }
      const at::Tensor& x = value(s.x);
      if ((rc = g_silu_mul(x.const_data_ptr(), value(s.up).const_data_ptr(), y.data_ptr(), x.numel(), elem_of(types[s.x]), stream))) return rc;
    }
    return 0;
  });
  if (rc == kDeclined) Py_RETURN_NONE;
  if (rc) return PyLong_FromLong(rc);
  PyObject* out = PyList_New(nret);
  if (!out) return nullptr;
  for (Py_ssize_t i = 0; i < nret; ++i) {
    PyObject* o;
    if (returns[i] < nargs) {
      o = PyList_GET_ITEM(a[0], returns[i]);
      Py_INCREF(o);
    } else {
      o = THPVariable_Wrap(made[returns[i]]);
    }
    PyList_SET_ITEM(out, i, o);
  }
  return out;
}

// The entry itself: what throws is declined.
template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject* self, PyObject* const* a, Py_ssize_t n) {
  try {
    return F(self, a, n);
  } catch (const std::exception&) {
    if (PyErr_Occurred()) PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// bind(addresses of qmm_quantized_matmul, qmm_moe_workspace_bytes, qmm_moe_experts_checked[, qmm_moe_silu_mul[, qmm_pack_dense_layer[, qmm_gated_matmul, qmm_gated_matmul_pays]]])
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n < 3 || n > 7) {
    PyErr_SetString(PyExc_TypeError, "bind takes the entry points' addresses");
    return nullptr;
  }
  g_quantized_matmul = reinterpret_cast<QuantizedMatmul>(PyLong_AsVoidPtr(a[0]));
  g_moe_workspace = reinterpret_cast<MoeWorkspace>(PyLong_AsVoidPtr(a[1]));
  g_moe_experts = reinterpret_cast<MoeExperts>(PyLong_AsVoidPtr(a[2]));
  if (n > 3) g_silu_mul = reinterpret_cast<SiluMul>(PyLong_AsVoidPtr(a[3]));
  if (n > 4) g_pack_layer = reinterpret_cast<PackLayer>(PyLong_AsVoidPtr(a[4]));
  if (n > 5) g_gated_matmul = reinterpret_cast<GatedMatmul>(PyLong_AsVoidPtr(a[5]));
  if (n > 6) g_gated_pays = reinterpret_cast<GatedPays>(PyLong_AsVoidPtr(a[6]));
  if (PyErr_Occurred()) return nullptr;
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(bind)), METH_FASTCALL, nullptr},
    {"quantized_matmul", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<quantized_matmul>)), METH_FASTCALL, nullptr},
    {"moe_experts", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<moe_experts>)), METH_FASTCALL, nullptr},
    {"pack_layer", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<pack_layer>)), METH_FASTCALL, nullptr},
    {"run_steps", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(guarded<run_steps>)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
