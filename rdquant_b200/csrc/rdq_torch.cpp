// CPython extension `_rdq_torch`: the per-call host path of a packed layer in native code.
//
// A `Layer` object is made once per packed layer from its dict of device tensors and keeps what a
// call needs (pointers, sizes, references that keep the tensors alive).  Its `linear(x, bias,
// flags)` checks the input, allocates the output with torch's CUDA allocator, takes torch's current
// stream and calls rdq_linear (include/rdq_b200.h).  What the fast path does not take -- another
// dtype, a non-contiguous or host tensor, a wrong last dimension, a tensor whose memory cannot be asked
// for (of tracing or vmap, a sparse layout: the accessors throw or answer null) -- returns None, and the
// caller's Python path handles or refuses it; so does a call whose scratch does not fit on the device.
// No C++ exception leaves an entry point.
//
// Why native: a decode step calls dozens of linears whose kernels take 5-10 us, and the same
// checks, allocation and ctypes call written in Python took 25-33 us per call.
//
// Reference counterpart: the pybind wrappers of rdquant/csrc/bindings.cpp:156-201.
#include <Python.h>

#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cuda_runtime_api.h>

#include <algorithm>
#include <initializer_list>
#include <new>
#include <vector>

#include "../../include/rdq_b200.h"

namespace {

struct LayerObject {
  PyObject_HEAD
  rdq_layer layer;
  int64_t n_out;
  c10::DeviceIndex device;
  std::vector<at::Tensor> *keep;
};

// makes `device` current while it lives
struct OnDevice {
  c10::DeviceIndex prev;
  bool changed;
  explicit OnDevice(c10::DeviceIndex device) : prev(c10::cuda::current_device()), changed(prev != device) {
    if (changed) c10::cuda::set_device(device);
  }
  ~OnDevice() {
    if (changed) c10::cuda::set_device(prev);
  }
};

// Words of rdq_linear_words.  They are zero between launches, so the calls of a stream share a set; a
// stream that is being captured has one per capture, which the graph zeroes on every replay.  A set that
// is dropped goes back to torch's allocator, which gives it to later work of the same stream only.  At
// most kMostSets are kept, the last used; all are dropped with the last layer.  (Under the GIL.)
struct Words {
  c10::DeviceIndex device;
  c10::StreamId stream;
  unsigned long long capture;
  at::Tensor t;
};
constexpr size_t kMostSets = 64;
std::vector<Words> *word_sets = new std::vector<Words>();  // not destroyed at exit: CUDA may be gone by then
long layers_alive = 0;

// `fresh`: the words have any content
int32_t *words_of(c10::DeviceIndex device, const c10::cuda::CUDAStream &stream, bool *fresh) {
  const c10::StreamId id = stream.id();
  unsigned long long capture = 0;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamGetCaptureInfo(stream.stream(), &status, &capture) != cudaSuccess)
    cudaGetLastError();  // (a launch on such a stream will say what is wrong with it)
  if (status != cudaStreamCaptureStatusActive) capture = 0;
  auto &sets = *word_sets;
  sets.erase(std::remove_if(sets.begin(), sets.end(), [&](const Words &w) { return w.capture != 0 && w.capture != capture; }), sets.end());
  auto it = std::find_if(sets.begin(), sets.end(),
                         [&](const Words &w) { return w.device == device && w.stream == id && w.capture == capture; });
  *fresh = it == sets.end();
  if (*fresh) {
    if (sets.size() >= kMostSets) sets.erase(sets.begin());
    const int64_t sizes[1] = {RDQ_LINEAR_WORDS};
    sets.push_back({device, id, capture,
                    at::detail::empty_cuda(at::IntArrayRef(sizes, 1), at::kInt, c10::Device(c10::kCUDA, device), std::nullopt)});
  } else if (it + 1 != sets.end()) {
    std::rotate(it, it + 1, sets.end());
  }
  return static_cast<int32_t *>(sets.back().t.data_ptr());
}

// f() with a C++ exception as a RuntimeError (a Python exception behind it stays what it is) and null
template <typename F>
PyObject *guarded(F f) {
  try {
    return f();
  } catch (const std::exception &e) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
  } catch (...) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "unknown C++ exception");
  }
  return nullptr;
}
// f(), a look at arguments: false also where an accessor throws
template <typename F>
bool accepts(F f) {
  try {
    return f();
  } catch (...) {
    PyErr_Clear();
    return false;
  }
}

bool take(LayerObject *self, PyObject *dict, const char *key, const void **out) {
  *out = nullptr;
  PyObject *v = PyDict_GetItemString(dict, key);  // borrowed
  if (v == nullptr || v == Py_None) return true;
  if (!THPVariable_Check(v)) {
    PyErr_Format(PyExc_TypeError, "%s must be a tensor or None", key);
    return false;
  }
  const at::Tensor &t = THPVariable_Unpack(v);
  if (!t.is_cuda() || !t.is_contiguous()) {
    PyErr_Format(PyExc_RuntimeError, "%s must be a contiguous CUDA tensor", key);
    return false;
  }
  if (self->device < 0) self->device = t.get_device();
  if (t.get_device() != self->device) {
    PyErr_Format(PyExc_RuntimeError, "%s is on another device than the rest of the layer", key);
    return false;
  }
  *out = t.data_ptr();
  if (*out == nullptr && t.numel() != 0) {
    PyErr_Format(PyExc_RuntimeError, "%s has no memory", key);
    return false;
  }
  self->keep->push_back(t);
  return true;
}

bool take_int(PyObject *dict, const char *key, int *out) {
  PyObject *v = PyDict_GetItemString(dict, key);
  if (v == nullptr) {
    PyErr_Format(PyExc_KeyError, "%s", key);
    return false;
  }
  *out = static_cast<int>(PyLong_AsLong(v));
  return !(PyErr_Occurred());
}

// the fields of a new object; false with an exception set
bool fill_layer(LayerObject *self, PyObject *dict) {
  rdq_layer &l = self->layer;
  const void *s8 = nullptr, *perm = nullptr, *inv = nullptr, *ws = nullptr, *cnt = nullptr;
  bool ok = take_int(dict, "n_fp4", &l.n_fp4) && take_int(dict, "n_fp8", &l.n_fp8) &&
            take_int(dict, "n_fp16", &l.n_fp16) && take_int(dict, "k", &l.K) && take(self, dict, "w_fp4_q", &l.w_fp4) &&
            take(self, dict, "w_fp4_scales", &l.w_fp4_scales) && take(self, dict, "w_fp8_q", &l.w_fp8) &&
            take(self, dict, "w_fp8_scales", &s8) && take(self, dict, "w_fp16", &l.w_fp16) &&
            take(self, dict, "w_tiled", &l.w_tiled) && take(self, dict, "perm", &perm) && take(self, dict, "inv_perm", &inv) &&
            take(self, dict, "workspace", &ws) && take(self, dict, "tile_counters", &cnt);
  l.w_fp4_global_scale = 1.0f;
  if (ok) {
    if (PyObject *gs = PyDict_GetItemString(dict, "w_fp4_global_scale")) {
      l.w_fp4_global_scale = static_cast<float>(PyFloat_AsDouble(gs));
      ok = !PyErr_Occurred();
    }
  }
  if (!ok) return false;
  l.w_fp8_scales = static_cast<const float *>(s8);
  l.perm = static_cast<const int32_t *>(perm);
  l.inv_perm = static_cast<const int32_t *>(inv);
  l.gemv_ws = const_cast<void *>(ws);
  l.gemv_counters = static_cast<int32_t *>(const_cast<void *>(cnt));
  self->n_out = static_cast<int64_t>(l.n_fp4) + l.n_fp8 + l.n_fp16;
  return true;
}

PyObject *layer_new(PyTypeObject *type, PyObject *args, PyObject *) {
  PyObject *dict = nullptr;
  if (!PyArg_ParseTuple(args, "O!", &PyDict_Type, &dict)) return nullptr;
  LayerObject *self = reinterpret_cast<LayerObject *>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  ++layers_alive;
  self->layer = rdq_layer{};
  self->device = -1;
  self->keep = nullptr;
  PyObject *made = guarded([&]() -> PyObject * {
    self->keep = new std::vector<at::Tensor>();
    return fill_layer(self, dict) ? reinterpret_cast<PyObject *>(self) : nullptr;
  });
  if (made == nullptr) Py_DECREF(self);
  return made;
}

void layer_dealloc(PyObject *obj) {
  delete reinterpret_cast<LayerObject *>(obj)->keep;
  if (--layers_alive == 0) word_sets->clear();
  Py_TYPE(obj)->tp_free(obj);
}

// linear(x, bias or None, flags) -> y, or None when the fast path does not take this input
PyObject *layer_linear(PyObject *obj, PyObject *const *args, Py_ssize_t nargs) {
  LayerObject *self = reinterpret_cast<LayerObject *>(obj);
  if (nargs != 3 || !THPVariable_Check(args[0])) {
    PyErr_SetString(PyExc_TypeError, "linear(x, bias, flags)");
    return nullptr;
  }
  const long flags = PyLong_AsLong(args[2]);
  if (flags == -1 && PyErr_Occurred()) return nullptr;
  const rdq_layer &l = self->layer;
  const at::Tensor &x = THPVariable_Unpack(args[0]);
  int64_t dims = 0, m = 0;
  auto type = at::kHalf;
  const void *xp = nullptr, *bias = nullptr;
  const bool ok = accepts([&] {
    dims = x.dim();
    type = x.scalar_type();
    if (!x.is_cuda() || x.get_device() != self->device || dims < 1 || x.size(dims - 1) != l.K || !x.is_contiguous() ||
        (type != at::kHalf && type != at::kBFloat16) || l.K == 0)
      return false;
    m = x.numel() / l.K;
    xp = x.data_ptr();
    if (m == 0 || m > 0x7fffffff || xp == nullptr || (reinterpret_cast<uintptr_t>(xp) & 15)) return false;
    if (args[1] == Py_None) return true;
    if (!THPVariable_Check(args[1])) return false;
    const at::Tensor &b = THPVariable_Unpack(args[1]);
    if (!b.is_cuda() || b.get_device() != self->device || b.scalar_type() != at::kHalf || !b.is_contiguous() ||
        b.numel() != self->n_out)
      return false;
    bias = b.data_ptr();
    return bias != nullptr || self->n_out == 0;
  });
  if (!ok) Py_RETURN_NONE;
  return guarded([&]() -> PyObject * {
    OnDevice guard(self->device);
    const c10::Device device(c10::kCUDA, self->device);
    at::Tensor y;
    if (dims == 2) {
      const int64_t sizes[2] = {m, self->n_out};
      y = at::detail::empty_cuda(at::IntArrayRef(sizes, 2), type, device, std::nullopt);
    } else {
      std::vector<int64_t> sizes(x.sizes().begin(), x.sizes().end());
      sizes.back() = self->n_out;
      y = at::detail::empty_cuda(sizes, type, device, std::nullopt);
    }
    const int xt = type == at::kBFloat16 ? RDQ_BF16 : RDQ_F16;
    size_t need = 0;
    int rc = rdq_linear_workspace_size(&l, static_cast<int>(m), xt, &need);
    if (rc == RDQ_OK) {
      // scratch of this call alone: the allocator orders its reuse behind the work queued here
      at::Tensor ws;
      if (need) {
        const int64_t sizes[1] = {static_cast<int64_t>(need)};
        try {
          ws = at::detail::empty_cuda(at::IntArrayRef(sizes, 1), at::kByte, device, std::nullopt);
        } catch (const c10::OutOfMemoryError &) {
          Py_RETURN_NONE;  // the caller's path has kernels that need none
        }
      }
      const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(self->device);
      // (without a workspace it is a decode kernel, and a GEMM of whole tiles counts nothing either)
      int32_t *words = nullptr;
      bool fresh = false;
      if (need && rdq_linear_uses_words(&l, static_cast<int>(m), xt)) words = words_of(self->device, stream, &fresh);
      rc = rdq_linear_words(&l, xp, xt, static_cast<int>(m), bias, y.data_ptr(), need ? ws.data_ptr() : nullptr, need, words,
                            static_cast<int>(flags) | (fresh ? RDQ_LINEAR_FRESH : 0), stream.stream());
      if (fresh && rc != RDQ_OK) word_sets->pop_back();  // perhaps not zeroed
    }
    if (rc != RDQ_OK) {
      PyErr_Format(PyExc_RuntimeError, "rdq_linear failed (code %d): %s", rc, rdq_last_error());
      return nullptr;
    }
    return THPVariable_Wrap(std::move(y));
  });
}

at::Tensor cuda_empty(at::IntArrayRef sizes, at::ScalarType type, c10::DeviceIndex device) {
  return at::detail::empty_cuda(sizes, type, c10::Device(c10::kCUDA, device), std::nullopt);
}
PyObject *wrap_or_none(at::Tensor t) {
  if (!t.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(t));
}
// a contiguous CUDA tensor of one of the given types on `device` (any device if < 0), or null
const at::Tensor *cuda_arg(PyObject *o, c10::DeviceIndex device, std::initializer_list<at::ScalarType> types) {
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor &t = THPVariable_Unpack(o);
  if (!t.is_cuda() || !t.is_contiguous() || (device >= 0 && t.get_device() != device)) return nullptr;
  for (auto type : types)
    if (t.scalar_type() == type) return &t;
  return nullptr;
}
bool int_args(PyObject *const *args, int n, long *out) {
  for (int i = 0; i < n; ++i) {
    out[i] = PyLong_AsLong(args[i]);
    if (out[i] == -1 && PyErr_Occurred()) return false;
  }
  return true;
}

// quantize_layer(weight [N, K], perm int64 [N], n4, n8, n16) -> (codes, scales, global_scale, fp8, fp8_scale,
// fp16, inv_perm, splits int32 [3] on the host), absent groups None; None when the input needs conversions first
PyObject *quantize_layer(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  long n[3];
  if (nargs != 5) {
    PyErr_SetString(PyExc_TypeError, "quantize_layer(weight, perm, n4, n8, n16)");
    return nullptr;
  }
  if (!int_args(args + 2, 3, n)) return nullptr;
  const at::Tensor *w = nullptr;
  const void *wp = nullptr;
  const long long *pp = nullptr;
  int64_t N = 0, K = 0;
  c10::DeviceIndex dev = -1;
  const bool ok = accepts([&] {
    w = cuda_arg(args[0], -1, {at::kHalf, at::kFloat});
    if (w == nullptr || w->dim() != 2) return false;
    dev = w->get_device();
    N = w->size(0);
    K = w->size(1);
    const at::Tensor *perm = cuda_arg(args[1], dev, {at::kLong});
    if (perm == nullptr || perm->numel() != N || n[0] < 0 || n[1] < 0 || n[2] < 0 || n[0] + n[1] + n[2] != N || K % 16 || K == 0 ||
        N == 0 || N > 0x7fffffff || K > 0x7fffffff)
      return false;
    wp = w->data_ptr();
    pp = static_cast<const long long *>(perm->data_ptr());
    return wp != nullptr && pp != nullptr && (reinterpret_cast<uintptr_t>(wp) & 15) == 0;
  });
  if (!ok) Py_RETURN_NONE;
  return guarded([&]() -> PyObject * {
    OnDevice guard(dev);
    at::Tensor codes, scales, top, fp8, fp8_scale, fp16;
    if (n[0]) {
      codes = cuda_empty({n[0], K / 2}, at::kByte, dev);
      scales = cuda_empty({n[0], K / 16}, at::kByte, dev);
      top = cuda_empty({1}, at::kFloat, dev);
    }
    if (n[1]) {
      fp8 = cuda_empty({n[1], K}, at::kByte, dev);
      fp8_scale = cuda_empty({n[1]}, at::kFloat, dev);
    }
    if (n[2]) fp16 = cuda_empty({n[2], K}, at::kBFloat16, dev);
    at::Tensor inv = cuda_empty({N}, at::kInt, dev), scratch = cuda_empty({RDQ_QUANTIZE_LAYER_SCRATCH}, at::kFloat, dev);
    auto ptr = [](const at::Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; };
    const int rc = rdq_quantize_layer(wp, w->scalar_type() == at::kFloat, pp,
                                      static_cast<int>(n[0]), static_cast<int>(n[1]), static_cast<int>(n[2]), static_cast<int>(K),
                                      ptr(codes), ptr(scales), static_cast<float *>(ptr(top)), ptr(fp8),
                                      static_cast<float *>(ptr(fp8_scale)), ptr(fp16), static_cast<int32_t *>(inv.data_ptr()),
                                      static_cast<float *>(scratch.data_ptr()), c10::cuda::getCurrentCUDAStream(dev).stream());
    if (rc != RDQ_OK) {
      PyErr_Format(PyExc_RuntimeError, "rdq_quantize_layer failed (code %d): %s", rc, rdq_last_error());
      return nullptr;
    }
    at::Tensor splits = at::detail::empty_cpu({3}, at::kInt);
    for (int i = 0; i < 3; ++i) static_cast<int32_t *>(splits.data_ptr())[i] = static_cast<int32_t>(n[i]);
    return Py_BuildValue("NNNNNNNN", wrap_or_none(std::move(codes)), wrap_or_none(std::move(scales)), wrap_or_none(std::move(top)),
                         wrap_or_none(std::move(fp8)), wrap_or_none(std::move(fp8_scale)), wrap_or_none(std::move(fp16)),
                         wrap_or_none(std::move(inv)), wrap_or_none(std::move(splits)));
  });
}

// dequantize(w4, s4, w8, s8, w16, inv_perm or None, n4, n8, n16, k) -> f16 [N, K], or None when an argument needs the
// checked path.  Groups of size 0 are not looked at.
PyObject *dequantize(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  long n[4];
  if (nargs != 10) {
    PyErr_SetString(PyExc_TypeError, "dequantize(w4, s4, w8, s8, w16, inv_perm, n4, n8, n16, k)");
    return nullptr;
  }
  if (!int_args(args + 6, 4, n)) return nullptr;
  const int64_t K = n[3], N = n[0] + n[1] + n[2];
  if (n[0] < 0 || n[1] < 0 || n[2] < 0 || N <= 0 || K <= 0) Py_RETURN_NONE;
  c10::DeviceIndex dev = -1;
  const void *p[6] = {};
  bool bf16 = false;
  auto take_arg = [&](int i, std::initializer_list<at::ScalarType> types, int64_t numel) {
    const at::Tensor *t = cuda_arg(args[i], dev, types);
    if (t == nullptr || t->numel() != numel) return false;
    if (i != 3 && i != 5 && (t->dim() != 2 || t->size(0) != (i == 4 ? n[2] : n[i / 2]))) return false;
    dev = t->get_device();
    p[i] = t->data_ptr();
    if (p[i] == nullptr) return false;
    if (i == 4) bf16 = t->scalar_type() == at::kBFloat16;
    return true;
  };
  const bool ok = accepts([&] {
    if (n[0] && !(take_arg(0, {at::kByte}, n[0] * (K / 2)) && take_arg(1, {at::kByte}, n[0] * (K / 16)))) return false;
    if (n[1] && !(take_arg(2, {at::kByte}, n[1] * K) && take_arg(3, {at::kFloat}, n[1]))) return false;
    if (n[2] && !take_arg(4, {at::kHalf, at::kBFloat16}, n[2] * K)) return false;
    return args[5] == Py_None || take_arg(5, {at::kInt}, N);
  });
  if (!ok) Py_RETURN_NONE;
  return guarded([&]() -> PyObject * {
    OnDevice guard(dev);
    at::Tensor out = cuda_empty({N, K}, at::kHalf, dev);
    const int rc = rdq_dequant_packed(p[0], p[1], 1.0f, p[2], static_cast<const float *>(p[3]), p[4], bf16,
                                      static_cast<const int32_t *>(p[5]), out.data_ptr(), 0, static_cast<int>(n[0]),
                                      static_cast<int>(n[1]), static_cast<int>(n[2]), static_cast<int>(K),
                                      c10::cuda::getCurrentCUDAStream(dev).stream());
    if (rc != RDQ_OK) {
      PyErr_Format(PyExc_RuntimeError, "rdq_dequant_packed failed (code %d): %s", rc, rdq_last_error());
      return nullptr;
    }
    return THPVariable_Wrap(std::move(out));
  });
}

// drop_words() -> number of sets dropped: the next calls start with zeroed ones (after a time-out, which
// leaves counts behind)
PyObject *drop_words(PyObject *, PyObject *) {
  const size_t n = word_sets->size();
  word_sets->clear();
  return PyLong_FromSize_t(n);
}

PyMethodDef module_methods[] = {
    {"drop_words", drop_words, METH_NOARGS, "forget the words of rdq_linear_words, which a time-out leaves in disorder"},
    {"quantize_layer", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(quantize_layer)), METH_FASTCALL,
     "packed tensors of a layer, or None when the input needs conversions first"},
    {"dequantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(dequantize)), METH_FASTCALL,
     "f16 weight of a packed layer, or None when an argument needs the checked path"},
    {nullptr, nullptr, 0, nullptr}};

PyMethodDef layer_methods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(layer_linear)), METH_FASTCALL,
     "linear(x, bias, flags): y = x @ W.T (+ bias), or None when the input needs the checked path"},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject layer_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_rdq_torch", "native host path of the packed layers", -1, module_methods};

}  // namespace

PyMODINIT_FUNC PyInit__rdq_torch(void) {
  layer_type.tp_name = "_rdq_torch.Layer";
  layer_type.tp_basicsize = sizeof(LayerObject);
  layer_type.tp_flags = Py_TPFLAGS_DEFAULT;
  layer_type.tp_new = layer_new;
  layer_type.tp_dealloc = layer_dealloc;
  layer_type.tp_methods = layer_methods;
  layer_type.tp_doc = "Layer(fd): a packed layer ready to be called";
  if (PyType_Ready(&layer_type) < 0) return nullptr;
  PyObject *m = PyModule_Create(&module_def);
  if (m == nullptr) return nullptr;
  Py_INCREF(&layer_type);
  if (PyModule_AddObject(m, "Layer", reinterpret_cast<PyObject *>(&layer_type)) < 0) {
    Py_DECREF(&layer_type);
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
