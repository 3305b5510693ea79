// Python binding of the layer call: what the host does per call, in native code.
//
// A transformer layer of few rows takes about 15 us on the GPU.  Looked up, checked and called from Python (ctypes), the
// same call cost 30 us of interpreter time: 12 parameters to compare with what the packed weights were made from, shapes
// and types of five tensors, two allocations, 16 converted arguments.  Here the interpreter makes one call.
//
// `LayerPlan` holds what a layer's native call needs (the parameter block, the tensors behind it) and what it was made
// from: dictionary entries of the modules (parameters, submodules, options) with the objects found there, and for tensors
// their storage, version counter, type and layout.  `layer_forward` returns None when anything has changed or anything about
// the arguments is out of the ordinary; the Python side then validates, rebuilds or raises.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/TracerMode.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <memory>
#include <optional>
#include <utility>
#include <vector>

#include "../../../include/fast_mimi_b200.h"

namespace {

// What a tensor's contents are known by.  The storage counts by its identity: assigning a parameter's .data moves no version
// counter, and an address is given out again once its storage is gone.  The weak reference keeps the identity, not the memory.
// Throws for tensors without storage (wrappers of transforms) and without a version counter (made in inference mode): such a
// one cannot be watched.
struct Stamp {
  explicit Stamp(const at::Tensor& t)
      : storage(t.storage().getWeakStorageImpl()), data(t.const_data_ptr()), version(static_cast<uint32_t>(t._version())),
        dtype(t.scalar_type()), sizes(t.sizes()), strides(t.strides()) {}
  bool still(const at::Tensor& t) const {
    return t.storage().unsafeGetStorageImpl() == storage._unsafe_get_target() && t.const_data_ptr() == data &&
           static_cast<uint32_t>(t._version()) == version && t.scalar_type() == dtype && t.sizes() == at::IntArrayRef(sizes) &&
           t.strides() == at::IntArrayRef(strides);
  }
  c10::weak_intrusive_ptr<c10::StorageImpl> storage;
  const void* data;
  uint32_t version;
  c10::ScalarType dtype;
  c10::DimVector sizes, strides;
};

struct Watch {
  PyObject* dict;
  PyObject* key;
  PyObject* value;
  std::optional<Stamp> stamp;      // of a tensor
};

struct LayerPlan {
  PyObject_HEAD
  std::vector<Watch>* watches;
  PyObject* keep;            // tuple of tensors the parameter block points into
  fm_layer_params params;
  int* status;
  c10::ScalarType dtype;     // of the residual stream
  c10::ScalarType value;     // of the ring's V
  c10::DeviceIndex device;
};

void plan_dealloc(PyObject* self_obj) {
  LayerPlan* self = reinterpret_cast<LayerPlan*>(self_obj);
  PyObject_GC_UnTrack(self_obj);
  if (self->watches != nullptr) {
    for (Watch& w : *self->watches) {
      Py_XDECREF(w.dict);
      Py_XDECREF(w.key);
      Py_XDECREF(w.value);
    }
    delete self->watches;
  }
  Py_XDECREF(self->keep);
  Py_TYPE(self_obj)->tp_free(self_obj);
}

int plan_traverse(PyObject* self_obj, visitproc visit, void* arg) {
  LayerPlan* self = reinterpret_cast<LayerPlan*>(self_obj);
  if (self->watches != nullptr)
    for (Watch& w : *self->watches) {
      Py_VISIT(w.dict);
      Py_VISIT(w.value);
    }
  Py_VISIT(self->keep);
  return 0;
}

int plan_clear(PyObject* self_obj) {
  LayerPlan* self = reinterpret_cast<LayerPlan*>(self_obj);
  if (self->watches != nullptr)
    for (Watch& w : *self->watches) {
      Py_CLEAR(w.dict);
      Py_CLEAR(w.value);
    }
  Py_CLEAR(self->keep);
  return 0;
}

// LayerPlan(watches, keep, params_address, status, like, value_like): watches is a list of (dict, key); keep the tensors
// behind the parameter block at params_address (copied); status an int32 tensor; like / value_like tensors whose type and
// device activations / ring values must have.
PyObject* plan_new(PyTypeObject* type, PyObject* args, PyObject*) {
  PyObject *list, *keep, *status, *like, *value_like;
  unsigned long long address;
  if (!PyArg_ParseTuple(args, "O!O!KOOO", &PyList_Type, &list, &PyTuple_Type, &keep, &address, &status, &like, &value_like)) return nullptr;
  if (!THPVariable_Check(status) || !THPVariable_Check(like) || !THPVariable_Check(value_like)) {
    PyErr_SetString(PyExc_TypeError, "status, like and value_like must be tensors");
    return nullptr;
  }
  LayerPlan* self = reinterpret_cast<LayerPlan*>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  self->watches = new std::vector<Watch>();
  Py_INCREF(keep);
  self->keep = keep;
  self->params = *reinterpret_cast<const fm_layer_params*>(address);
  self->params.weights_settled = 0;
  self->status = static_cast<int*>(THPVariable_Unpack(status).data_ptr());
  self->dtype = THPVariable_Unpack(like).scalar_type();
  self->value = THPVariable_Unpack(value_like).scalar_type();
  self->device = THPVariable_Unpack(like).device().index();
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(list); ++i) {
    PyObject *dict, *key;
    if (!PyArg_ParseTuple(PyList_GET_ITEM(list, i), "O!O", &PyDict_Type, &dict, &key)) {
      Py_DECREF(self);
      return nullptr;
    }
    PyObject* value = PyDict_GetItemWithError(dict, key);
    if (value == nullptr) {
      if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, key);
      Py_DECREF(self);
      return nullptr;
    }
    Watch w = {dict, key, value, std::nullopt};
    try {
      if (THPVariable_Check(value)) w.stamp.emplace(THPVariable_Unpack(value));
    } catch (const std::exception&) {
      PyErr_SetObject(PyExc_KeyError, key);
      Py_DECREF(self);
      return nullptr;
    }
    Py_INCREF(dict);
    Py_INCREF(key);
    Py_INCREF(value);
    self->watches->push_back(std::move(w));
  }
  return reinterpret_cast<PyObject*>(self);
}

bool unchanged(const LayerPlan* plan) {
  for (const Watch& w : *plan->watches) {
    if (PyDict_GetItemWithError(w.dict, w.key) != w.value) {
      PyErr_Clear();
      return false;
    }
    if (w.stamp && !w.stamp->still(THPVariable_Unpack(w.value))) return false;
  }
  return true;
}

PyTypeObject plan_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

// An int argument, or -1 for what is none (a value for the Python side to look at).
long int_of(PyObject* o) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) PyErr_Clear();
  return v;
}

// layer_forward(plan, x, cos, sin, ring_k, ring_v, layer, past) -> tensor, or None: not the ordinary case.  The rings are those
// of all layers, [layers, streams, 8, slots, 64]: the caller's own tensors, of which nothing is kept.
PyObject* layer_forward_checked(PyObject* const* a, Py_ssize_t n) {
  if (n != 8 || !PyObject_TypeCheck(a[0], &plan_type)) {
    PyErr_SetString(PyExc_TypeError, "layer_forward(plan, x, cos, sin, ring_k, ring_v, layer, past)");
    return nullptr;
  }
  LayerPlan* plan = reinterpret_cast<LayerPlan*>(a[0]);
  if (!THPVariable_Check(a[1]) || !THPVariable_Check(a[2]) || !THPVariable_Check(a[3])) Py_RETURN_NONE;
  const at::Tensor &x = THPVariable_Unpack(a[1]), &cos = THPVariable_Unpack(a[2]), &sin = THPVariable_Unpack(a[3]);
  if (!x.is_cuda() || x.scalar_type() != plan->dtype || x.device().index() != plan->device || x.dim() != 3 || x.size(2) != 512 ||
      !x.is_contiguous())
    Py_RETURN_NONE;
  const int64_t B = x.size(0), T = x.size(1);
  if (B * T > 0x7fffffff || B * T == 0) Py_RETURN_NONE;
  for (const at::Tensor* t : {&cos, &sin})
    if (!t->is_cuda() || t->scalar_type() != at::kFloat || t->dim() != 3 || t->size(1) != T || t->size(2) != 64 ||
        (t->size(0) != 1 && t->size(0) != B) || !t->is_contiguous())
      Py_RETURN_NONE;
  if (cos.size(0) != sin.size(0)) Py_RETURN_NONE;
  void *ring_k = nullptr, *ring_v = nullptr;
  int past = 0, slots = 0;
  if (a[4] != Py_None) {
    if (!THPVariable_Check(a[4]) || !THPVariable_Check(a[5])) Py_RETURN_NONE;
    const at::Tensor &k = THPVariable_Unpack(a[4]), &v = THPVariable_Unpack(a[5]);
    const long layer = int_of(a[6]), p = int_of(a[7]);
    if (!k.is_cuda() || k.scalar_type() != at::kBFloat16 || k.dim() != 5 || k.size(1) != B || k.size(2) != 8 || k.size(4) != 64 ||
        layer < 0 || layer >= k.size(0) || !k.is_contiguous() || !v.is_cuda() || v.scalar_type() != plan->value || v.sizes() != k.sizes() || !v.is_contiguous())
      Py_RETURN_NONE;
    slots = static_cast<int>(k.size(3));
    ring_k = static_cast<uint16_t*>(k.data_ptr()) + layer * k.stride(0);
    ring_v = static_cast<uint16_t*>(v.data_ptr()) + layer * k.stride(0);
    if (p < 0 || p > 0x7fffffffL - T) Py_RETURN_NONE;
    past = static_cast<int>(p);
  }
  if (!unchanged(plan)) Py_RETURN_NONE;
  const fm_layer_params& q = plan->params;
  const int64_t elem = static_cast<int64_t>(x.element_size());
  int64_t bytes = B * T * (2048 + 512 * elem + (2 * q.ffn > 3072 ? 2 * q.ffn : 3072)) + 4096;
  if (ring_k != nullptr) bytes += 2048 * B * ((past < q.window - 1 ? past : q.window - 1) + T);
  const at::Tensor workspace = at::empty({bytes}, x.options().dtype(at::kByte));
  at::Tensor y = at::empty(x.sizes(), x.options());
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const long long bstride = cos.size(0) == 1 ? 0 : T * 64;
  // every address before the interpreter lock is given up: what has none throws
  const void* x_data = x.const_data_ptr();
  const float *cos_data = cos.const_data_ptr<float>(), *sin_data = sin.const_data_ptr<float>();
  void *y_data = y.data_ptr(), *space = workspace.data_ptr();
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS
  rc = fm_layer_forward(&q, x_data, y_data, space, bytes, cos_data, sin_data, bstride, static_cast<int>(B), static_cast<int>(T),
                        ring_k, ring_v, past, slots, plan->status, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) return PyLong_FromLong(rc);
  plan->params.weights_settled = 1;
  return THPVariable_Wrap(std::move(y));
}

// No C++ exception leaves the module: whatever threw did so before the launch, and the Python side runs into it again and
// raises it in its own type (out of memory, tensors without storage).
PyObject* layer_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    return layer_forward_checked(a, n);
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
}

// ---- The calls around the quantiser.  Nothing is kept between them: the tensors come with every call.  They return None for
// anything out of the ordinary, (name, status) for a native call that refused, and leave raising to the Python side.

const at::Tensor* tensor(PyObject* o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

// A plain CUDA tensor of a type and rank on the current device.
bool plain(const at::Tensor* t, c10::ScalarType type, int64_t dim) {
  return t != nullptr && t->is_cuda() && t->scalar_type() == type && t->dim() == dim && t->device().index() == c10::cuda::current_device();
}

// FP16 hi + lo parts of a weight [n, k] as the split-precision products take them.
bool weight_parts(const at::Tensor* hi, const at::Tensor* lo, int64_t k) {
  return plain(hi, at::kHalf, 2) && plain(lo, at::kHalf, 2) && hi->is_contiguous() && lo->is_contiguous() && hi->sizes() == lo->sizes() &&
         hi->size(1) == k && k % 64 == 0 && hi->size(0) % 256 == 0 && hi->size(0) > 0;
}

PyObject* refused(const char* name, int rc) { return Py_BuildValue("(si)", name, rc); }

// One allocation for two FP16 matrices of a size.
at::Tensor two_parts(int64_t values, const at::Tensor& like) { return at::empty({2, values}, like.options().dtype(at::kHalf)); }

// conv_frames(x [B, C, T], w_hi, w_lo, kernel, stride, status) -> [B, C_out, ceil(T / stride)]
PyObject* conv_frames_checked(PyObject* const* a, Py_ssize_t n) {
  if (n != 6) {
    PyErr_SetString(PyExc_TypeError, "conv_frames(x, w_hi, w_lo, kernel, stride, status)");
    return nullptr;
  }
  const at::Tensor *x = tensor(a[0]), *hi = tensor(a[1]), *lo = tensor(a[2]), *status = tensor(a[5]);
  const long kernel = int_of(a[3]), stride = int_of(a[4]);
  if (!plain(x, at::kFloat, 3) || stride < 1 || kernel < stride || kernel > 16 || !plain(status, at::kInt, 1)) Py_RETURN_NONE;
  const int64_t B = x->size(0), C = x->size(1), T = x->size(2), t_out = (T + stride - 1) / stride;
  if (!weight_parts(hi, lo, kernel * C) || B * T == 0 || B * (t_out + kernel) > 0x7fffffff || T > 0x7fffffff) Py_RETURN_NONE;
  const int64_t n_out = hi->size(0);
  const bool direct = C % 64 == 0 && fm_split_direct(B * t_out, static_cast<int>(n_out), static_cast<int>(kernel * C));
  if (!direct && (kernel % stride != 0 || stride * C % 64 != 0)) Py_RETURN_NONE;
  const at::Tensor frames = x->transpose(1, 2).contiguous();
  const int64_t extra = kernel / stride - 1, rows = B * (t_out + extra), cols = stride * C;
  at::Tensor parts;
  if (!direct) parts = two_parts(rows * cols, frames);
  const at::Tensor y = at::empty({B, t_out, n_out}, frames.options());
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const float* src = frames.const_data_ptr<float>();
  const void *w_hi = hi->const_data_ptr(), *w_lo = lo->const_data_ptr();
  float* out = y.data_ptr<float>();
  int* st = status->data_ptr<int>();
  uint16_t* part = direct ? nullptr : static_cast<uint16_t*>(parts.data_ptr());
  const int b = static_cast<int>(B), t = static_cast<int>(T), c = static_cast<int>(C), ker = static_cast<int>(kernel), str = static_cast<int>(stride),
            outs = static_cast<int>(n_out);
  int rc = 0;
  const char* what = "fm_conv_frames_f32";
  Py_BEGIN_ALLOW_THREADS
  if (direct) {
    rc = fm_conv_frames_f32(src, w_hi, w_lo, out, b, t, c, ker, str, outs, st, stream);
  } else {
    what = "fm_conv_parts_f32";
    rc = fm_conv_parts_f32(src, part, part + rows * cols, w_hi, w_lo, out, b, t, c, ker, str, outs, st, stream);
  }
  Py_END_ALLOW_THREADS
  if (rc != 0) return refused(what, rc);
  return THPVariable_Wrap(y.transpose(1, 2));
}

// rvq_encode(embeddings [B, C, T], w_hi, w_lo, ((vectors, half, sq, e_max, layers), (..)), tau_rel, status): both branches' input projections
// and their searches, then what the status word says -> codes [layers, B, T], or that word
PyObject* rvq_encode_checked(PyObject* const* a, Py_ssize_t n) {
  if (n != 6) {
    PyErr_SetString(PyExc_TypeError, "rvq_encode(embeddings, w_hi, w_lo, stacks, tau_rel, status)");
    return nullptr;
  }
  const at::Tensor *x = tensor(a[0]), *hi = tensor(a[1]), *lo = tensor(a[2]), *status = tensor(a[5]);
  if (!plain(x, at::kFloat, 3) || !plain(status, at::kInt, 1) || !PyTuple_Check(a[3]) || PyTuple_GET_SIZE(a[3]) != 2 || !PyFloat_Check(a[4])) Py_RETURN_NONE;
  const int64_t B = x->size(0), C = x->size(1), T = x->size(2), rows = B * T;
  if (!weight_parts(hi, lo, C) || hi->size(0) != 512 || rows == 0 || rows > 0x7fffffff / 512) Py_RETURN_NONE;
  constexpr int kMaxLayers = 64;
  fm_rvq_stack stacks[2];
  float e_max[2][kMaxLayers];
  int64_t layers = 0, entries = 0;
  for (int i = 0; i < 2; ++i) {
    PyObject* s = PyTuple_GET_ITEM(a[3], i);
    if (!PyTuple_Check(s) || PyTuple_GET_SIZE(s) != 5) Py_RETURN_NONE;
    const at::Tensor *vectors = tensor(PyTuple_GET_ITEM(s, 0)), *half = tensor(PyTuple_GET_ITEM(s, 1)), *sq = tensor(PyTuple_GET_ITEM(s, 2));
    PyObject* norms = PyTuple_GET_ITEM(s, 3);
    const long count = int_of(PyTuple_GET_ITEM(s, 4));
    if (!plain(vectors, at::kFloat, 3) || !plain(half, at::kHalf, 3) || !plain(sq, at::kFloat, 2) || !vectors->is_contiguous() || !half->is_contiguous() ||
        !sq->is_contiguous() || half->sizes() != vectors->sizes() || vectors->size(2) != 256 || sq->size(0) != vectors->size(0) ||
        sq->size(1) != vectors->size(1) || !PyList_Check(norms) || count < 1 || count > vectors->size(0) || count > kMaxLayers || PyList_GET_SIZE(norms) < count)
      Py_RETURN_NONE;
    if (i == 1 && vectors->size(1) != entries) Py_RETURN_NONE;
    entries = vectors->size(1);
    for (long l = 0; l < count; ++l) {
      if (!PyFloat_Check(PyList_GET_ITEM(norms, l))) Py_RETURN_NONE;
      e_max[i][l] = static_cast<float>(PyFloat_AS_DOUBLE(PyList_GET_ITEM(norms, l)));
    }
    stacks[i] = {nullptr, half->const_data_ptr(), vectors->const_data_ptr<float>(), sq->const_data_ptr<float>(), e_max[i], nullptr, static_cast<int>(count)};
    layers += count;
  }
  const at::Tensor frames = x->transpose(1, 2).contiguous();
  at::Tensor codes = at::empty({layers, B, T}, frames.options().dtype(at::kLong));
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const float* src = frames.const_data_ptr<float>();
  const void *w_hi = hi->const_data_ptr(), *w_lo = lo->const_data_ptr();
  int* st = status->data_ptr<int>();
  stacks[0].codes = reinterpret_cast<long long*>(codes.data_ptr<int64_t>());
  stacks[1].codes = stacks[0].codes + stacks[0].layers * rows;
  const float tau_rel = static_cast<float>(PyFloat_AS_DOUBLE(a[4]));
  const int width = static_cast<int>(C), n_codes = static_cast<int>(entries);
  int words[2] = {0, 0};
  const char* what = "fm_rvq_encode_frames_f32";
  int rc = fm_rvq_encode_frames_f32(src, width, w_hi, w_lo, stacks, 2, rows, n_codes, tau_rel, st, stream);
  at::Tensor projected, parts, space;
  float* both = nullptr;
  uint16_t* part = nullptr;
  uint8_t* ws = nullptr;
  const bool chain = rc == -9;             // the projections, then the search
  const int64_t half_bytes = rows * 512, record_bytes = rows * (entries / 64) * 16;
  if (chain) {
    projected = at::empty({2, rows, 256}, frames.options());
    space = at::empty({half_bytes + record_bytes + rows * 4}, frames.options().dtype(at::kByte));
    if (!fm_split_direct(rows, 512, width)) {
      parts = two_parts(rows * C, frames);
      part = static_cast<uint16_t*>(parts.data_ptr());
    }
    both = projected.data_ptr<float>();
    ws = static_cast<uint8_t*>(space.data_ptr());
    stacks[0].residual = both;
    stacks[1].residual = both + rows * 256;
  }
  Py_BEGIN_ALLOW_THREADS
  if (chain) {
    if (part == nullptr) {
      what = "fm_linear_rows_f32";
      rc = fm_linear_rows_f32(src, w_hi, w_lo, both, rows, 2, 512, width, st, stream);
    } else {
      what = "fm_split_half";
      rc = fm_split_half(src, part, part + rows * C, rows * C, stream);
      if (rc == 0) {
        what = "fm_linear_split_f32";
        rc = fm_linear_split_f32(part, part + rows * C, rows, width, w_hi, w_lo, both, rows, 1, 1, 0, 2, 512, width, st, stream);
      }
    }
    if (rc == 0) {
      what = "fm_rvq_encode_stacks_f32";
      rc = fm_rvq_encode_stacks_f32(stacks, 2, ws, reinterpret_cast<float*>(ws + half_bytes + record_bytes), ws + half_bytes, rows, n_codes, tau_rel, st,
                                    stream);
    }
  }
  if (rc == 0) {
    what = "fm_read_words";
    rc = fm_read_words(st, nullptr, words, stream);
  }
  Py_END_ALLOW_THREADS
  if (rc != 0) return refused(what, rc);
  if (words[0] != 0) return PyLong_FromLong(words[0]);
  return THPVariable_Wrap(std::move(codes));
}

// rvq_decode_project(codes [B, K, T], books0, books1 or None, w_hi, w_lo, status) -> (y [B, n, T], status word, whether a code was out of range)
PyObject* rvq_decode_project_checked(PyObject* const* a, Py_ssize_t n) {
  if (n != 6) {
    PyErr_SetString(PyExc_TypeError, "rvq_decode_project(codes, books0, books1, w_hi, w_lo, status)");
    return nullptr;
  }
  const at::Tensor *codes = tensor(a[0]), *books0 = tensor(a[1]), *books1 = a[2] == Py_None ? nullptr : tensor(a[2]);
  const at::Tensor *hi = tensor(a[3]), *lo = tensor(a[4]), *status = tensor(a[5]);
  const bool two = a[2] != Py_None;
  if (!plain(codes, at::kLong, 3) || !plain(books0, at::kFloat, 3) || (two && !plain(books1, at::kFloat, 3)) || !plain(status, at::kInt, 1)) Py_RETURN_NONE;
  const int64_t B = codes->size(0), K = codes->size(1), T = codes->size(2), n0 = two ? books0->size(0) : K, rows = B * T, width = two ? 512 : 256;
  if (n0 < 1 || n0 > books0->size(0) || (two && (K <= n0 || K - n0 > books1->size(0))) || rows == 0 || rows > 0x7fffffff / 512 ||
      !weight_parts(hi, lo, width) || books0->size(2) != 256 || !books0->is_contiguous() || (two && (books1->size(2) != 256 || !books1->is_contiguous())))
    Py_RETURN_NONE;
  const at::Tensor index = codes->contiguous();
  const at::Tensor parts = two_parts(rows * width, *books0);
  const int64_t n_out = hi->size(0);
  at::Tensor y = at::empty({B, n_out, T}, books0->options());
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const long long* c = reinterpret_cast<const long long*>(index.const_data_ptr<int64_t>());
  const float *first = books0->const_data_ptr<float>(), *second = two ? books1->const_data_ptr<float>() : nullptr;
  uint16_t* part = static_cast<uint16_t*>(parts.data_ptr());
  const void *w_hi = hi->const_data_ptr(), *w_lo = lo->const_data_ptr();
  float* out = y.data_ptr<float>();
  int* st = status->data_ptr<int>();
  const int n_codes0 = static_cast<int>(books0->size(1)), n_codes1 = two ? static_cast<int>(books1->size(1)) : 0;
  int rc = 0, words[2] = {0, 0};
  Py_BEGIN_ALLOW_THREADS
  rc = fm_rvq_decode_project_f32(c, first, second, part, part + rows * width, w_hi, w_lo, out, static_cast<int>(B), static_cast<int>(T), static_cast<int>(K),
                                 static_cast<int>(n0), n_codes0, n_codes1, static_cast<int>(n_out), st, words, stream);
  Py_END_ALLOW_THREADS
  if (rc == -8) Py_RETURN_NONE;
  if (rc != 0) return refused("fm_rvq_decode_project_f32", rc);
  return Py_BuildValue("(Nii)", THPVariable_Wrap(std::move(y)), words[0], words[1]);
}

// upsample(x [B, C, T], weight [C, 1, 4]) -> [B, C, 2 T]
PyObject* upsample_checked(PyObject* const* a, Py_ssize_t n) {
  if (n != 2) {
    PyErr_SetString(PyExc_TypeError, "upsample(x, weight)");
    return nullptr;
  }
  const at::Tensor *x = tensor(a[0]), *w = tensor(a[1]);
  if (!plain(x, at::kFloat, 3) || !plain(w, at::kFloat, 3) || !x->is_contiguous() || !w->is_contiguous()) Py_RETURN_NONE;
  const int64_t B = x->size(0), C = x->size(1), T = x->size(2);
  if (w->numel() != 4 * C || C % 32 != 0 || B > 65535 || B * C * T == 0 || T > 0x3fffffff) Py_RETURN_NONE;
  const at::Tensor y = at::empty({B, 2 * T, C}, x->options());
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream().stream();
  const float *src = x->const_data_ptr<float>(), *taps = w->const_data_ptr<float>();
  float* out = y.data_ptr<float>();
  int rc = 0;
  Py_BEGIN_ALLOW_THREADS
  rc = fm_upsample2_channels_f32(src, taps, out, static_cast<int>(B), static_cast<int>(T), static_cast<int>(C), stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) return refused("fm_upsample2_channels_f32", rc);
  return THPVariable_Wrap(y.transpose(1, 2));
}

// No C++ exception leaves the module (as in layer_forward); what threw did so before the first launch.  A call that torch.jit.trace records is left to
// the Python side, too, whose sizes are tensors then: the search and a transposed convolution that learns refuse it, where a recording of this
// module's calls would be one of their allocations alone.
template <PyObject* (*kFn)(PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (at::tracer::impl::is_dispatch_enabled()) Py_RETURN_NONE;
  try {
    return kFn(a, n);
  } catch (const std::exception&) {
    Py_RETURN_NONE;
  }
}

constexpr const char* kStampsName = "_fm_bind.stamps";

void stamps_free(PyObject* capsule) {
  delete static_cast<std::vector<Stamp>*>(PyCapsule_GetPointer(capsule, kStampsName));
}

// stamps(*tensors) -> an object for still().
PyObject* stamps(PyObject*, PyObject* const* a, Py_ssize_t n) {
  try {
    auto made = std::make_unique<std::vector<Stamp>>();
    for (Py_ssize_t i = 0; i < n; ++i) {
      if (!THPVariable_Check(a[i])) {
        PyErr_SetString(PyExc_TypeError, "stamps(*tensors)");
        return nullptr;
      }
      made->emplace_back(THPVariable_Unpack(a[i]));
    }
    PyObject* capsule = PyCapsule_New(made.get(), kStampsName, stamps_free);
    if (capsule != nullptr) made.release();
    return capsule;
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

// still(stamps, *tensors) -> whether these are the stamped tensors, unchanged.
PyObject* still(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n < 1) {
    PyErr_SetString(PyExc_TypeError, "still(stamps, *tensors)");
    return nullptr;
  }
  const auto* seen = static_cast<const std::vector<Stamp>*>(PyCapsule_GetPointer(a[0], kStampsName));
  if (seen == nullptr) return nullptr;
  if (static_cast<Py_ssize_t>(seen->size()) != n - 1) Py_RETURN_FALSE;
  try {
    for (Py_ssize_t i = 1; i < n; ++i)
      if (!THPVariable_Check(a[i]) || !(*seen)[i - 1].still(THPVariable_Unpack(a[i]))) Py_RETURN_FALSE;
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
  Py_RETURN_TRUE;
}

template <PyObject* (*kFn)(PyObject*, PyObject* const*, Py_ssize_t)>
PyCFunction fast_call() {
  return reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(kFn));
}

PyMethodDef methods[] = {
    {"stamps", fast_call<stamps>(), METH_FASTCALL, "stamps(*tensors) -> what their contents are known by"},
    {"still", fast_call<still>(), METH_FASTCALL, "still(stamps, *tensors) -> whether these are the stamped tensors, unchanged"},
    {"layer_forward", fast_call<layer_forward>(), METH_FASTCALL,
     "layer_forward(plan, x, cos, sin, ring_k, ring_v, layer, past) -> tensor, an int (native status), or None (not the ordinary case)"},
    {"conv_frames", fast_call<guarded<conv_frames_checked>>(), METH_FASTCALL,
     "conv_frames(x, w_hi, w_lo, kernel, stride, status) -> tensor, (name, native status), or None (not the ordinary case)"},
    {"rvq_encode", fast_call<guarded<rvq_encode_checked>>(), METH_FASTCALL,
     "rvq_encode(embeddings, w_hi, w_lo, stacks, tau_rel, status) -> codes, a status word, (name, native status), or None (not the ordinary case)"},
    {"rvq_decode_project", fast_call<guarded<rvq_decode_project_checked>>(), METH_FASTCALL,
     "rvq_decode_project(codes, books0, books1, w_hi, w_lo, status) -> (tensor, status word, bad code), (name, native status), or None (not the ordinary case)"},
    {"upsample", fast_call<guarded<upsample_checked>>(), METH_FASTCALL,
     "upsample(x, weight) -> tensor, (name, native status), or None (not the ordinary case)"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fm_bind", "host side of the native calls", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__fm_bind(void) {
  plan_type.tp_name = "_fm_bind.LayerPlan";
  plan_type.tp_basicsize = sizeof(LayerPlan);
  plan_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
  plan_type.tp_new = plan_new;
  plan_type.tp_dealloc = plan_dealloc;
  plan_type.tp_traverse = plan_traverse;
  plan_type.tp_clear = plan_clear;
  if (PyType_Ready(&plan_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module);
  if (m == nullptr) return nullptr;
  Py_INCREF(&plan_type);
  if (PyModule_AddObject(m, "LayerPlan", reinterpret_cast<PyObject*>(&plan_type)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
