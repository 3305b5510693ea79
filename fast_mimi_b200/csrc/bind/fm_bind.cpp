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
