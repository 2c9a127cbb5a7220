// Host path of the modules as native code. A decode-sized call is 20 to 50 us of GPU work; the
// same call prepared in Python (pointers of 4 E parameters compared, views of the workspace, ctypes)
// took 100 us and more, so the GPU waited for its host. Here one method call checks that nothing
// the call was prepared for has changed, allocates the outputs and launches.
//
// Division of labour: the Python modules prepare (validation with error messages, plan, workspace,
// merged LoRA weights) and bind() the result; forward() answers from what is bound, or returns None
// for every call that differs from it in any way, and the Python side then prepares again.
// What is bound is found changed by identity: the module tree's own dictionaries must still hold
// the same submodules and parameters, and every parameter the same storage.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <string>
#include <vector>

#include "../../../include/moe_b200.h"
#include "../internal.h"

namespace {

using at::Tensor;

PyObject* g_error = nullptr;    // gemmallm_b200._cabi.MoeB200Error
PyObject* s_weight = nullptr;
PyObject* s_bias = nullptr;
PyObject* s_parameters = nullptr;
PyObject* s_eps = nullptr;

PyObject* fail(int rc, const char* what) {
  if (g_error == nullptr) {
    PyObject* m = PyImport_ImportModule("gemmallm_b200._cabi");
    if (m == nullptr) return nullptr;
    g_error = PyObject_GetAttrString(m, "MoeB200Error");
    Py_DECREF(m);
    if (g_error == nullptr) return nullptr;
  }
  PyErr_Format(g_error, "%s failed with code %d: %s", what, rc, moe_b200_last_error_string());
  return nullptr;
}

// One entry of the module tree a bound call depends on: dict[key] must still be `value`.
struct Watch {
  PyObject* dict;
  PyObject* key;
  PyObject* value;
  const void* data;      // parameters: storage address; nullptr for submodules
};

class WatchList {
 public:
  ~WatchList() { clear(); }
  void clear() {
    for (Watch& w : items_) {
      Py_DECREF(w.dict);
      Py_DECREF(w.key);
      Py_DECREF(w.value);
    }
    items_.clear();
    params_.clear();
  }
  // seq: a list of (dict, key) pairs; tensors become parameters, in order
  bool bind(PyObject* seq) {
    clear();
    const Py_ssize_t n = PyList_Size(seq);
    if (n < 0) return false;
    items_.reserve(n);
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject *dict, *key;
      if (!PyArg_ParseTuple(PyList_GET_ITEM(seq, i), "O!O", &PyDict_Type, &dict, &key)) return false;
      PyObject* v = PyDict_GetItemWithError(dict, key);
      if (v == nullptr) {
        if (!PyErr_Occurred()) PyErr_SetObject(PyExc_KeyError, key);
        return false;
      }
      Py_INCREF(dict);
      Py_INCREF(key);
      Py_INCREF(v);
      const bool tensor = THPVariable_Check(v);
      items_.push_back(Watch{dict, key, v, tensor ? THPVariable_Unpack(v).const_data_ptr() : nullptr});
      if (tensor) params_.push_back((int)items_.size() - 1);
    }
    return true;
  }
  bool unchanged() const {
    for (const Watch& w : items_) {
      if (PyDict_GetItemWithError(w.dict, w.key) != w.value) {
        PyErr_Clear();
        return false;
      }
      if (w.data != nullptr && THPVariable_Unpack(w.value).const_data_ptr() != w.data) return false;
    }
    return true;
  }
  const Tensor& param(int i) const { return THPVariable_Unpack(items_[params_[i]].value); }
  int num_params() const { return (int)params_.size(); }
  bool empty() const { return items_.empty(); }

 private:
  std::vector<Watch> items_;
  std::vector<int> params_;
};

// A Linear with its LoRA pair, merged again whenever one of the six tensors was written since
// (torch's version counters): indices of weight, bias, a.weight, a.bias, b.weight, b.bias.
struct LoraJob {
  int p[6];
  int64_t version[6];
  double scale;
  int out_f, in_f, rank;
  void* out_w;
  void* out_b;
};

class LoraJobs {
 public:
  bool bind(PyObject* seq, const WatchList& w) {
    jobs_.clear();
    if (seq == Py_None) return true;
    const Py_ssize_t n = PyList_Size(seq);
    if (n < 0) return false;
    for (Py_ssize_t i = 0; i < n; ++i) {
      LoraJob j;
      unsigned long long ow, ob;
      if (!PyArg_ParseTuple(PyList_GET_ITEM(seq, i), "iiiiiidiiiKK", &j.p[0], &j.p[1], &j.p[2], &j.p[3], &j.p[4],
                            &j.p[5], &j.scale, &j.out_f, &j.in_f, &j.rank, &ow, &ob))
        return false;
      j.out_w = reinterpret_cast<void*>(ow);
      j.out_b = reinterpret_cast<void*>(ob);
      for (int q = 0; q < 6; ++q) {
        if (j.p[q] < 0 || j.p[q] >= w.num_params()) {
          PyErr_SetString(PyExc_IndexError, "parameter index");
          return false;
        }
        j.version[q] = (int64_t)w.param(j.p[q])._version();
      }
      jobs_.push_back(j);
    }
    return true;
  }
  int refresh(const WatchList& w, int dtype, void* stream) {
    for (LoraJob& j : jobs_) {
      bool stale = false;
      for (int q = 0; q < 6; ++q) {
        const int64_t v = (int64_t)w.param(j.p[q])._version();
        stale |= v != j.version[q];
        j.version[q] = v;
      }
      if (!stale) continue;
      const int rc = moe_b200_lora_merge(
          w.param(j.p[0]).const_data_ptr(), w.param(j.p[1]).const_data_ptr(), w.param(j.p[2]).const_data_ptr(),
          w.param(j.p[3]).const_data_ptr(), w.param(j.p[4]).const_data_ptr(), w.param(j.p[5]).const_data_ptr(),
          (float)j.scale, j.out_f, j.in_f, j.rank, dtype, j.out_w, j.out_b, stream);
      if (rc != 0) {
        j.version[0] = -1;
        return rc;
      }
    }
    return 0;
  }

 private:
  std::vector<LoraJob> jobs_;
};

at::ScalarType scalar_of(int dtype) { return dtype == MOE_B200_BF16 ? at::kBFloat16 : at::kFloat; }

// ---- the Mixture-of-Experts block ------------------------------------------------------------

struct Block {
  PyObject_HEAD
  WatchList* watch;       // [0], [1]: the router's weight and bias, then the experts' tensors
  LoraJobs* lora;
  Tensor* workspace;
  const void* plan;
  void* ws_base;
  size_t ws_bytes;
  int64_t N;
  int d, f, E, k, dtype, device;
};

// The caller's LayerNorm: false when it is not an affine one over d elements of the call's dtype.
bool read_norm(PyObject* norm, int d, int dtype, int device, const void** w, const void** b, double* eps) {
  PyObject* dict = PyObject_GetAttr(norm, s_parameters);
  if (dict == nullptr) return false;
  bool ok = false;
  if (PyDict_Check(dict)) {
    PyObject* pw = PyDict_GetItemWithError(dict, s_weight);
    PyObject* pb = PyDict_GetItemWithError(dict, s_bias);
    if (pw != nullptr && pb != nullptr && THPVariable_Check(pw) && THPVariable_Check(pb)) {
      const Tensor& tw = THPVariable_Unpack(pw);
      const Tensor& tb = THPVariable_Unpack(pb);
      ok = tw.is_cuda() && tw.device().index() == device && tw.scalar_type() == scalar_of(dtype) &&
           tw.dim() == 1 && tw.size(0) == d && tw.is_contiguous() && tb.is_cuda() &&
           tb.device().index() == device && tb.scalar_type() == scalar_of(dtype) && tb.dim() == 1 &&
           tb.size(0) == d && tb.is_contiguous();
      if (ok) {
        *w = tw.const_data_ptr();
        *b = tb.const_data_ptr();
      }
    }
  }
  Py_DECREF(dict);
  if (!ok) return false;
  PyObject* e = PyObject_GetAttr(norm, s_eps);
  if (e == nullptr) return false;
  *eps = PyFloat_AsDouble(e);
  Py_DECREF(e);
  return !PyErr_Occurred();
}

PyObject* block_new(PyTypeObject* type, PyObject*, PyObject*) {
  Block* self = reinterpret_cast<Block*>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  self->watch = new WatchList();
  self->lora = new LoraJobs();
  self->workspace = new Tensor();
  return reinterpret_cast<PyObject*>(self);
}

void block_dealloc(PyObject* o) {
  Block* self = reinterpret_cast<Block*>(o);
  PyTypeObject* type = Py_TYPE(o);
  delete self->watch;
  delete self->lora;
  delete self->workspace;
  type->tp_free(o);
  Py_DECREF(type);
}

// bind(watch, lora or None, plan, workspace tensor, base, bytes, N, d, f, E, k, dtype, device index)
PyObject* block_bind(PyObject* o, PyObject* args) {
  HANDLE_TH_ERRORS
  Block* self = reinterpret_cast<Block*>(o);
  PyObject *watch, *lora, *ws;
  unsigned long long plan, base, bytes;
  long long N;
  int d, f, E, k, dtype, device;
  if (!PyArg_ParseTuple(args, "O!OKOKKLiiiiii", &PyList_Type, &watch, &lora, &plan, &ws, &base, &bytes, &N, &d, &f,
                        &E, &k, &dtype, &device))
    return nullptr;
  if (!THPVariable_Check(ws)) {
    PyErr_SetString(PyExc_TypeError, "workspace must be a tensor");
    return nullptr;
  }
  if (!self->watch->bind(watch) || !self->lora->bind(lora, *self->watch)) {
    self->watch->clear();
    return nullptr;
  }
  *self->workspace = THPVariable_Unpack(ws);
  self->plan = reinterpret_cast<const void*>(plan);
  self->ws_base = reinterpret_cast<void*>(base);
  self->ws_bytes = (size_t)bytes;
  self->N = N;
  self->d = d;
  self->f = f;
  self->E = E;
  self->k = k;
  self->dtype = dtype;
  self->device = device;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* block_unbind(PyObject* o, PyObject*) {
  Block* self = reinterpret_cast<Block*>(o);
  self->watch->clear();
  *self->workspace = Tensor();
  Py_RETURN_NONE;
}

// a contiguous tensor of the bound device, dtype and row width with n rows
bool rows_match(const Tensor& t, int device, int dtype, int d, int64_t n) {
  return t.is_cuda() && t.device().index() == device && t.scalar_type() == scalar_of(dtype) && t.dim() >= 1 &&
         t.size(-1) == d && t.numel() == n * d && t.is_contiguous();
}

// forward(tensor, residual or None, norm or None) -> (out, loss), or None: prepare again
PyObject* block_forward(PyObject* o, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Block* self = reinterpret_cast<Block*>(o);
  if (nargs != 3) {
    PyErr_SetString(PyExc_TypeError, "forward(tensor, residual, norm)");
    return nullptr;
  }
  if (self->watch->empty() || !THPVariable_Check(args[0])) Py_RETURN_NONE;
  const Tensor& x = THPVariable_Unpack(args[0]);
  if (self->N <= 0 || !rows_match(x, self->device, self->dtype, self->d, self->N)) Py_RETURN_NONE;
  const void* res = nullptr;
  if (args[1] != Py_None) {
    if (!THPVariable_Check(args[1])) Py_RETURN_NONE;
    const Tensor& r = THPVariable_Unpack(args[1]);
    if (!rows_match(r, self->device, self->dtype, self->d, self->N) || r.sizes() != x.sizes()) Py_RETURN_NONE;
    res = r.const_data_ptr();
  }
  const void *nw = nullptr, *nb = nullptr;
  double eps = 0.0;
  if (args[2] != Py_None && !read_norm(args[2], self->d, self->dtype, self->device, &nw, &nb, &eps)) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (!self->watch->unchanged()) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
  void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream();
  int rc = self->lora->refresh(*self->watch, self->dtype, stream);
  if (rc != 0) return fail(rc, "lora_merge");
  Tensor out = at::empty(x.sizes(), x.options());
  Tensor aux = at::empty({}, x.options().dtype(at::kFloat));
  rc = moe::forward_into(x.const_data_ptr(), self->watch->param(0).const_data_ptr(),
                         self->watch->param(1).const_data_ptr(), self->plan, res, nw, nb, (float)eps, self->N,
                         self->d, self->f, self->E, self->k, self->dtype, MOE_B200_FLAG_WS_CLEAN, self->ws_base,
                         self->ws_bytes, out.data_ptr(), aux.data_ptr<float>(), stream);
  if (rc != 0) return fail(rc, "forward");
  PyObject* t = PyTuple_New(2);
  if (t == nullptr) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(aux)));
  return t;
  END_HANDLE_TH_ERRORS
}

// a copy or an unpickled module starts unbound
PyObject* fresh_reduce(PyObject* o, PyObject*) { return Py_BuildValue("O()", (PyObject*)Py_TYPE(o)); }

PyMethodDef block_methods[] = {
    {"bind", block_bind, METH_VARARGS, nullptr},
    {"unbind", block_unbind, METH_NOARGS, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(block_forward)), METH_FASTCALL, nullptr},
    {"__reduce__", fresh_reduce, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyType_Slot block_slots[] = {{Py_tp_new, reinterpret_cast<void*>(block_new)},
                             {Py_tp_dealloc, reinterpret_cast<void*>(block_dealloc)},
                             {Py_tp_methods, block_methods},
                             {0, nullptr}};
PyType_Spec block_spec = {"gemmallm_b200._host.Block", sizeof(Block), 0, Py_TPFLAGS_DEFAULT, block_slots};

// ---- the dense feed-forward ------------------------------------------------------------------

struct Ffn {
  PyObject_HEAD
  WatchList* watch;
  LoraJobs* lora;
  Tensor* offsets;        // int32 [0, M]
  Tensor* status;         // int32 [16], written only when a wait inside a kernel ran out
  const void* plan;
  int64_t M;
  int d, f, dtype, device;
};

PyObject* ffn_new(PyTypeObject* type, PyObject*, PyObject*) {
  Ffn* self = reinterpret_cast<Ffn*>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  self->watch = new WatchList();
  self->lora = new LoraJobs();
  self->offsets = new Tensor();
  self->status = new Tensor();
  return reinterpret_cast<PyObject*>(self);
}

void ffn_dealloc(PyObject* o) {
  Ffn* self = reinterpret_cast<Ffn*>(o);
  PyTypeObject* type = Py_TYPE(o);
  delete self->watch;
  delete self->lora;
  delete self->offsets;
  delete self->status;
  type->tp_free(o);
  Py_DECREF(type);
}

// bind(watch, lora or None, plan, offsets, status, M, d, f, dtype, device index)
PyObject* ffn_bind(PyObject* o, PyObject* args) {
  HANDLE_TH_ERRORS
  Ffn* self = reinterpret_cast<Ffn*>(o);
  PyObject *watch, *lora, *offsets, *status;
  unsigned long long plan;
  long long M;
  int d, f, dtype, device;
  if (!PyArg_ParseTuple(args, "O!OKOOLiiii", &PyList_Type, &watch, &lora, &plan, &offsets, &status, &M, &d, &f,
                        &dtype, &device))
    return nullptr;
  if (!THPVariable_Check(offsets) || !THPVariable_Check(status)) {
    PyErr_SetString(PyExc_TypeError, "offsets and status must be tensors");
    return nullptr;
  }
  if (!self->watch->bind(watch) || !self->lora->bind(lora, *self->watch)) {
    self->watch->clear();
    return nullptr;
  }
  *self->offsets = THPVariable_Unpack(offsets);
  *self->status = THPVariable_Unpack(status);
  self->plan = reinterpret_cast<const void*>(plan);
  self->M = M;
  self->d = d;
  self->f = f;
  self->dtype = dtype;
  self->device = device;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* ffn_unbind(PyObject* o, PyObject*) {
  reinterpret_cast<Ffn*>(o)->watch->clear();
  Py_RETURN_NONE;
}

// forward(tensor) -> y, or None: prepare again
PyObject* ffn_forward(PyObject* o, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Ffn* self = reinterpret_cast<Ffn*>(o);
  if (nargs != 1) {
    PyErr_SetString(PyExc_TypeError, "forward(tensor)");
    return nullptr;
  }
  if (self->watch->empty() || self->M <= 0 || !THPVariable_Check(args[0])) Py_RETURN_NONE;
  const Tensor& x = THPVariable_Unpack(args[0]);
  if (!rows_match(x, self->device, self->dtype, self->d, self->M) || !self->watch->unchanged()) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
  void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream();
  int rc = self->lora->refresh(*self->watch, self->dtype, stream);
  if (rc != 0) return fail(rc, "lora_merge");
  Tensor h = at::empty({self->M, self->f}, x.options());
  Tensor y = at::empty(x.sizes(), x.options());
  rc = moe_b200_experts(x.const_data_ptr(), self->offsets->const_data_ptr<int32_t>(), self->plan, self->M, self->d,
                        self->f, 1, self->dtype, 0, h.data_ptr(), y.data_ptr(), self->status->data_ptr<int32_t>(),
                        stream);
  if (rc != 0) return fail(rc, "experts");
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyMethodDef ffn_methods[] = {
    {"bind", ffn_bind, METH_VARARGS, nullptr},
    {"unbind", ffn_unbind, METH_NOARGS, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(ffn_forward)), METH_FASTCALL, nullptr},
    {"__reduce__", fresh_reduce, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyType_Slot ffn_slots[] = {{Py_tp_new, reinterpret_cast<void*>(ffn_new)},
                           {Py_tp_dealloc, reinterpret_cast<void*>(ffn_dealloc)},
                           {Py_tp_methods, ffn_methods},
                           {0, nullptr}};
PyType_Spec ffn_spec = {"gemmallm_b200._host.Ffn", sizeof(Ffn), 0, Py_TPFLAGS_DEFAULT, ffn_slots};

PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, nullptr, nullptr, nullptr, nullptr, nullptr};

bool add_type(PyObject* m, const char* name, PyType_Spec* spec) {
  PyObject* t = PyType_FromSpec(spec);
  if (t == nullptr) return false;
  const int rc = PyModule_AddObjectRef(m, name, t);
  Py_DECREF(t);
  return rc == 0;
}

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&module_def);
  if (m == nullptr) return nullptr;
  s_weight = PyUnicode_InternFromString("weight");
  s_bias = PyUnicode_InternFromString("bias");
  s_parameters = PyUnicode_InternFromString("_parameters");
  s_eps = PyUnicode_InternFromString("eps");
  if (!add_type(m, "Block", &block_spec) || !add_type(m, "Ffn", &ffn_spec)) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
