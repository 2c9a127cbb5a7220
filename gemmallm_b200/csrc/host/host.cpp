// Host path of the modules as native code. A decode-sized call is 20 to 50 us of GPU work; the
// same call prepared in Python (pointers of 4 E parameters compared, views of the workspace, ctypes)
// took 100 us and more, so the GPU waited for its host. Here one method call checks that nothing
// the call was prepared for has changed, allocates the outputs and launches.
//
// Division of labour: the Python modules prepare (validation with error messages, plan, workspace,
// merged LoRA weights) and bind() the result; forward() answers from what is bound, or returns None
// for every call that differs from it in any way, and the Python side then prepares again.
// What is bound is found changed by identity: the module tree's own dictionaries must still hold
// the same submodules, parameters and plain attributes (scales of experts), and every parameter the same storage. Plain
// attributes of the module itself come with the call: a binding that held its module's dictionary would keep the
// module, and the memory of its weights, until the garbage collector ran.
//
// Lifetime: a bound call owns every buffer whose address it has (plan, workspaces, merged weights): the Python side may
// replace its own, and the parameters may leave and come back (weights exchanged for an evaluation) with the binding
// still in place. Of merged weights there is one record of what they hold, kept with them. The parameters themselves it does not own, so that moving a module away frees them; an autograd node
// does, from its forward to its backward, because the plan that it will use has their addresses.
#include <Python.h>
#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <algorithm>
#include <memory>
#include <mutex>
#include <string>
#include <tuple>
#include <utility>
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
PyObject* s_normalized_shape = nullptr;

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
  const void* data;      // parameters: storage address; nullptr for submodules and plain attributes
};

class WatchList {
 public:
  ~WatchList() { clear(); }
  void clear() {
    std::vector<Watch> old;
    old.swap(items_);
    params_.clear();
    for (Watch& w : old) {
      Py_DECREF(w.dict);
      Py_DECREF(w.key);
      Py_DECREF(w.value);
    }
  }
  // seq: a list of (dict, key) pairs; tensors become parameters, in order. Nothing is bound after an error.
  bool bind(PyObject* seq) {
    bool ok = false;
    try {
      ok = fill(seq);
    } catch (...) {      // a parameter without an address
      clear();
      throw;
    }
    if (!ok) clear();
    return ok;
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
  int traverse(visitproc visit, void* arg) const {
    for (const Watch& w : items_) {
      Py_VISIT(w.dict);
      Py_VISIT(w.key);
      Py_VISIT(w.value);
    }
    return 0;
  }
  const Tensor& param(int i) const { return THPVariable_Unpack(items_[params_[i]].value); }
  int num_params() const { return (int)params_.size(); }
  bool empty() const { return items_.empty(); }

 private:
  bool fill(PyObject* seq) {
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
      const bool tensor = THPVariable_Check(v);
      items_.push_back(Watch{dict, key, v, tensor ? THPVariable_Unpack(v).const_data_ptr() : nullptr});
      Py_INCREF(dict);
      Py_INCREF(key);
      Py_INCREF(v);
      if (tensor) params_.push_back((int)items_.size() - 1);
    }
    return true;
  }
  std::vector<Watch> items_;
  std::vector<int> params_;
};

bool tensor_list(PyObject* seq, std::vector<Tensor>* out) {
  out->clear();
  const Py_ssize_t n = PyList_Size(seq);
  if (n < 0) return false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* t = PyList_GET_ITEM(seq, i);
    if (!THPVariable_Check(t)) {
      PyErr_SetString(PyExc_TypeError, "a list of tensors is needed");
      return false;
    }
    out->push_back(THPVariable_Unpack(t));
  }
  return true;
}

bool float_list(PyObject* seq, std::vector<double>* out) {
  out->clear();
  const Py_ssize_t n = PyList_Size(seq);
  if (n < 0) return false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    out->push_back(PyFloat_AsDouble(PyList_GET_ITEM(seq, i)));
    if (PyErr_Occurred()) return false;
  }
  return true;
}

// A parameter as a call finds it: its address, the storage that keeps it alive, and torch's version counter.
struct Held {
  c10::Storage storage;
  const void* data;
  c10::VariableVersion version;
  explicit Held(const Tensor& t)
      : storage(t.storage()), data(t.const_data_ptr()), version(t.unsafeGetTensorImpl()->version_counter()) {}
};

// Merged copies W' = W + s B A, b' = b + s (B a + b_lora) of the two Linears of a list of experts, and the one record of
// what they hold: storages, addresses, versions and scale of the last merge (weak references: an address alone may have
// been given to other weights since, and weights that were moved away must be freed). Every call that reads them, bound or not, forward
// or backward, compares its own parameters with that record first, so that adapters that were exchanged in between, by
// whichever call, are merged again. Parameters are counted as in moe.py: twelve an expert.
class Merged {
 public:
  bool fill(PyObject* seq) {
    const Py_ssize_t n = PyList_Size(seq);
    if (n < 0) return false;
    for (Py_ssize_t i = 0; i < n; ++i) {
      Job j;
      PyObject *w, *b;
      if (!PyArg_ParseTuple(PyList_GET_ITEM(seq, i), "iiiOO", &j.out_f, &j.in_f, &j.rank, &w, &b)) return false;
      if (!THPVariable_Check(w) || !THPVariable_Check(b)) {
        PyErr_SetString(PyExc_TypeError, "merged weights must be tensors");
        return false;
      }
      j.w = THPVariable_Unpack(w);
      j.b = THPVariable_Unpack(b);
      jobs_.push_back(std::move(j));
    }
    return true;
  }
  size_t num_params() const { return jobs_.size() * 6; }
  // param(i) -> (address, version, storage) of the i-th parameter; scale of every expert
  template <typename Param>
  int refresh(Param param, const std::vector<double>& scales, int dtype, void* stream) {
    const std::lock_guard<std::mutex> lock(mutex_);      // a backward runs on another thread
    std::vector<moe::LoraMerge> todo;
    std::vector<Job*> jobs;
    for (size_t i = 0; i < jobs_.size(); ++i) {
      Job& j = jobs_[i];
      const size_t first = i / 2 * 12, l = i % 2;
      // weight, bias, a.weight, a.bias, b.weight, b.bias
      const size_t at[6] = {first + 2 * l, first + 2 * l + 1, first + 4 + 4 * l, first + 5 + 4 * l, first + 6 + 4 * l,
                            first + 7 + 4 * l};
      const void* data[6];
      int64_t version[6];
      const c10::Storage* storage[6];
      bool same = j.valid && j.scale == scales[i / 2];
      for (int q = 0; q < 6; ++q) {
        std::tie(data[q], version[q], storage[q]) = param(at[q]);
        same = same && data[q] == j.data[q] && version[q] == j.version[q] &&
               storage[q]->unsafeGetStorageImpl() == j.storage[q]._unsafe_get_target();
      }
      if (same) continue;
      j.valid = false;
      todo.push_back({data[0], data[1], data[2], data[3], data[4], data[5], j.w.data_ptr(), j.b.data_ptr(),
                      (float)scales[i / 2], j.out_f, j.in_f, j.rank});
      jobs.push_back(&j);
      std::copy(data, data + 6, j.data);
      std::copy(version, version + 6, j.version);
      j.storage.clear();
      for (const c10::Storage* s : storage) j.storage.push_back(s->getWeakStorageImpl());
      j.scale = scales[i / 2];
    }
    if (todo.empty()) return 0;
    const int rc = moe::lora_merges(todo.data(), (int)todo.size(), dtype, stream);
    for (Job* j : jobs) j->valid = rc == 0;
    return rc;
  }

 private:
  struct Job {
    Tensor w, b;
    int out_f = 0, in_f = 0, rank = 0;
    bool valid = false;
    const void* data[6];
    int64_t version[6];
    std::vector<c10::weak_intrusive_ptr<c10::StorageImpl>> storage;
    double scale = 0.0;
  };
  std::vector<Job> jobs_;
  std::mutex mutex_;
};

// What a bound call has of it; nothing without LoRA branches.
struct MergedUse {
  std::shared_ptr<Merged> merged;
  std::vector<double> scales;
  size_t first = 0;       // place of the first expert's parameters among the call's

  bool has_scale(double scale) const { return merged == nullptr || scales[0] == scale; }      // of the only expert

  int refresh(const WatchList& w, int dtype, void* stream) const {
    if (merged == nullptr) return 0;
    return merged->refresh(
        [&](size_t i) {
          const Tensor& t = w.param((int)(first + i));
          return std::make_tuple(t.const_data_ptr(), (int64_t)t._version(), &t.storage());
        },
        scales, dtype, stream);
  }
  int refresh(const std::vector<Held>& h, int dtype, void* stream) const {
    if (merged == nullptr) return 0;
    return merged->refresh(
        [&](size_t i) {
          const Held& p = h[first + i];
          return std::make_tuple(p.data, (int64_t)p.version.current_version(), &p.storage);
        },
        scales, dtype, stream);
  }
};

struct MergedObject {
  PyObject_HEAD
  std::shared_ptr<Merged>* merged;
};

PyTypeObject* g_merged_type = nullptr;

// Merged([(out, in, rank, W', b')]): gate_and_up and down of every expert
PyObject* merged_new(PyTypeObject* type, PyObject* args, PyObject*) {
  HANDLE_TH_ERRORS
  PyObject* jobs;
  if (!PyArg_ParseTuple(args, "O!", &PyList_Type, &jobs)) return nullptr;
  auto m = std::make_shared<Merged>();
  if (!m->fill(jobs)) return nullptr;
  MergedObject* self = reinterpret_cast<MergedObject*>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  self->merged = new std::shared_ptr<Merged>(std::move(m));
  return reinterpret_cast<PyObject*>(self);
  END_HANDLE_TH_ERRORS
}

void merged_dealloc(PyObject* o) {
  PyTypeObject* type = Py_TYPE(o);
  delete reinterpret_cast<MergedObject*>(o)->merged;
  type->tp_free(o);
  Py_DECREF(type);
}

// refresh(parameters, scales, dtype, device index)
PyObject* merged_refresh(PyObject* o, PyObject* args) {
  HANDLE_TH_ERRORS
  PyObject *params, *scales;
  int dtype, device;
  if (!PyArg_ParseTuple(args, "O!O!ii", &PyList_Type, &params, &PyList_Type, &scales, &dtype, &device)) return nullptr;
  Merged& m = **reinterpret_cast<MergedObject*>(o)->merged;
  std::vector<Tensor> t;
  std::vector<double> s;
  if (!tensor_list(params, &t) || !float_list(scales, &s)) return nullptr;
  if (t.size() != m.num_params() || s.size() * 12 != t.size()) {
    PyErr_SetString(PyExc_ValueError, "twelve parameters and a scale for every expert");
    return nullptr;
  }
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
  void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream();
  const int rc = m.refresh(
      [&](size_t i) { return std::make_tuple(t[i].const_data_ptr(), (int64_t)t[i]._version(), &t[i].storage()); }, s, dtype,
      stream);
  if (rc != 0) return fail(rc, "lora_merge");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// (merged or None, scales) of a bind(); `params`: how many parameters the call has, the first expert's at `first`
bool read_merged(PyObject* merged, PyObject* scales, size_t first, size_t params, MergedUse* out) {
  *out = MergedUse();
  if (merged == Py_None) return true;
  if (!PyObject_TypeCheck(merged, g_merged_type)) {
    PyErr_SetString(PyExc_TypeError, "merged must be a Merged");
    return false;
  }
  if (!float_list(scales, &out->scales)) return false;
  out->merged = *reinterpret_cast<MergedObject*>(merged)->merged;
  out->first = first;
  // params is 0 for a module tree that cannot be watched: its calls never refresh from the watched parameters
  if (out->scales.size() * 12 != out->merged->num_params() ||
      (params != 0 && params != first + out->merged->num_params())) {
    PyErr_SetString(PyExc_ValueError, "twelve parameters and a scale for every expert");
    return false;
  }
  return true;
}

// ---- training -----------------------------------------------------------------------------------
// The forward of a module under .train() as one autograd node, without Python on either way: the node keeps
// what its backward needs (the prepared call, the input, the call's seed) and hands every gradient that is wanted
// a place of its own, so that nothing is copied out of a workspace afterwards.

using torch::autograd::Edge;
using torch::autograd::edge_list;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

// Number of forwards on a training workspace, of all bindings that share it: a backward must belong to the last.
struct Generation {
  PyObject_HEAD
  std::shared_ptr<int64_t>* count;
};

PyObject* generation_new(PyTypeObject* type, PyObject*, PyObject*) {
  Generation* self = reinterpret_cast<Generation*>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  self->count = new std::shared_ptr<int64_t>(std::make_shared<int64_t>(0));
  return reinterpret_cast<PyObject*>(self);
}

void generation_dealloc(PyObject* o) {
  PyTypeObject* type = Py_TYPE(o);
  delete reinterpret_cast<Generation*>(o)->count;
  type->tp_free(o);
  Py_DECREF(type);
}

PyTypeObject* g_generation_type = nullptr;

bool read_generation(PyObject* o, std::shared_ptr<int64_t>* out) {
  if (!PyObject_TypeCheck(o, g_generation_type)) {
    PyErr_SetString(PyExc_TypeError, "generation must be a Generation");
    return false;
  }
  *out = *reinterpret_cast<Generation*>(o)->count;
  return true;
}

// What a prepared training call works on; shared by the module and the nodes of its calls.
struct TrainCall {
  Tensor ws, tws, offsets, status, lora_tab;    // buffers kept alive
  std::vector<Tensor> owned;                    // the plan likewise
  MergedUse lora;
  const void* plan = nullptr;
  void *ws_base = nullptr, *tws_base = nullptr;
  size_t ws_bytes = 0, tws_bytes = 0;
  int64_t N = 0;
  int d = 0, f = 0, E = 0, k = 0, device = 0;
  std::vector<int> ranks;      // of gate_and_up and down of every expert; empty without LoRA branches
  std::shared_ptr<int64_t> gen;
};

uint64_t draw_seed() {      // torch's CPU generator, as torch.randint(0, 2**62, (1,)) in Python
  return (uint64_t)at::randint((int64_t)1 << 62, {1}, at::TensorOptions().dtype(at::kLong)).item<int64_t>();
}

// From a backward pass, on a thread that does not hold the GIL: the same MoeB200Error.
void check_rc(int rc, const char* what) {
  if (rc == 0) return;
  const PyGILState_STATE gil = PyGILState_Ensure();
  python_error e;
  fail(rc, what);
  e.persist();
  PyGILState_Release(gil);
  throw e;
}

// Gradients of the experts' parameters: per expert w1, b1, w2, b2 and, with LoRA, weight and bias of
// gate_and_up a, b and down a, b; `wanted(i)` says whether the i-th of them (counted over the experts) is.
struct ExpertGrads {
  Tensor w1, b1, w2, b2, scratch;
  std::vector<Tensor> lora;      // eight an expert
  moe::LoraGrads lora_args = {};
  int per = 4;

  // the arguments of the pass; LoRA gradients are wanted if lora_args has runs
  template <typename Wanted>
  void prepare(const TrainCall& c, const at::TensorOptions& opt, moe::TrainGrads* g, Wanted wanted) {
    const int64_t E = c.E, d = c.d, f = c.f;
    per = c.ranks.empty() ? 4 : 12;
    bool need[12] = {};
    for (int64_t e = 0; e < E; ++e)
      for (int i = 0; i < per; ++i) need[i] |= wanted(e * per + i);
    bool with_lora = false;
    for (int i = 4; i < per; ++i) with_lora |= need[i];
    // (what the LoRA gradients need of these and nobody wants lies in the training workspace)
    if (need[0]) w1 = at::empty({E, 2 * f, d}, opt);
    if (need[1]) b1 = at::empty({E, 2 * f}, opt);
    if (need[2]) w2 = at::empty({E, d, f}, opt);
    if (need[3]) b2 = at::empty({E, d}, opt);
    auto ptr = [](Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; };
    g->w1 = ptr(w1);
    g->b1 = ptr(b1);
    g->w2 = ptr(w2);
    g->b2 = ptr(b2);
    if (!with_lora) return;
    // experts of one rank and scale, which is all of them unless someone replaced some, in one run
    bool alike = true;
    for (int64_t e = 1; e < E; ++e)
      alike = alike && c.ranks[2 * e] == c.ranks[0] && c.ranks[2 * e + 1] == c.ranks[1] && c.lora.scales[e] == c.lora.scales[0];
    const int64_t ne = alike ? E : 1;
    lora.resize(8 * E);
    size_t floats = 0;
    const int64_t in[2] = {d, f}, out[2] = {2 * f, d};
    for (int64_t e0 = 0; e0 < E; e0 += ne) {
      moe::LoraRun run = {};
      run.first = (int)e0;
      run.count = (int)ne;
      run.scale = (float)c.lora.scales[e0];
      for (int l = 0; l < 2; ++l) {
        const int64_t r = run.rank[l] = c.ranks[2 * e0 + l];
        Tensor t[4] = {at::empty({ne, r, in[l]}, opt), at::empty({ne, r}, opt), at::empty({ne, out[l], r}, opt),
                       at::empty({ne, out[l]}, opt)};
        run.dA[l] = t[0].data_ptr();
        run.da[l] = t[1].data_ptr();
        run.dB[l] = t[2].data_ptr();
        run.db[l] = t[3].data_ptr();
        for (int64_t e = 0; e < ne; ++e)
          for (int q = 0; q < 4; ++q) lora[(e0 + e) * 8 + l * 4 + q] = t[q].select(0, e);
      }
      floats = std::max(floats, moe::lora_grads_scratch_floats(c.d, c.f, run));
      lora_args.runs.push_back(run);
    }
    scratch = at::empty({(int64_t)floats}, opt.dtype(at::kFloat));
    lora_args.tab = static_cast<const void* const*>(c.lora_tab.const_data_ptr());
    lora_args.scratch = scratch.data_ptr<float>();
  }
  const moe::LoraGrads* lora_grads() const { return per == 12 ? &lora_args : nullptr; }
  void zero() {
    for (Tensor* t : {&w1, &b1, &w2, &b2})
      if (t->defined()) t->zero_();
    for (Tensor& t : lora) t.zero_();
  }
  template <typename Wanted>
  void collect(int64_t E, variable_list* out, size_t first, Wanted wanted) {
    Tensor* base[4] = {&w1, &b1, &w2, &b2};
    for (int64_t e = 0; e < E; ++e)
      for (int i = 0; i < per; ++i)
        if (wanted(e * per + i)) (*out)[first + e * per + i] = i < 4 ? base[i]->select(0, e) : lora[e * 8 + i - 4];
  }
};

Tensor output_grad(const Tensor& g, const Tensor& like) {
  if (!g.defined()) return at::zeros_like(like);
  return g.to(like.scalar_type()).contiguous();
}

// A saved tensor of N rows of `cols`, whatever hooks made of it in between.
Tensor unpacked(const SavedVariable& v, const TrainCall& c, int64_t cols) {
  Tensor t = v.unpack();
  TORCH_CHECK(t.is_cuda() && t.device().index() == c.device && t.scalar_type() == at::kBFloat16 && t.numel() == c.N * cols,
              "a saved tensor came back with another size, dtype or device");
  return t.contiguous();
}

void check_generation(const TrainCall& c, int64_t gen) {
  if (*c.gen != gen)
    throw std::runtime_error("this module ran another training forward before the backward of this one: its "
                             "workspace holds the later call's tensors");
}

// inputs: x, residual (an empty edge without one), gate weight, gate bias, the experts' parameters
struct BlockBackward : public Node {
  std::shared_ptr<TrainCall> call;
  SavedVariable x;
  Tensor gate_w;
  std::vector<Held> weights;    // the parameters whose addresses the plan has
  int64_t gen = 0;
  uint64_t seed = 0;
  double p = 0.0;

  std::string name() const override { return "MOEBackward"; }
  void release_variables() override {
    x.reset_data();
    weights.clear();
  }
  variable_list apply(variable_list&& grads) override {
    const TrainCall& c = *call;
    check_generation(c, gen);
    at::AutoGradMode no_grad(false);
    const Tensor xv = unpacked(x, c, c.d);
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)c.device);
    void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)c.device).stream();
    const Tensor go = output_grad(grads[0], xv);
    Tensor aux = grads[1];
    if (aux.defined()) aux = aux.to(xv.options().dtype(at::kFloat)).contiguous();
    variable_list out(next_edges().size());
    const auto opt = xv.options();
    moe::TrainGrads g = {};
    Tensor gx, gwg, gbg;
    if (task_should_compute_output(0)) gx = at::empty(xv.sizes(), opt);
    if (task_should_compute_output(2)) gwg = at::empty({c.E, c.d}, opt);
    if (task_should_compute_output(3)) gbg = at::empty({c.E}, opt);
    g.x = gx.defined() ? gx.data_ptr() : nullptr;
    g.wg = gwg.defined() ? gwg.data_ptr() : nullptr;
    g.bg = gbg.defined() ? gbg.data_ptr() : nullptr;
    auto wanted = [&](int64_t i) { return task_should_compute_output(4 + (size_t)i); };
    ExpertGrads eg;
    eg.prepare(c, opt, &g, wanted);
    if (c.N > 0) {
      check_rc(c.lora.refresh(weights, MOE_B200_BF16, stream), "lora_merge");
      check_rc(moe::backward_into(xv.const_data_ptr(), gate_w.const_data_ptr(), c.plan, go.const_data_ptr(), 0.f,
                                  aux.defined() ? aux.const_data_ptr<float>() : nullptr, c.N, c.d, c.f, c.E, c.k,
                                  MOE_B200_BF16, (float)p, seed, c.ws_base, c.ws_bytes, c.tws_base, c.tws_bytes, g,
                                  eg.lora_grads(), stream),
               "backward");
    } else {
      for (Tensor* t : {&gwg, &gbg})
        if (t->defined()) t->zero_();
      eg.zero();
    }
    out[0] = gx;
    if (task_should_compute_output(1)) out[1] = grads[0].defined() ? grads[0] : go;
    out[2] = gwg;
    out[3] = gbg;
    eg.collect(c.E, &out, 4, wanted);
    return out;
  }
};

// inputs: x, the parameters
struct FfnBackward : public Node {
  std::shared_ptr<TrainCall> call;
  SavedVariable x, h;
  std::vector<Held> weights;
  int64_t gen = 0;
  uint64_t seed = 0;
  double p = 0.0;

  std::string name() const override { return "FeedForwardBackward"; }
  void release_variables() override {
    x.reset_data();
    h.reset_data();
    weights.clear();
  }
  variable_list apply(variable_list&& grads) override {
    const TrainCall& c = *call;
    check_generation(c, gen);
    at::AutoGradMode no_grad(false);
    const Tensor xv = unpacked(x, c, c.d), hv = unpacked(h, c, c.f);
    c10::cuda::CUDAGuard guard((c10::DeviceIndex)c.device);
    void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)c.device).stream();
    const Tensor go = output_grad(grads[0], xv);
    variable_list out(next_edges().size());
    const auto opt = xv.options();
    moe::TrainGrads g = {};
    Tensor gx;
    if (task_should_compute_output(0)) gx = at::empty(xv.sizes(), opt);
    g.x = gx.defined() ? gx.data_ptr() : nullptr;
    auto wanted = [&](int64_t i) { return task_should_compute_output(1 + (size_t)i); };
    ExpertGrads eg;
    eg.prepare(c, opt, &g, wanted);
    if (c.N > 0) {
      check_rc(c.lora.refresh(weights, MOE_B200_BF16, stream), "lora_merge");
      check_rc(moe::experts_backward_into(xv.const_data_ptr(), hv.const_data_ptr(), c.offsets.const_data_ptr<int32_t>(),
                                          c.plan, go.const_data_ptr(), c.N, c.d, c.f, 1, (float)p, seed, c.tws_base,
                                          c.tws_bytes, g, eg.lora_grads(), c.status.data_ptr<int32_t>(), stream),
               "experts_backward");
    } else {
      eg.zero();
    }
    out[0] = gx;
    eg.collect(1, &out, 1, wanted);
    return out;
  }
};

// Two ranks for every expert that `lora` merges.
bool read_ranks(PyObject* seq, const MergedUse& lora, std::vector<int>* out) {
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(seq); ++i) {
    out->push_back((int)PyLong_AsLong(PyList_GET_ITEM(seq, i)));
    if (PyErr_Occurred()) return false;
  }
  if (out->size() != 2 * lora.scales.size()) {
    PyErr_SetString(PyExc_ValueError, "two ranks for every expert");
    return false;
  }
  return true;
}

// Edges of a call's inputs, and those of them that are parameters.
class Edges {
 public:
  void add_param(const Tensor& t) {
    add(t);
    weights_.emplace_back(t);
  }
  void add(const Tensor& t) {
    any_ |= t.requires_grad();
    tangent_ |= t._fw_grad(0).defined();
    list_.push_back(torch::autograd::impl::gradient_edge(t));
  }
  void add_empty() { list_.emplace_back(); }
  bool wanted() const { return any_ && at::GradMode::is_enabled(); }
  // The node has no forward-mode derivative: a call on dual tensors would lose their tangents.
  void refuse_tangents() const {
    TORCH_CHECK_NOT_IMPLEMENTED(!tangent_, "training mode has no forward-mode derivative (jvp)");
  }
  edge_list take() { return std::move(list_); }
  std::vector<Held> take_weights() { return std::move(weights_); }

 private:
  edge_list list_;
  std::vector<Held> weights_;
  bool any_ = false, tangent_ = false;
};

at::ScalarType scalar_of(int dtype) { return dtype == MOE_B200_BF16 ? at::kBFloat16 : at::kFloat; }

// ---- the Mixture-of-Experts block ------------------------------------------------------------

struct Block {
  PyObject_HEAD
  WatchList* watch;       // [0], [1]: the router's weight and bias, then the experts' tensors
  MergedUse* lora;
  Tensor* workspace;
  std::vector<Tensor>* owned;     // the plan
  std::shared_ptr<TrainCall>* train;
  const void* plan;
  void* ws_base;
  size_t ws_bytes;
  int64_t N;
  int d, f, E, k, dtype, device;
};

// The caller's LayerNorm: false when it is not an affine one over d elements of the call's dtype. (normalized_shape is
// what tells it from other norms with d weights, which would be taken for one otherwise.)
bool read_norm(PyObject* norm, int d, int dtype, int device, const void** w, const void** b, double* eps) {
  PyObject* shape = PyObject_GetAttr(norm, s_normalized_shape);
  if (shape == nullptr) return false;
  const bool over_d = PyTuple_Check(shape) && PyTuple_GET_SIZE(shape) == 1 && PyLong_Check(PyTuple_GET_ITEM(shape, 0)) &&
                      PyLong_AsLong(PyTuple_GET_ITEM(shape, 0)) == d;
  Py_DECREF(shape);
  if (!over_d) return false;
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
  self->lora = new MergedUse();
  self->workspace = new Tensor();
  self->owned = new std::vector<Tensor>();
  self->train = new std::shared_ptr<TrainCall>();
  return reinterpret_cast<PyObject*>(self);
}

// (A tree whose parts refer to the module is a cycle through the binding.)
int block_traverse(PyObject* o, visitproc visit, void* arg) {
  Py_VISIT(Py_TYPE(o));
  const WatchList* w = reinterpret_cast<Block*>(o)->watch;
  return w != nullptr ? w->traverse(visit, arg) : 0;
}

PyObject* block_unbind(PyObject* o, PyObject*);

int block_clear(PyObject* o) {
  Py_XDECREF(block_unbind(o, nullptr));
  return 0;
}

void block_dealloc(PyObject* o) {
  PyObject_GC_UnTrack(o);
  Block* self = reinterpret_cast<Block*>(o);
  PyTypeObject* type = Py_TYPE(o);
  delete self->watch;
  delete self->lora;
  delete self->workspace;
  delete self->owned;
  delete self->train;
  type->tp_free(o);
  Py_DECREF(type);
}

// bind(watch, merged or None, scales, plan, owned buffers, workspace tensor, base, bytes, N, d, f, E, k, dtype, device index)
PyObject* block_bind(PyObject* o, PyObject* args) {
  HANDLE_TH_ERRORS
  Block* self = reinterpret_cast<Block*>(o);
  PyObject *watch, *merged, *scales, *owned, *ws;
  unsigned long long plan, base, bytes;
  long long N;
  int d, f, E, k, dtype, device;
  if (!PyArg_ParseTuple(args, "O!OOKO!OKKLiiiiii", &PyList_Type, &watch, &merged, &scales, &plan, &PyList_Type, &owned, &ws, &base, &bytes, &N, &d, &f,
                        &E, &k, &dtype, &device))
    return nullptr;
  if (!THPVariable_Check(ws)) {
    PyErr_SetString(PyExc_TypeError, "workspace must be a tensor");
    return nullptr;
  }
  if (!tensor_list(owned, self->owned) || !self->watch->bind(watch) ||
      !read_merged(merged, scales, 2, (size_t)self->watch->num_params(), self->lora)) {
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
  self->owned->clear();
  *self->lora = MergedUse();
  self->train->reset();
  Py_RETURN_NONE;
}

// bind_train(training workspace, base, bytes, LoRA pointer table or None, ranks, generation): after bind()
PyObject* block_bind_train(PyObject* o, PyObject* args) {
  HANDLE_TH_ERRORS
  Block* self = reinterpret_cast<Block*>(o);
  PyObject *tws, *tab, *ranks, *gen;
  unsigned long long base, bytes;
  if (!PyArg_ParseTuple(args, "OKKOO!O", &tws, &base, &bytes, &tab, &PyList_Type, &ranks, &gen)) return nullptr;
  auto c = std::make_shared<TrainCall>();
  c->lora = *self->lora;
  if (!read_generation(gen, &c->gen) || !read_ranks(ranks, c->lora, &c->ranks)) return nullptr;
  c->ws = *self->workspace;
  c->owned = *self->owned;
  c->tws = THPVariable_Unpack(tws);
  if (tab != Py_None) c->lora_tab = THPVariable_Unpack(tab);
  c->plan = self->plan;
  c->ws_base = self->ws_base;
  c->ws_bytes = self->ws_bytes;
  c->tws_base = reinterpret_cast<void*>(base);
  c->tws_bytes = (size_t)bytes;
  c->N = self->N;
  c->d = self->d;
  c->f = self->f;
  c->E = self->E;
  c->k = self->k;
  c->device = self->device;
  *self->train = std::move(c);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// a contiguous tensor of the bound device, dtype and row width with n rows
bool rows_match(const Tensor& t, int device, int dtype, int d, int64_t n) {
  return t.is_cuda() && t.device().index() == device && t.scalar_type() == scalar_of(dtype) && t.dim() >= 1 &&
         t.size(-1) == d && t.numel() == n * d && t.is_contiguous();
}

// forward(tensor, residual or None, norm or None, slots) -> (out, loss), or None: prepare again
PyObject* block_forward(PyObject* o, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Block* self = reinterpret_cast<Block*>(o);
  if (nargs != 4) {
    PyErr_SetString(PyExc_TypeError, "forward(tensor, residual, norm, slots)");
    return nullptr;
  }
  const long k = PyLong_AsLong(args[3]);
  if (k == -1 && PyErr_Occurred()) return nullptr;
  if (self->watch->empty() || !THPVariable_CheckExact(args[0])) Py_RETURN_NONE;    // the result is of the input's class
  const Tensor& x = THPVariable_Unpack(args[0]);
  if (self->N <= 0 || k != self->k || !rows_match(x, self->device, self->dtype, self->d, self->N)) Py_RETURN_NONE;
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

// train(tensor, residual or None, dropout p, parameters or None, slots) -> (out, loss, seed), or None: prepare again.
// Without a list the parameters are the watched ones.
PyObject* block_train(PyObject* o, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Block* self = reinterpret_cast<Block*>(o);
  if (nargs != 5) {
    PyErr_SetString(PyExc_TypeError, "train(tensor, residual, p, parameters, slots)");
    return nullptr;
  }
  const long k = PyLong_AsLong(args[4]);
  if (k == -1 && PyErr_Occurred()) return nullptr;
  if (*self->train == nullptr || !THPVariable_Check(args[0])) Py_RETURN_NONE;
  if (args[3] == Py_None && !THPVariable_CheckExact(args[0])) Py_RETURN_NONE;    // the result is of the input's class
  if (args[3] == Py_None && torch::jit::tracer::isTracing()) Py_RETURN_NONE;
  const std::shared_ptr<TrainCall> c = *self->train;
  const Tensor& x = THPVariable_Unpack(args[0]);
  if (k != c->k || !rows_match(x, c->device, MOE_B200_BF16, c->d, c->N)) Py_RETURN_NONE;
  const bool has_res = args[1] != Py_None;
  if (has_res && !THPVariable_Check(args[1])) Py_RETURN_NONE;
  Tensor res;
  if (has_res) {
    res = THPVariable_Unpack(args[1]);
    if (!rows_match(res, c->device, MOE_B200_BF16, c->d, c->N) || res.sizes() != x.sizes()) Py_RETURN_NONE;
  }
  const double p = PyFloat_AsDouble(args[2]);
  if (PyErr_Occurred()) return nullptr;
  Edges edges;
  edges.add(x);
  if (has_res) edges.add(res); else edges.add_empty();
  Tensor gate_w, gate_b;
  if (args[3] == Py_None) {
    if (self->watch->empty() || !self->watch->unchanged()) Py_RETURN_NONE;
    gate_w = self->watch->param(0);
    gate_b = self->watch->param(1);
    for (int i = 0; i < self->watch->num_params(); ++i) edges.add_param(self->watch->param(i));
  } else {
    const Py_ssize_t n = PyList_Size(args[3]);
    if (n < 2) {
      PyErr_SetString(PyExc_TypeError, "parameters must be a list");
      return nullptr;
    }
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* v = PyList_GET_ITEM(args[3], i);
      if (!THPVariable_Check(v)) {
        PyErr_SetString(PyExc_TypeError, "parameters must be tensors");
        return nullptr;
      }
      edges.add_param(THPVariable_Unpack(v));
    }
    gate_w = THPVariable_Unpack(PyList_GET_ITEM(args[3], 0));
    gate_b = THPVariable_Unpack(PyList_GET_ITEM(args[3], 1));
  }
  edges.refuse_tangents();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)c->device);
  void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)c->device).stream();
  if (args[3] == Py_None) {
    const int rc = self->lora->refresh(*self->watch, MOE_B200_BF16, stream);
    if (rc != 0) return fail(rc, "lora_merge");
  }
  const uint64_t seed = draw_seed();
  Tensor out, aux;
  {
    at::AutoGradMode no_grad(false);
    out = at::empty(x.sizes(), x.options());
    aux = c->N > 0 ? at::empty({}, x.options().dtype(at::kFloat)) : at::zeros({}, x.options().dtype(at::kFloat));
    const int rc = moe::forward_train_into(
        x.const_data_ptr(), gate_w.const_data_ptr(), gate_b.const_data_ptr(), c->plan,
        has_res ? res.const_data_ptr() : nullptr, c->N, c->d, c->f, c->E, c->k, MOE_B200_BF16, (float)p, seed, c->ws_base,
        c->ws_bytes, c->tws_base, c->tws_bytes, out.data_ptr(), aux.data_ptr<float>(), !c->ranks.empty(), stream);
    if (rc != 0) return fail(rc, "forward_train");
  }
  ++*c->gen;
  if (edges.wanted()) {
    auto node = std::shared_ptr<BlockBackward>(new BlockBackward(), torch::autograd::deleteNode);
    node->set_next_edges(edges.take());
    node->weights = edges.take_weights();
    node->call = c;
    node->gen = *c->gen;
    node->seed = seed;
    node->p = p;
    node->gate_w = gate_w.detach();
    node->x = SavedVariable(x, false);
    torch::autograd::set_history({out, aux}, node);
  }
  PyObject* t = PyTuple_New(3);
  if (t == nullptr) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(aux)));
  PyTuple_SET_ITEM(t, 2, PyLong_FromUnsignedLongLong(seed));
  return t;
  END_HANDLE_TH_ERRORS
}

// a copy or an unpickled module starts unbound
PyObject* fresh_reduce(PyObject* o, PyObject*) { return Py_BuildValue("O()", (PyObject*)Py_TYPE(o)); }

PyMethodDef block_methods[] = {
    {"bind", block_bind, METH_VARARGS, nullptr},
    {"unbind", block_unbind, METH_NOARGS, nullptr},
    {"bind_train", block_bind_train, METH_VARARGS, nullptr},
    {"train", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(block_train)), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(block_forward)), METH_FASTCALL, nullptr},
    {"__reduce__", fresh_reduce, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyType_Slot block_slots[] = {{Py_tp_new, reinterpret_cast<void*>(block_new)},
                             {Py_tp_dealloc, reinterpret_cast<void*>(block_dealloc)},
                             {Py_tp_traverse, reinterpret_cast<void*>(block_traverse)},
                             {Py_tp_clear, reinterpret_cast<void*>(block_clear)},
                             {Py_tp_methods, block_methods},
                             {0, nullptr}};
PyType_Spec block_spec = {"gemmallm_b200._host.Block", sizeof(Block), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC,
                          block_slots};

// ---- the dense feed-forward ------------------------------------------------------------------

struct Ffn {
  PyObject_HEAD
  WatchList* watch;
  MergedUse* lora;
  std::vector<Tensor>* owned;   // the plan
  Tensor* offsets;        // int32 [0, M]
  Tensor* status;         // int32 [16], written only when a wait inside a kernel ran out
  std::shared_ptr<TrainCall>* train;
  const void* plan;
  int64_t M;
  int d, f, dtype, device;
};

PyObject* ffn_new(PyTypeObject* type, PyObject*, PyObject*) {
  Ffn* self = reinterpret_cast<Ffn*>(type->tp_alloc(type, 0));
  if (self == nullptr) return nullptr;
  self->watch = new WatchList();
  self->lora = new MergedUse();
  self->owned = new std::vector<Tensor>();
  self->offsets = new Tensor();
  self->status = new Tensor();
  self->train = new std::shared_ptr<TrainCall>();
  return reinterpret_cast<PyObject*>(self);
}

int ffn_traverse(PyObject* o, visitproc visit, void* arg) {
  Py_VISIT(Py_TYPE(o));
  const WatchList* w = reinterpret_cast<Ffn*>(o)->watch;
  return w != nullptr ? w->traverse(visit, arg) : 0;
}

PyObject* ffn_unbind(PyObject* o, PyObject*);

int ffn_clear(PyObject* o) {
  Py_XDECREF(ffn_unbind(o, nullptr));
  return 0;
}

void ffn_dealloc(PyObject* o) {
  PyObject_GC_UnTrack(o);
  Ffn* self = reinterpret_cast<Ffn*>(o);
  PyTypeObject* type = Py_TYPE(o);
  delete self->watch;
  delete self->lora;
  delete self->owned;
  delete self->offsets;
  delete self->status;
  delete self->train;
  type->tp_free(o);
  Py_DECREF(type);
}

// bind(watch, merged or None, scales, plan, owned buffers, offsets, status, M, d, f, dtype, device index)
PyObject* ffn_bind(PyObject* o, PyObject* args) {
  HANDLE_TH_ERRORS
  Ffn* self = reinterpret_cast<Ffn*>(o);
  PyObject *watch, *merged, *scales, *owned, *offsets, *status;
  unsigned long long plan;
  long long M;
  int d, f, dtype, device;
  if (!PyArg_ParseTuple(args, "O!OOKO!OOLiiii", &PyList_Type, &watch, &merged, &scales, &plan, &PyList_Type, &owned, &offsets, &status, &M, &d, &f,
                        &dtype, &device))
    return nullptr;
  if (!THPVariable_Check(offsets) || !THPVariable_Check(status)) {
    PyErr_SetString(PyExc_TypeError, "offsets and status must be tensors");
    return nullptr;
  }
  if (!tensor_list(owned, self->owned) || !self->watch->bind(watch) ||
      !read_merged(merged, scales, 0, (size_t)self->watch->num_params(), self->lora)) {
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
  Ffn* self = reinterpret_cast<Ffn*>(o);
  self->watch->clear();
  self->owned->clear();
  *self->lora = MergedUse();
  self->train->reset();
  Py_RETURN_NONE;
}

// bind_train(training workspace, base, bytes, LoRA pointer table or None, ranks, generation): after bind()
PyObject* ffn_bind_train(PyObject* o, PyObject* args) {
  HANDLE_TH_ERRORS
  Ffn* self = reinterpret_cast<Ffn*>(o);
  PyObject *tws, *tab, *ranks, *gen;
  unsigned long long base, bytes;
  if (!PyArg_ParseTuple(args, "OKKOO!O", &tws, &base, &bytes, &tab, &PyList_Type, &ranks, &gen)) return nullptr;
  auto c = std::make_shared<TrainCall>();
  c->lora = *self->lora;
  if (!read_generation(gen, &c->gen) || !read_ranks(ranks, c->lora, &c->ranks)) return nullptr;
  c->tws = THPVariable_Unpack(tws);
  c->owned = *self->owned;
  c->offsets = *self->offsets;
  c->status = *self->status;
  if (tab != Py_None) c->lora_tab = THPVariable_Unpack(tab);
  c->plan = self->plan;
  c->tws_base = reinterpret_cast<void*>(base);
  c->tws_bytes = (size_t)bytes;
  c->N = self->M;
  c->d = self->d;
  c->f = self->f;
  c->E = 1;
  c->k = 1;
  c->device = self->device;
  *self->train = std::move(c);
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// train(tensor, dropout p, parameters or None, LoRA scale) -> (y, seed), or None: prepare again
PyObject* ffn_train(PyObject* o, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Ffn* self = reinterpret_cast<Ffn*>(o);
  if (nargs != 4) {
    PyErr_SetString(PyExc_TypeError, "train(tensor, p, parameters, scale)");
    return nullptr;
  }
  const double scale = PyFloat_AsDouble(args[3]);
  if (PyErr_Occurred()) return nullptr;
  if (*self->train == nullptr || !THPVariable_Check(args[0])) Py_RETURN_NONE;
  // (under a tracer the module takes a way that the tracer sees)
  if (args[2] == Py_None && torch::jit::tracer::isTracing()) Py_RETURN_NONE;
  const std::shared_ptr<TrainCall> c = *self->train;
  const Tensor& x = THPVariable_Unpack(args[0]);
  if (!c->lora.has_scale(scale) || !rows_match(x, c->device, MOE_B200_BF16, c->d, c->N)) Py_RETURN_NONE;
  const double p = PyFloat_AsDouble(args[1]);
  if (PyErr_Occurred()) return nullptr;
  Edges edges;
  edges.add(x);
  if (args[2] == Py_None) {
    if (self->watch->empty() || !self->watch->unchanged()) Py_RETURN_NONE;
    for (int i = 0; i < self->watch->num_params(); ++i) edges.add_param(self->watch->param(i));
  } else {
    const Py_ssize_t n = PyList_Size(args[2]);
    if (n < 0) return nullptr;
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* v = PyList_GET_ITEM(args[2], i);
      if (!THPVariable_Check(v)) {
        PyErr_SetString(PyExc_TypeError, "parameters must be tensors");
        return nullptr;
      }
      edges.add_param(THPVariable_Unpack(v));
    }
  }
  edges.refuse_tangents();
  c10::cuda::CUDAGuard guard((c10::DeviceIndex)c->device);
  void* stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)c->device).stream();
  if (args[2] == Py_None) {
    const int rc = self->lora->refresh(*self->watch, MOE_B200_BF16, stream);
    if (rc != 0) return fail(rc, "lora_merge");
  }
  const uint64_t seed = draw_seed();
  Tensor h, y;
  {
    at::AutoGradMode no_grad(false);
    h = at::empty({c->N, c->f}, x.options());
    y = at::empty(x.sizes(), x.options());
    const int rc = moe::experts_train_into(x.const_data_ptr(), c->offsets.const_data_ptr<int32_t>(), c->plan, c->N, c->d,
                                           c->f, 1, (float)p, seed, c->tws_base, c->tws_bytes, h.data_ptr(), y.data_ptr(),
                                           !c->ranks.empty(), c->status.data_ptr<int32_t>(), stream);
    if (rc != 0) return fail(rc, "experts_train");
  }
  ++*c->gen;
  if (edges.wanted()) {
    auto node = std::shared_ptr<FfnBackward>(new FfnBackward(), torch::autograd::deleteNode);
    node->set_next_edges(edges.take());
    node->weights = edges.take_weights();
    node->call = c;
    node->gen = *c->gen;
    node->seed = seed;
    node->p = p;
    node->x = SavedVariable(x, false);
    node->h = SavedVariable(h, false);
    torch::autograd::set_history(y, node);
  }
  PyObject* t = PyTuple_New(2);
  if (t == nullptr) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(y)));
  PyTuple_SET_ITEM(t, 1, PyLong_FromUnsignedLongLong(seed));
  return t;
  END_HANDLE_TH_ERRORS
}

// forward(tensor, LoRA scale) -> y, or None: prepare again
PyObject* ffn_forward(PyObject* o, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  Ffn* self = reinterpret_cast<Ffn*>(o);
  if (nargs != 2) {
    PyErr_SetString(PyExc_TypeError, "forward(tensor, scale)");
    return nullptr;
  }
  const double scale = PyFloat_AsDouble(args[1]);
  if (PyErr_Occurred()) return nullptr;
  if (self->watch->empty() || self->M <= 0 || !THPVariable_Check(args[0])) Py_RETURN_NONE;
  const Tensor& x = THPVariable_Unpack(args[0]);
  if (!self->lora->has_scale(scale) || !rows_match(x, self->device, self->dtype, self->d, self->M) ||
      !self->watch->unchanged())
    Py_RETURN_NONE;
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
    {"bind_train", ffn_bind_train, METH_VARARGS, nullptr},
    {"train", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(ffn_train)), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(ffn_forward)), METH_FASTCALL, nullptr},
    {"__reduce__", fresh_reduce, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyMethodDef merged_methods[] = {{"refresh", merged_refresh, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyType_Slot merged_slots[] = {{Py_tp_new, reinterpret_cast<void*>(merged_new)},
                              {Py_tp_dealloc, reinterpret_cast<void*>(merged_dealloc)},
                              {Py_tp_methods, merged_methods},
                              {0, nullptr}};
PyType_Spec merged_spec = {"gemmallm_b200._host.Merged", sizeof(MergedObject), 0, Py_TPFLAGS_DEFAULT, merged_slots};

PyMethodDef generation_methods[] = {{"__reduce__", fresh_reduce, METH_NOARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};
PyType_Slot generation_slots[] = {{Py_tp_new, reinterpret_cast<void*>(generation_new)},
                                  {Py_tp_dealloc, reinterpret_cast<void*>(generation_dealloc)},
                                  {Py_tp_methods, generation_methods},
                                  {0, nullptr}};
PyType_Spec generation_spec = {"gemmallm_b200._host.Generation", sizeof(Generation), 0, Py_TPFLAGS_DEFAULT, generation_slots};

PyType_Slot ffn_slots[] = {{Py_tp_new, reinterpret_cast<void*>(ffn_new)},
                           {Py_tp_dealloc, reinterpret_cast<void*>(ffn_dealloc)},
                           {Py_tp_traverse, reinterpret_cast<void*>(ffn_traverse)},
                           {Py_tp_clear, reinterpret_cast<void*>(ffn_clear)},
                           {Py_tp_methods, ffn_methods},
                           {0, nullptr}};
PyType_Spec ffn_spec = {"gemmallm_b200._host.Ffn", sizeof(Ffn), 0, Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC, ffn_slots};

// ---- the decoder layer's attention and first LayerNorm in inference --------------------------------
// Nothing is bound or kept: every tensor comes with the call. None for what is left to the Python side (other classes of
// tensors, modes that see Python calls, tracing, autocast). A layer call of one short sequence is 90 us of GPU work; with
// its ten launches made from Python it took 119.

bool plain_call() {
  return !at::impl::torch_function_mode_enabled() && !torch::jit::tracer::isTracing() &&
         !at::autocast::is_autocast_enabled(at::kCUDA);
}

// attention(x, qkv weight, bias, gate weight, bias, o weight, bias, table, mask or None, q heads, kv heads, head_dim, scaler,
//           status [, norm weight, bias, eps]). With the LayerNorm: on its output, and x is added (the skip connection); None
// where attention_supported() says no.
PyObject* host_attention(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 14 && nargs != 17) {
    PyErr_SetString(PyExc_TypeError, "attention() takes 14 or 17 arguments");
    return nullptr;
  }
  const bool masked = args[8] != Py_None, layer = nargs == 17;
  for (int i = 0; i < (masked ? 9 : 8); ++i)
    if (!THPVariable_CheckExact(args[i])) Py_RETURN_NONE;
  if (!THPVariable_CheckExact(args[13])) Py_RETURN_NONE;
  if (layer && (!THPVariable_CheckExact(args[14]) || !THPVariable_CheckExact(args[15]))) Py_RETURN_NONE;
  const long heads = PyLong_AsLong(args[9]), kv = PyLong_AsLong(args[10]), hd = PyLong_AsLong(args[11]);
  const double scaler = PyFloat_AsDouble(args[12]), eps = layer ? PyFloat_AsDouble(args[16]) : 0.;
  if (PyErr_Occurred()) return nullptr;
  auto t = [&](int i) -> const Tensor& { return THPVariable_Unpack(args[i]); };
  const Tensor &x = t(0), &table = t(7), &status = t(13);
  if (!plain_call() || !x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() != 3 || !x.is_contiguous() || heads < 1 ||
      kv < 1 || hd < 1)
    Py_RETURN_NONE;
  const int64_t B = x.size(0), S = x.size(1), hidden = x.size(2), inner = heads * hd;
  for (int i = 1; i < 7; ++i)
    if (t(i).device() != x.device() || t(i).scalar_type() != at::kBFloat16) Py_RETURN_NONE;
  if (t(1).dim() != 2 || t(1).size(0) != (heads + 2 * kv) * hd || t(3).dim() != 2 || t(3).size(0) != heads) Py_RETURN_NONE;
  if (table.device() != x.device() || table.scalar_type() != at::kFloat || !table.is_contiguous() || table.dim() != 2 ||
      table.size(0) < S || table.size(1) != 2 * hd)
    Py_RETURN_NONE;
  if (status.device() != x.device() || status.scalar_type() != at::kInt || status.numel() < MOE_B200_STATUS_INTS) Py_RETURN_NONE;
  const float* mask = nullptr;
  if (masked) {
    if (t(8).device() != x.device() || t(8).scalar_type() != at::kFloat || !t(8).is_contiguous() || t(8).numel() != S * S)
      Py_RETURN_NONE;
    mask = t(8).const_data_ptr<float>();
  }
  // the library's own launches throughout, where sizes and places allow (attention.py asks for the same) and nobody asks for
  // derivatives: torch's Linears give those of the output projection (the core has none, so no other Linear has any)
  bool derived = x._fw_grad(0).defined();
  for (int i = 1; i < 7; ++i)
    derived |= t(i)._fw_grad(0).defined() || (at::GradMode::is_enabled() && t(i).requires_grad());
  // (has_storage: a batch of weights under vmap has none)
  auto matrix = [](const Tensor& w, int64_t rows, int64_t cols) {
    return w.dim() == 2 && w.size(0) == rows && w.size(1) == cols && w.is_contiguous() && w.has_storage();
  };
  auto vector = [](const Tensor& b, int64_t n) { return b.numel() == n && b.is_contiguous() && b.has_storage(); };
  moe::AttentionArgs p = {};
  bool own = !derived && x.has_storage() && hidden <= 1 << 24 && inner <= 1 << 24 && B <= 1 << 24 && S <= 128 && matrix(t(1), (heads + 2 * kv) * hd, hidden) &&
             vector(t(2), (heads + 2 * kv) * hd) && matrix(t(3), heads, hidden) && vector(t(4), heads) &&
             matrix(t(5), hidden, inner) && vector(t(6), hidden);
  if (own) {
    p.x = x.const_data_ptr();
    if (layer) {
      for (int i = 14; i < 16; ++i)
        if (t(i).device() != x.device() || t(i).scalar_type() != at::kBFloat16 || !vector(t(i), hidden)) Py_RETURN_NONE;
      p.norm_weight = t(14).const_data_ptr();
      p.norm_bias = t(15).const_data_ptr();
      p.eps = (float)eps;
      p.skip = p.x;
    }
    p.wqkv = t(1).const_data_ptr(); p.bqkv = t(2).const_data_ptr();
    p.wgate = t(3).const_data_ptr(); p.bgate = t(4).const_data_ptr();
    p.wo = t(5).const_data_ptr(); p.bo = t(6).const_data_ptr();
    p.pos_emb = table.const_data_ptr<float>();
    p.mask = mask;
    p.B = B; p.S = (int)S; p.hidden = (int)hidden;
    p.q_heads = (int)heads; p.kv_heads = (int)kv; p.head_dim = (int)hd;
    p.scaler = (float)scaler;
    p.status = status.data_ptr<int32_t>();
    own = moe::attention_supported(p);
  }
  if (layer) {
    if (!own) Py_RETURN_NONE;
    for (int i : {0, 14, 15})
      if (t(i)._fw_grad(0).defined() || (at::GradMode::is_enabled() && t(i).requires_grad())) Py_RETURN_NONE;
  }
  c10::cuda::CUDAGuard guard(x.device());
  Tensor result;
  int rc = 0;
  {
    pybind11::gil_scoped_release no_gil;
    void* stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    if (own) {
      // qkv, the core's output, the normalised rows and the gate in one piece (rows of 16-byte multiples, the gate last)
      const int64_t N = B * S, qkv = N * (heads + 2 * kv) * hd, apart = moe::attention_normalises_apart(p) ? N * hidden : 0;
      const Tensor scratch = at::empty({qkv + N * inner + apart + N * heads}, x.options());
      result = at::empty({B, S, hidden}, x.options());
      char* at_byte = static_cast<char*>(scratch.data_ptr());
      p.qkv = at_byte;
      p.core = at_byte + qkv * 2;
      p.xn = at_byte + (qkv + N * inner) * 2;
      p.gate = at_byte + (qkv + N * inner + apart) * 2;
      p.out = result.data_ptr();
      rc = moe::attention_layer(p, stream);
    } else {
      const Tensor qkv = at::linear(x, t(1), t(2)), gate = at::linear(x, t(3), t(4));
      const Tensor out = at::empty({B, S, inner}, x.options());
      rc = moe_b200_attention(qkv.const_data_ptr(), gate.const_data_ptr(), table.const_data_ptr<float>(), mask, B, (int)S,
                              (int)heads, (int)kv, (int)hd, (float)scaler, out.data_ptr(), stream);
      if (rc == 0) result = at::linear(out, t(5), t(6));
    }
  }
  if (rc != 0) return fail(rc, "attention");
  return THPVariable_Wrap(std::move(result));
  END_HANDLE_TH_ERRORS
}

// layernorm(x, weight, bias, eps) by the library's row kernel, over the last dimension
PyObject* host_layernorm(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4) {
    PyErr_SetString(PyExc_TypeError, "layernorm(x, weight, bias, eps)");
    return nullptr;
  }
  for (int i = 0; i < 3; ++i)
    if (!THPVariable_CheckExact(args[i])) Py_RETURN_NONE;
  const double eps = PyFloat_AsDouble(args[3]);
  if (PyErr_Occurred()) return nullptr;
  const Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]), &b = THPVariable_Unpack(args[2]);
  const auto type = x.scalar_type();
  if (!plain_call() || !x.is_cuda() || (type != at::kBFloat16 && type != at::kFloat) || x.dim() < 1 || !x.is_contiguous())
    Py_RETURN_NONE;
  const int64_t d = x.size(-1);
  if (d < 8 || d % 8 != 0 || x.numel() == 0) Py_RETURN_NONE;
  for (const Tensor* p : {&w, &b})
    if (p->device() != x.device() || p->scalar_type() != type || !p->is_contiguous() || p->numel() != d) Py_RETURN_NONE;
  if (at::GradMode::is_enabled() && (x.requires_grad() || w.requires_grad() || b.requires_grad())) Py_RETURN_NONE;
  c10::cuda::CUDAGuard guard(x.device());
  Tensor out = at::empty_like(x);
  const int rc = moe_b200_layernorm(x.const_data_ptr(), w.const_data_ptr(), b.const_data_ptr(), (float)eps, x.numel() / d,
                                    (int)d, type == at::kFloat ? MOE_B200_F32 : MOE_B200_BF16, out.data_ptr(),
                                    c10::cuda::getCurrentCUDAStream(x.device().index()).stream());
  if (rc == MOE_B200_ERR_ALIGN) Py_RETURN_NONE;      // tensors at an odd place
  if (rc != 0) return fail(rc, "layernorm");
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyMethodDef module_methods[] = {
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(host_attention)), METH_FASTCALL, nullptr},
    {"layernorm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(host_layernorm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

bool add_type(PyObject* m, const char* name, PyType_Spec* spec, PyTypeObject** keep = nullptr) {
  PyObject* t = PyType_FromSpec(spec);
  if (t == nullptr) return false;
  const int rc = PyModule_AddObjectRef(m, name, t);
  if (keep != nullptr && rc == 0) {
    *keep = reinterpret_cast<PyTypeObject*>(t);      // for the life of the process
  } else {
    Py_DECREF(t);
  }
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
  s_normalized_shape = PyUnicode_InternFromString("normalized_shape");
  if (!add_type(m, "Block", &block_spec) || !add_type(m, "Ffn", &ffn_spec) ||
      !add_type(m, "Generation", &generation_spec, &g_generation_type) ||
      !add_type(m, "Merged", &merged_spec, &g_merged_type)) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
