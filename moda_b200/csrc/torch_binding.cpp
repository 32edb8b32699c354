// PyTorch binding of libmoda_b200.so: argument checks, allocation of results and scratch, and the
// autograd nodes of the operators, in one native call per operator.
//
// The smallest calls of the operators run for some ten microseconds on the GPU; a binding through
// ctypes with torch.autograd.Function in Python cost 50 us (forward) and 240 us (forward and
// backward) of host time per call on the same machine, so that they were bound by the host.
// Everything between the user's call and the library's C ABI therefore lives here: the arguments of
// a well-formed call are checked natively (a call that is not well-formed, or that asks for a
// warning, returns None and takes the Python wrapper, which says what is wrong), and the backward
// is a torch::autograd::Node that the engine runs without entering Python.
//
// Functions (module moda_b200._native):
//   attention(q, k, v, cached_k, cached_v, scale, G, mode, return_depth_grads, warn_shape, checked)
//   forward(q, k, v, cached_k, cached_v, scale, G, mode, chunk_rows)
//   backward(q, k, v, cached_k, cached_v, o, lse, dout, scale, G, mode, chunk_rows)
//   cache_state([grad_k, grad_v]), cache_grads(state), cache_append(...), cache_attention(...): DepthKVCache
//   set_path(path), set_check(fn)
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/empty.h>
#include <c10/core/Event.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <atomic>
#include <cmath>
#include <memory>
#include <optional>

#include "../../include/moda_b200.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

constexpr int kChunkRows = 64;        // query rows of a chunk of the chunk-visible operator (moda_v16.py:581-585)
std::atomic<int> g_path{MODA_PATH_AUTO};
PyObject* g_check = nullptr;          // Python callable (status, what): raises for a status that is not 0

// Raises what the Python side raises for a library status (also from the autograd engine's threads).
void check_status(int rc, const char* what) {
  if (rc == MODA_OK) return;
  PyGILState_STATE gil = PyGILState_Ensure();
  PyObject* r = g_check ? PyObject_CallFunction(g_check, "is", rc, what) : nullptr;
  Py_XDECREF(r);
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s: status %d", what, rc);
  python_error err;
  err.persist();
  PyGILState_Release(gil);
  throw err;
}

bool usable(const Tensor& x) {        // the library reads this layout in place
  if (x.stride(-1) != 1 || (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15u) != 0) return false;
  for (int64_t i = 0; i + 1 < x.dim(); ++i)
    if (x.size(i) > 1 && (x.stride(i) <= 0 || x.stride(i) % 8 != 0)) return false;
  return true;
}
Tensor in_place_or_copy(const Tensor& x) {
  if (!x.defined() || usable(x)) return x;
  return x.is_contiguous() ? x.clone() : x.contiguous();     // contiguous, but not on a 16-byte boundary: a copy is
}

struct T4 {
  moda_tensor4 t{};
  bool set = false;
  explicit T4(const Tensor& x) {
    if (!x.defined()) return;
    set = true;
    t.data = const_cast<void*>(x.const_data_ptr());
    t.stride_b = x.stride(0); t.stride_t = x.stride(1); t.stride_h = x.stride(2);
  }
  const moda_tensor4* p() const { return set ? &t : nullptr; }
};

// One call: the operator's scalars and, for a layer cache, how many of its layers are valid.
struct Op {
  double scale = 0.;
  int G = 1, mode = 0, chunk_rows = kChunkRows;
  int layers = -1, capacity = 0;      // layers >= 0: depth tensors are an in-place cache [B, T * capacity, H, D]
};

moda_problem problem(const Op& op, const Tensor& q, bool use_depth, const Tensor& ck, bool accumulate) {
  moda_problem pr{};
  pr.B = (int32_t)q.size(0);
  pr.T_kv = (int32_t)(q.size(1) / op.G);
  pr.H = (int32_t)q.size(2);
  pr.D = (int32_t)q.size(3);
  pr.G = op.G;
  pr.L = !use_depth ? 0 : op.layers >= 0 ? op.layers : pr.T_kv > 0 ? (int32_t)(ck.size(1) / pr.T_kv) : 0;
  pr.mode = op.mode;
  pr.chunk_rows = op.chunk_rows;
  pr.dtype = q.scalar_type() == at::kBFloat16 ? MODA_BF16 : MODA_FP16;
  pr.path = g_path.load(std::memory_order_relaxed);
  pr.scale = (float)op.scale;
  pr.device = q.get_device();
  pr.depth_rows_per_pos = op.layers >= 0 ? op.capacity : 0;
  pr.accumulate_depth_grads = accumulate ? 1 : 0;
  return pr;
}

struct Out { Tensor o, lse; };
Out run_forward(const Op& op, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& ck_, const Tensor& cv_) {
  const bool use_depth = ck_.defined() && cv_.defined();
  const Tensor q = in_place_or_copy(q_), k = in_place_or_copy(k_), v = in_place_or_copy(v_);
  const Tensor ck = use_depth ? in_place_or_copy(ck_) : Tensor(), cv = use_depth ? in_place_or_copy(cv_) : Tensor();
  const moda_problem pr = problem(op, q, use_depth, ck, false);
  Out r;
  r.o = at::empty(q.sizes(), q.options());
  r.lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
  const c10::cuda::CUDAGuard guard(q.device());
  check_status(moda_b200_fwd(&pr, T4(q).p(), T4(k).p(), T4(v).p(), T4(ck).p(), T4(cv).p(), T4(r.o).p(),
                             r.lse.mutable_data_ptr<float>(), c10::cuda::getCurrentCUDAStream().stream()),
               "moda_b200_fwd");
  return r;
}

struct Grads { Tensor dq, dk, dv, dck, dcv; };
// dck / dcv given: gradient caches of the depth tensors' layout, added to when `accumulate`.
Grads run_backward(const Op& op, const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& ck_, const Tensor& cv_,
                   const Tensor& o_, const Tensor& lse_, const Tensor& dout_, const Tensor& dck, const Tensor& dcv, bool accumulate) {
  const bool use_depth = ck_.defined() && cv_.defined();
  const Tensor q = in_place_or_copy(q_), k = in_place_or_copy(k_), v = in_place_or_copy(v_), o = in_place_or_copy(o_);
  const Tensor dout = in_place_or_copy(dout_), lse = lse_.contiguous();
  const Tensor ck = use_depth ? in_place_or_copy(ck_) : Tensor(), cv = use_depth ? in_place_or_copy(cv_) : Tensor();
  const moda_problem pr = problem(op, q, use_depth, ck, accumulate);
  auto like = [](const Tensor& x) { return x.defined() ? at::empty(x.sizes(), x.options()) : Tensor(); };
  Grads g;
  g.dq = like(q); g.dk = like(k); g.dv = like(v);
  g.dck = dck.defined() ? dck : like(ck);
  g.dcv = dcv.defined() ? dcv : like(cv);
  size_t bytes = 0;
  check_status(moda_b200_bwd_workspace_bytes(&pr, &bytes), "moda_b200_bwd_workspace_bytes");
  const Tensor ws = at::empty({(int64_t)(bytes > 256 ? bytes : 256)}, q.options().dtype(at::kByte));
  const c10::cuda::CUDAGuard guard(q.device());
  check_status(moda_b200_bwd(&pr, T4(q).p(), T4(k).p(), T4(v).p(), T4(ck).p(), T4(cv).p(), T4(o).p(), lse.const_data_ptr<float>(),
                             T4(dout).p(), T4(g.dq).p(), T4(g.dk).p(), T4(g.dv).p(), T4(g.dck).p(), T4(g.dcv).p(),
                             ws.mutable_data_ptr(), (size_t)ws.numel(), c10::cuda::getCurrentCUDAStream().stream()),
               "moda_b200_bwd");
  return g;
}

// ------------------------------------------------------------------ depth-KV cache: state of one backward
// Gradient caches of a DepthKVCache, shared by the nodes of one forward pass.  The first `filled`
// layers hold gradients: the first attention whose backward runs (as a rule the last layer, which
// read every slot) stores its depth gradients there, the others add theirs, so that nothing has
// to be zeroed; a later one that read more layers than are filled gets those zeroed first.
// They belong to one run of the engine: a second one over the same forward (a retained graph, losses of
// single layers) starts with caches of its own, and hands on nothing that an earlier one left.
// They pass from node to node outside the engine's sight, which orders two nodes' streams only along
// defined gradients: whoever uses them on another stream than the last user waits for that one.
struct CacheState {
  Tensor grad_k, grad_v;
  int filled = 0;
  int run = -1;                                    // the engine's number of its run
  std::optional<c10::cuda::CUDAStream> last;       // stream of the last use
  void enter(int now) {
    if (run != now) *this = CacheState();
    run = now;
  }
  void used_on(const c10::cuda::CUDAStream& now) {
    if (last && *last != now) {
      c10::Event event(c10::DeviceType::CUDA);
      event.record(last->unwrap());
      event.block(now.unwrap());
      grad_k.record_stream(now.unwrap());
      grad_v.record_stream(now.unwrap());
    }
    last = now;
  }
};
using CacheStatePtr = std::shared_ptr<CacheState>;

// ------------------------------------------------------------------ autograd nodes
struct MoDAAttentionBackward : public Node {
  Op op;
  SavedVariable q, k, v, ck, cv, o, lse;
  CacheStatePtr state;                 // layer cache: its tensors are appended to in place after this
  Tensor cache_k, cache_v;             // node was made, in rows it does not read, so they are kept as they are

  std::string name() const override { return "MoDAAttentionBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q, &k, &v, &ck, &cv, &o, &lse}) s->reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    variable_list out(next_edges().size());
    if (!grads[0].defined()) return out;
    std::unique_lock<std::mutex> lock(mutex_);
    const Tensor q_ = q.unpack(), k_ = k.unpack(), v_ = v.unpack();
    const Tensor ck_ = state ? cache_k : ck.unpack(), cv_ = state ? cache_v : cv.unpack();
    const Tensor o_ = o.unpack(getptr()), lse_ = lse.unpack();
    lock.unlock();
    at::AutoGradMode no_grad(false);
    const Tensor dout = grads[0].scalar_type() == q_.scalar_type() ? grads[0] : grads[0].to(q_.scalar_type());
    Grads g;
    if (state && op.layers > 0) {
      bool accumulate = true;
      state->enter(torch::autograd::get_current_graph_task_id());
      if (!state->grad_k.defined()) {
        state->grad_k = at::empty(cache_k.sizes(), cache_k.options());
        state->grad_v = at::empty(cache_v.sizes(), cache_v.options());
      }
      state->used_on(c10::cuda::getCurrentCUDAStream(q_.device().index()));
      if (state->filled == 0) {
        accumulate = false;
      } else if (op.layers > state->filled) {
        for (const Tensor& x : {state->grad_k, state->grad_v})
          x.view({x.size(0), -1, op.capacity, x.size(2), x.size(3)}).slice(2, state->filled, op.layers).zero_();
      }
      if (op.layers > state->filled) state->filled = op.layers;
      g = run_backward(op, q_, k_, v_, ck_, cv_, o_, lse_, dout, state->grad_k, state->grad_v, accumulate);
    } else if (state) {
      Op plain = op;
      plain.layers = -1;
      g = run_backward(plain, q_, k_, v_, Tensor(), Tensor(), o_, lse_, dout, Tensor(), Tensor(), false);
    } else {
      g = run_backward(op, q_, k_, v_, ck_, cv_, o_, lse_, dout, Tensor(), Tensor(), false);
    }
    out[0] = std::move(g.dq);
    out[1] = std::move(g.dk);
    out[2] = std::move(g.dv);
    if (!state) { out[3] = std::move(g.dck); out[4] = std::move(g.dcv); }   // else out[3] is the token's: none
    return out;
  }
};

// The copy of one layer's k and v into its slot of a layer cache.  Its backward hands the slot's
// gradients to k and v; the chain of tokens makes the engine run it only after every attention that
// read the slot (each attention takes the newest token, each append the one before it).
struct MoDADepthAppendBackward : public Node {
  CacheStatePtr state;
  moda_problem pr{};
  int slot = 0;
  std::string name() const override { return "MoDADepthAppendBackward"; }
  variable_list apply(variable_list&&) override {
    variable_list out(3);
    state->enter(torch::autograd::get_current_graph_task_id());
    if (!state->grad_k.defined() || slot >= state->filled) return out;      // no attention that read the slot has run
    at::AutoGradMode no_grad(false);
    const Tensor& gk = state->grad_k;
    state->used_on(c10::cuda::getCurrentCUDAStream(gk.device().index()));
    const std::vector<int64_t> shape{gk.size(0), pr.T_kv, gk.size(2), gk.size(3)};
    out[0] = at::empty(shape, gk.options());
    out[1] = at::empty(shape, gk.options());
    const c10::cuda::CUDAGuard guard(gk.device());
    check_status(moda_b200_depth_take(&pr, T4(gk).p(), T4(state->grad_v).p(), slot, T4(out[0]).p(), T4(out[1]).p(),
                                      c10::cuda::getCurrentCUDAStream().stream()),
                 "moda_b200_depth_take");
    return out;
  }
};

bool wants_grad(std::initializer_list<const Tensor*> xs) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* x : xs)
    if (x->defined() && x->requires_grad()) return true;
  return false;
}

// There is no forward-mode derivative: a dual number's tangent must not be dropped in silence.
void refuse_tangents(std::initializer_list<const Tensor*> xs) {
  for (const Tensor* x : xs)
    TORCH_CHECK_NOT_IMPLEMENTED(!x->defined() || !x->_fw_grad(0).defined(), "moda_b200: forward-mode differentiation is not implemented");
}

Out attention(const Op& op, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& ck, const Tensor& cv,
              const CacheStatePtr& state, const Tensor& token) {
  refuse_tangents({&q, &k, &v, &ck, &cv});
  const bool grad = wants_grad({&q, &k, &v, state ? &token : &ck, state ? &token : &cv});
  Out r;
  {
    at::AutoGradMode no_grad(false);
    Op used = op;
    if (state && op.layers == 0) used.layers = -1;
    r = (state && op.layers == 0) ? run_forward(used, q, k, v, Tensor(), Tensor()) : run_forward(used, q, k, v, ck, cv);
  }
  if (!grad) return r;
  std::shared_ptr<MoDAAttentionBackward> node(new MoDAAttentionBackward(), torch::autograd::deleteNode);
  node->op = op;
  node->set_next_edges(state ? torch::autograd::collect_next_edges(q, k, v, token)
                             : torch::autograd::collect_next_edges(q, k, v, ck, cv));
  node->q = SavedVariable(q, false);
  node->k = SavedVariable(k, false);
  node->v = SavedVariable(v, false);
  if (state) { node->state = state; node->cache_k = ck; node->cache_v = cv; }
  else { node->ck = SavedVariable(ck, false); node->cv = SavedVariable(cv, false); }
  torch::autograd::set_history(r.o, node);
  node->o = SavedVariable(r.o, true);
  node->lse = SavedVariable(r.lse, false);
  return r;
}

// ------------------------------------------------------------------ Python side
struct NoGil {                        // ctypes dropped the interpreter lock around the library call; so does this
  PyThreadState* s = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(s); }
};
Tensor tensor_or_none(PyObject* x) { return x == Py_None ? Tensor() : THPVariable_Unpack(x); }
bool tensor_or_none_check(PyObject* x) { return x == Py_None || THPVariable_Check(x); }
PyObject* wrap(const Tensor& x) { return THPVariable_Wrap(x); }
PyObject* wrap(const Out& r) {
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, wrap(r.o));
  PyTuple_SET_ITEM(t, 1, wrap(r.lse));
  return t;
}
bool arg_count(Py_ssize_t n, Py_ssize_t want) {
  if (n == want) return true;
  PyErr_Format(PyExc_TypeError, "moda_b200._native: %zd arguments given, %zd expected", n, want);
  return false;
}
int as_int(PyObject* x) {
  const long v = PyLong_AsLong(x);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return (int)v;
}
double as_scale(PyObject* x, const Tensor& q) {
  if (x == Py_None) return 1. / std::sqrt((double)q.size(-1));
  const double v = PyFloat_AsDouble(x);
  if (v == -1. && PyErr_Occurred()) throw python_error();
  return v;
}

// A call the Python wrapper would let through without an error, a warning or a change of layout.
bool well_formed(const Tensor& q, const Tensor& k, const Tensor& v, Tensor& ck, Tensor& cv, int G, int mode,
                 bool return_depth_grads, bool warn_shape) {
  const bool need_kv = mode != MODA_DEPTH_ONLY;
  if (!q.defined() || q.dim() != 4 || !q.is_cuda() || G <= 0) return false;
  if (q.scalar_type() != at::kBFloat16 && q.scalar_type() != at::kHalf) return false;
  if (need_kv != k.defined() || need_kv != v.defined()) return false;
  const int64_t B = q.size(0), Tq = q.size(1), H = q.size(2), D = q.size(3);
  if (warn_shape && Tq < H) return false;
  if (Tq % G != 0) return false;
  if (mode == MODA_CHUNK_VISIBLE && kChunkRows % G != 0) return false;
  const int64_t T = Tq / G;
  auto same = [&](const Tensor& x, int64_t rows) {
    return x.dim() == 4 && x.scalar_type() == q.scalar_type() && x.device() == q.device() && x.size(0) == B && x.size(1) == rows &&
           x.size(2) == H && x.size(3) == D;
  };
  if (need_kv && (!same(k, T) || !same(v, T))) return false;
  if (!ck.defined() || !cv.defined()) {
    ck = Tensor(); cv = Tensor();
  } else {
    const int64_t rows = ck.dim() == 4 ? ck.size(1) : 0;
    if (T == 0 || rows == 0 || rows % T != 0 || !same(ck, rows) || !same(cv, rows)) return false;
    if (!return_depth_grads && (ck.requires_grad() || cv.requires_grad())) return false;
  }
  return need_kv || ck.defined();
}

// attention(q, k, v, cached_k, cached_v, scale, G, mode, return_depth_grads, warn_shape, checked)
//   -> (o, lse), or None for a call that the Python wrapper has to look at (never when `checked`).
// G is anything with __index__ (a NumPy integer, say).
PyObject* py_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 11)) return nullptr;
  const bool checked = a[10] == Py_True;
  for (int i = 0; i < 5; ++i)
    if (!tensor_or_none_check(a[i])) {
      if (!checked) Py_RETURN_NONE;
      PyErr_SetString(PyExc_TypeError, "moda_b200: the operands must be tensors");
      return nullptr;
    }
  if (!checked && !(PyIndex_Check(a[6]) && (a[5] == Py_None || PyFloat_Check(a[5]) || PyLong_Check(a[5])))) Py_RETURN_NONE;
  const Tensor q = tensor_or_none(a[0]), k = tensor_or_none(a[1]), v = tensor_or_none(a[2]);
  Tensor ck = tensor_or_none(a[3]), cv = tensor_or_none(a[4]);
  Op op;
  op.G = as_int(a[6]);
  op.mode = as_int(a[7]);
  if (!checked && !well_formed(q, k, v, ck, cv, op.G, op.mode, PyObject_IsTrue(a[8]) == 1, PyObject_IsTrue(a[9]) == 1)) Py_RETURN_NONE;
  op.scale = as_scale(a[5], q);
  Out r;
  {
    NoGil no_gil;
    r = attention(op, q, k, v, ck, cv, nullptr, Tensor());
  }
  return wrap(r);
  END_HANDLE_TH_ERRORS
}

// forward(q, k, v, cached_k, cached_v, scale, G, mode, chunk_rows) -> (o, lse); no autograd
PyObject* py_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 9)) return nullptr;
  const Tensor q = tensor_or_none(a[0]), k = tensor_or_none(a[1]), v = tensor_or_none(a[2]);
  const Tensor ck = tensor_or_none(a[3]), cv = tensor_or_none(a[4]);
  Op op;
  op.scale = as_scale(a[5], q);
  op.G = as_int(a[6]); op.mode = as_int(a[7]); op.chunk_rows = as_int(a[8]);
  Out r;
  {
    NoGil no_gil;
    at::AutoGradMode no_grad(false);
    r = run_forward(op, q, k, v, ck, cv);
  }
  return wrap(r);
  END_HANDLE_TH_ERRORS
}

// backward(q, k, v, cached_k, cached_v, o, lse, dout, scale, G, mode, chunk_rows) -> (dq, dk, dv, d_cached_k, d_cached_v)
PyObject* py_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 12)) return nullptr;
  Tensor t[8];
  for (int i = 0; i < 8; ++i) t[i] = tensor_or_none(a[i]);
  Op op;
  op.scale = as_scale(a[8], t[0]);
  op.G = as_int(a[9]); op.mode = as_int(a[10]); op.chunk_rows = as_int(a[11]);
  Grads g;
  {
    NoGil no_gil;
    at::AutoGradMode no_grad(false);
    g = run_backward(op, t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], Tensor(), Tensor(), false);
  }
  PyObject* r = PyTuple_New(5);
  if (!r) return nullptr;
  const Tensor* out[5] = {&g.dq, &g.dk, &g.dv, &g.dck, &g.dcv};
  for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(r, i, wrap(*out[i]));      // an undefined tensor wraps to None
  return r;
  END_HANDLE_TH_ERRORS
}

constexpr const char* kStateName = "moda_b200.cache_state";
CacheStatePtr as_state(PyObject* x) {
  auto* p = static_cast<CacheStatePtr*>(PyCapsule_GetPointer(x, kStateName));
  if (!p) throw python_error();
  return *p;
}
// cache_state() -> a new state; cache_state(grad_k, grad_v): with these gradient caches (a copy of another's)
PyObject* py_cache_state(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 0 && !arg_count(n, 2)) return nullptr;
  auto state = std::make_shared<CacheState>();
  if (n != 0) {
    state->grad_k = tensor_or_none(a[0]);
    state->grad_v = tensor_or_none(a[1]);
  }
  return PyCapsule_New(new CacheStatePtr(std::move(state)), kStateName,
                       [](PyObject* c) { delete static_cast<CacheStatePtr*>(PyCapsule_GetPointer(c, kStateName)); });
  END_HANDLE_TH_ERRORS
}
PyObject* py_cache_grads(PyObject*, PyObject* x) {
  HANDLE_TH_ERRORS
  const CacheStatePtr s = as_state(x);
  return wrap(Out{s->grad_k, s->grad_v});
  END_HANDLE_TH_ERRORS
}

// cache_append(k, v, cache_k, cache_v, capacity, slot, token, state) -> token: the new one, or, where nothing is
// recorded, the one that came in, which keeps the appends before it on the chain
PyObject* py_cache_append(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 8)) return nullptr;
  const Tensor k = tensor_or_none(a[0]), v = tensor_or_none(a[1]), cache_k = tensor_or_none(a[2]), cache_v = tensor_or_none(a[3]);
  const Tensor token = tensor_or_none(a[6]);
  Op op;
  op.layers = 0;
  op.capacity = as_int(a[4]);
  op.scale = 1.;
  const int slot = as_int(a[5]);
  const CacheStatePtr state = as_state(a[7]);
  Tensor next = token;
  {
    NoGil no_gil;
    refuse_tangents({&k, &v});
    const bool grad = wants_grad({&k, &v, &token});
    moda_problem pr;
    {
      at::AutoGradMode no_grad(false);
      const Tensor k_ = in_place_or_copy(k), v_ = in_place_or_copy(v);
      pr = problem(op, k_, false, Tensor(), false);
      const c10::cuda::CUDAGuard guard(k.device());
      check_status(moda_b200_depth_append(&pr, T4(k_).p(), T4(v_).p(), T4(cache_k).p(), T4(cache_v).p(), slot,
                                          c10::cuda::getCurrentCUDAStream().stream()),
                   "moda_b200_depth_append");
      if (grad) next = at::empty({}, k.options().dtype(at::kFloat));       // only its place in the graph is used
    }
    if (grad) {
      std::shared_ptr<MoDADepthAppendBackward> node(new MoDADepthAppendBackward(), torch::autograd::deleteNode);
      node->state = state;
      node->pr = pr;
      node->slot = slot;
      node->set_next_edges(torch::autograd::collect_next_edges(k, v, token));
      torch::autograd::set_history(next, node);
    }
  }
  return wrap(next);
  END_HANDLE_TH_ERRORS
}

// cache_attention(q, k, v, cache_k, cache_v, scale, G, mode, layers, capacity, token, state) -> (o, lse)
PyObject* py_cache_attention(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (!arg_count(n, 12)) return nullptr;
  Tensor t[5];
  for (int i = 0; i < 5; ++i) t[i] = tensor_or_none(a[i]);
  Op op;
  op.scale = as_scale(a[5], t[0]);
  op.G = as_int(a[6]); op.mode = as_int(a[7]); op.layers = as_int(a[8]); op.capacity = as_int(a[9]);
  const Tensor token = tensor_or_none(a[10]);
  const CacheStatePtr state = as_state(a[11]);
  Out r;
  {
    NoGil no_gil;
    r = attention(op, t[0], t[1], t[2], t[3], t[4], state, token);
  }
  return wrap(r);
  END_HANDLE_TH_ERRORS
}

PyObject* py_set_path(PyObject*, PyObject* x) {
  const long v = PyLong_AsLong(x);
  if (v == -1 && PyErr_Occurred()) return nullptr;
  return PyLong_FromLong(g_path.exchange((int)v));
}
PyObject* py_set_check(PyObject*, PyObject* x) {
  Py_INCREF(x);
  Py_XDECREF(g_check);
  g_check = x;
  Py_RETURN_NONE;
}

#define MODA_FAST(f) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(f)), METH_FASTCALL
PyMethodDef kMethods[] = {{"attention", MODA_FAST(py_attention), nullptr},
                          {"forward", MODA_FAST(py_forward), nullptr},
                          {"backward", MODA_FAST(py_backward), nullptr},
                          {"cache_state", MODA_FAST(py_cache_state), nullptr},
                          {"cache_grads", py_cache_grads, METH_O, nullptr},
                          {"cache_append", MODA_FAST(py_cache_append), nullptr},
                          {"cache_attention", MODA_FAST(py_cache_attention), nullptr},
                          {"set_path", py_set_path, METH_O, nullptr},
                          {"set_check", py_set_check, METH_O, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
