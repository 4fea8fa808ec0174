// Native host path of the functions that a circuit loop calls per gate:
// argument checks, batch rules, output allocation, the C ABI call and the
// autograd nodes, without the interpreter in between.  On a state of a few
// MB a gate is a few microseconds of GPU time, and the same steps in Python
// take 19 (and 60 more with a gradient).
//
// Every function here takes the ordinary call (plain CUDA tensors of the
// engine's types, the batch forms below, no tensor subclass, mode, transform
// or tracer) and returns None for anything else: the Python function of the
// same name then runs its own checks, raises its own errors and handles what
// is left.  The kernels and their results are the same.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/ExpandUtils.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/core/grad_mode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <array>
#include <optional>
#include <vector>

#include "gbsv.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::Variable;
using torch::autograd::variable_list;
using Sizes = std::vector<int64_t>;

constexpr int kMaxQubits = GBSV_MAX_DENSE_QUBITS;

// A failed status.  In a call it sends the call to the Python function,
// which fails in its own way; in a backward it is a RuntimeError with
// GbsvError's text.
struct StatusError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
void check(int rc, const char* what) {
  if (rc != GBSV_OK)
    throw StatusError(std::string(what) + ": " + gbsv_status_string(rc) +
                      ": " + gbsv_last_error() + " (status " +
                      std::to_string(rc) + ")");
}

// Nothing that would see or change the operations between Python and the
// kernel: dispatch or function modes, functorch transforms, a tracer.
bool plain_context() {
  return !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         at::impl::PythonTorchFunctionTLS::stack_len() == 0 &&
         !c10::impl::tls_is_dispatch_key_included(
             c10::DispatchKey::FuncTorchDynamicLayerFrontMode) &&
         !torch::jit::tracer::isTracing();
}

// An ordinary strided CUDA tensor (not conjugated or negated lazily).
bool ordinary(const Tensor& t) {
  static const c10::DispatchKeySet allowed =
      c10::DispatchKeySet({c10::DispatchKey::CUDA,
                           c10::DispatchKey::ADInplaceOrView,
                           c10::DispatchKey::AutogradCUDA,
                           c10::DispatchKey::AutocastCUDA});
  return t.defined() && t.is_cuda() &&
         (t.unsafeGetTensorImpl()->key_set().raw_repr() &
          ~allowed.raw_repr()) == 0;
}
// The same without a forward-mode tangent.
bool plain(const Tensor& t) {
  return ordinary(t) && !t._fw_grad(/*level=*/0).defined();
}

// The tensor of a Python argument, if it is exactly a Tensor or Parameter.
Tensor unpack(PyObject* o) {
  if (!THPVariable_CheckExact(o) &&
      reinterpret_cast<PyObject*>(Py_TYPE(o)) != ParameterClass)
    return Tensor();
  const Tensor& t = THPVariable_Unpack(o);
  return plain(t) ? t : Tensor();
}

// Other Python threads run while a call allocates and launches: both can
// wait for the device (a full allocator, a full queue, behind which a host
// callback may need the interpreter).  The same calls through ctypes do so.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};
template <typename F>
PyObject* without_gil(F f) {
  Tensor out;
  {
    const WithoutGil w;
    out = f();
  }
  return THPVariable_Wrap(std::move(out));
}

bool needs_grad(const Tensor& a, const Tensor& b) {
  return at::GradMode::is_enabled() && (a.requires_grad() || b.requires_grad());
}
bool needs_grad(const Tensor& a) {
  return at::GradMode::is_enabled() && a.requires_grad();
}

// log2 of a power of two, or -1
int log2_exact(int64_t x) {
  return x > 0 && (x & (x - 1)) == 0 ? __builtin_ctzll((uint64_t)x) : -1;
}

int complex_code(at::ScalarType t) {
  return t == at::kComplexFloat ? GBSV_C64
         : t == at::kComplexDouble ? GBSV_C128
                                   : -1;
}
int real_code(at::ScalarType t) {
  return t == at::kFloat ? GBSV_F32 : t == at::kDouble ? GBSV_F64 : -1;
}
at::ScalarType real_of(at::ScalarType t) {
  return t == at::kComplexFloat ? at::kFloat : at::kDouble;
}

void* stream_of(const Tensor& t) {
  return c10::cuda::getCurrentCUDAStream(t.device().index()).stream();
}

int64_t product(c10::IntArrayRef s) {
  int64_t p = 1;
  for (int64_t x : s) p *= x;
  return p;
}

Tensor scratch(size_t bytes, const Tensor& like) {
  return bytes ? at::empty({(int64_t)bytes}, like.options().dtype(at::kByte))
               : Tensor();
}
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// How an (operator batch, state batch) pair maps onto the C ABI's strides;
// false for the forms left to Python (an operator batch that broadcasts onto
// another state batch, empty batches, errors).  `tail` dims of the operator
// are matrices.
struct Batch {
  Sizes out;           // output shape
  int64_t num_states = 1, in_stride = 0, op_stride = 0;
  bool expanded = false;  // an unbatched state under an operator batch
};
bool plan(const Tensor& op, int tail, int64_t op_size, const Tensor& state,
          int n, Batch* b) {
  const auto ob = op.sizes().slice(0, op.dim() - tail);
  const auto sb = state.sizes().slice(0, state.dim() - 1);
  const int64_t per_op = product(ob);
  if (ob.empty()) {
    b->out = sb.vec();
  } else if (sb.empty()) {
    b->out = ob.vec();
    b->expanded = true;
  } else if (ob == sb) {
    b->out = sb.vec();
  } else {
    return false;
  }
  b->num_states = product(b->out);
  b->in_stride = b->expanded ? 0 : int64_t(1) << n;
  b->op_stride = per_op > 1 ? op_size : 0;
  b->out.push_back(int64_t(1) << n);
  return b->num_states > 0;
}

// The qubits of a list, tuple or range of plain ints, distinct and in
// [0, n); nothing else is consumed or converted.
bool parse_qubits(PyObject* o, int n, int32_t* q, int* k) {
  if (!PyList_CheckExact(o) && !PyTuple_CheckExact(o) && !PyRange_Check(o))
    return false;
  PyObject* seq = PySequence_Fast(o, "qubits");
  if (!seq) {
    PyErr_Clear();
    return false;
  }
  const Py_ssize_t len = PySequence_Fast_GET_SIZE(seq);
  bool ok = len <= kMaxQubits;
  uint64_t seen = 0;
  for (Py_ssize_t i = 0; ok && i < len; ++i) {
    PyObject* x = PySequence_Fast_GET_ITEM(seq, i);
    ok = PyLong_CheckExact(x);
    if (!ok) break;
    int over = 0;
    const long v = PyLong_AsLongAndOverflow(x, &over);
    ok = !over && v >= 0 && v < n && !((seen >> v) & 1);
    if (!ok) break;
    seen |= uint64_t(1) << v;
    q[i] = (int32_t)v;
  }
  Py_DECREF(seq);
  *k = (int)len;
  return ok;
}

// ------------------------------------------------------- apply_operator --
struct Gate {
  Batch b;
  int n = 0, k = 0;
  std::array<int32_t, kMaxQubits> q{};
};

Tensor run_gate(const Tensor& ops, const Tensor& state, const Gate& g) {
  Tensor out = at::empty(g.b.out, state.options());
  check(gbsv_apply_operator(state.data_ptr(), out.data_ptr(),
                            complex_code(state.scalar_type()), g.n,
                            g.b.num_states, g.b.in_stride, ops.data_ptr(),
                            g.b.op_stride, g.q.data(), g.k,
                            stream_of(state)),
        "apply_operator");
  return out;
}

Tensor dense_grad(Tensor g) {
  return g.resolve_conj().resolve_neg().contiguous();
}

// Gradients summed over the states of a broadcast (one) state.
Tensor state_grad(const Tensor& gs, const Batch& b, int n,
                  c10::IntArrayRef shape) {
  if (b.expanded) return gs.reshape({-1, int64_t(1) << n}).sum(0).view(shape);
  return gs.view(shape);
}

struct ApplyOperator : public Function<ApplyOperator> {
  static Variable forward(AutogradContext* ctx, const Variable& op,
                          const Variable& state, const Gate& g) {
    const Tensor ops = op.contiguous(), sc = state.contiguous();
    Tensor out = run_gate(ops, sc, g);
    ctx->saved_data["op_shape"] = op.sizes().vec();
    ctx->saved_data["shape"] = state.sizes().vec();
    ctx->saved_data["out"] = g.b.out;
    ctx->saved_data["ints"] =
        Sizes{g.b.num_states, g.b.in_stride, g.b.op_stride, g.b.expanded,
              g.n, g.k};
    ctx->saved_data["q"] = Sizes(g.q.begin(), g.q.begin() + g.k);
    // the operator enters the state's gradient only
    ctx->save_for_backward({sc, state.requires_grad() ? ops : Tensor()});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    at::NoGradGuard no_grad;
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &sc = saved[0], &ops = saved[1];
    Gate g;
    const auto ints = ctx->saved_data["ints"].toIntVector();
    const auto q = ctx->saved_data["q"].toIntVector();
    g.b.out = ctx->saved_data["out"].toIntVector();
    g.b.num_states = ints[0];
    g.b.in_stride = ints[1];
    g.b.op_stride = ints[2];
    g.b.expanded = ints[3];
    g.n = (int)ints[4];
    g.k = (int)ints[5];
    std::copy(q.begin(), q.end(), g.q.begin());
    const Tensor go = dense_grad(gout[0]);
    const bool need_op = ctx->needs_input_grad(0);
    const bool need_state = ctx->needs_input_grad(1);
    const int code = complex_code(go.scalar_type());
    Tensor gs, gop;
    // complex64 gates on 1 or 2 qubits: both gradients in one pass
    const bool both =
        need_op && need_state && (g.k == 1 || g.k == 2) && code == GBSV_C64;
    if (need_state) gs = at::empty(go.sizes(), go.options());
    if (need_state && !both) {
      const Tensor dag =
          ops.conj().transpose(-1, -2).resolve_conj().contiguous();
      check(gbsv_apply_operator(go.data_ptr(), gs.data_ptr(), code, g.n,
                                g.b.num_states, int64_t(1) << g.n,
                                dag.data_ptr(), g.b.op_stride, g.q.data(),
                                g.k, stream_of(go)),
            "apply_operator");
    }
    if (need_op) {
      const int shared = g.b.op_stride == 0;
      const size_t bytes = gbsv_operator_grad_scratch_bytes(
          g.b.num_states, g.n, g.k, shared);
      const Tensor sp = scratch(bytes, go);
      gop = at::empty(ctx->saved_data["op_shape"].toIntVector(),
                      go.options());
      check(gbsv_apply_operator_grad(
                go.data_ptr(), sc.data_ptr(), code, g.n, g.b.num_states,
                g.b.in_stride, ptr(ops), g.b.op_stride, g.q.data(), g.k,
                both ? gs.data_ptr() : nullptr, gop.data_ptr(), shared,
                ptr(sp), bytes, stream_of(go)),
            "operator_grad");
    }
    if (need_state)
      gs = state_grad(gs, g.b, g.n, ctx->saved_data["shape"].toIntVector());
    return {gop, gs, Variable()};
  }
};

PyObject* none() { Py_RETURN_NONE; }

#define GBSV_CALL   \
  HANDLE_TH_ERRORS  \
  try {
#define GBSV_END_CALL            \
  }                              \
  catch (const StatusError&) {   \
    return none();               \
  }                              \
  END_HANDLE_TH_ERRORS

PyObject* py_apply_operator(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  if (na != 3 || !plain_context()) return none();
  const Tensor op = unpack(args[0]), state = unpack(args[2]);
  if (!op.defined() || !state.defined() ||
      op.scalar_type() != state.scalar_type() ||
      complex_code(state.scalar_type()) < 0 ||
      op.device() != state.device() || op.dim() < 2 || state.dim() < 1)
    return none();
  Gate g;
  g.n = log2_exact(state.size(-1));
  if (g.n < 0 || g.n > 62 || !parse_qubits(args[1], g.n, g.q.data(), &g.k) ||
      op.size(-1) != (int64_t(1) << g.k) || op.size(-2) != op.size(-1) ||
      !plan(op, 2, int64_t(1) << (2 * g.k), state, g.n, &g.b))
    return none();
  return without_gil([&]() -> Tensor {
    if (needs_grad(op, state)) return ApplyOperator::apply(op, state, g);
    return run_gate(op.contiguous(), state.contiguous(), g);
  });
  GBSV_END_CALL
}

// ------------------------------------- apply_all_qubits / each_qubit -----
struct Layer {
  Batch b;
  int n = 0;
  int64_t op_qstride = 0;  // 4: one operator per qubit
};

struct ApplyLayer : public Function<ApplyLayer> {
  static Variable forward(AutogradContext* ctx, const Variable& op,
                          const Variable& state, const Layer& l, int passes) {
    const Tensor ops = op.contiguous(), sc = state.contiguous();
    variable_list kept{sc};
    std::vector<void*> outs;
    Tensor out;
    for (int i = 0; i < passes; ++i) {
      out = at::empty(l.b.out, state.options());
      outs.push_back(out.data_ptr());
      if (i + 1 < passes) kept.push_back(out);
    }
    check(gbsv_apply_all_qubits_passes(
              sc.data_ptr(), outs.data(), complex_code(sc.scalar_type()),
              l.n, l.b.num_states, l.b.in_stride, ops.data_ptr(),
              l.b.op_stride, l.op_qstride, stream_of(sc)),
          "apply_all_qubits");
    ctx->saved_data["op_shape"] = op.sizes().vec();
    ctx->saved_data["shape"] = state.sizes().vec();
    ctx->saved_data["ints"] =
        Sizes{l.b.num_states, l.b.in_stride, l.b.op_stride, l.b.expanded, l.n,
              l.op_qstride};
    kept.push_back(ops);
    ctx->save_for_backward(kept);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    at::NoGradGuard no_grad;
    variable_list kept = ctx->get_saved_variables();
    const Tensor ops = kept.back();
    kept.pop_back();
    const auto ints = ctx->saved_data["ints"].toIntVector();
    Batch b;
    b.num_states = ints[0];
    b.in_stride = ints[1];
    b.op_stride = ints[2];
    b.expanded = ints[3];
    const int n = (int)ints[4];
    const int64_t qs = ints[5];
    const Tensor go = dense_grad(gout[0]);
    const bool need_op = ctx->needs_input_grad(0);
    const bool need_state = ctx->needs_input_grad(1);
    const int code = complex_code(go.scalar_type());
    Tensor gs, gop;
    if (need_state || (need_op && kept.size() > 1))
      gs = at::empty(go.sizes(), go.options());
    if (need_op) {
      const int shared = b.op_stride == 0;
      const size_t bytes = gbsv_all_qubits_grad_scratch_bytes(
          b.num_states, n, shared, qs != 0);
      const Tensor sp = scratch(bytes, go);
      gop = at::empty(ctx->saved_data["op_shape"].toIntVector(),
                      go.options());
      std::vector<const void*> in;
      for (const Tensor& t : kept) in.push_back(t.data_ptr());
      check(gbsv_apply_all_qubits_grad(
                go.data_ptr(), in.data(), code, n, b.num_states, b.in_stride,
                ops.data_ptr(), b.op_stride, qs, ptr(gs), need_state,
                gop.data_ptr(), shared, ptr(sp), bytes, stream_of(go)),
            "apply_all_qubits_grad");
    } else if (need_state) {
      const Tensor dag =
          ops.conj().transpose(-1, -2).resolve_conj().contiguous();
      check(gbsv_apply_all_qubits(go.data_ptr(), gs.data_ptr(), code, n,
                                  b.num_states, int64_t(1) << n,
                                  dag.data_ptr(), b.op_stride, qs,
                                  stream_of(go)),
            "apply_all_qubits");
    }
    if (!need_state) return {gop, Variable(), Variable(), Variable()};
    return {gop,
            state_grad(gs, b, n, ctx->saved_data["shape"].toIntVector()),
            Variable(), Variable()};
  }
};

// (operator, state, each): operator (*b, 2, 2), or (*b, n, 2, 2) with each.
PyObject* py_apply_layer(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  if (na != 3 || !plain_context()) return none();
  const Tensor op = unpack(args[0]), state = unpack(args[1]);
  const bool each = args[2] == Py_True;
  const int tail = each ? 3 : 2;
  if (!op.defined() || !state.defined() ||
      op.scalar_type() != state.scalar_type() ||
      complex_code(state.scalar_type()) < 0 ||
      op.device() != state.device() || op.dim() < tail || state.dim() < 1 ||
      op.size(-1) != 2 || op.size(-2) != 2)
    return none();
  Layer l;
  l.n = log2_exact(state.size(-1));
  if (l.n < 1 || l.n > 62 || (each && op.size(-3) != l.n) ||
      !plan(op, tail, each ? 4 * l.n : 4, state, l.n, &l.b))
    return none();
  l.op_qstride = each ? 4 : 0;
  const int code = complex_code(state.scalar_type());
  const bool grad = needs_grad(op, state);
  const int passes = grad ? gbsv_all_qubits_passes(code, l.n) : 0;
  if (grad && !passes) return none();  // one node per qubit, in Python
  return without_gil([&]() -> Tensor {
    if (grad) return ApplyLayer::apply(op, state, l, passes);
    const Tensor ops = op.contiguous(), sc = state.contiguous();
    Tensor out = at::empty(l.b.out, state.options());
    check(gbsv_apply_all_qubits(sc.data_ptr(), out.data_ptr(), code, l.n,
                                l.b.num_states, l.b.in_stride, ops.data_ptr(),
                                l.b.op_stride, l.op_qstride, stream_of(sc)),
          "apply_all_qubits");
    return out;
  });
  GBSV_END_CALL
}

// ------------------------------------------------------- broadcasting ----
// Element strides of t, made contiguous, broadcast to `shape`.
Sizes bcast_strides(const Tensor& t, c10::IntArrayRef shape) {
  const int64_t nd = (int64_t)shape.size(), off = nd - t.dim();
  Sizes s(nd, 0);
  const bool dense = t.is_contiguous();
  int64_t stride = 1;
  for (int64_t i = t.dim() - 1; i >= 0; --i) {
    s[off + i] = t.size(i) == 1 && shape[off + i] != 1 ? 0
                 : dense                               ? t.stride(i)
                                                       : stride;
    stride *= t.size(i);
  }
  return s;
}

// Unit dims dropped, dims contiguous in both operands merged; false when
// more remain than the descriptor holds.
bool bcast_desc(c10::IntArrayRef shape, c10::IntArrayRef sa,
                c10::IntArrayRef sb, gbsv_bcast_t* d) {
  std::memset(d, 0, sizeof(*d));
  int nd = 0;
  for (size_t i = 0; i < shape.size(); ++i) {
    if (shape[i] == 1) continue;
    if (nd && d->stride_a[nd - 1] == sa[i] * shape[i] &&
        d->stride_b[nd - 1] == sb[i] * shape[i]) {
      d->shape[nd - 1] *= shape[i];
      d->stride_a[nd - 1] = sa[i];
      d->stride_b[nd - 1] = sb[i];
      continue;
    }
    if (nd == GBSV_MAX_DIMS) return false;
    d->shape[nd] = shape[i];
    d->stride_a[nd] = sa[i];
    d->stride_b[nd] = sb[i];
    ++nd;
  }
  if (nd == 0) {
    d->shape[0] = 1;
    nd = 1;
  }
  d->ndim = nd;
  return true;
}

std::optional<Sizes> broadcast(const Tensor& a, const Tensor& b) {
  const int64_t nd = std::max(a.dim(), b.dim());
  Sizes s(nd);
  for (int64_t i = 0; i < nd; ++i) {
    const int64_t x = i < nd - a.dim() ? 1 : a.size(i - (nd - a.dim()));
    const int64_t y = i < nd - b.dim() ? 1 : b.size(i - (nd - b.dim()));
    if (x != y && x != 1 && y != 1) return std::nullopt;
    s[i] = x == 1 ? y : x;
  }
  return s;
}

// Tensor.sum_to_size
Tensor sum_to_size(const Tensor& t, c10::IntArrayRef shape) {
  TORCH_CHECK(at::is_expandable_to(shape, t.sizes()), "size {", shape,
              "} is not expandable to size {", t.sizes(), "}.");
  return at::sum_to(t, shape);
}

// ---------------------------------------------------------- apply_phase --
Tensor run_phase(const Tensor& a, const Tensor& s, c10::IntArrayRef shape,
                 const gbsv_bcast_t& d) {
  const auto dt = a.scalar_type() == at::kDouble ||
                          s.scalar_type() == at::kComplexDouble
                      ? at::kComplexDouble
                      : at::kComplexFloat;
  Tensor out = at::empty(shape, s.options().dtype(dt));
  check(gbsv_apply_phase(a.data_ptr(), real_code(a.scalar_type()),
                         s.data_ptr(), complex_code(s.scalar_type()),
                         out.data_ptr(), complex_code(dt), &d, stream_of(s)),
        "apply_phase");
  return out;
}

struct ApplyPhase : public Function<ApplyPhase> {
  static Variable forward(AutogradContext* ctx, const Variable& angles,
                          const Variable& state, const Sizes& shape,
                          const gbsv_bcast_t& d) {
    Tensor out = run_phase(angles.contiguous(), state.contiguous(), shape, d);
    ctx->save_for_backward({angles, state, out});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &angles = saved[0], &state = saved[1], &out = saved[2];
    const bool need_a = ctx->needs_input_grad(0);
    const bool need_s = ctx->needs_input_grad(1);
    Tensor ga, gs;
    if (at::GradMode::is_enabled() && need_a) {
      // create_graph: the angles' gradient stays differentiable
      const Tensor g = gout[0];
      ga = at::real(g * out.conj() * c10::complex<double>(0, 1));
    }
    {
      at::NoGradGuard no_grad;
      const Tensor a = angles.detach().contiguous();
      const Tensor g = dense_grad(gout[0]);
      const bool kernel_a = need_a && !ga.defined();
      if (need_s) gs = at::empty(g.sizes(), g.options());
      if (kernel_a)
        ga = at::empty(g.sizes(),
                       g.options().dtype(real_of(g.scalar_type())));
      gbsv_bcast_t d;
      // the forward call's descriptor held, so this one does
      TORCH_CHECK(bcast_desc(g.sizes(), bcast_strides(a, g.sizes()),
                             bcast_strides(g, g.sizes()), &d),
                  "apply_phase: too many broadcast dims");
      check(gbsv_apply_phase_grad(
                a.data_ptr(), real_code(a.scalar_type()), g.data_ptr(),
                out.data_ptr(), complex_code(g.scalar_type()), &d, ptr(gs),
                kernel_a ? ga.data_ptr() : nullptr, stream_of(g)),
            "apply_phase_grad");
      if (need_s)
        gs = sum_to_size(gs.to(state.scalar_type()), state.sizes());
    }
    if (need_a) ga = sum_to_size(ga.to(angles.scalar_type()), angles.sizes());
    return {ga, gs, Variable(), Variable()};
  }
};

PyObject* py_apply_phase(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  if (na != 2 || !plain_context()) return none();
  const Tensor a = unpack(args[0]), s = unpack(args[1]);
  if (!a.defined() || !s.defined() || a.device() != s.device() ||
      real_code(a.scalar_type()) < 0 || complex_code(s.scalar_type()) < 0 ||
      a.numel() == 0 || s.numel() == 0)
    return none();
  const auto shape = broadcast(a, s);
  gbsv_bcast_t d;
  if (!shape || !bcast_desc(*shape, bcast_strides(a, *shape),
                            bcast_strides(s, *shape), &d))
    return none();
  return without_gil([&]() -> Tensor {
    if (needs_grad(a, s)) return ApplyPhase::apply(a, s, *shape, d);
    return run_phase(a.contiguous(), s.contiguous(), *shape, d);
  });
  GBSV_END_CALL
}

// ----------------------------------------------------------- reductions --
Tensor run_norm(const Tensor& state) {
  const Tensor s = state.contiguous();
  const int64_t dim = s.size(-1), rows = s.numel() / dim;
  const auto real = real_of(s.scalar_type());
  Tensor out = at::empty(s.sizes().slice(0, s.dim() - 1),
                         s.options().dtype(real));
  const size_t bytes = gbsv_reduce_scratch_bytes(rows, dim);
  const Tensor sp = scratch(bytes, s);
  check(gbsv_norm_squared(s.data_ptr(), complex_code(s.scalar_type()), rows,
                          dim, out.data_ptr(), real_code(real), ptr(sp),
                          bytes, stream_of(s)),
        "norm_squared");
  return out;
}

struct NormSquared : public Function<NormSquared> {
  static Variable forward(AutogradContext* ctx, const Variable& state) {
    ctx->save_for_backward({state});
    return run_norm(state);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor state = ctx->get_saved_variables()[0];
    return {2 * g[0].unsqueeze(-1) * state};
  }
};

Tensor run_abs(const Tensor& state) {
  const Tensor s = state.contiguous();
  Tensor out = at::empty(s.sizes(),
                         s.options().dtype(real_of(s.scalar_type())));
  check(gbsv_abs_squared(s.data_ptr(), complex_code(s.scalar_type()),
                         s.numel(), out.data_ptr(), stream_of(s)),
        "abs_squared");
  return out;
}

struct AbsSquared : public Function<AbsSquared> {
  static Variable forward(AutogradContext* ctx, const Variable& state) {
    ctx->save_for_backward({state});
    return run_abs(state);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const Tensor state = ctx->get_saved_variables()[0];
    return {2 * g[0] * state};
  }
};

// A complex state of at least one amplitude.
Tensor state_arg(PyObject* o) {
  const Tensor s = unpack(o);
  return s.defined() && s.dim() >= 1 && s.numel() > 0 &&
                 complex_code(s.scalar_type()) >= 0
             ? s
             : Tensor();
}

PyObject* py_norm_squared(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  const Tensor s =
      na == 1 && plain_context() ? state_arg(args[0]) : Tensor();
  if (!s.defined()) return none();
  return without_gil([&]() -> Tensor {
    return needs_grad(s) ? NormSquared::apply(s) : run_norm(s);
  });
  GBSV_END_CALL
}

PyObject* py_abs_squared(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  const Tensor s =
      na == 1 && plain_context() ? state_arg(args[0]) : Tensor();
  if (!s.defined()) return none();
  return without_gil([&]() -> Tensor {
    return needs_grad(s) ? AbsSquared::apply(s) : run_abs(s);
  });
  GBSV_END_CALL
}

// Rows of two broadcast (*batch, dim) tensors, made contiguous.
struct Rows {
  Sizes shape;  // without the inner dim
  gbsv_bcast_t d;
  int64_t dim = 1, ia = 0, ib = 0;
};
bool plan_rows(const Tensor& a, const Tensor& b, Rows* r) {
  const auto shape = broadcast(a, b);
  if (!shape || shape->empty()) return false;
  const Sizes sa = bcast_strides(a, *shape), sb = bcast_strides(b, *shape);
  const size_t nd = shape->size() - 1;
  r->dim = shape->back();
  r->ia = sa[nd];
  r->ib = sb[nd];
  r->shape.assign(shape->begin(), shape->begin() + nd);
  return bcast_desc(r->shape, c10::IntArrayRef(sa.data(), nd),
                    c10::IntArrayRef(sb.data(), nd), &r->d);
}

Tensor run_inner(const Tensor& a, const Tensor& b, const Rows& r) {
  Tensor out = at::empty(r.shape, a.options());
  const size_t bytes = gbsv_reduce_scratch_bytes(out.numel(), r.dim);
  const Tensor sp = scratch(bytes, a);
  const int code = complex_code(a.scalar_type());
  check(gbsv_inner_product(a.data_ptr(), b.data_ptr(), code, &r.d, r.dim,
                           r.ia, r.ib, out.data_ptr(), code, ptr(sp), bytes,
                           stream_of(a)),
        "inner_product");
  return out;
}

struct InnerProduct : public Function<InnerProduct> {
  static Variable forward(AutogradContext* ctx, const Variable& a,
                          const Variable& b, const Rows& r) {
    ctx->save_for_backward({a, b});
    return run_inner(a.contiguous(), b.contiguous(), r);
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &a = saved[0], &b = saved[1];
    const Tensor g = gout[0].unsqueeze(-1);
    Tensor ga, gb;
    if (ctx->needs_input_grad(0))
      ga = sum_to_size(g.conj() * b, a.sizes());
    if (ctx->needs_input_grad(1)) gb = sum_to_size(g * a, b.sizes());
    return {ga, gb, Variable()};
  }
};

PyObject* py_inner_product(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  if (na != 2 || !plain_context()) return none();
  const Tensor a = state_arg(args[0]), b = state_arg(args[1]);
  if (!a.defined() || !b.defined() || a.scalar_type() != b.scalar_type() ||
      a.device() != b.device())
    return none();
  Rows r;
  if (!plan_rows(a, b, &r)) return none();
  return without_gil([&]() -> Tensor {
    if (needs_grad(a, b)) return InnerProduct::apply(a, b, r);
    return run_inner(a.contiguous(), b.contiguous(), r);
  });
  GBSV_END_CALL
}

Tensor run_diag(const Tensor& d, const Tensor& s, const Rows& r) {
  const auto dt = at::promote_types(real_of(s.scalar_type()),
                                    d.scalar_type());
  Tensor out = at::empty(r.shape, s.options().dtype(dt));
  const size_t bytes = gbsv_reduce_scratch_bytes(out.numel(), r.dim);
  const Tensor sp = scratch(bytes, s);
  check(gbsv_diag_expectation(d.data_ptr(), real_code(d.scalar_type()),
                              s.data_ptr(), complex_code(s.scalar_type()),
                              &r.d, r.dim, r.ia, r.ib, out.data_ptr(),
                              real_code(dt), ptr(sp), bytes, stream_of(s)),
        "diag_expectation_value");
  return out;
}

struct DiagExpectation : public Function<DiagExpectation> {
  static Variable forward(AutogradContext* ctx, const Variable& d,
                          const Variable& s, const Rows& r) {
    ctx->save_for_backward({d, s});
    return run_diag(d.contiguous(), s.contiguous(), r);
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    const variable_list saved = ctx->get_saved_variables();
    const Tensor &d = saved[0], &s = saved[1];
    const Tensor g = gout[0].unsqueeze(-1);
    Tensor gd, gs;
    if (ctx->needs_input_grad(0))
      gd = sum_to_size((g * at::real(s.conj() * s)).to(d.scalar_type()),
                      d.sizes());
    if (ctx->needs_input_grad(1))
      gs = sum_to_size((2 * g * d * s).to(s.scalar_type()), s.sizes());
    return {gd, gs, Variable()};
  }
};

PyObject* py_diag(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  if (na != 2 || !plain_context()) return none();
  const Tensor d = unpack(args[0]), s = state_arg(args[1]);
  if (!d.defined() || !s.defined() || d.dim() < 1 || d.numel() == 0 ||
      real_code(d.scalar_type()) < 0 || d.device() != s.device())
    return none();
  Rows r;
  if (!plan_rows(d, s, &r)) return none();
  return without_gil([&]() -> Tensor {
    if (needs_grad(d, s)) return DiagExpectation::apply(d, s, r);
    return run_diag(d.contiguous(), s.contiguous(), r);
  });
  GBSV_END_CALL
}


// ------------------------------------------------------- rotation gates --
// The angles as the kernel reads them: a dim of any stride, or dense.
int64_t angle_stride(const Tensor& a) {
  return a.dim() == 1 && a.size(0) > 1 ? a.stride(0) : 1;
}

Tensor run_rotation(const Tensor& a, int axis) {
  const auto dt = a.scalar_type() == at::kDouble ? at::kComplexDouble
                                                 : at::kComplexFloat;
  Sizes shape = a.sizes().vec();
  shape.insert(shape.end(), {2, 2});
  Tensor out = at::empty(shape, a.options().dtype(dt));
  check(gbsv_rotation_gates(a.data_ptr(), complex_code(dt), angle_stride(a),
                            a.numel(), axis, out.data_ptr(), stream_of(a)),
        "rotation_gates");
  return out;
}

Tensor angles_of(const Tensor& a) {
  return a.dim() <= 1 && angle_stride(a) >= 0 ? a : a.contiguous();
}

struct Rotation : public Function<Rotation> {
  static Variable forward(AutogradContext* ctx, const Variable& angles,
                          int64_t axis) {
    ctx->save_for_backward({angles});
    ctx->saved_data["axis"] = axis;
    return run_rotation(angles_of(angles), (int)axis);
  }
  static variable_list backward(AutogradContext* ctx, variable_list gout) {
    const Tensor angles = ctx->get_saved_variables()[0];
    const int axis = (int)ctx->saved_data["axis"].toInt();
    if (at::GradMode::is_enabled()) {  // create_graph: differentiable again
      const Tensor g = gout[0];
      const Tensor g00 = g.select(-1, 0).select(-1, 0);
      const Tensor g01 = g.select(-1, 1).select(-1, 0);
      const Tensor g10 = g.select(-1, 0).select(-1, 1);
      const Tensor g11 = g.select(-1, 1).select(-1, 1);
      const Tensor off = axis == 0   ? -(at::imag(g01) + at::imag(g10))
                         : axis == 1 ? at::real(g10) - at::real(g01)
                                     : at::imag(g11) - at::imag(g00);
      return {angles.cos() * off -
                  angles.sin() * (at::real(g00) + at::real(g11)),
              Variable()};
    }
    const Tensor a = angles_of(angles.detach()), g = dense_grad(gout[0]);
    Tensor ga = at::empty(a.sizes(), a.options());
    check(gbsv_rotation_gates_grad(a.data_ptr(),
                                   complex_code(g.scalar_type()),
                                   angle_stride(a), a.numel(), axis,
                                   g.data_ptr(), ga.data_ptr(), stream_of(a)),
          "rotation_gates_grad");
    return {ga, Variable()};
  }
};

// (axis, angles): exp(-i a P), complex in the angles' precision.
PyObject* py_rotation(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  if (na != 2 || !PyLong_CheckExact(args[0]) || !plain_context())
    return none();
  const long axis = PyLong_AsLong(args[0]);
  const Tensor a = unpack(args[1]);
  if (!a.defined() || axis < 0 || axis > 2 || real_code(a.scalar_type()) < 0 ||
      a.numel() == 0)
    return none();
  return without_gil([&]() -> Tensor {
    return needs_grad(a) ? Rotation::apply(a, (int64_t)axis)
                         : run_rotation(angles_of(a), (int)axis);
  });
  GBSV_END_CALL
}

// (tensor): the tensor itself where its memory holds its values in order.
PyObject* py_dense(PyObject*, PyObject* const* args, Py_ssize_t na) {
  GBSV_CALL
  if (na != 1 || !THPVariable_CheckExact(args[0])) return none();
  const Tensor& t = THPVariable_Unpack(args[0]);
  if (!ordinary(t) || !t.is_contiguous()) return none();
  Py_INCREF(args[0]);
  return args[0];
  GBSV_END_CALL
}

PyMethodDef kMethods[] = {
    {"dense",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_dense)),
     METH_FASTCALL, "(tensor) -> the same Tensor or None"},
    {"rotation",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_rotation)),
     METH_FASTCALL, "(axis, angles) -> Tensor or None"},
    {"apply_operator",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_apply_operator)),
     METH_FASTCALL, "(operator, qubits, state) -> Tensor or None"},
    {"apply_layer",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_apply_layer)),
     METH_FASTCALL, "(operator, state, each) -> Tensor or None"},
    {"apply_phase",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_apply_phase)),
     METH_FASTCALL, "(angles, state) -> Tensor or None"},
    {"norm_squared",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_norm_squared)),
     METH_FASTCALL, "(state) -> Tensor or None"},
    {"abs_squared",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_abs_squared)),
     METH_FASTCALL, "(state) -> Tensor or None"},
    {"inner_product",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_inner_product)),
     METH_FASTCALL, "(state_1, state_2) -> Tensor or None"},
    {"diag_expectation_value",
     reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_diag)),
     METH_FASTCALL, "(diagonal, state) -> Tensor or None"},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_gbsv_host",
                       "Native host path of the engine's functions.", -1,
                       kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__gbsv_host(void) { return PyModule_Create(&kModule); }
