// Python binding of the autograd entry points: LFWFunction.apply, DFWFunction.apply,
// LFWFusedFunction.apply and lfw_decode_step as C functions of the extension module that this library
// also is.
//
// Why: a call on a small problem is bound by the host.  Through a Python autograd function and torch.ops
// one token of 32 rows cost 18 us of host time around a 3 us kernel, and a backward pass had to wait for
// the interpreter on the engine's thread.  Here the arguments are unpacked straight from the argument
// vector, the graph node is a C++ node, and without gradients no node is made at all.
//
// A call that is not the plain case (an argument that is no tensor, a tensor subclass, a dual tensor, a failed shape
// or type check, tracing, a function transform) is handed to the Python class, which then raises, or does,
// what it always did.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/object_ptr.h>
#include <torch/csrc/utils/pybind.h>
#include <ATen/core/PythonFallbackKernel.h>
#include <ATen/FuncTorchTLS.h>

#include "torch_ops.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// The last slot of a checkpoint array as a tensor of its own.  With gradients it is an ordinary view (an
// in-place change of it is then noticed by autograd); without, nothing is saved and the view's
// bookkeeping is left out.
Tensor last_slot(const Tensor &ckpt, bool tracked) {
  const int64_t slots = ckpt.size(1);
  if (tracked) return ckpt.select(1, slots - 1);
  Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(ckpt.storage()), ckpt.key_set(), ckpt.dtype());
  const int64_t D = ckpt.size(2), K = ckpt.size(3);
  const int64_t sizes[3] = {ckpt.size(0), D, K}, strides[3] = {slots * D * K, K, 1};
  t.unsafeGetTensorImpl()->set_sizes_and_strides(sizes, strides, ckpt.storage_offset() + (slots - 1) * D * K);
  return t;
}

// Gradients formed in grad mode (create_graph) from tensors that require gradients: there is no second derivative, so
// they hang on a node that raises when one runs into it.  Left as they are they would be constants, and that derivative
// silently zero.  The node's edges lead to those tensors, so that a search for a path to one of them finds it.
variable_list no_second_derivative(variable_list grads, const variable_list &upstream, const variable_list &saved) {
  if (!at::GradMode::is_enabled()) return grads;
  auto needs = [](const variable_list &l) {
    for (const Tensor &t : l)
      if (t.requires_grad()) return true;
    return false;
  };
  if (!needs(upstream) && !needs(saved)) return grads;
  std::shared_ptr<torch::autograd::Node> node(new torch::autograd::NotImplemented("the backward of t2fw's recurrences"),
                                              torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(upstream, saved));
  for (const Tensor &g : grads) torch::autograd::set_history(g, node);      // fresh tensors of this call
  return grads;
}

// `state` of a T > 1 call may be the strided last slot of another call's checkpoints: the operators ask for
// contiguous tensors and say so themselves.
struct LfwNode : torch::autograd::Function<LfwNode> {
  static variable_list forward(AutogradContext *ctx, const Tensor &x, const Tensor &f, const Tensor &q,
                               const Tensor &k, const Tensor &fk, const Tensor &s) {
    auto r = t2fw_ops::lfw_forward(x, f, q, k, fk, s);
    ctx->save_for_backward({x, f, q, k, fk, s, r[1]});
    return {r[0], last_slot(r[1], true)};
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    const auto v = ctx->get_saved_variables();
    return no_second_derivative(t2fw_ops::lfw_backward(g[0].contiguous(), g[1].contiguous(), v[0], v[1], v[2], v[3], v[4],
                                                       v[0], v[5], v[6]), g, v);
  }
};

struct DfwNode : torch::autograd::Function<DfwNode> {
  static variable_list forward(AutogradContext *ctx, const Tensor &q, const Tensor &k, const Tensor &v,
                               const Tensor &s) {
    auto r = t2fw_ops::dfw_forward(q, k, v, s);
    ctx->save_for_backward({q, k, r[2], r[1]});
    return {r[0], r[1]};
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    const auto v = ctx->get_saved_variables();
    return no_second_derivative(t2fw_ops::dfw_backward(g[0].contiguous(), g[1].contiguous(), v[0], v[1], v[2], v[3]), g, v);
  }
};

struct FusedNode : torch::autograd::Function<FusedNode> {
  static variable_list forward(AutogradContext *ctx, const Tensor &qkvg, const Tensor &state, int64_t n_head) {
    auto r = t2fw_ops::lfw_fused_forward(qkvg, state, n_head);
    ctx->save_for_backward({qkvg, state, r[1]});
    ctx->saved_data["n_head"] = n_head;
    return {r[0], last_slot(r[1], true)};
  }
  static variable_list backward(AutogradContext *ctx, variable_list g) {
    const auto v = ctx->get_saved_variables();
    auto r = no_second_derivative(t2fw_ops::lfw_fused_backward(g[0].contiguous(), g[1].contiguous(), v[0], v[1], v[2],
                                                               ctx->saved_data["n_head"].toInt()), g, v);
    return {r[0], r[1], Tensor()};
  }
};

// ---- argument handling --------------------------------------------------------------------------
PyObject *g_fallback[3] = {nullptr, nullptr, nullptr};      // Python's LFWFunction / DFWFunction / LFWFusedFunction apply

PyObject *call_fallback(int which, PyObject *const *args, Py_ssize_t n) {
  if (g_fallback[which] == nullptr) {
    PyErr_SetString(PyExc_RuntimeError, "t2fw: the Python classes are not loaded");
    return nullptr;
  }
  return PyObject_Vectorcall(g_fallback[which], args, (size_t)n, nullptr);
}

// plain tensors only: exact type (or nn.Parameter), no Python dispatch, no wrapped function-transform levels, no
// forward-mode tangent (which an entry point without a jvp would drop: the class raises)
bool plain_tensor(PyObject *o) {
  if (!THPVariable_Check(o)) return false;
  const Tensor &t = THPVariable_Unpack(o);
  if (!THPVariable_CheckExact(o) && !(ParameterClass != nullptr && (PyObject *)Py_TYPE(o) == ParameterClass)) return false;
  const auto ks = t.key_set();
  return t.defined() && t.is_cuda() && !ks.has(c10::DispatchKey::Python) && !ks.has(c10::DispatchKey::FuncTorchGradWrapper) &&
         !ks.has(c10::DispatchKey::FuncTorchBatched) &&
         (t.unsafeGetTensorImpl()->autograd_meta() == nullptr || !t._fw_grad(/*level=*/0).defined());
}

bool plain_mode() {
  const auto &ft = at::functorch::functorchTLSAccessor();
  if (ft) {
    try {
      ft->checkSupportsCppAutogradFunction();
    } catch (...) {
      return false;
    }
  }
  return !torch::jit::tracer::isTracing() && !c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::Python);
}

bool any_requires_grad(const Tensor *const *t, int n) {
  if (!at::GradMode::is_enabled()) return false;
  for (int i = 0; i < n; ++i)
    if (t[i]->requires_grad()) return true;
  return false;
}

PyObject *pair_to_python(Tensor a, Tensor b) {
  PyObject *tup = PyTuple_New(2);
  if (tup == nullptr) throw python_error();
  PyTuple_SET_ITEM(tup, 0, THPVariable_Wrap(std::move(a)));
  PyTuple_SET_ITEM(tup, 1, THPVariable_Wrap(std::move(b)));
  return tup;
}

PyObject *py_lfw_apply(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool ok = n == 6 && plain_mode();
  for (int i = 0; ok && i < 6; ++i) ok = plain_tensor(args[i]);
  if (ok) {
    const Tensor &x = THPVariable_Unpack(args[0]), &f = THPVariable_Unpack(args[1]), &q = THPVariable_Unpack(args[2]);
    const Tensor &k = THPVariable_Unpack(args[3]), &fk = THPVariable_Unpack(args[4]), &s = THPVariable_Unpack(args[5]);
    const auto dt = x.scalar_type();
    // the class's own assertions (same contract as t2fw/functional_lfw.py:42-49)
    if (x.sizes() == f.sizes() && q.sizes() == k.sizes() && q.sizes() == fk.sizes() && f.scalar_type() == dt &&
        q.scalar_type() == dt && fk.scalar_type() == dt && s.scalar_type() == dt) {
      const Tensor *all[6] = {&x, &f, &q, &k, &fk, &s};
      Tensor out, nxt;
      {
        pybind11::gil_scoped_release no_gil;
        if (any_requires_grad(all, 6)) {
          auto r = LfwNode::apply(x, f, q, k, fk, s);
          out = std::move(r[0]);
          nxt = std::move(r[1]);
        } else {
          auto r = t2fw_ops::lfw_forward(x, f, q, k, fk, s);
          out = std::move(r[0]);
          nxt = last_slot(r[1], false);
        }
      }
      return pair_to_python(std::move(out), std::move(nxt));
    }
  }
  return call_fallback(0, args, n);
  END_HANDLE_TH_ERRORS
}

PyObject *py_dfw_apply(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool ok = n == 4 && plain_mode();
  for (int i = 0; ok && i < 4; ++i) ok = plain_tensor(args[i]);
  if (ok) {
    const Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
    const Tensor &s = THPVariable_Unpack(args[3]);
    // the class's own assertions (same contract as t2fw/functional_dfw.py:38-40)
    if (q.sizes() == k.sizes() && q.scalar_type() == v.scalar_type() && s.scalar_type() == v.scalar_type()) {
      const Tensor *all[4] = {&q, &k, &v, &s};
      Tensor out, fin;
      {
        pybind11::gil_scoped_release no_gil;
        auto r = any_requires_grad(all, 4) ? DfwNode::apply(q, k, v, s) : t2fw_ops::dfw_forward(q, k, v, s);
        out = std::move(r[0]);
        fin = std::move(r[1]);
      }
      return pair_to_python(std::move(out), std::move(fin));
    }
  }
  return call_fallback(1, args, n);
  END_HANDLE_TH_ERRORS
}

PyObject *py_fused_apply(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n == 3 && plain_mode() && plain_tensor(args[0]) && plain_tensor(args[1]) && PyLong_CheckExact(args[2])) {
    const Tensor &qkvg = THPVariable_Unpack(args[0]), &state = THPVariable_Unpack(args[1]);
    int overflow = 0;      // then the number is -1, which the class refuses
    const long h = PyLong_AsLongAndOverflow(args[2], &overflow);
    if (h > 0 && qkvg.dim() == 3 && h <= qkvg.size(2) && qkvg.size(2) == 4 * h * 64 && state.dim() == 3 && state.size(0) == qkvg.size(0) * h &&
        state.size(1) == 64 && state.size(2) == 64 && qkvg.scalar_type() == state.scalar_type() &&
        qkvg.is_contiguous() && state.is_contiguous()) {
      const Tensor *all[2] = {&qkvg, &state};
      Tensor out, nxt;
      {
        pybind11::gil_scoped_release no_gil;
        if (any_requires_grad(all, 2)) {
          auto r = FusedNode::apply(qkvg, state, (int64_t)h);
          out = std::move(r[0]);
          nxt = std::move(r[1]);
        } else {
          auto r = t2fw_ops::lfw_fused_forward(qkvg, state, h);
          out = std::move(r[0]);
          nxt = last_slot(r[1], false);
        }
      }
      return pair_to_python(std::move(out), std::move(nxt));
    }
  }
  return call_fallback(2, args, n);
  END_HANDLE_TH_ERRORS
}

// decode_step(x, f, query, key, f_key, state_in, state_out, outputs): None, or NotImplemented if the
// arguments are not plain CUDA tensors (the caller then goes through torch.ops)
PyObject *py_decode_step(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool ok = n == 8 && plain_mode();
  for (int i = 0; ok && i < 8; ++i) ok = plain_tensor(args[i]);
  if (!ok) Py_RETURN_NOTIMPLEMENTED;
  const Tensor *t[8];
  for (int i = 0; i < 8; ++i) t[i] = &THPVariable_Unpack(args[i]);
  {
    pybind11::gil_scoped_release no_gil;
    t2fw_ops::lfw_decode_step(*t[0], *t[1], *t[2], *t[3], *t[4], *t[5], *t[6], *t[7]);
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// decode_ring(x, f, query, key, f_key, state, outputs): whether the whole ring was done in one launch
PyObject *py_decode_ring(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  bool ok = n == 7 && plain_mode();
  for (int i = 0; ok && i < 7; ++i) ok = plain_tensor(args[i]);
  if (!ok) Py_RETURN_FALSE;
  const Tensor *t[7];
  for (int i = 0; i < 7; ++i) t[i] = &THPVariable_Unpack(args[i]);
  {
    pybind11::gil_scoped_release no_gil;
    ok = t2fw_ops::lfw_decode_ring(*t[0], *t[1], *t[2], *t[3], *t[4], *t[5], *t[6]);
  }
  return PyBool_FromLong(ok);
  END_HANDLE_TH_ERRORS
}

// no_second_derivative(gradients, upstream and saved tensors) -> gradients: for the Python classes
PyObject *py_no_second_derivative(PyObject *, PyObject *const *args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  variable_list l[2];
  for (int i = 0; i < 2; ++i) {
    TORCH_CHECK(n == 2 && (PyTuple_Check(args[i]) || PyList_Check(args[i])), "no_second_derivative(gradients, tensors)");
    for (Py_ssize_t j = 0; j < PySequence_Fast_GET_SIZE(args[i]); ++j) {
      PyObject *o = PySequence_Fast_GET_ITEM(args[i], j);
      TORCH_CHECK(THPVariable_Check(o), "no_second_derivative: tensors expected");
      l[i].push_back(THPVariable_Unpack(o));
    }
  }
  const variable_list r = no_second_derivative(l[0], l[1], {});
  THPObjectPtr tup(PyTuple_New((Py_ssize_t)r.size()));
  if (!tup) throw python_error();
  for (size_t j = 0; j < r.size(); ++j) PyTuple_SET_ITEM(tup.get(), (Py_ssize_t)j, THPVariable_Wrap(r[j]));
  return tup.release();
  END_HANDLE_TH_ERRORS
}

// set_fallback(which, callable): 0 LFWFunction, 1 DFWFunction, 2 LFWFusedFunction
PyObject *py_set_fallback(PyObject *, PyObject *const *args, Py_ssize_t n) {
  const long w = n == 2 ? PyLong_AsLong(args[0]) : -1;
  if (w < 0 || w > 2 || !PyCallable_Check(args[1])) {
    PyErr_SetString(PyExc_ValueError, "set_fallback(which, callable)");
    return nullptr;
  }
  Py_INCREF(args[1]);
  Py_XSETREF(g_fallback[w], args[1]);
  Py_RETURN_NONE;
}

#define T2FW_METHOD(name, fn, doc) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, doc}
PyMethodDef g_methods[] = {
    T2FW_METHOD("lfw_apply", py_lfw_apply, "apply(value, forget, query, key, f_key, state) -> (outputs, next_state)"),
    T2FW_METHOD("dfw_apply", py_dfw_apply, "apply(query, key, value, state) -> (outputs, final_state)"),
    T2FW_METHOD("fused_apply", py_fused_apply, "apply(qkvg, state, n_head) -> (outputs, next_state)"),
    T2FW_METHOD("decode_step", py_decode_step, "decode_step(x, f, query, key, f_key, state_in, state_out, outputs)"),
    T2FW_METHOD("decode_ring", py_decode_ring, "decode_ring(x, f, query, key, f_key, state, outputs) -> bool"),
    T2FW_METHOD("no_second_derivative", py_no_second_derivative, "no_second_derivative(gradients, tensors) -> gradients"),
    T2FW_METHOD("set_fallback", py_set_fallback, "set_fallback(which, callable)"),
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "t2fw_torch_ops", "Autograd entry points of t2fw_b200.", -1, g_methods,
                        nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_t2fw_torch_ops(void) { return PyModule_Create(&g_module); }
