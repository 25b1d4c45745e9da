// Python module `_native`: the eager route of the public operators.
#include "tpf_torch.h"

#include <c10/core/impl/LocalDispatchKeySet.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>

#include <atomic>

namespace tpf_torch {

bool plain_cuda(const Tensor& t) {
  using c10::DispatchKey;
  static const c10::DispatchKeySet special({DispatchKey::Python, DispatchKey::PythonTLSSnapshot,
                                            DispatchKey::FuncTorchBatched, DispatchKey::FuncTorchGradWrapper,
                                            DispatchKey::Functionalize, DispatchKey::Conjugate, DispatchKey::Negative,
                                            DispatchKey::ZeroTensor});
  return t.is_cuda() && t.layout() == at::kStrided && !t.key_set().has_any(special);
}

// Parameter carries torch's marker for "no __torch_function__", and a subclass inherits it unless it defines one.
bool plain_type(py::handle h) {
  if (THPVariable_CheckExact(h.ptr())) return true;
  if (!THPVariable_Check(h.ptr())) return false;
  return py::getattr(py::type::handle_of(h), "__torch_function__", py::none())
      .is(py::module_::import("torch._C").attr("_disabled_torch_function_impl"));
}

bool plain_context() {
  using c10::DispatchKey;
  static const c10::DispatchKeySet special({DispatchKey::Python, DispatchKey::FuncTorchDynamicLayerFrontMode,
                                            DispatchKey::FuncTorchDynamicLayerBackMode, DispatchKey::Functionalize,
                                            DispatchKey::Tracer});  // (torch.jit.trace)
  return !c10::impl::tls_local_dispatch_key_set().included_.has_any(special);
}

bool device_supported(const Tensor& t) {
  static std::atomic<int> table[64];  // 0: unknown, 1: no, 2: yes
  const int dev = t.device().index();
  if (dev < 0 || dev >= 64) return false;
  int v = table[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    v = at::cuda::getDeviceProperties(dev)->major == 10 ? 2 : 1;
    table[dev].store(v, std::memory_order_relaxed);
  }
  return v == 2;
}

// The raising node leads to everything the gradients depend on: the operator's inputs (the edges of the node that is
// running) and the incoming gradients.  Without those edges a second pass that asks for certain inputs only
// (autograd.grad) would prune it and leave the term out.
variable_list first_order(const variable_list& incoming, variable_list grads) {
  namespace ag = torch::autograd;
  if (!at::GradMode::is_enabled()) return grads;
  ag::edge_list edges = ag::get_current_node()->next_edges();
  for (const Tensor& t : incoming)
    if (t.defined()) edges.push_back(ag::impl::gradient_edge(t));
  auto node = std::make_shared<ag::Error>(
      "the triangle operators are differentiable once: there is no second derivative (create_graph=True)",
      std::move(edges));
  for (Tensor& g : grads) {
    if (!g.defined()) continue;
    g = g.variable_data();
    ag::set_history(g, node);
  }
  return grads;
}

}  // namespace tpf_torch

PYBIND11_MODULE(_native, m) {
  m.def("attention", &tpf_torch::py_attention);
  m.def("attn_fwd", &tpf_torch::attn_fwd);
  m.def("attn_bwd", &tpf_torch::attn_bwd);
  m.def("trimul", &tpf_torch::py_trimul);
  m.def("trimul_fwd", &tpf_torch::trimul_fwd);
  m.def("pair_block", &tpf_torch::py_pair_block);
  m.def("trimul_bwd", &tpf_torch::trimul_bwd);
}
