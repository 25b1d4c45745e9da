// Python module `_native`: the eager route of the public operators.
#include "tpf_torch.h"

#include <c10/core/impl/LocalDispatchKeySet.h>

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

bool plain_context() {
  using c10::DispatchKey;
  static const c10::DispatchKeySet special({DispatchKey::Python, DispatchKey::FuncTorchDynamicLayerFrontMode,
                                            DispatchKey::FuncTorchDynamicLayerBackMode, DispatchKey::Functionalize});
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
