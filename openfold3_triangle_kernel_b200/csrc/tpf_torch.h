// Shared pieces of the native torch layer (tpf_torch*.cpp): the Python module `_native` that carries the eager
// calls of the public operators, their autograd nodes included, without going through Python-level dispatch.
#pragma once

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "../../include/tpf_b200.h"

namespace tpf_torch {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

inline void check(int rc, const char* who) {
  if (rc == TPF_OK) return;
  if (rc == TPF_ERR_INVALID_ARGUMENT || rc == TPF_ERR_UNSUPPORTED)
    TORCH_CHECK_VALUE(false, who, ": ", tpf_last_error_string());
  TORCH_CHECK(false, who, " failed: ", tpf_last_error_string());
}

inline void* stream() { return at::cuda::getCurrentCUDAStream().stream(); }

inline Tensor empty_bf16(at::IntArrayRef s, const Tensor& like) { return at::empty(s, like.options().dtype(at::kBFloat16)); }
inline Tensor empty_f32(at::IntArrayRef s, const Tensor& like) { return at::empty(s, like.options().dtype(at::kFloat)); }
inline Tensor empty_bytes(int64_t n, const Tensor& like) {
  return at::empty({n < 256 ? 256 : n}, like.options().dtype(at::kByte));
}
inline float* fptr(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }

// An fp32 contiguous view or copy of a parameter.
inline Tensor f32c(const Tensor& t) {
  if (t.scalar_type() == at::kFloat && t.is_contiguous()) return t;
  return t.detach().to(at::kFloat).contiguous();
}

// A plain eager CUDA tensor: no functorch wrapper, no lazy conjugation or negation, no subclass that dispatches.  Anything
// else (and any active dispatch mode) takes the torch.library route, which every such mechanism sees.
bool plain_cuda(const Tensor& t);
// ... and no subclass whose __torch_function__ wants to see the call, which the Python object tells: tensors, parameters and
// subclasses of Parameter without one of their own pass.
bool plain_type(py::handle h);
bool plain_context();

// Compute capability 10.x, cached per device.
bool device_supported(const Tensor& t);

// Last step of every backward.  The gradients have no derivative of their own; when the engine records them
// (create_graph=True) they get a node that raises if one is asked for, instead of counting as constants.
variable_list first_order(const variable_list& incoming, variable_list grads);

// Hands out 256-byte aligned pieces of one allocation: an operator call keeps a dozen intermediate tensors, and one
// allocation is cheaper on the host than twelve.
struct Arena {
  int64_t off = 0;
  char* base = nullptr;
  int64_t take(int64_t bytes) {
    const int64_t o = off;
    off += (bytes + 255) / 256 * 256;
    return o;
  }
};

// ---- attention (tpf_torch_attention.cpp) ----------------------------------------------------
py::object py_attention(py::handle q, py::handle k, py::handle v, py::handle bias, py::handle mask, bool return_lse);
std::tuple<Tensor, Tensor> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& mask,
                                    const Tensor& bias, double scale);
std::tuple<Tensor, Tensor, Tensor, Tensor> attn_bwd(const Tensor& q, const Tensor& k, const Tensor& v,
                                                    const Tensor& d_out, const Tensor& out, const Tensor& lse,
                                                    const Tensor& mask, const Tensor& bias, double scale);

// ---- triangle multiplicative update (tpf_torch_trimul.cpp) ----------------------------------
py::object py_trimul(py::handle z, bool incoming, py::handle mask, py::tuple weights);
std::vector<Tensor> trimul_fwd(const Tensor& z, const Tensor& mask, std::vector<Tensor> w, bool incoming);
std::vector<Tensor> trimul_bwd(const Tensor& d_out, const Tensor& z, const Tensor& mask, std::vector<Tensor> w,
                               bool incoming, std::vector<Tensor> saved);

// ---- pair-stack block (tpf_torch_block.cpp) -------------------------------------------------
py::object py_pair_block(py::handle z, py::handle mask, py::tuple tri_out, py::tuple tri_in, py::tuple start,
                         py::tuple end, int64_t heads);

}  // namespace tpf_torch
