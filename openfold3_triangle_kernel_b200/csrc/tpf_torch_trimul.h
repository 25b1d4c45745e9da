// TriMul helpers shared by the operator (tpf_torch_trimul.cpp) and the pair block (tpf_torch_block.cpp).
#pragma once

#include "tpf_internal.h"
#include "tpf_torch.h"

namespace tpf_torch {

int mask_type(const Tensor& t);  // -1: not a mask type
Tensor trimul_bind(tpf::TrimulCall& t, const Tensor& z, const Tensor& mask, const std::vector<Tensor>& w, bool incoming,
                   bool keep, const Tensor& arena_in);
void trimul_grad_bind(tpf::TrimulGrads& g, std::vector<Tensor>& out, const Tensor& like, int64_t C);
Tensor flat_pair_mask(const Tensor& mask, const Tensor& z, int64_t B);
Tensor aligned_bf16(const Tensor& t);
bool trimul_supported(const Tensor& z, const Tensor& mask, const std::vector<Tensor>& w);

}  // namespace tpf_torch
