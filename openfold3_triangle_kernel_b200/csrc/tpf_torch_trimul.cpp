// turbo_trimul for eager CUDA tensors: contract check, launch and autograd node.
#include "tpf_internal.h"
#include "tpf_torch.h"
#include "tpf_torch_trimul.h"

namespace tpf_torch {

int mask_type(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return 0;
    case at::kBFloat16: return 1;
    case at::kHalf: return 2;
    case at::kBool: return 3;
    default: return -1;
  }
}

// Sets the fields that follow from the shapes, and the intermediates' addresses inside one arena.  `keep`: every
// intermediate is kept for the backward; otherwise tensors whose lives do not overlap share memory.
Tensor trimul_bind(tpf::TrimulCall& t, const Tensor& z, const Tensor& mask, const std::vector<Tensor>& w, bool incoming,
                   bool keep, const Tensor& arena_in) {
  const int64_t nd = z.dim(), N = z.size(-2), C = z.size(-1);
  t.B = 1;
  for (int64_t i = 0; i < nd - 3; ++i) t.B *= z.size(i);
  t.N = N;
  t.Np = (N + 7) / 8 * 8;
  t.C = C;
  t.incoming = incoming ? 1 : 0;
  t.z = z.data_ptr();
  const float* ws[8];
  for (int i = 0; i < 8; ++i) ws[i] = fptr(w[i]);
  t.w = {ws[0], ws[1], ws[2], ws[3], ws[4], ws[5], ws[6], ws[7]};
  bool own_mask = true;
  if (mask.defined()) {
    t.mask = mask.data_ptr();
    t.mask_type = mask_type(mask);
    for (int i = 0; i < 3; ++i) t.mask_stride[i] = mask.stride(i);
    own_mask = !(t.mask_type == 0 && t.Np == N && mask.is_contiguous());
  }
  const int64_t R = t.B * t.Np * t.Np;
  Arena a;
  const int64_t packed = a.take(tpf::trimul_fwd_workspace_bytes(t.B, t.Np, C));
  if (!keep && tpf::trimul_fused(C)) {
    const int64_t x[3] = {a.take(R * C * 2), a.take(R * C * 2), a.take(R * C * 2)}, stats = a.take(2 * R * 4);
    Tensor arena = arena_in.defined() ? arena_in : empty_bytes(a.off, z);
    char* base = static_cast<char*>(arena.data_ptr());
    t.packed = base + packed;
    t.infer = true;
    t.a_cm = base + x[0];
    t.b_cm = base + x[1];
    t.x_cm = base + x[2];
    t.z_stats = reinterpret_cast<float*>(base + stats);
    return arena;
  }
  const int64_t zln = a.take(R * C * 2), acm = a.take(R * C * 2), bcm = a.take(R * C * 2), gate = a.take(R * C * 2);
  const int64_t xcm = keep ? a.take(R * C * 2) : zln;  // zln is dead once a, b and the gate exist,
  const int64_t xln = keep ? a.take(R * C * 2) : acm;  // a once x exists
  const int64_t stats = keep ? a.take(4 * R * 4) : 0;
  const int64_t mgrid = own_mask ? a.take(R * 4) : 0;
  Tensor arena = arena_in.defined() ? arena_in : empty_bytes(a.off, z);
  char* base = static_cast<char*>(arena.data_ptr());
  t.packed = base + packed;
  t.zln = base + zln;
  t.a_cm = base + acm;
  t.b_cm = base + bcm;
  t.gate = base + gate;
  t.x_cm = base + xcm;
  t.xln = base + xln;
  if (keep) {
    float* s = reinterpret_cast<float*>(base + stats);
    t.mean_in = s;
    t.rstd_in = s + R;
    t.mean_out = s + 2 * R;
    t.rstd_out = s + 3 * R;
  }
  if (own_mask) t.mask_grid = reinterpret_cast<float*>(base + mgrid);
  return arena;
}

// Gradient buffers of the eight parameters in one allocation each kind; `order` of the operator's weight list.
void trimul_grad_bind(tpf::TrimulGrads& g, std::vector<Tensor>& out, const Tensor& like, int64_t C) {
  const int64_t rows[4] = {2 * C, 2 * C, C, C};
  for (int i = 0; i < 4; ++i) out.push_back(empty_f32({rows[i], C}, like));
  for (int i = 0; i < 4; ++i) out.push_back(empty_f32({C}, like));
  g.p_in = fptr(out[0]);
  g.g_in = fptr(out[1]);
  g.p_out = fptr(out[2]);
  g.g_out = fptr(out[3]);
  g.norm_in_w = fptr(out[4]);
  g.norm_in_b = fptr(out[5]);
  g.norm_out_w = fptr(out[6]);
  g.norm_out_b = fptr(out[7]);
}

Tensor flat_pair_mask(const Tensor& mask, const Tensor& z, int64_t B) {
  if (!mask.defined()) return mask;
  const auto lead = z.sizes().slice(0, z.dim() - 1);
  if (z.dim() == 4 && mask.sizes() == lead) return mask.detach();
  return mask.detach().expand(lead).reshape({B, z.size(-2), z.size(-2)});
}

Tensor aligned_bf16(const Tensor& t) {
  Tensor c = t.scalar_type() == at::kBFloat16 ? t.contiguous() : t.to(at::kBFloat16).contiguous();
  return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15) ? c.clone() : c;
}

namespace {

cudaStream_t cu_stream() { return static_cast<cudaStream_t>(stream()); }

// inputs: z, mask (an absent one is an empty optional: the node cannot take an undefined tensor as an input), then p_in,
// g_in, p_out, g_out, norm_in_w, norm_in_b, norm_out_w, norm_out_b
struct TrimulFn : public torch::autograd::Function<TrimulFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& z_in, const std::optional<Tensor>& mask_in, const Tensor& w0,
                        const Tensor& w1, const Tensor& w2, const Tensor& w3, const Tensor& w4, const Tensor& w5,
                        const Tensor& w6, const Tensor& w7, bool incoming, bool save) {
    const Tensor z = aligned_bf16(z_in.detach());
    std::vector<Tensor> w;
    for (const Tensor* t : {&w0, &w1, &w2, &w3, &w4, &w5, &w6, &w7}) w.push_back(f32c(*t));
    const Tensor mask = flat_pair_mask(mask_in.value_or(Tensor()), z, z.numel() / (z.size(-1) * z.size(-2) * z.size(-2)));
    tpf::TrimulCall t = {};
    Tensor arena = trimul_bind(t, z, mask, w, incoming, save, Tensor());
    Tensor out = empty_bf16(z.sizes(), z);
    t.out = out.data_ptr();
    check(tpf::trimul_forward(t, cu_stream()), "tpf_trimul_fwd");
    if (save) {
      // of the weights only the two norm weights are read again: the matrices live on as packed bf16 copies
      ctx->save_for_backward({z, mask, arena, out, w[4], w[6]});
      std::vector<int64_t> m{incoming ? 1 : 0};
      for (const Tensor* x : {&w0, &w1, &w2, &w3, &w4, &w5, &w6, &w7}) m.push_back((int64_t)x->scalar_type());
      ctx->saved_data["m"] = std::move(m);
    }
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return first_order(grads, gradients(ctx, grads));
  }

  static variable_list gradients(AutogradContext* ctx, const variable_list& grads) {
    variable_list r(12);
    if (!grads[0].defined()) return r;
    const auto saved = ctx->get_saved_variables();
    const Tensor& z = saved[0];
    const auto m = ctx->saved_data["m"].toIntVector();
    c10::cuda::CUDAGuard guard(z.device());
    at::NoGradGuard no_grad;
    const Tensor d_out = aligned_bf16(grads[0]);
    std::vector<Tensor> w(8);
    w[4] = saved[4];
    w[6] = saved[5];
    tpf::TrimulCall t = {};
    trimul_bind(t, z, saved[1], w, m[0] != 0, true, saved[2]);
    t.out = saved[3].data_ptr();
    tpf::TrimulGrads g = {};
    std::vector<Tensor> gw;
    trimul_grad_bind(g, gw, z, t.C);
    Tensor d_z = empty_bf16(z.sizes(), z);
    g.d_out = d_out.data_ptr();
    g.d_z = d_z.data_ptr();
    const int64_t ws_bytes = tpf::trimul_bwd_workspace_bytes(t.B, t.Np * t.Np, t.C);
    Tensor ws = empty_bytes(ws_bytes, z);
    check(tpf::trimul_backward(t, g, ws.data_ptr(), ws_bytes, cu_stream()), "tpf_trimul_bwd");
    r[0] = d_z;
    for (int i = 0; i < 8; ++i) {
      const auto type = (at::ScalarType)m[1 + i];
      r[2 + i] = gw[i].scalar_type() == type ? gw[i] : gw[i].to(type);
    }
    return r;
  }
};

}  // namespace

bool trimul_supported(const Tensor& z, const Tensor& mask, const std::vector<Tensor>& w) {
  if (!plain_cuda(z) || !device_supported(z) || z.dim() < 4 || z.scalar_type() != at::kBFloat16 || z.numel() == 0)
    return false;
  const int64_t N = z.size(-2), C = z.size(-1);
  if (z.size(-3) != N || (C != 32 && C != 64 && C != 96 && C != 128)) return false;
  if (mask.defined()) {
    if (!plain_cuda(mask) || mask.device() != z.device() || mask_type(mask) < 0 || mask.requires_grad() ||
        mask.dim() > z.dim() - 1)
      return false;
    for (int64_t i = 0; i < mask.dim(); ++i) {
      const int64_t a = mask.size(mask.dim() - 1 - i), b = z.size(z.dim() - 2 - i);
      if (a != b && a != 1) return false;
    }
  }
  const int64_t rows[4] = {2 * C, 2 * C, C, C};
  for (int i = 0; i < 8; ++i) {
    if (!plain_cuda(w[i]) || w[i].device() != z.device() || !w[i].is_floating_point()) return false;
    if (i < 4 ? (w[i].dim() != 2 || w[i].size(0) != rows[i] || w[i].size(1) != C) : (w[i].dim() != 1 || w[i].size(0) != C))
      return false;
  }
  return true;
}

// The eager call.  Returns None when the arguments need the Python route (see py_attention).
py::object py_trimul(py::handle hz, bool incoming, py::handle hm, py::tuple weights) {
  if (!plain_type(hz) || weights.size() != 8) return py::none();
  const Tensor& z = THPVariable_Unpack(hz.ptr());
  Tensor mask;
  if (!hm.is_none()) {
    if (!plain_type(hm)) return py::none();
    mask = THPVariable_Unpack(hm.ptr());
  }
  std::vector<Tensor> w;
  bool grad = z.requires_grad();
  for (int i = 0; i < 8; ++i) {
    py::handle h = weights[i];
    if (!plain_type(h)) return py::none();
    w.push_back(THPVariable_Unpack(h.ptr()));
    grad = grad || w.back().requires_grad();
  }
  if (!plain_context() || !trimul_supported(z, mask, w)) return py::none();
  const bool save = grad && at::GradMode::is_enabled();
  const std::optional<Tensor> opt_mask = mask.defined() ? std::optional<Tensor>(mask) : std::nullopt;
  Tensor out;
  {
    py::gil_scoped_release release;
    c10::cuda::CUDAGuard guard(z.device());
    if (save) {
      out = TrimulFn::apply(z, opt_mask, w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], incoming, true);
    } else {
      at::NoGradGuard no_grad;
      out = TrimulFn::forward(nullptr, z, opt_mask, w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], incoming, false);
    }
  }
  return py::cast(out);
}

// Launches behind the torch.library operators: z [B,N,N,C] with N a multiple of 8, mask fp32 [B,N,N].
std::vector<Tensor> trimul_fwd(const Tensor& z_, const Tensor& mask_, std::vector<Tensor> w_, bool incoming) {
  c10::cuda::CUDAGuard guard(z_.device());
  const Tensor z = aligned_bf16(z_), mask = mask_.to(at::kFloat).contiguous();
  const int64_t B = z.size(0), N = z.size(1), C = z.size(3), R = B * N * N;
  std::vector<Tensor> w;
  for (const Tensor& t : w_) w.push_back(f32c(t));
  std::vector<Tensor> o{empty_bf16({B, N, N, C}, z)};                       // out
  auto bf = [&](at::IntArrayRef s) { o.push_back(empty_bf16(s, z)); };
  auto f = [&]() { o.push_back(empty_f32({R}, z)); };
  bf({R, C}); f(); f();                                                     // zln, mean_in, rstd_in
  bf({B * C, N * N}); bf({B * C, N * N}); bf({R, C}); bf({B * C, N * N});   // a_cm, b_cm, gate, x_cm
  bf({R, C}); f(); f();                                                     // xln, mean_out, rstd_out
  const int64_t nbytes = tpf_trimul_fwd_workspace_bytes(B, N, C);
  Tensor ws = empty_bytes(nbytes, z);
  check(tpf_trimul_fwd(z.data_ptr(), fptr(mask), fptr(w[0]), fptr(w[1]), fptr(w[2]), fptr(w[3]), fptr(w[4]), fptr(w[5]),
                       fptr(w[6]), fptr(w[7]), incoming ? 1 : 0, B, N, C, o[0].data_ptr(), o[1].data_ptr(), fptr(o[2]),
                       fptr(o[3]), o[4].data_ptr(), o[5].data_ptr(), o[6].data_ptr(), o[7].data_ptr(), o[8].data_ptr(),
                       fptr(o[9]), fptr(o[10]), ws.data_ptr(), nbytes, stream()),
        "tpf_trimul_fwd");
  return o;
}

// w: p_in, g_in, p_out, g_out, norm_in_w, norm_out_w.  Returns d_z and the eight parameter gradients.
std::vector<Tensor> trimul_bwd(const Tensor& d_out_, const Tensor& z_, const Tensor& mask_, std::vector<Tensor> w_,
                               bool incoming, std::vector<Tensor> s) {
  c10::cuda::CUDAGuard guard(z_.device());
  const Tensor z = aligned_bf16(z_), mask = mask_.to(at::kFloat).contiguous(), d_out = aligned_bf16(d_out_);
  const int64_t B = z.size(0), N = z.size(1), C = z.size(3);
  std::vector<Tensor> w;
  for (const Tensor& t : w_) w.push_back(f32c(t));
  std::vector<Tensor> gw;
  tpf::TrimulGrads g = {};
  trimul_grad_bind(g, gw, z, C);
  Tensor d_z = empty_bf16(z.sizes(), z);
  const int64_t nbytes = tpf_trimul_bwd_workspace_bytes(B, N, C);
  Tensor ws = empty_bytes(nbytes, z);
  check(tpf_trimul_bwd(d_out.data_ptr(), z.data_ptr(), fptr(mask), fptr(w[0]), fptr(w[1]), fptr(w[2]), fptr(w[3]),
                       fptr(w[4]), fptr(w[5]), incoming ? 1 : 0, B, N, C, s[0].data_ptr(), s[1].data_ptr(), fptr(s[2]),
                       fptr(s[3]), s[4].data_ptr(), s[5].data_ptr(), s[6].data_ptr(), s[7].data_ptr(), s[8].data_ptr(),
                       fptr(s[9]), fptr(s[10]), d_z.data_ptr(), g.p_in, g.g_in, g.p_out, g.g_out, g.norm_in_w,
                       g.norm_in_b, g.norm_out_w, g.norm_out_b, ws.data_ptr(), nbytes, stream()),
        "tpf_trimul_bwd");
  std::vector<Tensor> r{d_z};
  for (Tensor& t : gw) r.push_back(t);
  return r;
}

}  // namespace tpf_torch
