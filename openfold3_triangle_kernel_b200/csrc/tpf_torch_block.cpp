// The pair-stack block for eager CUDA tensors: TriMul outgoing, TriMul incoming, attention starting node, attention
// ending node, each with its residual add inside its last kernel.  Four autograd nodes.
#include "tpf_torch_trimul.h"

namespace tpf_torch {

namespace {

cudaStream_t cu_stream() { return static_cast<cudaStream_t>(stream()); }

std::vector<int64_t> scalar_types(at::ArrayRef<Tensor> w) {
  std::vector<int64_t> m;
  for (const Tensor& t : w) m.push_back((int64_t)t.scalar_type());
  return m;
}

Tensor as_type(const Tensor& g, int64_t type) {
  return g.scalar_type() == (at::ScalarType)type ? g : g.to((at::ScalarType)type);
}

// z + TriMul(z).  w: p_in, g_in, p_out, g_out, norm_in_w, norm_in_b, norm_out_w, norm_out_b
struct TrimulResidualFn : public torch::autograd::Function<TrimulResidualFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& z_in, const Tensor& mask, const Tensor& w0,
                        const Tensor& w1, const Tensor& w2, const Tensor& w3, const Tensor& w4, const Tensor& w5,
                        const Tensor& w6, const Tensor& w7, bool incoming, bool save) {
    const Tensor z = aligned_bf16(z_in.detach());
    const Tensor in[8] = {w0, w1, w2, w3, w4, w5, w6, w7};
    std::vector<Tensor> w;
    for (const Tensor& t : in) w.push_back(f32c(t));
    tpf::TrimulCall t = {};
    Tensor arena = trimul_bind(t, z, mask, w, incoming, save, Tensor());
    Tensor sum = empty_bf16(z.sizes(), z), out;
    t.sum = sum.data_ptr();
    if (save) {  // the backward of the output gate reads the update itself
      out = empty_bf16(z.sizes(), z);
      t.out = out.data_ptr();
    }
    check(tpf::trimul_forward(t, cu_stream()), "tpf_trimul_fwd");
    if (save) {
      ctx->save_for_backward({z, mask, arena, out, w[4], w[6]});
      std::vector<int64_t> m = scalar_types(in);
      m.push_back(incoming ? 1 : 0);
      ctx->saved_data["m"] = std::move(m);
    }
    return sum;
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
    std::vector<Tensor> w(8), gw;
    w[4] = saved[4];
    w[6] = saved[5];
    tpf::TrimulCall t = {};
    trimul_bind(t, z, saved[1], w, m[8] != 0, true, saved[2]);
    t.out = saved[3].data_ptr();
    tpf::TrimulGrads g = {};
    trimul_grad_bind(g, gw, z, t.C);
    Tensor d_z = empty_bf16(z.sizes(), z);
    g.d_out = g.d_res = d_out.data_ptr();
    g.d_z = d_z.data_ptr();
    const int64_t n = tpf::trimul_bwd_workspace_bytes(t.B, t.Np * t.Np, t.C);
    Tensor ws = empty_bytes(n, z);
    check(tpf::trimul_backward(t, g, ws.data_ptr(), n, cu_stream()), "tpf_trimul_bwd");
    r[0] = d_z;
    for (int i = 0; i < 8; ++i) r[2 + i] = as_type(gw[i], m[i]);
    return r;
  }
};

constexpr double kInf = 1e9;

Tensor attn_bind(tpf::PairAttnCall& t, const Tensor& z, const Tensor& mask, const std::vector<Tensor>& w, int64_t heads,
                 int64_t d, bool ending, bool keep, const Tensor& arena_in) {
  t.B = z.size(0);
  t.N = z.size(1);
  t.C = z.size(3);
  t.H = heads;
  t.D = d;
  t.ending = ending ? 1 : 0;
  t.z = z.data_ptr();
  t.mask = mask.data_ptr();
  t.mask_type = mask_type(mask);
  for (int i = 0; i < 3; ++i) t.mask_stride[i] = mask.stride(i);
  t.inf = (float)kInf;
  t.w = {fptr(w[0]), fptr(w[1]), fptr(w[2]), fptr(w[3]), fptr(w[4]), fptr(w[5]), fptr(w[6]), fptr(w[7])};
  const int64_t R = t.B * t.N * t.N, HD = heads * d;
  Arena a;
  const int64_t packed = a.take(tpf::pair_attn_packed_bytes(t.C, heads, d));
  const int64_t x = a.take(R * t.C * 2), qkvg = a.take(4 * R * HD * 2);
  const int64_t og = keep || HD > t.C ? a.take(R * HD * 2) : x;  // x is dead once it is projected
  const int64_t bias = a.take(t.B * heads * t.N * ((t.N + 7) / 8 * 8) * 2);
  const int64_t madd = a.take(t.B * t.N * ((t.N + 3) / 4 * 4) * 4);
  const int64_t stats = keep ? a.take((2 * R + R * heads) * 4) : 0;
  Tensor arena = arena_in.defined() ? arena_in : empty_bytes(a.off, z);
  char* base = static_cast<char*>(arena.data_ptr());
  t.packed = base + packed;
  t.x = base + x;
  t.qkvg = base + qkvg;
  t.og = base + og;
  t.bias = base + bias;
  t.mask_add = reinterpret_cast<float*>(base + madd);
  if (keep) {
    t.mean = reinterpret_cast<float*>(base + stats);
    t.rstd = t.mean + R;
    t.lse = t.mean + 2 * R;
  }
  return arena;
}

// z + attention update.  w: ln_w, ln_b, w_z, w_q, w_k, w_v, w_g, w_o
struct PairAttnFn : public torch::autograd::Function<PairAttnFn> {
  static Tensor forward(AutogradContext* ctx, const Tensor& z_in, const Tensor& mask, const Tensor& w0,
                        const Tensor& w1, const Tensor& w2, const Tensor& w3, const Tensor& w4, const Tensor& w5,
                        const Tensor& w6, const Tensor& w7, int64_t heads, bool ending, bool save) {
    const Tensor z = aligned_bf16(z_in.detach());
    const Tensor in[8] = {w0, w1, w2, w3, w4, w5, w6, w7};
    std::vector<Tensor> w;
    for (const Tensor& t : in) w.push_back(f32c(t));
    const int64_t d = w[3].size(0) / heads;
    tpf::PairAttnCall t = {};
    Tensor arena = attn_bind(t, z, mask, w, heads, d, ending, save, Tensor());
    Tensor out = empty_bf16(z.sizes(), z);
    t.out = out.data_ptr();
    check(tpf::pair_attn_forward(t, cu_stream()), "pair attention forward");
    if (save) {
      ctx->save_for_backward({z, mask, arena, w[0]});
      std::vector<int64_t> m = scalar_types(in);
      for (int64_t x : {heads, d, (int64_t)ending}) m.push_back(x);
      ctx->saved_data["m"] = std::move(m);
    }
    return out;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return first_order(grads, gradients(ctx, grads));
  }

  static variable_list gradients(AutogradContext* ctx, const variable_list& grads) {
    variable_list r(13);
    if (!grads[0].defined()) return r;
    const auto saved = ctx->get_saved_variables();
    const Tensor& z = saved[0];
    const auto m = ctx->saved_data["m"].toIntVector();
    c10::cuda::CUDAGuard guard(z.device());
    at::NoGradGuard no_grad;
    const Tensor d_out = aligned_bf16(grads[0]);
    std::vector<Tensor> w(8);
    w[0] = saved[3];
    const int64_t H = m[8], D = m[9], HD = H * D, C = z.size(3);
    tpf::PairAttnCall t = {};
    attn_bind(t, z, saved[1], w, H, D, m[10] != 0, true, saved[2]);
    Tensor d_z = empty_bf16(z.sizes(), z);
    const Tensor gw[8] = {empty_f32({C}, z),     empty_f32({C}, z),     empty_f32({H, C}, z),  empty_f32({HD, C}, z),
                          empty_f32({HD, C}, z), empty_f32({HD, C}, z), empty_f32({HD, C}, z), empty_f32({C, HD}, z)};
    const tpf::PairAttnGrads g{d_out.data_ptr(), d_z.data_ptr(), fptr(gw[0]), fptr(gw[1]), fptr(gw[2]),
                               fptr(gw[3]),      fptr(gw[4]),    fptr(gw[5]), fptr(gw[6]), fptr(gw[7])};
    const int64_t n = tpf::pair_attn_bwd_workspace_bytes(t.B, t.N, C, H, D);
    Tensor ws = empty_bytes(n, z);
    check(tpf::pair_attn_backward(t, g, ws.data_ptr(), n, cu_stream()), "pair attention backward");
    r[0] = d_z;
    for (int i = 0; i < 8; ++i) r[2 + i] = as_type(gw[i], m[i]);
    return r;
  }
};

bool attn_weights_ok(const std::vector<Tensor>& w, const Tensor& z, int64_t heads) {
  const int64_t C = z.size(3);
  for (const Tensor& t : w)
    if (!plain_cuda(t) || t.device() != z.device() || !t.is_floating_point()) return false;
  for (int i = 0; i < 2; ++i)
    if (w[i].dim() != 1 || w[i].size(0) != C) return false;
  for (int i = 2; i < 8; ++i)
    if (w[i].dim() != 2) return false;
  const int64_t HD = w[3].size(0);
  if (heads <= 0 || HD % heads || w[2].size(0) != heads || w[2].size(1) != C) return false;
  for (int i = 3; i < 7; ++i)
    if (w[i].size(0) != HD || w[i].size(1) != C) return false;
  return w[7].size(0) == C && w[7].size(1) == HD && tpf::pair_attn_supported(C, heads, HD / heads);
}

bool unpack(const py::tuple& p, std::vector<Tensor>& w, bool& grad) {
  if (p.size() != 8) return false;
  for (py::handle h : p) {
    if (!plain_type(h)) return false;
    w.push_back(THPVariable_Unpack(h.ptr()));
    grad = grad || w.back().requires_grad();
  }
  return true;
}

}  // namespace

// The eager call.  `tri_out`, `tri_in`: weights in the order of py_trimul; `start`, `end`: ln_w, ln_b, w_z, w_q, w_k,
// w_v, w_g, w_o.  Returns None when the arguments need the Python route.
py::object py_pair_block(py::handle hz, py::handle hm, py::tuple tri_out, py::tuple tri_in, py::tuple start,
                         py::tuple end, int64_t heads) {
  if (!plain_type(hz) || !plain_type(hm)) return py::none();
  const Tensor &z = THPVariable_Unpack(hz.ptr()), &mask = THPVariable_Unpack(hm.ptr());
  std::vector<Tensor> w[4];
  bool grad = z.requires_grad();
  const py::tuple* parts[4] = {&tri_out, &tri_in, &start, &end};
  for (int i = 0; i < 4; ++i)
    if (!unpack(*parts[i], w[i], grad)) return py::none();
  if (z.dim() != 4 || mask.dim() != 3 || !plain_context() || !trimul_supported(z, mask, w[0]) ||
      !trimul_supported(z, mask, w[1]) || mask.sizes() != z.sizes().slice(0, 3) || !attn_weights_ok(w[2], z, heads) ||
      !attn_weights_ok(w[3], z, heads))
    return py::none();
  const bool save = grad && at::GradMode::is_enabled();
  Tensor x = z;
  {
    py::gil_scoped_release release;
    c10::cuda::CUDAGuard guard(z.device());
    if (save) {
      for (int i = 0; i < 2; ++i) {
        const auto& v = w[i];
        x = TrimulResidualFn::apply(x, mask, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], i == 1, true);
      }
      for (int i = 2; i < 4; ++i) {
        const auto& v = w[i];
        x = PairAttnFn::apply(x, mask, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], heads, i == 3, true);
      }
    } else {
      at::NoGradGuard no_grad;
      for (int i = 0; i < 2; ++i) {
        const auto& v = w[i];
        x = TrimulResidualFn::forward(nullptr, x, mask, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], i == 1, false);
      }
      for (int i = 2; i < 4; ++i) {
        const auto& v = w[i];
        x = PairAttnFn::forward(nullptr, x, mask, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], heads, i == 3, false);
      }
    }
  }
  return py::cast(x);
}

}  // namespace tpf_torch
