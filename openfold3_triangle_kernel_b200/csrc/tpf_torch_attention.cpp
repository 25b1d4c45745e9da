// turbo_attention for eager CUDA tensors: contract check, operand preparation, launch and autograd node.
#include <cmath>

#include "tpf_internal.h"
#include "tpf_torch.h"

namespace tpf_torch {

namespace {

struct Shape {
  int64_t B, O, H, N, D, G;  // D: lane width of the kernels; G: bias batch (1 or B)
};

// A tensor the TMA descriptors can read in place: last dim contiguous, base and strides multiples of 16 bytes.
Tensor kernel_layout(const Tensor& t) {
  const auto st = t.strides();
  const int64_t nd = t.dim();
  bool ok = st[nd - 1] == 1 && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
  for (int64_t i = 0; ok && i < nd - 1; ++i) ok = (st[i] * 2) % 16 == 0;
  return ok ? t : t.contiguous();
}

int prep_type(const Tensor& t) {
  return t.scalar_type() == at::kFloat ? tpf::kPrepF32 : t.scalar_type() == at::kBFloat16 ? tpf::kPrepBF16 : tpf::kPrepF16;
}

struct Operands {
  Tensor mask, bias;  // fp32 [B,O,mp], bf16 [G,H,N,bp]
  int64_t mp, bp;
};

// mask [B,O,N] (any float type and strides), bias [G,H,N,N] -> kernel layout, in place where they have it already.
Operands prepare(const Tensor& mask, const Tensor& bias, const Shape& s) {
  Operands o{mask, bias, (s.N + 3) / 4 * 4, (s.N + 7) / 8 * 8};
  tpf::PrepSource ps_bias{nullptr, 0, {0, 0, 0, 0}}, ps_mask{nullptr, 0, {0, 0, 0, 0}};
  const bool mask_ok = mask.scalar_type() == at::kFloat && o.mp == s.N && mask.is_contiguous() &&
                       (reinterpret_cast<uintptr_t>(mask.data_ptr()) & 15) == 0;
  const bool bias_ok = bias.scalar_type() == at::kBFloat16 && o.bp == s.N && bias.is_contiguous() &&
                       (reinterpret_cast<uintptr_t>(bias.data_ptr()) & 15) == 0;
  if (!mask_ok) {
    o.mask = empty_f32({s.B, s.O, o.mp}, mask);
    ps_mask.src = mask.data_ptr();
    ps_mask.type = prep_type(mask);
    for (int i = 0; i < 3; ++i) ps_mask.stride[i] = mask.stride(i);
  }
  if (!bias_ok) {
    o.bias = empty_bf16({s.G, s.H, s.N, o.bp}, bias);
    ps_bias.src = bias.data_ptr();
    ps_bias.type = prep_type(bias);
    for (int i = 0; i < 4; ++i) ps_bias.stride[i] = bias.stride(i);
  }
  if (!mask_ok || !bias_ok)
    check(tpf::attn_prep(ps_bias, s.G, s.H, bias_ok ? nullptr : o.bias.data_ptr(), o.bp, ps_mask, s.B, s.O,
                         mask_ok ? nullptr : fptr(o.mask), o.mp, s.N, static_cast<cudaStream_t>(stream())),
          "attn_prep");
  return o;
}

void launch_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Operands& op, const Shape& s, double scale,
                const Tensor& out, const Tensor& lse) {
  check(tpf_attn_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), q.strides().data(), k.strides().data(),
                     v.strides().data(), fptr(op.mask), op.mp, op.bias.data_ptr(), op.bp, s.G, out.data_ptr(),
                     fptr(lse), s.B, s.O, s.H, s.N, s.D, (float)scale, stream()),
        "tpf_attn_fwd");
}

struct Grads {
  Tensor dq, dk, dv, dbias;
};

Grads launch_bwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& d_out, const Tensor& out,
                 const Tensor& lse, const Operands& op, const Shape& s, double scale, int stages) {
  Grads g;
  if (stages & TPF_ATTN_BWD_STAGE_DQKV)
    for (Tensor* t : {&g.dq, &g.dk, &g.dv}) *t = empty_bf16({s.B, s.O, s.H, s.N, s.D}, q);
  if (stages & TPF_ATTN_BWD_STAGE_DBIAS) g.dbias = empty_f32({s.G, s.H, s.N, s.N}, q);
  const int64_t ws_bytes = tpf_attn_bwd_workspace_bytes(s.B, s.O, s.H, s.N, s.D, s.G);
  Tensor ws = empty_bytes(ws_bytes + s.B * s.O * s.H * s.N * 4 + 512, q);  // kernel scratch, then delta
  char* base = static_cast<char*>(ws.data_ptr());
  float* delta = reinterpret_cast<float*>(base + (ws_bytes + 255) / 256 * 256);
  auto p = [](const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; };
  check(tpf_attn_bwd_stages(q.data_ptr(), k.data_ptr(), v.data_ptr(), d_out.data_ptr(), q.strides().data(),
                            k.strides().data(), v.strides().data(), out.data_ptr(), fptr(lse), fptr(op.mask), op.mp,
                            op.bias.data_ptr(), op.bp, s.G, p(g.dq), p(g.dk), p(g.dv), fptr(g.dbias), delta, base,
                            ws_bytes, s.B, s.O, s.H, s.N, s.D, (float)scale, stages, stream()),
        "tpf_attn_bwd");
  return g;
}

Tensor pad_lane(const Tensor& t, int64_t lane) {
  return t.size(-1) == lane ? t : at::constant_pad_nd(t, {0, lane - t.size(-1)});
}

// The autograd node of the eager call.  It takes the caller's tensors in the caller's shapes, so that no view nodes
// surround it.  An absent mask is an empty optional: the node cannot take an undefined tensor as an input.
struct AttentionFn : public torch::autograd::Function<AttentionFn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in,
                               const Tensor& bias_in, const std::optional<Tensor>& mask_in, bool save) {
    const auto qs = q_in.sizes();
    const int64_t nd = q_in.dim(), D = qs[nd - 1], lane = D <= 16 ? 16 : D <= 32 ? 32 : 64;
    Shape s{1, qs[nd - 4], qs[nd - 3], qs[nd - 2], lane, 1};
    for (int64_t i = 0; i < nd - 4; ++i) s.B *= qs[i];
    auto flat = [&](const Tensor& t) {
      Tensor x = pad_lane(t.detach(), lane);
      if (nd != 5) x = x.reshape({s.B, s.O, s.H, s.N, lane});
      return kernel_layout(x);
    };
    const Tensor q = flat(q_in), k = flat(k_in), v = flat(v_in);
    const auto prefix = qs.slice(0, nd - 4);

    auto expanded = [&](const Tensor& t, int64_t group) {  // prefix broadcast to q's, then flattened
      if (t.dim() - 4 == nd - 4 && t.sizes().slice(0, nd - 4) == prefix && nd == 5) return t;
      std::vector<int64_t> full(prefix.begin(), prefix.end());
      for (int64_t i = t.dim() - 4; i < t.dim(); ++i) full.push_back(t.size(i));
      std::vector<int64_t> to{group};
      for (int64_t i = t.dim() - 4; i < t.dim(); ++i) to.push_back(t.size(i));
      return t.expand(full).reshape(to);
    };
    bool shared = true;  // a bias whose whole prefix is 1 is read as one plane set for every batch entry
    for (int64_t i = 0; i < bias_in.dim() - 4; ++i) shared = shared && bias_in.size(i) == 1;
    s.G = shared ? 1 : s.B;
    Tensor bias = bias_in.detach();
    if (shared) bias = bias.dim() == 5 ? bias.select(0, 0) : bias.reshape({1, s.H, s.N, s.N});  // [1,H,N,N]
    else bias = expanded(bias, s.B).select(1, 0);                                              // [B,H,N,N]
    Tensor mask;
    if (mask_in) mask = expanded(mask_in->detach(), s.B).select(3, 0).select(2, 0);   // [B,O,N]
    else mask = at::zeros({s.B, s.O, s.N}, q.options().dtype(at::kFloat));

    const double scale = 1.0 / std::sqrt((double)D);
    const Operands op = prepare(mask, bias, s);
    Tensor out = empty_bf16({s.B, s.O, s.N, s.H, lane}, q), lse = empty_f32({s.B, s.O, s.H, s.N}, q);
    launch_fwd(q, k, v, op, s, scale, out, lse);

    if (save) {
      ctx->save_for_backward({q, k, v, op.mask, op.bias, out, lse});
      ctx->saved_data["s"] = std::vector<int64_t>{s.B, s.O, s.H, s.N, s.D, s.G, D, op.mp, op.bp};
      ctx->saved_data["q"] = qs.vec();
      ctx->saved_data["bias"] = bias_in.sizes().vec();
      ctx->saved_data["type"] = (int64_t)bias_in.scalar_type();
    }
    Tensor o = lane != D ? out.slice(4, 0, D) : out, l = lse;
    if (nd != 5) {
      std::vector<int64_t> os(prefix.begin(), prefix.end()), ls = os;
      for (int64_t x : {s.O, s.N, s.H, D}) os.push_back(x);
      for (int64_t x : {s.O, s.H, s.N}) ls.push_back(x);
      o = o.reshape(os);
      l = lse.reshape(ls);
    }
    // the log-sum-exp is a by-product for callers that ask for it, not a differentiable output
    if (save) ctx->mark_non_differentiable({l});
    return {o, l};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return first_order(grads, gradients(ctx, grads));
  }

  static variable_list gradients(AutogradContext* ctx, const variable_list& grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2], &out = saved[5], &lse = saved[6];
    const auto q_sizes = ctx->saved_data["q"].toIntVector();
    const auto m = ctx->saved_data["s"].toIntVector();
    const Shape s{m[0], m[1], m[2], m[3], m[4], m[5]};
    const int64_t D = m[6];
    c10::cuda::CUDAGuard guard(q.device());
    at::NoGradGuard no_grad;
    Tensor d_out = grads[0].reshape({s.B, s.O, s.N, s.H, D});
    if (d_out.scalar_type() != at::kBFloat16) d_out = d_out.to(at::kBFloat16);
    d_out = pad_lane(d_out, s.D).contiguous();
    if (reinterpret_cast<uintptr_t>(d_out.data_ptr()) & 15) d_out = d_out.clone();
    const bool need_qkv = ctx->needs_input_grad(0) || ctx->needs_input_grad(1) || ctx->needs_input_grad(2);
    const bool need_bias = ctx->needs_input_grad(3);
    const int stages = TPF_ATTN_BWD_STAGE_DELTA | (need_qkv ? TPF_ATTN_BWD_STAGE_DQKV : 0) |
                       (need_bias ? TPF_ATTN_BWD_STAGE_DBIAS : 0);
    Grads g = launch_bwd(q, k, v, d_out, out, lse, Operands{saved[3], saved[4], m[7], m[8]}, s,
                         1.0 / std::sqrt((double)D), stages);
    auto shaped = [&](Tensor t) {
      if (!t.defined()) return t;
      if (s.D != D) t = t.slice(4, 0, D);
      return q_sizes.size() == 5 ? t : t.reshape(q_sizes);
    };
    Tensor db;
    if (need_bias) {
      db = g.dbias;
      const auto bias_sizes = ctx->saved_data["bias"].toIntVector();
      const auto type = (at::ScalarType)ctx->saved_data["type"].toInt();
      if (s.G == 1) {
        db = db.view(bias_sizes);
      } else {
        std::vector<int64_t> full(q_sizes.begin(), q_sizes.end() - 4);
        for (int64_t x : {(int64_t)1, s.H, s.N, s.N}) full.push_back(x);
        db = at::sum_to(db.view(full), bias_sizes);
      }
      if (db.scalar_type() != type) db = db.to(type);
    }
    return {shaped(g.dq), shaped(g.dk), shaped(g.dv), db, Tensor(), Tensor()};
  }
};

bool float_mask(const Tensor& t) {
  return t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf;
}

// Prefix of `t` (all but its last four dimensions) broadcasts to q's prefix without extending it.
bool prefix_ok(const Tensor& t, const Tensor& q) {
  const int64_t pt = t.dim() - 4, pq = q.dim() - 4;
  if (pt > pq) return false;
  for (int64_t i = 0; i < pt; ++i) {
    const int64_t a = t.size(pt - 1 - i), b = q.size(pq - 1 - i);
    if (a != b && a != 1) return false;
  }
  return true;
}

}  // namespace

// The eager call.  Returns None when the arguments need the Python route: an unsupported case (which raises there,
// with its reason), a tensor subclass, an active dispatch mode.
py::object py_attention(py::handle hq, py::handle hk, py::handle hv, py::handle hb, py::handle hm, bool return_lse) {
  for (py::handle h : {hq, hk, hv, hb})
    if (!plain_type(h)) return py::none();
  const Tensor &q = THPVariable_Unpack(hq.ptr()), &k = THPVariable_Unpack(hk.ptr()), &v = THPVariable_Unpack(hv.ptr()),
               &bias = THPVariable_Unpack(hb.ptr());
  std::optional<Tensor> mask;
  if (!hm.is_none()) {
    if (!plain_type(hm)) return py::none();
    mask = THPVariable_Unpack(hm.ptr());
  }
  if (!plain_context() || !plain_cuda(q) || !plain_cuda(k) || !plain_cuda(v) || !plain_cuda(bias) ||
      (mask && !plain_cuda(*mask)) || !device_supported(q))
    return py::none();
  const int64_t nd = q.dim();
  if (nd < 5 || nd > 20 || q.numel() == 0 || q.size(-1) > 64 || bias.dim() < 4) return py::none();
  if (k.sizes() != q.sizes() || v.sizes() != q.sizes()) return py::none();
  for (const Tensor* t : {&q, &k, &v})
    if (t->scalar_type() != at::kBFloat16) return py::none();
  const int64_t O = q.size(-4), H = q.size(-3), N = q.size(-2);
  if (bias.size(-4) != 1 || bias.size(-3) != H || bias.size(-2) != N || bias.size(-1) != N || !prefix_ok(bias, q) ||
      (bias.scalar_type() != at::kBFloat16 && bias.scalar_type() != at::kFloat))
    return py::none();
  if (k.device() != q.device() || v.device() != q.device() || bias.device() != q.device()) return py::none();
  if (mask) {
    if (mask->dim() < 4 || mask->size(-4) != O || mask->size(-3) != 1 || mask->size(-2) != 1 || mask->size(-1) != N ||
        !prefix_ok(*mask, q) || !float_mask(*mask) || mask->requires_grad() || mask->device() != q.device())
      return py::none();
  }
  const bool save = at::GradMode::is_enabled() &&
                    (q.requires_grad() || k.requires_grad() || v.requires_grad() || bias.requires_grad());
  variable_list r;
  {
    py::gil_scoped_release release;
    c10::cuda::CUDAGuard guard(q.device());
    if (save) {
      r = AttentionFn::apply(q, k, v, bias, mask, true);
    } else {
      at::NoGradGuard no_grad;
      r = AttentionFn::forward(nullptr, q, k, v, bias, mask, false);
    }
  }
  if (return_lse) return py::make_tuple(r[0], r[1]);
  return py::cast(r[0]);
}

// Launches behind the torch.library operators: flattened batch, lane-padded head dim.
std::tuple<Tensor, Tensor> attn_fwd(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& mask,
                                    const Tensor& bias, double scale) {
  c10::cuda::CUDAGuard guard(q_.device());
  const Shape s{q_.size(0), q_.size(1), q_.size(2), q_.size(3), q_.size(4), bias.size(0)};
  const Tensor q = kernel_layout(q_), k = kernel_layout(k_), v = kernel_layout(v_);
  const Operands op = prepare(mask, bias, s);
  Tensor out = empty_bf16({s.B, s.O, s.N, s.H, s.D}, q), lse = empty_f32({s.B, s.O, s.H, s.N}, q);
  launch_fwd(q, k, v, op, s, scale, out, lse);
  return {out, lse};
}

std::tuple<Tensor, Tensor, Tensor, Tensor> attn_bwd(const Tensor& q_, const Tensor& k_, const Tensor& v_,
                                                    const Tensor& d_out, const Tensor& out, const Tensor& lse,
                                                    const Tensor& mask, const Tensor& bias, double scale) {
  c10::cuda::CUDAGuard guard(q_.device());
  const Shape s{q_.size(0), q_.size(1), q_.size(2), q_.size(3), q_.size(4), bias.size(0)};
  const Tensor q = kernel_layout(q_), k = kernel_layout(k_), v = kernel_layout(v_);
  const Grads g = launch_bwd(q, k, v, d_out.contiguous(), out.contiguous(), lse, prepare(mask, bias, s), s, scale,
                             TPF_ATTN_BWD_STAGE_ALL);
  return {g.dq, g.dk, g.dv, g.dbias};
}

}  // namespace tpf_torch
