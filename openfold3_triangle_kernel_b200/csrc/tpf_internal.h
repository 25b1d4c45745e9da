// C++ entry points of libtpf_b200.so that the native torch layer uses besides the C ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace tpf {

// One strided source operand of attn_prep: element type and element strides of its (up to four) dimensions.
enum PrepType : int { kPrepF32 = 0, kPrepBF16 = 1, kPrepF16 = 2, kPrepBool = 3 };
struct PrepSource {
  const void* src;
  int type;
  int64_t stride[4];
};

// bias (strides g,h,q,k) -> bf16 [G,H,N,bias_pitch]; mask (strides b,o,n) -> fp32 [B,O,mask_pitch]; one launch.
// A source with src == nullptr is skipped.  The mask comes out as (value + mask_add) * mask_mul.
int attn_prep(const PrepSource& bias, int64_t G, int64_t H, void* bias_dst, int64_t bias_pitch, const PrepSource& mask,
              int64_t B, int64_t O, float* mask_dst, int64_t mask_pitch, int64_t N, cudaStream_t stream,
              float mask_add = 0.f, float mask_mul = 1.f);

constexpr double kNoByteLimit = 1e300;

// One triangle-attention problem.  Strides are in elements, order (b, o, h, n); the last dimension is contiguous.
struct AttnCall {
  int64_t B, O, H, N, D, G;  // G: bias batch, 1 or B
  float scale;
  const void *q, *k, *v;     // bf16
  int64_t qs[4], ks[4], vs[4];
  const float* mask;         // fp32 [B,O,mask_pitch]
  int64_t mask_pitch;
  const void* bias;          // bf16 [G,H,N,bias_pitch]
  int64_t bias_pitch;
  void* out;                 // bf16
  int64_t os[4];
  const void* gate;          // bf16 logits: out = attention * sigmoid(gate); or nullptr
  int64_t gs[4];
  float* lse;                // fp32 [B,O,H,N]; may be nullptr in a forward without gate gradients
  // backward
  const void* d_out;         // bf16, gradient of the (ungated) attention result
  int64_t dos[4];
  float* delta;              // fp32 [B,O,H,N] = rowsum(d_out * attention result)
  void *dq, *dk, *dv;        // bf16
  int64_t ds[4];             // strides of dq, dk and dv
  float* dbias;              // fp32 [G,H,N,N]; or nullptr with dbias_rows:
  void* dbias_rows;          // bf16, row (g, i, j) of pitch dbias_ld holds the H bias gradients of pair (i, j), then
  int64_t dbias_ld;          //   zeros up to a multiple of 8 columns
  double dbias_limit = kNoByteLimit;  // most bytes of workspace that chunk planes of dbias may take
};
int attn_forward(const AttnCall& c, cudaStream_t stream);
int attn_backward_qkv(const AttnCall& c, void* workspace, int64_t workspace_bytes, cudaStream_t stream);
int attn_backward_bias(const AttnCall& c, void* workspace, int64_t workspace_bytes, cudaStream_t stream);
int64_t attn_bwd_workspace_bytes(int64_t B, int64_t O, int64_t H, int64_t N, int64_t D);
int64_t attn_dbias_workspace_bytes(int64_t B, int64_t O, int64_t H, int64_t N, int64_t G);
int64_t attn_dbias_rows_workspace_bytes(int64_t B, int64_t O, int64_t H, int64_t N, int64_t G);

// One triangle multiplicative update on the caller's [B,N,N,C] tensors, any N.  The intermediates live on an internal
// grid of B * Np * Np rows (Np = N rounded up to 8, padding rows are zeros), see tpf_pair_rows.cuh.
struct TrimulWeights {
  const float *p_in, *g_in, *p_out, *g_out, *norm_in_w, *norm_in_b, *norm_out_w, *norm_out_b;
};
struct TrimulCall {
  int64_t B, N, Np, C;
  int incoming;
  const void* z;      // bf16 [B,N,N,C]
  const void* mask;   // pair mask; mask_grid == nullptr: fp32 on the internal grid.  nullptr: all ones
  int mask_type;      // 0 fp32, 1 bf16, 2 fp16, 3 bool
  int64_t mask_stride[3];
  float* mask_grid;   // fp32 [B*Np*Np] that the forward fills from `mask`
  TrimulWeights w;
  void* packed;       // bf16 weights in kernel layout (trimul_fwd_workspace_bytes), written by the forward
  void* out;          // bf16 [B,N,N,C]; may be nullptr when `sum` is wanted alone
  void* sum;          // bf16 [B,N,N,C] = z + out, or nullptr
  void *zln, *a_cm, *b_cm, *gate, *x_cm, *xln;            // bf16 [B*Np*Np, C]
  float *mean_in, *rstd_in, *mean_out, *rstd_out;         // fp32 [B*Np*Np]
  // Nothing is kept for a backward (only where trimul_fused(C)): of the intermediates the forward then needs a_cm, b_cm and
  // x_cm alone, z_stats in place of the input norm's statistics, and no mask_grid.
  bool infer;
  float* z_stats;     // fp32 [B*Np*Np, 2]
};
// The forward's weights in kernel layout (tpf_trimul_fwd.cu): w = gamma W in bf16, rows [a_p; a_g; b_p; b_g; g] (input norm)
// and z (output norm), all halved (which is exact: p sigmoid(g) = p / 2 + p / 2 tanh(g / 2)); st: (sum of w, sum of beta W)
// of each row.
struct TrimulFused {
  const void* w;    // bf16 [6C, C]
  const float* st;  // fp32 [6C, 2]
};
bool trimul_fused(int64_t C);
// NN: internal rows per batch entry.  The first writes the statistics of z's rows (mean_in and rstd_in, or z_stats), which
// the second reads.
int trimul_project(const TrimulCall& t, const TrimulFused& w, int64_t NN, cudaStream_t stream);
int trimul_output(const TrimulCall& t, const TrimulFused& w, int64_t NN, cudaStream_t stream);
struct TrimulGrads {
  const void* d_out;  // bf16 [B,N,N,C]
  const void* d_res;  // gradient to add to d_z (residual connection), or nullptr
  void* d_z;
  float *p_in, *g_in, *p_out, *g_out, *norm_in_w, *norm_in_b, *norm_out_w, *norm_out_b;
};
int64_t trimul_fwd_workspace_bytes(int64_t B, int64_t N, int64_t C);
int64_t trimul_bwd_workspace_bytes(int64_t B, int64_t rows_per_batch, int64_t C);
int trimul_forward(const TrimulCall& t, cudaStream_t stream);
int trimul_backward(const TrimulCall& t, const TrimulGrads& g, void* workspace, int64_t workspace_bytes,
                    cudaStream_t stream);

// Triangle attention as the pair block uses it: out = z + Linear_o(sigmoid(gate) * attention(LayerNorm(z))), with the
// bias-free q / k / v / gate / bias projections of the normalised rows.  `ending`: the node attends along the first
// pair index (outer index = second), everything else stays in the caller's row order.
struct PairAttnWeights {
  const float *ln_w, *ln_b, *w_z, *w_q, *w_k, *w_v, *w_g, *w_o;
};
struct PairAttnCall {
  int64_t B, N, C, H, D;
  int ending;
  const void* z;     // bf16 [B,N,N,C]
  const void* mask;  // pair mask (1 keeps), type / strides as in TrimulCall
  int mask_type;
  int64_t mask_stride[3];
  float inf;
  PairAttnWeights w;
  void* out;         // bf16 [B,N,N,C]
  // intermediates; R = B*N*N rows
  void* packed;      // bf16 weights in kernel layout (pair_attn_packed_bytes), written by the forward
  void* x;           // bf16 [R,C] normalised rows
  void* qkvg;        // bf16 [4H][R][D]: q, k, v and gate-logit planes
  void* og;          // bf16 [R,H*D] gated attention result
  void* bias;        // bf16 [B,H,N,pitch 8]
  float* mask_add;   // fp32 [B,N,pitch 4] additive mask
  float *mean, *rstd;  // fp32 [R]; may be nullptr in a forward that keeps nothing
  float* lse;          // fp32 [B,N,H,N], likewise
};
struct PairAttnGrads {
  const void* d_out;  // bf16 [B,N,N,C]
  void* d_z;
  float *ln_w, *ln_b, *w_z, *w_q, *w_k, *w_v, *w_g, *w_o;
};
int64_t pair_attn_packed_bytes(int64_t C, int64_t H, int64_t D);
int64_t pair_attn_bwd_workspace_bytes(int64_t B, int64_t N, int64_t C, int64_t H, int64_t D);
bool pair_attn_supported(int64_t C, int64_t H, int64_t D);
int pair_attn_forward(const PairAttnCall& t, cudaStream_t stream);
int pair_attn_backward(const PairAttnCall& t, const PairAttnGrads& g, void* workspace, int64_t workspace_bytes,
                       cudaStream_t stream);

}  // namespace tpf
