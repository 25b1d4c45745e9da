// C++ entry points of libtpf_b200.so that the native torch layer uses besides the C ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace tpf {

// One strided source operand of attn_prep: element type and element strides of its (up to four) dimensions.
enum PrepType : int { kPrepF32 = 0, kPrepBF16 = 1, kPrepF16 = 2 };
struct PrepSource {
  const void* src;
  int type;
  int64_t stride[4];
};

// bias (strides g,h,q,k) -> bf16 [G,H,N,bias_pitch]; mask (strides b,o,n) -> fp32 [B,O,mask_pitch]; one launch.
// A source with src == nullptr is skipped.
int attn_prep(const PrepSource& bias, int64_t G, int64_t H, void* bias_dst, int64_t bias_pitch, const PrepSource& mask,
              int64_t B, int64_t O, float* mask_dst, int64_t mask_pitch, int64_t N, cudaStream_t stream);

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
};
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

}  // namespace tpf
