// Operand preparation of triangle attention: the additive mask and the pair bias in the layout the TMA
// descriptors need (mask fp32, row pitch a multiple of 4; bias bf16, row pitch a multiple of 8), from whatever
// type and strides the caller's tensors have.
//
// Both are small next to q / k / v (HBM bound: one read, one write, a few microseconds), so what counts is that
// they are ONE launch: a zero fill, a strided copy and a conversion per tensor took five.
#include <cuda_fp16.h>

#include "tpf_host.cuh"
#include "tpf_internal.h"
#include "tpf_ptx.cuh"

namespace tpf {

struct PrepParams {
  PrepSource bias, mask;       // src == nullptr: nothing to do for that operand
  __nv_bfloat16* bias_dst;     // [G,H,N,bias_pitch]
  float* mask_dst;             // [B,O,mask_pitch]
  int H, N, O, bias_pitch, mask_pitch;
  float mask_add, mask_mul;    // mask value = (source + add) * mul
  int64_t bias_groups, mask_groups;  // 8-element / 4-element pieces
  int bias_blocks;
};

__device__ __forceinline__ float prep_load(const PrepSource& s, int64_t off) {
  if (s.type == kPrepF32) return reinterpret_cast<const float*>(s.src)[off];
  if (s.type == kPrepBF16) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(s.src)[off]);
  if (s.type == kPrepBool) return reinterpret_cast<const uint8_t*>(s.src)[off] ? 1.f : 0.f;
  return __half2float(reinterpret_cast<const __half*>(s.src)[off]);
}

__global__ void __launch_bounds__(256) attn_prep_kernel(const PrepParams p) {
  griddep_wait();
  if ((int)blockIdx.x < p.bias_blocks) {
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= p.bias_groups) return;
    const int per_row = p.bias_pitch / 8;
    const int j0 = (int)(i % per_row) * 8;
    int64_t r = i / per_row;
    const int q = (int)(r % p.N);
    r /= p.N;
    const int64_t base = (r / p.H) * p.bias.stride[0] + (r % p.H) * p.bias.stride[1] + q * p.bias.stride[2];
    uint32_t o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int j = j0 + 2 * e;
      const float a = j < p.N ? prep_load(p.bias, base + j * p.bias.stride[3]) : 0.f;
      const float b = j + 1 < p.N ? prep_load(p.bias, base + (j + 1) * p.bias.stride[3]) : 0.f;
      o[e] = pack_bf16x2(a, b);
    }
    reinterpret_cast<uint4*>(p.bias_dst)[i] = make_uint4(o[0], o[1], o[2], o[3]);
  } else {
    const int64_t i = (int64_t)(blockIdx.x - p.bias_blocks) * 256 + threadIdx.x;
    if (i >= p.mask_groups) return;
    const int per_row = p.mask_pitch / 4;
    const int j0 = (int)(i % per_row) * 4;
    const int64_t r = i / per_row;
    const int64_t base = (r / p.O) * p.mask.stride[0] + (r % p.O) * p.mask.stride[1];
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      o[e] = j0 + e < p.N ? (prep_load(p.mask, base + (j0 + e) * p.mask.stride[2]) + p.mask_add) * p.mask_mul : 0.f;
    reinterpret_cast<float4*>(p.mask_dst)[i] = make_float4(o[0], o[1], o[2], o[3]);
  }
}

int attn_prep(const PrepSource& bias, int64_t G, int64_t H, void* bias_dst, int64_t bias_pitch, const PrepSource& mask,
              int64_t B, int64_t O, float* mask_dst, int64_t mask_pitch, int64_t N, cudaStream_t stream, float mask_add,
              float mask_mul) {
  PrepParams p = {};
  p.mask_add = mask_add;
  p.mask_mul = mask_mul;
  p.bias = bias;
  p.mask = mask;
  p.bias_dst = reinterpret_cast<__nv_bfloat16*>(bias_dst);
  p.mask_dst = mask_dst;
  p.H = (int)H; p.N = (int)N; p.O = (int)O;
  p.bias_pitch = (int)bias_pitch;
  p.mask_pitch = (int)mask_pitch;
  p.bias_groups = bias.src ? G * H * N * (bias_pitch / 8) : 0;
  p.mask_groups = mask.src ? B * O * (mask_pitch / 4) : 0;
  const int64_t nb = (p.bias_groups + 255) / 256, nm = (p.mask_groups + 255) / 256;
  TPF_REQUIRE(nb + nm < (1ll << 31), TPF_ERR_INVALID_ARGUMENT, "attn_prep: extent too large");
  p.bias_blocks = (int)nb;
  if (nb + nm == 0) return TPF_OK;
  launch_kernel(attn_prep_kernel, dim3((unsigned)(nb + nm)), dim3(256), 0, stream, p);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

}  // namespace tpf
