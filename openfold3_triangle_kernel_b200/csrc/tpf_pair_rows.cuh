// Row addressing of a pair tensor.  The kernels work on an internal grid of rows (b, i, j); the caller's tensor is
// [B, N, N, ...].  The two differ when N is not a multiple of 8 (the internal grid is padded, so that the channel-major
// tensors keep 16-byte rows) and when the kernels walk the transposed pair tensor.
#pragma once

#include <cuda_fp16.h>

#include "tpf_gemm.cuh"
#include "tpf_ptx.cuh"

namespace tpf {

__device__ __forceinline__ float bf16_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t u) { return __uint_as_float(u & 0xFFFF0000u); }

struct PairPos {
  int64_t src;  // the caller's row, -1: padding
  int b, i, j;  // the caller's coordinates (valid when the map is not the identity)
};

struct PairRows {
  int identity;     // internal row == the caller's row
  int transposed;   // internal (b, i, j) is the caller's (b, j, i)
  int N;            // the caller's extent
  FastDiv pitch;    // internal extent
  FastDiv plane;    // internal rows per batch entry
  static PairRows make(int64_t N, int64_t padded, bool transposed) {
    PairRows r;
    r.identity = (N == padded && !transposed) ? 1 : 0;
    r.transposed = transposed ? 1 : 0;
    r.N = (int)N;
    r.pitch = FastDiv::make((uint32_t)padded);
    r.plane = FastDiv::make((uint32_t)(padded * padded));
    return r;
  }
  __device__ __forceinline__ PairPos split(uint32_t row) const {
    PairPos p;
    p.b = (int)plane.div(row);
    const uint32_t in = row - p.b * plane.d;
    const int r0 = (int)pitch.div(in), r1 = (int)(in - r0 * pitch.d);
    p.i = transposed ? r1 : r0;
    p.j = transposed ? r0 : r1;
    p.src = (p.i < N && p.j < N) ? ((int64_t)p.b * N + p.i) * N + p.j : -1;
    return p;
  }
  __device__ __forceinline__ PairPos locate(uint32_t row) const {
    if (identity) return PairPos{(int64_t)row, 0, 0, (int)row};
    return split(row);
  }
};

// The caller's pair mask, any type and strides; absent: all ones.
struct PairMask {
  const void* src;
  int type;  // 0 fp32, 1 bf16, 2 fp16, 3 bool / uint8
  int64_t sb, si, sj;
  __device__ __forceinline__ float load(const PairPos& p) const {
    if (src == nullptr) return 1.f;
    const int64_t off = p.b * sb + p.i * si + p.j * sj;
    if (type == 0) return reinterpret_cast<const float*>(src)[off];
    if (type == 1) return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(src)[off]);
    if (type == 2) return __half2float(reinterpret_cast<const __half*>(src)[off]);
    return reinterpret_cast<const uint8_t*>(src)[off] ? 1.f : 0.f;
  }
};

// Address of column n0 of internal row `row` in the caller's [.., C] tensor; nullptr: no such row.
__device__ __forceinline__ __nv_bfloat16* row_address(__nv_bfloat16* base, const PairRows& rows, int row, int M, int C,
                                                      int n0) {
  if (row >= M) return nullptr;
  int64_t src = row;
  if (!rows.identity) src = rows.split((uint32_t)row).src;
  return src < 0 ? nullptr : base + src * C + n0;
}

// A warp's 32 rows x 64 bytes in the arrangement of warp_tile_store: access i covers rows 8 i .. 8 i + 7.
__device__ __forceinline__ void load_rows(const __nv_bfloat16* base, const PairRows& rows, int m_base, int M, int C,
                                          int n0, int lane, uint4 (&u)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat16* src =
        row_address(const_cast<__nv_bfloat16*>(base), rows, m_base + 8 * i + (lane >> 2), M, C, n0);
    u[i] = make_uint4(0u, 0u, 0u, 0u);
    if (src != nullptr) u[i] = *reinterpret_cast<const uint4*>(src + 8 * (lane & 3));
  }
}

__device__ __forceinline__ uint4 add_bf16x8(const uint4& x, const uint4& y) {
  const uint32_t a[4] = {x.x, x.y, x.z, x.w}, b[4] = {y.x, y.y, y.z, y.w};
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) o[e] = pack_bf16x2(bf16_lo(a[e]) + bf16_lo(b[e]), bf16_hi(a[e]) + bf16_hi(b[e]));
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Stores a warp's 32 x 32 bf16 block (lane = row, packed column pairs) of internal rows m_base.. at the caller's rows:
// `out` (may be null) receives the block, `sum` the block added to the residual `r` (from load_rows).  The block is
// rounded to bf16 first, as a separate add would see it.
__device__ __forceinline__ void store_rows_added(uint8_t* tile, int lane, const uint32_t (&pk)[16], const PairRows& rows,
                                                 int m_base, int M, int C, int n0, __nv_bfloat16* out,
                                                 __nv_bfloat16* sum, const uint4 (&r)[4]) {
  warp_tile_put(tile, lane, pk);
  __syncwarp();
  const int piece = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = 8 * i + (lane >> 2);
    __nv_bfloat16* dst = row_address(sum, rows, m_base + rr, M, C, n0);
    if (dst == nullptr) continue;
    const uint4 u = warp_tile_get(tile, rr, piece);
    if (out != nullptr) *reinterpret_cast<uint4*>(out + (dst - sum) + 8 * piece) = u;
    *reinterpret_cast<uint4*>(dst + 8 * piece) = add_bf16x8(u, r[i]);
  }
  __syncwarp();
}

}  // namespace tpf
