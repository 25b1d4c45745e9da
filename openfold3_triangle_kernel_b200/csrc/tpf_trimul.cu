// Triangle multiplicative update (outgoing / incoming), forward and backward, for sm_100a.
//
//   zn  = LayerNorm_in(z)                                  a = (zn Wap^T) * sigmoid(zn Wag^T) * mask
//   x[i,j,c] = sum_k a[i,k,c] b[j,k,c]   (outgoing)        b = (zn Wbp^T) * sigmoid(zn Wbg^T) * mask
//   x[i,j,c] = sum_k a[k,i,c] b[k,j,c]   (incoming)        out = (LayerNorm_out(x) Wz^T) * sigmoid(zn Wg^T)
//
// Stands in for the reference's native TriMul stages and the cuBLAS calls between them
// (openfold3/core/kernels/turbopairformer/turbopairformer_trimul_cuda.cu:634-1047, 1202-1470,
//  1541-1809, 226-438 and turbopairformer_trimul.py:184-392).  Rounding points follow the
// reference: fp32 master weights are rounded to bf16 once, LayerNorm statistics are fp32 with
// var = E[x^2] - mean^2 and eps = 1e-5, intermediates (zn, a, b, gate logits, x) are bf16,
// weight gradients are fp32 sums folded in a fixed order.  (The forward's kernels at C = 64 and 128 round gamma W instead
// of zn and of the weights, and their own gate not at all.)
//
// At C = 64 and 128 the forward's projections and output stage are the kernels of tpf_trimul_fwd.cu; every other
// GEMM-shaped stage runs on the tcgen05 engine of tpf_gemm.cuh, with gating, masking and the
// channel-major re-layout that the k-contraction wants fused into GEMM epilogues.  The
// a / b / x tensors live channel-major ([B*C][N*N]) so that the k-contraction is a plain batched
// GEMM in both directions (K-major operands when outgoing, MN-major when incoming).
#include <cuda_fp16.h>

#include <initializer_list>
#include <utility>

#include "tpf_gemm_host.cuh"
#include "tpf_internal.h"
#include "tpf_norm.cuh"
#include "tpf_pair_rows.cuh"

namespace tpf {

static __device__ int g_trimul_status;

int trimul_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  TPF_CUDA_OK(cudaMemcpyFromSymbol(&v, g_trimul_status, sizeof(int)));
  if (v) TPF_CUDA_OK(cudaMemcpyToSymbol(g_trimul_status, &zero, sizeof(int)));
  *out = v;
  return TPF_OK;
}

int bmm_bf16(const void* A, int64_t lda, int64_t bsa, int a_mn, const void* B, int64_t ldb, int64_t bsb, int b_mn,
             void* D, int64_t ldd, int64_t bsd, int out_f32, int64_t M, int64_t N, int64_t K, int64_t batch,
             int64_t k_per_split, int swizzle_bytes, cudaStream_t stream);

// =============================================================================================
// weight packing: fp32 masters -> bf16 W5 [5C,C] = [a_p; a_g; b_p; b_g; g], W5T [C,5C], Wz [C,C], WzT [C,C] (W5 null:
// not wanted), and what the fused forward reads (TrimulFused; fw null: not wanted).  One warp a row.
// =============================================================================================
__global__ void __launch_bounds__(64) trimul_pack_weights_kernel(const TrimulWeights w, bf16* __restrict__ W5,
                                                                  bf16* __restrict__ W5T, bf16* __restrict__ Wz,
                                                                  bf16* __restrict__ WzT, bf16* __restrict__ fw,
                                                                  float2* __restrict__ st, int C) {
  griddep_wait();
  const int row = (int)((blockIdx.x * 64 + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  const int blk = row / C, r = row % C;
  const float* src = blk == 0 ? w.p_in + r * C : blk == 1 ? w.g_in + r * C : blk == 2 ? w.p_in + (C + r) * C
                     : blk == 3 ? w.g_in + (C + r) * C : blk == 4 ? w.g_out + r * C : w.p_out + r * C;
  const float* gamma = blk == 5 ? w.norm_out_w : w.norm_in_w;
  const float* beta = blk == 5 ? w.norm_out_b : w.norm_in_b;
  float s = 0.f, t = 0.f, in[4], ga[4], be[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = lane + 32 * i;
    const bool ok = k < C;
    in[i] = ok ? src[k] : 0.f;
    ga[i] = ok && fw != nullptr ? gamma[k] : 0.f;
    be[i] = ok && fw != nullptr ? beta[k] : 0.f;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int k = lane + 32 * i;
    if (k >= C) break;
    const float v = in[i];
    if (W5 != nullptr) {
      const bf16 h = __float2bfloat16(v);
      if (blk < 5) {
        W5[row * C + k] = h;
        W5T[k * 5 * C + row] = h;
      } else {
        Wz[r * C + k] = h;
        WzT[k * C + r] = h;
      }
    }
    if (fw != nullptr) {
      const bf16 h = __float2bfloat16(0.5f * ga[i] * v);
      fw[row * C + k] = h;
      s += __bfloat162float(h);
      t += 0.5f * be[i] * v;
    }
  }
  if (fw == nullptr) return;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, off);
    t += __shfl_xor_sync(0xffffffffu, t, off);
  }
  if (lane == 0) st[row] = make_float2(s, t);
}

// =============================================================================================
// Output norm forward: channel-major x [B*C][NN] -> row-major LayerNorm(x) [R,C] + mean/rstd
// =============================================================================================
// The channel-major -> row-major turn is done on 8x8 blocks of bf16 by ldmatrix.trans instead of element by
// element through shared memory: the tile is stored as it is loaded (16 bytes = 8 pair rows of one
// channel), every lane then holds, per 8-channel group, two neighbouring channels of ONE pair row, so
// the LayerNorm statistics are a register sum plus two shuffles, and the normalised row goes back
// through a row-major staging tile that is read out in 16-byte pieces.  About one shared-memory
// instruction per element instead of four.
template <int C>
__global__ void __launch_bounds__(256, 2) trimul_xnorm_fwd_kernel(const bf16* __restrict__ x_cm,
                                                                  const float* __restrict__ gamma,
                                                                  const float* __restrict__ beta,
                                                                  bf16* __restrict__ xln, float* __restrict__ mean,
                                                                  float* __restrict__ rstd, int64_t NN,
                                                                  int tiles_per_batch, int n_tiles) {
  griddep_wait();
  constexpr int TR = 64;                    // pair rows per tile; warp w owns rows 8w .. 8w+7
  constexpr int IN_PITCH = TR * 2 + 16;     // bytes per channel row of the input tile (+16: conflict-free ldmatrix)
  constexpr int OUT_PITCH = C * 2 + 16;     // bytes per pair row of the staging tile
  constexpr int NG = C / 32;                // ldmatrix.x4 steps: 4 groups of 8 channels each
  extern __shared__ __align__(16) uint8_t xnorm_smem[];
  uint8_t* xs0 = xnorm_smem;                       // two input tiles: the next one is fetched (cp.async)
  uint8_t* ys = xnorm_smem + 2 * C * IN_PITCH;     // while the current one is processed
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int k2 = 2 * (lane & 3);            // this lane's channel pair inside an 8-channel group
  const int rr = 8 * warp + (lane >> 2);    // this lane's pair row inside the tile
  float2 g[NG][4], bt[NG][4];  // read one by one, once per CTA: a parameter may start at any element of a flat buffer
#pragma unroll
  for (int i = 0; i < NG; ++i)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int c = 32 * i + 8 * m + k2;
      g[i][m] = make_float2(gamma[c], gamma[c + 1]);
      bt[i][m] = make_float2(beta[c], beta[c + 1]);
    }
  // 16-byte copies: 8 consecutive pair rows of one channel (NN is a multiple of 8)
  auto fetch = [&](int tile, uint8_t* dst) {
    const int fb = tile / tiles_per_batch;
    const int64_t f0 = (int64_t)(tile % tiles_per_batch) * TR;
#pragma unroll
    for (int idx = threadIdx.x; idx < C * (TR / 8); idx += 256) {
      const int c = idx / (TR / 8), j8 = idx % (TR / 8);
      const bool ok = f0 + 8 * j8 < NN;
      cp_async_16(dst + c * IN_PITCH + 16 * j8, x_cm + ((int64_t)fb * C + c) * NN + (ok ? f0 + 8 * j8 : 0), ok);
    }
    cp_async_commit();
  };
  int buf = 0;
  if ((int)blockIdx.x < n_tiles) fetch(blockIdx.x, xs0);
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, buf ^= 1) {
    const int bb = tile / tiles_per_batch;
    const int64_t r0 = (int64_t)(tile % tiles_per_batch) * TR;
    uint8_t* xs = xs0 + buf * C * IN_PITCH;
    // the other buffer was last read (ldmatrix) before the barriers of the previous iteration
    if (tile + (int)gridDim.x < n_tiles) {
      fetch(tile + gridDim.x, xs0 + (buf ^ 1) * C * IN_PITCH);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    uint32_t fr[NG][4];
#pragma unroll
    for (int i = 0; i < NG; ++i)
      ldmatrix_x4_trans(fr[i], smem_u32(xs + (32 * i + lane) * IN_PITCH + 16 * warp));
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < NG; ++i)
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float v0 = bf16_lo(fr[i][m]), v1 = bf16_hi(fr[i][m]);
        s1 += v0 + v1;
        s2 += v0 * v0 + v1 * v1;
      }
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s2 += __shfl_xor_sync(0xffffffffu, s2, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    s2 += __shfl_xor_sync(0xffffffffu, s2, 2);
    const float mu = s1 * (1.f / C);
    const float rs = rsqrtf(fmaxf(s2 * (1.f / C) - mu * mu, 0.f) + 1e-5f);
#pragma unroll
    for (int i = 0; i < NG; ++i)
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float y0 = (bf16_lo(fr[i][m]) - mu) * rs * g[i][m].x + bt[i][m].x;
        const float y1 = (bf16_hi(fr[i][m]) - mu) * rs * g[i][m].y + bt[i][m].y;
        *reinterpret_cast<uint32_t*>(ys + rr * OUT_PITCH + (32 * i + 8 * m + k2) * 2) = pack_bf16x2(y0, y1);
      }
    if (mean != nullptr && (lane & 3) == 0 && r0 + rr < NN) {
      mean[(int64_t)bb * NN + r0 + rr] = mu;
      rstd[(int64_t)bb * NN + r0 + rr] = rs;
    }
    __syncthreads();
    // row-major stores: 16 bytes (8 channels) per thread, a warp covers two whole rows
#pragma unroll
    for (int idx = threadIdx.x; idx < TR * (C / 8); idx += 256) {
      const int j = idx / (C / 8), c8 = idx % (C / 8);
      if (r0 + j < NN)
        *reinterpret_cast<uint4*>(xln + ((int64_t)bb * NN + r0 + j) * C + 8 * c8) =
            *reinterpret_cast<const uint4*>(ys + j * OUT_PITCH + 16 * c8);
    }
    // the next iteration's first barrier orders these reads before the staging tile is rewritten; the
    // input tile is rewritten only after every warp has passed the barrier above, i.e. after its ldmatrix
  }
}

// =============================================================================================
// GEMM epilogues
// =============================================================================================
// Projection + gating (C = 32 and 96; the others: tpf_trimul_fwd.cu).  GEMM N axis = [a_p | a_g] [b_p | b_g] [g | pad],
// one tile of width 2C each.  a and b are stored channel-major.  Each lane owns one row of the accumulator tile, which
// would make 2-byte scattered stores; the 32x32 block is transposed through a per-warp smem tile so that each lane writes
// 32 consecutive rows of ONE channel (4 x 16 bytes).
// Integer divisions by run-time values cost a lone epilogue warp 300-600 cycles each (a chain of conversions and
// a reciprocal on the XU pipe), once per tile and on its critical path, so the epilogues avoid them: the tile
// kind comes from comparisons, and the batch entry of a row is found by division only when there is more than one.
__device__ __forceinline__ int tile_kind(int n0, int C) { return n0 >= 4 * C ? 2 : n0 >= 2 * C ? 1 : 0; }
__device__ __forceinline__ void split_row(int row, int64_t NN, int M, int& bb, int& rr) {
  if ((int64_t)M <= NN) {  // one batch entry
    bb = 0;
    rr = row;
  } else {
    bb = (int)((uint32_t)row / (uint32_t)NN);
    rr = row - bb * (int)NN;
  }
}

struct ProjGateParams {
  CUtensorMap map_gate;  // stores: [R][C]
  bf16* a_cm;        // [B*C][NN]
  bf16* b_cm;        // [B*C][NN]
  const float* mask; // [R]
  int C;
  int64_t NN;
};
struct EpiProjGate {
  using Params = ProjGateParams;
  static constexpr bool kPaired = true;
  static constexpr bool kStaged = false;
  static constexpr int kSmemPerWarp = 4608;  // staging tiles, or one 32 x 33 float block
  struct Pre {
    float mk;  // pair mask of this lane's row
  };
  __device__ static __forceinline__ void prefetch2(const Params& p, const GemmShape& sh, int, int m0, int rit, int,
                                                   int, int, Pre& pre) {
    const int m = m0 + rit;
    pre.mk = (m < sh.M) ? p.mask[m] : 0.f;
  }
  __device__ static __forceinline__ void apply2(const Params& p, const GemmShape& sh, int, int m0, int rit, int n0,
                                                int c0, const float (&v0)[32], const float (&v1)[32], float* wsm,
                                                int lane, const Pre& pre, int& buf) {
    const int which = tile_kind(n0, p.C);
    const int m = m0 + rit;
    const int m_base = m - lane;  // first row of this warp's 32-row block (a multiple of 32)
    if (which == 2) {
      uint32_t pk[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(v0[2 * i], v0[2 * i + 1]);
      if (m_base < sh.M)
        warp_tile_store_tma(reinterpret_cast<uint8_t*>(wsm), buf, lane, pk, &p.map_gate, c0, m_base, 0);
      return;
    }
    // a / b tile: each lane owns one row of the accumulator tile, which would
    // make 2-byte scattered stores; the 32x32 block is transposed through a per-warp smem tile so that each
    // lane writes 8 consecutive rows of four channels (4 x 16 bytes).
    bulk_wait_read<0>();  // the block shares its memory with the gate tiles' staging buffers
    __syncwarp();
    const float mk = pre.mk;
#pragma unroll
    for (int i = 0; i < 32; ++i) wsm[lane * 33 + i] = v0[i] * sigmoid_fast(v1[i]) * mk;
    __syncwarp();
    // four lanes per channel: each store instruction covers 8 channels x 64 contiguous bytes (32 rows)
    int bb, rr;
    split_row(m_base, p.NN, sh.M, bb, rr);
    const int piece = lane & 3;  // rows 8*piece .. 8*piece+7 of the block
    bf16* dst = (which == 0 ? p.a_cm : p.b_cm) + ((int64_t)bb * p.C + c0 + (lane >> 2)) * p.NN + rr + 8 * piece;
    const float* col = wsm + (8 * piece) * 33 + (lane >> 2);
    const bool ok = m_base + 8 * piece + 7 < sh.M;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float* cg = col + 8 * g;  // channel 8*g + lane/4
      uint4 u;
      u.x = pack_bf16x2(cg[0 * 33], cg[1 * 33]);
      u.y = pack_bf16x2(cg[2 * 33], cg[3 * 33]);
      u.z = pack_bf16x2(cg[4 * 33], cg[5 * 33]);
      u.w = pack_bf16x2(cg[6 * 33], cg[7 * 33]);
      if (ok) *reinterpret_cast<uint4*>(dst + (int64_t)(8 * g) * p.NN) = u;
    }
    __syncwarp();
  }
};

// Output projection: out = acc * sigmoid(gate), and with a residual input sum = res + out.  Rows of the internal
// (padded) grid are stored at the caller's positions; padding rows are dropped.
template <bool RES>
struct EpiOutGate {
  struct Params {
    CUtensorMap map_out;  // !RES, identity rows: out leaves by TMA
    bf16* out;        // caller's rows x C; may be null when `sum` is wanted alone
    bf16* sum;        // RES: caller's rows x C
    const bf16* res;  // RES: residual input, caller's rows x C
    const bf16* gate; // [R][C]
    PairRows rows;
    int C;
  };
  static constexpr bool kPaired = false;
  static constexpr bool kStaged = false;
  static constexpr int kSmemPerWarp = kTmaTiles;
  struct Pre {
    uint4 g[4];            // 32 gate logits of this lane's row
    uint4 r[RES ? 4 : 1];  // residual, in the arrangement of the stores (8 rows x 64 bytes per access)
  };
  __device__ static __forceinline__ void prefetch(const Params& p, const GemmShape& sh, int, int m, int n0, int lane,
                                                  Pre& pre) {
    if constexpr (RES) load_rows(p.res, p.rows, m - lane, sh.M, p.C, n0, lane, pre.r);
    if (m >= sh.M) return;
    const uint4* g = reinterpret_cast<const uint4*>(p.gate + (int64_t)m * p.C + n0);
#pragma unroll
    for (int i = 0; i < 4; ++i) pre.g[i] = g[i];
  }
  __device__ static __forceinline__ void apply(const Params& p, const GemmShape& sh, int, int m, int n0,
                                               const float (&v)[32], float* wsm, int lane, const Pre& pre, int& buf) {
    uint32_t ow[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 gu = m < sh.M ? pre.g[i] : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t gw[4] = {gu.x, gu.y, gu.z, gu.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        ow[4 * i + e] = pack_bf16x2(v[8 * i + 2 * e] * sigmoid_fast(bf16_lo(gw[e])),
                                    v[8 * i + 2 * e + 1] * sigmoid_fast(bf16_hi(gw[e])));
    }
    uint8_t* tile = reinterpret_cast<uint8_t*>(wsm);
    if constexpr (RES)
      store_rows_added(tile, lane, ow, p.rows, m - lane, sh.M, p.C, n0, p.out, p.sum, pre.r);
    else if (p.rows.identity) {
      if (m - lane < sh.M) warp_tile_store_tma(tile, buf, lane, ow, &p.map_out, n0, m - lane, 0);
    } else
      warp_tile_store(tile, lane, ow, [&](int r) { return row_address(p.out, p.rows, m - lane + r, sh.M, p.C, n0); });
  }
};

// Backward of the gated projections: recomputed (p, g) pair + incoming d_a / d_b -> d_proj5[:, 0:4C]
struct EpiGateSplitBwd {
  struct Params {
    CUtensorMap map_d;  // stores: d_proj5 [R][5C]
    const bf16* da_cm;  // [B*C][NN]
    const bf16* db_cm;
    const float* mask;  // [R]
    bf16* d_proj5;      // [R][5C]
    int C;
    int64_t NN;
  };
  static constexpr bool kPaired = true;
  static constexpr bool kStaged = true;
  static constexpr int kSmemPerWarp = kTmaTiles;  // a 32 x 34 bf16 block, then two staging tiles
  struct Pre {
    uint4 d[4];  // incoming gradient, channel-major: d[g] = 8 consecutive rows of channel 8*g + lane/4
    float mk;    // pair mask of this lane's row
  };
  __device__ static __forceinline__ void prefetch2(const Params& p, const GemmShape& sh, int, int m0, int rit, int n0,
                                                   int c0, int lane, Pre& pre) {
    const int which = tile_kind(n0, p.C);  // 0: a, 1: b
    const int m = m0 + rit;
    const int m_base = m - lane;
    int bb, rr;
    split_row(m_base, p.NN, sh.M, bb, rr);
    // four lanes per channel: load g reads rows 8*piece..+7 of channel 8*g + lane/4, so one load
    // instruction covers 8 channels x 64 contiguous bytes
    const int piece = lane & 3;
    const bf16* src = (which == 0 ? p.da_cm : p.db_cm) + ((int64_t)bb * p.C + c0 + (lane >> 2)) * p.NN + rr + 8 * piece;
    const bool ok = m_base + 8 * piece + 7 < sh.M;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      pre.d[g] = make_uint4(0u, 0u, 0u, 0u);
      if (ok) pre.d[g] = *reinterpret_cast<const uint4*>(src + (int64_t)(8 * g) * p.NN);
    }
    pre.mk = (m < sh.M) ? p.mask[m] : 0.f;
  }
  // The prefetched channel-major block is transposed through smem so that afterwards lane = row finds
  // its 32 channels in the 34 bf16 from lane * 34 on (17 words a row: no bank conflicts either way).
  __device__ static __forceinline__ void stage(const Pre& pre, float* wsm, int lane) {
    bulk_wait_read<0>();  // the staging tiles of the previous chunk lie in the same memory
    __syncwarp();
    uint16_t* col = reinterpret_cast<uint16_t*>(wsm) + (8 * (lane & 3)) * 34 + (lane >> 2);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const uint4 u = pre.d[g];
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        col[(2 * e) * 34 + 8 * g] = (uint16_t)w[e];
        col[(2 * e + 1) * 34 + 8 * g] = (uint16_t)(w[e] >> 16);
      }
    }
    __syncwarp();
  }
  __device__ static __forceinline__ void apply2(const Params& p, const GemmShape& sh, int, int m0, int rit, int n0,
                                                int c0, const float (&v0)[32], const float (&v1)[32], float* wsm,
                                                int lane, const Pre& pre, int& buf) {
    const int which = tile_kind(n0, p.C);  // 0: a, 1: b
    const int m = m0 + rit;
    // d = incoming gradient * mask; t = tanh(g / 2): sigmoid s = 0.5 + 0.5 t, s (1 - s) = 0.25 - 0.25 t^2.
    // Channel pairs (i, i + 1) go through packed fp32 arithmetic and are rounded to bf16 at once, so that
    // only the packed results stay live.
    const uint64_t mk2 = f2_pack(pre.mk, pre.mk);
    const uint64_t half2 = f2_pack(0.5f, 0.5f), quarter2 = f2_pack(0.25f, 0.25f), nquarter2 = f2_pack(-0.25f, -0.25f);
    const uint32_t* drow = reinterpret_cast<const uint32_t*>(wsm) + lane * 17;
    uint32_t pk0[16], pk1[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const uint32_t dw = drow[i];
      const uint64_t d2 = f2_mul(f2_pack(bf16_lo(dw), bf16_hi(dw)), mk2);
      float h0, h1, a0, a1, b0, b1;
      f2_unpack(f2_mul(f2_pack(v1[2 * i], v1[2 * i + 1]), half2), h0, h1);
      const uint64_t t2 = f2_pack(tanh_fast(h0), tanh_fast(h1));
      const uint64_t s2 = f2_fma(t2, half2, half2);
      const uint64_t ss2 = f2_fma(f2_mul(t2, nquarter2), t2, quarter2);
      f2_unpack(f2_mul(d2, s2), a0, a1);
      f2_unpack(f2_mul(f2_mul(d2, f2_pack(v0[2 * i], v0[2 * i + 1])), ss2), b0, b1);
      pk0[i] = pack_bf16x2(a0, a1);
      pk1[i] = pack_bf16x2(b0, b1);
    }
    __syncwarp();  // the transposed gradient block has been consumed: its smem is reused as staging tiles
    const int m_base = m - lane;
    if (m_base >= sh.M) return;
    const int col = which * 2 * p.C + c0;  // d_p; d_g lies C columns further
    warp_tile_store_tma(reinterpret_cast<uint8_t*>(wsm), buf, lane, pk0, &p.map_d, col, m_base, 0);
    warp_tile_store_tma(reinterpret_cast<uint8_t*>(wsm), buf, lane, pk1, &p.map_d, col + p.C, m_base, 0);
  }
};
// (300 bytes of spills instead of 40.  Per lane -> uniform, us at N = 384: C = 128, 256 columns 65.5 -> 104; C = 96, 192 columns, where
// the per-lane one spills 500 bytes, 96.5 -> 77; C = 64 31.4 -> 30.5; C = 32 22.6 -> 20.5.)
template <>
constexpr bool kPerLaneWarpIndex<EpiGateSplitBwd, 256> = true;

// =============================================================================================
// backward elementwise stages
// =============================================================================================
// d_y = d_out * sigmoid(g);  d_glogit = d_out * out * (1 - sigmoid(g))  -> d_proj5[:, 4C:5C]
// d_out and out have the caller's rows, the results the internal (padded) rows: zeros where no caller row exists.
__global__ void __launch_bounds__(256) trimul_out_gate_bwd_kernel(const bf16* __restrict__ d_out,
                                                                  const bf16* __restrict__ out,
                                                                  const bf16* __restrict__ gate, bf16* __restrict__ d_y,
                                                                  bf16* __restrict__ d_proj5, const PairRows rows,
                                                                  const FastDiv per_row, int64_t R, int C) {
  griddep_wait();
  const uint32_t n8 = (uint32_t)(R * C / 8);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += gridDim.x * blockDim.x) {
    const uint32_t row = per_row.div(i);
    const int col8 = (int)(i - row * per_row.d);
    const PairPos pos = rows.locate(row);
    uint32_t y[4] = {0u, 0u, 0u, 0u}, l[4] = {0u, 0u, 0u, 0u};
    if (pos.src >= 0) {
      const uint4 a = *reinterpret_cast<const uint4*>(d_out + pos.src * C + col8 * 8);
      const uint4 b = *reinterpret_cast<const uint4*>(out + pos.src * C + col8 * 8);
      const uint4 g = reinterpret_cast<const uint4*>(gate)[i];
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w}, gw[4] = {g.x, g.y, g.z, g.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float s0 = sigmoid_fast(bf16_lo(gw[e])), s1 = sigmoid_fast(bf16_hi(gw[e]));
        const float d0 = bf16_lo(aw[e]), d1 = bf16_hi(aw[e]);
        y[e] = pack_bf16x2(d0 * s0, d1 * s1);
        l[e] = pack_bf16x2(d0 * bf16_lo(bw[e]) * (1.f - s0), d1 * bf16_hi(bw[e]) * (1.f - s1));
      }
    }
    reinterpret_cast<uint4*>(d_y)[i] = make_uint4(y[0], y[1], y[2], y[3]);
    *reinterpret_cast<uint4*>(d_proj5 + (int64_t)row * 5 * C + 4 * C + col8 * 8) = make_uint4(l[0], l[1], l[2], l[3]);
  }
}

// Output-norm backward.  d_xln row-major [R,C], x channel-major -> d_x channel-major; per-CTA partial sums
// for d_gamma / d_beta (fixed order inside the CTA, folded in CTA order later).
//
// Same data movement as the forward norm: x is stored as loaded and turned by ldmatrix.trans, so that a
// lane holds, for ONE pair row, two neighbouring channels of each 8-channel group; d_xln is staged
// row-major and read back in that same arrangement; d_x goes back through stmatrix.trans into the
// channel-major tile (in place: a warp only touches its own 8 pair rows of every channel) and leaves
// in 16-byte pieces.  The d_gamma / d_beta sums of a lane's channels stay in registers over all the
// tiles of the CTA and are reduced once at the end.
template <int C>
__global__ void __launch_bounds__(256, 2) trimul_xnorm_bwd_kernel(const bf16* __restrict__ d_xln,
                                                                  const bf16* __restrict__ x_cm,
                                                                  const float* __restrict__ gamma,
                                                                  const float* __restrict__ mean,
                                                                  const float* __restrict__ rstd,
                                                                  bf16* __restrict__ dx_cm, float* __restrict__ partials,
                                                                  int64_t NN, int tiles_per_batch, int n_tiles) {
  griddep_wait();
  constexpr int TR = 64;
  constexpr int IN_PITCH = TR * 2 + 16;
  constexpr int OUT_PITCH = C * 2 + 16;
  constexpr int NG = C / 32;
  extern __shared__ __align__(16) uint8_t xnorm_smem[];
  // two (x, d_xln) tile pairs: the next pair is fetched (cp.async) while the current one is processed
  uint8_t* xs0 = xnorm_smem;                          // x, later d_x: [channel][pair row]
  uint8_t* ds0 = xnorm_smem + 2 * C * IN_PITCH;       // d_xln: [pair row][channel]
  __shared__ float2 gsm[C / 2];
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int k2 = 2 * (lane & 3);
  const int rr = 8 * warp + (lane >> 2);
  if (threadIdx.x < C / 2) gsm[threadIdx.x] = make_float2(gamma[2 * threadIdx.x], gamma[2 * threadIdx.x + 1]);
  float2 ag[NG][4], ab[NG][4];  // running sums of d * xhat and d for this lane's channels
#pragma unroll
  for (int i = 0; i < NG; ++i)
#pragma unroll
    for (int m = 0; m < 4; ++m) ag[i][m] = ab[i][m] = make_float2(0.f, 0.f);

  auto fetch = [&](int tile, uint8_t* xdst, uint8_t* ddst) {
    const int fb = tile / tiles_per_batch;
    const int64_t f0 = (int64_t)(tile % tiles_per_batch) * TR;
#pragma unroll
    for (int idx = threadIdx.x; idx < C * (TR / 8); idx += 256) {
      const int c = idx / (TR / 8), j8 = idx % (TR / 8);
      const bool ok = f0 + 8 * j8 < NN;
      cp_async_16(xdst + c * IN_PITCH + 16 * j8, x_cm + ((int64_t)fb * C + c) * NN + (ok ? f0 + 8 * j8 : 0), ok);
    }
#pragma unroll
    for (int idx = threadIdx.x; idx < TR * (C / 8); idx += 256) {
      const int j = idx / (C / 8), c8 = idx % (C / 8);
      const bool ok = f0 + j < NN;
      cp_async_16(ddst + j * OUT_PITCH + 16 * c8, d_xln + ((int64_t)fb * NN + (ok ? f0 + j : 0)) * C + 8 * c8, ok);
    }
    cp_async_commit();
  };
  int buf = 0;
  if ((int)blockIdx.x < n_tiles) fetch(blockIdx.x, xs0, ds0);
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, buf ^= 1) {
    const int bb = tile / tiles_per_batch;
    const int64_t r0 = (int64_t)(tile % tiles_per_batch) * TR;
    uint8_t* xs = xs0 + buf * C * IN_PITCH;
    uint8_t* ds = ds0 + buf * TR * OUT_PITCH;
    const bool row_ok = r0 + rr < NN;
    const float mu = row_ok ? mean[(int64_t)bb * NN + r0 + rr] : 0.f;
    const float rs = row_ok ? rstd[(int64_t)bb * NN + r0 + rr] : 0.f;
    // The other buffer pair was last touched in the previous iteration: its d_x read-out (plain loads) was
    // completed by every thread before that thread got here, but by OTHER threads only if they are past it too
    __syncthreads();
    if (tile + (int)gridDim.x < n_tiles) {
      fetch(tile + gridDim.x, xs0 + (buf ^ 1) * C * IN_PITCH, ds0 + (buf ^ 1) * TR * OUT_PITCH);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    uint32_t fx[NG][4], fd[NG][4];
#pragma unroll
    for (int i = 0; i < NG; ++i) {
      ldmatrix_x4_trans(fx[i], smem_u32(xs + (32 * i + lane) * IN_PITCH + 16 * warp));
#pragma unroll
      for (int m = 0; m < 4; ++m)
        fd[i][m] = *reinterpret_cast<const uint32_t*>(ds + rr * OUT_PITCH + (32 * i + 8 * m + k2) * 2);
    }
    float a1 = 0.f, a2 = 0.f;
#pragma unroll
    for (int i = 0; i < NG; ++i)
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float2 gm = gsm[(32 * i + 8 * m + k2) >> 1];
        const float x0 = (bf16_lo(fx[i][m]) - mu) * rs, x1 = (bf16_hi(fx[i][m]) - mu) * rs;
        const float d0 = bf16_lo(fd[i][m]), d1 = bf16_hi(fd[i][m]);
        const float g0 = gm.x * d0, g1 = gm.y * d1;
        a1 += g0 + g1;
        a2 += g0 * x0 + g1 * x1;
        ag[i][m].x += d0 * x0;
        ag[i][m].y += d1 * x1;
        ab[i][m].x += d0;
        ab[i][m].y += d1;
      }
    a1 += __shfl_xor_sync(0xffffffffu, a1, 1);
    a2 += __shfl_xor_sync(0xffffffffu, a2, 1);
    a1 += __shfl_xor_sync(0xffffffffu, a1, 2);
    a2 += __shfl_xor_sync(0xffffffffu, a2, 2);
    const float m1 = a1 * (1.f / C), m2 = a2 * (1.f / C);
#pragma unroll
    for (int i = 0; i < NG; ++i) {
      uint32_t out[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const float2 gm = gsm[(32 * i + 8 * m + k2) >> 1];
        const float x0 = (bf16_lo(fx[i][m]) - mu) * rs, x1 = (bf16_hi(fx[i][m]) - mu) * rs;
        const float v0 = rs * (gm.x * bf16_lo(fd[i][m]) - m1 - x0 * m2);
        const float v1 = rs * (gm.y * bf16_hi(fd[i][m]) - m1 - x1 * m2);
        out[m] = pack_bf16x2(v0, v1);
      }
      stmatrix_x4_trans(smem_u32(xs + (32 * i + lane) * IN_PITCH + 16 * warp), out);
    }
    __syncthreads();
#pragma unroll
    for (int idx = threadIdx.x; idx < C * (TR / 8); idx += 256) {
      const int c = idx / (TR / 8), j8 = idx % (TR / 8);
      if (r0 + 8 * j8 < NN)
        *reinterpret_cast<uint4*>(dx_cm + ((int64_t)bb * C + c) * NN + r0 + 8 * j8) =
            *reinterpret_cast<const uint4*>(xs + c * IN_PITCH + 16 * j8);
    }
  }

  // ---- d_gamma / d_beta partials of this CTA: the 8 pair rows of a warp (lanes that differ in lane / 4) in
  //      shuffle order, then the 8 warps in warp order; a fixed tree, no atomics
  __syncthreads();
  float* red = reinterpret_cast<float*>(ds0);  // [8 warps][2][C]
#pragma unroll
  for (int i = 0; i < NG; ++i)
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      float v[4] = {ag[i][m].x, ag[i][m].y, ab[i][m].x, ab[i][m].y};
#pragma unroll
      for (int off = 4; off < 32; off <<= 1)
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] += __shfl_xor_sync(0xffffffffu, v[e], off);
      if (lane < 4) {
        const int c = 32 * i + 8 * m + k2;
        red[(warp * 2 + 0) * C + c] = v[0];
        red[(warp * 2 + 0) * C + c + 1] = v[1];
        red[(warp * 2 + 1) * C + c] = v[2];
        red[(warp * 2 + 1) * C + c + 1] = v[3];
      }
    }
  __syncthreads();
  if (threadIdx.x < 2 * C) {
    const int which = threadIdx.x / C, c = threadIdx.x % C;
    float t = red[(0 * 2 + which) * C + c];
#pragma unroll
    for (int w = 1; w < 8; ++w) t += red[(w * 2 + which) * C + c];
    partials[(int64_t)blockIdx.x * 2 * C + which * C + c] = t;
  }
}

// =============================================================================================
// host orchestration
// =============================================================================================
struct TrimulPacked {
  bf16 *W5, *W5T, *Wz, *WzT;
};
static int64_t packed_weight_elems(int64_t C) { return 12 * C * C; }

static TrimulPacked packed_at(void* buf, int64_t C) {
  bf16* base = reinterpret_cast<bf16*>(buf);
  return TrimulPacked{base, base + 5 * C * C, base + 10 * C * C, base + 11 * C * C};
}
// behind them in the forward's workspace
static TrimulFused fused_at(void* buf, int64_t C) {
  bf16* w = reinterpret_cast<bf16*>(buf) + packed_weight_elems(C);
  return TrimulFused{w, reinterpret_cast<float*>(w + 6 * C * C)};
}
static int pack_weights(const TrimulWeights& w, const TrimulPacked* pk, const TrimulFused* fused, int C, cudaStream_t stream) {
  const TrimulPacked p = pk ? *pk : TrimulPacked{};
  const TrimulFused f = fused ? *fused : TrimulFused{};
  launch_kernel(trimul_pack_weights_kernel, dim3(6 * C / 2), dim3(64), 0, stream, w, p.W5, p.W5T, p.Wz, p.WzT,
                (bf16*)const_cast<void*>(f.w), reinterpret_cast<float2*>(const_cast<float*>(f.st)), C);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

// BLOCKS: weight blocks of C rows (a_p, a_g, b_p, b_g and, forward, g).
template <int C, int BLOCKS, class Epi>
static int proj_gemm(const bf16* zln, const bf16* W5, int64_t R, const typename Epi::Params& ep, int* status,
                     cudaStream_t stream) {
  // The gated epilogues are latency-bound: at C = 128 and 96 (four, three 32-column chunk pairs per tile) 16
  // epilogue warps keep one chunk pair each in flight; narrower tiles have work for 8 only.
  // The weights (all of them, or a tile of 2C rows x C) stay in shared memory; only the activations stream.
  const GemmShape sh{(int)R, BLOCKS * C, C, 1, 0};
  if (resident_pays(R, (BLOCKS + 1) / 2)) {
    using Cfg = GemmCfg<128, 2 * C, 128, false, 128, false, (C + 63) / 64, (C >= 96 ? 16 : 8), 3, (C + 63) / 64, BLOCKS * C>;
    return launch_gemm<Cfg, Epi>(zln, C, 0, W5, C, 0, sh, ep, status, stream);
  }
  using Cfg = GemmCfg<128, 2 * C, 128, false, 128, false, 4, (C >= 96 ? 16 : 8), 2, (C + 63) / 64>;
  return launch_gemm<Cfg, Epi>(zln, C, 0, W5, C, 0, sh, ep, status, stream);
}

template <int C>
static int trimul_fwd_t(const TrimulCall& t, const float* mask, const TrimulPacked& pk, const TrimulFused& fused, int64_t NN,
                        int stages, int* status, cudaStream_t stream) {
  // t.Np: internal extent (a multiple of 8); NN: internal rows per batch entry (Np * Np for a whole pair tensor,
  // N_local * N for a row shard).
  const int64_t B = t.B, N = t.Np, R = B * NN;
  const bf16* z = (const bf16*)t.z;
  bf16 *zln = (bf16*)t.zln, *xln = (bf16*)t.xln, *x_cm = (bf16*)t.x_cm;
  const PairRows rows = PairRows::make(t.N, t.Np, false);
  constexpr bool kFused = C % 64 == 0;
  int rc = TPF_OK;
  if (stages & 1) {
    if constexpr (kFused) {
      if ((rc = trimul_project(t, fused, NN, stream))) return rc;
    } else {
      const PairMask pm{t.mask, t.mask_type, t.mask_stride[0], t.mask_stride[1], t.mask_stride[2]};
      launch_kernel(rows.identity && !t.mask_grid ? ln_fwd_kernel<C, false> : ln_fwd_kernel<C, true>,
                    dim3(ln_fwd_blocks<C>(R)), dim3(256), 0, stream, z, t.w.norm_in_w, t.w.norm_in_b, zln, t.mean_in,
                    t.rstd_in, rows, pm, t.mask_grid, R);
      TPF_LAUNCH_OK();
      ProjGateParams ep{{}, (bf16*)t.a_cm, (bf16*)t.b_cm, mask, C, NN};
      if ((rc = make_store_tmap(&ep.map_gate, t.gate, C, R, C, 1, 0))) return rc;
      if ((rc = proj_gemm<C, 5, EpiProjGate>(zln, pk.W5, R, ep, status, stream))) return rc;
    }
  }
  if (stages & 2) {
    // k-contraction: batch = B*C problems of N x N x N
    rc = bmm_bf16(t.a_cm, N, NN, t.incoming, t.b_cm, N, NN, t.incoming, x_cm, N, NN, 0, N, N, N, B * C, 0, 128, stream);
    if (rc) return rc;
  }
  if (stages & 4) {
    if (!t.infer) {
      const int tiles = (int)((NN + 63) / 64);
      int grid = (int)(B * tiles);
      if (grid > 2 * sm_count()) grid = 2 * sm_count();
      auto kern = trimul_xnorm_fwd_kernel<C>;
      constexpr int smem = 2 * C * (64 * 2 + 16) + 64 * (C * 2 + 16);
      static PerDeviceOnce once;  // per instantiation
      if ((rc = ensure_dynamic_smem(kern, smem, once))) return rc;
      launch_kernel(kern, dim3(grid), dim3(256), smem, stream, x_cm, t.w.norm_out_w, t.w.norm_out_b, xln, t.mean_out,
                    t.rstd_out, NN, tiles, (int)(B * tiles));
      TPF_LAUNCH_OK();
    }
    if constexpr (kFused) return trimul_output(t, fused, NN, stream);
    GemmShape sh{(int)R, C, C, 1, 0};
    if (t.sum) {
      // The residual doubles the operands the epilogue keeps in flight: narrow tiles, so that a warp has one 32-column
      // chunk and 165 registers for it (wider tiles with two chunks, or with 16 warps of 96 registers, spill).  The
      // activations are read once more per tile column, from L2.
      using Cfg = GemmCfg<128, 32, 128, false, 128, false, 4>;
      typename EpiOutGate<true>::Params ep{{}, (bf16*)t.out, (bf16*)t.sum, z, (const bf16*)t.gate, rows, C};
      rc = launch_gemm<Cfg, EpiOutGate<true>>(xln, C, 0, pk.Wz, C, 0, sh, ep, status, stream);
    } else {
      using Cfg = GemmCfg<128, C, 128, false, 128, false, 4>;
      typename EpiOutGate<false>::Params ep{{}, (bf16*)t.out, nullptr, nullptr, (const bf16*)t.gate, rows, C};
      if (rows.identity && (rc = make_store_tmap(&ep.map_out, t.out, C, R, C, 1, 0))) return rc;
      rc = launch_gemm<Cfg, EpiOutGate<false>>(xln, C, 0, pk.Wz, C, 0, sh, ep, status, stream);
    }
    if (rc) return rc;
  }
  return TPF_OK;
}

static void split_plan(int64_t R, int tiles_mn, int* n_splits, int64_t* k_per_split) {
  int64_t s = sm_count() / (tiles_mn > 0 ? tiles_mn : 1);
  if (s < 1) s = 1;
  int64_t kps = ((R + s - 1) / s + 63) / 64 * 64;
  if (kps < 64) kps = 64;
  *k_per_split = kps;
  *n_splits = (int)((R + kps - 1) / kps);
}

struct TrimulBwdWorkspace {
  bf16 *wpack, *d_y, *d_proj5, *d_xln, *dx_cm, *da_cm, *db_cm;  // d_zln aliases d_xln
  float *part_w5, *part_wz, *part_ln_out, *part_ln_in;
  int splits_w5, splits_wz, blocks_ln_out, blocks_ln_in, rows_per_block_in;
  int64_t kps_w5, kps_wz;
  int64_t total_bytes;
};

static int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

static void plan_bwd_workspace(int64_t B, int64_t NN, int64_t C, char* base, TrimulBwdWorkspace* w) {
  const int64_t R = B * NN;
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  w->wpack = reinterpret_cast<bf16*>(take(packed_weight_elems(C) * 2));
  w->d_y = reinterpret_cast<bf16*>(take(R * C * 2));
  w->d_proj5 = reinterpret_cast<bf16*>(take(R * 5 * C * 2));
  w->d_xln = reinterpret_cast<bf16*>(take(R * C * 2));
  w->dx_cm = reinterpret_cast<bf16*>(take(R * C * 2));
  w->da_cm = reinterpret_cast<bf16*>(take(R * C * 2));
  w->db_cm = reinterpret_cast<bf16*>(take(R * C * 2));
  split_plan(R, (int)((5 * C + 127) / 128), &w->splits_w5, &w->kps_w5);
  split_plan(R, 1, &w->splits_wz, &w->kps_wz);
  w->part_w5 = reinterpret_cast<float*>(take((int64_t)w->splits_w5 * 5 * C * C * 4));
  w->part_wz = reinterpret_cast<float*>(take((int64_t)w->splits_wz * C * C * 4));
  {
    // one partial row per CTA of the output-norm backward kernel (persistent, two CTAs per SM)
    const int64_t tiles = B * ((NN + 63) / 64);
    w->blocks_ln_out = (int)(tiles < 2 * sm_count() ? tiles : 2 * sm_count());
  }
  w->rows_per_block_in = ln_bwd_rows_per_block(R);
  w->blocks_ln_in = (int)((R + w->rows_per_block_in - 1) / w->rows_per_block_in);
  w->part_ln_out = reinterpret_cast<float*>(take((int64_t)w->blocks_ln_out * 2 * C * 4));
  w->part_ln_in = reinterpret_cast<float*>(take((int64_t)w->blocks_ln_in * 2 * C * 4));
  w->total_bytes = off;
}

template <int C>
static int trimul_bwd_t(const TrimulCall& t, const TrimulGrads& g, const float* mask, const TrimulPacked* packed,
                        int64_t NN, int stages, bf16* dx_io, bf16* da_io, bf16* db_io, char* workspace, int* status,
                        cudaStream_t stream) {
  const int64_t B = t.B, N = t.Np, R = B * NN;
  const bf16 *z = (const bf16*)t.z, *zln = (const bf16*)t.zln, *xln = (const bf16*)t.xln, *a_cm = (const bf16*)t.a_cm,
             *b_cm = (const bf16*)t.b_cm, *d_out = (const bf16*)g.d_out;
  const PairRows rows = PairRows::make(t.N, t.Np, false);
  TrimulBwdWorkspace w;
  plan_bwd_workspace(B, NN, C, workspace, &w);
  if (dx_io) w.dx_cm = dx_io;  // staged (sharded) use: the caller moves these between ranks
  if (da_io) w.da_cm = da_io;
  if (db_io) w.db_cm = db_io;
  TrimulPacked pk = packed ? *packed : packed_at(w.wpack, C);
  int rc;
  if (!packed && (rc = pack_weights(t.w, &pk, nullptr, C, stream))) return rc;
  FoldList folds;

  if (stages & 1) {
  // 1. output gate: d_y, d_glogit
  {
    TPF_REQUIRE(R * C / 8 < (1ll << 31), TPF_ERR_INVALID_ARGUMENT, "trimul_bwd: extent too large");
    int blocks = (int)((R * C / 8 + 255) / 256);
    if (blocks > 16 * sm_count()) blocks = 16 * sm_count();
    launch_kernel(trimul_out_gate_bwd_kernel, dim3(blocks), dim3(256), 0, stream, d_out, (const bf16*)t.out,
                  (const bf16*)t.gate, w.d_y, w.d_proj5, rows, FastDiv::make(C / 8), R, C);
    TPF_LAUNCH_OK();
  }
  // 2. d_xln = d_y Wz ; d_wz = d_y^T xln
  {
    using Cfg = GemmCfg<128, 128, 128, false, 128, false, 4>;
    using Epi = EpiStore<bf16>;
    GemmShape sh{(int)R, C, C, 1, 0};
    typename Epi::Params ep;
    if ((rc = epi_store_params<bf16>(&ep, w.d_xln, C, 0, sh))) return rc;
    if ((rc = launch_gemm<Cfg, Epi>(w.d_y, C, 0, pk.WzT, C, 0, sh, ep, status, stream))) return rc;
  }
  rc = bmm_bf16(w.d_y, C, 0, 1, xln, C, 0, 1, w.part_wz, C, (int64_t)C * C, 1, C, C, R, w.splits_wz, w.kps_wz, 128,
                stream);
  if (rc) return rc;
  folds.add(w.part_wz, w.splits_wz, C * C, C * C, g.p_out);
  // 3. output norm backward -> d_x (channel-major), d_gamma_out, d_beta_out
  {
    const int tiles = (int)((NN + 63) / 64);
    auto kern = trimul_xnorm_bwd_kernel<C>;
    constexpr int smem = 2 * C * (64 * 2 + 16) + 2 * 64 * (C * 2 + 16);
    static PerDeviceOnce once;  // per instantiation
    if ((rc = ensure_dynamic_smem(kern, smem, once))) return rc;
    launch_kernel(kern, dim3(w.blocks_ln_out), dim3(256), smem, stream, w.d_xln, (const bf16*)t.x_cm, t.w.norm_out_w,
                  t.mean_out, t.rstd_out, w.dx_cm, w.part_ln_out, NN, tiles, (int)(B * tiles));
    TPF_LAUNCH_OK();
    folds.add(w.part_ln_out, w.blocks_ln_out, 2 * C, C, g.norm_out_w, g.norm_out_b);
  }
  }
  if (stages & 2) {
  // 4. contraction backward
  if (!t.incoming) {
    // d_a[c,i,k] = sum_j d_x[c,i,j] b[c,j,k] ; d_b[c,j,k] = sum_i d_x[c,i,j] a[c,i,k]
    if ((rc = bmm_bf16(w.dx_cm, N, NN, 0, b_cm, N, NN, 1, w.da_cm, N, NN, 0, N, N, N, B * C, 0, 128, stream))) return rc;
    if ((rc = bmm_bf16(w.dx_cm, N, NN, 1, a_cm, N, NN, 1, w.db_cm, N, NN, 0, N, N, N, B * C, 0, 128, stream))) return rc;
  } else {
    // d_a[c,k,i] = sum_j b[c,k,j] d_x[c,i,j] ; d_b[c,k,j] = sum_i a[c,k,i] d_x[c,i,j]
    if ((rc = bmm_bf16(b_cm, N, NN, 0, w.dx_cm, N, NN, 0, w.da_cm, N, NN, 0, N, N, N, B * C, 0, 128, stream))) return rc;
    if ((rc = bmm_bf16(a_cm, N, NN, 0, w.dx_cm, N, NN, 1, w.db_cm, N, NN, 0, N, N, N, B * C, 0, 128, stream))) return rc;
  }
  }
  if (stages & 4) {
  // 5. gated projections backward (recompute p, g) -> d_proj5[:, 0:4C]
  {
    EpiGateSplitBwd::Params ep{{}, w.da_cm, w.db_cm, mask, w.d_proj5, C, NN};
    if ((rc = make_store_tmap(&ep.map_d, w.d_proj5, 5 * C, R, 5 * C, 1, 0))) return rc;
    if ((rc = proj_gemm<C, 4, EpiGateSplitBwd>(zln, pk.W5, R, ep, status, stream))) return rc;
  }
  // 6. d_zln = d_proj5 W5 ; dW5 = d_proj5^T zln
  bf16* d_zln = w.d_xln;
  {
    // d_proj5 streams from DRAM (W5^T comes from L2): six stages keep enough of it in flight per SM
    using Cfg = GemmCfg<128, 128, 128, false, 128, false, 6>;
    using Epi = EpiStore<bf16>;
    GemmShape sh{(int)R, C, 5 * C, 1, 0};
    typename Epi::Params ep;
    if ((rc = epi_store_params<bf16>(&ep, d_zln, C, 0, sh))) return rc;
    if ((rc = launch_gemm<Cfg, Epi>(w.d_proj5, 5 * C, 0, pk.W5T, 5 * C, 0, sh, ep, status, stream))) return rc;
  }
  rc = bmm_bf16(w.d_proj5, 5 * C, 0, 1, zln, C, 0, 1, w.part_w5, C, (int64_t)5 * C * C, 1, 5 * C, C, R, w.splits_w5,
                w.kps_w5, 128, stream);
  if (rc) return rc;
  folds.add(w.part_w5, w.splits_w5, 5 * C * C, C * C, g.p_in, g.g_in, g.p_in + C * C, g.g_in + C * C, g.g_out);
  // 7. input norm backward
  launch_kernel(ln_bwd_kernel<C>, dim3(w.blocks_ln_in), dim3(256), 0, stream, d_zln, z, t.w.norm_in_w,
                t.mean_in, t.rstd_in, (bf16*)g.d_z, w.part_ln_in, rows, (const bf16*)g.d_res, R, w.rows_per_block_in);
  TPF_LAUNCH_OK();
  folds.add(w.part_ln_in, w.blocks_ln_in, 2 * C, C, g.norm_in_w, g.norm_in_b);
  }
  return folds.launch(stream);
}

static int check_trimul_rows(const char* who, int64_t N, int64_t NN, int stages) {
  TPF_REQUIRE(stages >= 1 && stages <= 7, TPF_ERR_INVALID_ARGUMENT, "%s: stages must be a non-empty mask of 1|2|4", who);
  TPF_REQUIRE(NN > 0 && NN % 64 == 0, TPF_ERR_UNSUPPORTED, "%s: rows per batch (%lld) must be a positive multiple of 64",
              who, (long long)NN);
  TPF_REQUIRE(NN == N * N || !(stages & 2), TPF_ERR_INVALID_ARGUMENT,
              "%s: the contraction stage needs whole pair tensors (rows per batch == N*N)", who);
  return TPF_OK;
}

static int check_trimul_shape(const char* who, int64_t B, int64_t N, int64_t C) {
  TPF_REQUIRE(B > 0 && N > 0, TPF_ERR_INVALID_ARGUMENT, "%s: B and N must be positive", who);
  TPF_REQUIRE(C == 32 || C == 64 || C == 96 || C == 128, TPF_ERR_UNSUPPORTED, "%s: C=%lld not in {32,64,96,128}", who,
              (long long)C);
  TPF_REQUIRE(N % 8 == 0, TPF_ERR_UNSUPPORTED, "%s: N=%lld must be a multiple of 8 (pad on the host side)", who,
              (long long)N);
  TPF_REQUIRE(B * N * N < (1ll << 31), TPF_ERR_INVALID_ARGUMENT, "%s: B*N*N too large", who);
  return TPF_OK;
}

int64_t trimul_fwd_workspace_bytes(int64_t B, int64_t N, int64_t C) {
  return align256(packed_weight_elems(C) * 2 + (trimul_fused(C) ? 6 * C * C * 2 + 6 * C * 8 : 0));
}

int64_t trimul_bwd_workspace_bytes(int64_t B, int64_t NN, int64_t C) {
  TrimulBwdWorkspace w;
  plan_bwd_workspace(B, NN, C, nullptr, &w);
  return w.total_bytes;
}

static int trimul_status(int** status) {
  static PerDeviceAddress cache;
  return device_symbol_address(g_trimul_status, cache, reinterpret_cast<void**>(status));
}

// The kernels' mask: the caller's own when it has the internal layout, else the copy the input norm writes.
static const float* grid_mask(const TrimulCall& t) {
  return t.mask_grid ? t.mask_grid : reinterpret_cast<const float*>(t.mask);
}

// The bf16 tensors are read and written 16 bytes at a time (masks, weights, statistics element by element).
static int check_trimul_aligned(const char* who, std::initializer_list<std::pair<const char*, const void*>> tensors) {
  for (const auto& t : tensors) TPF_REQUIRE_ALIGNED16(t.second, who, t.first);
  return TPF_OK;
}

static int trimul_fwd_run(const TrimulCall& t, int64_t NN, int stages, cudaStream_t stream) {
  int* status = nullptr;
  int rc = check_trimul_aligned("trimul_fwd", {{"z", t.z}, {"out", t.out}, {"sum", t.sum}, {"zln", t.zln}, {"a_cm", t.a_cm},
                                               {"b_cm", t.b_cm}, {"gate", t.gate}, {"x_cm", t.x_cm}, {"xln", t.xln},
                                               {"workspace", t.packed}});
  if (rc || (rc = trimul_status(&status))) return rc;
  const TrimulPacked pk = packed_at(t.packed, t.C);
  const TrimulFused fused = fused_at(t.packed, t.C);
  if ((rc = pack_weights(t.w, t.infer ? nullptr : &pk, trimul_fused(t.C) ? &fused : nullptr, (int)t.C, stream))) return rc;
  switch (t.C) {
    case 32: return trimul_fwd_t<32>(t, grid_mask(t), pk, fused, NN, stages, status, stream);
    case 64: return trimul_fwd_t<64>(t, grid_mask(t), pk, fused, NN, stages, status, stream);
    case 96: return trimul_fwd_t<96>(t, grid_mask(t), pk, fused, NN, stages, status, stream);
    case 128: return trimul_fwd_t<128>(t, grid_mask(t), pk, fused, NN, stages, status, stream);
  }
  return fail(TPF_ERR_UNSUPPORTED, "trimul_fwd: unsupported C");
}

static int trimul_bwd_run(const TrimulCall& t, const TrimulGrads& g, int64_t NN, int stages, void* dx_io, void* da_io,
                          void* db_io, void* workspace, cudaStream_t stream) {
  int* status = nullptr;
  int rc = check_trimul_aligned("trimul_bwd", {{"d_out", g.d_out}, {"d_res", g.d_res}, {"d_z", g.d_z}, {"z", t.z},
                                               {"out", t.out}, {"zln", t.zln}, {"a_cm", t.a_cm}, {"b_cm", t.b_cm},
                                               {"gate", t.gate}, {"x_cm", t.x_cm}, {"xln", t.xln}, {"dx_cm", dx_io},
                                               {"da_cm", da_io}, {"db_cm", db_io}, {"packed weights", t.packed}});
  if (rc || (rc = trimul_status(&status))) return rc;
  TrimulPacked pk = packed_at(t.packed, t.C);
  const TrimulPacked* packed = t.packed ? &pk : nullptr;
  bf16 *dx = (bf16*)dx_io, *da = (bf16*)da_io, *db = (bf16*)db_io;
  char* ws = (char*)workspace;
  switch (t.C) {
    case 32: return trimul_bwd_t<32>(t, g, grid_mask(t), packed, NN, stages, dx, da, db, ws, status, stream);
    case 64: return trimul_bwd_t<64>(t, g, grid_mask(t), packed, NN, stages, dx, da, db, ws, status, stream);
    case 96: return trimul_bwd_t<96>(t, g, grid_mask(t), packed, NN, stages, dx, da, db, ws, status, stream);
    case 128: return trimul_bwd_t<128>(t, g, grid_mask(t), packed, NN, stages, dx, da, db, ws, status, stream);
  }
  return fail(TPF_ERR_UNSUPPORTED, "trimul_bwd: unsupported C");
}

int trimul_forward(const TrimulCall& t, cudaStream_t stream) {
  int rc = check_trimul_shape("trimul_fwd", t.B, t.Np, t.C);
  if (rc) return rc;
  return trimul_fwd_run(t, t.Np * t.Np, 7, stream);
}

int trimul_backward(const TrimulCall& t, const TrimulGrads& g, void* workspace, int64_t workspace_bytes,
                    cudaStream_t stream) {
  int rc = check_trimul_shape("trimul_bwd", t.B, t.Np, t.C);
  if (rc) return rc;
  TPF_REQUIRE(workspace && workspace_bytes >= trimul_bwd_workspace_bytes(t.B, t.Np * t.Np, t.C) &&
                  (reinterpret_cast<uintptr_t>(workspace) & 255) == 0,
              TPF_ERR_WORKSPACE, "trimul_bwd: workspace too small or misaligned");
  return trimul_bwd_run(t, g, t.Np * t.Np, 7, nullptr, nullptr, nullptr, workspace, stream);
}

int trimul_fwd(const void* z, const float* mask, const float* p_in, const float* g_in, const float* p_out,
               const float* g_out, const float* gin, const float* bin, const float* gout, const float* bout,
               int incoming, int64_t B, int64_t N, int64_t C, void* out, void* zln, float* mean_in, float* rstd_in,
               void* a_cm, void* b_cm, void* gate, void* x_cm, void* xln, float* mean_out, float* rstd_out,
               void* workspace, int64_t workspace_bytes, int64_t NN, int stages, cudaStream_t stream) {
  int rc = check_trimul_shape("trimul_fwd", B, N, C);
  if (rc) return rc;
  if (NN == 0) NN = N * N;
  if ((rc = check_trimul_rows("trimul_fwd", N, NN, stages))) return rc;
  TPF_REQUIRE(z && mask && p_in && g_in && p_out && g_out && gin && bin && gout && bout && out && zln && mean_in &&
                  rstd_in && a_cm && b_cm && gate && x_cm && xln && mean_out && rstd_out,
              TPF_ERR_INVALID_ARGUMENT, "trimul_fwd: null pointer");
  TPF_REQUIRE(workspace && workspace_bytes >= trimul_fwd_workspace_bytes(B, N, C), TPF_ERR_WORKSPACE,
              "trimul_fwd: workspace of %lld bytes required", (long long)trimul_fwd_workspace_bytes(B, N, C));
  TrimulCall t = {};
  t.B = B; t.N = N; t.Np = N; t.C = C; t.incoming = incoming;
  t.z = z; t.mask = mask;
  t.w = {p_in, g_in, p_out, g_out, gin, bin, gout, bout};
  t.packed = workspace;
  t.out = out; t.zln = zln; t.mean_in = mean_in; t.rstd_in = rstd_in; t.a_cm = a_cm; t.b_cm = b_cm; t.gate = gate;
  t.x_cm = x_cm; t.xln = xln; t.mean_out = mean_out; t.rstd_out = rstd_out;
  return trimul_fwd_run(t, NN, stages, stream);
}

int trimul_bwd(const void* d_out, const void* z, const float* mask, const float* p_in, const float* g_in,
               const float* p_out, const float* g_out, const float* gin, const float* gout, int incoming, int64_t B,
               int64_t N, int64_t C, const void* out, const void* zln, const float* mean_in, const float* rstd_in,
               const void* a_cm, const void* b_cm, const void* gate, const void* x_cm, const void* xln,
               const float* mean_out, const float* rstd_out, void* d_z, float* d_p_in, float* d_g_in, float* d_p_out,
               float* d_g_out, float* d_gin, float* d_bin, float* d_gout, float* d_bout, void* workspace,
               int64_t workspace_bytes, int64_t NN, int stages, void* dx_io, void* da_io, void* db_io,
               cudaStream_t stream) {
  int rc = check_trimul_shape("trimul_bwd", B, N, C);
  if (rc) return rc;
  if (NN == 0) NN = N * N;
  if ((rc = check_trimul_rows("trimul_bwd", N, NN, stages))) return rc;
  TPF_REQUIRE(d_out && z && mask && p_in && g_in && p_out && g_out && gin && gout && out && zln && mean_in &&
                  rstd_in && a_cm && b_cm && gate && x_cm && xln && mean_out && rstd_out && d_z && d_p_in && d_g_in &&
                  d_p_out && d_g_out && d_gin && d_bin && d_gout && d_bout,
              TPF_ERR_INVALID_ARGUMENT, "trimul_bwd: null pointer");
  TPF_REQUIRE(workspace && workspace_bytes >= trimul_bwd_workspace_bytes(B, NN, C) &&
                  (reinterpret_cast<uintptr_t>(workspace) & 255) == 0,
              TPF_ERR_WORKSPACE, "trimul_bwd: 256-byte aligned workspace of %lld bytes required",
              (long long)trimul_bwd_workspace_bytes(B, NN, C));
  TrimulCall t = {};
  t.B = B; t.N = N; t.Np = N; t.C = C; t.incoming = incoming;
  t.z = z; t.mask = mask;
  t.w = {p_in, g_in, p_out, g_out, gin, nullptr, gout, nullptr};
  t.out = const_cast<void*>(out); t.zln = const_cast<void*>(zln);
  t.mean_in = const_cast<float*>(mean_in); t.rstd_in = const_cast<float*>(rstd_in);
  t.a_cm = const_cast<void*>(a_cm); t.b_cm = const_cast<void*>(b_cm); t.gate = const_cast<void*>(gate);
  t.x_cm = const_cast<void*>(x_cm); t.xln = const_cast<void*>(xln);
  t.mean_out = const_cast<float*>(mean_out); t.rstd_out = const_cast<float*>(rstd_out);
  const TrimulGrads g{d_out, nullptr, d_z, d_p_in, d_g_in, d_p_out, d_g_out, d_gin, d_bin, d_gout, d_bout};
  return trimul_bwd_run(t, g, NN, stages, dx_io, da_io, db_io, workspace, stream);
}

}  // namespace tpf
