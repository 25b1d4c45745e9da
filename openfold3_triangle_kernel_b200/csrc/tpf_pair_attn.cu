// Triangle attention as a module of the pair block (forward and backward) for sm_100a:
//
//   x = LayerNorm(z);  q, k, v, g, bias = x W^T;  og = sigmoid(g) * attention(q, k, v, bias, mask);  out = z + og Wo^T
//
// Stands in for the module around the operator (openfold3/core/model/layers/triangular_attention.py:245-409), which as
// separate framework operations is a dozen passes over pair-sized tensors: at N = 768 the norm, the five projections,
// the gate, the transposes and the residual add took 10 of the block's 21 ms.  Here the projections are ONE tensor-core
// GEMM whose epilogue writes q / k / v / gate as [head][row][D] planes (what the attention kernel's tile loads want,
// and whole cache lines per warp store) and the bias as [head][i][j]; the gate is applied where the attention kernel
// stores its rows; the output projection adds the residual.  The backward mirrors it: one GEMM turns d_out into the
// attention gradient, the gate gradient and delta = rowsum(d_o o); dq / dk / dv / dgate / dbias are columns of one row
// matrix, so that one GEMM gives d_x and one split GEMM all five weight gradients.
//
// The ending node is the same computation with the outer and the sequence index of the attention exchanged: only the
// strides handed to the attention kernels differ, nothing is transposed.  (A bias of the ending node indexed
// [query][key] of the transposed tensor is the natural [i][j] one.)
#include "tpf_gemm_host.cuh"
#include "tpf_internal.h"
#include "tpf_norm.cuh"
#include "tpf_pair_rows.cuh"

namespace tpf {

static __device__ int g_pair_attn_status;

int pair_attn_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  TPF_CUDA_OK(cudaMemcpyFromSymbol(&v, g_pair_attn_status, sizeof(int)));
  if (v) TPF_CUDA_OK(cudaMemcpyToSymbol(g_pair_attn_status, &zero, sizeof(int)));
  *out = v;
  return TPF_OK;
}

int bmm_bf16(const void* A, int64_t lda, int64_t bsa, int a_mn, const void* B, int64_t ldb, int64_t bsb, int b_mn,
             void* D, int64_t ldd, int64_t bsd, int out_f32, int64_t M, int64_t N, int64_t K, int64_t batch,
             int64_t k_per_split, int swizzle_bytes, cudaStream_t stream);

// Columns of the joint projection: [q | k | v | g] of H * D each, then H bias columns, zero-padded to a multiple of 8
// (the row pitch of the gradient matrix has to be a multiple of 16 bytes).
static int64_t proj_cols(int64_t H, int64_t D) { return 4 * H * D + (H + 7) / 8 * 8; }

// =============================================================================================
// weight packing: fp32 masters -> bf16 W [P,C], W^T [C,P], Wo [C,HD], Wo^T [HD,C]
// =============================================================================================
struct AttnPacked {
  bf16 *W, *WT, *Wo, *WoT;
};
static AttnPacked attn_packed_at(void* buf, int64_t C, int64_t H, int64_t D) {
  bf16* b = reinterpret_cast<bf16*>(buf);
  const int64_t P = proj_cols(H, D);
  return AttnPacked{b, b + P * C, b + 2 * P * C, b + 2 * P * C + C * H * D};
}

__global__ void __launch_bounds__(256) pair_attn_pack_kernel(const PairAttnWeights w, AttnPacked o, int C, int HD, int H,
                                                             int P) {
  griddep_wait();
  const int n1 = P * C, n = n1 + C * HD;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    if (i < n1) {
      const int p = i / C, c = i - p * C;
      float v = 0.f;
      if (p < HD) v = w.w_q[i];
      else if (p < 2 * HD) v = w.w_k[i - HD * C];
      else if (p < 3 * HD) v = w.w_v[i - 2 * HD * C];
      else if (p < 4 * HD) v = w.w_g[i - 3 * HD * C];
      else if (p < 4 * HD + H) v = w.w_z[i - 4 * HD * C];
      const bf16 h = __float2bfloat16(v);
      o.W[i] = h;
      o.WT[(int64_t)c * P + p] = h;
    } else {
      const int k = i - n1, c = k / HD, d = k - c * HD;
      const bf16 h = __float2bfloat16(w.w_o[k]);
      o.Wo[k] = h;
      o.WoT[d * C + c] = h;
    }
  }
}

// =============================================================================================
// GEMM epilogues
// =============================================================================================
// Joint projection: column chunks of q, k, v, g go to [plane][row][D]; the bias chunk to [b][h][i][j].
struct EpiQkvg {
  struct Params {
    CUtensorMap map;       // D = 32: stores [4H][R][D]
    bf16* planes;
    int64_t plane_stride;  // R * D
    int log_d, D;
    int HD4;               // first bias column
    bf16* bias;
    int H, N;
    int64_t bias_pitch;
    PairRows rows;
  };
  static constexpr bool kPaired = false;
  static constexpr bool kStaged = false;
  static constexpr int kSmemPerWarp = kTmaTiles;
  struct Pre {};
  __device__ static __forceinline__ void prefetch(const Params&, const GemmShape&, int, int, int, int, Pre&) {}
  __device__ static __forceinline__ void apply(const Params& p, const GemmShape& sh, int, int m, int n0,
                                               const float (&v)[32], float* wsm, int lane, const Pre&, int& buf) {
    const int m_base = m - lane;
    if (n0 < p.HD4) {
      uint32_t pk[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
      uint8_t* tile = reinterpret_cast<uint8_t*>(wsm);
      if (p.D == 32) {
        if (m_base < sh.M) warp_tile_store_tma(tile, buf, lane, pk, &p.map, 0, m_base, n0 >> 5);
        return;
      }
      warp_tile_put(tile, lane, pk);
      __syncwarp();
      const int piece = lane & 3, col = n0 + 8 * piece;
      bf16* dst = p.planes + (int64_t)(col >> p.log_d) * p.plane_stride + (col & (p.D - 1));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2);
        if (m_base + r < sh.M)
          *reinterpret_cast<uint4*>(dst + (int64_t)(m_base + r) * p.D) = warp_tile_get(tile, r, piece);
      }
      __syncwarp();
      return;
    }
    if (m < sh.M) {
      const PairPos pos = p.rows.split((uint32_t)m);
      bf16* dst = p.bias + (((int64_t)pos.b * p.H + (n0 - p.HD4)) * p.N + pos.i) * p.bias_pitch + pos.j;
#pragma unroll
      for (int h = 0; h < 32; ++h)
        if (n0 - p.HD4 + h < p.H) dst[(int64_t)h * p.N * p.bias_pitch] = __float2bfloat16(v[h]);
    }
  }
};

// Output projection with residual: out = res + acc.
struct EpiResidual {
  struct Params {
    bf16* out;
    const bf16* res;
    PairRows rows;
    int C;
  };
  static constexpr bool kPaired = false;
  static constexpr bool kStaged = false;
  static constexpr int kSmemPerWarp = 2048;
  struct Pre {
    uint4 r[4];
  };
  __device__ static __forceinline__ void prefetch(const Params& p, const GemmShape& sh, int, int m, int n0, int lane,
                                                  Pre& pre) {
    load_rows(p.res, p.rows, m - lane, sh.M, p.C, n0, lane, pre.r);
  }
  __device__ static __forceinline__ void apply(const Params& p, const GemmShape& sh, int, int m, int n0,
                                               const float (&v)[32], float* wsm, int lane, const Pre& pre, int&) {
    uint32_t pk[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
    store_rows_added(reinterpret_cast<uint8_t*>(wsm), lane, pk, p.rows, m - lane, sh.M, p.C, n0, nullptr, p.out, pre.r);
  }
};

// Backward of output projection and gate: acc = d_og = d_out Wo.  With s = sigmoid(g) and og = s o:
//   d_o = d_og s (planes),  d_g = d_og og (1 - s) (columns 3 HD.. of the row matrix),  delta = sum_d d_og og  per head.
// A 32-column chunk holds whole heads (D = 16 or 32), so delta is a sum inside one thread.
template <int D>
struct EpiGateBwd {
  struct Params {
    CUtensorMap map_o, map_g;  // stores: d_o planes (D = 32), the row matrix's gate columns
    const bf16* gate;      // gate-logit planes [H][R][D]
    const bf16* og;        // [R][HD]
    bf16* d_o;             // planes [H][R][D]
    int64_t plane_stride;
    bf16* d_rows;          // gradient row matrix at its gate columns
    int64_t ld;
    float* delta;          // [B,O,H,N]
    int ending, H, N, HD;
    PairRows rows;
  };
  static constexpr bool kPaired = false;
  static constexpr bool kStaged = false;
  static constexpr int kSmemPerWarp = kTmaTiles;
  struct Pre {
    uint4 g[4], o[4];
  };
  __device__ static __forceinline__ void prefetch(const Params& p, const GemmShape& sh, int, int m, int n0, int,
                                                  Pre& pre) {
    if (m >= sh.M) return;
    const uint4* o = reinterpret_cast<const uint4*>(p.og + (int64_t)m * p.HD + n0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      pre.o[i] = o[i];
      const int col = n0 + 8 * i;
      pre.g[i] = *reinterpret_cast<const uint4*>(p.gate + (int64_t)(col / D) * p.plane_stride + (int64_t)m * D + col % D);
    }
  }
  __device__ static __forceinline__ void apply(const Params& p, const GemmShape& sh, int, int m, int n0,
                                               const float (&v)[32], float* wsm, int lane, const Pre& pre, int& buf) {
    uint32_t po[16], pg[16];
    float sum[2] = {0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint4 gu = m < sh.M ? pre.g[i] : make_uint4(0u, 0u, 0u, 0u);
      const uint4 ou = m < sh.M ? pre.o[i] : make_uint4(0u, 0u, 0u, 0u);
      const uint32_t gw[4] = {gu.x, gu.y, gu.z, gu.w}, ow[4] = {ou.x, ou.y, ou.z, ou.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float d0 = v[8 * i + 2 * e], d1 = v[8 * i + 2 * e + 1];
        const float s0 = sigmoid_rel(bf16_lo(gw[e])), s1 = sigmoid_rel(bf16_hi(gw[e]));
        const float t0 = d0 * bf16_lo(ow[e]), t1 = d1 * bf16_hi(ow[e]);
        po[4 * i + e] = pack_bf16x2(d0 * s0, d1 * s1);
        pg[4 * i + e] = pack_bf16x2(t0 - t0 * s0, t1 - t1 * s1);
        sum[D == 16 ? i >> 1 : 0] += t0 + t1;
      }
    }
    if (m < sh.M) {
      const PairPos pos = p.rows.split((uint32_t)m);
      const int o = p.ending ? pos.j : pos.i, n = p.ending ? pos.i : pos.j;
      float* dst = p.delta + (((int64_t)pos.b * p.N + o) * p.H + n0 / D) * p.N + n;
      dst[0] = sum[0];
      if (D == 16) dst[p.N] = sum[1];
    }
    const int m_base = m - lane;
    if (m_base >= sh.M) return;
    uint8_t* tile = reinterpret_cast<uint8_t*>(wsm);
    if constexpr (D == 32) {
      warp_tile_store_tma(tile, buf, lane, po, &p.map_o, 0, m_base, n0 / D);
    } else {
      bulk_wait_read<0>();
      __syncwarp();
      warp_tile_put(tile, lane, po);
      __syncwarp();
      const int piece = lane & 3, col = n0 + 8 * piece;
      bf16* dst = p.d_o + (int64_t)(col / D) * p.plane_stride + col % D;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2);
        if (m_base + r < sh.M)
          *reinterpret_cast<uint4*>(dst + (int64_t)(m_base + r) * D) = warp_tile_get(tile, r, piece);
      }
      __syncwarp();
    }
    warp_tile_store_tma(tile, buf, lane, pg, &p.map_g, n0, m_base, 0);
  }
};

// =============================================================================================
// host orchestration
// =============================================================================================
static int64_t align256(int64_t x) { return (x + 255) / 256 * 256; }

bool pair_attn_supported(int64_t C, int64_t H, int64_t D) {
  return (C == 32 || C == 64 || C == 96 || C == 128) && (D == 16 || D == 32) && (H * D) % 32 == 0 && H <= 32;
}

int64_t pair_attn_packed_bytes(int64_t C, int64_t H, int64_t D) {
  return align256((2 * proj_cols(H, D) * C + 2 * C * H * D) * 2);
}

// strides (b, o, h, n) of a [H][B*N*N][D] plane set and of a [B*N*N][ld] row matrix (head h at column h * D)
static void plane_strides(int64_t* s, const PairAttnCall& t) {
  const int64_t N = t.N, D = t.D;
  s[0] = N * N * D;
  s[1] = t.ending ? D : N * D;
  s[2] = t.B * N * N * D;
  s[3] = t.ending ? N * D : D;
}
static void row_strides(int64_t* s, const PairAttnCall& t, int64_t ld) {
  s[0] = t.N * t.N * ld;
  s[1] = t.ending ? ld : t.N * ld;
  s[2] = t.D;
  s[3] = t.ending ? t.N * ld : ld;
}

static AttnCall attn_of(const PairAttnCall& t) {
  AttnCall a = {};
  const int64_t plane = t.B * t.N * t.N * t.D;
  const bf16* base = reinterpret_cast<const bf16*>(t.qkvg);
  a.B = t.B; a.O = t.N; a.H = t.H; a.N = t.N; a.D = t.D; a.G = t.B;
  a.scale = 1.f / sqrtf((float)t.D);
  a.q = base;
  a.k = base + t.H * plane;
  a.v = base + 2 * t.H * plane;
  for (int64_t* s : {a.qs, a.ks, a.vs, a.gs}) plane_strides(s, t);
  a.gate = base + 3 * t.H * plane;
  a.mask = t.mask_add;
  a.mask_pitch = (t.N + 3) / 4 * 4;
  a.bias = t.bias;
  a.bias_pitch = (t.N + 7) / 8 * 8;
  a.out = t.og;
  row_strides(a.os, t, t.H * t.D);
  a.lse = t.lse;
  return a;
}

static int pair_attn_status(int** status) {
  static PerDeviceAddress cache;
  return device_symbol_address(g_pair_attn_status, cache, reinterpret_cast<void**>(status));
}

template <int C>
static int out_proj(const PairAttnCall& t, const AttnPacked& pk, int* status, cudaStream_t stream) {
  const int64_t R = t.B * t.N * t.N, HD = t.H * t.D;
  using Cfg = GemmCfg<128, C, 128, false, 128, false, 4, (C > 64 ? 16 : 8)>;
  GemmShape sh{(int)R, C, (int)HD, 1, 0};
  EpiResidual::Params ep{(bf16*)t.out, (const bf16*)t.z, PairRows::make(t.N, t.N, false), C};
  return launch_gemm<Cfg, EpiResidual>(t.og, HD, 0, pk.Wo, HD, 0, sh, ep, status, stream);
}

template <int C>
static int layer_norm(const PairAttnCall& t, cudaStream_t stream) {
  const int64_t R = t.B * t.N * t.N;
  launch_kernel(ln_fwd_kernel<C, false>, dim3(ln_fwd_blocks<C>(R)), dim3(256), 0, stream, (const bf16*)t.z, t.w.ln_w,
                t.w.ln_b, (bf16*)t.x, t.mean, t.rstd, PairRows::make(t.N, t.N, false), PairMask{}, (float*)nullptr, R);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

static int check_pair_attn(const PairAttnCall& t) {
  TPF_REQUIRE(pair_attn_supported(t.C, t.H, t.D), TPF_ERR_UNSUPPORTED, "pair attention: C=%lld, H=%lld, D=%lld",
              (long long)t.C, (long long)t.H, (long long)t.D);
  TPF_REQUIRE(t.B > 0 && t.N > 0 && t.B * t.N * t.N < (1ll << 31), TPF_ERR_INVALID_ARGUMENT,
              "pair attention: B*N*N out of range");
  return TPF_OK;
}

int pair_attn_forward(const PairAttnCall& t, cudaStream_t stream) {
  int rc = check_pair_attn(t);
  if (rc) return rc;
  int* status = nullptr;
  if ((rc = pair_attn_status(&status))) return rc;
  const int64_t C = t.C, HD = t.H * t.D, P = proj_cols(t.H, t.D), R = t.B * t.N * t.N;
  const AttnPacked pk = attn_packed_at(t.packed, C, t.H, t.D);
  launch_kernel(pair_attn_pack_kernel, dim3((unsigned)((P * C + C * HD + 255) / 256)), dim3(256), 0, stream, t.w, pk,
                (int)C, (int)HD, (int)t.H, (int)P);
  TPF_LAUNCH_OK();
  {
    // additive mask inf * (mask - 1), [B, O, N] of the attention's orientation
    PrepSource none{}, m{t.mask, t.mask_type, {t.mask_stride[0], t.mask_stride[1], t.mask_stride[2], 0}};
    if (t.ending) {
      m.stride[1] = t.mask_stride[2];
      m.stride[2] = t.mask_stride[1];
    }
    rc = attn_prep(none, 0, 0, nullptr, 8, m, t.B, t.N, t.mask_add, (t.N + 3) / 4 * 4, t.N, stream, -1.f, t.inf);
    if (rc) return rc;
  }
  switch (C) {
    case 32: rc = layer_norm<32>(t, stream); break;
    case 64: rc = layer_norm<64>(t, stream); break;
    case 96: rc = layer_norm<96>(t, stream); break;
    default: rc = layer_norm<128>(t, stream);
  }
  if (rc) return rc;
  {
    int log_d = 0;
    while ((1 << log_d) < t.D) ++log_d;
    EpiQkvg::Params ep{{}, (bf16*)t.qkvg, R * t.D, log_d, (int)t.D, (int)(4 * HD), (bf16*)t.bias, (int)t.H, (int)t.N,
                       (t.N + 7) / 8 * 8, PairRows::make(t.N, t.N, false)};
    if (t.D == 32 && (rc = make_store_tmap(&ep.map, t.qkvg, t.D, R, t.D, 4 * t.H, R * t.D))) return rc;
    GemmShape sh{(int)R, (int)P, (int)C, 1, 0};
    // 4 HD + H columns in as few, as full tiles as possible: 3 x 192 at H * D = 128, 3 x 96 at 64.  The weights, or as
    // much of them as a tile needs, stay in shared memory while the rows stream past (see GemmCfg).  All of them at
    // H * D = 128 from 99 row tiles on: 13.4 -> 12.3 us at N = 192, 39.3 -> 34.9 at 384, 691 -> 482 at 1536, but
    // 6.2 -> 7.9 at 72.  At H * D = 64 no variant with all weights resident is built; it would pay there as well (measured
    // with 2 x 192 columns, C = 64: 32.2 -> 25.0 us at N = 384, 443 -> 326 at 1536).
    if (P > 272 && P <= 544 && resident_pays(R, 3)) {
      using Cfg = GemmCfg<128, 192, 128, false, 128, false, 3, 8, 3, 2, 544>;
      rc = launch_gemm<Cfg, EpiQkvg>(t.x, C, 0, pk.W, C, 0, sh, ep, status, stream);
    } else if (HD <= 64) {
      using Cfg = GemmCfg<128, 96, 128, false, 128, false, 4, 8, 2, 2>;
      rc = launch_gemm<Cfg, EpiQkvg>(t.x, C, 0, pk.W, C, 0, sh, ep, status, stream);
    } else {
      using Cfg = GemmCfg<128, 192, 128, false, 128, false, 4, 8, 2, 2>;
      rc = launch_gemm<Cfg, EpiQkvg>(t.x, C, 0, pk.W, C, 0, sh, ep, status, stream);
    }
    if (rc) return rc;
  }
  if ((rc = attn_forward(attn_of(t), stream))) return rc;
  switch (C) {
    case 32: return out_proj<32>(t, pk, status, stream);
    case 64: return out_proj<64>(t, pk, status, stream);
    case 96: return out_proj<96>(t, pk, status, stream);
    default: return out_proj<128>(t, pk, status, stream);
  }
}

struct PairAttnBwdWorkspace {
  bf16 *d_o, *d_rows, *d_x;
  float *delta, *part_w, *part_wo, *part_ln;
  char* attn;        // scratch of the attention backward kernels (the two use it one after the other)
  int64_t attn_qkv, attn_bias;
  int splits_w, splits_wo, rows_per_block, blocks_ln;
  int64_t kps_w, kps_wo, total;
};

static void split_rows(int64_t R, int64_t tiles, int* n, int64_t* kps) {
  int64_t s = sm_count() / tiles;
  if (s < 1) s = 1;
  *kps = ((R + s - 1) / s + 63) / 64 * 64;
  *n = (int)((R + *kps - 1) / *kps);
}

static void plan_pair_attn_bwd(int64_t B, int64_t N, int64_t C, int64_t H, int64_t D, char* base,
                               PairAttnBwdWorkspace* w) {
  const int64_t R = B * N * N, HD = H * D, P = proj_cols(H, D);
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    char* p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  w->d_o = (bf16*)take(R * HD * 2);
  w->d_rows = (bf16*)take(R * P * 2);
  w->d_x = (bf16*)take(R * C * 2);
  w->delta = (float*)take(R * H * 4);
  split_rows(R, (P + 127) / 128, &w->splits_w, &w->kps_w);
  split_rows(R, (HD + 127) / 128, &w->splits_wo, &w->kps_wo);
  w->part_w = (float*)take(w->splits_w * P * C * 4);
  w->part_wo = (float*)take(w->splits_wo * C * HD * 4);
  w->rows_per_block = ln_bwd_rows_per_block(R);
  w->blocks_ln = (int)((R + w->rows_per_block - 1) / w->rows_per_block);
  w->part_ln = (float*)take((int64_t)w->blocks_ln * 2 * C * 4);
  w->attn_qkv = attn_bwd_workspace_bytes(B, N, H, N, D);
  w->attn_bias = attn_dbias_rows_workspace_bytes(B, N, H, N, B);
  w->attn = take(w->attn_qkv > w->attn_bias ? w->attn_qkv : w->attn_bias);
  w->total = off;
}

int64_t pair_attn_bwd_workspace_bytes(int64_t B, int64_t N, int64_t C, int64_t H, int64_t D) {
  PairAttnBwdWorkspace w;
  plan_pair_attn_bwd(B, N, C, H, D, nullptr, &w);
  return w.total;
}

template <int D>
static int gate_bwd(const PairAttnCall& t, const void* d_out, const PairAttnBwdWorkspace& w, const AttnPacked& pk,
                    int* status, cudaStream_t stream) {
  const int64_t R = t.B * t.N * t.N, HD = t.H * D, P = proj_cols(t.H, D);
  // the epilogue keeps gate logits and gated outputs of the next tile in flight: one 32-column chunk per warp (see the
  // output projection of the multiplicative update)
  using Cfg = GemmCfg<128, 64, 128, false, 128, false, 4>;
  using Epi = EpiGateBwd<D>;
  typename Epi::Params ep{{}, {}, (const bf16*)t.qkvg + 3 * t.H * R * D, (const bf16*)t.og, w.d_o, R * D, w.d_rows + 3 * HD, P,
                          w.delta, t.ending, (int)t.H, (int)t.N, (int)HD, PairRows::make(t.N, t.N, false)};
  int rc = D == 32 ? make_store_tmap(&ep.map_o, w.d_o, D, R, D, t.H, R * D) : TPF_OK;
  if (rc || (rc = make_store_tmap(&ep.map_g, w.d_rows + 3 * HD, HD, R, P, 1, 0))) return rc;
  GemmShape sh{(int)R, (int)HD, (int)t.C, 1, 0};
  return launch_gemm<Cfg, Epi>(d_out, t.C, 0, pk.WoT, t.C, 0, sh, ep, status, stream);
}

template <int C>
static int norm_bwd(const PairAttnCall& t, const PairAttnGrads& g, const PairAttnBwdWorkspace& w, const AttnPacked& pk,
                    int* status, cudaStream_t stream) {
  const int64_t R = t.B * t.N * t.N, P = proj_cols(t.H, t.D);
  {
    using Cfg = GemmCfg<128, C, 128, false, 128, false, 6>;
    using Epi = EpiStore<bf16>;
    GemmShape sh{(int)R, C, (int)P, 1, 0};
    typename Epi::Params ep;
    if (int rc = epi_store_params<bf16>(&ep, w.d_x, C, 0, sh)) return rc;
    if (int rc = launch_gemm<Cfg, Epi>(w.d_rows, P, 0, pk.WT, P, 0, sh, ep, status, stream)) return rc;
  }
  launch_kernel(ln_bwd_kernel<C>, dim3(w.blocks_ln), dim3(256), 0, stream, (const bf16*)w.d_x, (const bf16*)t.z,
                t.w.ln_w, (const float*)t.mean, (const float*)t.rstd, (bf16*)g.d_z, w.part_ln,
                PairRows::make(t.N, t.N, false), (const bf16*)g.d_out, R, w.rows_per_block);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

int pair_attn_backward(const PairAttnCall& t, const PairAttnGrads& g, void* workspace, int64_t workspace_bytes,
                       cudaStream_t stream) {
  int rc = check_pair_attn(t);
  if (rc) return rc;
  int* status = nullptr;
  if ((rc = pair_attn_status(&status))) return rc;
  const int64_t B = t.B, N = t.N, C = t.C, H = t.H, D = t.D, HD = H * D, P = proj_cols(H, D), R = B * N * N;
  PairAttnBwdWorkspace w;
  plan_pair_attn_bwd(B, N, C, H, D, (char*)workspace, &w);
  TPF_REQUIRE(workspace && workspace_bytes >= w.total && (reinterpret_cast<uintptr_t>(workspace) & 255) == 0,
              TPF_ERR_WORKSPACE, "pair attention backward: workspace too small or misaligned");
  const AttnPacked pk = attn_packed_at(t.packed, C, H, D);
  FoldList folds;
  // 1. d_og = d_out Wo -> d_o, d_g, delta
  rc = D == 16 ? gate_bwd<16>(t, g.d_out, w, pk, status, stream) : gate_bwd<32>(t, g.d_out, w, pk, status, stream);
  if (rc) return rc;
  // 2. d_wo = d_out^T og
  rc = bmm_bf16(g.d_out, C, 0, 1, t.og, HD, 0, 1, w.part_wo, HD, C * HD, 1, C, HD, R, w.splits_wo, w.kps_wo, 128, stream);
  if (rc) return rc;
  folds.add(w.part_wo, w.splits_wo, (int)(C * HD), (int)(C * HD), g.w_o);
  // 3. attention backward -> columns of the row matrix
  AttnCall a = attn_of(t);
  a.d_out = w.d_o;
  plane_strides(a.dos, t);
  a.delta = w.delta;
  a.dq = w.d_rows;
  a.dk = w.d_rows + HD;
  a.dv = w.d_rows + 2 * HD;
  row_strides(a.ds, t, P);
  a.dbias_rows = w.d_rows + 4 * HD;
  a.dbias_ld = P;
  if ((rc = attn_backward_qkv(a, w.attn, w.attn_qkv, stream))) return rc;
  if ((rc = attn_backward_bias(a, w.attn, w.attn_bias, stream))) return rc;
  // 4. d_x = d_rows W, norm backward (adds the residual path's gradient)
  switch (C) {
    case 32: rc = norm_bwd<32>(t, g, w, pk, status, stream); break;
    case 64: rc = norm_bwd<64>(t, g, w, pk, status, stream); break;
    case 96: rc = norm_bwd<96>(t, g, w, pk, status, stream); break;
    default: rc = norm_bwd<128>(t, g, w, pk, status, stream);
  }
  if (rc) return rc;
  folds.add(w.part_ln, w.blocks_ln, (int)(2 * C), (int)C, g.ln_w, g.ln_b);
  // 5. weight gradients of the joint projection: d_rows^T x
  rc = bmm_bf16(w.d_rows, P, 0, 1, t.x, C, 0, 1, w.part_w, C, P * C, 1, P, C, R, w.splits_w, w.kps_w, 128, stream);
  if (rc) return rc;
  folds.add(w.part_w, w.splits_w, (int)(P * C), (int)(HD * C), g.w_q, g.w_k, g.w_v, g.w_g, g.w_z, (int)((4 * HD + H) * C));
  return folds.launch(stream);
}

}  // namespace tpf
