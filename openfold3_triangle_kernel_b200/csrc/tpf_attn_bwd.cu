// Triangle-attention backward for sm_100a: dQ, dK, dV (this file, kernel 1), the row
// scalar delta (kernel 0) and dBias (kernel 2 + fold).
//
// Reference interface replaced: turbopairformer_triangle_delta_out and
// turbopairformer_triangle_sr_backward_out
// (openfold3/core/kernels/turbopairformer/turbopairformer_triangle_delta.cu:343-414,
//  openfold3/core/kernels/turbopairformer/turbopairformer_triangle_dq_dbias.cu:2526-2648).
// Same math: P = exp(S - lse) (0 where lse < -2^24, -inf among it: no key is kept), dP = dO V^T, dS = P (dP - delta),
// dV = P^T dO, dK = scale dS^T Q, dQ = scale dS K, dBias = sum over outer rows of dS; P and dS
// are rounded to bf16 only as UMMA operands, all accumulation is fp32, no atomics anywhere.
//
// Machine mapping (differs from the reference, which keeps 64-key leaves and writes bf16
// dQ partials and dBias leaf planes to HBM):
//  * kernel 1 owns whole (b, o, h) planes.  For each 128x128 (query, key) tile the five GEMMs
//    run on tcgen05; dK/dV of up to KS key tiles and dQ of the current query tile stay in
//    TMEM until complete, so for N <= 128*KS nothing but the final gradients is written.
//    Longer sequences walk key strips and keep a per-CTA fp32 dQ running sum in a small
//    private scratch (same thread, fixed order).
//  * kernel 2 owns a (h, query tile, key tile) of dBias and walks the outer rows, recomputing
//    S and dP (two cheap K = D GEMMs) and summing dS in fp32 registers in ascending o.
//    A few independent o-chunks per tile fill the machine; their partial planes are folded
//    in fixed order by a tiny kernel.
#include <math.h>
#include <stdlib.h>

#include "tpf_host.cuh"
#include "tpf_internal.h"
#include "tpf_ptx.cuh"

namespace tpf {

static __device__ int g_attn_bwd_status;

int attn_bwd_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  TPF_CUDA_OK(cudaMemcpyFromSymbol(&v, g_attn_bwd_status, sizeof(int)));
  if (v) TPF_CUDA_OK(cudaMemcpyToSymbol(g_attn_bwd_status, &zero, sizeof(int)));
  *out = v;
  return TPF_OK;
}

static int attn_bwd_status_address(int** out) {
  static PerDeviceAddress cache;
  return device_symbol_address(g_attn_bwd_status, cache, reinterpret_cast<void**>(out));
}

// =============================================================================================
// kernel 0: delta[b,o,h,q] = sum_d dO[b,o,q,h,d] * O[b,o,q,h,d]      (HBM bound)
// =============================================================================================
template <int D>
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ d_out,
                                                         const __nv_bfloat16* __restrict__ out,
                                                         float* __restrict__ delta, int64_t rows, int H, int N) {
  griddep_wait();
  // one thread handles D/8 ... : LANES threads per (b,o,q,h) row of D elements, 8 elements each
  constexpr int LANES = D / 8;
  const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t r = gid / LANES;  // flat (b,o,q,h)
  const int part = (int)(gid % LANES);
  float acc = 0.f;
  if (r < rows) {
    const uint4 a = *reinterpret_cast<const uint4*>(d_out + r * D + part * 8);
    const uint4 b = *reinterpret_cast<const uint4*>(out + r * D + part * 8);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc = fmaf(__uint_as_float(aw[i] << 16), __uint_as_float(bw[i] << 16), acc);
      acc = fmaf(__uint_as_float(aw[i] & 0xFFFF0000u), __uint_as_float(bw[i] & 0xFFFF0000u), acc);
    }
  }
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (r < rows && part == 0) {
    const int h = (int)(r % H);
    const int64_t t = r / H;
    const int q = (int)(t % N);
    const int64_t bo = t / N;
    delta[(bo * H + h) * N + q] = acc;
  }
}

// =============================================================================================
// kernel 1: dQ, dK, dV
// =============================================================================================
struct AttnBwdParams {
  __nv_bfloat16 *dq, *dk, *dv;
  int64_t gb, go, gh, gn;       // their element strides
  const float* lse;             // [B,O,H,N]
  const float* delta;           // [B,O,H,N]
  const float* mask;            // [B,O,mask_pitch]
  int64_t mask_pitch;
  float* dq_scratch;            // per-CTA [N][D] fp32 when the key axis needs several strips
  int B, O, H, N;
  int q_tiles, k_tiles, n_strips;
  int bias_broadcast;
  float scale;
  float logit_scale;            // scale, kept away from zero: what the added operands are divided by
  int n_items;
  FastDiv div_h, div_o;
};

// Numbers that are added to every logit of a row or of a column enter S and dP by one more UMMA of K = 16: an fp32 value is
// three bf16 parts in three K columns (24 bits, as many as fp32 has), met by ones on the other side.  A tile of such rows has
// 32 bytes per row, as a D = 16 operand tile; rows hold their values in the first 16 bytes, the second half is zero.
struct Bf16x3 {
  uint32_t hi, mid, lo;  // bf16 bits
};
__device__ __forceinline__ Bf16x3 split_bf16x3(float x) {
  const float hi = __bfloat162float(__float2bfloat16_rn(x));
  const float r = hi - hi != 0.f ? 0.f : x - hi;  // infinity or NaN: one part carries it
  const float mid = __bfloat162float(__float2bfloat16_rn(r));
  return {__float_as_uint(hi) >> 16, __float_as_uint(mid) >> 16, pack_bf16x2(r - mid, 0.f)};
}
__device__ __forceinline__ void store_added(uint8_t* tile, int row, uint4 v) {
  *reinterpret_cast<uint4*>(tile + row * 32 + ((row >> 2) & 1) * 16) = v;  // (the 32-byte swizzle)
}
constexpr uint32_t kOnesBf16x2 = 0x3F803F80u;
// A row whose log-sum-exp is below -2^24 has masked keys only (by -inf or by a large finite value such as -1e9).  fp32 numbers are
// two or more apart there, so what its logits and its log-sum-exp differ by is rounding, and exp of that is any number
// (probabilities of 3e5 under a mask of -1e9, of 3.6 under -1e8).  It gets no gradient.
constexpr float kMaskedLse = -16777216.f;

template <int D_>
struct AttnBwdCfg {
  static constexpr int D = D_;
  static constexpr int KS = D <= 32 ? 3 : 1;   // key tiles whose dK/dV stay in TMEM together
  // With one key tile per strip K and V stay for the strip; else they are loaded for every tile, and K, which dQ reads last,
  // three tiles deep (with two the loads of the next tile came late: 800 cycles of a tile of 3250).
  static constexpr bool KV_STAYS = KS == 1;
  static constexpr int NK = KV_STAYS ? 2 : 3, NV = 2, NQ = 2;
  static constexpr int NB = D <= 32 ? 2 : 1;   // bias stages
  static constexpr int NCW = 16;               // compute warps: two groups of eight, 64 queries each
  static constexpr int THREADS = 32 * (NCW + 7);
  static constexpr int WARP_TMA = NCW, WARP_MMA = NCW + 1, WARP_ADD = NCW + 2;  // then four that store finished gradients
  static constexpr int SWZ = 2 * D;
  static constexpr int TILE = 128 * D * 2;
  static constexpr int ADD_TILE = 128 * 32;
  static constexpr int BIAS_STAGE = 32768, DS_BYTES = 32768;
  static constexpr int OFF_BIAS = 0;
  static constexpr int OFF_DS = OFF_BIAS + NB * BIAS_STAGE;
  static constexpr int OFF_Q = OFF_DS + DS_BYTES;        // [NQ]
  static constexpr int OFF_DO = OFF_Q + NQ * TILE;       // [NQ]
  static constexpr int OFF_K = OFF_DO + NQ * TILE;       // [NK]
  static constexpr int OFF_V = OFF_K + NK * TILE;        // [NV]
  // added operands: -lse and a row of ones with Q, -delta with dO, ones and the mask (with V's stages), ones with V
  static constexpr int OFF_QADD = OFF_V + NV * TILE;         // [NQ]
  static constexpr int OFF_DOADD = OFF_QADD + NQ * ADD_TILE;  // [NQ]
  static constexpr int OFF_KADD = OFF_DOADD + NQ * ADD_TILE;  // [NV]
  static constexpr int OFF_VADD = OFF_KADD + NV * ADD_TILE;
  static constexpr int ADD_BYTES = (2 * NQ + NV + 1) * ADD_TILE;
  // D <= 32: per storing warp two 32-row blocks of a finished tile on their way out (at D = 64 there is no room)
  static constexpr bool STAGED = D <= 32;
  static constexpr int STG_BYTES = 32 * D * 2;
  static constexpr int OFF_STG = OFF_VADD + ADD_TILE;
  static constexpr int OFF_BAR = OFF_STG + (STAGED ? 8 * STG_BYTES : 0);
  static constexpr int N_BAR = 2 * NB + 2 * NQ + 2 * NK + 2 * NV + 8 + 2 * KS;
  static constexpr int SMEM_BYTES = OFF_BAR + N_BAR * 8 + 16 + 1024;
  // S^T and dP^T of the two groups (64 queries each); P^T and dS^T, bf16, take their place
  static constexpr int TM_S = 0, TM_DP = 128, TM_DQ = 256, TM_DK = 320, TM_DV = 320 + KS * D;
  static constexpr int TMEM_COLS = 512;
  static_assert(TM_DV + KS * D <= 512, "TMEM budget");
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

// Walks the (item, strip, query tile, key tile) sequence of one CTA.
struct BwdWalk {
  int n_items, q_tiles, k_tiles, KS, n_strips, step;
  int item, strip, qt, kk;
  __device__ void init(int first, int step_, int n_items_, int q_tiles_, int k_tiles_, int KS_, int n_strips_) {
    n_items = n_items_; q_tiles = q_tiles_; k_tiles = k_tiles_; KS = KS_; n_strips = n_strips_; step = step_;
    item = first; strip = 0; qt = 0; kk = 0;
  }
  __device__ bool valid() const { return item < n_items; }
  __device__ int strip_len() const { return min(KS, k_tiles - strip * KS); }
  __device__ int kt() const { return strip * KS + kk; }
  __device__ bool first_kk() const { return kk == 0; }
  __device__ bool last_kk() const { return kk == strip_len() - 1; }
  __device__ bool first_qt() const { return qt == 0; }
  __device__ bool last_qt() const { return qt == q_tiles - 1; }
  __device__ void next() {
    if (++kk < strip_len()) return;
    kk = 0;
    if (++qt < q_tiles) return;
    qt = 0;
    if (++strip < n_strips) return;
    strip = 0;
    item += step;
  }
};

// S and dP are computed transposed (S^T = K Q^T, TMEM lane = key, column = query), so that bf16 P^T and dS^T, written over them,
// are the A operands of dV += P^T dO and dK += dS^T Q straight from TMEM; only dS goes through shared memory, for dQ += dS K.
// The log-sum-exp, the mask and delta are in S and dP already (see Bf16x3): what is left per logit is the bias, an ex2 and a
// product.
// The sixteen compute warps are two groups, each with the 64 queries of one half of a 128 x 128 tile and S / dP columns of its
// own: while one group's UMMAs run, the other one computes.  A thread has the 32 queries of one key.
//
// What bounds it: the chain of a half tile, 1200 cycles of arithmetic and 1000 between P being written and the next S being
// there (hand-shakes, 14 UMMAs, completion), of which the other group hides most; the ex2 pipe alone needs 1024 cycles a tile.
// Before, with a thread per query row, P and dS went through shared memory for three products of 128 x 128 tiles, whose operand
// traffic kept it busy for 2400 cycles a tile, and one S / dP pair left all warps waiting together.  Measured, H = 4, us:
// N = 384, D = 32 188 -> 133; N = 768 1523 -> 1010; N = 257, D = 64 233 -> 156; N = 128, D = 16, B = 4 35.4 -> 30.4.
// Waiting for S and dP apart was slower (136 us at N = 384), so was a warp of its own for dQ's UMMAs (137).
//
// TAIL: the last tile has rows beyond the last key.  They are zeros, and an infinite query times zero is a NaN, which the added -inf
// does not mask; their dS is written over with zeros, so that dQ of a query whose logits are all -inf is zero, as at any other
// length.  (dK and dV of such rows are not stored.)  Without -> with that, us: N = 400 250 -> 252,
// N = 517 455 -> 457, N = 510 320 -> 319; as a select of the registers in one kernel for every length N = 384 140 -> 144, N = 517 474.
//
// RAGGED: a warp whose rows or keys of a tile all lie beyond the last one only keeps the barriers going, and the UMMAs leave its
// part of their K extent out; the others have the pipes to themselves.
template <class Cfg, bool TAIL, bool RAGGED>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                const __grid_constant__ CUtensorMap tmBias, const __grid_constant__ CUtensorMap tmDQ,
                const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDV, const AttnBwdParams p, int* __restrict__ status) {
  griddep_wait();
  constexpr int D = Cfg::D, KS = Cfg::KS, NK = Cfg::NK, NV = Cfg::NV, NQ = Cfg::NQ, NB = Cfg::NB, NCW = Cfg::NCW;
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* b_full = bars;
  uint64_t* b_empty = b_full + NB;
  uint64_t* q_full = b_empty + NB;
  uint64_t* q_empty = q_full + NQ;
  uint64_t* k_full = q_empty + NQ;
  uint64_t* k_empty = k_full + NK;
  uint64_t* v_full = k_empty + NK;  // V and the added operand of the keys
  uint64_t* v_empty = v_full + NV;
  uint64_t* misc = v_empty + NV;
  uint64_t* sdp_full = misc + 0;   // [2] S and dP of a group's half tile are in TMEM
  uint64_t* pds_ready = misc + 2;  // [2] ... and P and dS have taken their place
  uint64_t* ds_ready = misc + 4;   // dS of a tile is in shared memory
  uint64_t* ds_free = misc + 5;    // ... and has been consumed; so have P and dS in TMEM
  uint64_t* dq_full = misc + 6;    // dQ of a query tile is complete
  uint64_t* dq_free = misc + 7;    // ... and has been read
  uint64_t* dkv_full = misc + 8;   // [KS] dK and dV of a key tile are complete
  uint64_t* dkv_free = dkv_full + KS;  // ... and have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::N_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wctx{abort_flag, status};

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NB; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], NCW);
    }
    for (int s = 0; s < NQ; ++s) {
      mbar_init(&q_full[s], 2);  // the copies, the added operands
      mbar_init(&q_empty[s], 1);
    }
    for (int s = 0; s < NK; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < NV; ++s) {
      mbar_init(&v_full[s], 2);
      mbar_init(&v_empty[s], 1);
    }
    for (int g = 0; g < 2; ++g) {
      mbar_init(&sdp_full[g], 1);
      mbar_init(&pds_ready[g], NCW / 2);
    }
    mbar_init(ds_ready, NCW);
    mbar_init(ds_free, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_free, 4);
    for (int s = 0; s < KS; ++s) {
      mbar_init(&dkv_full[s], 1);
      mbar_init(&dkv_free[s], 8);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
    tma_prefetch_desc(&tmBias);
  }
  for (int i = threadIdx.x; i < Cfg::ADD_BYTES / 4; i += blockDim.x)
    reinterpret_cast<uint32_t*>(smem + Cfg::OFF_QADD)[i] = i >= (Cfg::OFF_VADD - Cfg::OFF_QADD) / 4 ? kOnesBf16x2 : 0u;
  fence_async_smem();
  if (warp == Cfg::WARP_MMA) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  auto decode = [&](int item, int& b, int& o, int& h) {
    const int r = (int)p.div_h.div((uint32_t)item);
    h = item - r * p.H;
    b = (int)p.div_o.div((uint32_t)r);
    o = r - b * p.O;
  };

  if (warp == Cfg::WARP_TMA) {
    // ------------------------------------------------------------------ TMA producer
    const uint32_t el = elect_one();
    int q_s = 0, k_s = 0, v_s = 0, b_s = 0;
    uint32_t q_ph = 1, k_ph = 1, v_ph = 1, b_ph = 1;
    int b = 0, o = 0, h = 0, cur = -1;
    BwdWalk w;
    for (w.init(blockIdx.x, gridDim.x, p.n_items, p.q_tiles, p.k_tiles, KS, p.n_strips); w.valid(); w.next()) {
      if (w.item != cur) {
        cur = w.item;
        decode(cur, b, o, h);
      }
      if (w.first_kk()) {
        warp_wait(&q_empty[q_s], q_ph, wctx);
        mbar_expect_tx(el, &q_full[q_s], 2 * Cfg::TILE);
        tma_load_5d(el, smem + Cfg::OFF_Q + q_s * Cfg::TILE, &tmQ, &q_full[q_s], 0, w.qt * 128, h, o, b);
        tma_load_5d(el, smem + Cfg::OFF_DO + q_s * Cfg::TILE, &tmDO, &q_full[q_s], 0, w.qt * 128, h, o, b);
        if (++q_s == NQ) {
          q_s = 0;
          q_ph ^= 1;
        }
      }
      const int kt = w.kt();
      if (!Cfg::KV_STAYS || w.first_qt()) {
        warp_wait2(&v_empty[v_s], v_ph, &k_empty[k_s], k_ph, wctx);
        mbar_expect_tx(el, &v_full[v_s], Cfg::TILE);
        tma_load_5d(el, smem + Cfg::OFF_V + v_s * Cfg::TILE, &tmV, &v_full[v_s], 0, kt * 128, h, o, b);
        mbar_expect_tx(el, &k_full[k_s], Cfg::TILE);
        tma_load_5d(el, smem + Cfg::OFF_K + k_s * Cfg::TILE, &tmK, &k_full[k_s], 0, kt * 128, h, o, b);
        if (++v_s == NV) {
          v_s = 0;
          v_ph ^= 1;
        }
        if (++k_s == NK) {
          k_s = 0;
          k_ph ^= 1;
        }
      }
      warp_wait(&b_empty[b_s], b_ph, wctx);
      mbar_expect_tx(el, &b_full[b_s], Cfg::BIAS_STAGE);
      tma_load_4d(el, smem + Cfg::OFF_BIAS + b_s * Cfg::BIAS_STAGE, &tmBias, &b_full[b_s], kt * 128, w.qt * 128, h,
                  p.bias_broadcast ? 0 : b);
      if (++b_s == NB) {
        b_s = 0;
        b_ph ^= 1;
      }
    }
  } else if (warp == Cfg::WARP_ADD) {
    // ------------------------------------------------------------------ the added operands
    // (By the loading warp between its copies they made the loads late.  Kernel, us: N = 128, D = 16, B = 4 33.9 -> 30.4,
    // N = 257, D = 64 162 -> 156; N = 384 and 768, D = 32 no change.)
    int q_s = 0, v_s = 0;
    uint32_t q_ph = 1, v_ph = 1;
    BwdWalk w;
    w.init(blockIdx.x, gridDim.x, p.n_items, p.q_tiles, p.k_tiles, KS, p.n_strips);
    const float inv = 1.f / p.logit_scale;
    const float no_row = copysignf(1e30f, -p.logit_scale);  // makes exp2 zero, and no NaN with masked keys
    // The next step's values are requested before this step's waits.
    struct Step {
      float4 mask;
      float l[4], d[4];
    } cur, nxt;
    auto request = [&](const BwdWalk& at, Step& s) {
      const int k0 = at.kt() * 128 + 4 * lane;
      if (k0 < p.N && (!Cfg::KV_STAYS || at.first_qt())) {
        const float* m = p.mask + (int64_t)p.div_h.div((uint32_t)at.item) * p.mask_pitch + k0;
        if (k0 + 3 < p.N) s.mask = __ldg(reinterpret_cast<const float4*>(m));
        else s.mask = make_float4(__ldg(m), k0 + 1 < p.N ? __ldg(m + 1) : 0.f, k0 + 2 < p.N ? __ldg(m + 2) : 0.f, 0.f);
      }
      if (at.first_kk()) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int q = at.qt * 128 + 32 * i + lane;
          if (q < p.N) {
            const int64_t idx = (int64_t)at.item * p.N + q;  // items are numbered as their planes lie in memory
            s.l[i] = __ldg(p.lse + idx);
            s.d[i] = __ldg(p.delta + idx);
          }
        }
      }
    };
    cur.mask = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) cur.l[i] = cur.d[i] = 0.f;
    if (w.valid()) request(w, cur);
    nxt = cur;
    BwdWalk next = w;
    while (w.valid()) {
      next.next();
      if (next.valid()) request(next, nxt);
      if (w.first_kk()) {
        warp_wait(&q_empty[q_s], q_ph, wctx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = 32 * i + lane;
          const bool ok = w.qt * 128 + row < p.N;
          const Bf16x3 l = split_bf16x3(ok && !(cur.l[i] < kMaskedLse) ? -cur.l[i] * inv : no_row);
          const Bf16x3 d = split_bf16x3(ok ? -cur.d[i] : 0.f);
          store_added(smem + Cfg::OFF_QADD + q_s * Cfg::ADD_TILE, row,
                      make_uint4(l.hi | l.mid << 16, l.lo | 0x3F800000u, kOnesBf16x2, 0u));
          store_added(smem + Cfg::OFF_DOADD + q_s * Cfg::ADD_TILE, row, make_uint4(d.hi | d.mid << 16, d.lo, 0u, 0u));
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full[q_s]);
        if (++q_s == NQ) {
          q_s = 0;
          q_ph ^= 1;
        }
      }
      if (!Cfg::KV_STAYS || w.first_qt()) {
        const int kt = w.kt();
        warp_wait(&v_empty[v_s], v_ph, wctx);
        const float mv[4] = {cur.mask.x, cur.mask.y, cur.mask.z, cur.mask.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int key = 4 * lane + i;
          const Bf16x3 m = split_bf16x3(kt * 128 + key < p.N ? mv[i] * inv : copysignf(INFINITY, -p.logit_scale));
          store_added(smem + Cfg::OFF_KADD + v_s * Cfg::ADD_TILE, key,
                      make_uint4(kOnesBf16x2, 0x3F80u | m.hi << 16, m.mid | m.lo << 16, 0u));
        }
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&v_full[v_s]);
        if (++v_s == NV) {
          v_s = 0;
          v_ph ^= 1;
        }
      }
      w = next;
      cur = nxt;
    }
  } else if (warp == Cfg::WARP_MMA) {
    // ------------------------------------------------------------------ UMMA issuer
    const uint32_t el = elect_one();
    constexpr uint32_t idesc_sd = make_idesc_bf16(128, 64, false, false);  // S^T, dP^T
    constexpr uint32_t idesc_kv = make_idesc_bf16(128, D, false, true);    // dV, dK
    constexpr uint32_t idesc_dq = make_idesc_bf16(128, D, true, true);     // dQ
    constexpr uint32_t swz = swizzle_mode_for_bytes(Cfg::SWZ);
    // Lower descriptor words of stage 0 of every operand; a stage, a half or a k-step only changes the start-address
    // field (bits 0-13, 16-byte units).
    constexpr uint32_t hi = smem_desc_hi(8 * Cfg::SWZ, swz);                       // q, k, v, dO tiles, K-major and MN-major
    constexpr uint32_t hi_ds = smem_desc_hi(1024, swizzle_mode_for_bytes(128));
    constexpr uint32_t hi_add = smem_desc_hi(256, swizzle_mode_for_bytes(32));
    constexpr uint32_t kMn = (128 * Cfg::SWZ - 16) >> 4 << 16;                     // from a tile's K-major word to its MN-major one
    const uint32_t d_q = smem_desc_lo(smem_u32(smem + Cfg::OFF_Q), 16);
    const uint32_t d_k = smem_desc_lo(smem_u32(smem + Cfg::OFF_K), 16);
    const uint32_t d_do = smem_desc_lo(smem_u32(smem + Cfg::OFF_DO), 16);
    const uint32_t d_v = smem_desc_lo(smem_u32(smem + Cfg::OFF_V), 16);
    const uint32_t d_ds = smem_desc_lo(smem_u32(smem + Cfg::OFF_DS), 16384);
    const uint32_t d_qadd = smem_desc_lo(smem_u32(smem + Cfg::OFF_QADD), 16);
    const uint32_t d_doadd = smem_desc_lo(smem_u32(smem + Cfg::OFF_DOADD), 16);
    const uint32_t d_kadd = smem_desc_lo(smem_u32(smem + Cfg::OFF_KADD), 16);
    const uint32_t d_vadd = smem_desc_lo(smem_u32(smem + Cfg::OFF_VADD), 16);
    constexpr uint32_t kTile16 = Cfg::TILE >> 4, kAdd16 = Cfg::ADD_TILE >> 4;

    // stage trackers for the "ahead" stream (S, dP) and the "behind" stream (dV, dK, dQ)
    int aq_s = 0, ak_s = 0, av_s = 0;
    uint32_t aq_ph = 0, ak_ph = 0, av_ph = 0;
    int bq_s = 0, bk_s = 0;
    uint32_t pds_ph[2] = {0, 0}, dsready_ph = 0, dqfree_ph = 1, dkvfree_ph = ~0u;  // (dkvfree_ph: a bit per key tile of a strip)

    BwdWalk wa, wb;  // ahead / behind
    wa.init(blockIdx.x, gridDim.x, p.n_items, p.q_tiles, p.k_tiles, KS, p.n_strips);
    wb = wa;

    // whether the second half of a query tile has rows
    auto two_halves = [&](int qt) { return !RAGGED || qt * 128 + 64 < p.N; };
    auto wait_sdp = [&]() {  // for the operands of tile wa
      if (Cfg::KV_STAYS && !wa.first_qt()) warp_wait(&q_full[aq_s], aq_ph, wctx);
      else if (wa.first_kk()) warp_wait3(&q_full[aq_s], aq_ph, &k_full[ak_s], ak_ph, &v_full[av_s], av_ph, wctx);
      else warp_wait2(&k_full[ak_s], ak_ph, &v_full[av_s], av_ph, wctx);
      tc_fence_after();
    };
    auto issue_sdp = [&](int g) {  // S^T and dP^T of half g of tile wa
      const uint32_t qo = aq_s * kTile16 + g * 4 * Cfg::SWZ, ko = ak_s * kTile16, vo = av_s * kTile16;
      const uint32_t qa = aq_s * kAdd16 + g * 128;
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        umma_ss_w<hi, hi, idesc_sd>(el, tmem_base + Cfg::TM_S + 64 * g, d_k + ko + 2 * ks, d_q + qo + 2 * ks, ks != 0);
      umma_ss_w<hi_add, hi_add, idesc_sd>(el, tmem_base + Cfg::TM_S + 64 * g, d_kadd + av_s * kAdd16, d_qadd + qa, 1u);
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks)
        umma_ss_w<hi, hi, idesc_sd>(el, tmem_base + Cfg::TM_DP + 64 * g, d_v + vo + 2 * ks, d_do + qo + 2 * ks, ks != 0);
      umma_ss_w<hi_add, hi_add, idesc_sd>(el, tmem_base + Cfg::TM_DP + 64 * g, d_vadd, d_doadd + qa, 1u);
      umma_commit(el, &sdp_full[g]);
    };
    auto next_sdp = [&]() {
      if (!Cfg::KV_STAYS || wa.last_qt()) {
        umma_commit(el, &v_empty[av_s]);
        if (++av_s == NV) {
          av_s = 0;
          av_ph ^= 1;
        }
        if (++ak_s == NK) {
          ak_s = 0;
          ak_ph ^= 1;
        }
      }
      const bool last_kk = wa.last_kk();
      wa.next();
      if (last_kk) {
        if (++aq_s == NQ) {
          aq_s = 0;
          aq_ph ^= 1;
        }
      }
    };

    if (wa.valid()) {
      wait_sdp();
      issue_sdp(0);
      if (two_halves(wa.qt)) issue_sdp(1);
      next_sdp();
    }
    while (wb.valid()) {
      const uint32_t qo = bq_s * kTile16, ko = bk_s * kTile16;
      const uint32_t acc_kv = wb.first_qt() ? 0u : 1u;
      const int q_left = p.N - wb.qt * 128, k_left = p.N - wb.kt() * 128;
      const bool ahead = wa.valid();
      if (ahead) wait_sdp();  // (here the answer of the probe is not waited for in the chain of a tile)
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        if (g == 0 || two_halves(wb.qt)) {
          warp_wait(&pds_ready[g], pds_ph[g], wctx);
          pds_ph[g] ^= 1;
          if (g == 0 && wb.first_qt()) {
            // the first accumulation overwrites dK/dV: those of the previous strip must have been read out
            warp_wait(&dkv_free[wb.kk], (dkvfree_ph >> wb.kk) & 1u, wctx);
            dkvfree_ph ^= 1u << wb.kk;
          }
          tc_fence_after();
          // dV(kt) (+)= P^T dO ; dK(kt) (+)= dS^T Q   (16 queries per step; a warp's 32 queries start at its own 32 columns)
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            if (!RAGGED || 64 * g + 32 * (ks >> 1) < q_left)
              umma_ts_w<hi, idesc_kv>(el, tmem_base + Cfg::TM_DV + wb.kk * D, tmem_base + Cfg::TM_S + 64 * g + (ks >> 1) * 32 + (ks & 1) * 8,
                                      d_do + kMn + qo + (4 * g + ks) * Cfg::SWZ, (g | ks) != 0 ? 1u : acc_kv);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            if (!RAGGED || 64 * g + 32 * (ks >> 1) < q_left)
              umma_ts_w<hi, idesc_kv>(el, tmem_base + Cfg::TM_DK + wb.kk * D, tmem_base + Cfg::TM_DP + 64 * g + (ks >> 1) * 32 + (ks & 1) * 8,
                                      d_q + kMn + qo + (4 * g + ks) * Cfg::SWZ, (g | ks) != 0 ? 1u : acc_kv);
        }
        if (g == 1 && wb.last_qt()) umma_commit(el, &dkv_full[wb.kk]);
        if (g == 1 && wb.last_kk()) {
          umma_commit(el, &q_empty[bq_s]);
          if (++bq_s == NQ) bq_s = 0;
        }
        // S and dP of the next tile's half, over P and dS, which the UMMAs just issued still have to read.  PTX states the order
        // of UMMAs for one accumulator and shape only, and these have others.  What this rests on is that the UMMAs of one
        // issuing thread go through the CTA's one tensor pipe in the order of issue, which attention kernels that keep P in
        // the columns of S are commonly built on; tests compare the bits of 170 equal planes.  A completion in between would
        // put a commit and a probe (500 cycles) into the chain of every half tile.
        if (ahead) {
          if (g == 0 || two_halves(wa.qt)) issue_sdp(g);
          if (g == 1) next_sdp();
        }
      }
      // dQ(qt) (+)= dS K   (16 keys per step)
      warp_wait(ds_ready, dsready_ph, wctx);
      dsready_ph ^= 1;
      if (wb.first_kk()) {  // overwrites dQ
        warp_wait(dq_free, dqfree_ph, wctx);
        dqfree_ph ^= 1;
      }
      tc_fence_after();
      const uint32_t acc_q = wb.first_kk() ? 0u : 1u;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks)
        if (!RAGGED || 32 * (ks >> 1) < k_left)
          umma_ss_w<hi_ds, hi, idesc_dq>(el, tmem_base + Cfg::TM_DQ, d_ds + ks * 128, d_k + kMn + ko + ks * Cfg::SWZ,
                                         (ks != 0) ? 1u : acc_q);
      umma_commit(el, ds_free);
      if (wb.last_kk()) umma_commit(el, dq_full);
      if (!Cfg::KV_STAYS || wb.last_qt()) {
        umma_commit(el, &k_empty[bk_s]);
        if (++bk_s == NK) bk_s = 0;
      }
      wb.next();
    }
  } else if (warp > Cfg::WARP_ADD) {
    // ------------------------------------------------------------------ finished gradients
    // Four warps, one per TMEM lane quarter, read dQ after the last key tile of a query tile, and dK and dV of every key tile of
    // a strip after the last query tile, as they are finished: 32 rows go through shared memory and leave by one TMA (D = 64:
    // from registers).  With several strips dQ is summed in the CTA's scratch, in the order of the strips.
    // (By the compute warps between two tiles this was 450 cycles of a tile's 2550.)
    const int lane_base = 32 * (warp & 3);
    const float scale = p.scale;
    uint32_t dqfull_ph = 0, dkvfull_ph = 0;
    [[maybe_unused]] int stg_buf = 0;
    // tile rows n0 .. n0 + 127 in TMEM columns col ..; part: the tile is a part of the sum, `strip` of n_strips
    auto drain = [&](uint32_t col, float mul, const CUtensorMap* map, __nv_bfloat16* plane, int n0, uint64_t* free_bar, bool part,
                     int strip, int b, int o, int h) {
      const int r0 = n0 + lane_base, row = r0 + lane;
      const uint32_t src = tmem_addr(tmem_base, lane_base, col);
      const bool out = !part || strip + 1 == p.n_strips;
      if (r0 >= p.N) {
        if (lane == 0) mbar_arrive(free_bar);
        return;
      }
      // scratch of 32 rows (fewer at the end): 4 columns of every row, the next 4 ..., so that a warp's accesses are contiguous
      const int rows = min(32, p.N - r0);
      float4* const sums = reinterpret_cast<float4*>(p.dq_scratch + ((int64_t)blockIdx.x * p.N + r0) * D) + lane;
      uint8_t* const stg = smem + Cfg::OFF_STG + ((warp & 3) * 2 + stg_buf) * Cfg::STG_BYTES;
      if constexpr (Cfg::STAGED) {
        if (out) {  // every use of a buffer is followed by its store: all stores but the newest have left the other one
          stg_buf ^= 1;
          bulk_wait_read<1>();
          __syncwarp();
        }
      }
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        uint32_t r[16];
        tmem_ld16(src + c, r);
        tmem_ld_wait();
        if (c + 16 == D) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(free_bar);
        }
        if (part && row < p.N) {
          if (strip > 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 a = sums[(c / 4 + i) * rows];
              r[4 * i] = __float_as_uint(__uint_as_float(r[4 * i]) + a.x);
              r[4 * i + 1] = __float_as_uint(__uint_as_float(r[4 * i + 1]) + a.y);
              r[4 * i + 2] = __float_as_uint(__uint_as_float(r[4 * i + 2]) + a.z);
              r[4 * i + 3] = __float_as_uint(__uint_as_float(r[4 * i + 3]) + a.w);
            }
          }
          if (!out) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              sums[(c / 4 + i) * rows] = make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]),
                                                     __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
          }
        }
        if (!out) continue;
        uint4 w[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * i + e]) * mul;
          w[i] = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        }
        if constexpr (Cfg::STAGED) {
          const int sw = D == 32 ? (lane >> 1) & 3 : (lane >> 2) & 1;  // the maps' 64- / 32-byte swizzle
#pragma unroll
          for (int i = 0; i < 2; ++i) *reinterpret_cast<uint4*>(stg + lane * (2 * D) + (((c >> 3) + i) ^ sw) * 16) = w[i];
        } else if (row < p.N) {
          uint4* dst = reinterpret_cast<uint4*>(plane + row * p.gn + c);
          dst[0] = w[0];
          dst[1] = w[1];
        }
      }
      if constexpr (Cfg::STAGED) {
        fence_async_smem();
        __syncwarp();
        if (out) tma_store_5d(lane == 0, map, stg, 0, r0, h, o, b);
      }
    };
    for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
      int b, o, h;
      decode(item, b, o, h);
      const int64_t off = b * p.gb + o * p.go + h * p.gh;
      for (int strip = 0; strip < p.n_strips; ++strip) {
        const int tiles_k = min(KS, p.k_tiles - strip * KS);
        for (int qt = 0; qt < p.q_tiles; ++qt) {
          if (qt == p.q_tiles - 1) {
            for (int kk = 0; kk < tiles_k; ++kk) {
              warp_wait(&dkv_full[kk], (dkvfull_ph >> kk) & 1u, wctx);
              dkvfull_ph ^= 1u << kk;
              tc_fence_after();
              const int n0 = (strip * KS + kk) * 128;
              // (each of the two reads arrives: dkv_free counts eight)
              drain(Cfg::TM_DK + kk * D, scale, &tmDK, p.dk + off, n0, &dkv_free[kk], false, 0, b, o, h);
              drain(Cfg::TM_DV + kk * D, 1.f, &tmDV, p.dv + off, n0, &dkv_free[kk], false, 0, b, o, h);
            }
          }
          warp_wait(dq_full, dqfull_ph, wctx);
          dqfull_ph ^= 1;
          tc_fence_after();
          drain(Cfg::TM_DQ, scale, &tmDQ, p.dq + off, qt * 128, dq_free, p.n_strips > 1, strip, b, o, h);
        }
      }
    }
    if constexpr (Cfg::STAGED) bulk_wait_all();
  } else {
    // ------------------------------------------------------------------ compute warps
    const int part = warp >> 2;                 // which 32 queries of the tile
    const int g = part >> 1;                    // group
    const int lane_base = 32 * (warp & 3);
    const int row = lane_base + lane;           // key in the tile == TMEM lane
    const uint32_t t_s = tmem_addr(tmem_base, lane_base, Cfg::TM_S + 32 * part);
    const uint32_t t_dp = tmem_addr(tmem_base, lane_base, Cfg::TM_DP + 32 * part);
    // dS^T tile: a row per key, 128 bytes = the 64 queries of a group; the thread's 32 queries are four 16-byte pieces
    uint8_t* const ds_row = smem + Cfg::OFF_DS + g * 16384 + row * 128;
    const int piece0 = (part & 1) * 4;
    // bias tile: a row per query, 256 bytes = 128 keys, not swizzled: the lanes of a warp read 64 consecutive bytes
    const uint8_t* const bias_col = smem + Cfg::OFF_BIAS + part * (32 * 256) + row * 2;
    constexpr float kLog2e = 1.4426950408889634f;
    const uint64_t c1 = f2_pack(p.logit_scale * kLog2e, p.logit_scale * kLog2e);
    const uint64_t log2e2 = f2_pack(kLog2e, kLog2e);
    [[maybe_unused]] const int tail_keys = p.N - (p.k_tiles - 1) * 128;  // of the last key tile
    [[maybe_unused]] const bool tail_warp = lane_base + 32 > tail_keys;

    uint32_t sdpfull_ph = 0, dsfree_ph = 1, b_ph = 0;
    int b_s = 0;
    // The (item, strip, query tile, key tile) sequence as plain loops: the scalar part of a step is on the path between
    // two UMMA batches.
    for (int item = blockIdx.x; item < p.n_items; item += gridDim.x) {
    for (int strip = 0; strip < p.n_strips; ++strip) {
      const int tiles_k = min(KS, p.k_tiles - strip * KS);
    for (int qt = 0; qt < p.q_tiles; ++qt) {
      bool no_half = false, no_rows = false;  // the group's / this warp's queries all lie beyond the last one
      if constexpr (RAGGED) {
        no_half = qt * 128 + 64 * g >= p.N;
        no_rows = qt * 128 + 32 * part >= p.N;
      }
    for (int kk = 0; kk < tiles_k; ++kk) {
      uint32_t dpk[16];  // bf16 pairs of dS of this thread's 32 queries
      bool dead = false;
      if constexpr (RAGGED) dead = no_rows || (strip * KS + kk) * 128 + lane_base >= p.N;
      if (RAGGED && no_half) {
        warp_wait(&b_full[b_s], b_ph, wctx);
      } else {
        warp_wait2(&sdp_full[g], sdpfull_ph, &b_full[b_s], b_ph, wctx);
        sdpfull_ph ^= 1;
      }
      tc_fence_after();
      const uint8_t* bias = bias_col + b_s * Cfg::BIAS_STAGE;
      if (dead) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&b_empty[b_s]);
      } else {
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {  // 16 queries per step
          uint32_t rs[16], rd[16], bu[16];
          tmem_ld16(t_s + 16 * ch, rs);
          tmem_ld16(t_dp + 16 * ch, rd);
#pragma unroll
          for (int e = 0; e < 16; ++e) bu[e] = *reinterpret_cast<const uint16_t*>(bias + (16 * ch + e) * 256);
          tmem_ld_wait();
          uint32_t ppk[8], dtm[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const uint64_t bl = f2_mul(f2_pack_bits(bu[2 * e] << 16, bu[2 * e + 1] << 16), log2e2);
            float a0, a1;
            f2_unpack(f2_fma(f2_pack_bits(rs[2 * e], rs[2 * e + 1]), c1, bl), a0, a1);
            const float p0 = ex2_approx(a0), p1 = ex2_approx(a1);
            float d0, d1;
            f2_unpack(f2_mul(f2_pack(p0, p1), f2_pack_bits(rd[2 * e], rd[2 * e + 1])), d0, d1);
            ppk[e] = pack_bf16x2(p0, p1);
            dtm[e] = dpk[8 * ch + e] = pack_bf16x2(d0, d1);
          }
          if (ch == 1) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&b_empty[b_s]);
          }
          tmem_st8(t_s + 8 * ch, ppk);
          tmem_st8(t_dp + 8 * ch, dtm);
        }
        tmem_st_wait();
      }
      if (!(RAGGED && no_half)) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&pds_ready[g]);
      }
      if (++b_s == NB) {
        b_s = 0;
        b_ph ^= 1;
      }

      // the dQ UMMAs of the previous tile are done: the dS tile is free
      warp_wait(ds_free, dsfree_ph, wctx);
      dsfree_ph ^= 1;
      if (!dead) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          *reinterpret_cast<uint4*>(ds_row + (((piece0 + u) ^ (row & 7)) << 4)) =
              make_uint4(dpk[4 * u], dpk[4 * u + 1], dpk[4 * u + 2], dpk[4 * u + 3]);
        if (TAIL && tail_warp && strip * KS + kk == p.k_tiles - 1 && row >= tail_keys) {
#pragma unroll
          for (int u = 0; u < 4; ++u)
            *reinterpret_cast<uint4*>(ds_row + (((piece0 + u) ^ (row & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
    }  // key tiles
    }  // query tiles
    }
    }
    // the UMMAs of this CTA's last tile have to be over before it ends
    warp_wait(ds_free, dsfree_ph, wctx);
    tc_fence_after();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::WARP_MMA) {
    __syncwarp();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// The additive mask of a tile's 128 keys as an operand of S (see Bf16x3; the A operand is ones).  Called by the issuing warp;
// returns whether there is anything to add.  A lane makes the rows of four keys.
__device__ __forceinline__ bool mask_operand(uint8_t* dst, const float* mask_row, int lane, float inv_scale) {
  const float4 m = reinterpret_cast<const float4*>(mask_row)[lane];
  float v[4] = {m.x, m.y, m.z, m.w};
  bool any = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) any |= v[i] != 0.f;
  if (!__any_sync(0xffffffffu, any)) return false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const Bf16x3 x = split_bf16x3(v[i] * inv_scale);
    store_added(dst, 4 * lane + i, make_uint4(x.hi | x.mid << 16, x.lo, 0u, 0u));
  }
  fence_async_smem();
  __syncwarp();
  return true;
}

// =============================================================================================
// kernel 2: dBias partial planes.  One CTA = one (group, h, query tile, key tile) and a chunk of
// outer planes; dS summed over the chunk in ascending plane order, fp32, in registers.
// =============================================================================================
struct AttnDbiasParams {
  float* part;        // [n_chunks][G][H][N][N] fp32 (or the final buffer when n_chunks == 1)
  const float* lse;   // [B,O,H,N]
  const float* delta; // [B,O,H,N]
  int B, O, H, N;
  int G;              // bias batch (1 or B)
  int planes;         // outer planes per group = (B / G) * O
  int n_chunks, chunk_len;
  int q_tiles, k_tiles;
  float scale;
};

template <int D_>
struct AttnDbiasCfg {
  static constexpr int D = D_;
  static constexpr int SWZ = 2 * D;
  static constexpr int TILE = 128 * D * 2;
  static constexpr int STAGE = 4 * TILE + 1024;  // Q, dO, K, V, mask row
  static constexpr int NST = D <= 32 ? 4 : 2;
  static constexpr int NCW = 16;                 // compute warps: four threads per query row, 32 keys each
  static constexpr int OFF_BIAS32 = 0;           // the CTA's bias tile as fp32 * log2(e), 64 KiB, thread-major
  static constexpr int OFF_ST = 65536;
  // the bf16 bias tile is staged once: in the last stage buffer when that is large enough (the
  // producer waits for the conversion before it first fills that buffer), else in a region of its own
  static constexpr bool STAGE_HOLDS_BIAS = STAGE >= 32768 + 1024;
  static constexpr int OFF_BSTG = STAGE_HOLDS_BIAS ? OFF_ST + (NST - 1) * STAGE : OFF_ST + NST * STAGE;
  // the mask as an operand (see mask_operand): ones [128][16], and the mask of each S buffer [128][16]
  static constexpr int OFF_ONES = OFF_ST + NST * STAGE + (STAGE_HOLDS_BIAS ? 0 : 32768);
  static constexpr int OFF_MOP = OFF_ONES + 4096;
  static constexpr int OFF_BAR = OFF_MOP + 2 * 4096;
  static constexpr int N_BAR = 2 * NST + 4 + 2;
  static constexpr int SMEM_BYTES = OFF_BAR + N_BAR * 8 + 16 + 1024;
  static constexpr int TMEM_COLS = 512;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

// 16 compute warps: four threads share one query row (TMEM lane) and take 32 of the 128 keys of the
// tile each.  The bias tile of a CTA never changes, so it is converted once to fp32 (already
// multiplied by log2 e) and read back with conflict-free 16-byte loads; per logit the inner loop is
// four packed fp32x2 operations per pair and one ex2.  The mask is no business of these warps: where a plane has one in this key
// range, the issuing warp adds it to S by one more UMMA (K = 16).  As an add in the loop, behind a vote, it cost every plane
// and made the CTAs of the masked keys the last to finish.  Measured, N = 384 with 5 % of the keys masked: 115 -> 85 us, N = 768
// 844 -> 603.  Columns beyond N are computed with the zeros that TMA fills in and never stored.
template <class Cfg>
__global__ void __launch_bounds__(32 * (Cfg::NCW + 2), 1)
attn_dbias_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                  const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO,
                  const __grid_constant__ CUtensorMap tmBias, const __grid_constant__ CUtensorMap tmMask,
                  const AttnDbiasParams p, int* __restrict__ status) {
  griddep_wait();
  constexpr int D = Cfg::D, NST = Cfg::NST, NCW = Cfg::NCW;
  constexpr int WARP_TMA = NCW, WARP_MMA = NCW + 1;
  constexpr int CPT = 32;                   // key columns per thread
  // the declared alignment makes every address below a constant: 904 -> 868 us at N = 768
  extern __shared__ __align__(1024) uint8_t smem_al[];
  uint8_t* smem = smem_al + ((1024u - (smem_u32(smem_al) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* full = bars;
  uint64_t* empty = full + NST;
  uint64_t* sdp_full = empty + NST;   // [2]
  uint64_t* sdp_free = sdp_full + 2;  // [2]
  uint64_t* bias_full = sdp_free + 2;
  uint64_t* bias_done = bias_full + 1;  // the compute warps have converted the staged bias tile
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::N_BAR);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wctx{abort_flag, status};
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  uint8_t* bias_stage = smem + Cfg::OFF_BSTG;  // bf16 tile as TMA delivers it

  // work item
  int it = blockIdx.x;
  const int chunk = it % p.n_chunks; it /= p.n_chunks;
  const int kt = it % p.k_tiles; it /= p.k_tiles;
  const int qt = it % p.q_tiles; it /= p.q_tiles;
  const int h = it % p.H;
  const int g = it / p.H;
  const int pl0 = chunk * p.chunk_len;
  const int pl1 = min(p.planes, pl0 + p.chunk_len);
  const int b_per_g = p.B / p.G;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NST; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sdp_full[s], 1);
      mbar_init(&sdp_free[s], NCW);
    }
    mbar_init(bias_full, 1);
    mbar_init(bias_done, NCW);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
    tma_prefetch_desc(&tmBias);
    tma_prefetch_desc(&tmMask);
  }
  for (int i = threadIdx.x; i < 3 * 1024; i += blockDim.x)
    reinterpret_cast<uint32_t*>(smem + Cfg::OFF_ONES)[i] = i < 1024 ? 0x3F803F80u : 0u;
  fence_async_smem();
  if (warp == WARP_MMA) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == WARP_TMA) {
    {
      const uint32_t el = elect_one();
      mbar_expect_tx(el, bias_full, 32768);
      tma_load_4d(el, bias_stage, &tmBias, bias_full, kt * 128, qt * 128, h, g);
      tma_load_4d(el, bias_stage + 16384, &tmBias, bias_full, kt * 128 + 64, qt * 128, h, g);
      int s = 0;
      uint32_t ph = 1;
      for (int pl = pl0; pl < pl1; ++pl) {
        const int b = g * b_per_g + pl / p.O, o = pl % p.O;
        if (pl - pl0 == NST - 1) warp_wait(bias_done, 0, wctx);  // first use of the buffer the bias was staged in
        warp_wait(&empty[s], ph, wctx);
        mbar_expect_tx(el, &full[s], 4 * Cfg::TILE + 512);
        uint8_t* st = smem + Cfg::OFF_ST + s * Cfg::STAGE;
        tma_load_5d(el, st, &tmQ, &full[s], 0, qt * 128, h, o, b);
        tma_load_5d(el, st + Cfg::TILE, &tmDO, &full[s], 0, qt * 128, h, o, b);
        tma_load_5d(el, st + 2 * Cfg::TILE, &tmK, &full[s], 0, kt * 128, h, o, b);
        tma_load_5d(el, st + 3 * Cfg::TILE, &tmV, &full[s], 0, kt * 128, h, o, b);
        tma_load_3d(el, st + 4 * Cfg::TILE, &tmMask, &full[s], kt * 128, o, b);
        if (++s == NST) {
          s = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp == WARP_MMA) {
    {
      const uint32_t el = elect_one();
      constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, false);
      constexpr uint32_t swz = swizzle_mode_for_bytes(Cfg::SWZ);
      const uint64_t ones_desc = make_smem_desc(smem_u32(smem + Cfg::OFF_ONES), 16, 256, swizzle_mode_for_bytes(32));
      const uint64_t mop_desc = make_smem_desc(smem_u32(smem + Cfg::OFF_MOP), 16, 256, swizzle_mode_for_bytes(32));
      const float inv_scale = 1.f / p.scale;
      int s = 0, buf = 0;
      uint32_t ph = 0, free_ph[2] = {1, 1};
      for (int pl = pl0; pl < pl1; ++pl) {
        warp_wait2(&full[s], ph, &sdp_free[buf], free_ph[buf], wctx);
        free_ph[buf] ^= 1;
        tc_fence_after();
        const uint32_t st = smem_u32(smem + Cfg::OFF_ST + s * Cfg::STAGE);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          umma_ss(el, tmem_base + buf * 256, make_smem_desc(st + ks * 32, 16, 8 * Cfg::SWZ, swz),
                  make_smem_desc(st + 2 * Cfg::TILE + ks * 32, 16, 8 * Cfg::SWZ, swz), idesc, ks != 0);
        // (S of this buffer has been read, so the UMMA that used its mask operand is done)
        if (mask_operand(smem + Cfg::OFF_MOP + buf * 4096, reinterpret_cast<const float*>(smem + Cfg::OFF_ST + s * Cfg::STAGE + 4 * Cfg::TILE),
                         lane, inv_scale))
          umma_ss(el, tmem_base + buf * 256, ones_desc, mop_desc + (uint64_t)(buf * (4096 >> 4)), idesc, 1u);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          umma_ss(el, tmem_base + buf * 256 + 128, make_smem_desc(st + Cfg::TILE + ks * 32, 16, 8 * Cfg::SWZ, swz),
                  make_smem_desc(st + 3 * Cfg::TILE + ks * 32, 16, 8 * Cfg::SWZ, swz), idesc, ks != 0);
        umma_commit(el, &sdp_full[buf]);
        umma_commit(el, &empty[s]);
        buf ^= 1;
        if (++s == NST) {
          s = 0;
          ph ^= 1;
        }
      }
    }
  } else if (warp < NCW) {
    const int part = warp >> 2;               // which 32-column slice of the tile
    const int row = 32 * (warp & 3) + lane;
    const uint32_t lane_base = 32 * (warp & 3);
    constexpr float kLog2e = 1.4426950408889634f;
    const float c1 = p.scale * kLog2e;
    const uint64_t c2 = f2_pack(c1, c1);
    const int q = qt * 128 + row;

    // ---- bias tile -> fp32 * log2(e), laid out [part][16-column half][4-column group][row][4] so that
    //      the 32 lanes of a warp read 32 consecutive 16-byte pieces
    float4* bias32 = reinterpret_cast<float4*>(smem + Cfg::OFF_BIAS32);
    warp_wait(bias_full, 0, wctx);
    {
      const int col0 = CPT * part;
      const uint8_t* brow = bias_stage + (col0 >> 6) * 16384 + row * 128;
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // 8 columns per 16-byte piece of the bf16 tile
        const uint4 bv = *reinterpret_cast<const uint4*>(brow + (((((col0 & 63) >> 3) + u) ^ (row & 7)) << 4));
        const float4 lo = make_float4(__uint_as_float(bv.x << 16) * kLog2e, __uint_as_float(bv.x & 0xFFFF0000u) * kLog2e,
                                      __uint_as_float(bv.y << 16) * kLog2e, __uint_as_float(bv.y & 0xFFFF0000u) * kLog2e);
        const float4 hi = make_float4(__uint_as_float(bv.z << 16) * kLog2e, __uint_as_float(bv.z & 0xFFFF0000u) * kLog2e,
                                      __uint_as_float(bv.w << 16) * kLog2e, __uint_as_float(bv.w & 0xFFFF0000u) * kLog2e);
        // piece u covers columns 8u .. 8u+7 of the slice: half = u / 2, groups 2 (u % 2) and 2 (u % 2) + 1
        bias32[(((part * 2 + (u >> 1)) * 4 + 2 * (u & 1)) * 128) + row] = lo;
        bias32[(((part * 2 + (u >> 1)) * 4 + 2 * (u & 1) + 1) * 128) + row] = hi;
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(bias_done);

    uint64_t acc[CPT / 2];
#pragma unroll
    for (int i = 0; i < CPT / 2; ++i) acc[i] = 0ull;

    // lse / delta of (plane, h, q): planes of one group are consecutive in memory, so the index
    // advances by H * N per step (no division in the loop)
    const int64_t row_stride = (int64_t)p.H * p.N;
    const int64_t row_idx0 = ((int64_t)g * b_per_g * p.O * p.H + h) * p.N + q;
    auto load_row_scalars = [&](int pl, float& l, float& dl) {
      l = INFINITY;  // a row without a finite log-sum-exp (fully masked, or past N) contributes nothing
      dl = 0.f;
      if (pl < pl1 && q < p.N) {
        const int64_t idx = row_idx0 + (int64_t)pl * row_stride;
        l = __ldg(p.lse + idx);
        dl = __ldg(p.delta + idx);
      }
    };

    int buf = 0;
    uint32_t full_ph[2] = {0, 0};
    // row scalars travel two planes ahead of their use (they come from HBM on first touch)
    float l_n1, dl_n1, l_n2, dl_n2;
    load_row_scalars(pl0, l_n1, dl_n1);
    load_row_scalars(pl0 + 1, l_n2, dl_n2);
    for (int pl = pl0; pl < pl1; ++pl) {
      // exp2(t - lse log2e) of a fully masked row must give 0, not NaN or infinity
      const float nl = (l_n1 < kMaskedLse || l_n1 == INFINITY) ? -INFINITY : -l_n1 * kLog2e;
      const uint64_t nl2 = f2_pack(nl, nl);
      const uint64_t nd2 = f2_pack(-dl_n1, -dl_n1);
      l_n1 = l_n2;
      dl_n1 = dl_n2;
      load_row_scalars(pl + 2, l_n2, dl_n2);
      warp_wait(&sdp_full[buf], full_ph[buf], wctx);
      full_ph[buf] ^= 1;
      tc_fence_after();
      const uint32_t t_s = tmem_addr(tmem_base, lane_base, buf * 256 + CPT * part);
      const uint32_t t_dp = tmem_addr(tmem_base, lane_base, buf * 256 + 128 + CPT * part);
      // 8 columns per step; the TMEM loads of step c+1 are in flight while step c is computed
      uint32_t rs[2][8], rd[2][8];
      tmem_ld8(t_s, rs[0]);
      tmem_ld8(t_dp, rd[0]);
#pragma unroll
      for (int c = 0; c < CPT / 8; ++c) {
        const float4 bb0 = bias32[((part * 2 + (c >> 1)) * 4 + 2 * (c & 1)) * 128 + row];
        const float4 bb1 = bias32[((part * 2 + (c >> 1)) * 4 + 2 * (c & 1) + 1) * 128 + row];
        tmem_ld_wait();  // step c has landed
        if (c + 1 < CPT / 8) {
          tmem_ld8(t_s + 8 * (c + 1), rs[(c + 1) & 1]);
          tmem_ld8(t_dp + 8 * (c + 1), rd[(c + 1) & 1]);
        } else {
          // the whole TMEM tile is in registers: the next S / dP pair may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sdp_free[buf]);
        }
        const uint32_t(&s8)[8] = rs[c & 1];
        const uint32_t(&d8)[8] = rd[c & 1];
        uint64_t t2[4];
        t2[0] = f2_fma(f2_pack_bits(s8[0], s8[1]), c2, f2_pack(bb0.x, bb0.y));
        t2[1] = f2_fma(f2_pack_bits(s8[2], s8[3]), c2, f2_pack(bb0.z, bb0.w));
        t2[2] = f2_fma(f2_pack_bits(s8[4], s8[5]), c2, f2_pack(bb1.x, bb1.y));
        t2[3] = f2_fma(f2_pack_bits(s8[6], s8[7]), c2, f2_pack(bb1.z, bb1.w));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float a0, a1;
          f2_unpack(f2_add(t2[i], nl2), a0, a1);
          const uint64_t pr = f2_pack(ex2_approx(a0), ex2_approx(a1));
          const uint64_t gd = f2_add(f2_pack_bits(d8[2 * i], d8[2 * i + 1]), nd2);
          acc[4 * c + i] = f2_fma(pr, gd, acc[4 * c + i]);
        }
      }
      buf ^= 1;
    }

    if (q < p.N) {
      const int k0 = kt * 128 + CPT * part;
      float* dst = p.part + ((((int64_t)chunk * p.G + g) * p.H + h) * p.N + q) * p.N + k0;
      float a[CPT];
#pragma unroll
      for (int i = 0; i < CPT / 2; ++i) f2_unpack(acc[i], a[2 * i], a[2 * i + 1]);
      if ((p.N & 3) == 0 && k0 + CPT <= p.N) {
#pragma unroll
        for (int i = 0; i < CPT; i += 4)
          *reinterpret_cast<float4*>(dst + i) = make_float4(a[i], a[i + 1], a[i + 2], a[i + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < CPT; ++i)
          if (k0 + i < p.N) dst[i] = a[i];
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == WARP_MMA) {
    __syncwarp();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// dbias[i] = ((part[0][i] + part[1][i]) + part[2][i]) + ...   (ascending chunk order, fp32)
__global__ void __launch_bounds__(256) attn_dbias_fold_kernel(const float* __restrict__ part, float* __restrict__ out,
                                                              int64_t n, int n_chunks) {
  griddep_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    float a = part[i];
    for (int c = 1; c < n_chunks; ++c) a = __fadd_rn(a, part[(int64_t)c * n + i]);
    out[i] = a;
  }
}

// The same sum, written as bf16 rows: row (g, i, j) of `out` (pitch ld) gets the H gradients of pair (i, j), then zeros
// up to a multiple of 8 columns (they are K columns of the GEMM that follows).
__global__ void __launch_bounds__(256) attn_dbias_rows_kernel(const float* __restrict__ part,
                                                              __nv_bfloat16* __restrict__ out, int64_t ld, int H,
                                                              int64_t NN, int64_t n_rows, int n_chunks) {
  griddep_wait();
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t g = r / NN, ij = r - g * NN;
    const int64_t plane = n_rows * H;
    for (int h0 = 0; h0 < H; h0 += 8) {
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        v[e] = 0.f;
        if (h0 + e < H) {
          const float* src = part + (g * H + h0 + e) * NN + ij;
          float a = src[0];
          for (int c = 1; c < n_chunks; ++c) a = __fadd_rn(a, src[c * plane]);
          v[e] = a;
        }
      }
      *reinterpret_cast<uint4*>(out + r * ld + h0) =
          make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
int make_qkv_tmap(CUtensorMap* tm, const void* base, int64_t B, int64_t O, int64_t H, int64_t N, int64_t D,
                  const int64_t* st, int swz);
int make_bias_tmap(CUtensorMap* tm, const void* base, int64_t Bb, int64_t H, int64_t N, int64_t pitch);
int make_bias_tmap_plain(CUtensorMap* tm, const void* base, int64_t Bb, int64_t H, int64_t N, int64_t pitch);
int make_mask_tmap(CUtensorMap* tm, const void* base, int64_t B, int64_t O, int64_t N, int64_t pitch);
int make_qkv_tmap_rows(CUtensorMap* tm, const void* base, int64_t B, int64_t O, int64_t H, int64_t N, int64_t D,
                       const int64_t* st, int swz, int rows);

// What is added to the logits by UMMAs is divided by the softmax scale first.  A scale of zero (or nearly) leaves the logits
// themselves out of fp32 sums with these quotients, which is what it asks for.
static float logit_scale(float scale) { return fabsf(scale) < 1e-20f ? copysignf(1e-20f, scale) : scale; }

template <int D>
int launch_attn_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                    const CUtensorMap& tb, const CUtensorMap& tdq, const CUtensorMap& tdk, const CUtensorMap& tdv,
                    AttnBwdParams& p, int* status, int grid, cudaStream_t stream) {
  using Cfg = AttnBwdCfg<D>;
  const bool ragged = p.N % 128 != 0 && p.N % 128 <= 96;  // some 32-row (32-key) block of the last tile is empty
  const int form = p.N % 128 == 0 ? 0 : ragged ? 2 : 1;
  auto kern = form == 0   ? attn_bwd_kernel<Cfg, false, false>
              : form == 1 ? attn_bwd_kernel<Cfg, true, false>
                          : attn_bwd_kernel<Cfg, true, true>;
  static PerDeviceOnce once[3];  // per instantiation
  if (int rc = ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, once[form])) return rc;
  launch_kernel(kern, dim3(grid), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, stream, tq, tk, tv, tdo, tb, tdq, tdk, tdv, p, status);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

static int bwd_key_strip(int64_t D) { return D <= 32 ? 3 : 1; }

int64_t attn_bwd_workspace_bytes(int64_t B, int64_t O, int64_t H, int64_t N, int64_t D) {
  const int64_t k_tiles = (N + 127) / 128;
  const int64_t strips = (k_tiles + bwd_key_strip(D) - 1) / bwd_key_strip(D);
  if (strips <= 1) return 0;
  int64_t grid = sm_count();
  if (grid > B * O * H) grid = B * O * H;
  return grid * N * D * 4;
}

int attn_bwd_dqkv(const void* q, const void* k, const void* v, const void* d_out, const int64_t* q_strides,
                  const int64_t* k_strides, const int64_t* v_strides, const void* out, const float* lse,
                  const float* mask, int64_t mask_pitch, const void* bias, int64_t bias_pitch, int64_t bias_batch,
                  void* dq, void* dk, void* dv, float* delta, void* workspace, int64_t workspace_bytes, int64_t B,
                  int64_t O, int64_t H, int64_t N, int64_t D, float scale, int stages, cudaStream_t stream) {
  TPF_REQUIRE(q && k && v && d_out && out && lse && mask && bias && delta && (!(stages & 2) || (dq && dk && dv)),
              TPF_ERR_INVALID_ARGUMENT, "attn_bwd: null pointer");
  TPF_REQUIRE(B > 0 && O > 0 && H > 0 && N > 0, TPF_ERR_INVALID_ARGUMENT, "attn_bwd: B,O,H,N must be positive");
  TPF_REQUIRE(D == 16 || D == 32 || D == 64, TPF_ERR_UNSUPPORTED, "attn_bwd: head dim %lld not in {16,32,64}",
              (long long)D);
  TPF_REQUIRE(bias_batch == 1 || bias_batch == B, TPF_ERR_INVALID_ARGUMENT, "attn_bwd: bias batch must be 1 or B");
  TPF_REQUIRE(bias_pitch >= N && bias_pitch % 8 == 0, TPF_ERR_INVALID_ARGUMENT,
              "attn_bwd: bias row pitch must be >= N and a multiple of 8 elements");
  TPF_REQUIRE(mask_pitch >= N && mask_pitch % 4 == 0, TPF_ERR_INVALID_ARGUMENT,
              "attn_bwd: mask row pitch must be >= N and a multiple of 4 elements");
  TPF_REQUIRE(B * O * H < (1ll << 31) && N <= (1 << 24), TPF_ERR_INVALID_ARGUMENT, "attn_bwd: extent too large");
  // dq / dk / dv rows and the delta pass's operands are accessed with 16-byte vectors
  TPF_REQUIRE_ALIGNED16(dq, "attn_bwd", "dq");
  TPF_REQUIRE_ALIGNED16(dk, "attn_bwd", "dk");
  TPF_REQUIRE_ALIGNED16(dv, "attn_bwd", "dv");
  TPF_REQUIRE_ALIGNED16(d_out, "attn_bwd", "d_out");
  TPF_REQUIRE_ALIGNED16(out, "attn_bwd", "out");
  const int64_t need = attn_bwd_workspace_bytes(B, O, H, N, D);
  TPF_REQUIRE(need == 0 || (workspace && workspace_bytes >= need), TPF_ERR_WORKSPACE,
              "attn_bwd: workspace of %lld bytes required, %lld given", (long long)need, (long long)workspace_bytes);
  TPF_REQUIRE(need == 0 || (reinterpret_cast<uintptr_t>(workspace) & 15) == 0, TPF_ERR_WORKSPACE,
              "attn_bwd: workspace must be 16-byte aligned");

  // delta = rowsum(dO * O)
  if (stages & 1) {
    const int64_t rows = B * O * N * H;
    const int lanes = (int)D / 8;
    const int64_t threads = rows * lanes;
    const int64_t blocks = (threads + 255) / 256;
    TPF_REQUIRE(blocks < (1ll << 31), TPF_ERR_INVALID_ARGUMENT, "attn_bwd: too many rows");
    const __nv_bfloat16* a = reinterpret_cast<const __nv_bfloat16*>(d_out);
    const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(out);
    if (D == 16) launch_kernel(attn_delta_kernel<16>, dim3((unsigned)blocks), dim3(256), 0, stream, a, b, delta, rows, (int)H, (int)N);
    else if (D == 32) launch_kernel(attn_delta_kernel<32>, dim3((unsigned)blocks), dim3(256), 0, stream, a, b, delta, rows, (int)H, (int)N);
    else launch_kernel(attn_delta_kernel<64>, dim3((unsigned)blocks), dim3(256), 0, stream, a, b, delta, rows, (int)H, (int)N);
    TPF_LAUNCH_OK();
  }

  if (!(stages & 2)) return TPF_OK;
  AttnCall c = {};
  c.B = B; c.O = O; c.H = H; c.N = N; c.D = D; c.G = bias_batch;
  c.scale = scale;
  c.q = q; c.k = k; c.v = v;
  for (int i = 0; i < 4; ++i) {
    c.qs[i] = q_strides[i];
    c.ks[i] = k_strides[i];
    c.vs[i] = v_strides[i];
  }
  c.mask = mask; c.mask_pitch = mask_pitch;
  c.bias = bias; c.bias_pitch = bias_pitch;
  c.lse = const_cast<float*>(lse);
  c.d_out = d_out;  // [B,O,N,H,D]
  c.dos[0] = O * N * H * D; c.dos[1] = N * H * D; c.dos[2] = D; c.dos[3] = H * D;
  c.delta = delta;
  c.dq = dq; c.dk = dk; c.dv = dv;  // [B,O,H,N,D]
  c.ds[0] = O * H * N * D; c.ds[1] = H * N * D; c.ds[2] = N * D; c.ds[3] = D;
  return attn_backward_qkv(c, workspace, workspace_bytes, stream);
}

int attn_backward_qkv(const AttnCall& c, void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
  const int64_t B = c.B, O = c.O, H = c.H, N = c.N, D = c.D;
  const int64_t need = attn_bwd_workspace_bytes(B, O, H, N, D);
  TPF_REQUIRE(need == 0 || (workspace && workspace_bytes >= need), TPF_ERR_WORKSPACE, "attn_bwd: workspace too small");
  TPF_REQUIRE_ALIGNED16(c.mask, "attn_bwd", "mask");  // rows are read with 16-byte loads
  const int swz = 2 * (int)D;
  CUtensorMap tq, tk, tv, tdo, tb, tdq = {}, tdk = {}, tdv = {};
  int rc;
  if ((rc = make_qkv_tmap(&tq, c.q, B, O, H, N, D, c.qs, swz))) return rc;
  if ((rc = make_qkv_tmap(&tk, c.k, B, O, H, N, D, c.ks, swz))) return rc;
  if ((rc = make_qkv_tmap(&tv, c.v, B, O, H, N, D, c.vs, swz))) return rc;
  if ((rc = make_qkv_tmap(&tdo, c.d_out, B, O, H, N, D, c.dos, swz))) return rc;
  if ((rc = make_bias_tmap_plain(&tb, c.bias, c.G, H, N, c.bias_pitch))) return rc;
  if (D <= 32 && ((rc = make_qkv_tmap_rows(&tdq, c.dq, B, O, H, N, D, c.ds, swz, 32)) ||
                  (rc = make_qkv_tmap_rows(&tdk, c.dk, B, O, H, N, D, c.ds, swz, 32)) ||
                  (rc = make_qkv_tmap_rows(&tdv, c.dv, B, O, H, N, D, c.ds, swz, 32))))
    return rc;
  AttnBwdParams p;
  p.dq = reinterpret_cast<__nv_bfloat16*>(c.dq);
  p.dk = reinterpret_cast<__nv_bfloat16*>(c.dk);
  p.dv = reinterpret_cast<__nv_bfloat16*>(c.dv);
  p.gb = c.ds[0]; p.go = c.ds[1]; p.gh = c.ds[2]; p.gn = c.ds[3];
  p.lse = c.lse;
  p.delta = c.delta;
  p.mask = c.mask;
  p.mask_pitch = c.mask_pitch;
  p.dq_scratch = reinterpret_cast<float*>(workspace);
  p.B = (int)B; p.O = (int)O; p.H = (int)H; p.N = (int)N;
  p.q_tiles = (int)((N + 127) / 128);
  p.k_tiles = p.q_tiles;
  const int ks = bwd_key_strip(D);
  p.n_strips = (p.k_tiles + ks - 1) / ks;
  p.bias_broadcast = c.G == 1 && B > 1 ? 1 : 0;
  p.scale = c.scale;
  p.logit_scale = logit_scale(c.scale);
  p.n_items = (int)(B * O * H);
  p.div_h = FastDiv::make((uint32_t)H);
  p.div_o = FastDiv::make((uint32_t)O);
  int grid = sm_count();
  if (grid > p.n_items) grid = p.n_items;
  int* status = nullptr;
  if ((rc = attn_bwd_status_address(&status))) return rc;
  if (D == 16) return launch_attn_bwd<16>(tq, tk, tv, tdo, tb, tdq, tdk, tdv, p, status, grid, stream);
  if (D == 32) return launch_attn_bwd<32>(tq, tk, tv, tdo, tb, tdq, tdk, tdv, p, status, grid, stream);
  return launch_attn_bwd<64>(tq, tk, tv, tdo, tb, tdq, tdk, tdv, p, status, grid, stream);
}

template <int D>
int launch_attn_dbias(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                      const CUtensorMap& tb, const CUtensorMap& tmk, AttnDbiasParams& p, int* status, int grid,
                      cudaStream_t stream) {
  using Cfg = AttnDbiasCfg<D>;
  auto kern = attn_dbias_kernel<Cfg>;
  static PerDeviceOnce once;  // per instantiation
  if (int rc = ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, once)) return rc;
  launch_kernel(kern, dim3(grid), dim3(32 * (Cfg::NCW + 2)), Cfg::SMEM_BYTES, stream, tq, tk, tv, tdo, tb, tmk, p, status);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

// How the outer planes of one dBias tile are split into independent chunks: the split with the shortest schedule, i.e.
// waves of CTAs (one per SM) times planes per CTA, plus about three planes' time for a CTA's start and its partial
// plane.  With one chunk whenever there are more tiles than SMs (N = 1021: 256 tiles) the last wave left half the
// machine idle.  Chunk planes take at most `max_bytes`; one chunk needs none.
// dBias and its fold, us by number of chunks (H = 4, D = 32, O = N; * is what the rule takes, with its workspace):
//   N =  384   1: 312   2: 167   4: 97*    8: 110            9 MiB
//   N =  400   1: 322   2: 174   4: 183    9: 179*          22 MiB
//   N =  512   1: 407   2: 220   9: 226*  16: 257           36 MiB
//   N =  640   1: 509   4: 415   7: 419   10: 425*          62 MiB
//   N =  704   1: 560*  5: 593                               0
//   N =  768   1: 619*  2: 626   4: 648    8: 726            0
//   N = 1024   1: 1688  2: 1761  4: 1585*                   64 MiB
// The count leaves out the fold, which reads every chunk plane; the steps between schedules are larger.  Where the rule misses,
// by 2 to 3 % (N = 400, 512, 640): planes have become a quarter cheaper than when the three were fitted, a CTA's start has not;
// ten planes' time for it would take 2, 2 and 4 chunks there.
static void dbias_plan(int64_t B, int64_t O, int64_t H, int64_t N, int64_t G, double max_bytes, int* n_chunks,
                       int* chunk_len) {
  const int64_t tiles = G * H * ((N + 127) / 128) * ((N + 127) / 128);
  const int64_t planes = (B / G) * O;
  const double chunk_bytes = 4.0 * G * H * N * N;
  const int64_t sms = sm_count();
  int64_t best = 0, best_cost = 0;
  for (int64_t c = 1; c <= planes && (c == 1 || (tiles * c <= 8 * sms && c * chunk_bytes <= max_bytes)); ++c) {
    const int64_t len = (planes + c - 1) / c;
    const int64_t cost = (tiles * c + sms - 1) / sms * (len + 3);
    if (best == 0 || cost < best_cost) {
      best = c;
      best_cost = cost;
    }
  }
  const int64_t len = (planes + best - 1) / best;
  *n_chunks = (int)((planes + len - 1) / len);
  *chunk_len = (int)len;
}

int64_t attn_dbias_workspace_bytes(int64_t B, int64_t O, int64_t H, int64_t N, int64_t G) {
  int c, len;
  dbias_plan(B, O, H, N, G, kNoByteLimit, &c, &len);
  return c > 1 ? (int64_t)c * G * H * N * N * 4 : 0;
}

int64_t attn_dbias_rows_workspace_bytes(int64_t B, int64_t O, int64_t H, int64_t N, int64_t G) {
  int c, len;
  dbias_plan(B, O, H, N, G, kNoByteLimit, &c, &len);
  return (int64_t)c * G * H * N * N * 4;
}

int attn_bwd_dbias(const void* q, const void* k, const void* v, const void* d_out, const int64_t* q_strides,
                   const int64_t* k_strides, const int64_t* v_strides, const float* lse, const float* delta,
                   const float* mask, int64_t mask_pitch, const void* bias, int64_t bias_pitch, int64_t bias_batch,
                   float* dbias, void* workspace, int64_t workspace_bytes, int64_t B, int64_t O, int64_t H, int64_t N,
                   int64_t D, float scale, cudaStream_t stream, double dbias_limit) {
  TPF_REQUIRE(dbias != nullptr, TPF_ERR_INVALID_ARGUMENT, "attn_bwd: dbias is NULL");
  TPF_REQUIRE_ALIGNED16(dbias, "attn_bwd", "dbias");  // rows are written with float4 stores
  AttnCall c = {};
  c.B = B; c.O = O; c.H = H; c.N = N; c.D = D; c.G = bias_batch;
  c.scale = scale;
  c.q = q; c.k = k; c.v = v;
  for (int i = 0; i < 4; ++i) {
    c.qs[i] = q_strides[i];
    c.ks[i] = k_strides[i];
    c.vs[i] = v_strides[i];
  }
  c.mask = mask; c.mask_pitch = mask_pitch;
  c.bias = bias; c.bias_pitch = bias_pitch;
  c.lse = const_cast<float*>(lse);
  c.d_out = d_out;
  c.dos[0] = O * N * H * D; c.dos[1] = N * H * D; c.dos[2] = D; c.dos[3] = H * D;
  c.delta = const_cast<float*>(delta);
  c.dbias = dbias;
  c.dbias_limit = dbias_limit;
  return attn_backward_bias(c, workspace, workspace_bytes, stream);
}

int attn_backward_bias(const AttnCall& c, void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
  const int64_t B = c.B, O = c.O, H = c.H, N = c.N, D = c.D, G = c.G;
  int n_chunks, chunk_len;
  dbias_plan(B, O, H, N, G, c.dbias_limit, &n_chunks, &chunk_len);
  const bool rows = c.dbias == nullptr;  // fp32 planes go to the workspace, bf16 rows come out
  const int64_t need = n_chunks > 1 || rows ? n_chunks * G * H * N * N * 4 : 0;
  TPF_REQUIRE(need == 0 || (workspace && workspace_bytes >= need), TPF_ERR_WORKSPACE,
              "attn_bwd: dBias workspace of %lld bytes required, %lld given", (long long)need,
              (long long)workspace_bytes);
  TPF_REQUIRE(need == 0 || (reinterpret_cast<uintptr_t>(workspace) & 15) == 0, TPF_ERR_WORKSPACE,
              "attn_bwd: dBias workspace must be 16-byte aligned");
  const int swz = 2 * (int)D;
  CUtensorMap tq, tk, tv, tdo, tb, tm;
  int rc;
  if ((rc = make_qkv_tmap(&tq, c.q, B, O, H, N, D, c.qs, swz))) return rc;
  if ((rc = make_qkv_tmap(&tk, c.k, B, O, H, N, D, c.ks, swz))) return rc;
  if ((rc = make_qkv_tmap(&tv, c.v, B, O, H, N, D, c.vs, swz))) return rc;
  if ((rc = make_qkv_tmap(&tdo, c.d_out, B, O, H, N, D, c.dos, swz))) return rc;
  if ((rc = make_bias_tmap(&tb, c.bias, G, H, N, c.bias_pitch))) return rc;
  if ((rc = make_mask_tmap(&tm, c.mask, B, O, N, c.mask_pitch))) return rc;
  AttnDbiasParams p;
  p.part = n_chunks > 1 || rows ? reinterpret_cast<float*>(workspace) : c.dbias;
  p.lse = c.lse;
  p.delta = c.delta;
  p.B = (int)B; p.O = (int)O; p.H = (int)H; p.N = (int)N;
  p.G = (int)G;
  p.planes = (int)((B / G) * O);
  p.n_chunks = n_chunks;
  p.chunk_len = chunk_len;
  p.q_tiles = (int)((N + 127) / 128);
  p.k_tiles = p.q_tiles;
  p.scale = logit_scale(c.scale);
  const int64_t grid = (int64_t)G * H * p.q_tiles * p.k_tiles * n_chunks;
  TPF_REQUIRE(grid < (1ll << 31), TPF_ERR_INVALID_ARGUMENT, "attn_bwd: dBias grid too large");
  int* status = nullptr;
  if ((rc = attn_bwd_status_address(&status))) return rc;
  if (D == 16) rc = launch_attn_dbias<16>(tq, tk, tv, tdo, tb, tm, p, status, (int)grid, stream);
  else if (D == 32) rc = launch_attn_dbias<32>(tq, tk, tv, tdo, tb, tm, p, status, (int)grid, stream);
  else rc = launch_attn_dbias<64>(tq, tk, tv, tdo, tb, tm, p, status, (int)grid, stream);
  if (rc) return rc;
  const int64_t n = rows ? G * N * N : G * H * N * N;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 4 * sm_count()) blocks = 4 * sm_count();
  if (rows) {
    launch_kernel(attn_dbias_rows_kernel, dim3(blocks), dim3(256), 0, stream, p.part,
                  reinterpret_cast<__nv_bfloat16*>(c.dbias_rows), c.dbias_ld, (int)H, N * N, n, n_chunks);
    TPF_LAUNCH_OK();
  } else if (n_chunks > 1) {
    launch_kernel(attn_dbias_fold_kernel, dim3(blocks), dim3(256), 0, stream, p.part, c.dbias, n, n_chunks);
    TPF_LAUNCH_OK();
  }
  return TPF_OK;
}

// =============================================================================================
// Backward with library-owned scratch: for callers that cannot allocate device memory themselves
// =============================================================================================
// Some hosts of this library may not call cudaMalloc (or any allocating routine) around the
// backward pass: code running between graph-capture begin/end, real-time or plugin hosts whose
// memory is handed out once at start-up, and foreign runtimes that own the device heap.  For them
// the scratch of the backward pass (per-CTA dQ running sums, dBias chunk planes) lives in a fixed
// array that is part of the library image.  Every GPU that loads the library holds these
// kStaticScratchBytes until the process exits.
constexpr int64_t kStaticScratchBytes = 16ll << 20;  // 16 MiB
static __device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

int64_t attn_bwd_static_scratch_capacity() { return kStaticScratchBytes; }

// In host code `g_static_scratch` is only a handle for the runtime, not a device address; the
// address is looked up once per device (with that device current) and cached.
static int static_scratch_address(void** out) {
  static PerDeviceAddress cache;
  int rc = device_symbol_address(g_static_scratch, cache, out);
  if (rc) return rc;
  TPF_REQUIRE((reinterpret_cast<uintptr_t>(*out) & 255) == 0, TPF_ERR_CUDA,
              "static scratch address lookup returned a misaligned pointer");
  return TPF_OK;
}

int attn_bwd_static_scratch(const void* q, const void* k, const void* v, const void* d_out, const int64_t* q_strides,
                            const int64_t* k_strides, const int64_t* v_strides, const void* out, const float* lse,
                            const float* mask, int64_t mask_pitch, const void* bias, int64_t bias_pitch,
                            int64_t bias_batch, void* dq, void* dk, void* dv, float* dbias, float* delta, int64_t B,
                            int64_t O, int64_t H, int64_t N, int64_t D, float scale, cudaStream_t stream) {
  TPF_REQUIRE(B > 0 && O > 0 && H > 0 && N > 0 && (bias_batch == 1 || bias_batch == B), TPF_ERR_INVALID_ARGUMENT,
              "attn_bwd (library scratch): bad extents");
  TPF_REQUIRE(D == 16 || D == 32 || D == 64, TPF_ERR_UNSUPPORTED,
              "attn_bwd (library scratch): head dim %lld not in {16,32,64}", (long long)D);
  const int64_t ws_a = (attn_bwd_workspace_bytes(B, O, H, N, D) + 255) / 256 * 256;
  // The dQ sums have to fit; dBias takes as many chunk planes as the rest of the array holds, down to one chunk, which
  // needs none.  (Chunks planned without that limit took up to 8 * SMs tiles of 64 KiB: N = 640, H = 4 would need 74 MiB.)
  TPF_REQUIRE(ws_a <= kStaticScratchBytes, TPF_ERR_WORKSPACE,
              "attn_bwd (library scratch): this shape needs %lld bytes of scratch, the built-in array holds %lld; "
              "use tpf_attn_bwd with a caller-provided workspace",
              (long long)ws_a, (long long)kStaticScratchBytes);
  const int64_t ws_b = kStaticScratchBytes - ws_a;
  void* base = nullptr;
  int rc = static_scratch_address(&base);
  if (rc) return rc;
  // Nothing in the scratch has to start at zero: the dQ running sums are written by the first key
  // strip before they are read, and every dBias chunk plane is fully overwritten.
  rc = attn_bwd_dqkv(q, k, v, d_out, q_strides, k_strides, v_strides, out, lse, mask, mask_pitch, bias, bias_pitch,
                     bias_batch, dq, dk, dv, delta, base, ws_a, B, O, H, N, D, scale, 3, stream);
  if (rc) return rc;
  return attn_bwd_dbias(q, k, v, d_out, q_strides, k_strides, v_strides, lse, delta, mask, mask_pitch, bias,
                        bias_pitch, bias_batch, dbias, static_cast<char*>(base) + ws_a, ws_b, B, O, H, N, D, scale,
                        stream, (double)ws_b);
}

}  // namespace tpf
