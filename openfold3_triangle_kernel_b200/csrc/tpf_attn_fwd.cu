// Triangle-attention forward for sm_100a.
//
//   S[q,k]  = (Q K^T)[q,k] * scale + mask[k] + bias[q,k]      (fp32, logits never leave the SM)
//   out     = softmax_k(S) V  -> bf16 [B,O,N,H,D];   lse = logsumexp_k(S) -> fp32 [B,O,H,N]
//
// Stands in for the reference forward kernels
// (openfold3/core/kernels/turbopairformer/turbopairformer_triangle_forward.cu:775-1256 and :451-766):
// same math and rounding points (fp32 running max / sum, probabilities rounded to bf16 for P V,
// fully masked rows give out = 0 and lse = -inf), different machine mapping:
//
//  * A work item is one (b, o, h, 128-query tile); a CTA walks its items and, inside an item, the 64-key tiles.
//    Three CTAs (two at D = 64) of five warps share an SM: four softmax warps with one thread per query row
//    (= TMEM lane), and one warp that issues every TMA load and UMMA.
//  * A softmax thread holds the 64 logits of its row in registers: one pass of TMEM loads (after which Q K^T of a later
//    tile may use the buffer), bias add, maximum, exponentials, row sum.  What bounds the kernel is the length of that
//    instruction stream (about 440 instructions per tile and warp against 64 exponentials; the MUFU pipe is half busy)
//    so it carries no bookkeeping: S and P are double-buffered, and the issuing warp needs no "empty" barriers (see
//    there).  The bf16 probabilities overwrite their S buffer in TMEM and P V takes them as its A operand; O accumulates
//    in TMEM across key tiles.
//  * The reference maximum of a row is raised - and the row's partial results rescaled - only when a tile exceeds
//    it by more than a fixed gap.
//  * The finished row of an item is normalised, gated and stored under the next item's first tile, when its last P V
//    has long completed.
//  * Items are numbered with the query tile fastest: CTAs running at the same time share K and V of an outer row (and
//    each bias strip stays in L2 anyway).  With the outer row fastest K and V came from DRAM once per query tile.
//  * A tile whose mask row is all zero and that has no ragged key tail (the common case) skips the mask add; warps
//    whose 32 query rows lie beyond N, the second half of a key tile with at most 32 keys, and the exponentials of a tile
//    whose keys are all masked, are skipped.
//
// Measured (B200, H = 4, D = 32, cold L2, 5 % of the keys masked): N = 384 102 us, N = 768 711, N = 1021 1.66 ms;
// D = 64, N = 257 74 us.  Before the tiles with a mask got code of their own and one store path for an item's rows: 109, 765,
// 1.78 and 78.
#include "tpf_host.cuh"
#include "tpf_internal.h"
#include "tpf_ptx.cuh"

namespace tpf {

static __device__ int g_attn_fwd_status;

int attn_fwd_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  TPF_CUDA_OK(cudaMemcpyFromSymbol(&v, g_attn_fwd_status, sizeof(int)));
  if (v) TPF_CUDA_OK(cudaMemcpyToSymbol(g_attn_fwd_status, &zero, sizeof(int)));
  *out = v;
  return TPF_OK;
}

struct AttnFwdParams {
  __nv_bfloat16* out;
  int64_t ob, oo, oh, on;   // element strides of out
  const __nv_bfloat16* gate;  // logits of the output gate, or null
  int64_t gb, go, gh, gn;
  float* lse;          // [B,O,H,N] or null
  int B, O, H, N;
  int q_tiles, k_tiles;  // 128-query tiles, 64-key tiles
  int bias_broadcast;    // 1: one bias for all b
  float scale;           // softmax scale applied to Q K^T
  int n_items;
};

template <int D_>
struct AttnFwdCfg {
  static constexpr int D = D_;
  static constexpr int KEYS = 64;                // keys per tile
  static constexpr int CTAS_PER_SM = D <= 32 ? 3 : 2;
  static constexpr int SWZ = 2 * D;              // bytes per smem row of a Q/K/V tile
  static constexpr int Q_TILE = 128 * D * 2;
  static constexpr int KV_TILE = KEYS * D * 2;
  static constexpr int NS = 3;                   // K / mask slots
  static constexpr int NB = 2;                   // bias / V slots
  static constexpr int BIAS_STAGE = 128 * KEYS * 2;
  static constexpr int OFF_BIAS = 0;
  static constexpr int OFF_Q = OFF_BIAS + NB * BIAS_STAGE;       // [2]
  static constexpr int OFF_K = OFF_Q + 2 * Q_TILE;               // [NS]
  static constexpr int OFF_V = OFF_K + NS * KV_TILE;             // [NB]
  static constexpr int OFF_MASK = OFF_V + NB * KV_TILE;          // [NS] x 256 B
  static constexpr int OFF_BAR = OFF_MASK + NS * 256;
  static constexpr int N_BAR = NB + 2 + NS + 6;
  static constexpr int SMEM_BYTES = OFF_BAR + N_BAR * 8 + 32 + 1024;
  // two S buffers (fp32, 64 columns); the bf16 probabilities of a tile overwrite the first 32 columns of its S buffer
  static constexpr int S_COLS = 128;
  static constexpr int O_COLS = D <= 32 ? 32 : 64;
  static constexpr int THREADS = 160;            // 4 softmax warps, one warp that issues TMA loads and UMMAs
  static constexpr int WARP_MMA = 4;
  static_assert(D == 16 || D == 32 || D == 64, "head dim lanes");
  static_assert((S_COLS + O_COLS) * CTAS_PER_SM <= 512, "TMEM budget");
  static_assert((SMEM_BYTES + 1024) * CTAS_PER_SM <= 233472, "shared memory budget");
  static_assert(KV_TILE % 1024 == 0 && Q_TILE % 1024 == 0, "tile buffers keep 1024-byte alignment");
};

template <bool B>
struct BoolTag {
  static constexpr bool value = B;
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::CTAS_PER_SM)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmBias,
                const __grid_constant__ CUtensorMap tmMask, const AttnFwdParams p, int* __restrict__ status) {
  griddep_wait();
  constexpr int D = Cfg::D, NS = Cfg::NS, NB = Cfg::NB, KEYS = Cfg::KEYS;
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* smem = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* b_full = bars;                  // [NB]
  uint64_t* q_full = b_full + NB;           // [2]
  uint64_t* k_full = q_full + 2;            // [NS]
  uint64_t* s_full = k_full + NS;          // [2]
  uint64_t* p_ready = s_full + 2;           // [2]
  uint64_t* pv_done = p_ready + 2;          // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + Cfg::N_BAR);  // S, O
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 2);
  const WaitCtx wctx{abort_flag, status};

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < NB; ++s) mbar_init(&b_full[s], 1);
    for (int s = 0; s < NS; ++s) mbar_init(&k_full[s], 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_ready[s], 4);
      mbar_init(&pv_done[s], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmBias);
    tma_prefetch_desc(&tmMask);
  }
  if (warp == Cfg::WARP_MMA) {
    tmem_alloc(tmem_slot, Cfg::S_COLS);
    tmem_alloc(tmem_slot + 1, Cfg::O_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_s = tmem_slot[0], tmem_o = tmem_slot[1];

  const int KT = p.k_tiles;

  // item -> (b, h, o, qt), the query tile fastest.
  // The coordinates are a mixed-radix counter advanced by the grid size: the divisions happen once, not per
  // item (an integer division by a run-time value costs a warp several hundred cycles on its critical path).
  struct ItemWalk {
    int qt, o, h, b;      // current item
    int sq, so, sh, sb;   // the step, decomposed
    int Q, O, H;
    __device__ void init(int item, int step, int O_, int Q_, int H_) {
      O = O_; Q = Q_; H = H_;
      qt = item % Q; int r = item / Q;
      o = r % O; r /= O;
      h = r % H; b = r / H;
      sq = step % Q; r = step / Q;
      so = r % O; r /= O;
      sh = r % H; sb = r / H;
    }
    __device__ __forceinline__ void next() {
      qt += sq;
      int c = qt >= Q ? 1 : 0;
      qt -= c * Q;
      o += so + c;
      c = o >= O ? 1 : 0;
      o -= c * O;
      h += sh + c;
      c = h >= H ? 1 : 0;
      h -= c * H;
      b += sb + c;
    }
  };

  if (warp == Cfg::WARP_MMA) {
    // ------------------------------------------------------------------ TMA loads and UMMAs
    // One thread issues both.  p_ready(t) says that the softmax warps have read S, bias and mask of tile t, and the
    // completion of P V (t) that every buffer of tile t is free: no "empty" barriers are needed.  Q K^T runs two tiles
    // ahead of P V (its S buffer is free once P V (t), whose P lies in it, is done), K / mask loads run three
    // tiles ahead, bias and V loads two.
    {
      const uint32_t el = elect_one();
      constexpr uint32_t idesc_qk = make_idesc_bf16(128, KEYS, false, false);
      constexpr uint32_t idesc_pv = make_idesc_bf16(128, D, false, true);
      constexpr uint32_t swz = swizzle_mode_for_bytes(Cfg::SWZ);
      const uint64_t q_desc0 = make_smem_desc(smem_u32(smem + Cfg::OFF_Q), 16, 8 * Cfg::SWZ, swz);
      const uint64_t k_desc0 = make_smem_desc(smem_u32(smem + Cfg::OFF_K), 16, 8 * Cfg::SWZ, swz);
      const uint64_t v_desc0 = make_smem_desc(smem_u32(smem + Cfg::OFF_V), KEYS * Cfg::SWZ, 8 * Cfg::SWZ, swz);
      const int my_items = (p.n_items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
      const int tiles = my_items * KT;

      // K / mask stream (and Q, at an item's first tile)
      ItemWalk kw;
      kw.init(blockIdx.x, gridDim.x, p.O, p.q_tiles, p.H);
      int kj = 0, k_s = 0, kq = 0;
      auto load_k = [&]() {
        if (kj == 0) {
          mbar_expect_tx(el, &q_full[kq], Cfg::Q_TILE);
          tma_load_5d(el, smem + Cfg::OFF_Q + kq * Cfg::Q_TILE, &tmQ, &q_full[kq], 0, kw.qt * 128, kw.h, kw.o, kw.b);
          kq ^= 1;
        }
        mbar_expect_tx(el, &k_full[k_s], Cfg::KV_TILE + 256);
        tma_load_5d(el, smem + Cfg::OFF_K + k_s * Cfg::KV_TILE, &tmK, &k_full[k_s], 0, kj * KEYS, kw.h, kw.o, kw.b);
        tma_load_3d(el, smem + Cfg::OFF_MASK + k_s * 256, &tmMask, &k_full[k_s], kj * KEYS, kw.o, kw.b);
        if (++k_s == NS) k_s = 0;
        if (++kj == KT) {
          kj = 0;
          kw.next();
        }
      };
      // bias / V stream
      ItemWalk bw;
      bw.init(blockIdx.x, gridDim.x, p.O, p.q_tiles, p.H);
      int bj = 0, b_s = 0;
      auto load_bv = [&]() {
        mbar_expect_tx(el, &b_full[b_s], Cfg::BIAS_STAGE + Cfg::KV_TILE);
        tma_load_4d(el, smem + Cfg::OFF_BIAS + b_s * Cfg::BIAS_STAGE, &tmBias, &b_full[b_s], bj * KEYS, bw.qt * 128, bw.h,
                    p.bias_broadcast ? 0 : bw.b);
        tma_load_5d(el, smem + Cfg::OFF_V + b_s * Cfg::KV_TILE, &tmV, &b_full[b_s], 0, bj * KEYS, bw.h, bw.o, bw.b);
        b_s ^= 1;
        if (++bj == KT) {
          bj = 0;
          bw.next();
        }
      };
      // Q K^T stream
      int qj = 0, q_s = 0, qk_s = 0, qk_buf = 0;
      uint32_t q_ph = 0, qk_ph = 0;
      auto issue_qk = [&]() {
        if (qj == 0) warp_wait2(&q_full[q_s], q_ph, &k_full[qk_s], qk_ph, wctx);
        else warp_wait(&k_full[qk_s], qk_ph, wctx);
        const uint64_t qd = q_desc0 + (uint64_t)((q_s * Cfg::Q_TILE) >> 4);
        const uint64_t kd = k_desc0 + (uint64_t)((qk_s * Cfg::KV_TILE) >> 4);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks)
          umma_ss(el, tmem_s + 64 * qk_buf, qd + 2 * ks, kd + 2 * ks, idesc_qk, ks != 0);
        umma_commit(el, &s_full[qk_buf]);
        qk_buf ^= 1;
        if (++qk_s == NS) {
          qk_s = 0;
          qk_ph ^= 1;
        }
        if (++qj == KT) {
          qj = 0;
          q_s ^= 1;
          if (q_s == 0) q_ph ^= 1;
        }
      };

      load_k();
      load_bv();
      if (tiles > 1) {
        load_k();
        load_bv();
      }
      if (tiles > 2 && KT > 1) load_k();
      issue_qk();
      if (tiles > 1) issue_qk();
      if (tiles > 2 && KT == 1) {
        // the third tile is the third item, whose Q goes where the first one's lies: not before that has been used
        warp_wait(&s_full[0], 0, wctx);
        load_k();
      }
      int j = 0;
      for (int t = 0; t < tiles; ++t) {
        const int buf = t & 1;
        const uint32_t ph = (t >> 1) & 1;
        warp_wait(&p_ready[buf], ph, wctx);
        tc_fence_after();
        const uint64_t vd = v_desc0 + (uint64_t)((buf * Cfg::KV_TILE) >> 4);
        // 16 keys per step; A = P from TMEM (8 columns of bf16 pairs).  A tail of at most 32 keys has no P beyond them.
        const bool half = j + 1 == KT && p.N - j * KEYS <= 32;
#pragma unroll
        for (int ks = 0; ks < KEYS / 16; ++ks)
          if (ks < 2 || !half)
            umma_ts(el, tmem_o, tmem_s + 64 * buf + 8 * ks, vd + (uint64_t)(ks * Cfg::SWZ), idesc_pv, (ks | j) != 0);
        umma_commit(el, &pv_done[buf]);
        if (++j == KT) j = 0;
        if (t + 2 < tiles) {
          warp_wait(&pv_done[buf], ph, wctx);
          tc_fence_after();
          issue_qk();
          load_bv();
          if (t + 3 < tiles) load_k();
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax warps: one thread per query row
    const int row = 32 * warp + lane;  // query row inside the tile == TMEM lane
    const uint32_t t_s = tmem_addr(tmem_s, 32 * warp, 0);
    const uint32_t t_o = tmem_addr(tmem_o, 32 * warp, 0);
    constexpr float kLog2e = 1.4426950408889634f;
    constexpr float kLn2 = 0.6931471805599453f;
    constexpr float kGap = 12.0f;  // largest exponent (natural units) a probability may have relative to m
    // A maximum below this belongs to a row that has met masked keys only, by a large finite value.  From 2^31 on m log2(e) is
    // rounded by up to 2^7: the exponentials, made with one fma, would be infinite or zero.  Such a row subtracts m first.
    constexpr float kFar = -1.4e9f;
    const uint64_t scale2 = f2_pack(p.scale, p.scale);
    const uint64_t log2e2 = f2_pack(kLog2e, kLog2e);

    int m_s = 0;
    int t = 0;  // tiles done by this CTA: tile t uses S / P buffer t & 1 for the (t >> 1)-th time
    bool pend = false;
    int f_q = 0, f_b = 0, f_o = 0, f_h = 0;
    float f_m = 0.f, f_l = 0.f;
    // normalise, gate and store the output row of the item whose last P V was tile t - 1
    auto finish_item = [&]() {
      warp_wait(&pv_done[(t - 1) & 1], ((t - 1) >> 1) & 1, wctx);
      tc_fence_after();
      const float inv = f_l > 0.f ? __fdividef(1.f, f_l) : 0.f;
      const bool f_ok = f_q < p.N;
      __nv_bfloat16* f_out = p.out + f_b * p.ob + f_o * p.oo + f_h * p.oh + (int64_t)f_q * p.on;
      const __nv_bfloat16* f_gate = p.gate + f_b * p.gb + f_o * p.go + f_h * p.gh + (int64_t)f_q * p.gn;
#pragma unroll
      for (int c = 0; c < D; c += 16) {
        uint32_t ro[16];
        tmem_ld16(t_o + c, ro);
        uint4 g0 = make_uint4(0u, 0u, 0u, 0u), g1 = g0;
        if (p.gate != nullptr && f_ok) {
          g0 = *reinterpret_cast<const uint4*>(f_gate + c);
          g1 = *reinterpret_cast<const uint4*>(f_gate + c + 8);
        }
        tmem_ld_wait();
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(ro[i]) * inv;
        if (p.gate != nullptr) {
          const uint32_t gw[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            v[2 * i] *= sigmoid_rel(__uint_as_float(gw[i] << 16));
            v[2 * i + 1] *= sigmoid_rel(__uint_as_float(gw[i] & 0xFFFF0000u));
          }
        }
        if (f_ok) {
          *reinterpret_cast<uint4*>(f_out + c) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                                                            pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
          *reinterpret_cast<uint4*>(f_out + c + 8) = make_uint4(pack_bf16x2(v[8], v[9]), pack_bf16x2(v[10], v[11]),
                                                                pack_bf16x2(v[12], v[13]), pack_bf16x2(v[14], v[15]));
        }
      }
      if (f_ok && p.lse != nullptr)
        p.lse[(((int64_t)f_b * p.O + f_o) * p.H + f_h) * p.N + f_q] = f_l > 0.f ? f_m + log2f(f_l) * kLn2 : -INFINITY;
    };

    ItemWalk iw;
    iw.init(blockIdx.x, gridDim.x, p.O, p.q_tiles, p.H);
    for (int item = blockIdx.x; item < p.n_items; item += gridDim.x, iw.next()) {
      float m_use = -INFINITY, l_run = 0.f;
      const bool live = iw.qt * 128 + 32 * warp < p.N;  // a warp without query rows only keeps the barriers going
      for (int j = 0; j < KT; ++j, ++t) {
        const int buf = t & 1;
        const uint32_t ph = (t >> 1) & 1;
        // s_full completes after Q K^T of this tile, hence after the K tile and the mask row that
        // arrives on the same barrier have landed
        warp_wait2(&s_full[buf], ph, &b_full[buf], ph, wctx);
        tc_fence_after();
        float* mask_row = reinterpret_cast<float*>(smem + Cfg::OFF_MASK + m_s * 256);
        if (++m_s == NS) m_s = 0;
        const int n_keys = p.N - j * KEYS;
        const float2 mprobe = *reinterpret_cast<const float2*>(mask_row + 2 * lane);
        const bool general = n_keys < KEYS || __any_sync(0xffffffffu, (mprobe.x != 0.f) || (mprobe.y != 0.f));
        const uint8_t* bias_row = smem + Cfg::OFF_BIAS + buf * Cfg::BIAS_STAGE + row * 128;
        // A tile from its logits to its probabilities.  GENERAL: with a mask or a ragged tail.  Two copies, because as a
        // branch between the bias and the maximum it cost every tile: the 64 logits had to be in the same registers on
        // both ways, and the stages before and after it could not be interleaved.
        auto tile = [&](auto general_tag) {
          constexpr bool GENERAL = decltype(general_tag)::value;
          if (GENERAL && n_keys < KEYS) {
            // no keys there: every warp writes the same values over the zeros that the copy filled in
            if (lane >= n_keys) mask_row[lane] = -INFINITY;
            if (lane + 32 >= n_keys) mask_row[lane + 32] = -INFINITY;
            fence_async_smem();  // the next copy into this slot comes after these stores
            __syncwarp();
          }
          uint32_t raw[64];  // this row's logits
          tmem_ld32(t_s + 64 * buf, *reinterpret_cast<uint32_t(*)[32]>(raw));
          tmem_ld32(t_s + 64 * buf + 32, *reinterpret_cast<uint32_t(*)[32]>(raw + 32));
          tmem_ld_wait();
          // Keys that are not there (key 63 is one in a tail tile) are zeros, and an infinite query times zero is a NaN, which
          // -inf does not mask.
          if (GENERAL && n_keys < KEYS && __any_sync(0xffffffffu, __uint_as_float(raw[63]) != 0.f)) {
#pragma unroll
            for (int i = 0; i < 64; ++i)
              if (i >= n_keys) raw[i] = 0u;
          }
          float cm0 = -INFINITY, cm1 = -INFINITY;
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            if (GENERAL && u == 4 && n_keys <= 32) break;
            const uint4 bv = *reinterpret_cast<const uint4*>(bias_row + ((u ^ (row & 7)) << 4));
            const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
            float4 mk[2];
            if (GENERAL) {
              mk[0] = *reinterpret_cast<const float4*>(mask_row + 8 * u);
              mk[1] = *reinterpret_cast<const float4*>(mask_row + 8 * u + 4);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int i = 8 * u + 2 * e;
              uint64_t v = f2_fma(f2_pack_bits(raw[i], raw[i + 1]), scale2, f2_pack_bits(bw[e] << 16, bw[e] & 0xFFFF0000u));
              if (GENERAL) v = f2_add(v, e & 1 ? f2_pack(mk[e >> 1].z, mk[e >> 1].w) : f2_pack(mk[e >> 1].x, mk[e >> 1].y));
              float v0, v1;
              f2_unpack(v, v0, v1);
              raw[i] = __float_as_uint(v0);
              raw[i + 1] = __float_as_uint(v1);
              float& cm = e & 1 ? cm1 : cm0;
              cm = GENERAL ? max3_nan(cm, v0, v1) : max3(cm, v0, v1);
            }
          }
          const float cmax = GENERAL ? max3_nan(cm0, cm1, cm1) : fmaxf(cm0, cm1);
          if (__any_sync(0xffffffffu, cmax > (m_use < kFar ? -INFINITY : m_use + kGap))) {
            // Raise the reference maximum of the rows that need it (f = 1 for the others) and rescale what
            // those rows have accumulated.  Runs for the first finite tile of every row and then only
            // when the logits of a row grow by more than kGap, or while a row has nothing but keys far below zero.
            const bool grow = cmax > m_use + kGap;
            const float f = grow ? ex2_approx((m_use - cmax) * kLog2e) : 1.f;  // m_use = -inf gives 0; nothing accumulated then
            if (grow) m_use = cmax;
            l_run *= f;
            if (j > 0) {
              warp_wait(&pv_done[(t - 1) & 1], ((t - 1) >> 1) & 1, wctx);
              tc_fence_after();
#pragma unroll 1
              for (int cc = 0; cc < D; cc += 8) {
                uint32_t ro[8];
                tmem_ld8(t_o + cc, ro);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i) ro[i] = __float_as_uint(__uint_as_float(ro[i]) * f);
                tmem_st8(t_o + cc, ro);
              }
            }
            const float shift = m_use < kFar && m_use != -INFINITY ? m_use : 0.f;
            if (__any_sync(0xffffffffu, shift != 0.f)) {
#pragma unroll
              for (int i = 0; i < 64; ++i) raw[i] = __float_as_uint(__uint_as_float(raw[i]) - shift);
            }
          }
          if (GENERAL && !__any_sync(0xffffffffu, !(cmax < m_use - 104.f))) {
            // masked keys only: every probability is below the smallest fp32 number (no NaN among the logits either)
            const uint32_t zero[8] = {};
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_st8(t_s + 64 * buf + 8 * c, zero);
            return;
          }
          const float neg_m = m_use < kFar ? 0.f : -m_use * kLog2e;
          const uint64_t neg_m2 = f2_pack(neg_m, neg_m);
          uint64_t rs2a = 0ull, rs2b = 0ull;  // packed partial row sums of this tile
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (GENERAL && c == 2 && n_keys <= 32) break;
            uint32_t pk[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              float a0, a1;
              f2_unpack(f2_fma(f2_pack_bits(raw[16 * c + 2 * e], raw[16 * c + 2 * e + 1]), log2e2, neg_m2), a0, a1);
              const float e0 = ex2_approx(a0), e1 = ex2_approx(a1);
              if (e & 1) rs2b = f2_add(rs2b, f2_pack(e0, e1));
              else rs2a = f2_add(rs2a, f2_pack(e0, e1));
              pk[e] = pack_bf16x2(e0, e1);
            }
            tmem_st8(t_s + 64 * buf + 8 * c, pk);
          }
          float r0, r1;
          f2_unpack(f2_add(rs2a, rs2b), r0, r1);
          l_run += r0 + r1;
        };
        if (!live) {
        } else if (general) tile(BoolTag<true>{});
        else tile(BoolTag<false>{});
        // the previous item's row leaves before this item's first P V overwrites the accumulator
        if (j == 0 && pend) finish_item();
        if (j == 0) pend = false;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_ready[buf]);
      }
      pend = live;
      f_q = iw.qt * 128 + row; f_b = iw.b; f_o = iw.o; f_h = iw.h;
      f_m = m_use;
      f_l = l_run;
    }
    if (pend) finish_item();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::WARP_MMA) {
    __syncwarp();
    tmem_dealloc(tmem_s, Cfg::S_COLS);
    tmem_dealloc(tmem_o, Cfg::O_COLS);
  }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------

// 5-D map over a [B,O,H,N,D] bf16 tensor with element strides (sb, so, sh, sn), D contiguous.
// `rows` = sequence positions per box.
int make_qkv_tmap_rows(CUtensorMap* tm, const void* base, int64_t B, int64_t O, int64_t H, int64_t N, int64_t D,
                       const int64_t* st, int swz, int rows) {
  uint64_t dims[5] = {(uint64_t)D, (uint64_t)N, (uint64_t)H, (uint64_t)O, (uint64_t)B};
  uint64_t strides[4] = {(uint64_t)st[3] * 2, (uint64_t)st[2] * 2, (uint64_t)st[1] * 2, (uint64_t)st[0] * 2};
  uint32_t box[5] = {(uint32_t)D, (uint32_t)rows, 1, 1, 1};
  return make_tmap_bf16(tm, base, 5, dims, strides, box, swz);
}
int make_qkv_tmap(CUtensorMap* tm, const void* base, int64_t B, int64_t O, int64_t H, int64_t N, int64_t D,
                  const int64_t* st, int swz) {
  return make_qkv_tmap_rows(tm, base, B, O, H, N, D, st, swz, 128);
}

// 4-D map over the bf16 bias [Bb,H,N,N] whose rows are `pitch` elements apart.
int make_bias_tmap(CUtensorMap* tm, const void* base, int64_t Bb, int64_t H, int64_t N, int64_t pitch) {
  uint64_t dims[4] = {(uint64_t)N, (uint64_t)N, (uint64_t)H, (uint64_t)Bb};
  uint64_t strides[3] = {(uint64_t)pitch * 2, (uint64_t)pitch * N * 2, (uint64_t)pitch * N * H * 2};
  uint32_t box[4] = {64, 128, 1, 1};
  return make_tmap_bf16(tm, base, 4, dims, strides, box, 128);
}

// The same with boxes of 128 x 128, not swizzled.
int make_bias_tmap_plain(CUtensorMap* tm, const void* base, int64_t Bb, int64_t H, int64_t N, int64_t pitch) {
  uint64_t dims[4] = {(uint64_t)N, (uint64_t)N, (uint64_t)H, (uint64_t)Bb};
  uint64_t strides[3] = {(uint64_t)pitch * 2, (uint64_t)pitch * N * 2, (uint64_t)pitch * N * H * 2};
  uint32_t box[4] = {128, 128, 1, 1};
  return make_tmap_bf16(tm, base, 4, dims, strides, box, 0);
}

// 3-D map over the fp32 additive mask [B,O,N] whose rows are `pitch` elements apart.
int make_mask_tmap_cols(CUtensorMap* tm, const void* base, int64_t B, int64_t O, int64_t N, int64_t pitch, int cols) {
  uint64_t dims[3] = {(uint64_t)N, (uint64_t)O, (uint64_t)B};
  uint64_t strides[2] = {(uint64_t)pitch * 4, (uint64_t)pitch * O * 4};
  uint32_t box[3] = {(uint32_t)cols, 1, 1};
  return make_tmap_f32(tm, base, 3, dims, strides, box);
}
int make_mask_tmap(CUtensorMap* tm, const void* base, int64_t B, int64_t O, int64_t N, int64_t pitch) {
  return make_mask_tmap_cols(tm, base, B, O, N, pitch, 128);
}

template <int D>
int launch_attn_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tb,
                    const CUtensorMap& tmk, const AttnFwdParams& p, int* status, cudaStream_t stream) {
  using Cfg = AttnFwdCfg<D>;
  auto kern = attn_fwd_kernel<Cfg>;
  static PerDeviceOnce once;  // per instantiation
  if (int rc = ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, once)) return rc;
  int grid = Cfg::CTAS_PER_SM * sm_count();
  if (grid > p.n_items) grid = p.n_items;
  launch_kernel(kern, dim3(grid), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, stream, tq, tk, tv, tb, tmk, p, status);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

int attn_forward(const AttnCall& c, cudaStream_t stream) {
  const int64_t B = c.B, O = c.O, H = c.H, N = c.N, D = c.D;
  TPF_REQUIRE(c.q && c.k && c.v && c.mask && c.bias && c.out, TPF_ERR_INVALID_ARGUMENT, "attn_fwd: null pointer");
  TPF_REQUIRE(B > 0 && O > 0 && H > 0 && N > 0, TPF_ERR_INVALID_ARGUMENT, "attn_fwd: B,O,H,N must be positive");
  TPF_REQUIRE(D == 16 || D == 32 || D == 64, TPF_ERR_UNSUPPORTED,
              "attn_fwd: head dim %lld not in {16,32,64} (pad on the host side)", (long long)D);
  TPF_REQUIRE(c.G == 1 || c.G == B, TPF_ERR_INVALID_ARGUMENT, "attn_fwd: bias batch must be 1 or B");
  TPF_REQUIRE(c.bias_pitch >= N && c.bias_pitch % 8 == 0, TPF_ERR_INVALID_ARGUMENT,
              "attn_fwd: bias row pitch must be >= N and a multiple of 8 elements");
  TPF_REQUIRE(c.mask_pitch >= N && c.mask_pitch % 4 == 0, TPF_ERR_INVALID_ARGUMENT,
              "attn_fwd: mask row pitch must be >= N and a multiple of 4 elements");
  TPF_REQUIRE(N <= (1 << 24) && B * O * H < (1ll << 31), TPF_ERR_INVALID_ARGUMENT, "attn_fwd: extent too large");
  TPF_REQUIRE_ALIGNED16(c.out, "attn_fwd", "out");
  TPF_REQUIRE((reinterpret_cast<uintptr_t>(c.lse) & 3) == 0, TPF_ERR_INVALID_ARGUMENT,
              "attn_fwd: lse must be 4-byte aligned");
  const int swz = 2 * (int)D;
  CUtensorMap tq, tk, tv, tb, tm;
  int rc;
  if ((rc = make_qkv_tmap(&tq, c.q, B, O, H, N, D, c.qs, swz))) return rc;
  if ((rc = make_qkv_tmap_rows(&tk, c.k, B, O, H, N, D, c.ks, swz, 64))) return rc;
  if ((rc = make_qkv_tmap_rows(&tv, c.v, B, O, H, N, D, c.vs, swz, 64))) return rc;
  if ((rc = make_bias_tmap(&tb, c.bias, c.G, H, N, c.bias_pitch))) return rc;
  if ((rc = make_mask_tmap_cols(&tm, c.mask, B, O, N, c.mask_pitch, 64))) return rc;
  AttnFwdParams p;
  p.out = reinterpret_cast<__nv_bfloat16*>(c.out);
  p.ob = c.os[0]; p.oo = c.os[1]; p.oh = c.os[2]; p.on = c.os[3];
  p.gate = reinterpret_cast<const __nv_bfloat16*>(c.gate);
  p.gb = c.gs[0]; p.go = c.gs[1]; p.gh = c.gs[2]; p.gn = c.gs[3];
  p.lse = c.lse;
  p.B = (int)B; p.O = (int)O; p.H = (int)H; p.N = (int)N;
  p.q_tiles = (int)((N + 127) / 128);
  p.k_tiles = (int)((N + 63) / 64);
  p.bias_broadcast = c.G == 1 && B > 1 ? 1 : 0;
  p.scale = c.scale;
  const int64_t items = B * H * p.q_tiles * O;
  TPF_REQUIRE(items < (1ll << 31), TPF_ERR_INVALID_ARGUMENT, "attn_fwd: too many work items");
  p.n_items = (int)items;
  int* status = nullptr;
  {
    static PerDeviceAddress cache;
    if ((rc = device_symbol_address(g_attn_fwd_status, cache, reinterpret_cast<void**>(&status)))) return rc;
  }
  if (D == 16) return launch_attn_fwd<16>(tq, tk, tv, tb, tm, p, status, stream);
  if (D == 32) return launch_attn_fwd<32>(tq, tk, tv, tb, tm, p, status, stream);
  return launch_attn_fwd<64>(tq, tk, tv, tb, tm, p, status, stream);
}

int attn_fwd(const void* q, const void* k, const void* v, const int64_t* q_strides, const int64_t* k_strides,
             const int64_t* v_strides, const float* mask, int64_t mask_pitch, const void* bias, int64_t bias_pitch,
             int64_t bias_batch, void* out, float* lse, int64_t B, int64_t O, int64_t H, int64_t N, int64_t D,
             float scale, cudaStream_t stream) {
  TPF_REQUIRE(lse, TPF_ERR_INVALID_ARGUMENT, "attn_fwd: null pointer");
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
  c.out = out;
  c.os[0] = O * N * H * D; c.os[1] = N * H * D; c.os[2] = D; c.os[3] = H * D;
  c.lse = lse;
  return attn_forward(c, stream);
}

}  // namespace tpf
