// Triangle multiplicative update, forward: the two kernels around the k-contraction, each with its LayerNorm inside
// (C = 64 and 128).
//
//   project:  zln = LN(z);  a = mask (zln Wap^T) sigmoid(zln Wag^T), b likewise           -> channel-major
//   output :  out = (LN(x) Wz^T) sigmoid(LN(z) Wg^T)  [+ z],   x = contraction, channel-major
//
// What bounds the update is passes over [R, C] tensors: with separate norms and a stored gate it makes 14 of them, here 9
// when nothing is kept for a backward.  The normalised rows are never an operand: the tensor cores work on the rows as
// they are,
//
//   LN(x) W^T = rs (x W'^T - mu S) + T,     W' = gamma W rounded to bf16,  S = sum_k W',  T = sum_k beta W,
//
// and the epilogue applies a row's rs and mu.  S is summed from the rounded W', so the mean cancels up to fp32 rounding,
// and of the two roundings of the other order (of the normalised rows and of W) one is left: 4.5e-3 from an fp64
// evaluation instead of 5.5e-3.  Nor does the gate pass through memory: its logits are computed where they are used, from
// z, which costs the read that the gate would have cost.  Of what a backward reads, the projection writes zln, the statistics
// and the mask of its rows, the output kernel the gate logits, and the output norm (a kernel of tpf_trimul.cu) xln.
//
// Both kernels are persistent and warp-specialised like the GEMM engine.  The weights stay in shared memory; a few warps
// read each landed tile once more for the sums of its rows, in 16-byte accesses without bank conflicts (normalising the
// tile in place instead, before the UMMAs, took 249 and 190 us where this took 215 and 135).
//
// Measured, C = 128, nothing kept: N = 1024 763 -> 550 us of kernels (norm 99 + projection 223 -> projection 207; norm 100
// + output 126 -> output 133; contraction 210 either way), N = 517 248 -> 178 us.  The output kernel runs at the copy
// rate (805 MB).  The projection does not (124 us): a tile takes an SM 7100 cycles, of which its 32 UMMAs of 128 x 128 x
// 16 need all of the shared memory bandwidth for 2050, beside 16 epilogue warps that take about 1650 cycles of arithmetic
// and 600 of staging and fence for 32 x 32 elements.  With a backward behind it, N = 384: norm 17 + projection 36 + output
// 22 -> projection 38 + output 30 us (which then stores the gate that the projection stored before).  A kernel of its own
// for zln read z a second time: 17 + 32 instead of 38 us.  Two warps for the rows, as without zln, take 52.
#include <type_traits>

#include "tpf_gemm_host.cuh"
#include "tpf_internal.h"
#include "tpf_norm.cuh"
#include "tpf_pair_rows.cuh"

namespace tpf {

static __device__ int g_trimul_fwd_status;

int trimul_fwd_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  TPF_CUDA_OK(cudaMemcpyFromSymbol(&v, g_trimul_fwd_status, sizeof(int)));
  if (v) TPF_CUDA_OK(cudaMemcpyToSymbol(g_trimul_fwd_status, &zero, sizeof(int)));
  *out = v;
  return TPF_OK;
}

// 64 channels of 128 rows of z in the internal grid, 64 rows a copy where they lie in one line of the pair tensor, else
// eight (the padded extent of a line is a multiple of eight).  Coordinates beyond the caller's tensor read as zeros.
__device__ __forceinline__ void load_z_block(uint32_t el, uint8_t* dst, const CUtensorMap* map64, const CUtensorMap* map8,
                                             uint64_t* bar, const PairRows& rows, int c0, int m0) {
  mbar_expect_tx(el, bar, 16384);
#pragma unroll 1
  for (int h = 0; h < 128; h += 64) {
    if (rows.identity) {
      tma_load_4d(el, dst + h * 128, map64, bar, c0, m0 + h, 0, 0);
      continue;
    }
    const uint32_t row = (uint32_t)(m0 + h);
    int b = (int)rows.plane.div(row);
    const uint32_t in = row - b * rows.plane.d;
    int i = (int)rows.pitch.div(in), j = (int)(in - i * rows.pitch.d);
    const int Np = (int)rows.pitch.d;
    if (j + 64 <= Np) {
      tma_load_4d(el, dst + h * 128, map64, bar, c0, j, i, b);
      continue;
    }
#pragma unroll 1
    for (int r = 0; r < 64; r += 8) {
      tma_load_4d(el, dst + (h + r) * 128, map8, bar, c0, j, i, b);
      j += 8;
      if (j == Np) {
        j = 0;
        if (++i == Np) {
          i = 0;
          ++b;
        }
      }
    }
  }
}

__device__ __forceinline__ void unpack_pairs(const uint4& u, uint64_t (&x)[4]) {
  x[0] = f2_pack(bf16_lo(u.x), bf16_hi(u.x));
  x[1] = f2_pack(bf16_lo(u.y), bf16_hi(u.y));
  x[2] = f2_pack(bf16_lo(u.z), bf16_hi(u.z));
  x[3] = f2_pack(bf16_lo(u.w), bf16_hi(u.w));
}
struct RowStats {
  float mu, rs;
};
template <int C>
__device__ __forceinline__ RowStats row_stats(float s1, float s2) {
  const float mu = s1 * (1.f / C);
  return RowStats{mu, rsqrtf(fmaxf(s2 * (1.f / C) - mu * mu, 0.f) + 1e-5f)};
}

// Sum and sum of squares of a lane's channels: eight of each 64.
template <int C, class Load>
__device__ __forceinline__ void lane_sums(Load load, float& s1, float& s2) {
  uint64_t t1 = 0ull, t2 = 0ull;
#pragma unroll
  for (int k = 0; k < C / 64; ++k) {
    uint64_t x[4];
    unpack_pairs(load(k), x);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      t1 = f2_add(t1, x[e]);
      t2 = f2_fma(x[e], x[e], t2);
    }
  }
  float lo, hi;
  f2_unpack(t1, lo, hi);
  s1 = lo + hi;
  f2_unpack(t2, lo, hi);
  s2 = lo + hi;
}

// Sums of ROWS consecutive rows of a K-major tile (64-channel blocks kb[] of 128 rows x 128 bytes, 128-byte swizzle) by one
// warp: eight lanes a row, 16 bytes of each block, four steps of four rows in flight.  `store` is called in one lane a row,
// all four rows behind one branch (with a branch for each row the projection took 225 instead of 207 us at N = 1024: its
// tiles wait for these warps); `each`, if there is one, in all lanes, with the place of the lane's 16 bytes.
struct NoEach {};
template <int C, int ROWS, class Store, class Each = NoEach>
__device__ __forceinline__ void stats_rows(const uint8_t* const (&kb)[C / 64], int row0, int lane, Store store,
                                           Each each = {}) {
  constexpr int U = 4;
#pragma unroll 1
  for (int r = 0; r < ROWS; r += 4 * U) {
    float s1[U], s2[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int row = row0 + r + 4 * u + (lane >> 3);
      const int off = row * 128 + (((lane & 7) ^ (row & 7)) << 4);
      lane_sums<C>([&](int k) { return *reinterpret_cast<const uint4*>(kb[k] + off); }, s1[u], s2[u]);
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        s1[u] += __shfl_xor_sync(0xffffffffu, s1[u], off);
        s2[u] += __shfl_xor_sync(0xffffffffu, s2[u], off);
      }
    if ((lane & 7) == 0) {
#pragma unroll
      for (int u = 0; u < U; ++u) store(row0 + r + 4 * u + (lane >> 3), row_stats<C>(s1[u], s2[u]));
    }
    if constexpr (!std::is_same<Each, NoEach>::value) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int row = row0 + r + 4 * u + (lane >> 3);
        each(row, row * 128 + (((lane & 7) ^ (row & 7)) << 4), row_stats<C>(s1[u], s2[u]));
      }
    }
  }
}

// Sums of the 64 rows of an MN-major tile (C lines of 128 bytes, one a channel, 128-byte swizzle) by one warp: a lane
// takes eight neighbouring rows (16 bytes) of every fourth channel.
template <int C, class Store>
__device__ __forceinline__ void stats_lines(const uint8_t* tile, int lane, Store store) {
  const int piece = lane & 7, cl = lane >> 3;
  uint64_t s1[4], s2[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) s1[e] = s2[e] = 0ull;
  // channels cl, cl + 4: their swizzles repeat every eight
  const uint8_t* p0 = tile + cl * 128 + ((piece ^ cl) << 4);
  const uint8_t* p1 = tile + (cl + 4) * 128 + ((piece ^ (cl + 4)) << 4);
#pragma unroll 4
  for (int c = 0; c < C; c += 8) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint64_t x[4];
      unpack_pairs(*reinterpret_cast<const uint4*>((h ? p1 : p0) + c * 128), x);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        s1[e] = f2_add(s1[e], x[e]);
        s2[e] = f2_fma(x[e], x[e], s2[e]);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float a0, a1, q0, q1;
    f2_unpack(s1[e], a0, a1);
    f2_unpack(s2[e], q0, q1);
#pragma unroll
    for (int off = 8; off <= 16; off <<= 1) {
      a0 += __shfl_xor_sync(0xffffffffu, a0, off);
      a1 += __shfl_xor_sync(0xffffffffu, a1, off);
      q0 += __shfl_xor_sync(0xffffffffu, q0, off);
      q1 += __shfl_xor_sync(0xffffffffu, q1, off);
    }
    if (cl == e) {
      store(8 * piece + 2 * e, row_stats<C>(a0, q0));
      store(8 * piece + 2 * e + 1, row_stats<C>(a1, q1));
    }
  }
}

// =============================================================================================
// project
// =============================================================================================
struct TrimulProjectParams {
  const float2* st;  // (S, T) of the weight rows
  PairRows rows;
  FastDiv per_entry;       // internal rows per batch entry
  PairMask mask;           // the caller's,
  const float* mask_grid;  // or, if not null, [R]
  float2* z_stats;         // [R] for the output kernel; KEEP: in its place
  float *mean, *rstd;      // [R]
  const float *gamma, *beta;
  bf16* zln;               // [R, C] normalised rows, zeros where the grid has no row of the caller
  float* mask_out;         // [R], or null: the mask has the internal layout
  int R;                   // internal rows
};

// KEEP: what a backward reads of the norm and the mask is written.
template <int C_, bool KEEP_>
struct TrimulProjectCfg {
  static constexpr int C = C_;
  static constexpr bool KEEP = KEEP_;
  static constexpr int NT = C / 64;              // accumulator tiles of 128 channels: the 2 C channels of [a, b]
  static constexpr int KB = C / 64;
  static constexpr int W_BYTES = 4 * C * C * 2;  // per 64 channels of k: projection rows [a, b], gate rows [a, b]
  static constexpr int NST = 3;                  // slots of 64 channels x 128 rows
  static constexpr int NCW = 16, NSW = KEEP ? 4 : 2;  // epilogue warps, warps that sum rows (96 or 80 registers)
  static constexpr int SR = 128 / NSW;           // rows of a tile that one of the latter sums
  static_assert(!KEEP || SR == 32, "one ballot tells which of its rows exist");
  static constexpr int THREADS = 32 * (2 + NCW + NSW);
  static constexpr int OFF_A = W_BYTES;
  // Tiles whose row scalars are kept: what is loaded ahead, two accumulators, and one being written.
  static constexpr int NRB = C == 64 ? 8 : 4;
  static constexpr int OFF_STG = OFF_A + NST * 16384;
  static constexpr int OFF_ROW = OFF_STG + NCW * 2048;  // [NRB] x {rs, -rs mu, mask} x 128
  static constexpr int OFF_BAR = OFF_ROW + NRB * 1536;
  static constexpr int SMEM_BYTES = OFF_BAR + 256;
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
trimul_project_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmZ8,
                      const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmAB0,
                      const __grid_constant__ CUtensorMap tmAB1, const TrimulProjectParams p, int* __restrict__ status) {
  griddep_wait();
  constexpr int C = Cfg::C, NT = Cfg::NT, KB = Cfg::KB, NST = Cfg::NST, NRB = Cfg::NRB;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {  // the launch checks it: no write beyond the block's memory
    if (threadIdx.x == 0) *status = (int)kStatusWaitTimeout;
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* w_full = bars;
  uint64_t* a_full = w_full + 1;      // [NST] 64 channels of a z tile have landed
  uint64_t* a_empty = a_full + NST;   // [NST] ... have been multiplied, and summed
  uint64_t* r_full = a_empty + NST;   // [NRB] the rows' scalars of a tile are there
  uint64_t* tfull = r_full + NRB;     // [2]
  uint64_t* tempty = tfull + 2;       // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wctx{abort_flag, status};
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int tiles = (p.R + 127) / 128;

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int s = 0; s < NST; ++s) {
      mbar_init(&a_full[s], 1);
      mbar_init(&a_empty[s], 1 + Cfg::NSW);
    }
    for (int s = 0; s < NRB; ++s) mbar_init(&r_full[s], Cfg::NSW);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], Cfg::NCW / 2);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmZ);
    tma_prefetch_desc(&tmW);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA loads
    const uint32_t el = elect_one();
    int s = 0;
    uint32_t ph = 1;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      for (int kb = 0; kb < KB; ++kb) {
        warp_wait(&a_empty[s], ph, wctx);
        load_z_block(el, smem + Cfg::OFF_A + s * 16384, &tmZ, &tmZ8, &a_full[s], p.rows, 64 * kb, tile * 128);
        if (++s == NST) {
          s = 0;
          ph ^= 1;
        }
      }
      if (tile == (int)blockIdx.x) {
        // packed weight blocks of C rows: projection a, gate a, projection b, gate b
        mbar_expect_tx(el, w_full, Cfg::W_BYTES);
        for (int kb = 0; kb < KB; ++kb)
          for (int blk = 0; blk < 4; ++blk) {
            const int dst = (blk & 1) * 2 * C + (blk >> 1) * C;
            for (int r = 0; r < C; r += 32)
              tma_load_3d(el, smem + (kb * 4 * C + dst + r) * 128, &tmW, w_full, 64 * kb, blk * C + r, 0);
          }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ UMMAs, accumulator lane = channel, column = row
    const uint32_t el = elect_one();
    constexpr uint32_t idesc = make_idesc_bf16(128, 128, false, false);
    constexpr uint32_t sw = swizzle_mode_for_bytes(128);
    const uint64_t w_desc = make_smem_desc(smem_u32(smem), 16, 1024, sw);
    const uint64_t a_desc = make_smem_desc(smem_u32(smem + Cfg::OFF_A), 16, 1024, sw);
    int s = 0, acc = 0;
    uint32_t ph = 0, acc_ph = 1;
    warp_wait(w_full, 0, wctx);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
      const int s_tile = s;
      const uint32_t ph_tile = ph;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        s = s_tile;
        ph = ph_tile;
        warp_wait(&tempty[acc], acc_ph, wctx);
        const uint32_t d = tmem_base + 256 * acc;
        for (int kb = 0; kb < KB; ++kb) {
          if (n == 0) warp_wait(&a_full[s], ph, wctx);
          tc_fence_after();
          const uint64_t ad = a_desc + ((s * 16384) >> 4), wd = w_desc + ((kb * 4 * C * 128 + n * 16384) >> 4);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            umma_ss(el, d, wd + 2 * k, ad + 2 * k, idesc, (kb | k) != 0);
            umma_ss(el, d + 128, wd + ((2 * C * 128) >> 4) + 2 * k, ad + 2 * k, idesc, (kb | k) != 0);
          }
          if (n + 1 == NT) umma_commit(el, &a_empty[s]);
          if (++s == NST) {
            s = 0;
            ph ^= 1;
          }
        }
        umma_commit(el, &tfull[acc]);
        if (++acc == 2) {
          acc = 0;
          acc_ph ^= 1;
        }
      }
    }
  } else if (warp < 2 + Cfg::NCW) {
    // ------------------------------------------------------------------ epilogue: norm, mask, gate, channel-major store
    // Eight warps an accumulator: while one set computes, the other waits, loads and stores.  A warp takes 64 rows of 32
    // channels, 32 at a time.
    const int ew = warp - 2, quarter = warp & 3, acc = ew >> 3, c0 = 64 * ((ew >> 2) & 1);
    uint8_t* stg = smem + Cfg::OFF_STG + ew * 2048;
    int i = 0;
    uint32_t acc_ph = 0;
    // this lane's channels: (S, T) of the projection and of the gate.  The set of an accumulator sees one of the two
    // tiles of 128 channels, or every second tile of rows.
    const int ch0 = (NT == 2 ? acc : 0) * 128 + 32 * quarter;  // of the warp's first lane, in [a, b]
    const int wrow = ((ch0 + lane) / C) * 2 * C + (ch0 + lane) % C;
    const float2 wv = p.st[wrow], wg = p.st[wrow + C];
    const uint64_t vs = f2_pack(wv.x, wv.x), vt = f2_pack(wv.y, wv.y), gs = f2_pack(wg.x, wg.x), gt = f2_pack(wg.y, wg.y);
    const CUtensorMap* map = ch0 < C ? &tmAB0 : &tmAB1;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      if (NT == 1 && (i & 1) != acc) continue;
      warp_wait2(&tfull[acc], acc_ph, &r_full[i % NRB], (i / NRB) & 1, wctx);
      acc_ph ^= 1;
      tc_fence_after();
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const int r0 = tile * 128 + c0 + 32 * h;
        const ulonglong2* row_rs =
            reinterpret_cast<const ulonglong2*>(smem + Cfg::OFF_ROW + (i % NRB) * 1536 + (c0 + 32 * h) * 4);
        bulk_wait_read<0>();  // (lane 0) the last store from the staging tile has read it
        __syncwarp();
        // 16 rows at a time: 32 at a time take 64 registers, which leaves too few to keep the broadcasts ahead
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const uint32_t t = tmem_addr(tmem_base, 32 * quarter, 256 * acc + c0 + 32 * h + 16 * hh);
          uint32_t v[16], g[16];  // of this lane's channel
          tmem_ld16(t, v);
          tmem_ld16(t + 128, g);
          tmem_ld_wait();
          if (hh == 1 && h == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tempty[acc]);
          }
          uint32_t ow[8];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            // four rows' rs, -rs mu, mask: the same address in every lane, one broadcast each
            const ulonglong2 rs = row_rs[4 * hh + q], nm = row_rs[32 + 4 * hh + q], mk = row_rs[64 + 4 * hh + q];
            const uint64_t rss[2] = {rs.x, rs.y}, nms[2] = {nm.x, nm.y}, mks[2] = {mk.x, mk.y};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int k = 4 * q + 2 * e;
              float h0, h1, o0, o1;
              f2_unpack(f2_fma(f2_pack_bits(g[k], g[k + 1]), rss[e], f2_fma(nms[e], gs, gt)), h0, h1);
              const uint64_t pv = f2_mul(f2_fma(f2_pack_bits(v[k], v[k + 1]), rss[e], f2_fma(nms[e], vs, vt)), mks[e]);
              f2_unpack(f2_fma(pv, f2_pack(tanh_fast(h0), tanh_fast(h1)), pv), o0, o1);
              ow[2 * q + e] = pack_bf16x2(o0, o1);
            }
          }
#pragma unroll
          for (int q = 0; q < 2; ++q)
            *reinterpret_cast<uint4*>(stg + lane * 64 + (((2 * hh + q) ^ ((lane >> 1) & 3)) << 4)) =
                make_uint4(ow[4 * q], ow[4 * q + 1], ow[4 * q + 2], ow[4 * q + 3]);
        }
        fence_async_smem();
        __syncwarp();
        // rows are a multiple of 64, so the 32-row chunk lies inside one batch entry and is inside R or not at all
        if (r0 < p.R) {
          const int bb = (int)p.per_entry.div((uint32_t)r0);
          tma_store_3d(lane == 0, map, stg, r0 - bb * (int)p.per_entry.d, ch0 & (C - 1), bb);
        }
      }
    }
    bulk_wait_all();
  } else {
    // ------------------------------------------------------------------ row sums
    const int sw0 = warp - 2 - Cfg::NCW;
    int i = 0, s = 0;
    uint32_t ph = 0;
    // KEEP: gamma and beta of this lane's channels, eight of each 64 (a parameter may start at any element: one by one)
    uint64_t ga[KB][4], be[KB][4];
    if constexpr (Cfg::KEEP) {
#pragma unroll
      for (int k = 0; k < KB; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = 64 * k + 8 * (lane & 7) + 2 * e;
          ga[k][e] = f2_pack(p.gamma[c], p.gamma[c + 1]);
          be[k][e] = f2_pack(p.beta[c], p.beta[c + 1]);
        }
    }
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      float* rs = reinterpret_cast<float*>(smem + Cfg::OFF_ROW + (i % NRB) * 1536);
      constexpr int NH = Cfg::SR / 32;
      float mk[NH];
      uint32_t real[NH];  // KEEP: which of the rows exist in the caller's tensor
#pragma unroll
      for (int h = 0; h < NH; ++h) {  // (the map costs two divisions: before the wait)
        const int r = tile * 128 + Cfg::SR * sw0 + 32 * h + lane;
        mk[h] = 0.f;
        bool there = r < p.R;
        if (there) {
          if (p.mask_grid != nullptr) {
            mk[h] = p.mask_grid[r];
          } else {
            const PairPos pos = p.rows.split((uint32_t)r);
            there = pos.src >= 0;
            if (there) mk[h] = p.mask.load(pos);
            if (Cfg::KEEP) p.mask_out[r] = mk[h];
          }
        }
        if constexpr (Cfg::KEEP) real[h] = __ballot_sync(0xffffffffu, there);
      }
      const uint8_t* kb[KB];
      int slot[KB];
#pragma unroll
      for (int k = 0; k < KB; ++k) {
        warp_wait(&a_full[s], ph, wctx);
        kb[k] = smem + Cfg::OFF_A + s * 16384;
        slot[k] = s;
        if (++s == NST) {
          s = 0;
          ph ^= 1;
        }
      }
      auto store = [&](int row, const RowStats& v) {
        const int m = tile * 128 + row;
        rs[row] = v.rs;
        rs[128 + row] = -v.rs * v.mu;
        if (m < p.R) {
          if constexpr (Cfg::KEEP) {
            p.mean[m] = v.mu;
            p.rstd[m] = v.rs;
          } else {
            p.z_stats[m] = make_float2(v.rs, -v.rs * v.mu);
          }
        }
      };
      if constexpr (Cfg::KEEP) {
        // the normalised row, 128 bytes by eight lanes
        stats_rows<C, Cfg::SR>(kb, Cfg::SR * sw0, lane, store, [&](int row, int off, const RowStats& v) {
          const int m = tile * 128 + row;
          const bool there = (real[0] >> (row & 31)) & 1;
          const uint64_t r2 = f2_pack(v.rs, v.rs), m2 = f2_pack(-v.mu, -v.mu);
#pragma unroll
          for (int k = 0; k < KB; ++k) {
            uint64_t x[4];
            unpack_pairs(*reinterpret_cast<const uint4*>(kb[k] + off), x);
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float lo, hi;
              f2_unpack(f2_fma(f2_mul(f2_add(x[e], m2), r2), ga[k][e], be[k][e]), lo, hi);
              o[e] = there ? pack_bf16x2(lo, hi) : 0u;
            }
            if (m < p.R)
              *reinterpret_cast<uint4*>(p.zln + (int64_t)m * C + 64 * k + 8 * (lane & 7)) =
                  make_uint4(o[0], o[1], o[2], o[3]);
          }
        });
      } else {
        stats_rows<C, Cfg::SR>(kb, Cfg::SR * sw0, lane, store);
      }
#pragma unroll
      for (int h = 0; h < NH; ++h) rs[256 + Cfg::SR * sw0 + 32 * h + lane] = mk[h];
      __syncwarp();
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < KB; ++k) mbar_arrive(&a_empty[slot[k]]);
        mbar_arrive(&r_full[i % NRB]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

// =============================================================================================
// output
// =============================================================================================
struct TrimulOutputParams {
  const float2 *st_x, *st_z;  // (S, T) of the rows of Wz and Wg
  const float2* z_stats;      // (rs, -rs mu) of the rows of z; KEEP: their mean and rs in two arrays
  const float *z_mean, *z_rstd;
  PairRows rows;
  FastDiv per_entry;
  bf16* gate;        // KEEP: [R, C]
  bf16 *out, *sum;   // caller's rows; without a residual `out` alone, else `sum` and, if not null, `out`
  int R;
};

// RES: a residual is added.  KEEP: the gate logits are stored.
template <int C_, bool RES_, bool KEEP_>
struct TrimulOutputCfg {
  static constexpr int C = C_;
  static constexpr bool RES = RES_, KEEP = KEEP_;
  static constexpr int KB = C / 64;
  static constexpr int W_BYTES = 2 * C * C * 2;  // Wz, Wg
  static constexpr int T_BYTES = 128 * C * 2;    // an x or z tile
  static constexpr int NCW = 8;                  // epilogue warps, then four that sum rows of x
  static constexpr int THREADS = 32 * (2 + NCW + 4);
  static constexpr int OFF_X = W_BYTES;          // [2]
  static constexpr int OFF_Z = OFF_X + 2 * T_BYTES;
  static constexpr int OFF_STG = OFF_Z + 2 * T_BYTES;
  static constexpr int OFF_COL = OFF_STG + NCW * 2048;   // {S, S, T, T} of channel pairs, for x and for z
  static constexpr int OFF_ROW = OFF_COL + 2 * C * 8;    // [4] x {rs, -rs mu} of x x 128: they outlive their tile's slots
  static constexpr int OFF_BAR = OFF_ROW + 4 * 1024;
  static constexpr int SMEM_BYTES = OFF_BAR + 256;
  static constexpr int ACC = 2 * C;              // TMEM columns of an accumulator pair
  static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
trimul_output_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmZ,
                     const __grid_constant__ CUtensorMap tmZ8, const __grid_constant__ CUtensorMap tmW,
                     const __grid_constant__ CUtensorMap tmOut, const __grid_constant__ CUtensorMap tmGate,
                     const TrimulOutputParams p, int* __restrict__ status) {
  griddep_wait();
  constexpr int C = Cfg::C, KB = Cfg::KB;
  extern __shared__ __align__(1024) uint8_t smem[];
  if ((smem_u32(smem) & 1023u) != 0) {  // the launch checks it: no write beyond the block's memory
    if (threadIdx.x == 0) *status = (int)kStatusWaitTimeout;
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Cfg::OFF_BAR);
  uint64_t* w_full = bars;
  uint64_t* x_full = bars + 1;    // [2]
  uint64_t* z_full = bars + 3;    // [2]
  uint64_t* a_empty = bars + 5;   // [2] x and z of a slot have been multiplied, and summed (and z added)
  uint64_t* tfull = bars + 7;     // [2]
  uint64_t* tempty = bars + 9;    // [2]
  uint64_t* r_full = bars + 11;   // [4] the rows' scalars of a tile are there
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const WaitCtx wctx{abort_flag, status};
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int tiles = (p.R + 127) / 128;
  float* col = reinterpret_cast<float*>(smem + Cfg::OFF_COL);

  if (threadIdx.x == 0) {
    mbar_init(w_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&x_full[s], 1);
      mbar_init(&z_full[s], KB);  // one arrival a block of 64 channels
      mbar_init(&a_empty[s], 1 + 2 + (Cfg::RES ? Cfg::NCW : 0));
      mbar_init(&tfull[s], 1);
      mbar_init(&tempty[s], Cfg::NCW);
    }
    for (int s = 0; s < 4; ++s) mbar_init(&r_full[s], 2);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmZ);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * Cfg::ACC);
    tmem_relinquish();
  }
  for (int c = threadIdx.x; c < 2 * C; c += Cfg::THREADS) {
    const float2 v = c < C ? p.st_x[c] : p.st_z[c - C];
    col[4 * (c / 2) + (c & 1)] = v.x;
    col[4 * (c / 2) + 2 + (c & 1)] = v.y;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA loads
    const uint32_t el = elect_one();
    int i = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      const int s = i & 1;
      warp_wait(&a_empty[s], ((i >> 1) & 1) ^ 1, wctx);
      mbar_expect_tx(el, &x_full[s], Cfg::T_BYTES);
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // 64 rows lie inside one batch entry
        const uint32_t r = (uint32_t)(tile * 128 + 64 * h);
        const int b = (int)p.per_entry.div(r);
        tma_load_3d(el, smem + Cfg::OFF_X + s * Cfg::T_BYTES + h * C * 128, &tmX, &x_full[s],
                    (int)(r - b * p.per_entry.d), 0, b);
      }
      for (int kb = 0; kb < KB; ++kb)
        load_z_block(el, smem + Cfg::OFF_Z + s * Cfg::T_BYTES + kb * 16384, &tmZ, &tmZ8, &z_full[s], p.rows, 64 * kb,
                     tile * 128);
      if (i == 0) {
        mbar_expect_tx(el, w_full, Cfg::W_BYTES);
        for (int kb = 0; kb < KB; ++kb) {
          tma_load_3d(el, smem + kb * C * 128, &tmW, w_full, 64 * kb, C, 0);  // rows [g; z]
          tma_load_3d(el, smem + C * C * 2 + kb * C * 128, &tmW, w_full, 64 * kb, 0, 0);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ UMMAs, accumulator lane = row
    const uint32_t el = elect_one();
    constexpr uint32_t idesc_x = make_idesc_bf16(128, C, true, false);
    constexpr uint32_t idesc_z = make_idesc_bf16(128, C, false, false);
    constexpr uint32_t sw = swizzle_mode_for_bytes(128);
    const uint64_t w_desc = make_smem_desc(smem_u32(smem), 16, 1024, sw);
    const uint64_t x_desc = make_smem_desc(smem_u32(smem + Cfg::OFF_X), C * 128, 1024, sw);
    const uint64_t z_desc = make_smem_desc(smem_u32(smem + Cfg::OFF_Z), 16, 1024, sw);
    int i = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      const int s = i & 1;
      const uint32_t ph = (i >> 1) & 1;
      warp_wait3(&tempty[s], ph ^ 1, &x_full[s], ph, &z_full[s], ph, wctx);
      if (i == 0) warp_wait(w_full, 0, wctx);
      tc_fence_after();
      const uint32_t d = tmem_base + Cfg::ACC * s;
#pragma unroll
      for (int k = 0; k < C / 16; ++k) {
        const uint64_t wd = w_desc + (((k >> 2) * C * 128) >> 4) + 2 * (k & 3);
        umma_ss(el, d, x_desc + ((s * Cfg::T_BYTES + k * 2048) >> 4), wd, idesc_x, k != 0);
        umma_ss(el, d + C, z_desc + ((s * Cfg::T_BYTES + (k >> 2) * 16384) >> 4) + 2 * (k & 3), wd + ((C * C * 2) >> 4),
                idesc_z, k != 0);
      }
      umma_commit(el, &a_empty[s]);
      umma_commit(el, &tfull[s]);
    }
  } else if (warp < 2 + Cfg::NCW) {
    // ------------------------------------------------------------------ epilogue: gate, residual, row-major store
    const int quarter = warp & 3, par = (warp - 2) >> 2;
    uint8_t* stg = smem + Cfg::OFF_STG + (warp - 2) * 2048;
    int i = 0, buf = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      const int s = i & 1;
      const int m_base = tile * 128 + 32 * quarter;
      float2 zst = make_float2(0.f, 0.f);
      if (m_base + lane < p.R) {
        if constexpr (Cfg::KEEP) {
          const float mu = p.z_mean[m_base + lane], rs = p.z_rstd[m_base + lane];
          zst = make_float2(rs, -rs * mu);
        } else {
          zst = p.z_stats[m_base + lane];
        }
      }
      warp_wait2(&tfull[s], (i >> 1) & 1, &r_full[i & 3], (i >> 2) & 1, wctx);
      tc_fence_after();
      const float* row = reinterpret_cast<const float*>(smem + Cfg::OFF_ROW + (i & 3) * 1024) + 32 * quarter + lane;
      const uint64_t xr = f2_pack(row[0], row[0]), xm = f2_pack(row[128], row[128]);
      const uint64_t zr = f2_pack(zst.x, zst.x), zm = f2_pack(zst.y, zst.y);
#pragma unroll
      for (int k = 0; k < C / 64; ++k) {
        const int n0 = 32 * (par + 2 * k);
        const uint32_t t = tmem_addr(tmem_base, 32 * quarter, Cfg::ACC * s + n0);
        uint32_t v[32], g[32];
        tmem_ld32(t, v);
        tmem_ld32(t + C, g);
        tmem_ld_wait();
        if (k + 1 == C / 64) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[s]);
        }
        const ulonglong2* cx = reinterpret_cast<const ulonglong2*>(col) + n0 / 2;
        uint32_t ow[16];
        if constexpr (Cfg::KEEP) {
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const ulonglong2 sz = cx[C / 2 + e];
            float h0, h1;
            f2_unpack(f2_fma(f2_pack_bits(g[2 * e], g[2 * e + 1]), zr, f2_fma(zm, sz.x, sz.y)), h0, h1);
            g[2 * e] = __float_as_uint(h0);
            g[2 * e + 1] = __float_as_uint(h1);
            ow[e] = pack_bf16x2(2.f * h0, 2.f * h1);
          }
          // By TMA, or with a residual, whose rows are stored by the threads too, by the threads (block training at
          // N = 768: 203 us an update by TMA, 175 this way; without one 29 and 35 us at N = 384).
          if constexpr (Cfg::RES) {
            warp_tile_store(stg, lane, ow, [&](int q) {
              return m_base + q < p.R ? p.gate + (int64_t)(m_base + q) * C + n0 : nullptr;
            });
          } else if (m_base < p.R) {
            warp_tile_store_tma<1>(stg, buf, lane, ow, &tmGate, n0, m_base, 0);
          }
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const ulonglong2 sx = cx[e];  // the same address in every lane: one broadcast
          float h0 = __uint_as_float(g[2 * e]), h1 = __uint_as_float(g[2 * e + 1]), o0, o1;
          if constexpr (!Cfg::KEEP) {
            const ulonglong2 sz = cx[C / 2 + e];
            f2_unpack(f2_fma(f2_pack(h0, h1), zr, f2_fma(zm, sz.x, sz.y)), h0, h1);
          }
          const uint64_t y = f2_fma(f2_pack_bits(v[2 * e], v[2 * e + 1]), xr, f2_fma(xm, sx.x, sx.y));
          f2_unpack(f2_fma(y, f2_pack(tanh_fast(h0), tanh_fast(h1)), y), o0, o1);
          ow[e] = pack_bf16x2(o0, o1);
        }
        if constexpr (Cfg::KEEP && !Cfg::RES) {
          if (!p.rows.identity) {  // these stores use the staging tile at once
            bulk_wait_read<0>();
            __syncwarp();
          }
        }
        if constexpr (Cfg::RES) {
          // the residual is the z tile, in the arrangement of the stores: 8 rows x 64 bytes an access
          uint4 r[4];
          const uint8_t* zt = smem + Cfg::OFF_Z + s * Cfg::T_BYTES + (n0 >> 6) * 16384;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int zrow = 32 * quarter + 8 * q + (lane >> 2), piece = ((n0 & 63) >> 3) + (lane & 3);
            r[q] = *reinterpret_cast<const uint4*>(zt + zrow * 128 + ((piece ^ (zrow & 7)) << 4));
          }
          store_rows_added(stg, lane, ow, p.rows, m_base, p.R, C, n0, p.out, p.sum, r);
          // Not before the residual has been used: released while those loads were in flight, the slot was refilled under
          // them now and then (one pass in four at C = 64, N = 528).
          if (k + 1 == C / 64) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_empty[s]);
          }
        }
        else if (p.rows.identity) {
          if (m_base < p.R) warp_tile_store_tma<1>(stg, buf, lane, ow, &tmOut, n0, m_base, 0);
        } else
          warp_tile_store(stg, lane, ow, [&](int q) { return row_address(p.out, p.rows, m_base + q, p.R, C, n0); });
      }
    }
    bulk_wait_all();
  } else {
    // ------------------------------------------------------------------ row sums of x, two warps a slot
    const int sw = warp - 2 - Cfg::NCW, h = sw & 1;
    int i = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      const int s = i & 1;
      if (s != sw >> 1) continue;
      float* row = reinterpret_cast<float*>(smem + Cfg::OFF_ROW + (i & 3) * 1024);
      warp_wait(&x_full[s], (i >> 1) & 1, wctx);
      stats_lines<C>(smem + Cfg::OFF_X + s * Cfg::T_BYTES + h * C * 128, lane, [&](int q, const RowStats& v) {
        row[64 * h + q] = v.rs;
        row[128 + 64 * h + q] = -v.rs * v.mu;
      });
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&a_empty[s]);
        mbar_arrive(&r_full[i & 3]);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, 2 * Cfg::ACC);
  }
}

// =============================================================================================
// host
// =============================================================================================
// z as the kernels load it: the caller's rows flat, or (c, j, i, b) of the caller's tensor; boxes of 64 and of 8 rows
static int make_z_tmaps(CUtensorMap* tm64, CUtensorMap* tm8, const TrimulCall& t, const PairRows& rows, int64_t R) {
  const uint64_t C = (uint64_t)t.C, N = (uint64_t)t.N, B = (uint64_t)t.B;
  uint64_t dims[4] = {C, N, N, B};
  uint64_t strides[3] = {2 * C, 2 * C * N, 2 * C * N * N};
  if (rows.identity) {
    dims[1] = (uint64_t)R;
    dims[2] = dims[3] = 1;
    strides[1] = strides[2] = 2 * C * (uint64_t)R;
  }
  uint32_t box[4] = {64, 64, 1, 1};
  if (int rc = make_tmap_bf16(tm64, t.z, 4, dims, strides, box, 128)) return rc;
  if (rows.identity) {  // not used
    *tm8 = *tm64;
    return TPF_OK;
  }
  box[1] = 8;
  return make_tmap_bf16(tm8, t.z, 4, dims, strides, box, 128);
}

static int fwd_status(int** status) {
  static PerDeviceAddress cache;
  return device_symbol_address(g_trimul_fwd_status, cache, reinterpret_cast<void**>(status));
}

static int row_tile_grid(int64_t R) {
  const int64_t tiles = (R + 127) / 128;
  return (int)(tiles < sm_count() ? tiles : sm_count());
}

template <int C, bool KEEP>
static int project(const TrimulCall& t, const TrimulFused& w, int64_t NN, cudaStream_t stream) {
  using Cfg = TrimulProjectCfg<C, KEEP>;
  const int64_t R = t.B * NN;
  int* status = nullptr;
  int rc = fwd_status(&status);
  if (rc) return rc;
  TrimulProjectParams p{};
  p.st = reinterpret_cast<const float2*>(w.st);
  p.rows = PairRows::make(t.N, t.Np, false);
  p.per_entry = FastDiv::make((uint32_t)NN);
  p.mask = PairMask{t.mask, t.mask_type, t.mask_stride[0], t.mask_stride[1], t.mask_stride[2]};
  // A mask without a copy of its own, of a forward that keeps what it makes, has the internal layout.
  p.mask_grid = KEEP && t.mask_grid == nullptr ? reinterpret_cast<const float*>(t.mask) : nullptr;
  p.z_stats = reinterpret_cast<float2*>(t.z_stats);
  if (KEEP) {
    p.mean = t.mean_in;
    p.rstd = t.rstd_in;
    p.gamma = t.w.norm_in_w;
    p.beta = t.w.norm_in_b;
    p.zln = (bf16*)t.zln;
    p.mask_out = t.mask_grid;
  }
  p.R = (int)R;
  CUtensorMap tz, tz8, tw, ta, tb;
  if ((rc = make_z_tmaps(&tz, &tz8, t, p.rows, R)) ||
      (rc = make_operand_tmap(&tw, w.w, false, 4 * C, C, C, 1, 0, 128, 32, 64)) ||
      (rc = make_store_tmap(&ta, t.a_cm, NN, C, NN, t.B, C * NN)) ||
      (rc = make_store_tmap(&tb, t.b_cm, NN, C, NN, t.B, C * NN)))
    return rc;
  auto kern = trimul_project_kernel<Cfg>;
  static PerDeviceOnce once;  // per instantiation
  if ((rc = ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, once, 1024))) return rc;
  launch_kernel(kern, dim3(row_tile_grid(R)), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, stream, tz, tz8, tw, ta, tb, p, status);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

template <int C, bool RES, bool KEEP>
static int output(const TrimulCall& t, const TrimulFused& w, int64_t NN, cudaStream_t stream) {
  using Cfg = TrimulOutputCfg<C, RES, KEEP>;
  const int64_t R = t.B * NN;
  int* status = nullptr;
  int rc = fwd_status(&status);
  if (rc) return rc;
  TrimulOutputParams p{};
  p.st_z = reinterpret_cast<const float2*>(w.st) + 4 * C;
  p.st_x = p.st_z + C;
  p.z_stats = reinterpret_cast<const float2*>(t.z_stats);
  p.z_mean = t.mean_in;
  p.z_rstd = t.rstd_in;
  p.rows = PairRows::make(t.N, t.Np, false);
  p.per_entry = FastDiv::make((uint32_t)NN);
  p.gate = (bf16*)t.gate;
  p.out = (bf16*)t.out;
  p.sum = (bf16*)t.sum;
  p.R = (int)R;
  CUtensorMap tx, tz, tz8, tw, to = {}, tg = {};
  uint64_t dims[3] = {(uint64_t)NN, (uint64_t)C, (uint64_t)t.B};
  uint64_t strides[2] = {(uint64_t)NN * 2, (uint64_t)(C * NN) * 2};
  uint32_t box[3] = {64, C, 1};
  if ((rc = make_z_tmaps(&tz, &tz8, t, p.rows, R)) || (rc = make_tmap_bf16(&tx, t.x_cm, 3, dims, strides, box, 128)) ||
      (rc = make_operand_tmap(&tw, (const bf16*)w.w + 4 * C * C, false, 2 * C, C, C, 1, 0, 128, C, 64)))
    return rc;
  if (!RES && p.rows.identity && (rc = make_store_tmap(&to, t.out, C, R, C, 1, 0))) return rc;
  if (KEEP && !RES && (rc = make_store_tmap(&tg, t.gate, C, R, C, 1, 0))) return rc;
  auto kern = trimul_output_kernel<Cfg>;
  static PerDeviceOnce once;  // per instantiation
  if ((rc = ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, once, 1024))) return rc;
  launch_kernel(kern, dim3(row_tile_grid(R)), dim3(Cfg::THREADS), Cfg::SMEM_BYTES, stream, tx, tz, tz8, tw, to, tg, p,
                status);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

template <int C>
static int output(const TrimulCall& t, const TrimulFused& w, int64_t NN, cudaStream_t stream) {
  if (t.infer) return t.sum ? output<C, true, false>(t, w, NN, stream) : output<C, false, false>(t, w, NN, stream);
  return t.sum ? output<C, true, true>(t, w, NN, stream) : output<C, false, true>(t, w, NN, stream);
}

bool trimul_fused(int64_t C) { return C == 64 || C == 128; }

// NN: internal rows per batch entry.
int trimul_project(const TrimulCall& t, const TrimulFused& w, int64_t NN, cudaStream_t stream) {
  if (t.infer) return t.C == 64 ? project<64, false>(t, w, NN, stream) : project<128, false>(t, w, NN, stream);
  return t.C == 64 ? project<64, true>(t, w, NN, stream) : project<128, true>(t, w, NN, stream);
}
int trimul_output(const TrimulCall& t, const TrimulFused& w, int64_t NN, cudaStream_t stream) {
  return t.C == 64 ? output<64>(t, w, NN, stream) : output<128>(t, w, NN, stream);
}

}  // namespace tpf
