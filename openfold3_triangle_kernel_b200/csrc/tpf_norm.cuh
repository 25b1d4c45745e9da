// Row-wise LayerNorm kernels (forward, backward) and the fixed-order folds of split gradient sums: used by the triangle
// multiplicative update and by the attention module of the pair block.
#pragma once

#include "tpf_host.cuh"
#include "tpf_pair_rows.cuh"
#include "tpf_ptx.cuh"

namespace tpf {

typedef __nv_bfloat16 bf16;

// =============================================================================================
// LayerNorm over the last dim of a row-major [R,C] bf16 tensor (input norm), forward
// =============================================================================================
// Row-wise LayerNorm kernels: a lane owns 8 consecutive channels (one 16-byte load), the lanes of a row
// sit in a slot of LS lanes (a power of two; the lanes beyond C / 8 of a slot idle when C = 96), and a warp
// works on 32 / LS rows at a time.
template <int C>
struct RowLanes {
  static constexpr int LPR = C / 8;                               // lanes that hold a row
  static constexpr int LS = LPR <= 4 ? 4 : LPR <= 8 ? 8 : 16;     // lanes per row slot
  static constexpr int RPW = 32 / LS;                             // rows per warp step
};

template <int C>
__device__ __forceinline__ float slot_sum(float v) {
#pragma unroll
  for (int off = RowLanes<C>::LS / 2; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&x)[8]) {
  x[0] = bf16_lo(u.x); x[1] = bf16_hi(u.x); x[2] = bf16_lo(u.y); x[3] = bf16_hi(u.y);
  x[4] = bf16_lo(u.z); x[5] = bf16_hi(u.z); x[6] = bf16_lo(u.w); x[7] = bf16_hi(u.w);
}

// MAPPED: the caller's rows differ from the internal ones, or the mask has to be converted (see PairRows); kept apart
// because the row map costs the plain case 5 % (98.6 -> 103.5 us at R = 1024^2, C = 128).
template <int C, bool MAPPED>
__global__ void __launch_bounds__(256) ln_fwd_kernel(const bf16* __restrict__ z, const float* __restrict__ gamma,
                                                            const float* __restrict__ beta, bf16* __restrict__ zln,
                                                            float* __restrict__ mean, float* __restrict__ rstd,
                                                            const PairRows rows, const PairMask pmask,
                                                            float* __restrict__ mask_out, int64_t R) {
  griddep_wait();
  using L = RowLanes<C>;
  constexpr int G = 4;  // row groups per warp, all loads issued before the first use
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int sub = lane / L::LS, part = lane % L::LS;
  const bool on = part < L::LPR;
  float g[8], b[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    g[e] = on ? gamma[part * 8 + e] : 0.f;
    b[e] = on ? beta[part * 8 + e] : 0.f;
  }
  uint4 u[G];
  bool active[G], real[G];  // real: the row exists in the caller's tensor (padding rows come out as zeros)
#pragma unroll
  for (int r = 0; r < G; ++r) {
    const int64_t row = (warp * G + r) * L::RPW + sub;
    active[r] = on && row < R;
    real[r] = active[r];
    u[r] = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (MAPPED) {
      const PairPos pos = rows.split((uint32_t)(row < R ? row : 0));
      real[r] = active[r] && pos.src >= 0;
      if (real[r]) u[r] = *reinterpret_cast<const uint4*>(z + pos.src * C + part * 8);
      if (mask_out != nullptr && active[r] && part == 0) mask_out[row] = real[r] ? pmask.load(pos) : 0.f;
    } else {
      if (real[r]) u[r] = *reinterpret_cast<const uint4*>(z + row * C + part * 8);
    }
  }
#pragma unroll
  for (int r = 0; r < G; ++r) {
    const int64_t row = (warp * G + r) * L::RPW + sub;
    float x[8];
    unpack8(u[r], x);
    float a1 = 0.f, a2 = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      a1 += x[e];
      a2 += x[e] * x[e];
    }
    const float s1 = slot_sum<C>(a1);
    const float s2 = slot_sum<C>(a2);
    const float mu = s1 * (1.f / C);
    const float var = fmaxf(s2 * (1.f / C) - mu * mu, 0.f);
    const float rs = rsqrtf(var + 1e-5f);
    if (active[r]) {
      uint4 o = make_uint4(0u, 0u, 0u, 0u);
      if (!MAPPED || real[r]) {
      o.x = pack_bf16x2((x[0] - mu) * rs * g[0] + b[0], (x[1] - mu) * rs * g[1] + b[1]);
      o.y = pack_bf16x2((x[2] - mu) * rs * g[2] + b[2], (x[3] - mu) * rs * g[3] + b[3]);
      o.z = pack_bf16x2((x[4] - mu) * rs * g[4] + b[4], (x[5] - mu) * rs * g[5] + b[5]);
      o.w = pack_bf16x2((x[6] - mu) * rs * g[6] + b[6], (x[7] - mu) * rs * g[7] + b[7]);
      }
      *reinterpret_cast<uint4*>(zln + row * C + part * 8) = o;
      if (part == 0 && mean != nullptr) {
        mean[row] = mu;
        rstd[row] = rs;
      }
    }
  }
}

// Input-norm backward, row-major.  d_z = rstd (gamma d_zln - mean(gamma d_zln) - xhat mean(gamma d_zln xhat))
template <int C>
__global__ void __launch_bounds__(256) ln_bwd_kernel(const bf16* __restrict__ d_zln, const bf16* __restrict__ z,
                                                            const float* __restrict__ gamma,
                                                            const float* __restrict__ mean,
                                                            const float* __restrict__ rstd, bf16* __restrict__ d_z,
                                                            float* __restrict__ partials, const PairRows rows,
                                                            const bf16* __restrict__ d_res, int64_t R,
                                                            int rows_per_block) {
  griddep_wait();
  using L = RowLanes<C>;
  __shared__ float red[8][2][C];
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int sub = lane / L::LS, part = lane % L::LS;
  const bool on = part < L::LPR;
  const int64_t row_begin = (int64_t)blockIdx.x * rows_per_block;
  float g[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) g[e] = on ? gamma[part * 8 + e] : 0.f;
  float ag[8], ab[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) ag[e] = ab[e] = 0.f;
  constexpr int G = 4;  // row groups in flight per warp: all their loads are issued before the first use
  for (int it0 = warp * L::RPW; it0 < rows_per_block; it0 += G * 8 * L::RPW) {
    uint4 du[G], zu[G], ru[G];  // ru: the gradient that reaches z past the update (residual connection)
    float mu[G], rs[G];
    int64_t src[G];  // the caller's row
    bool active[G];
#pragma unroll
    for (int r = 0; r < G; ++r) {
      const int it = it0 + r * 8 * L::RPW;
      const int64_t row = row_begin + it + sub;
      active[r] = on && it + sub < rows_per_block && row < R;
      src[r] = active[r] ? rows.locate((uint32_t)row).src : -1;
      active[r] = src[r] >= 0;
      du[r] = zu[r] = ru[r] = make_uint4(0u, 0u, 0u, 0u);
      mu[r] = rs[r] = 0.f;
      if (active[r]) {
        du[r] = *reinterpret_cast<const uint4*>(d_zln + row * C + part * 8);
        zu[r] = *reinterpret_cast<const uint4*>(z + src[r] * C + part * 8);
        if (d_res != nullptr) ru[r] = *reinterpret_cast<const uint4*>(d_res + src[r] * C + part * 8);
        mu[r] = mean[row];
        rs[r] = rstd[row];
      }
    }
#pragma unroll
    for (int r = 0; r < G; ++r) {
      float d[8], xh[8];
      unpack8(du[r], d);
      unpack8(zu[r], xh);
      float gd[8], a1 = 0.f, a2 = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        xh[e] = active[r] ? (xh[e] - mu[r]) * rs[r] : 0.f;
        gd[e] = g[e] * d[e];
        a1 += gd[e];
        a2 += gd[e] * xh[e];
      }
      const float m1 = slot_sum<C>(a1) * (1.f / C);
      const float m2 = slot_sum<C>(a2) * (1.f / C);
      if (active[r]) {
        float res[8];
        unpack8(ru[r], res);
        uint32_t o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          o[e] = pack_bf16x2(res[2 * e] + rs[r] * (gd[2 * e] - m1 - xh[2 * e] * m2),
                             res[2 * e + 1] + rs[r] * (gd[2 * e + 1] - m1 - xh[2 * e + 1] * m2));
        *reinterpret_cast<uint4*>(d_z + src[r] * C + part * 8) = make_uint4(o[0], o[1], o[2], o[3]);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          ag[e] += d[e] * xh[e];
          ab[e] += d[e];
        }
      }
    }
  }
  // fixed-order fold: the row slots of a warp (sub = 0 .. RPW-1), then the 8 warps
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float vg = ag[e], vb = ab[e];
    for (int s = 1; s < L::RPW; ++s) {
      const float og = __shfl_sync(0xffffffffu, ag[e], part + s * L::LS);
      const float ob = __shfl_sync(0xffffffffu, ab[e], part + s * L::LS);
      vg += og;
      vb += ob;
    }
    if (sub == 0 && on) {
      red[warp][0][part * 8 + e] = vg;
      red[warp][1][part * 8 + e] = vb;
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 * C) {
    const int which = threadIdx.x / C, c = threadIdx.x % C;
    float s = red[0][which][c];
    for (int w = 1; w < 8; ++w) s += red[w][which][c];
    partials[(int64_t)blockIdx.x * 2 * C + which * C + c] = s;
  }
}

// Every fixed-order fold of the backward in one launch: the split-K weight-gradient partials and the per-CTA sums
// of the two LayerNorm backward kernels.  Each job is tiny (latency bound: a few dependent batches of loads), so what
// they cost is launches; six of them, folded one after the other, took longer than the sums.
//   weight gradients: out[r][c] = sum over splits of part[s][m][c], rows routed in blocks of C to up to five
//                     destinations (W5 = [a_p; a_g; b_p; b_g; g]);
//   norm gradients:   out[j] = sum over CTAs of partials[blk][j], j < 2C, the halves going to d_gamma and d_beta.
// A CTA owns 32 output elements (8 of a job with many terms); thread group g adds its contiguous range of terms in
// ascending order (a batch of 8 loads is in flight before the first add), then the 8 (32) range sums are added in range
// order: a fixed summation tree, no atomics.
struct FoldJob {
  const float* part;
  int terms, width;   // width: distance between consecutive terms
  int used;           // outputs wanted (the columns beyond are padding)
  int C;              // elements per destination row block: C * C (weights) or C (norms)
  int log_lanes;      // a CTA folds 1 << log_lanes outputs, with 256 >> log_lanes threads each
  float* dst[5];
};
struct FoldJobs {
  FoldJob job[4];
  int first[5];  // first CTA of each job; first[n_jobs] = grid
  int n_jobs;
};
static __global__ void __launch_bounds__(256) fold_kernel(const __grid_constant__ FoldJobs jobs) {
  griddep_wait();
  __shared__ float red[256];
  int n = 0;
  while (n + 1 < jobs.n_jobs && (int)blockIdx.x >= jobs.first[n + 1]) ++n;
  const FoldJob& jb = jobs.job[n];
  const int lanes = 1 << jb.log_lanes, groups = 256 >> jb.log_lanes;
  const int g = threadIdx.x >> jb.log_lanes, lane = threadIdx.x & (lanes - 1);
  const int i = (blockIdx.x - jobs.first[n]) * lanes + lane;
  const int per = (jb.terms + groups - 1) >> (8 - jb.log_lanes);
  const int k0 = g * per, k1 = min(jb.terms, k0 + per);
  float s = 0.f;
  if (i < jb.used) {
    const float* src = jb.part + i;
    for (int k = k0; k < k1; k += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = k + u < k1 ? src[(int64_t)(k + u) * jb.width] : 0.f;
#pragma unroll
      for (int u = 0; u < 8; ++u) s = __fadd_rn(s, v[u]);
    }
  }
  red[threadIdx.x] = s;
  __syncthreads();
  if (g == 0 && i < jb.used) {
    float t = red[lane];
    for (int w = 1; w < groups; ++w) t = __fadd_rn(t, red[w * lanes + lane]);
    const int d = i / jb.C;
    jb.dst[d][i - d * jb.C] = t;
  }
}

struct FoldList {
  FoldJobs j = {};
  void add(const float* part, int terms, int width, int C, float* d0, float* d1 = nullptr, float* d2 = nullptr,
           float* d3 = nullptr, float* d4 = nullptr, int used = 0) {
    if (used == 0) used = width;
    // Few outputs with many terms (the norms: 2 C outputs, a term per CTA of the backward pass) are a chain of load
    // latencies: 8 outputs per CTA (a sector of each row) leave 32 threads for the terms of each, where 32 outputs left
    // 8 threads with 148 terms each.
    const int log_lanes = terms > 256 ? 3 : 5;
    const FoldJob job{part, terms, width, used, C, log_lanes, {d0, d1, d2, d3, d4}};
    // The CTAs of the job with the longest chains come first: the input norm's, added last, ended long after the others
    // (update with C = 128, N = 384: 13.6 -> 9.5 us; a block at N = 768, four folds: 46 -> 36 us).
    int at = j.n_jobs++;
    for (; at > 0 && chain(j.job[at - 1]) < chain(job); --at) j.job[at] = j.job[at - 1];
    j.job[at] = job;
  }
  static int chain(const FoldJob& job) { return job.terms >> (8 - job.log_lanes); }  // terms a thread
  int launch(cudaStream_t stream) {
    if (j.n_jobs == 0) return TPF_OK;
    for (int n = 0; n < j.n_jobs; ++n)
      j.first[n + 1] = j.first[n] + ((j.job[n].used + (1 << j.job[n].log_lanes) - 1) >> j.job[n].log_lanes);
    launch_kernel(fold_kernel, dim3(j.first[j.n_jobs]), dim3(256), 0, stream, j);
    TPF_LAUNCH_OK();
    return TPF_OK;
  }
};

template <int C>
inline unsigned ln_fwd_blocks(int64_t R) {
  const int64_t warps = (R + 4 * RowLanes<C>::RPW - 1) / (4 * RowLanes<C>::RPW);
  return (unsigned)((warps + 7) / 8);
}
// at most 8 CTAs per SM, so that few partial rows are left to fold
inline int ln_bwd_rows_per_block(int64_t R) {
  return (int)(((R + 8 * sm_count() - 1) / (8 * sm_count()) + 127) / 128 * 128);
}

}  // namespace tpf
