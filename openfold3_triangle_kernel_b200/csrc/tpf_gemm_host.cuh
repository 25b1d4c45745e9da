// Host-side launch helpers for the tcgen05 GEMM engine (tpf_gemm.cuh).
#pragma once

#include "tpf_gemm.cuh"
#include "tpf_host.cuh"

namespace tpf {

// Tensor map for one GEMM operand.  K-major: memory [batch][mn][k]; MN-major: memory [batch][k][mn].
inline int make_operand_tmap(CUtensorMap* tm, const void* base, bool mn_major, int64_t mn, int64_t k, int64_t ld,
                      int64_t batch, int64_t batch_stride, int swz, int tile_mn, int bk) {
  uint64_t dims[3];
  uint64_t strides[2] = {(uint64_t)ld * 2, (uint64_t)(batch_stride ? batch_stride : 8) * 2};
  uint32_t box[3];
  if (!mn_major) {
    dims[0] = (uint64_t)k; dims[1] = (uint64_t)mn; dims[2] = (uint64_t)batch;
    box[0] = (uint32_t)bk; box[1] = (uint32_t)tile_mn; box[2] = 1;
  } else {
    dims[0] = (uint64_t)mn; dims[1] = (uint64_t)k; dims[2] = (uint64_t)batch;
    box[0] = (uint32_t)(swz / 2); box[1] = (uint32_t)bk; box[2] = 1;
  }
  return make_tmap_bf16(tm, base, 3, dims, strides, box, swz);
}

// Tensor map of a bf16 output [batch][rows][cols] for warp_tile_store_tma: 32 x 32 boxes, 64-byte swizzle.
inline int make_store_tmap(CUtensorMap* tm, const void* base, int64_t cols, int64_t rows, int64_t ld, int64_t batch,
                           int64_t batch_stride) {
  uint64_t dims[3] = {(uint64_t)cols, (uint64_t)rows, (uint64_t)batch};
  uint64_t strides[2] = {(uint64_t)ld * 2, (uint64_t)(batch_stride ? batch_stride : 8) * 2};
  uint32_t box[3] = {32, 32, 1};
  return make_tmap_bf16(tm, base, 3, dims, strides, box, 64);
}
// Parameters of EpiStore; bf16 outputs with 16-byte aligned rows get a tensor map.
template <typename OutT, int BUFS = 2>
inline int epi_store_params(typename EpiStore<OutT, BUFS>::Params* ep, OutT* D, int64_t ldd, int64_t batch_stride,
                            const GemmShape& sh) {
  *ep = {};
  ep->D = D;
  ep->ldd = ldd;
  ep->batch_stride = batch_stride;
  if (sizeof(OutT) == 2 && ldd % 8 == 0 && batch_stride % 8 == 0 && (reinterpret_cast<uintptr_t>(D) & 15) == 0) {
    ep->has_map = 1;
    return make_store_tmap(&ep->map, D, sh.N, sh.M, ldd, sh.batch, batch_stride);
  }
  return TPF_OK;
}

// B resident in every CTA, or one tile column of it per CTA (GemmCfg::STAT 3 or 2) for R rows and nt tile columns?
// Compared by the longest sequence of tiles a CTA gets: with few rows the second divides the work better.  At (nearly)
// equal lengths the first wins, by its single read of A.
inline bool resident_pays(int64_t R, int64_t nt) {
  const int64_t mt = (R + 127) / 128, sms = sm_count();
  return 8 * nt * ((mt + sms - 1) / sms) <= 9 * ((mt * nt + sms - 1) / sms);
}

template <class Cfg, class Epi>
int launch_gemm(const void* A, int64_t lda, int64_t bsa, const void* B, int64_t ldb, int64_t bsb,
                const GemmShape& sh, const typename Epi::Params& ep, int* status, cudaStream_t stream,
                int max_ctas = 0) {
  CUtensorMap tmA, tmB;
  const int64_t tensor_batch = sh.k_per_split > 0 ? 1 : sh.batch;
  int rc = make_operand_tmap(&tmA, A, Cfg::A_MN, sh.M, sh.K, lda, tensor_batch, bsa, Cfg::SWZ_A, Cfg::BM, Cfg::BK);
  if (rc) return rc;
  rc = make_operand_tmap(&tmB, B, Cfg::B_MN, sh.N, sh.K, ldb, tensor_batch, bsb, Cfg::SWZ_B, Cfg::B_BOX, Cfg::BK);
  if (rc) return rc;
  auto kern = gemm_umma_kernel<Cfg, Epi>;
  constexpr int smem_bytes = Cfg::SMEM_BYTES + Cfg::EPI_WARPS * Epi::kSmemPerWarp;
  static_assert(smem_bytes <= 232448, "shared memory budget");
  static PerDeviceOnce once;  // per instantiation
  if ((rc = ensure_dynamic_smem(kern, smem_bytes, once))) return rc;
  const int mt = (sh.M + Cfg::BM - 1) / Cfg::BM, nt = (sh.N + Cfg::BN - 1) / Cfg::BN;
  const int tiles = sh.batch * mt * nt;
  int grid = sm_count();
  if (max_ctas > 0 && grid > max_ctas) grid = max_ctas;
  if (grid > (Cfg::RESIDENT ? mt : tiles)) grid = Cfg::RESIDENT ? mt : tiles;
  if (grid < 1) return TPF_OK;
  if constexpr (Cfg::STAT != 0) {
    const int k_len = sh.k_per_split > 0 ? sh.k_per_split : sh.K;
    TPF_REQUIRE(k_len <= Cfg::STAT_KB * Cfg::BK, TPF_ERR_UNSUPPORTED,
                "gemm: K = %d exceeds the stationary operand buffer (%d)", k_len, Cfg::STAT_KB * Cfg::BK);
    if constexpr (Cfg::RESIDENT) {
      TPF_REQUIRE(sh.batch == 1 && sh.N <= Cfg::B_ROWS, TPF_ERR_UNSUPPORTED, "gemm: B does not fit as a whole");
    }
    const int per = Cfg::RESIDENT ? 1 : (tiles + grid - 1) / grid;  // contiguous tiles per CTA; CTAs that would get none are not launched
    if (!Cfg::RESIDENT) grid = (tiles + per - 1) / per;
  }
  launch_kernel(kern, dim3(grid), dim3(Cfg::THREADS), smem_bytes, stream, tmA, tmB, sh, ep, status);
  TPF_LAUNCH_OK();
  return TPF_OK;
}

}  // namespace tpf
