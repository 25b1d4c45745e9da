// Batched bf16 GEMM on the tcgen05 engine: D[b] = A[b] * B[b]^T with either
// operand K-major or MN-major.  This is the TriMul k-contraction
// (reference: torch.bmm at turbopairformer_trimul.py:244-249 and :357-362) and
// the building block the other TriMul GEMM stages reuse with fused epilogues.
#include "tpf_gemm_host.cuh"

namespace tpf {

static __device__ int g_bmm_status;

int bmm_status_fetch_and_clear(int* out) {
  int v = 0, zero = 0;
  TPF_CUDA_OK(cudaMemcpyFromSymbol(&v, g_bmm_status, sizeof(int)));
  if (v) TPF_CUDA_OK(cudaMemcpyToSymbol(g_bmm_status, &zero, sizeof(int)));
  *out = v;
  return TPF_OK;
}

// Width of the output tiles.  A tile of 128 x BN moves (128 + BN) operand rows per k step through shared memory twice
// (TMA writes them, the tensor pipe reads them) for 128 x BN products: at BN = 128 that is 256 bytes a clock at full
// tensor rate where shared memory gives 128, so such tiles end at half the peak (1.16 of 2.3 PFLOP/s measured at
// N = 1024), and wider ones at 0.6 (192) and 0.67 (256) of it.  The time of a tile is therefore taken as 128 + BN,
// and the width with the shortest sequence of tiles per CTA is used; ragged widths and nearly empty last rounds count.
// Wide tiles have fewer stages and a longer start and end, so they have to promise a tenth.  Alone, 128 channels, K-major,
// us at 128 / 192 / 256 columns (* is what the rule takes; the count relative to 128 columns in brackets):
//   N =  264   24.1*  25.8 (0.94)   30.9 (1.13)        N =  520   93.8   75.3* (0.74)   87.4 (0.89)
//   N =  320   18.6*  19.5 (0.94)   21.6 (1.13)        N =  576   66.8   59.8* (0.74)   63.4 (0.89)
//   N =  384   24.0*  26.7 (0.94)   28.4 (1.13)        N =  640   78.1   82.4  (1.02)   75.1* (0.89)
//   N =  392   53.5   53.6 (0.98)   50.0* (0.75)       N =  896  195    191    (0.90)  183*   (0.87)
//   N =  512   44.0   46.2 (0.98)   40.4* (0.75)       N = 1024  280    282    (0.94)  240*   (0.75)
// At 64 channels N = 640 stays at 128 columns (46.1 us; 46.3 at 256, 0.955).  Over these and six more lengths, 64 and 128
// channels, both operand majors, the choice is at most 2.5 % behind the best of the three.
static int tile_width(const GemmShape& sh) {
  const int64_t mt = (int64_t)sh.batch * ((sh.M + 127) / 128), sms = sm_count();
  int best = 128;
  int64_t best_cost = INT64_MAX;
  for (int bn = 128; bn <= 256; bn += 64) {
    const int64_t tiles = mt * ((sh.N + bn - 1) / bn);
    const int64_t cost = (tiles + sms - 1) / sms * (128 + bn) * (bn == 128 ? 9 : 10);
    if (cost < best_cost) {
      best = bn;
      best_cost = cost;
    }
  }
  return best;
}

template <int BN, int SWZ, bool A_MN, bool B_MN, typename OutT>
int bmm_run(const void* A, int64_t lda, int64_t bsa, const void* B, int64_t ldb, int64_t bsb, void* D,
            int64_t ldd, int64_t bsd, const GemmShape& sh, int* status, cudaStream_t stream) {
  constexpr int kBK = (A_MN && B_MN) ? 64 : SWZ / 2;
  constexpr int kBufs = BN == 256 ? 1 : 2;  // one staging tile per warp makes room for the fourth stage
  constexpr int kFit = (BN == 128 ? 196608 : BN == 192 ? 163840 : 196608) / ((128 + BN) * kBK * 2);
  using Cfg = GemmCfg<128, BN, SWZ, A_MN, SWZ, B_MN, (kFit > 8 ? 8 : kFit), (BN == 128 ? 8 : 16)>;
  using Epi = EpiStore<OutT, kBufs>;
  typename Epi::Params ep;
  if (int rc = epi_store_params<OutT, kBufs>(&ep, reinterpret_cast<OutT*>(D), ldd, bsd, sh)) return rc;
  return launch_gemm<Cfg, Epi>(A, lda, bsa, B, ldb, bsb, sh, ep, status, stream);
}

template <int SWZ, bool A_MN, bool B_MN, typename OutT>
int bmm_dispatch(const void* A, int64_t lda, int64_t bsa, const void* B, int64_t ldb, int64_t bsb, void* D,
                 int64_t ldd, int64_t bsd, const GemmShape& sh, int* status, cudaStream_t stream) {
  if constexpr (SWZ == 128 && sizeof(OutT) == 2) {  // the others (split K, narrow swizzles) are not tensor-bound
    const int bn = tile_width(sh);
    if (bn == 256)
      return bmm_run<256, SWZ, A_MN, B_MN, OutT>(A, lda, bsa, B, ldb, bsb, D, ldd, bsd, sh, status, stream);
    if (bn == 192)
      return bmm_run<192, SWZ, A_MN, B_MN, OutT>(A, lda, bsa, B, ldb, bsb, D, ldd, bsd, sh, status, stream);
  }
  return bmm_run<128, SWZ, A_MN, B_MN, OutT>(A, lda, bsa, B, ldb, bsb, D, ldd, bsd, sh, status, stream);
}

int bmm_bf16(const void* A, int64_t lda, int64_t bsa, int a_mn, const void* B, int64_t ldb, int64_t bsb, int b_mn,
             void* D, int64_t ldd, int64_t bsd, int out_f32, int64_t M, int64_t N, int64_t K, int64_t batch,
             int64_t k_per_split, int swizzle_bytes, cudaStream_t stream) {
  TPF_REQUIRE(A && B && D, TPF_ERR_INVALID_ARGUMENT, "bmm: null pointer");
  TPF_REQUIRE(M > 0 && N > 0 && K > 0 && batch > 0, TPF_ERR_INVALID_ARGUMENT, "bmm: M,N,K,batch must be positive");
  TPF_REQUIRE(M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31) && batch < (1ll << 31),
              TPF_ERR_INVALID_ARGUMENT, "bmm: extent too large");
  TPF_REQUIRE(lda % 8 == 0 && ldb % 8 == 0 && bsa % 8 == 0 && bsb % 8 == 0, TPF_ERR_INVALID_ARGUMENT,
              "bmm: leading dimensions and batch strides must be multiples of 8 elements (16 bytes)");
  TPF_REQUIRE(k_per_split >= 0 && k_per_split % 64 == 0, TPF_ERR_INVALID_ARGUMENT,
              "bmm: k_per_split must be a non-negative multiple of 64");
  GemmShape sh{(int)M, (int)N, (int)K, (int)batch, (int)k_per_split};
  int* status = nullptr;
  {
    static PerDeviceAddress cache;
    if (int rc = device_symbol_address(g_bmm_status, cache, reinterpret_cast<void**>(&status))) return rc;
  }
#define TPF_BMM_CASE(SWZ, AM, BM)                                                                              \
  if (swizzle_bytes == SWZ && (a_mn != 0) == AM && (b_mn != 0) == BM)                                          \
    return out_f32 ? bmm_dispatch<SWZ, AM, BM, float>(A, lda, bsa, B, ldb, bsb, D, ldd, bsd, sh, status, stream) \
                   : bmm_dispatch<SWZ, AM, BM, __nv_bfloat16>(A, lda, bsa, B, ldb, bsb, D, ldd, bsd, sh, status, \
                                                              stream);
  TPF_BMM_CASE(128, false, false)
  TPF_BMM_CASE(128, true, true)
  TPF_BMM_CASE(128, true, false)
  TPF_BMM_CASE(128, false, true)
  TPF_BMM_CASE(64, false, false)
  TPF_BMM_CASE(64, true, true)
  TPF_BMM_CASE(32, false, false)
  TPF_BMM_CASE(32, true, true)
#undef TPF_BMM_CASE
  return fail(TPF_ERR_UNSUPPORTED, "bmm: unsupported (swizzle=%d, a_mn=%d, b_mn=%d)", swizzle_bytes, a_mn, b_mn);
}

}  // namespace tpf
