// Kernel and launch of the CTA-pair GEMM (256 x BN tiles over two SMs, gemm_2cta.cuh) for the sources that use it.
#pragma once
#include "api.h"
#include "gemm_2cta.cuh"

namespace b200 {

template <int BN, int STAGES, bool A_MN, bool B_MN, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G2_THREADS, 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmC, int M, int N, int K, Gemm2Params ep, uint32_t* status) {
  gemm2_mainloop<BN, STAGES, A_MN, B_MN, EPI>(&tmA, &tmB, &tmC, M, N, K, ep, status);
}

// How many CTA pairs can be resident at once (asked once per kernel and device; <= num_sms / 2).
template <class Kern>
static int max_pairs(Kern kern, int smem_bytes, int num_sms, int threads = G2_THREADS) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * (num_sms / 2), 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem_bytes;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) {
    (void)cudaGetLastError();
    n = num_sms / 2;
  }
  return n < num_sms / 2 ? n : num_sms / 2;
}

template <int BN, int STAGES, bool A_MN, bool B_MN, int EPI>
static int launch_gemm2(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                        long long ldc, const Gemm2Params& ep, uint32_t* status, int num_sms, cudaStream_t stream) {
  CUtensorMap tmA, tmB, tmC;
  if (A_MN ? make_tmap_2d(&tmA, A, K, M, lda, 64, 64, 2) : make_tmap_2d(&tmA, A, M, K, lda, G2_BM_CTA, G2_BK, 2))
    return B200_ERR_TENSORMAP;
  if (B_MN ? make_tmap_2d(&tmB, B, K, N, ldb, 64, 64, 2) : make_tmap_2d(&tmB, B, N, K, ldb, BN / 2, G2_BK, 2))
    return B200_ERR_TENSORMAP;
  const int n_cols = EPI == G2_EPI_SWIGLU ? N / 2 : N;
  if (make_tmap_out(&tmC, C, M, n_cols, ldc, ep.out_fp32)) return B200_ERR_TENSORMAP;
  using SM = Gemm2Smem<BN, STAGES>;
  auto kern = gemm2_bf16_kernel<BN, STAGES, A_MN, B_MN, EPI>;
  static int pairs[16] = {0};  // per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return B200_ERR_RUNTIME;
  if (pairs[dev] == 0) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL) != cudaSuccess)
      return B200_ERR_LAUNCH;
    pairs[dev] = max_pairs(kern, SM::TOTAL, num_sms);
  }
  constexpr int OUT_BN = EPI == G2_EPI_SWIGLU ? BN / 2 : BN;
  const int tiles = ((M + G2_BM - 1) / G2_BM) * ((n_cols + OUT_BN - 1) / OUT_BN);
  int np = pairs[dev];
  if (num_sms / 2 < np) np = num_sms / 2;  // the caller may reserve SMs for kernels on other streams
  if (np < 1) np = 1;
  const int grid = 2 * (tiles < np ? tiles : np);
  kern<<<grid, G2_THREADS, SM::TOTAL, stream>>>(tmA, tmB, tmC, M, N, K, ep, status);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

}  // namespace b200
