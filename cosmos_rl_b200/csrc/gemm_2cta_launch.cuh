// Kernel and launch of the CTA-pair GEMM (256 x BN tiles over two SMs, gemm_2cta.cuh) for the sources that use it.
#pragma once
#include "api.h"
#include "gemm_2cta.cuh"

namespace b200 {

template <int BN, int STAGES, bool A_MN, bool B_MN, int EPI, bool TAIL = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(g2_threads(EPI), 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                  const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmW, int M, int N, int K,
                  Gemm2Params ep, uint32_t* status) {
  gemm2_mainloop<BN, STAGES, A_MN, B_MN, EPI, TAIL>(&tmA, &tmB, &tmC, &tmW, M, N, K, ep, status);
}

// C of the cut tiles: the sum of their shares (+ bias) (+ C). A warp has one row of a tile, a lane eight columns; rows of C
// start on 16-byte boundaries. Above 128 rows the sum is added to C in memory, like the tiles that are not cut: whatever else
// adds to C at that time, no value is lost. Fewer rows, all of whose tiles come this way, read C and write it like the single-CTA
// kernel, and round once.
// Grid (rest, 256 / 8).
template <int BN>
__global__ void __launch_bounds__(256)
gemm2_sum_shares_kernel(const float* __restrict__ ws, void* __restrict__ C, long long ldc, int M, int N, Gemm2Params ep) {
  pdl_wait();
  const int num_m = (M + G2_BM - 1) / G2_BM, num_n = (N + BN - 1) / BN;
  int m_blk, n_blk;
  g2_tile_coords(blockIdx.x, num_m, num_n, ep.group_m > 0 ? ep.group_m : 8, m_blk, n_blk);
  const int r = blockIdx.y * 8 + (threadIdx.x >> 5);
  const long long row = (long long)m_blk * G2_BM + r;
  if (row >= M) return;
#pragma unroll
  for (int c = (threadIdx.x & 31) * 8; c < BN; c += 256) {
    const int col = n_blk * BN + c;
    if (col >= N) continue;
    const float* p = ws + ((long long)blockIdx.x * G2_BM + r) * BN + c;
    const long long step = (long long)ep.rest * G2_BM * BN;
    float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float4 x[8][2];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < ep.splits) {
        x[s][0] = *reinterpret_cast<const float4*>(p + s * step);
        x[s][1] = *reinterpret_cast<const float4*>(p + s * step + 4);
      }
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < ep.splits) {
        v[0] += x[s][0].x; v[1] += x[s][0].y; v[2] += x[s][0].z; v[3] += x[s][0].w;
        v[4] += x[s][1].x; v[5] += x[s][1].y; v[6] += x[s][1].z; v[7] += x[s][1].w;
      }
    if (ep.bias != nullptr) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col + j < N)
          v[j] += ep.bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ep.bias)[col + j])
                               : reinterpret_cast<const float*>(ep.bias)[col + j];
    }
    const bool add = ep.accumulate && M > 128;
    if (ep.out_fp32) {
      float* dst = reinterpret_cast<float*>(C) + row * ldc + col;
      if (add) {
        if (col + 8 <= N) {
          red_add(dst, v[0], v[1], v[2], v[3]);
          red_add(dst + 4, v[4], v[5], v[6], v[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (col + j < N) atomicAdd(dst + j, v[j]);
        }
        continue;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (col + j < N) dst[j] = ep.accumulate ? dst[j] + v[j] : v[j];
    } else {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(C) + row * ldc + col;
      if (add) {
        if (col + 8 <= N) {
          red_add(dst, pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (col + j < N) atomicAdd(dst + j, __float2bfloat16(v[j]));
        }
        continue;
      }
      if (col + 8 <= N) {
        if (ep.accumulate) {
          const uint4 old = *reinterpret_cast<const uint4*>(dst);
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(h[j]);
            v[2 * j] += f.x;
            v[2 * j + 1] += f.y;
          }
        }
        *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                                    pack_bf16x2(v[6], v[7]));
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (col + j < N) dst[j] = __float2bfloat16(ep.accumulate ? __bfloat162float(dst[j]) + v[j] : v[j]);
      }
    }
  }
}

// How many CTA pairs of `kern` run at once on `num_sms` SMs: a caller may reserve some for kernels on other streams. `whole` is
// the kernel's own (per device): what the device has room for, asked once and whatever the first call's num_sms is. Also makes
// the kernel's shared memory available. 0 or an error code.
template <class Kern>
static int resident_pairs(Kern kern, int (&whole)[16], int smem_bytes, int threads, int num_sms, int& np) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return B200_ERR_RUNTIME;
  if (whole[dev] == 0) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return B200_ERR_RUNTIME;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes) != cudaSuccess) return B200_ERR_LAUNCH;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (sms / 2), 1, 1);
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
      n = sms / 2;
    }
    whole[dev] = n < sms / 2 ? n : sms / 2;
  }
  np = whole[dev] < num_sms / 2 ? whole[dev] : num_sms / 2;
  if (np < 1) np = 1;
  return 0;
}

// Contraction blocks that a cut has to save a pair: the shares' way through memory and the kernel that adds them. Weight
// gradients, us, uncut and cut: 1500 tokens (24 blocks), 6144 x 4096 57 and 61; 2048 tokens (32 blocks) 74 and 77. Of 64 blocks
// and more every cut pays: 300 x 4096 x 28672 141 and 89, 1500 x 4096 x 14336 149 and 125, 1500 x 4096 x 4096 49 and 44.
constexpr int G2_CUT_BLOCKS = 30;
// Tiles of the last round that are cut along the contraction, into how many shares; 0: none.
inline int g2_rest(long long tiles, int pairs, int num_kb, int& splits) {
  const int rest = (int)(tiles % pairs);
  splits = rest > 0 ? pairs / rest : 0;
  if (splits > 8) splits = 8;
  if (splits > num_kb / 8) splits = num_kb / 8;
  if (splits < 2 || num_kb - num_kb / splits < G2_CUT_BLOCKS) return splits = 0;
  return rest;
}

// The same, but with `all` every tile, in one share if there is nothing to cut: sums that are to be rounded once pass through the
// kernel that adds the shares. All tiles run at once then.
inline int g2_shared_tiles(long long tiles, int pairs, int num_kb, bool all, int& splits) {
  const int rest = g2_rest(tiles, pairs, num_kb, splits);
  if (!all || rest == tiles) return rest;
  splits = 1;
  return (int)tiles;
}

// Few rows that are added to bf16 values: the single-CTA kernel rounds the sum only, TMA adds round the product before it as well.
inline bool g2_round_once(int M, int out_fp32, int accumulate) { return M <= G2_BM_CTA && accumulate && !out_fp32; }

// Scratch of a launch that cuts `rest` tiles (Gemm2Params::ws), in elements.
constexpr long long g2_ws_floats(int rest, int splits, int bn) { return (long long)rest * splits * G2_BM * bn; }

// allow_cut: a launch that would gain from a workspace and has too little (ep.ws, ws_floats) returns B200_NEED_WORKSPACE
template <int BN, int STAGES, bool A_MN, bool B_MN, int EPI, bool TAIL>
static int launch_gemm2_form(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                             long long ldc, Gemm2Params ep, uint32_t* status, int num_sms, cudaStream_t stream,
                             bool allow_cut, long long ws_floats) {
  CUtensorMap tmA, tmB, tmC, tmW;
  const int n_cols = EPI == G2_EPI_SWIGLU ? N / 2 : N;
  using SM = Gemm2Smem<BN, STAGES>;
  auto kern = gemm2_bf16_kernel<BN, STAGES, A_MN, B_MN, EPI, TAIL>;
  static int whole[16] = {0};
  int np = 0;
  if (const int rc = resident_pairs(kern, whole, SM::TOTAL, G2_THREADS, num_sms, np)) return rc;
  constexpr int OUT_BN = EPI == G2_EPI_SWIGLU ? BN / 2 : BN;
  const int tiles = ((M + G2_BM - 1) / G2_BM) * ((n_cols + OUT_BN - 1) / OUT_BN);
  const bool all = g2_round_once(M, ep.out_fp32, ep.accumulate) && tiles <= np;
  ep.rest = EPI == G2_EPI_STORE && allow_cut ? g2_shared_tiles(tiles, np, (K + G2_BK - 1) / G2_BK, all, ep.splits)
                                             : (ep.splits = 0);
  if (ep.rest > 0 && (ep.ws == nullptr || ws_floats < g2_ws_floats(ep.rest, ep.splits, BN))) return B200_NEED_WORKSPACE;
  const int a_rows = !A_MN && M < G2_BM_CTA ? M : G2_BM_CTA;
  ep.a_bytes = a_rows * G2_BK * 2;
  if (A_MN ? make_tmap_2d(&tmA, A, K, M, lda, 64, 64, 2) : make_tmap_2d(&tmA, A, M, K, lda, a_rows, G2_BK, 2))
    return B200_ERR_TENSORMAP;
  if (B_MN ? make_tmap_2d(&tmB, B, K, N, ldb, 64, 64, 2) : make_tmap_2d(&tmB, B, N, K, ldb, BN / 2, G2_BK, 2))
    return B200_ERR_TENSORMAP;
  ep.C = C;
  ep.ldc = ldc;
  const int whole_cols = whole16(n_cols, ep.out_fp32);   // 0: nothing is stored through the map
  if (make_tmap_out(&tmC, C, M, whole_cols ? whole_cols : (ep.out_fp32 ? 4 : 8), ldc, ep.out_fp32)) return B200_ERR_TENSORMAP;
  tmW = tmC;
  if (ep.rest > 0 && make_tmap_out(&tmW, ep.ws, (uint64_t)ep.rest * ep.splits * G2_BM, BN, BN, 1)) return B200_ERR_TENSORMAP;
  const int grid = 2 * (ep.rest > 0 || tiles >= np ? np : tiles);
  kern<<<grid, G2_THREADS, SM::TOTAL, stream>>>(tmA, tmB, tmC, tmW, M, N, K, ep, status);
  if (cudaGetLastError() != cudaSuccess) return B200_ERR_LAUNCH;
  if constexpr (EPI == G2_EPI_STORE)
    if (ep.rest > 0 && launch_pdl(gemm2_sum_shares_kernel<BN>, dim3(ep.rest, G2_BM / 8), dim3(256), 0, stream,
                                  (const float*)ep.ws, C, ldc, M, N, ep) != cudaSuccess)
      return B200_ERR_LAUNCH;
  return 0;
}

template <int BN, int STAGES, bool A_MN, bool B_MN, int EPI>
static int launch_gemm2(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                        long long ldc, const Gemm2Params& ep, uint32_t* status, int num_sms, cudaStream_t stream,
                        bool allow_cut = false, long long ws_floats = 0) {
  const int n_cols = EPI == G2_EPI_SWIGLU ? N / 2 : N;
  auto launch = whole16(n_cols, ep.out_fp32) == n_cols ? launch_gemm2_form<BN, STAGES, A_MN, B_MN, EPI, false>
                                                       : launch_gemm2_form<BN, STAGES, A_MN, B_MN, EPI, true>;
  return launch(A, B, C, M, N, K, lda, ldb, ldc, ep, status, num_sms, stream, allow_cut, ws_floats);
}

}  // namespace b200
