// Dense bf16 GEMM on tcgen05/TMEM:  C[M,N] = A[M,K] * B[N,K]^T  (+ optional fp32 accumulate-into).
// A and B are row-major with K contiguous (the layout of activations x and nn.Linear weights),
// C is row-major bf16 or fp32. Building block for the fused kernels of this library; replaces
// the library GEMM the reference reaches through nn.Linear (cosmos_rl/policy/model/gpt/__init__.py:284-316).
#include "gemm_core.cuh"
#include "gemm_2cta_launch.cuh"
#include "api.h"

namespace b200 {

struct StoreEpilogue {
  struct Params {
    void* C;
    long long ldc;
    int M, N;
    int out_fp32;     // 0: bf16, 1: fp32
    int accumulate;   // C += result
    int bn;
  };
  __device__ __forceinline__ void tile_begin(const Params&, const TileInfo&, int) {}
  __device__ __forceinline__ void tile_end(const Params&, const TileInfo&, int) {}
  __device__ __forceinline__ void finish(const Params&) {}
  __device__ __forceinline__ void chunk(const Params& p, const TileInfo& t, int row, int col0, const float (&v)[32]) {
    store_chunk(p.C, p.ldc, p.M, p.N, p.out_fp32, p.accumulate, (long long)t.m_blk * GEMM_BM + row,
                t.n_blk * p.bn + col0, v);
  }
  static __device__ __forceinline__ void store_chunk(void* C, long long ldc, long long M, int N, int out_fp32,
                                                     int accumulate, long long r, int c, const float (&v)[32]) {
    if (r >= M || c >= N) return;
    if (out_fp32) {
      float* dst = reinterpret_cast<float*>(C) + r * ldc + c;
      if (c + 32 <= N && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          float4 o = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
          if (accumulate) {
            float4 old = *reinterpret_cast<float4*>(dst + i);
            o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
          }
          *reinterpret_cast<float4*>(dst + i) = o;
        }
      } else {
        for (int i = 0; i < 32 && c + i < N; ++i) dst[i] = accumulate ? dst[i] + v[i] : v[i];
      }
    } else {
      __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(C) + r * ldc + c;
      if (c + 32 <= N && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          float w[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) w[j] = v[i + j];
          if (accumulate) {
            uint4 old = *reinterpret_cast<uint4*>(dst + i);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              float2 f = __bfloat1622float2(h[j]);
              w[2 * j] += f.x;
              w[2 * j + 1] += f.y;
            }
          }
          uint4 o;
          o.x = pack_bf16x2(w[0], w[1]);
          o.y = pack_bf16x2(w[2], w[3]);
          o.z = pack_bf16x2(w[4], w[5]);
          o.w = pack_bf16x2(w[6], w[7]);
          *reinterpret_cast<uint4*>(dst + i) = o;
        }
      } else {
        for (int i = 0; i < 32 && c + i < N; ++i)
          dst[i] = __float2bfloat16(accumulate ? __bfloat162float(dst[i]) + v[i] : v[i]);
      }
    }
  }
};

template <int BN, int STAGES, bool A_MN, bool B_MN>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N, int K,
                 StoreEpilogue::Params ep, uint32_t* status) {
  gemm_mainloop<BN, STAGES, StoreEpilogue, RasterSchedule, GemmTraits<A_MN, B_MN>>(&tmA, &tmB, M, N, K, ep, status);
}

template <int BN, int STAGES, bool A_MN, bool B_MN>
static int launch_gemm(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                       long long ldc, int out_fp32, int accumulate, uint32_t* status, int num_sms,
                       cudaStream_t stream) {
  CUtensorMap tmA, tmB;
  // K-major operand: stored [MN, K], box = (tile rows) x 64 contraction elements.
  // MN-major operand: stored [K, MN], box = 64 contraction rows x 64 MN elements.
  if (A_MN ? make_tmap_2d(&tmA, A, K, M, lda, 64, 64, 2) : make_tmap_2d(&tmA, A, M, K, lda, GEMM_BM, GEMM_BK, 2))
    return B200_ERR_TENSORMAP;
  if (B_MN ? make_tmap_2d(&tmB, B, K, N, ldb, 64, 64, 2) : make_tmap_2d(&tmB, B, N, K, ldb, BN, GEMM_BK, 2))
    return B200_ERR_TENSORMAP;
  using SM = GemmSmem<BN, STAGES>;
  auto kern = gemm_bf16_kernel<BN, STAGES, A_MN, B_MN>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL) != cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  StoreEpilogue::Params ep{C, ldc, M, N, out_fp32, accumulate, BN};
  int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * ((N + BN - 1) / BN);
  int grid = tiles < num_sms ? tiles : num_sms;
  kern<<<grid, GEMM_THREADS, SM::TOTAL, stream>>>(tmA, tmB, M, N, K, ep, status);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

template <bool A_MN, bool B_MN>
static int dispatch_bn(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                       long long ldc, int out_fp32, int accumulate, uint32_t* status, int num_sms, cudaStream_t stream) {
  // Wide tiles amortise shared-memory traffic; narrow N uses the 128-wide tile.
  if (N >= 256)
    return launch_gemm<256, 4, A_MN, B_MN>(A, B, C, M, N, K, lda, ldb, ldc, out_fp32, accumulate, status, num_sms, stream);
  return launch_gemm<128, 6, A_MN, B_MN>(A, B, C, M, N, K, lda, ldb, ldc, out_fp32, accumulate, status, num_sms, stream);
}

// 128-wide tiles, whose product takes 0.6 of the time of a 256-wide one, where those would fill more than half of one round of
// pairs (so that it is not cut) and these one round and at most a third of the next, which is cut then. us, 256 and 128 wide:
// 700 x 3584 x 18944 (42 tiles) 99 and 80, 600 x 4096 x 14336 (48) 79 and 70, the same with B stored [K, N]; 1003 x 4096 x 14336
// (64) 84 and 91. Narrow tiles fetch A twice as often. Stored [K, M] with M no multiple of 64, it has boxes that lie partly
// outside, which take longer: 600 x 4096 x 14336 86 and 101, 648 x 3584 x 8192 52 and 52 to 54, 704 x 3584 x 18944 102 and 79.
static bool narrow_tiles(int M, int N, int K, bool a_mn, int pairs) {
  const int num_m = (M + G2_BM - 1) / G2_BM;
  const long long wide = (long long)num_m * ((N + 255) / 256), narrow = (long long)num_m * ((N + 127) / 128);
  return wide <= pairs && 2 * wide > pairs && narrow > pairs && 3 * (narrow - pairs) <= pairs && K >= 64 * G2_BK &&
         !(a_mn && M % 64);
}

// The CTA pairs that the rules below reckon with: as many as run at once.
static int gemm_pairs(int num_sms) {
  static int whole[16] = {0};
  int np = 0;
  const int rc = resident_pairs(gemm2_bf16_kernel<256, 6, false, false, G2_EPI_STORE>, whole, Gemm2Smem<256, 6>::TOTAL, G2_THREADS,
                                num_sms, np);
  return rc ? num_sms / 2 : np;
}

static int pair_tile_width(int M, int N, int K, bool a_mn, int out_fp32, int accumulate, bool cut, int num_sms) {
  return N > 128 && (g2_round_once(M, out_fp32, accumulate) || !(cut && narrow_tiles(M, N, K, a_mn, gemm_pairs(num_sms)))) ? 256 : 128;
}

template <bool A_MN, bool B_MN>
static int dispatch_gemm2(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                          long long ldc, const Gemm2Params& ep, int epi, bool cut, long long ws_floats, uint32_t* status,
                          int num_sms, cudaStream_t stream) {
  if (epi == G2_EPI_SWIGLU) {
    if constexpr (!A_MN && !B_MN)
      return launch_gemm2<256, 6, false, false, G2_EPI_SWIGLU>(A, B, C, M, N, K, lda, ldb, ldc, ep, status, num_sms, stream);
    else
      return B200_ERR_ARG;
  }
  if (pair_tile_width(M, N, K, A_MN, ep.out_fp32, ep.accumulate, cut, num_sms) == 256)
    return launch_gemm2<256, 6, A_MN, B_MN, G2_EPI_STORE>(A, B, C, M, N, K, lda, ldb, ldc, ep, status, num_sms, stream, cut, ws_floats);
  return launch_gemm2<128, 8, A_MN, B_MN, G2_EPI_STORE>(A, B, C, M, N, K, lda, ldb, ldc, ep, status, num_sms, stream, cut, ws_floats);
}

// Up to 128 rows the pair kernel is the faster one when all its tiles run at once, with or without a cut (100 rows, us, single
// CTAs and pairs: 4096 x 28672 165 and 51, 14336 x 4096 36 and 29; 28672 x 4096, 112 tiles, 51 and 56), and the rows of C are
// whole 16 bytes, which is what its stores write. With 129 to 255 columns a pair has one tile of 256 where single CTAs have two of
// 128, and unless it is cut its results take longer to write (7 x 184 x 960 11.0 us and 9.1; 8 x 112 x 1280 7.8 and 9.4).
static bool pairs_for_few_rows(int M, int N, int K, int out_fp32, int num_sms) {
  if (M > 128 || (N + 255) / 256 > gemm_pairs(num_sms) || ((N * (out_fp32 ? 4 : 2)) & 15)) return false;
  if (N <= 128 || N >= 256) return true;
  int splits = 0;
  return g2_rest(1, gemm_pairs(num_sms), (K + G2_BK - 1) / G2_BK, splits) > 0;
}

// Whether a call takes the CTA-pair kernel. rows16: the rows of C start on 16-byte boundaries; without that there is none.
static bool takes_pairs(bool rows16, int M, int N, int K, int out_fp32, bool bias, int epilogue, int path,
                        bool cut, int num_sms) {
  if (epilogue == G2_EPI_SWIGLU || bias || path == 2) return true;   // what only this kernel has
  return path != 1 && rows16 && (M > 128 || (cut && pairs_for_few_rows(M, N, K, out_fp32, num_sms)));
}

}  // namespace b200

// C[M,N] (+)= op(A) * op(B)^T with fp32 accumulation.
//   a_mn = 0: A stored [M, K] (lda = row stride)      a_mn = 1: A stored [K, M]
//   b_mn = 0: B stored [N, K] (ldb = row stride)      b_mn = 1: B stored [K, N]
// forward  y = x W^T      : a_mn 0, b_mn 0        dgrad dx = dy W : a_mn 0, b_mn 1 (W stored [N_contract, K_out])
// wgrad dW = dy^T x       : a_mn 1, b_mn 1 (both stored [tokens, features])
// (reason << 24) | CUresult of the last tensor-map encode that failed in this process (0: none); see gemm_core.cuh
extern "C" int b200_last_tmap_error() { return b200::last_tmap_error(); }

// cut: a call whose tiles leave half of their last round of CTA pairs idle cuts it along the contraction. ws: scratch of
// ws_floats elements for that; with less than b200_gemm_scratch says such a call returns B200_NEED_WORKSPACE and has launched
// nothing.
extern "C" int b200_gemm_bf16_ws(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                 long long ldb, long long ldc, int a_mn, int b_mn, int out_fp32, int accumulate,
                                 const void* bias, int bias_bf16, int epilogue, int up_row0, int path, int cut, float* ws,
                                 long long ws_floats, uint32_t* status, int num_sms, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return B200_ERR_ARG;
  // TMA needs 16-byte aligned row strides; MN-major tiles are fetched in 64-element columns
  if ((lda & 7) || (ldb & 7)) return B200_ERR_ARG;
  using namespace b200;
  const bool rows16 = !(reinterpret_cast<uintptr_t>(C) & 15) && !((ldc * (out_fp32 ? 4 : 2)) & 15);
  if (takes_pairs(rows16, M, N, K, out_fp32, bias != nullptr, epilogue, path, cut != 0, num_sms)) {
    if (!rows16) return B200_ERR_ARG;
    if (epilogue == G2_EPI_SWIGLU && (a_mn || b_mn || (N & 1) || accumulate)) return B200_ERR_ARG;
    Gemm2Params ep{bias, bias_bf16, out_fp32, accumulate, up_row0, 8, 0, 0, 0, ws, nullptr, 0, {}};
    auto go = [&](auto am, auto bm) {
      return dispatch_gemm2<decltype(am)::value, decltype(bm)::value>(A, B, C, M, N, K, lda, ldb, ldc, ep, epilogue, cut != 0,
                                                                      ws_floats, status, num_sms, stream);
    };
    if (!a_mn && !b_mn) return go(std::false_type{}, std::false_type{});
    if (!a_mn && b_mn) return go(std::false_type{}, std::true_type{});
    if (a_mn && b_mn) return go(std::true_type{}, std::true_type{});
    return go(std::true_type{}, std::false_type{});
  }
  if (!a_mn && !b_mn) return dispatch_bn<false, false>(A, B, C, M, N, K, lda, ldb, ldc, out_fp32, accumulate, status, num_sms, stream);
  if (!a_mn && b_mn) return dispatch_bn<false, true>(A, B, C, M, N, K, lda, ldb, ldc, out_fp32, accumulate, status, num_sms, stream);
  if (a_mn && b_mn) return dispatch_bn<true, true>(A, B, C, M, N, K, lda, ldb, ldc, out_fp32, accumulate, status, num_sms, stream);
  return dispatch_bn<true, false>(A, B, C, M, N, K, lda, ldb, ldc, out_fp32, accumulate, status, num_sms, stream);
}

extern "C" int b200_gemm_bf16_ex(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                 long long ldb, long long ldc, int a_mn, int b_mn, int out_fp32, int accumulate,
                                 const void* bias, int bias_bf16, int epilogue, int up_row0, int path,
                                 uint32_t* status, int num_sms, cudaStream_t stream) {
  return b200_gemm_bf16_ws(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate, bias, bias_bf16, epilogue, up_row0,
                           path, 0, nullptr, 0, status, num_sms, stream);
}

// Scratch that such a call with `cut` wants, in elements; 0: it is not cut. rows16: C and its row stride are multiples of 16 bytes.
extern "C" long long b200_gemm_scratch(int M, int N, int K, int a_mn, int rows16, int out_fp32, int accumulate, int bias, int epilogue,
                                       int path, int num_sms) {
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0 || num_sms < 2 || epilogue == G2_EPI_SWIGLU || !rows16) return 0;
  if (!takes_pairs(true, M, N, K, out_fp32, bias != 0, epilogue, path, true, num_sms)) return 0;
  const int bn = pair_tile_width(M, N, K, a_mn != 0, out_fp32, accumulate, true, num_sms);
  const int pairs = gemm_pairs(num_sms);
  const long long tiles = (long long)((M + G2_BM - 1) / G2_BM) * ((N + bn - 1) / bn);
  int splits = 0;
  const int rest = g2_shared_tiles(tiles, pairs, (K + G2_BK - 1) / G2_BK, g2_round_once(M, out_fp32, accumulate) && tiles <= pairs,
                                   splits);
  return g2_ws_floats(rest, splits, bn);
}

extern "C" int b200_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                              long long ldb, long long ldc, int a_mn, int b_mn, int out_fp32, int accumulate,
                              uint32_t* status, int num_sms, cudaStream_t stream) {
  return b200_gemm_bf16_ex(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_fp32, accumulate, nullptr, 0, 0, 0, 0,
                           status, num_sms, stream);
}

extern "C" int b200_gemm_bf16_nt(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                                 long long ldb, long long ldc, int out_fp32, int accumulate, uint32_t* status,
                                 int num_sms, cudaStream_t stream) {
  return b200_gemm_bf16(A, B, C, M, N, K, lda, ldb, ldc, 0, 0, out_fp32, accumulate, status, num_sms, stream);
}
