// The two dense GEMMs of a gated MLP that its activation hangs on, in training: gate/up projection with the product formed in its
// epilogue, and the product's gradient with the activation's gradient formed in its. Both on the CTA-pair main loop
// (gemm_2cta.cuh), with two epilogue warps a TMEM lane quadrant. A pass over [T, 2 I] and [T, I] of its own is bound by HBM, which
// the GEMM hardly uses. 8192 x 18944 x 3584, us, GEMM and pass, and one kernel, cold and in a long run under the power cap: forward
// 1530 and 1417, 1820 and 1610; backward 1052 and 913, 1120 and 930. 1003 x 14336 x 4096: 205 and 194, 136 and 126.
#include "api.h"
#include "gemm_2cta_launch.cuh"

namespace b200 {

constexpr int MLP_STAGES = 5;   // with the staging slabs of eight warps

// Tiles that were cut along the contraction: the sum of their shares, in the order of the contraction, and the epilogue on it. A
// warp has one row of a tile. Grid (rest, 256 / 8).
template <int EPI>
__global__ void __launch_bounds__(256)
gemm2_sum_gated_kernel(const float* __restrict__ ws, const __nv_bfloat16* __restrict__ gate_up, __nv_bfloat16* __restrict__ halves,
                       __nv_bfloat16* __restrict__ act, int M, int I, Gemm2Params ep) {
  pdl_wait();
  constexpr bool FWD = EPI == G2_EPI_GATE_UP;
  constexpr int OUT_BN = FWD ? 128 : 256;
  int m_blk, n_blk;
  g2_tile_coords(blockIdx.x, (M + G2_BM - 1) / G2_BM, (I + OUT_BN - 1) / OUT_BN, ep.group_m, m_blk, n_blk);
  const int r = blockIdx.y * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const long long row = (long long)m_blk * G2_BM + r;
  // eight accumulators a lane: four gates and the ups that belong to them, or two fours of the product's gradient
  const int c0 = 4 * lane, c1 = 128 + 4 * lane, col0 = n_blk * OUT_BN + c0;
  if (row >= M || col0 >= I) return;
  const float* p = ws + ((long long)blockIdx.x * G2_BM + r) * 256;
  const long long step = (long long)ep.rest * G2_BM * 256;
  float v[2][4] = {};
  for (int s = 0; s < ep.splits; ++s) {
    const float4 a = *reinterpret_cast<const float4*>(p + s * step + c0), b = *reinterpret_cast<const float4*>(p + s * step + c1);
    v[0][0] += a.x; v[0][1] += a.y; v[0][2] += a.z; v[0][3] += a.w;
    v[1][0] += b.x; v[1][1] += b.y; v[1][2] += b.z; v[1][3] += b.w;
  }
  // four values as they are stored, and back
  auto round4 = [](const float (&x)[4]) { return make_uint2(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3])); };
  auto values = [](const uint2& x, float (&f)[4]) {
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x.y));
    f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
  };
  if constexpr (FWD) {
    const uint2 g = round4(v[0]), u = round4(v[1]);
    *reinterpret_cast<uint2*>(halves + row * 2 * I + col0) = g;
    *reinterpret_cast<uint2*>(halves + row * 2 * I + I + col0) = u;
    float a[4], b[4];
    values(g, a);
    values(u, b);
    swiglu_values(a, b, a);
    *reinterpret_cast<uint2*>(act + row * I + col0) = round4(a);
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int col = col0 + 128 * h;
      if (col >= I) continue;
      const long long at = row * 2 * I + col;
      float a[4], b[4], d[4];
      values(*reinterpret_cast<const uint2*>(gate_up + at), a);
      values(*reinterpret_cast<const uint2*>(gate_up + at + I), b);
      values(round4(v[h]), d);
      swiglu_grads(a, b, d);
      *reinterpret_cast<uint2*>(halves + at) = round4(a);
      *reinterpret_cast<uint2*>(halves + at + I) = round4(b);
    }
  }
}

static long long mlp_tiles(int M, int I, bool backward) {
  const int cols = backward ? 256 : 128;
  return (long long)((M + G2_BM - 1) / G2_BM) * ((I + cols - 1) / cols);
}

template <bool B_MN, int EPI>
static int launch_mlp(const void* A, const void* B, const void* gate_up, void* halves, void* act, int M, int N, int I, int K,
                      long long lda, long long ldb, float* ws, long long ws_floats, uint32_t* status, int num_sms,
                      cudaStream_t stream) {
  using SM = Gemm2Smem<256, MLP_STAGES, EPI>;
  constexpr bool BACKWARD = EPI == G2_EPI_DGATE_UP;
  auto kern = gemm2_bf16_kernel<256, MLP_STAGES, false, B_MN, EPI>;
  static int whole[16] = {0};
  int np = 0;
  if (const int rc = resident_pairs(kern, whole, SM::TOTAL, g2_threads(EPI), num_sms, np)) return rc;
  const long long tiles = mlp_tiles(M, I, BACKWARD);
  if (tiles > INT_MAX) return B200_ERR_TOO_LARGE;
  Gemm2Params ep{};
  ep.up_row0 = I;
  ep.group_m = 8;
  ep.a_bytes = SM::A_BYTES;
  ep.ws = ws;
  ep.rest = ws != nullptr ? g2_rest(tiles, np, (K + G2_BK - 1) / G2_BK, ep.splits) : 0;
  if (ep.rest > 0 && ws_floats < g2_ws_floats(ep.rest, ep.splits, 256)) ep.rest = 0;
  CUtensorMap tmA, tmB, tmC, tmW;
  if (make_tmap_2d(&tmA, A, M, K, lda, G2_BM_CTA, G2_BK, 2)) return B200_ERR_TENSORMAP;
  if (B_MN ? make_tmap_2d(&tmB, B, K, N, ldb, 64, 64, 2) : make_tmap_2d(&tmB, B, N, K, ldb, 128, G2_BK, 2)) return B200_ERR_TENSORMAP;
  const int cols = BACKWARD ? 32 : 64;
  const CUtensorMapSwizzle swizzle = BACKWARD ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
  if (make_tmap_halves(&tmW, halves, M, I, cols, swizzle)) return B200_ERR_TENSORMAP;
  if (BACKWARD ? make_tmap_halves(&tmC, gate_up, M, I, cols, swizzle) : make_tmap_out(&tmC, act, M, I, I, 0)) return B200_ERR_TENSORMAP;
  kern<<<2 * (int)(ep.rest > 0 || tiles >= np ? np : tiles), g2_threads(EPI), SM::TOTAL, stream>>>(tmA, tmB, tmC, tmW, M, N, K, ep,
                                                                                                status);
  if (cudaGetLastError() != cudaSuccess) return B200_ERR_LAUNCH;
  if (ep.rest > 0 && launch_pdl(gemm2_sum_gated_kernel<EPI>, dim3(ep.rest, G2_BM / 8), dim3(256), 0, stream, (const float*)ws,
                                (const __nv_bfloat16*)gate_up, (__nv_bfloat16*)halves, (__nv_bfloat16*)act, M, I, ep) != cudaSuccess)
    return B200_ERR_LAUNCH;
  return 0;
}

static bool misaligned(const void* p) { return reinterpret_cast<uintptr_t>(p) & 15; }

}  // namespace b200

extern "C" {

int b200_gemm_gate_up(const void* x, const void* W, void* gate_up, void* act, int M, int I, int K, long long ldx, long long ldw,
                      float* ws, long long ws_floats, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (M <= G2_BM_CTA || I <= 0 || I > INT_MAX / 2 || (I & 7) || K <= 0 || (ldx & 7) || (ldw & 7) || misaligned(gate_up) ||
      misaligned(act))
    return B200_ERR_ARG;
  // a tile has 128 gates and their 128 ups
  return launch_mlp<false, G2_EPI_GATE_UP>(x, W, nullptr, gate_up, act, M, 2 * I, I, K, ldx, ldw, ws, ws_floats, status, num_sms, stream);
}

int b200_gemm_dgate_up(const void* dy, const void* W, const void* gate_up, void* dgate_up, int M, int I, int K, long long lddy,
                       long long ldw, float* ws, long long ws_floats, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (M <= G2_BM_CTA || I <= 0 || (I & 7) || K <= 0 || (lddy & 7) || (ldw & 7) || misaligned(gate_up) || misaligned(dgate_up))
    return B200_ERR_ARG;
  return launch_mlp<true, G2_EPI_DGATE_UP>(dy, W, gate_up, dgate_up, nullptr, M, I, I, K, lddy, ldw, ws, ws_floats, status, num_sms,
                                           stream);
}

long long b200_gemm_gated_scratch(int M, int I, int K, int backward, int num_sms) {
  using namespace b200;
  if (M <= G2_BM_CTA || I <= 0 || K <= 0 || num_sms < 2) return 0;
  int splits = 0;
  const int rest = g2_rest(mlp_tiles(M, I, backward), num_sms / 2, (K + G2_BK - 1) / G2_BK, splits);
  return g2_ws_floats(rest, splits, 256);
}

}  // extern "C"
