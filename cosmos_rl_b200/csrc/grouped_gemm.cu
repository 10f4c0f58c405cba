// Grouped (per-expert) bf16 GEMMs for mixture-of-experts layers on tcgen05/TMEM, replacing the
// grouped_gemm / torch._grouped_mm library calls of the reference (cosmos_rl/policy/kernel/moe/moe.py:420-443,
// moe/grouped_gemm.py:33-165).
//
// Tokens routed to the local experts are stored sorted by expert in one [Mp, *] buffer in which every
// expert's block starts on a multiple of 128 rows (padding rows are zero). Then a 128-row output tile belongs
// to exactly one expert and a 64-row contraction block never straddles two experts, so all three GEMMs run on
// the dense pipelines of gemm_core.cuh and, on CTA pairs, gemm_2cta.cuh with a different tile schedule and 3-D tensor maps
// over the stacked expert weights [E, N, K]:
//   forward  Y[Mp, N]   = X[Mp, K] . W[e]^T                      (A 2-D K-major, B 3-D K-major, z = expert)
//   dgrad    dX[Mp, K]  = dY[Mp, N] . W[e]                       (A 2-D K-major, B 3-D MN-major)
//   wgrad    dW[e][N,K] (+)= dY[rows of e]^T . X[rows of e]      (A, B 2-D MN-major, contraction = the expert's rows)
// Tile counts and expert boundaries are read from device memory (tile_expert / expert_offsets / n_tiles), so
// no host synchronisation sits between routing and the expert GEMMs.
#include "gemm_core.cuh"
#include "gemm_2cta_launch.cuh"
#include "api.h"

namespace b200 {

struct GroupedParams {
  const CUtensorMap* tm_out;  // output as [batches, rows, N] (batches = experts for wgrad, else 1): boxes of 32 rows x 128 bytes
  const CUtensorMap* tm_act;  // gate/up projection: [rows, N / 2] activation, and tm_out is [rows][2][N / 2]
  const __nv_bfloat16* old;   // bf16 output that is accumulated into: its values are added in fp32 before the one rounding
  long long ld_old, batch_old;
  int N;                      // output columns
  int rows_limit;             // fwd/dgrad: allocated rows of C; wgrad: output rows per expert
  int out_fp32, accumulate, bn, batched;
  const int* tile_expert;     // [max_tiles] expert of each 128-row tile (fwd/dgrad)
  const int* expert_offsets;  // [E + 1] padded row offsets (wgrad)
  const int* filled;          // [E] rows that are not padding (wgrad), nullable
  const int* n_tiles;         // [1] number of 128-row tiles in use
  int num_experts;
};

// Each warp turns its 32 accumulator rows into slabs of 32 rows x 128 bytes in swizzled shared memory and hands them to
// TMA stores (reduce-adds when an fp32 result is accumulated), which clip rows and columns outside the output. The weight
// gradient is bound by these stores: an expert of 256 tokens has four contraction blocks per 64 KB of output.
struct GroupedEpilogue {
  using Params = GroupedParams;
  static constexpr bool CUSTOM_TILE = true;
  uint32_t slab_idx = 0;
  __device__ __forceinline__ void finish(const Params&) {
    if (elect_one()) tma_store_wait<0>();
  }
  __device__ __forceinline__ void tile(const Params& p, const TileInfo& t, int, uint32_t taddr, uint8_t* epi_smem) {
    const int lane = threadIdx.x & 31, quad = (threadIdx.x >> 5) & 3;
    uint8_t* slab0 = epi_smem + quad * 8192;
    const uint32_t sw = (uint32_t)(lane & 7);   // 128-byte swizzle: 16-byte chunk j of row r sits at chunk j ^ (r & 7)
    const int row0 = t.m_blk * GEMM_BM + quad * 32;
    const int batch = p.batched ? t.batch : 0;
    const int slab_cols = p.out_fp32 ? 32 : 64;
#pragma unroll 1
    for (int c = 0; c < p.bn; c += slab_cols) {
      const int gc = t.n_blk * p.bn + c;
      if (gc >= p.N) break;
      uint8_t* slab = slab0 + (slab_idx & 1) * 4096;
      if (elect_one()) tma_store_wait_read<1>();   // the store issued two slabs ago has finished reading this buffer
      __syncwarp();
      uint8_t* my_row = slab + lane * 128;
      uint32_t r[2][32];
      tmem_ld_32x32b_x32(taddr + c, r[0]);
      if (!p.out_fp32) tmem_ld_32x32b_x32(taddr + c + 32, r[1]);
      tmem_ld_wait();
      if (t.num_kb == 0) {   // an expert without rows
#pragma unroll
        for (int j = 0; j < 32; ++j) r[0][j] = r[1][j] = 0u;
      }
      if (p.old != nullptr && row0 + lane < p.rows_limit) {
        const __nv_bfloat16* o = p.old + batch * p.batch_old + (long long)(row0 + lane) * p.ld_old + gc;
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (gc + j < p.N) r[j >> 5][j & 31] = __float_as_uint(__uint_as_float(r[j >> 5][j & 31]) + __bfloat162float(o[j]));
      }
      if (p.out_fp32) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(my_row + ((((uint32_t)j) ^ sw) << 4)) =
              make_uint4(r[0][4 * j], r[0][4 * j + 1], r[0][4 * j + 2], r[0][4 * j + 3]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t(&v)[32] = r[j >> 2];
          const int k = (j & 3) * 8;
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(v[k]), __uint_as_float(v[k + 1]));
          o.y = pack_bf16x2(__uint_as_float(v[k + 2]), __uint_as_float(v[k + 3]));
          o.z = pack_bf16x2(__uint_as_float(v[k + 4]), __uint_as_float(v[k + 5]));
          o.w = pack_bf16x2(__uint_as_float(v[k + 6]), __uint_as_float(v[k + 7]));
          *reinterpret_cast<uint4*>(my_row + ((((uint32_t)j) ^ sw) << 4)) = o;
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (elect_one()) {
        if (row0 < p.rows_limit) {
          if (p.accumulate && p.out_fp32) tma_reduce_add_3d(p.tm_out, slab, gc, row0, batch);
          else tma_store_3d(p.tm_out, slab, gc, row0, batch);
        }
        tma_store_commit();
      }
      ++slab_idx;
    }
  }
};

// Gate/up projection: 128 gate columns and the 128 up columns that go with them; they leave as they are, and with their
// activation, which is formed from the rounded values and has the bits of a pass over them. The pass read and wrote 12 bytes an
// element of it at memory speed; here it is 4, written under the next tile's products (4096 tokens, 8 of 128 experts of 768 each:
// 217 us for the product and 36 for the pass, 232). On CTA pairs G2_EPI_GROUPED_GATE_UP does the same (16 experts, 4096 tokens: the
// layer forward and backward 1040 us with the pass, 1018).
struct GroupedGateUpEpilogue {
  using Params = GroupedParams;
  static constexpr bool CUSTOM_TILE = true;
  uint32_t slab_idx = 0;
  __device__ __forceinline__ void finish(const Params&) {
    if (elect_one()) tma_store_wait<0>();
  }
  __device__ __forceinline__ void tile(const Params& p, const TileInfo& t, int, uint32_t taddr, uint8_t* epi_smem) {
    const int lane = threadIdx.x & 31, quad = (threadIdx.x >> 5) & 3;
    uint8_t* slab0 = epi_smem + quad * 8192;
    const uint32_t sw = (uint32_t)(lane & 7);
    const int row0 = t.m_blk * GEMM_BM + quad * 32, inter = p.N / 2;
    auto put = [&](const uint32_t (&v)[32], auto store) {   // 64 columns as bf16 pairs, through the next staging slab
      uint8_t* slab = slab0 + (slab_idx++ & 1) * 4096;
      if (elect_one()) tma_store_wait_read<1>();   // the store issued two slabs ago has finished reading this buffer
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(slab + lane * 128 + ((((uint32_t)j) ^ sw) << 4)) =
            make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      fence_proxy_async_smem();
      __syncwarp();
      if (elect_one()) {
        store(slab);
        tma_store_commit();
      }
    };
    auto fetch = [&](uint32_t col, uint32_t (&v)[32]) {   // accumulator columns col .. col + 63, rounded
      uint32_t r[2][32];
      tmem_ld_32x32b_x32(taddr + col, r[0]);
      tmem_ld_32x32b_x32(taddr + col + 32, r[1]);
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 32; ++j)
        v[j] = pack_bf16x2(__uint_as_float(r[j >> 4][2 * (j & 15)]), __uint_as_float(r[j >> 4][2 * (j & 15) + 1]));
    };
#pragma unroll 1
    for (int c = 0; c < 128; c += 64) {
      const int gc = t.n_blk * 128 + c;
      if (gc >= inter) break;
      uint32_t g[32], u[32];
      fetch(c, g);
      put(g, [&](uint8_t* slab) { tma_store_3d(p.tm_out, slab, gc, 0, row0); });
      fetch(128 + c, u);
      put(u, [&](uint8_t* slab) { tma_store_3d(p.tm_out, slab, gc, 1, row0); });
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float a[8], b[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          a[2 * j] = __uint_as_float(g[4 * q + j] << 16);
          a[2 * j + 1] = __uint_as_float(g[4 * q + j] & 0xffff0000u);
          b[2 * j] = __uint_as_float(u[4 * q + j] << 16);
          b[2 * j + 1] = __uint_as_float(u[4 * q + j] & 0xffff0000u);
        }
        swiglu_values(a, b, a);
#pragma unroll
        for (int j = 0; j < 4; ++j) g[4 * q + j] = pack_bf16x2(a[2 * j], a[2 * j + 1]);
      }
      put(g, [&](uint8_t* slab) { tma_store_2d(p.tm_act, slab, gc, row0); });
    }
  }
};

// forward / dgrad: tiles = (128-row tile of the padded token buffer) x (BN-column tile)
struct TokenTileSchedule {
  int num_n, total, num_kb, bn;
  const int* tile_expert;
  __device__ __forceinline__ void init(int, int N, int K, int BN, const GroupedParams& p) {
    num_n = (N + BN - 1) / BN;
    total = p.n_tiles[0] * num_n;
    num_kb = (K + GEMM_BK - 1) / GEMM_BK;
    tile_expert = p.tile_expert;
    bn = BN;
  }
  __device__ __forceinline__ bool get(int it, TileInfo& t) const {
    int i = blockIdx.x + it * gridDim.x;
    if (i >= total) return false;
    // n fastest: CTAs running at the same time share the token tile's expert, i.e. the same weight slice in L2
    t.m_blk = i / num_n;
    t.n_blk = i - t.m_blk * num_n;
    t.a_mn0 = t.m_blk * GEMM_BM;
    t.b_mn0 = t.n_blk * bn;
    t.k0 = 0;
    t.num_kb = num_kb;
    t.batch = tile_expert[t.m_blk];
    return true;
  }
};

// gate/up projection: the same with 128 columns of either half of N
struct GateUpTileSchedule : TokenTileSchedule {
  int inter;
  __device__ __forceinline__ void init(int M, int N, int K, int BN, const GroupedParams& p) {
    TokenTileSchedule::init(M, N / 2, K, BN / 2, p);
    inter = N / 2;
  }
  __device__ __forceinline__ bool get(int it, TileInfo& t) const {
    if (!TokenTileSchedule::get(it, t)) return false;
    t.b_mn1 = inter + t.b_mn0;
    return true;
  }
};

// wgrad: tiles = expert x (128-row tile of dW) x (BN-column tile of dW); contraction over the expert's rows
struct ExpertWgradSchedule {
  int num_m, num_n, per_expert, total, bn;
  const int *off, *filled;
  __device__ __forceinline__ void init(int M, int N, int, int BN, const GroupedParams& p) {
    num_m = (M + GEMM_BM - 1) / GEMM_BM;
    num_n = (N + BN - 1) / BN;
    per_expert = num_m * num_n;
    total = per_expert * p.num_experts;
    off = p.expert_offsets;
    filled = p.filled;
    bn = BN;
  }
  __device__ __forceinline__ bool get(int it, TileInfo& t) const {
    int i = blockIdx.x + it * gridDim.x;
    if (i >= total) return false;
    const int e = i / per_expert, r = i - e * per_expert;
    t.m_blk = r / num_n;
    t.n_blk = r - t.m_blk * num_n;
    t.a_mn0 = t.m_blk * GEMM_BM;
    t.b_mn0 = t.n_blk * bn;
    t.k0 = off[e];
    t.num_kb = (off[e + 1] - off[e]) / GEMM_BK;
    if (filled) t.num_kb = min(t.num_kb, (filled[e] + GEMM_BK - 1) / GEMM_BK);
    t.batch = e;
    return true;
  }
};

constexpr int GG_BN = 256, GG_STAGES = 4;

__global__ void __launch_bounds__(GEMM_THREADS, 1)
grouped_fwd_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmC, int M, int N, int K, GroupedParams ep, uint32_t* status) {
  ep.tm_out = &tmC;
  gemm_mainloop<GG_BN, GG_STAGES, GroupedEpilogue, TokenTileSchedule, GemmTraits<false, false, false, true>>(
      &tmA, &tmB, M, N, K, ep, status);
}
__global__ void __launch_bounds__(GEMM_THREADS, 1)
grouped_gate_up_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                       const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmD, int M, int N, int K,
                       GroupedParams ep, uint32_t* status) {
  ep.tm_out = &tmC;
  ep.tm_act = &tmD;
  gemm_mainloop<GG_BN, GG_STAGES, GroupedGateUpEpilogue, GateUpTileSchedule, GemmTraits<false, false, false, true, 0, false, true>>(
      &tmA, &tmB, M, N, K, ep, status);
}
__global__ void __launch_bounds__(GEMM_THREADS, 1)
grouped_dgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, int M, int N, int K, GroupedParams ep, uint32_t* status) {
  ep.tm_out = &tmC;
  gemm_mainloop<GG_BN, GG_STAGES, GroupedEpilogue, TokenTileSchedule, GemmTraits<false, true, false, true>>(
      &tmA, &tmB, M, N, K, ep, status);
}
__global__ void __launch_bounds__(GEMM_THREADS, 1)
grouped_wgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, int M, int N, int K, GroupedParams ep, uint32_t* status) {
  ep.tm_out = &tmC;
  gemm_mainloop<GG_BN, GG_STAGES, GroupedEpilogue, ExpertWgradSchedule, GemmTraits<true, true>>(&tmA, &tmB, M, N, K,
                                                                                                  ep, status);
}

// [batches, rows, cols] output, boxes of 32 rows x 128 bytes, 128-byte swizzle
static int make_tmap_grouped_out(CUtensorMap* out, const void* ptr, uint64_t batches, uint64_t rows, uint64_t cols,
                                 uint64_t ld, uint64_t ld_batch, int fp32) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) { last_tmap_error() = 1 << 24; return -1; }
  const uint64_t eb = fp32 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || ((ld * eb) & 15) || ((ld_batch * eb) & 15)) {
    last_tmap_error() = (2 << 24) | 0x40000;
    return -2;
  }
  cuuint64_t gdim[3] = {cols, rows, batches};
  cuuint64_t gstr[2] = {ld * eb, ld_batch * eb};
  cuuint32_t box[3] = {(cuuint32_t)(128 / eb), 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode_with_context([&] {
    return enc(out, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr),
               gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) last_tmap_error() = (3 << 24) | 0x40000 | (int)r;
  return r == CUDA_SUCCESS ? 0 : -3;
}

template <class Kern>
static int set_smem(Kern k, bool& done) {
  if (!done) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<GG_BN, GG_STAGES>::TOTAL_WITH_EPI) !=
        cudaSuccess)
      return B200_ERR_LAUNCH;
    done = true;
  }
  return 0;
}

// CTA pairs of a call of expert weight gradients, 0: single CTAs, or an error code. Single CTAs are bound by operands out of L2 (4.9
// blocks of 48 KB for 64 KB of result, 4096 tokens on 128 experts), and a pair on a 256 x 256 tile fetches two thirds of that. us,
// single CTAs and pairs, 1536 x 2048 a gradient: 256 rows for each of 128 experts 290 and 260, 512 rows 465 and 400, 2048 rows for
// each of 16 165 and 143; few rows are bound by the epilogue, of which a pair has the less: 44 rows 190 and 216, 6 rows 166 and
// 191. max_rows is what there is room for, up to 128 rows an expert more than there are. What the larger tiles waste at the edges
// and in the last round counts against them: with a fifth more rounds than single CTAs have they are still no slower (58 experts of
// 640 x 1144 58.1 and 58.3), with more they are (101 of 360 x 688, 1334 rows, 104 and 118; 8 of 1112 x 352, two rounds for one, 9.8
// and 13.1). A result in fp32 that is added to is bound by its way through memory up to twice as many rows (92 of 504 x 4064, 537
// rows, 356 and 418). A bf16 result that is added to keeps its one rounding in the other kernel.
using WG_SMEM = Gemm2Smem<256, 6>;
static int wgrad_pairs(int max_rows, int N, int K, int num_experts, int out_fp32, int accumulate, int num_sms) {
  if ((accumulate && !out_fp32) || num_sms < 2 || max_rows < (accumulate ? 640ll : 320ll) * num_experts) return 0;
  static int whole[16] = {0};
  int np = 0;
  if (const int rc = resident_pairs(gemm2_bf16_kernel<256, 6, true, true, G2_EPI_EXPERTS>, whole, WG_SMEM::TOTAL, G2_THREADS,
                                    num_sms, np))
    return rc;
  auto tiles = [&](int rows) { return (long long)num_experts * ((N + rows - 1) / rows) * ((K + 255) / 256); };
  auto rounds = [](long long n, int at_once) { return (n + at_once - 1) / at_once; };
  const long long pair_tiles = tiles(G2_BM);
  if (pair_tiles < np || pair_tiles >= (1ll << 31)) return 0;
  return 5 * rounds(pair_tiles, np) <= 6 * rounds(tiles(GEMM_BM), num_sms) ? np : 0;
}

// CTA pairs of a call of grouped GEMMs, 0: single CTAs, or an error code. A single CTA fetches 48 KB out of L2 for a block of
// 128 x 256 x 64, and that bounds it (770 cycles a block, products 512); a pair fetches 64 KB for twice the work. us, single CTAs
// and pairs (a cold L2), rows an expert in brackets: 16 experts of 1536 x 2048 94 and 80 (1024), 155 and 140 (2048); 16 of 1024 x 512
// 44 and 38 (2048); 8 of 28672 x 4096 2028 and 1398 (1024); input gradient of 8 of 14336 x 4096 905 and 699 (1024).
// Up to 128 rows half of a pair stands idle: 153 and 159 (64). Tiles of 256 rows are rounded up once an expert: with a tenth more
// rounds than single CTAs have pairs are no slower (64 of 1408 x 2048 151 and 143 (384)), with more it varies (128 of 1536 x 2048,
// 1.2, 224 and 226; of 2048 x 768 126 and 120; 5 rounds for 4, 413 and 433; 3 for 2, 19.4 and 23.6). Short contractions and few tiles
// are bound by what a tile costs beside its products (16 of 256 x 256 15.3 and 17.4 (2048)). max_rows is what there is room for,
// about 64 rows an expert more than the padded rows there are, from which both numbers of tiles are estimated.
using GR_SMEM = Gemm2Smem<256, 6, G2_EPI_GROUPED>;
template <bool B_MN>
constexpr auto grouped_pair_kernel = gemm2_bf16_kernel<256, 6, false, B_MN, G2_EPI_GROUPED>;
static int grouped_pairs(int max_rows, int N, int K, int num_experts, int mode, int num_sms) {
  if (num_sms < 2 || (N & 7) || K < 512 || max_rows < 320ll * num_experts) return 0;
  static int whole[2][16] = {};
  int np = 0;
  if (const int rc = resident_pairs(mode == 0 ? grouped_pair_kernel<false> : grouped_pair_kernel<true>, whole[mode != 0],
                                    GR_SMEM::TOTAL, G2_THREADS, num_sms, np))
    return rc;
  const long long num_n = (N + 255) / 256, pair_tiles = max_rows * num_n / G2_BM;
  const long long tiles = (max_rows - 64ll * num_experts) * num_n / GEMM_BM;
  if (pair_tiles < 2 * np || pair_tiles >= (1ll << 30)) return 0;
  return 10 * ((pair_tiles + np - 1) / np) <= 11 * ((tiles + num_sms - 1) / num_sms) ? np : 0;
}

}  // namespace b200

extern "C" {

// mode 0: Y[Mp, N] = X[Mp, K] . W[e]^T with W [E, N, K]
// mode 1: dX[Mp, N] = dY[Mp, K] . W[e]   with W [E, K, N]   (K is the contraction = rows of W[e])
// expert_offsets [E + 1] (nullable): the experts' first rows, for tiles of 256 rows that begin with each
int b200_grouped_gemm_rows(const void* X, const void* W, void* Y, int max_rows, int N, int K, int num_experts,
                           long long ldx, long long ldy, const int* expert_offsets, const int* tile_expert, const int* n_tiles,
                           int mode, int accumulate, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (max_rows <= 0 || N <= 0 || K <= 0 || (ldx & 7) || (max_rows % GEMM_BM)) return B200_ERR_ARG;
  const int np = expert_offsets && !accumulate ? grouped_pairs(max_rows, N, K, num_experts, mode, num_sms) : 0;
  if (np < 0) return np;
  CUtensorMap tmA, tmB, tmC;
  if (np > 0 ? make_tmap_out(&tmC, Y, max_rows, N, ldy, 0)
             : make_tmap_grouped_out(&tmC, Y, 1, max_rows, N, ldy, (uint64_t)max_rows * ldy, 0))
    return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tmA, X, max_rows, K, ldx, GEMM_BM, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  // W[e] stored [K(contraction), N(out)]: MN-major B, boxes of 64 contraction rows x 64 output columns
  if (mode == 0 ? make_tmap_3d(&tmB, W, num_experts, N, K, K, (uint64_t)N * K, np > 0 ? 128 : GG_BN, GEMM_BK, 2)
                : make_tmap_3d(&tmB, W, num_experts, K, N, N, (uint64_t)N * K, 64, 64, 2))
    return B200_ERR_TENSORMAP;
  if (np > 0) {
    Gemm2Params ep2{};
    ep2.a_bytes = GR_SMEM::A_BYTES;
    ep2.offsets = expert_offsets;
    ep2.experts = num_experts;
    const auto pair_kern = mode == 0 ? grouped_pair_kernel<false> : grouped_pair_kernel<true>;
    pair_kern<<<2 * np, G2_THREADS, GR_SMEM::TOTAL, stream>>>(tmA, tmB, tmC, tmC, max_rows, N, K, ep2, status);
    return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
  }
  static bool s0 = false, s1 = false;
  GroupedParams ep{nullptr, nullptr, accumulate ? (const __nv_bfloat16*)Y : nullptr, ldy, 0, N, max_rows, 0, accumulate, GG_BN, 0, tile_expert, nullptr, nullptr, n_tiles, num_experts};
  if (mode == 0 ? set_smem(grouped_fwd_kernel, s0) : set_smem(grouped_dgrad_kernel, s1)) return B200_ERR_LAUNCH;
  const auto kern = mode == 0 ? grouped_fwd_kernel : grouped_dgrad_kernel;
  kern<<<num_sms, GEMM_THREADS, GemmSmem<GG_BN, GG_STAGES>::TOTAL_WITH_EPI, stream>>>(tmA, tmB, tmC, max_rows, N, K, ep, status);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

// h1[Mp, 2 I] = X[Mp, K] . W[e]^T with W [E, 2 I, K] (gate rows, then up rows), act[Mp, I] = silu(gate) o up of the rounded h1.
int b200_grouped_gate_up(const void* X, const void* W, void* h1, void* act, int max_rows, int I, int K, int num_experts,
                         long long ldx, const int* expert_offsets, const int* tile_expert, const int* n_tiles, uint32_t* status,
                         int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (max_rows <= 0 || I <= 0 || I > (1 << 30) || (I & 7) || K <= 0 || (ldx & 7) || (max_rows % GEMM_BM)) return B200_ERR_ARG;
  int np = grouped_pairs(max_rows, 2 * I, K, num_experts, 0, num_sms);
  if (np < 0) return np;
  CUtensorMap tmA, tmB, tmC, tmD;   // both take boxes of 128 rows of A and of 128 gate or up rows
  if (make_tmap_2d(&tmA, X, max_rows, K, ldx, GEMM_BM, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_3d(&tmB, W, num_experts, 2 * I, K, K, (uint64_t)2 * I * K, GG_BN / 2, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_halves(&tmC, h1, max_rows, I, 64, CU_TENSOR_MAP_SWIZZLE_128B)) return B200_ERR_TENSORMAP;
  if (make_tmap_out(&tmD, act, max_rows, I, I, 0)) return B200_ERR_TENSORMAP;
  if (np > 0) {
    using SM = Gemm2Smem<256, 5, G2_EPI_GROUPED_GATE_UP>;
    auto kern = gemm2_bf16_kernel<256, 5, false, false, G2_EPI_GROUPED_GATE_UP>;
    static int whole[16] = {0};
    if (const int rc = resident_pairs(kern, whole, SM::TOTAL, g2_threads(G2_EPI_GROUPED_GATE_UP), num_sms, np)) return rc;
    Gemm2Params ep2{};
    ep2.up_row0 = I;
    ep2.a_bytes = SM::A_BYTES;
    ep2.offsets = expert_offsets;
    ep2.experts = num_experts;
    kern<<<2 * np, g2_threads(G2_EPI_GROUPED_GATE_UP), SM::TOTAL, stream>>>(tmA, tmB, tmD, tmC, max_rows, 2 * I, K, ep2, status);
    return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
  }
  static bool done = false;
  if (set_smem(grouped_gate_up_kernel, done)) return B200_ERR_LAUNCH;
  GroupedParams ep{nullptr, nullptr, nullptr, 2 * I, 0, 2 * I, max_rows, 0, 0, GG_BN, 0, tile_expert, nullptr, nullptr, n_tiles,
                   num_experts};
  grouped_gate_up_kernel<<<num_sms, GEMM_THREADS, GemmSmem<GG_BN, GG_STAGES>::TOTAL_WITH_EPI, stream>>>(tmA, tmB, tmC, tmD, max_rows,
                                                                                                       2 * I, K, ep, status);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

// Whether such a call that is given the experts' first rows takes CTA pairs.
int b200_grouped_gemm_pairs(int max_rows, int N, int K, int num_experts, int mode, int num_sms) {
  return b200::grouped_pairs(max_rows, N, K, num_experts, mode, num_sms) > 0;
}

int b200_grouped_gemm(const void* X, const void* W, void* Y, int max_rows, int N, int K, int num_experts,
                      long long ldx, long long ldy, const int* tile_expert, const int* n_tiles, int mode,
                      int accumulate, uint32_t* status, int num_sms, cudaStream_t stream) {
  return b200_grouped_gemm_rows(X, W, Y, max_rows, N, K, num_experts, ldx, ldy, nullptr, tile_expert, n_tiles, mode, accumulate,
                                status, num_sms, stream);
}

// Whether such a call of expert weight gradients takes CTA pairs.
int b200_grouped_wgrad_pairs(int max_rows, int N, int K, int num_experts, int out_fp32, int accumulate, int num_sms) {
  return b200::wgrad_pairs(max_rows, N, K, num_experts, out_fp32, accumulate, num_sms) > 0;
}

// dW[e][N, K] (+)= dY[rows of e, N]^T . X[rows of e, K]; rows of e = [expert_offsets[e], expert_offsets[e+1]). With `filled` only
// the first filled[e] of them count and the rest is zero: blocks of 64 rows that hold nothing else are left out (half of the
// experts have one; 4096 tokens, 8 of 128 experts each, 1536 x 2048 and 2048 x 768 a gradient: 395 us with them, 385).
int b200_grouped_wgrad_filled(const void* dY, const void* X, void* dW, int max_rows, int N, int K, int num_experts,
                              long long lddy, long long ldx, const int* expert_offsets, const int* filled, int out_fp32,
                              int accumulate, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (max_rows <= 0 || N <= 0 || K <= 0 || (lddy & 7) || (ldx & 7)) return B200_ERR_ARG;
  CUtensorMap tmA, tmB, tmC;
  if (make_tmap_grouped_out(&tmC, dW, num_experts, N, K, K, (uint64_t)N * K, out_fp32)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tmA, dY, max_rows, N, lddy, 64, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tmB, X, max_rows, K, ldx, 64, 64, 2)) return B200_ERR_TENSORMAP;
  const int np = wgrad_pairs(max_rows, N, K, num_experts, out_fp32, accumulate, num_sms);
  if (np < 0) return np;
  if (np > 0) {
    Gemm2Params ep2{};
    ep2.out_fp32 = out_fp32;
    ep2.accumulate = accumulate;
    ep2.a_bytes = WG_SMEM::A_BYTES;
    ep2.offsets = expert_offsets;
    ep2.filled = filled;
    ep2.experts = num_experts;
    gemm2_bf16_kernel<256, 6, true, true, G2_EPI_EXPERTS><<<2 * np, G2_THREADS, WG_SMEM::TOTAL, stream>>>(
        tmA, tmB, tmC, tmC, N, K, 0, ep2, status);
    return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
  }
  static bool s2 = false;
  if (set_smem(grouped_wgrad_kernel, s2)) return B200_ERR_LAUNCH;
  GroupedParams ep{nullptr, nullptr, accumulate && !out_fp32 ? (const __nv_bfloat16*)dW : nullptr, K, (long long)N * K, K, N, out_fp32,
                   accumulate, GG_BN, 1, nullptr, expert_offsets, filled, nullptr, num_experts};
  grouped_wgrad_kernel<<<num_sms, GEMM_THREADS, GemmSmem<GG_BN, GG_STAGES>::TOTAL_WITH_EPI, stream>>>(tmA, tmB, tmC, N, K,
                                                                                                     0, ep, status);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

int b200_grouped_wgrad(const void* dY, const void* X, void* dW, int max_rows, int N, int K, int num_experts,
                       long long lddy, long long ldx, const int* expert_offsets, int out_fp32, int accumulate,
                       uint32_t* status, int num_sms, cudaStream_t stream) {
  return b200_grouped_wgrad_filled(dY, X, dW, max_rows, N, K, num_experts, lddy, ldx, expert_offsets, nullptr, out_fp32,
                                   accumulate, status, num_sms, stream);
}

}  // extern "C"
