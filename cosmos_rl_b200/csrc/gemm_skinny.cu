// Weight-streaming GEMM for decode-sized batches (M <= 256 rows) and the fused reductions that follow it.
//
//   y[M, N] = x[M, K] * W[N, K]^T      x, W bf16 (K contiguous)
//
// With so few rows the cost of a projection is reading W once from HBM, so the work is cut into
// (column tile, contraction split) units until every SM streams its own slice of W: a tile is 128 rows x 128
// columns on the tcgen05 pipeline of gemm_core.cuh, a split covers a contiguous range of 64-wide contraction
// blocks. With one split the epilogue writes bf16 (+ bias, or SwiGLU of a fused gate/up weight) directly;
// with several it writes fp32 partial tiles to a workspace [splits, M, N] that stays in L2, and one of the
// reduction kernels below finishes the layer step it belongs to:
//   * splitk_reduce                      y = sum (+ bias)
//   * splitk_reduce_residual_rmsnorm     res' = sum + res;  y = rmsnorm(res') * w          (o_proj, down_proj)
//   * splitk_reduce_qkv_rope_append      q = rope(sum + bias), K/V rows written into the paged cache (qkv_proj)
// so the decode layer has no separate bias / RoPE / cache-append / residual / norm launches. This replaces what
// the reference gets from vLLM's fused decode kernels (cosmos_rl/rollout/vllm_rollout/vllm_rollout.py:249-339).
#include "gemm_core.cuh"
#include "api.h"

namespace b200 {

// Tile widths: 128 columns when the contraction has to be split to occupy the machine, 256 columns when the column
// tiles alone do: a wider tile re-reads the activation rows half as often, and with 128 rows per tile that traffic out
// of L2 is as large as the weight stream itself. Up to 16 or 64 rows only those rows are kept per stage and the room
// goes into more stages, i.e. more of the weight stream in flight.
template <int BN, int A_ROWS>
struct SkinnyCfg {
  static constexpr int STAGES = BN == 256 ? (A_ROWS == 16 ? 5 : 4) : (A_ROWS == 16 ? 10 : A_ROWS == 64 ? 8 : 6);
  static constexpr int ROW_STORE_STAGES = A_ROWS == 16 ? 6 : A_ROWS == 64 ? 5 : 4;   // 256 wide, no store staging
  static constexpr int SMEM_LIMIT = 227 * 1024;
  static_assert(GemmSmem<BN, STAGES, A_ROWS>::TOTAL_WITH_EPI <= SMEM_LIMIT, "shared memory");
  static_assert(GemmSmem<256, ROW_STORE_STAGES, A_ROWS>::TOTAL <= SMEM_LIMIT, "shared memory");
};

// Gate value of accumulator rows that belong to no row of x and are not stored. What they hold (zeros, whatever follows the
// tile) sends the whole warp through the division's path for special operands: gate/up of 14336 x 4096, 5 rows 57.6 us, 45.
constexpr float SKINNY_NO_ROW = 1.f;

struct SkinnyParams {
  const CUtensorMap* tm_out;  // bf16 [M, N] (direct output) or fp32 [splits, M, N] (partials), boxes of 32 rows x 128 bytes
  const void* bias;           // [N], nullable (direct output only; the reduce kernels add it otherwise)
  int bias_bf16;
  int to_ws;                  // 1: fp32 partials through the 3-D map; 0: bf16 result through the 2-D map
  int M, N;                   // N = columns of the output (for SwiGLU: the intermediate size)
  int splits;
  __nv_bfloat16* out;         // direct output: the row-store epilogue, and what the tensor map leaves out
  long long ldo;
  int up_row0;                // SwiGLU: first "up" row of W
  int b_rows;                 // rows of W per tile (BN, or the width chosen at launch)
  int a_bytes;                // bytes of A a stage: the rows that are fetched
  int prefetch_kb;            // contraction blocks a CTA brings into L2 before it waits for the previous kernel
};

template <int BN, bool SWIGLU>
struct SkinnySchedule {
  int num_m, num_n, splits, num_kb, total, up_row0, out_bn;
  __device__ __forceinline__ void init(int M, int N, int K, int, const SkinnyParams& p) {
    num_m = (M + GEMM_BM - 1) / GEMM_BM;
    out_bn = SWIGLU ? p.b_rows / 2 : BN;
    num_n = (p.N + out_bn - 1) / out_bn;
    splits = p.splits;
    num_kb = (K + GEMM_BK - 1) / GEMM_BK;
    total = num_m * num_n * splits;
    up_row0 = p.up_row0;
  }
  // units that share a slice of W (the row blocks of one (column tile, split)) are neighbours in the launch
  // order, so the slice is read from HBM once and from L2 by the others
  __device__ __forceinline__ bool get(int it, TileInfo& t) const {
    const int u = blockIdx.x + it * gridDim.x;
    if (u >= total) return false;
    t.m_blk = u % num_m;
    const int r = u / num_m;
    const int s = r % splits;
    t.n_blk = r / splits;
    const int kb0 = (int)(((long long)s * num_kb) / splits);
    const int kb1 = (int)(((long long)(s + 1) * num_kb) / splits);
    t.a_mn0 = t.m_blk * GEMM_BM;
    if (SWIGLU) {
      t.b_mn0 = t.n_blk * out_bn;
      t.b_mn1 = up_row0 + t.n_blk * out_bn;
    } else {
      t.b_mn0 = t.n_blk * BN;
      t.b_mn1 = 0;
    }
    t.k0 = kb0 * GEMM_BK;
    t.num_kb = kb1 - kb0;
    t.batch = s;
    return true;
  }
};

// Epilogue: each warp turns its 32 accumulator rows into slabs of 32 rows x 128 bytes (32 fp32 or 64 bf16 columns) in
// swizzled shared memory and hands them to TMA stores, which clip rows >= M and columns >= N; the columns of a last, incomplete 16
// bytes of a bf16 row are left to the threads (TAIL: there are any; a test in the loop took 0.5 us of a decode block's 115).
template <int BN, bool SWIGLU, bool TAIL>
struct SkinnyEpilogue {
  using Params = SkinnyParams;
  static constexpr bool CUSTOM_TILE = true;
  uint32_t slab_idx = 0;
  __device__ __forceinline__ void finish(const Params&) {
    if (elect_one()) tma_store_wait<0>();
  }
  __device__ __forceinline__ void tile(const Params& p, const TileInfo& t, int row, uint32_t taddr, uint8_t* epi_smem) {
    constexpr int OUT_BN = SWIGLU ? BN / 2 : BN;
    const int lane = threadIdx.x & 31;
    const int quad = (threadIdx.x >> 5) & 3;
    uint8_t* slab0 = epi_smem + quad * 8192;
    const uint32_t sw = (uint32_t)(lane & 7);
    const int row0 = t.m_blk * GEMM_BM + quad * 32;
    if (row0 >= p.M) return;
    const int slab_cols = p.to_ws ? 32 : 64;
#pragma unroll 1
    for (int c = 0; c < OUT_BN; c += slab_cols) {
      uint8_t* slab = slab0 + (slab_idx & 1) * 4096;
      if (elect_one()) tma_store_wait_read<1>();  // the store issued two slabs ago has finished reading this buffer
      __syncwarp();
      uint8_t* my_row = slab + lane * 128;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (p.to_ws && h == 1) break;
        const int cc = c + h * 32;
        uint32_t a[32];
        float v[32];
        tmem_ld_32x32b_x32(taddr + cc, a);
        if constexpr (SWIGLU) {
          uint32_t u[32];
          tmem_ld_32x32b_x32(taddr + BN / 2 + cc, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = row0 + lane < p.M ? __uint_as_float(a[j]) : SKINNY_NO_ROW;
          swiglu_values(v, reinterpret_cast<const float(&)[32]>(u), v);
        } else {
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = (t.num_kb > 0) ? __uint_as_float(a[j]) : 0.f;
        }
        if (p.to_ws) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(my_row + ((((uint32_t)j) ^ sw) << 4)) =
                make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else {
          if (p.bias != nullptr) {
            const int gc = t.n_blk * OUT_BN + cc;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (gc + j < p.N)
                v[j] += p.bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[gc + j])
                                    : reinterpret_cast<const float*>(p.bias)[gc + j];
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 o;
            o.x = pack_bf16x2(v[8 * j], v[8 * j + 1]);
            o.y = pack_bf16x2(v[8 * j + 2], v[8 * j + 3]);
            o.z = pack_bf16x2(v[8 * j + 4], v[8 * j + 5]);
            o.w = pack_bf16x2(v[8 * j + 6], v[8 * j + 7]);
            *reinterpret_cast<uint4*>(my_row + ((((uint32_t)(4 * h + j)) ^ sw) << 4)) = o;
          }
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      const int gc = t.n_blk * OUT_BN + c;
      if (elect_one()) {
        if (gc < (TAIL ? whole16(p.N, 0) : p.N) && row0 < p.M) {
          if (p.to_ws) tma_store_3d(p.tm_out, slab, gc, row0, t.batch);
          else tma_store_2d(p.tm_out, slab, gc, row0);
        }
        tma_store_commit();
      }
      if constexpr (TAIL)
        if (row0 + lane < p.M) store_tail(p.out + (long long)(row0 + lane) * p.ldo, slab, gc, p.N, false);
      ++slab_idx;
    }
  }
};

// SwiGLU tiles of any width (a multiple of 8 columns): a tile's edge need not be a multiple of a store box, so rows are
// written with plain 16-byte stores.
struct SwigluRowsEpilogue {
  using Params = SkinnyParams;
  static constexpr bool CUSTOM_TILE = true;
  __device__ __forceinline__ void finish(const Params&) {}
  __device__ __forceinline__ void tile(const Params& p, const TileInfo& t, int row, uint32_t taddr, uint8_t*) {
    const int width = p.b_rows / 2, r = t.m_blk * GEMM_BM + row, gc0 = t.n_blk * width;
    if (r - (int)(threadIdx.x & 31) >= p.M) return;   // none of the warp's rows
    __nv_bfloat16* dst = p.out + (long long)r * p.ldo + gc0;
#pragma unroll 1
    for (int c = 0; c < width; c += 16) {
      uint32_t a[16], u[16];
      tmem_ld_32x32b_x16(taddr + c, a);
      tmem_ld_32x32b_x16(taddr + width + c, u);
      tmem_ld_wait();
      float v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = r < p.M ? __uint_as_float(a[j]) : SKINNY_NO_ROW;
      swiglu_values(v, reinterpret_cast<const float(&)[16]>(u), v);
      if (r >= p.M) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cc = c + 8 * h;
        if (cc >= width) continue;
        if (gc0 + cc + 8 <= p.N) {
          uint4 o;
          o.x = pack_bf16x2(v[8 * h], v[8 * h + 1]);
          o.y = pack_bf16x2(v[8 * h + 2], v[8 * h + 3]);
          o.z = pack_bf16x2(v[8 * h + 4], v[8 * h + 5]);
          o.w = pack_bf16x2(v[8 * h + 6], v[8 * h + 7]);
          *reinterpret_cast<uint4*>(dst + cc) = o;
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (gc0 + cc + j < p.N) dst[cc + j] = __float2bfloat16(v[8 * h + j]);
        }
      }
    }
  }
};

template <int BN, bool SWIGLU, int A_ROWS, bool TAIL>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmO, int M, int N, int K, SkinnyParams ep, uint32_t* status) {
  ep.tm_out = &tmO;
  if (threadIdx.x == 0) tma_prefetch_desc(&tmO);
  gemm_mainloop<BN, SkinnyCfg<BN, A_ROWS>::STAGES, SkinnyEpilogue<BN, SWIGLU, TAIL>, SkinnySchedule<BN, SWIGLU>,
                GemmTraits<false, false, false, false, 0, false, SWIGLU, true, A_ROWS, false, true>>(&tmA, &tmB, M, N, K, ep, status);
}

template <int A_ROWS>
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_skinny_swiglu_rows_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M,
                               int N, int K, SkinnyParams ep, uint32_t* status) {
  gemm_mainloop<256, SkinnyCfg<256, A_ROWS>::ROW_STORE_STAGES, SwigluRowsEpilogue, SkinnySchedule<256, true>,
                GemmTraits<false, false, false, false, 0, false, true, true, A_ROWS, true, true>>(&tmA, &tmB, M, N, K, ep, status);
}

// fp32 [splits, M, N] partials: boxes of 32 rows x 32 columns, 128-byte swizzle
static int make_tmap_ws(CUtensorMap* out, const float* ws, int splits, int M, int N) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) return -1;
  if ((reinterpret_cast<uintptr_t>(ws) & 15) || (N & 3)) return -2;
  cuuint64_t gdim[3] = {(cuuint64_t)N, (cuuint64_t)M, (cuuint64_t)splits};
  cuuint64_t gstr[2] = {(cuuint64_t)N * 4, (cuuint64_t)M * N * 4};
  cuuint32_t box[3] = {32, 32, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode_with_context([&] {
    return enc(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ws), gdim, gstr, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) last_tmap_error() = (3 << 24) | 0x20000 | (int)r;
  return r == CUDA_SUCCESS ? 0 : -3;
}

// bf16 [M, N] result: boxes of 32 rows x 64 columns, 128-byte swizzle
static int make_tmap_out16(CUtensorMap* out, const void* ptr, int M, int N, long long ld) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) return -1;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (ld & 7)) return -2;
  cuuint64_t gdim[2] = {(cuuint64_t)N, (cuuint64_t)M};
  cuuint64_t gstr[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {64, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_with_context([&] {
    return enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), gdim, gstr, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) last_tmap_error() = (3 << 24) | 0x30000 | (int)r;
  return r == CUDA_SUCCESS ? 0 : -3;
}

// ---------------------------------------------------------------------------------------------------
// reductions over the split-K workspace
// ---------------------------------------------------------------------------------------------------
__device__ __forceinline__ float bias_at(const void* bias, int bias_bf16, int i) {
  return bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(bias)[i])
                   : reinterpret_cast<const float*>(bias)[i];
}

// y[r, :] = sum_s ws[s, r, :] (+ bias); N % 4 == 0
__global__ void splitk_reduce_kernel(const float* __restrict__ ws, int splits, int M, int N, const void* bias,
                                     int bias_bf16, __nv_bfloat16* __restrict__ out, long long ldo) {
  pdl_launch_dependents();
  pdl_wait();
  const long long n4 = (long long)M * (N / 4);
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / (N / 4)), c = (int)(i % (N / 4)) * 4;
    float4 acc = *reinterpret_cast<const float4*>(ws + (long long)r * N + c);
#pragma unroll 4
    for (int s = 1; s < splits; ++s) {
      const float4 v = *reinterpret_cast<const float4*>(ws + ((long long)s * M + r) * N + c);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    if (bias) {
      acc.x += bias_at(bias, bias_bf16, c); acc.y += bias_at(bias, bias_bf16, c + 1);
      acc.z += bias_at(bias, bias_bf16, c + 2); acc.w += bias_at(bias, bias_bf16, c + 3);
    }
    uint2 o;
    o.x = pack_bf16x2(acc.x, acc.y);
    o.y = pack_bf16x2(acc.z, acc.w);
    *reinterpret_cast<uint2*>(out + (long long)r * ldo + c) = o;
  }
}

// Sum over the splits of four neighbouring columns. The first BATCH partials are loaded before any is used: with one item a
// thread, the latency of one round trip to L2 is what these kernels cost.
template <int BATCH>
struct SplitSum {
  float4 t[BATCH];
  __device__ __forceinline__ void load(const float* p, long long stride, int splits) {
#pragma unroll
    for (int s = 0; s < BATCH; ++s)
      if (s < splits) t[s] = *reinterpret_cast<const float4*>(p + s * stride);
  }
  __device__ __forceinline__ float4 sum(const float* p, long long stride, int splits) const {
    float4 a = t[0];
#pragma unroll
    for (int s = 1; s < BATCH; ++s)
      if (s < splits) { a.x += t[s].x; a.y += t[s].y; a.z += t[s].z; a.w += t[s].w; }
    for (int s = BATCH; s < splits; ++s) {
      const float4 v = *reinterpret_cast<const float4*>(p + s * stride);
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
    return a;
  }
};

// One CTA per row: res_out = sum_s ws[s, r, :] (+ res_in);  y = res_out * rsqrt(mean(res_out^2) + eps) * w.
// Four columns a thread, VPT times (H <= MAX_THREADS * VPT * 4); the row stays in registers between the two passes.
constexpr int RN_MAX_THREADS = 1024;
template <int VPT, int MAX_THREADS, int MIN_CTAS>
__global__ void __launch_bounds__(MAX_THREADS, MIN_CTAS)
splitk_reduce_residual_rmsnorm_kernel(const float* __restrict__ ws, int splits, int M, int H,
                                      const __nv_bfloat16* __restrict__ res_in, const __nv_bfloat16* __restrict__ w,
                                      float eps, __nv_bfloat16* __restrict__ res_out, __nv_bfloat16* __restrict__ y) {
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.x;
  const int n4 = H / 4;
  const long long split_stride = (long long)M * H;
  float4 v[VPT];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int c4 = threadIdx.x + j * blockDim.x;
    v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c4 < n4) {
      const float* p = ws + (long long)r * H + c4 * 4;
      SplitSum<VPT <= 2 ? 8 : 2> sum;
      sum.load(p, split_stride, splits);
      uint2 rr = make_uint2(0u, 0u);
      if (res_in) rr = *reinterpret_cast<const uint2*>(res_in + (long long)r * H + c4 * 4);
      float4 acc = sum.sum(p, split_stride, splits);
      if (res_in) {
        const float2 ra = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&rr.x));
        const float2 rb = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&rr.y));
        acc.x += ra.x; acc.y += ra.y; acc.z += rb.x; acc.w += rb.y;
      }
      // the residual stream is stored in bf16; normalise what is stored
      uint2 o;
      o.x = pack_bf16x2(acc.x, acc.y);
      o.y = pack_bf16x2(acc.z, acc.w);
      *reinterpret_cast<uint2*>(res_out + (long long)r * H + c4 * 4) = o;
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o.y));
      v[j] = make_float4(a.x, a.y, b.x, b.y);
      ss += a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y;
    }
  }
  __shared__ float red[RN_MAX_THREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  float tot = (threadIdx.x & 31) < (blockDim.x >> 5) ? red[threadIdx.x & 31] : 0.f;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  const float rstd = rsqrtf(tot / (float)H + eps);
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int c4 = threadIdx.x + j * blockDim.x;
    if (c4 < n4) {
      const uint2 ww = *reinterpret_cast<const uint2*>(w + c4 * 4);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ww.x));
      const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ww.y));
      uint2 o;
      o.x = pack_bf16x2(v[j].x * rstd * a.x, v[j].y * rstd * a.y);
      o.y = pack_bf16x2(v[j].z * rstd * b.x, v[j].w * rstd * b.y);
      *reinterpret_cast<uint2*>(y + (long long)r * H + c4 * 4) = o;
    }
  }
}

// The fused qkv projection ([hq + 2 hkv] heads of d): sums the split-K partials, adds the bias, rotates q and k
// (rotate-half RoPE at positions[r]), writes q [B, hq * d] and puts the K row and the V row of every kv head into the
// paged cache [pages, 2, hkv, page, d] at slot_mapping[r] (V slab transposed to [d, page] when v_transposed). A negative
// slot skips the cache write (padded batch rows). grid (row, part of the row); one thread = (head, four rotation pairs).
constexpr int QR_THREADS = 128;
__global__ void __launch_bounds__(QR_THREADS)
splitk_reduce_qkv_rope_append_kernel(const float* __restrict__ ws, int splits, int M, int hq, int hkv, int d,
                                     const void* bias, int bias_bf16, const long long* __restrict__ positions,
                                     const int* __restrict__ slot_mapping, float log2_theta,
                                     __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ cache,
                                     int page_size, int v_transposed) {
  pdl_launch_dependents();
  pdl_wait();
  const int r = blockIdx.x;
  const int half = d >> 1;
  const int q4 = half >> 2;  // groups of four rotation pairs per head
  const int N = (hq + 2 * hkv) * d;
  const int idx = blockIdx.y * QR_THREADS + threadIdx.x;
  if (idx >= (hq + 2 * hkv) * q4) return;
  const int h = idx / q4, i0 = (idx % q4) * 4;
  const int c0 = h * d + i0, c1 = c0 + half;
  const long long split_stride = (long long)M * N;
  const float* p0 = ws + (long long)r * N + c0;
  const float* p1 = p0 + half;
  SplitSum<8> s0, s1;
  s0.load(p0, split_stride, splits);
  s1.load(p1, split_stride, splits);
  const int slot = slot_mapping[r];
  float sn[4], cs[4];
  if (h < hq + hkv) {   // while the partial sums are on their way
    const float pos = (float)positions[r];
#pragma unroll
    for (int j = 0; j < 4; ++j) sincosf(pos * exp2f(-(2.0f * (float)(i0 + j) / (float)d) * log2_theta), &sn[j], &cs[j]);
  }
  const float4 a4 = s0.sum(p0, split_stride, splits), b4 = s1.sum(p1, split_stride, splits);
  float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
  if (bias) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      a[j] += bias_at(bias, bias_bf16, c0 + j);
      b[j] += bias_at(bias, bias_bf16, c1 + j);
    }
  }
  if (h < hq + hkv) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      // the unfused path rounds the projection to bf16 before rotating; do the same
      const float x = __bfloat162float(__float2bfloat16(a[j])), y = __bfloat162float(__float2bfloat16(b[j]));
      a[j] = x * cs[j] - y * sn[j];
      b[j] = y * cs[j] + x * sn[j];
    }
  }
  uint2 oa, ob;
  oa.x = pack_bf16x2(a[0], a[1]); oa.y = pack_bf16x2(a[2], a[3]);
  ob.x = pack_bf16x2(b[0], b[1]); ob.y = pack_bf16x2(b[2], b[3]);
  if (h < hq) {
    *reinterpret_cast<uint2*>(q_out + (long long)r * hq * d + c0) = oa;
    *reinterpret_cast<uint2*>(q_out + (long long)r * hq * d + c1) = ob;
  } else if (slot >= 0) {
    const int page = slot / page_size, off = slot % page_size;
    const long long slab = (long long)page_size * d;
    if (h < hq + hkv) {
      __nv_bfloat16* kd = cache + ((long long)(page * 2 + 0) * hkv + (h - hq)) * slab + (long long)off * d;
      *reinterpret_cast<uint2*>(kd + i0) = oa;
      *reinterpret_cast<uint2*>(kd + i0 + half) = ob;
    } else {
      __nv_bfloat16* vd = cache + ((long long)(page * 2 + 1) * hkv + (h - hq - hkv)) * slab;
      if (v_transposed) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          vd[(long long)(i0 + j) * page_size + off] = __float2bfloat16(a[j]);
          vd[(long long)(i0 + j + half) * page_size + off] = __float2bfloat16(b[j]);
        }
      } else {
        *reinterpret_cast<uint2*>(vd + (long long)off * d + i0) = oa;
        *reinterpret_cast<uint2*>(vd + (long long)off * d + i0 + half) = ob;
      }
    }
  }
}

}  // namespace b200

// Column tile width for a shape: 256 when that still leaves every SM at least two tiles (the second tile's main
// loop hides the first one's epilogue), else 128 (with contraction splits where the tiles are too few). Measured on
// the Qwen2.5-7B decode shapes at 128 rows: lm_head (594 wide tiles) 197 us against 210 us with narrow tiles;
// gate/up (148 wide tiles = one per SM) 57 us against 55 us.
static int skinny_bn(int M, int N, int swiglu, int num_sms) {
  const int num_m = (M + b200::GEMM_BM - 1) / b200::GEMM_BM;
  const int out_bn = swiglu ? 128 : 256;
  const int tiles256 = num_m * ((N + out_bn - 1) / out_bn);
  return tiles256 >= 2 * num_sms ? 256 : 128;
}

// SwiGLU: columns per tile when every SM gets one tile of that width, or 0 when fixed 64-column tiles are as good. Tiles
// of 64 columns cost whole rounds: 14336 columns are 224 tiles, two rounds of 148 SMs for 1.5 rounds of work, while
// 104-column tiles are one round of 138 (16 to 128 rows x 4096: 46 to 49 us, in 64-column tiles 52 to 55; 12288 columns: 40 to
// 42 and 51 to 53). A width that saves less than a twentieth loses to the store boxes of the fixed tiles: 18944 columns, where
// it would be 128 in one round instead of 64 in two, 16 rows x 3584: 50.8 us, fixed 47.5.
static int swiglu_width(int M, int N, int num_sms) {
  const int num_m = (M + b200::GEMM_BM - 1) / b200::GEMM_BM;
  if (num_m > num_sms) return 0;
  const int per_sm = num_sms / num_m;                       // column tiles that fit in one round
  const int w = ((N + per_sm - 1) / per_sm + 7) / 8 * 8;
  const int rounds64 = (num_m * ((N + 63) / 64) + num_sms - 1) / num_sms;
  return w <= 128 && w < 64 * rounds64 * 0.95f ? w : 0;
}

template <class Kern>
static int launch_skinny_kernel(Kern kern, bool& attr_set, int smem, int units, int num_sms) {
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -1;
    attr_set = true;
  }
  return units < num_sms ? units : num_sms;   // grid
}

template <int BN, bool SWIGLU, int A_ROWS, bool TAIL>
static int launch_skinny(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmO, int M, int N, int K,
                         const b200::SkinnyParams& ep, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  using SM = GemmSmem<BN, SkinnyCfg<BN, A_ROWS>::STAGES, A_ROWS>;
  auto kern = gemm_skinny_kernel<BN, SWIGLU, A_ROWS, TAIL>;
  static bool attr_set = false;
  constexpr int OUT_BN = SWIGLU ? BN / 2 : BN;
  const int units = ((M + GEMM_BM - 1) / GEMM_BM) * ((N + OUT_BN - 1) / OUT_BN) * ep.splits;
  const int grid = launch_skinny_kernel(kern, attr_set, SM::TOTAL_WITH_EPI, units, num_sms);
  if (grid < 0) return B200_ERR_LAUNCH;
  return launch_pdl(kern, dim3(grid), dim3(GEMM_THREADS), SM::TOTAL_WITH_EPI, stream, tmA, tmB, tmO, M, N, K, ep,
                    status) == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

template <int A_ROWS>
static int launch_swiglu_rows(const CUtensorMap& tmA, const CUtensorMap& tmB, int M, int N, int K,
                              const b200::SkinnyParams& ep, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  using SM = GemmSmem<256, SkinnyCfg<256, A_ROWS>::ROW_STORE_STAGES, A_ROWS>;
  auto kern = gemm_skinny_swiglu_rows_kernel<A_ROWS>;
  static bool attr_set = false;
  const int width = ep.b_rows / 2, units = ((M + GEMM_BM - 1) / GEMM_BM) * ((N + width - 1) / width);
  const int grid = launch_skinny_kernel(kern, attr_set, SM::TOTAL, units, num_sms);
  if (grid < 0) return B200_ERR_LAUNCH;
  return launch_pdl(kern, dim3(grid), dim3(GEMM_THREADS), SM::TOTAL, stream, tmA, tmB, M, N, K, ep, status) == cudaSuccess
             ? 0 : B200_ERR_LAUNCH;
}

// rows of the A tile that are kept in shared memory
static int skinny_a_rows(int M) { return M <= 16 ? 16 : M <= 64 ? 64 : b200::GEMM_BM; }

extern "C" {

// How many contraction splits fill the machine for this shape (1 = the GEMM can write its result directly).
int b200_gemm_skinny_splits(int M, int N, int K, int swiglu, int num_sms) {
  using namespace b200;
  if (swiglu) return 1;
  const int bn = skinny_bn(M, N, 0, num_sms);
  const int tiles = ((M + GEMM_BM - 1) / GEMM_BM) * ((N + bn - 1) / bn);
  const int num_kb = (K + GEMM_BK - 1) / GEMM_BK;
  int s = num_sms / (tiles > 0 ? tiles : 1);
  if (s > num_kb / 4) s = num_kb / 4;  // at least four contraction blocks per unit
  if (s > 16) s = 16;
  if (s < 1) s = 1;
  return s;
}

// x [M, K] (M <= 256), W [N_w, K]; swiglu: W is a fused gate/up weight, N = intermediate size, up rows start at up_row0.
// ws == NULL: out (bf16 [M, ldo]) is written (+ bias), splits must be 1. Otherwise ws (fp32 [splits, M, N]) receives
// the partial results and one of the b200_splitk_reduce* kernels must follow.
int b200_gemm_skinny(const void* x, const void* W, void* out, float* ws, int M, int N, int K, long long ldx,
                     long long ldw, long long ldo, const void* bias, int bias_bf16, int swiglu, int up_row0,
                     int splits, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0 || splits < 1 || (ldx & 7) || (ldw & 7)) return B200_ERR_ARG;
  if (splits > 1 && (!ws || swiglu)) return B200_ERR_ARG;
  if (!ws && !out) return B200_ERR_ARG;
  const int n_rows_w = swiglu ? up_row0 + N : N;
  const int width = swiglu ? swiglu_width(M, N, num_sms) : 0;
  const int bn = width ? 256 : skinny_bn(M, N, swiglu, num_sms);
  const int b_rows = width ? 2 * width : bn, a_rows = skinny_a_rows(M);
  // Exactly the rows there are: a row of a box that lies outside the tensor takes longer than one that is fetched.
  const int box_rows = M < a_rows ? M : a_rows;
  CUtensorMap tmA, tmB, tmO;
  if (make_tmap_2d(&tmA, x, M, K, ldx, box_rows, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tmB, W, n_rows_w, K, ldw, swiglu ? b_rows / 2 : b_rows, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  if (ws ? make_tmap_ws(&tmO, ws, splits, M, N) : make_tmap_out16(&tmO, out, M, N < 8 ? 8 : whole16(N, 0), ldo)) return B200_ERR_TENSORMAP;
  // Blocks of weights that a CTA brings into L2 ahead of its predecessor's end: a decode block of five sequences (8B) takes
  // 135.5 us without, 131.7 with half or all of this, 134.4 with twice as much; at 128 sequences (7B) 180.2, 179.7, 180.3 and
  // 182.3: more than the pipeline's own depth competes with the kernel that still runs.
  SkinnyParams ep{nullptr, ws ? nullptr : bias, bias_bf16, ws ? 1 : 0, M, N, splits, (__nv_bfloat16*)out, ldo, up_row0,
                  b_rows, box_rows * GEMM_BK * 2, pdl_enabled() ? (bn == 256 ? 8 : 16) : 0};
  auto launch = [&](auto rows, auto tail) -> int {
    constexpr int R = decltype(rows)::value;
    constexpr bool T = decltype(tail)::value;
    if (width) return launch_swiglu_rows<R>(tmA, tmB, M, N, K, ep, status, num_sms, stream);
    if (bn == 256)
      return swiglu ? launch_skinny<256, true, R, T>(tmA, tmB, tmO, M, N, K, ep, status, num_sms, stream)
                    : launch_skinny<256, false, R, T>(tmA, tmB, tmO, M, N, K, ep, status, num_sms, stream);
    return swiglu ? launch_skinny<128, true, R, T>(tmA, tmB, tmO, M, N, K, ep, status, num_sms, stream)
                  : launch_skinny<128, false, R, T>(tmA, tmB, tmO, M, N, K, ep, status, num_sms, stream);
  };
  auto launch_rows = [&](auto tail) -> int {
    if (a_rows == 16) return launch(std::integral_constant<int, 16>{}, tail);
    if (a_rows == 64) return launch(std::integral_constant<int, 64>{}, tail);
    return launch(std::integral_constant<int, GEMM_BM>{}, tail);
  };
  return !ws && whole16(N, 0) != N ? launch_rows(std::true_type{}) : launch_rows(std::false_type{});
}

int b200_splitk_reduce(const float* ws, int splits, int M, int N, const void* bias, int bias_bf16, void* out,
                       long long ldo, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || (N & 3) || (ldo & 3) || splits < 1) return B200_ERR_ARG;
  const long long n4 = (long long)M * (N / 4);
  const int grid = (int)((n4 + 255) / 256 < 2048 ? (n4 + 255) / 256 : 2048);
  return b200::launch_pdl(b200::splitk_reduce_kernel, dim3(grid), dim3(256), 0, stream, ws, splits, M, N, bias, bias_bf16,
                          (__nv_bfloat16*)out, ldo) == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

// y [M, N] bf16 = x W^T (+ bias) in one call: the split is chosen here and reduced when there is one. ws: fp32 scratch of
// ws_floats elements (splits * M * N are used); null with ws_floats 0 until a shape is split, which then returns
// B200_NEED_WORKSPACE without having launched anything.
int b200_skinny_linear(const void* x, const void* W, const void* bias, int bias_bf16, void* out, float* ws,
                       long long ws_floats, int M, int N, int K, long long ldx, long long ldw, long long ldo,
                       uint32_t* status, int num_sms, cudaStream_t stream) {
  const int splits = b200_gemm_skinny_splits(M, N, K, 0, num_sms);
  // Short contractions stay whole: the second kernel costs more than shares save up to 16 blocks of rows on the 128-byte grid. us,
  // split and whole: 57 rows, 1024 x 512 5.9 and 4.6, 512 x 1024 6.2 and 5.7, 8192 x 1024 8.9 and 6.9; one row 6.0 and 5.7 (1024 x
  // 1024); of 32 blocks 57 x 2048 x 2048 8.6 and 8.8, one row 7.7 and 8.7. Rows off that grid take half as long again to fetch, and
  // there the line is at 11 blocks: 118 rows, 1024 x 648 7.8 and 7.6, x 712 7.3 and 7.9, x 1000 7.7 and 9.5. What only the reduction
  // can write (results off the 16-byte grid) is split.
  const int most = (K | ldx | ldw) & 63 ? 11 : 16;
  const bool whole = K <= most * b200::GEMM_BK && !(N & 7) && !(ldo & 7) && !(reinterpret_cast<uintptr_t>(out) & 15);
  if (splits == 1 || whole)
    return b200_gemm_skinny(x, W, out, nullptr, M, N, K, ldx, ldw, ldo, bias, bias_bf16, 0, 0, 1, status, num_sms, stream);
  if (ws == nullptr) return B200_NEED_WORKSPACE;
  if ((long long)splits * M * N > ws_floats) return B200_ERR_TOO_LARGE;
  const int rc = b200_gemm_skinny(x, W, nullptr, ws, M, N, K, ldx, ldw, 0, nullptr, 0, 0, 0, splits, status, num_sms, stream);
  return rc ? rc : b200_splitk_reduce(ws, splits, M, N, bias, bias_bf16, out, ldo, stream);
}

int b200_splitk_reduce_residual_rmsnorm(const float* ws, int splits, int M, int H, const void* res_in, const void* w,
                                        float eps, void* res_out, void* y, cudaStream_t stream) {
  using namespace b200;
  if (M <= 0 || H <= 0 || (H & 3) || H > RN_MAX_THREADS * 2 * 4 || splits < 1) return B200_ERR_ARG;
  // A CTA of so many threads has an SM to itself. With more rows than SMs that is two rounds, so long rows (of which there are
  // at most two splits then) take a quarter of the threads there and two rows share an SM: projection and reduction of 256 x
  // 8192 (K 4096) 29.3 us, with half the threads 33.3; 256 x 6144 27.7 and 30.0.
  const int n4 = H / 4, vpt = n4 <= RN_MAX_THREADS ? 1 : M > 148 ? 4 : 2;
  const int threads = ((n4 + vpt - 1) / vpt + 31) / 32 * 32;
  auto kern = vpt == 1   ? splitk_reduce_residual_rmsnorm_kernel<1, RN_MAX_THREADS, 1>
              : vpt == 2 ? splitk_reduce_residual_rmsnorm_kernel<2, RN_MAX_THREADS, 1>
                         : splitk_reduce_residual_rmsnorm_kernel<4, RN_MAX_THREADS / 2, 2>;
  return launch_pdl(kern, dim3(M), dim3(threads), 0, stream, ws, splits, M, H, (const __nv_bfloat16*)res_in,
                    (const __nv_bfloat16*)w, eps, (__nv_bfloat16*)res_out, (__nv_bfloat16*)y) == cudaSuccess
             ? 0 : B200_ERR_LAUNCH;
}

int b200_splitk_reduce_qkv_rope_append(const float* ws, int splits, int M, int hq, int hkv, int d, const void* bias,
                                       int bias_bf16, const long long* positions, const int* slot_mapping,
                                       float theta, void* q_out, void* cache, int page_size, int v_transposed,
                                       cudaStream_t stream) {
  if (M <= 0 || hq <= 0 || hkv <= 0 || d <= 0 || (d & 7) || splits < 1) return B200_ERR_ARG;
  const int items = (hq + 2 * hkv) * (d / 8);
  return b200::launch_pdl(b200::splitk_reduce_qkv_rope_append_kernel,
                          dim3(M, (items + b200::QR_THREADS - 1) / b200::QR_THREADS), dim3(b200::QR_THREADS), 0, stream, ws, splits, M, hq,
                          hkv, d, bias, bias_bf16, positions, slot_mapping, log2f(theta), (__nv_bfloat16*)q_out,
                          (__nv_bfloat16*)cache, page_size, v_transposed) == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

}  // extern "C"
