// Mixture-of-experts routing and token movement kernels for sm_100a: fused softmax + top-k router,
// expert histogram / padded offsets, permute (gather rows by expert) and weighted un-permute (combine), with
// their backward forms. They replace the eager router (cosmos_rl/policy/kernel/moe/moe.py:563-635), the Triton
// permute / un-permute kernels (cosmos_rl/policy/kernel/megatron_moe/permutation.py:35-676) and the index
// converters of the reference. Every expert's block in the permuted buffer starts on a multiple of 128 rows so
// the grouped GEMMs (grouped_gemm.cu) never see a tile that straddles two experts; nothing here needs a host
// synchronisation: counts, offsets and the tile -> expert table stay on the device.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "api.h"

namespace {

constexpr int MOE_ALIGN = 128;

// ---- router: one warp per token, E <= 256, k <= 8 ---------------------------------------------------
__global__ void route_topk_kernel(const float* __restrict__ logits, int T, int E, int k, int renorm,
                                  float* __restrict__ probs, int* __restrict__ idx, int* __restrict__ counts) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= T) return;
  const float* row = logits + (long long)warp * E;
  float v[8];
  float mx = -INFINITY;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    int e = lane + 32 * i;
    v[i] = e < E ? row[e] : -INFINITY;
    mx = fmaxf(mx, v[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] = (lane + 32 * i) < E ? __expf(v[i] - mx) : 0.f;
    s += v[i];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float inv = 1.f / s;
  float topv[8];
  int topi[8];
  float tsum = 0.f;
  for (int j = 0; j < k; ++j) {
    float bv = -1.f;
    int bi = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (v[i] > bv) { bv = v[i]; bi = lane + 32 * i; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    topv[j] = bv * inv;
    topi[j] = bi;
    tsum += topv[j];
    if ((bi & 31) == lane) v[bi >> 5] = -1.f;  // remove the winner
  }
  if (lane == 0) {
    const float r = renorm ? 1.f / tsum : 1.f;
    for (int j = 0; j < k; ++j) {
      probs[(long long)warp * k + j] = topv[j] * r;
      idx[(long long)warp * k + j] = topi[j];
      if (counts) atomicAdd(&counts[topi[j]], 1);
    }
  }
}

// ---- offsets: one block; padded exclusive scan + tile -> expert table --------------------------------
constexpr int OFF_THREADS = 256;
__global__ void __launch_bounds__(OFF_THREADS)
offsets_kernel(const int* __restrict__ counts, int E, int* __restrict__ offsets, int* __restrict__ tile_expert,
               int* __restrict__ n_tiles, int* __restrict__ cursor, int max_tiles) {
  __shared__ int warp_tot[OFF_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;   // tiles of the experts before this round of the loop
  for (int e0 = 0; e0 < E; e0 += OFF_THREADS) {
    const int e = e0 + threadIdx.x;
    const int tiles = e < E ? (counts[e] + MOE_ALIGN - 1) / MOE_ALIGN : 0;
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    int before = base;
    for (int w = 0; w < warp; ++w) before += warp_tot[w];
    for (int w = 0; w < OFF_THREADS / 32; ++w) base += warp_tot[w];
    __syncthreads();
    if (e < E) {
      const int first = before + incl - tiles;
      offsets[e] = first * MOE_ALIGN;
      cursor[e] = 0;
      for (int t = first; t < first + tiles && t < max_tiles; ++t) tile_expert[t] = e;
    }
  }
  if (threadIdx.x == 0) {
    offsets[E] = base * MOE_ALIGN;
    n_tiles[0] = min(base, max_tiles);
  }
}

// ---- rows of the expert-sorted buffer. One block per token; a thread moves 16 bytes of the token's row at a time and
// touches all k choices with it, so the token's own row is read once and the k rows are in flight together. ---------
constexpr int ROW_MAX_THREADS = 256;

// permute: claim a slot per (token, choice), copy the row
__global__ void __launch_bounds__(ROW_MAX_THREADS)
permute_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ idx, const int* __restrict__ offsets,
               int* __restrict__ cursor, int* __restrict__ row_map, __nv_bfloat16* __restrict__ xp, int k, int H) {
  extern __shared__ int pos_sh[];
  const long long t = blockIdx.x;
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    const int e = idx[t * k + j];
    pos_sh[j] = row_map[t * k + j] = offsets[e] + atomicAdd(&cursor[e], 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
    const uint4 v = reinterpret_cast<const uint4*>(x + t * H)[i];
#pragma unroll 4
    for (int j = 0; j < k; ++j) reinterpret_cast<uint4*>(xp + (long long)pos_sh[j] * H)[i] = v;
  }
}

// the rows between an expert's last filled row and the next expert's first: the GEMMs contract over them
__global__ void __launch_bounds__(ROW_MAX_THREADS)
zero_padding_kernel(const int* __restrict__ filled, const int* __restrict__ offsets, __nv_bfloat16* __restrict__ xp,
                    int max_rows, int H) {
  const int e = blockIdx.x, end = min(offsets[e + 1], max_rows);   // counts that are only an upper bound may add up to more
  for (int r = offsets[e] + filled[e] + blockIdx.y; r < end; r += gridDim.y)
    for (int i = threadIdx.x; i < H / 8; i += blockDim.x)
      reinterpret_cast<uint4*>(xp + (long long)r * H)[i] = make_uint4(0u, 0u, 0u, 0u);
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(p[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// spread rows through an existing row_map (backward of combine: dy[pos] = prob * dout[t])
__global__ void __launch_bounds__(ROW_MAX_THREADS)
scatter_scaled_kernel(const __nv_bfloat16* __restrict__ src, const float* __restrict__ probs,
                      const int* __restrict__ row_map, __nv_bfloat16* __restrict__ dst, int k, int H) {
  const long long t = blockIdx.x;
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
    float f[8];
    unpack8(reinterpret_cast<const uint4*>(src + t * H)[i], f);
#pragma unroll 4
    for (int j = 0; j < k; ++j) {
      const float p = probs ? probs[t * k + j] : 1.f;
      float o[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) o[c] = f[c] * p;
      reinterpret_cast<uint4*>(dst + (long long)row_map[t * k + j] * H)[i] = pack8(o);
    }
  }
}

// ---- combine: out[t] = sum_j prob[t,j] * y[row_map[t,j]]  (probs null: plain sum) ------------------------
__global__ void __launch_bounds__(ROW_MAX_THREADS)
combine_kernel(const __nv_bfloat16* __restrict__ y, const float* __restrict__ probs, const int* __restrict__ row_map,
               __nv_bfloat16* __restrict__ out, int k, int H) {
  const long long t = blockIdx.x;
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int j = 0; j < k; ++j) {
      const float p = probs ? probs[t * k + j] : 1.f;
      float f[8];
      unpack8(reinterpret_cast<const uint4*>(y + (long long)row_map[t * k + j] * H)[i], f);
#pragma unroll
      for (int c = 0; c < 8; ++c) a[c] += p * f[c];
    }
    reinterpret_cast<uint4*>(out + t * H)[i] = pack8(a);
  }
}

// dprob[t,j] = <dout[t], y[row_map[t,j]]>, eight choices at a time
__global__ void __launch_bounds__(ROW_MAX_THREADS)
combine_dprob_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ y,
                     const int* __restrict__ row_map, float* __restrict__ dprob, int k, int H) {
  __shared__ float sh[ROW_MAX_THREADS / 32][8];
  const long long t = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j0 = 0; j0 < k; j0 += 8) {
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
      float f[8];
      unpack8(reinterpret_cast<const uint4*>(dout + t * H)[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j0 + j < k) {
          float g[8];
          unpack8(reinterpret_cast<const uint4*>(y + (long long)row_map[t * k + j0 + j] * H)[i], g);
#pragma unroll
          for (int c = 0; c < 8; ++c) s[j] += f[c] * g[c];
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
      if (lane == 0) sh[warp][j] = s[j];
    }
    __syncthreads();
    if (threadIdx.x < 8 && j0 + (int)threadIdx.x < k) {
      float r = 0.f;
      for (int w = 0; w < (int)blockDim.x / 32; ++w) r += sh[w][threadIdx.x];
      dprob[t * k + j0 + threadIdx.x] = r;
    }
    __syncthreads();
  }
}

// threads of a block that moves rows of H elements
inline int row_threads(int H) {
  const int t = (H / 8 + 31) / 32 * 32;
  return t < ROW_MAX_THREADS ? t : ROW_MAX_THREADS;
}

inline int ok() { return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH; }

}  // namespace

extern "C" {

int b200_moe_route_topk(const float* logits, int T, int E, int k, int renorm, float* probs, int* idx, int* counts,
                        cudaStream_t stream) {
  if (T <= 0) return 0;
  if (E > 256 || k > 8 || k > E) return B200_ERR_ARG;
  route_topk_kernel<<<(T * 32 + 255) / 256, 256, 0, stream>>>(logits, T, E, k, renorm, probs, idx, counts);
  return ok();
}

int b200_moe_offsets(const int* counts, int E, int* offsets, int* tile_expert, int* n_tiles, int* cursor,
                     int max_tiles, cudaStream_t stream) {
  offsets_kernel<<<1, OFF_THREADS, 0, stream>>>(counts, E, offsets, tile_expert, n_tiles, cursor, max_tiles);
  return ok();
}

int b200_moe_permute(const void* x, const int* idx, const int* offsets, int* cursor, int* row_map, void* xp, int T,
                     int k, int H, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((H & 7) || k <= 0 || k > 4096) return B200_ERR_ARG;
  permute_kernel<<<T, row_threads(H), k * sizeof(int), stream>>>((const __nv_bfloat16*)x, idx, offsets, cursor, row_map,
                                                                 (__nv_bfloat16*)xp, k, H);
  return ok();
}

int b200_moe_zero_padding(const int* filled, const int* offsets, void* xp, int E, int max_rows, int H, cudaStream_t stream) {
  if (E <= 0) return 0;
  if (H & 7) return B200_ERR_ARG;
  zero_padding_kernel<<<dim3(E, E < 64 ? 32 : 16), row_threads(H), 0, stream>>>(filled, offsets, (__nv_bfloat16*)xp, max_rows, H);
  return ok();
}

int b200_moe_scatter_scaled(const void* src, const float* probs, const int* row_map, void* dst, int T, int k, int H,
                            cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return B200_ERR_ARG;
  scatter_scaled_kernel<<<T, row_threads(H), 0, stream>>>((const __nv_bfloat16*)src, probs, row_map, (__nv_bfloat16*)dst,
                                                          k, H);
  return ok();
}

int b200_moe_combine(const void* y, const float* probs, const int* row_map, void* out, int T, int k, int H,
                     cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return B200_ERR_ARG;
  combine_kernel<<<T, row_threads(H), 0, stream>>>((const __nv_bfloat16*)y, probs, row_map, (__nv_bfloat16*)out, k, H);
  return ok();
}

int b200_moe_combine_dprob(const void* dout, const void* y, const int* row_map, float* dprob, int T, int k, int H,
                           cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return B200_ERR_ARG;
  combine_dprob_kernel<<<T, row_threads(H), 0, stream>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)y, row_map,
                                                         dprob, k, H);
  return ok();
}

}  // extern "C"
