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
#include "sm100.cuh"

namespace {

constexpr int MOE_ALIGN = 128;

// ---- router: one warp per token, E <= 256, k <= 8 ---------------------------------------------------
// Lane j keeps the j-th choice and every lane's logits stay in registers. A block counts its choices in shared memory and adds the
// sums: one by one they queue at the address of a popular expert. 4096 tokens, 8 of 128 experts: 9.8 us, with choices in
// arrays and counted one by one 16.0; 8192 tokens, 8 of 16 experts: 17.4 and 50.
constexpr int ROUTE_THREADS = 512;
__global__ void __launch_bounds__(ROUTE_THREADS)
route_topk_kernel(const float* __restrict__ logits, int T, int E, int k, int renorm, float* __restrict__ probs,
                  int* __restrict__ idx, int* __restrict__ counts) {
  __shared__ int hist[256];
  for (int e = threadIdx.x; e < E; e += ROUTE_THREADS) hist[e] = 0;
  __syncthreads();
  const int token = blockIdx.x * (ROUTE_THREADS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (token < T) {
    const float* row = logits + (long long)token * E;
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
    // A logit that is not a number leaves that in the token's weights; to the choice it is the least of values, so that every token
    // has k experts of its own that exist, whatever its logits are: the kernels that follow address memory with them.
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (lane + 32 * i) < E ? fmaxf(v[i], 0.f) : -1.f;
    const float inv = 1.f / s;
    float prob = 0.f, tsum = 0.f;
    int choice = 0;
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
      if (lane == j) {
        prob = bv * inv;
        choice = bi;
      }
      tsum += bv * inv;
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (lane + 32 * i == bi) v[i] = -1.f;  // remove the winner
    }
    if (lane < k) {
      probs[(long long)token * k + lane] = prob * (renorm ? 1.f / tsum : 1.f);
      idx[(long long)token * k + lane] = choice;
      atomicAdd(&hist[choice], 1);
    }
  }
  if (counts) {
    __syncthreads();
    for (int e = threadIdx.x; e < E; e += ROUTE_THREADS)
      if (hist[e]) atomicAdd(&counts[e], hist[e]);
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

// the rows between an expert's last filled row and the next expert's first: the GEMMs contract over them. row_info (nullable) says
// that they belong to no (token, choice).
__global__ void __launch_bounds__(ROW_MAX_THREADS)
zero_padding_kernel(const int* __restrict__ filled, const int* __restrict__ offsets, __nv_bfloat16* __restrict__ xp,
                    int2* __restrict__ row_info, int max_rows, int H) {
  const int e = blockIdx.x, end = min(offsets[e + 1], max_rows);   // counts that are only an upper bound may add up to more
  for (int r = offsets[e] + filled[e] + blockIdx.y; r < end; r += gridDim.y) {
    for (int i = threadIdx.x; i < H / 8; i += blockDim.x)
      reinterpret_cast<uint4*>(xp + (long long)r * H)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (row_info && threadIdx.x == 0) row_info[r] = make_int2(-1, 0);
  }
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

// Backward of combine, without the weights (expert_swiglu_bwd_kernel brings them in): the k rows of a token get its gradient, and
// row_info says which (token, choice) a row belongs to and what its weight is.
__global__ void __launch_bounds__(ROW_MAX_THREADS)
spread_kernel(const __nv_bfloat16* __restrict__ src, const float* __restrict__ probs, const int* __restrict__ row_map,
              __nv_bfloat16* __restrict__ dst, int2* __restrict__ row_info, int k, int H) {
  const long long t = blockIdx.x;
  for (int j = threadIdx.x; j < k; j += blockDim.x)
    row_info[row_map[t * k + j]] = make_int2((int)(t * k + j), __float_as_int(probs[t * k + j]));
  for (int i = threadIdx.x; i < H / 8; i += blockDim.x) {
    const uint4 v = reinterpret_cast<const uint4*>(src + t * H)[i];
#pragma unroll 4
    for (int j = 0; j < k; ++j) reinterpret_cast<uint4*>(dst + (long long)row_map[t * k + j] * H)[i] = v;
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

// Backward of the experts' middle. With a = silu(g) o u, the row's output is p (a Wd^T) and dact = dout Wd lacks the weight p:
//   dprob = <a, dact>,  dh1 = p dact d(a)/d(g, u),  ap = p a (what the gradient of Wd contracts with the unweighted dout).
// So the weights' gradient needs neither the experts' output nor a pass over it, a is not formed in a pass of its own, and the
// gradient is spread as it is. Bound by HBM (12 bytes an element of a; 4096 tokens on 128 experts of 768, 8 each: 59 us, 0.88 of
// copy speed; the passes it stands for, a, the gradient of a and dprob, took 126). One warp a row, since dprob is the row's sum;
// 40 warps an SM hide the way from a row's number to its data better than three vectors a lane on their way with 16 or 24 warps
// (73 and 64 us), and several warps a row add a barrier (80).
__global__ void __launch_bounds__(256, 5)
expert_swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dact, const __nv_bfloat16* __restrict__ h1,
                         const int2* __restrict__ row_info, const int* __restrict__ n_tiles, __nv_bfloat16* __restrict__ dh1,
                         __nv_bfloat16* __restrict__ ap, float* __restrict__ dprob, int I) {
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);   // there is room for whole blocks of rows
  const int2 info = row_info[row];
  if (row >= (long long)n_tiles[0] * MOE_ALIGN) return;
  const int lane = threadIdx.x & 31, nvec = I >> 3;
  uint4* out = reinterpret_cast<uint4*>(dh1 + row * 2 * I);
  uint4* out_a = reinterpret_cast<uint4*>(ap + row * I);
  if (info.x < 0) {   // padding
    for (int v = lane; v < nvec; v += 32) out[v] = out[nvec + v] = out_a[v] = make_uint4(0u, 0u, 0u, 0u);
    return;
  }
  const uint4* in = reinterpret_cast<const uint4*>(h1 + row * 2 * I);
  const uint4* in_d = reinterpret_cast<const uint4*>(dact + row * I);
  const float p = __int_as_float(info.y);
  float dot = 0.f;
  for (int v = lane; v < nvec; v += 32) {
    const uint4 gv = in[v], uv = in[nvec + v], dv = in_d[v];
    float a[8], b[8], c[8], s[8];
    unpack8(gv, a);
    unpack8(uv, b);
    unpack8(dv, c);
    b200::sigmoids(a, s);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float silu = a[j] * s[j], act = silu * b[j], pd = p * c[j];
      dot += act * c[j];
      a[j] = pd * b[j] * (s[j] + silu * (1.f - s[j]));
      b[j] = pd * silu;
      c[j] = p * act;
    }
    out[v] = pack8(a);
    out[nvec + v] = pack8(b);
    out_a[v] = pack8(c);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
  if (lane == 0) dprob[info.x] = dot;
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
  const int per = ROUTE_THREADS / 32;
  route_topk_kernel<<<(T + per - 1) / per, ROUTE_THREADS, 0, stream>>>(logits, T, E, k, renorm, probs, idx, counts);
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

int b200_moe_zero_padding(const int* filled, const int* offsets, void* xp, void* row_info, int E, int max_rows, int H,
                          cudaStream_t stream) {
  if (E <= 0) return 0;
  if (H & 7) return B200_ERR_ARG;
  zero_padding_kernel<<<dim3(E, E < 64 ? 32 : 16), row_threads(H), 0, stream>>>(filled, offsets, (__nv_bfloat16*)xp,
                                                                                (int2*)row_info, max_rows, H);
  return ok();
}

int b200_moe_spread(const void* src, const float* probs, const int* row_map, void* dst, void* row_info, int T, int k, int H,
                    cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return B200_ERR_ARG;
  spread_kernel<<<T, row_threads(H), 0, stream>>>((const __nv_bfloat16*)src, probs, row_map, (__nv_bfloat16*)dst,
                                                  (int2*)row_info, k, H);
  return ok();
}

int b200_moe_combine(const void* y, const float* probs, const int* row_map, void* out, int T, int k, int H,
                     cudaStream_t stream) {
  if (T <= 0) return 0;
  if (H & 7) return B200_ERR_ARG;
  combine_kernel<<<T, row_threads(H), 0, stream>>>((const __nv_bfloat16*)y, probs, row_map, (__nv_bfloat16*)out, k, H);
  return ok();
}

int b200_moe_swiglu_bwd(const void* dact, const void* h1, const void* row_info, const int* n_tiles, void* dh1, void* ap,
                        float* dprob, int max_rows, int I, cudaStream_t stream) {
  if (max_rows <= 0) return 0;
  if ((I & 7) || (max_rows & 7)) return B200_ERR_ARG;
  expert_swiglu_bwd_kernel<<<max_rows / 8, 256, 0, stream>>>((const __nv_bfloat16*)dact, (const __nv_bfloat16*)h1,
                                                                   (const int2*)row_info, n_tiles, (__nv_bfloat16*)dh1,
                                                                   (__nv_bfloat16*)ap, dprob, I);
  return ok();
}

}  // extern "C"
