// Bandwidth-bound ops of the policy model and optimizer for sm_100a: RMSNorm (+ fused residual add)
// forward/backward, rotary embedding, SwiGLU forward/backward, fused AdamW with bf16 shadow write,
// gradient sum-of-squares and clip coefficient. All math in fp32, 16-byte vector accesses.
// Reference semantics: cosmos_rl/policy/kernel/norm.py:36-41, rope.py:33-57, fused.py:31-37,
// cosmos_rl/policy/trainer/optm/__init__.py:365-400, cosmos_rl/utils/distributed.py:306-407.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "api.h"
#include "sm100.cuh"

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float r = (threadIdx.x < THREADS / 32) ? sh[threadIdx.x] : 0.f;
  if (w == 0) {
    r = warp_sum(r);
    if (l == 0) sh[0] = r;
  }
  __syncthreads();
  return sh[0];
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&f)[8]) {
  const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(p[i]);
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

// ------------------------------------------------------------------------------------------------
// RMSNorm. A row is spread over one CTA (VPT 16-byte vectors a thread); a CTA works on ROWS rows at a time so that the
// loads of all of them are in flight before the first sum is needed, and one barrier pair serves all their sums.
// ------------------------------------------------------------------------------------------------
constexpr int NORM_MAX_THREADS = 512;
constexpr int NORM_MAX_H = NORM_MAX_THREADS * 8 * 2;
constexpr int RMSNORM_WS_ROWS = 296;   // persistent blocks of the backward pass, two per SM

// sums of ROWS values over the block, the result in every thread; `sh` holds [ROWS][16] and is reused by the next call
// only after another barrier of the caller's loop (two buffers alternate)
template <int ROWS>
__device__ __forceinline__ void block_sums(float (&v)[ROWS], float (*sh)[16]) {
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    v[r] = warp_sum(v[r]);
    if (l == 0) sh[r][w] = v[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ROWS; ++r) v[r] = warp_sum(l < nw ? sh[r][l] : 0.f);
}

template <int VPT, int ROWS>
__global__ void __launch_bounds__(NORM_MAX_THREADS)
rmsnorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
                   const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ y,
                   __nv_bfloat16* __restrict__ res_out, float* __restrict__ rstd_out, int T, int H, float eps) {
  __shared__ float sh[ROWS][16];
  const int nvec = H >> 3;
  const long long row0 = (long long)blockIdx.x * ROWS;
  uint4 h[ROWS][VPT];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      h[r][i] = make_uint4(0u, 0u, 0u, 0u);
      if (v < nvec && row0 + r < T) h[r][i] = reinterpret_cast<const uint4*>(x + (row0 + r) * H)[v];
    }
  if (res) {
    uint4 q[ROWS][VPT];
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int v = threadIdx.x + i * blockDim.x;
        q[r][i] = make_uint4(0u, 0u, 0u, 0u);
        if (v < nvec && row0 + r < T) q[r][i] = reinterpret_cast<const uint4*>(res + (row0 + r) * H)[v];
      }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
      for (int i = 0; i < VPT; ++i) {
        const int v = threadIdx.x + i * blockDim.x;
        float f[8], g[8];
        unpack8(h[r][i], f);
        unpack8(q[r][i], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] += g[j];
        h[r][i] = pack8(f);   // the norm sees the bf16-rounded residual stream
        if (res_out && v < nvec && row0 + r < T) reinterpret_cast<uint4*>(res_out + (row0 + r) * H)[v] = h[r][i];
      }
  }
  float ss[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    ss[r] = 0.f;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      float f[8];
      unpack8(h[r][i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss[r] += f[j] * f[j];
    }
  }
  block_sums<ROWS>(ss, sh);
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    ss[r] = rsqrtf(ss[r] / (float)H + eps);
    if (threadIdx.x == 0 && rstd_out && row0 + r < T) rstd_out[row0 + r] = ss[r];
  }
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    if (v >= nvec) continue;
    float g[8];
    unpack8(reinterpret_cast<const uint4*>(w)[v], g);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      float f[8], o[8];
      unpack8(h[r][i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = f[j] * ss[r] * g[j];
      if (row0 + r < T) reinterpret_cast<uint4*>(y + (row0 + r) * H)[v] = pack8(o);
    }
  }
}

// RMSNorm backward of wide rows: dx (+ dres) and the weight gradient in one pass over dy and x. Persistent CTAs walk pairs of
// adjacent rows; a thread keeps the weight-gradient sums of its own columns in registers and writes them once, to its block's row
// of dw_partial (null: no weight gradient).
// Bound by HBM, if enough rows are on their way: a row is dy, x and dres, and rows come through a ring of NORM_STAGES in shared
// memory as bulk copies, three rows ahead of the one that is worked on. 8192 x 3584: 40.2 us, with the loads of two rows in
// registers, whose way the CTA waited for, 49.7 (36 are the bytes); 16384 x 5120 122 and 164; 64 x 3584 3.6 and 3.4.
constexpr int NORM_STAGES = 4;
template <int VPT, int MIN_CTAS>
__global__ void __launch_bounds__(NORM_MAX_THREADS, MIN_CTAS)
rmsnorm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                   const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx,
                   float* __restrict__ dw_partial, long long T, int H) {
  extern __shared__ __align__(16) uint8_t ring[];   // [NORM_STAGES][dy, x, dres][H]
  __shared__ float sh[2][1][16];
  __shared__ uint64_t full[NORM_STAGES];
  const int nvec = H >> 3;
  const uint32_t row_bytes = (uint32_t)H * 2;
  // the it-th row of this CTA: both rows of a pair, then the pair a grid further
  auto row_of = [&](int it) { return ((long long)blockIdx.x + (long long)(it >> 1) * gridDim.x) * 2 + (it & 1); };
  auto fetch = [&](int it) {
    const long long row = row_of(it);
    if (row >= T) return;
    uint8_t* dst = ring + (it % NORM_STAGES) * 3 * row_bytes;
    uint64_t* bar = &full[it % NORM_STAGES];
    b200::mbar_arrive_expect_tx(bar, (dres ? 3 : 2) * row_bytes);
    b200::bulk_load(dst, dy + row * H, row_bytes, bar);
    b200::bulk_load(dst + row_bytes, x + row * H, row_bytes, bar);
    if (dres) b200::bulk_load(dst + 2 * row_bytes, dres + row * H, row_bytes, bar);
  };
  b200::pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < NORM_STAGES; ++s) b200::mbar_init(&full[s], 1);
    b200::mbar_fence_init();
    for (int s = 0; s < NORM_STAGES - 1; ++s) fetch(s);
  }
  uint4 wv[VPT];
  float dw[VPT][8];
#pragma unroll
  for (int i = 0; i < VPT; ++i) {
    const int v = threadIdx.x + i * blockDim.x;
    wv[i] = make_uint4(0u, 0u, 0u, 0u);
    if (v < nvec) wv[i] = reinterpret_cast<const uint4*>(w)[v];
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[i][j] = 0.f;
  }
  __syncthreads();
  for (int it = 0;; ++it) {
    const long long row = row_of(it);
    if (row >= T) break;   // the pair's second row is the tensor's last row but one pair: nothing follows
    float rs = rstd[row];
    const uint4* in = reinterpret_cast<const uint4*>(ring + (it % NORM_STAGES) * 3 * row_bytes);
    if (!b200::mbar_wait(&full[it % NORM_STAGES], (it / NORM_STAGES) & 1)) rs = __int_as_float(0x7fffffff);   // NaN shows it
    uint4 a[VPT], b[VPT];
    float dot[1] = {0.f};
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      a[i] = b[i] = make_uint4(0u, 0u, 0u, 0u);
      if (v < nvec) {
        a[i] = in[v];
        b[i] = in[nvec + v];
      }
      float fa[8], fb[8], g[8];
      unpack8(a[i], fa);
      unpack8(b[i], fb);
      unpack8(wv[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = fb[j] * rs;
        dw[i][j] += fa[j] * xh;
        dot[0] += fa[j] * g[j] * xh;
      }
    }
    block_sums<1>(dot, sh[it & 1]);
    // its barrier says that every thread is through with the row before, whose stage takes the row three ahead
    if (threadIdx.x == 0) fetch(it + NORM_STAGES - 1);
    dot[0] /= (float)H;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v >= nvec) continue;
      float fa[8], fb[8], g[8], o[8];
      unpack8(a[i], fa);
      unpack8(b[i], fb);
      unpack8(wv[i], g);
      unpack8(dres ? in[2 * nvec + v] : make_uint4(0u, 0u, 0u, 0u), o);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] += rs * (fa[j] * g[j] - fb[j] * rs * dot[0]);
      reinterpret_cast<uint4*>(dx + row * H)[v] = pack8(o);
    }
  }
  if (dw_partial) {
    float4* out = reinterpret_cast<float4*>(dw_partial + (long long)blockIdx.x * H);
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int v = threadIdx.x + i * blockDim.x;
      if (v < nvec) {
        out[2 * v] = make_float4(dw[i][0], dw[i][1], dw[i][2], dw[i][3]);
        out[2 * v + 1] = make_float4(dw[i][4], dw[i][5], dw[i][6], dw[i][7]);
      }
    }
  }
}

// dw[c] = sum of the rows of partial [rows, H], as bf16: a warp takes every eighth row of 32 columns. Its CTAs are there when the
// kernel before ends (8192 x 3584, both: 43.0 us, one after the other 45.1).
__global__ void __launch_bounds__(256)
rmsnorm_dw_sum_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ dw, int rows, int H) {
  __shared__ float sh[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x * 32 + lane;
  b200::pdl_wait();
  float s = 0.f;
  if (c < H) {
#pragma unroll 8
    for (int r = warp; r < rows; r += 8) s += partial[(long long)r * H + c];
  }
  sh[warp][lane] = s;
  __syncthreads();
  if (warp == 0 && c < H) {
#pragma unroll
    for (int w = 1; w < 8; ++w) s += sh[w][lane];
    dw[c] = __float2bfloat16(s);
  }
}

// ---- RMSNorm backward of narrow rows (H <= 1024, the per-head q/k norms): two bandwidth-shaped kernels -----
// dx: one warp per row. dw: column strips, each block streams a strip of rows for 256 columns into the strip's row of
// dw_partial.
// H % 8 == 0, up to 4 vectors per lane
__global__ void __launch_bounds__(256)
rmsnorm_dx_warp_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                       const __nv_bfloat16* __restrict__ w, const float* __restrict__ rstd,
                       const __nv_bfloat16* __restrict__ dres, __nv_bfloat16* __restrict__ dx, long long T, int H) {
  const long long row = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= T) return;
  const int lane = threadIdx.x & 31, nvec = H >> 3;
  const uint4* dyr = reinterpret_cast<const uint4*>(dy + row * H);
  const uint4* xr = reinterpret_cast<const uint4*>(x + row * H);
  const uint4* wr = reinterpret_cast<const uint4*>(w);
  const float rs = rstd[row];
  float xh[4][8], dxh[4][8];
  float dot = 0.f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int v = lane + 32 * i;
    if (v < nvec) {
      float a[8], b[8], g[8];
      unpack8(dyr[v], a);
      unpack8(xr[v], b);
      unpack8(wr[v], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[i][j] = b[j] * rs;
        dxh[i][j] = a[j] * g[j];
        dot += dxh[i][j] * xh[i][j];
      }
    }
  }
  dot = warp_sum(dot) / (float)H;
  uint4* dxr = reinterpret_cast<uint4*>(dx + row * H);
  const uint4* drr = dres ? reinterpret_cast<const uint4*>(dres + row * H) : nullptr;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    int v = lane + 32 * i;
    if (v < nvec) {
      float o[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = rs * (dxh[i][j] - xh[i][j] * dot);
      if (drr) {
        float r[8];
        unpack8(drr[v], r);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] += r[j];
      }
      dxr[v] = pack8(o);
    }
  }
}

// dw_partial[strip, c] = sum_t dy[t,c] * x[t,c] * rstd[t] over the strip; grid (ceil(H/256), row strips), 8 warps per CTA split the strip
__global__ void __launch_bounds__(256)
rmsnorm_dw_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                  const float* __restrict__ rstd, float* __restrict__ dw_partial, long long T, int H) {
  __shared__ float sh[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = blockIdx.x * 256 + lane * 8;
  const long long rows_per_cta = (T + gridDim.y - 1) / gridDim.y;
  const long long r0 = blockIdx.y * rows_per_cta, r1 = min(T, r0 + rows_per_cta);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (c0 < H) {
    for (long long r = r0 + warp; r < r1; r += 8) {
      float a[8], b[8];
      unpack8(*reinterpret_cast<const uint4*>(dy + r * H + c0), a);
      unpack8(*reinterpret_cast<const uint4*>(x + r * H + c0), b);
      const float rs = rstd[r];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += a[j] * b[j] * rs;
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) sh[warp][lane * 8 + j] = acc[j];
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < H) {
    float s = 0.f;
#pragma unroll
    for (int wv = 0; wv < 8; ++wv) s += sh[wv][threadIdx.x];
    dw_partial[(long long)blockIdx.y * H + c] = s;
  }
}

// ------------------------------------------------------------------------------------------------
// RoPE (rotate-half convention), in place, cos/sin evaluated in fp32 from the integer position
// ------------------------------------------------------------------------------------------------
__global__ void rope_kernel(__nv_bfloat16* __restrict__ q, __nv_bfloat16* __restrict__ k,
                            const long long* __restrict__ pos, int T, int hq, int hkv, int d, long long q_stride,
                            long long k_stride, float log2_theta, float sign) {
  const int half = d >> 1;
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)T * half) return;
  const int i = (int)(idx % half);
  const long long t = idx / half;
  const float inv_freq = exp2f(-(2.0f * (float)i / (float)d) * log2_theta);
  float s, c;
  sincosf((float)pos[t] * inv_freq, &s, &c);
  s *= sign;
  __nv_bfloat16* qp = q + t * q_stride;
  for (int h = 0; h < hq; ++h) {
    float a = __bfloat162float(qp[h * d + i]), b = __bfloat162float(qp[h * d + i + half]);
    qp[h * d + i] = __float2bfloat16(a * c - b * s);
    qp[h * d + i + half] = __float2bfloat16(b * c + a * s);
  }
  if (k) {
    __nv_bfloat16* kp = k + t * k_stride;
    for (int h = 0; h < hkv; ++h) {
      float a = __bfloat162float(kp[h * d + i]), b = __bfloat162float(kp[h * d + i + half]);
      kp[h * d + i] = __float2bfloat16(a * c - b * s);
      kp[h * d + i + half] = __float2bfloat16(b * c + a * s);
    }
  }
}

// Vectorised form. A CTA has ROWS tokens: a thread has 8 rotation pairs of a head of each (16-byte loads and stores), and the tokens'
// sines and cosines are formed once, in shared memory, while those are on their way. `plain` heads behind the rotated ones are
// copied (the values of a gradient that is not rotated in place). 32 heads of 128, in place: 8192 tokens 26.1 us, with the
// angles formed again for every four heads 28.8 (20 are the bytes); 57 tokens, 6 heads 2.3 and 4.0. Persistent CTAs that
// fetch a token ahead have the angles of one token after the other: 40. In place q_out is q and k_out is k, so neither is
// __restrict__: a thread reads its vectors before it writes them, and nobody else touches them.
constexpr int ROPE_MAX_D = 512, ROPE_MAX_THREADS = 512;
template <int ROWS>
__global__ void __launch_bounds__(ROPE_MAX_THREADS)
rope_vec_kernel(const __nv_bfloat16* q, const __nv_bfloat16* k, __nv_bfloat16* q_out, __nv_bfloat16* k_out,
                const long long* __restrict__ pos, int T, int hq, int hkv, int plain, int d, long long q_stride, long long k_stride,
                long long q_out_stride, long long k_out_stride, float log2_theta, float sign) {
  __shared__ float2 sc[ROWS][ROPE_MAX_D / 2];   // sine, cosine
  const int half = d >> 1, vecs = half >> 3, items = (hq + hkv + plain) * vecs;
  const long long t0 = (long long)blockIdx.x * ROWS;
  uint4 lo[ROWS], hi[ROWS];
  auto load = [&](int item) {
    const int h = item / vecs, v = item - h * vecs;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      lo[r] = hi[r] = make_uint4(0u, 0u, 0u, 0u);
      if (t0 + r >= T) continue;
      const __nv_bfloat16* src =
          (h < hq ? q + (t0 + r) * q_stride + (long long)h * d : k + (t0 + r) * k_stride + (long long)(h - hq) * d) + v * 8;
      lo[r] = *reinterpret_cast<const uint4*>(src);
      hi[r] = *reinterpret_cast<const uint4*>(src + half);
    }
  };
  if (threadIdx.x < items) load(threadIdx.x);
  for (int i = threadIdx.x; i < ROWS * half; i += blockDim.x) {
    const int r = i / half, f = i - r * half;
    if (t0 + r >= T) break;
    const float inv_freq = exp2f(-(2.0f * (float)f / (float)d) * log2_theta);
    float s, c;
    sincosf((float)pos[t0 + r] * inv_freq, &s, &c);
    sc[r][f] = make_float2(s * sign, c);
  }
  __syncthreads();
  for (int item = threadIdx.x; item < items; item += blockDim.x) {
    if (item != threadIdx.x) load(item);
    const int h = item / vecs, v = item - h * vecs;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      if (t0 + r >= T) break;
      if (h < hq + hkv) {
        float a[8], b[8], oa[8], ob[8];
        unpack8(lo[r], a);
        unpack8(hi[r], b);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 w = sc[r][v * 8 + j];
          oa[j] = a[j] * w.y - b[j] * w.x;
          ob[j] = b[j] * w.y + a[j] * w.x;
        }
        lo[r] = pack8(oa);
        hi[r] = pack8(ob);
      }
      __nv_bfloat16* dst =
          (h < hq ? q_out + (t0 + r) * q_out_stride + (long long)h * d : k_out + (t0 + r) * k_out_stride + (long long)(h - hq) * d) + v * 8;
      *reinterpret_cast<uint4*>(dst) = lo[r];
      *reinterpret_cast<uint4*>(dst + half) = hi[r];
    }
  }
}

// ------------------------------------------------------------------------------------------------
// SwiGLU on a fused [T, 2I] gate|up projection
// ------------------------------------------------------------------------------------------------
// Positions are found with 32-bit divisions unless the tensor is too large for them. row_tiles (nullable, device): only the
// first row_tiles[0] * 128 rows are in use. A thread of the forward works on ITEMS vectors of 8 columns whose loads are all in
// flight before the first is used. The quotient is a division, as in the epilogues that form SwiGLU elsewhere: the same gate and
// up values give the same bits there and here, which a product with the reciprocal (one rounding more, 8192 x 18944 in 153 us)
// does not. Zero gates would send it through its path for special operands, so a thread that has nothing else (rows of padding)
// does not divide: 8192 x 18944 165 us, all zero 135 (163 and 300 if it does).
template <class Index, int ITEMS>
__global__ void __launch_bounds__(256)
swiglu_fwd_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, long long T, int I,
                  const int* __restrict__ row_tiles) {
  const Index nvec = I >> 3;
  const Index total = (Index)(row_tiles ? min((long long)row_tiles[0] * 128, T) : T) * nvec;
  const Index first = (Index)blockIdx.x * (256 * ITEMS) + threadIdx.x;
  uint4 g[ITEMS], u[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    const Index idx = first + k * 256;
    g[k] = make_uint4(0, 0, 0, 0);
    if (idx >= total) continue;
    const Index t = idx / nvec, v = idx - t * nvec;
    const uint4* row = reinterpret_cast<const uint4*>(gu + (long long)t * 2 * I);
    g[k] = row[v];
    u[k] = row[nvec + v];
  }
  uint32_t any = 0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) any |= g[k].x | g[k].y | g[k].z | g[k].w;
  auto write = [&](auto silu) {
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      const Index idx = first + k * 256;
      if (idx >= total) continue;
      float a[8], b[8], o[8];
      unpack8(g[k], a);
      unpack8(u[k], b);
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = silu(a[j]) * b[j];
      reinterpret_cast<uint4*>(out)[idx] = pack8(o);
    }
  };
  if (any & 0x7fff7fffu) write([](float x) { return x / (1.f + __expf(-x)); });
  else write([](float x) { return x; });
}

template <class Index>
__global__ void __launch_bounds__(256)
swiglu_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ gu,
                  __nv_bfloat16* __restrict__ dgu, long long T, int I, const int* __restrict__ row_tiles) {
  const Index nvec = I >> 3;
  const Index total = (Index)(row_tiles ? min((long long)row_tiles[0] * 128, T) : T) * nvec;
  const Index idx = (Index)blockIdx.x * 256 + threadIdx.x;
  if (idx >= total) return;
  const Index t = idx / nvec, v = idx - t * nvec;
  const uint4* in = reinterpret_cast<const uint4*>(gu + (long long)t * 2 * I);
  const uint4 g = in[v], u = in[nvec + v], dd = reinterpret_cast<const uint4*>(dout)[idx];
  float a[8], b[8], d[8], dg[8], du[8];
  unpack8(g, a);
  unpack8(u, b);
  unpack8(dd, d);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float s = 1.f / (1.f + __expf(-a[j]));
    float silu = a[j] * s;
    dg[j] = d[j] * b[j] * (s + silu * (1.f - s));
    du[j] = d[j] * silu;
  }
  uint4* out = reinterpret_cast<uint4*>(dgu + (long long)t * 2 * I);
  out[v] = pack8(dg);
  out[nvec + v] = pack8(du);
}

// ------------------------------------------------------------------------------------------------
// AdamW on flat buffers
// ------------------------------------------------------------------------------------------------
template <bool GRAD_FP32>
__global__ void __launch_bounds__(256)
adamw_kernel(float* __restrict__ master, float* __restrict__ m, float* __restrict__ v, const void* __restrict__ grad,
             __nv_bfloat16* __restrict__ shadow, long long n, float lr, float b1, float b2, float eps, float wd,
             float bias1, float bias2, const float* __restrict__ gscale) {
  const float gs = gscale ? *gscale : 1.f;
  const float step = lr / bias1;
  const float inv_sqrt_b2 = rsqrtf(bias2);
  long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  const long long stride = (long long)gridDim.x * blockDim.x * 4;
  for (; i + 3 < n; i += stride) {
    float4 p = *reinterpret_cast<float4*>(master + i);
    float4 mm = *reinterpret_cast<float4*>(m + i);
    float4 vv = *reinterpret_cast<float4*>(v + i);
    float g[4];
    if (GRAD_FP32) {
      float4 t = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(grad) + i);
      g[0] = t.x; g[1] = t.y; g[2] = t.z; g[3] = t.w;
    } else {
      uint2 t = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(grad) + i);
      float2 lo = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&t.x));
      float2 hi = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&t.y));
      g[0] = lo.x; g[1] = lo.y; g[2] = hi.x; g[3] = hi.y;
    }
    float pp[4] = {p.x, p.y, p.z, p.w}, pm[4] = {mm.x, mm.y, mm.z, mm.w}, pv[4] = {vv.x, vv.y, vv.z, vv.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float gj = g[j] * gs;
      pp[j] *= (1.f - lr * wd);
      pm[j] = b1 * pm[j] + (1.f - b1) * gj;
      pv[j] = b2 * pv[j] + (1.f - b2) * gj * gj;
      pp[j] -= step * pm[j] / (sqrtf(pv[j]) * inv_sqrt_b2 + eps);
    }
    *reinterpret_cast<float4*>(master + i) = make_float4(pp[0], pp[1], pp[2], pp[3]);
    *reinterpret_cast<float4*>(m + i) = make_float4(pm[0], pm[1], pm[2], pm[3]);
    *reinterpret_cast<float4*>(v + i) = make_float4(pv[0], pv[1], pv[2], pv[3]);
    if (shadow) {
      uint2 o;
      *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(pp[0], pp[1]);
      *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(pp[2], pp[3]);
      *reinterpret_cast<uint2*>(shadow + i) = o;
    }
  }
  // tail (n not a multiple of 4): handled by the first thread
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (long long t = n & ~3ll; t < n; ++t) {
      float gj = (GRAD_FP32 ? reinterpret_cast<const float*>(grad)[t]
                            : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(grad)[t])) * gs;
      float p = master[t] * (1.f - lr * wd);
      float mm = b1 * m[t] + (1.f - b1) * gj;
      float vv = b2 * v[t] + (1.f - b2) * gj * gj;
      p -= step * mm / (sqrtf(vv) * inv_sqrt_b2 + eps);
      master[t] = p; m[t] = mm; v[t] = vv;
      if (shadow) shadow[t] = __float2bfloat16(p);
    }
  }
}

template <bool FP32>
__global__ void __launch_bounds__(256) sumsq_kernel(const void* __restrict__ x, long long n, float* __restrict__ out) {
  __shared__ float sh[32];
  float s = 0.f;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (FP32) {
    const float* p = reinterpret_cast<const float*>(x);
    for (; i < n; i += stride) { float t = p[i]; s += t * t; }
  } else {
    const __nv_bfloat16* p = reinterpret_cast<const __nv_bfloat16*>(x);
    const long long nvec = n >> 3;
    const uint4* pv = reinterpret_cast<const uint4*>(p);
    for (long long v = i; v < nvec; v += stride) {
      float f[8];
      unpack8(pv[v], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) s += f[j] * f[j];
    }
    for (long long t = (nvec << 3) + i; t < n; t += stride) { float f = __bfloat162float(p[t]); s += f * f; }
  }
  s = block_sum<256>(s, sh);
  if (threadIdx.x == 0) atomicAdd(out, s);
}

__global__ void clip_coef_kernel(const float* sumsq, float max_norm, float* coef, float* norm_out) {
  float n = sqrtf(*sumsq);
  if (norm_out) *norm_out = n;
  float c = max_norm > 0.f ? max_norm / (n + 1e-6f) : 1.f;
  *coef = c < 1.f ? c : 1.f;
}

// threads of a CTA and vectors per thread for a row of H elements
struct NormShape {
  int vpt, threads;
  explicit NormShape(int H) {
    const int nvec = H >> 3;
    vpt = nvec <= NORM_MAX_THREADS ? 1 : 2;
    threads = ((nvec + vpt - 1) / vpt + 31) / 32 * 32;
  }
};

inline int ok() { return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH; }

}  // namespace

constexpr int ROPE_ROWS = 2;
static int launch_rope_vec(const void* q, const void* k, void* q_out, void* k_out, const long long* positions, int T, int hq, int hkv,
                           int plain, int d, long long q_stride, long long k_stride, long long q_out_stride, long long k_out_stride,
                           float theta, int backward, cudaStream_t stream) {
  // a token that is more than 512 vectors is taken in equal parts
  const int items = (hq + hkv + plain) * (d / 16);
  if (items <= 0) return B200_ERR_ARG;
  const int parts = (items + ROPE_MAX_THREADS - 1) / ROPE_MAX_THREADS;
  const int threads = ((items + parts - 1) / parts + 31) / 32 * 32, rows = T >= 148 * 4 ? ROPE_ROWS : 1;
  auto kern = rows == 1 ? rope_vec_kernel<1> : rope_vec_kernel<ROPE_ROWS>;
  kern<<<(unsigned)((T + rows - 1) / rows), threads, 0, stream>>>(
      (const __nv_bfloat16*)q, (const __nv_bfloat16*)k, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_out, positions, T, hq, hkv, plain, d,
      q_stride, k_stride, q_out_stride, k_out_stride, log2f(theta), backward ? -1.f : 1.f);
  return ok();
}

extern "C" {

int b200_rmsnorm_fwd(const void* x, const void* residual, const void* w, void* y, void* residual_out, float* rstd,
                     int T, int H, float eps, cudaStream_t stream) {
  if (T <= 0) return 0;
  if ((H & 7) || H > NORM_MAX_H) return B200_ERR_ARG;
  const NormShape n(H);
  // two rows a CTA once every SM has several CTAs of work anyway
  const int rows = T >= 148 * 8 ? 2 : 1;
  const unsigned grid = (unsigned)((T + rows - 1) / rows);
  auto go = [&](auto kern) {
    kern<<<grid, n.threads, 0, stream>>>((const __nv_bfloat16*)x, (const __nv_bfloat16*)residual, (const __nv_bfloat16*)w,
                                         (__nv_bfloat16*)y, (__nv_bfloat16*)residual_out, rstd, T, H, eps);
  };
  if (n.vpt == 1) rows == 2 ? go(rmsnorm_fwd_kernel<1, 2>) : go(rmsnorm_fwd_kernel<1, 1>);
  else rows == 2 ? go(rmsnorm_fwd_kernel<2, 2>) : go(rmsnorm_fwd_kernel<2, 1>);
  return ok();
}

// dx (+ dres) and dw (bf16; null: no weight gradient). ws: fp32 scratch of RMSNORM_WS_ROWS * max(H, 1024) elements.
int b200_rmsnorm_bwd2(const void* dy, const void* x, const void* w, const float* rstd, const void* dres, void* dx,
                      void* dw, float* ws, long long T, int H, cudaStream_t stream) {
  if (T <= 0) return dw ? (cudaMemsetAsync(dw, 0, (size_t)H * 2, stream) == cudaSuccess ? 0 : B200_ERR_RUNTIME) : 0;
  if ((H & 7) || H > NORM_MAX_H || (dw && !ws)) return B200_ERR_ARG;
  if (!dw) ws = nullptr;
  int rows = 0;   // of partial weight gradients
  if (H <= 1024) {
    rmsnorm_dx_warp_kernel<<<(unsigned)((T + 7) / 8), 256, 0, stream>>>(
        (const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, rstd, (const __nv_bfloat16*)dres,
        (__nv_bfloat16*)dx, T, H);
    if (dw) {
      const int col_blocks = (H + 255) / 256;
      long long strips = RMSNORM_WS_ROWS * 4 / col_blocks;   // col_blocks * 256 <= 1024 columns of the scratch
      if (strips > (T + 63) / 64) strips = (T + 63) / 64;
      rows = (int)strips;
      rmsnorm_dw_kernel<<<dim3(col_blocks, rows), 256, 0, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x,
                                                                    rstd, ws, T, H);
    }
  } else {
    const NormShape n(H);
    if (((uintptr_t)dy | (uintptr_t)x | (uintptr_t)dres) & 15) return B200_ERR_ARG;
    const int smem = NORM_STAGES * 3 * H * 2;
    auto go = [&](auto kern, int ctas) {
      const long long pairs = (T + 1) / 2;
      rows = (int)(pairs < ctas ? pairs : ctas);
      kern<<<rows, n.threads, smem, stream>>>((const __nv_bfloat16*)dy, (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, rstd,
                                              (const __nv_bfloat16*)dres, (__nv_bfloat16*)dx, ws, T, H);
    };
    // the limit is the device's, not the process's
    static bool raised[16] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) return B200_ERR_RUNTIME;
    if (!raised[dev]) {
      constexpr int most = NORM_STAGES * 3 * NORM_MAX_H * 2;
      if (cudaFuncSetAttribute(rmsnorm_bwd_kernel<1, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, most / 2) != cudaSuccess ||
          cudaFuncSetAttribute(rmsnorm_bwd_kernel<2, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess)
        return B200_ERR_LAUNCH;
      raised[dev] = true;
    }
    if (n.vpt == 1) go(rmsnorm_bwd_kernel<1, 2>, RMSNORM_WS_ROWS);
    else go(rmsnorm_bwd_kernel<2, 1>, RMSNORM_WS_ROWS / 2);
  }
  if (dw && b200::launch_pdl(rmsnorm_dw_sum_kernel, dim3((H + 31) / 32), dim3(256), 0, stream, (const float*)ws,
                             (__nv_bfloat16*)dw, rows, H) != cudaSuccess)
    return B200_ERR_LAUNCH;
  return ok();
}

int b200_rope_inplace(void* q, void* k, const long long* positions, int T, int hq, int hkv, int d, long long q_stride,
                      long long k_stride, float theta, int backward, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (d & 1) return B200_ERR_ARG;
  const bool aligned = !(d & 15) && d <= ROPE_MAX_D && !(q_stride & 7) && !(k_stride & 7) && !((uintptr_t)q & 15) && !((uintptr_t)k & 15);
  if (aligned)
    return launch_rope_vec(q, k, q, k, positions, T, hq, k ? hkv : 0, 0, d, q_stride, k_stride, q_stride, k_stride, theta, backward,
                           stream);
  long long n = (long long)T * (d / 2);
  rope_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>((__nv_bfloat16*)q, (__nv_bfloat16*)k, positions, T, hq,
                                                              hkv, d, q_stride, k_stride, log2f(theta),
                                                              backward ? -1.f : 1.f);
  return ok();
}

int b200_rope_qkv(const void* src, void* dst, const long long* positions, int T, int hq, int hkv, int d, long long src_stride,
                  long long dst_stride, float theta, int backward, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (hq <= 0 || hkv <= 0 || d <= 0 || (d & 15) || d > ROPE_MAX_D || (src_stride & 7) || (dst_stride & 7) || ((uintptr_t)src & 15) ||
      ((uintptr_t)dst & 15))
    return B200_ERR_ARG;
  const long long k_at = (long long)hq * d;
  return launch_rope_vec(src, (const __nv_bfloat16*)src + k_at, dst, (__nv_bfloat16*)dst + k_at, positions, T, hq, hkv, hkv, d,
                         src_stride, src_stride, dst_stride, dst_stride, theta, backward, stream);
}

int b200_swiglu_fwd(const void* gate_up, void* out, long long T, int I, const int* row_tiles, cudaStream_t stream) {
  if (T <= 0) return 0;
  if (I & 7) return B200_ERR_ARG;
  // Two vectors a thread once they fill the machine several times over: 2000 x 14336 32.2 us, with one 33.6; 1000 x 14336 16.0
  // and 16.1. Below that more threads hide more: 57 x 768 2.7 and 2.1.
  const long long n = T * (I / 8);
  const int items = n >= (3ll << 19) ? 2 : 1, per = 256 * items;
  auto kern = n >= (1ll << 32) - 1024 ? swiglu_fwd_kernel<unsigned long long, 2>
              : items == 2            ? swiglu_fwd_kernel<uint32_t, 2>
                                      : swiglu_fwd_kernel<uint32_t, 1>;
  kern<<<(unsigned)((n + per - 1) / per), 256, 0, stream>>>((const __nv_bfloat16*)gate_up, (__nv_bfloat16*)out, T, I,
                                                            row_tiles);
  return ok();
}

int b200_swiglu_bwd(const void* dout, const void* gate_up, void* dgate_up, long long T, int I, const int* row_tiles,
                    cudaStream_t stream) {
  if (T <= 0) return 0;
  if (I & 7) return B200_ERR_ARG;
  // One vector a thread (8192 x 18944: 223 us, with two 241; 57 x 768: 2.3 and 3.1)
  const long long n = T * (I / 8);
  auto kern = n >= (1ll << 32) - 512 ? swiglu_bwd_kernel<unsigned long long> : swiglu_bwd_kernel<uint32_t>;
  kern<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>((const __nv_bfloat16*)dout, (const __nv_bfloat16*)gate_up,
                                                        (__nv_bfloat16*)dgate_up, T, I, row_tiles);
  return ok();
}

int b200_adamw(float* master, float* m, float* v, const void* grad, int grad_fp32, void* param_bf16, long long n,
               float lr, float beta1, float beta2, float eps, float weight_decay, float bias1, float bias2,
               const float* grad_scale_dev, cudaStream_t stream) {
  if (n <= 0) return 0;
  long long want = (n / 4 + 255) / 256;
  int grid = (int)(want < 148 * 16 ? (want > 0 ? want : 1) : 148 * 16);
  if (grad_fp32)
    adamw_kernel<true><<<grid, 256, 0, stream>>>(master, m, v, grad, (__nv_bfloat16*)param_bf16, n, lr, beta1, beta2,
                                                 eps, weight_decay, bias1, bias2, grad_scale_dev);
  else
    adamw_kernel<false><<<grid, 256, 0, stream>>>(master, m, v, grad, (__nv_bfloat16*)param_bf16, n, lr, beta1,
                                                  beta2, eps, weight_decay, bias1, bias2, grad_scale_dev);
  return ok();
}

int b200_sumsq(const void* x, int is_fp32, long long n, float* out_accum, cudaStream_t stream) {
  if (n <= 0) return 0;
  long long want = (n / 8 + 255) / 256;
  int grid = (int)(want < 148 * 8 ? (want > 0 ? want : 1) : 148 * 8);
  if (is_fp32)
    sumsq_kernel<true><<<grid, 256, 0, stream>>>(x, n, out_accum);
  else
    sumsq_kernel<false><<<grid, 256, 0, stream>>>(x, n, out_accum);
  return ok();
}

int b200_clip_coef(const float* sumsq, float max_norm, float* coef_out, float* norm_out, cudaStream_t stream) {
  clip_coef_kernel<<<1, 1, 0, stream>>>(sumsq, max_norm, coef_out, norm_out);
  return ok();
}

}  // extern "C"
