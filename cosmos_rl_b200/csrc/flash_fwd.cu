// Varlen (packed) causal flash-attention forward on tcgen05 / TMEM / TMA for head_dim 128, GQA.
//
// One CTA = (sequence, 256 queries, query head) as two tiles of 128 queries that share every K / V tile. Per tile t and
// 128-key block j:
//     S_t  = Q_t K_j^T          tcgen05.mma M=128 (queries) N=128 (keys) K=128 (d), both operands K-major (TMA, SW128)
//     P_t  = exp2(S_t*c - m)    one thread per query row (TMEM lane) holds the whole row in registers: no shuffles, no
//                               shared memory; P goes back as bf16 over the columns of S_t
//     O_t += P_t V_j            A = P_t out of TMEM, B = V MN-major, so the [token, d] layout is used as stored
// While the softmax warps of one tile work, the tensor core runs the two products of the other. Reading P out of TMEM
// and sharing K / V between the tiles leaves 192 KB of shared-memory reads per key block for 2048 tensor-core cycles;
// 2 x 128 x 128 exponentials at 16 per cycle take the same 2048, so the exponentials and the products bound the kernel
// together. Timing: profiles/flash_attention_B16_L4096.md.
// O stays in TMEM for the whole item and is rescaled lazily: the running maximum only moves when it grows by more than
// 2^8, so the TMEM read-modify-write of O is rare. S_t(j+1) is issued after P_t(j) V_j by the same thread and the tensor
// core keeps that order, so "S_t(j+1) is ready" also says that P_t(j) has been read and O_t updated.
// Roles: warp 0 TMA producer, warp 1 MMA issuer, warps 2-5 / 6-9 softmax and epilogue of tile 0 / 1.
// Outputs O [T, hq, d] bf16 and LSE [hq, T] fp32 (natural log of the softmax denominator of the scaled scores).
// Queries are aligned to the END of the keys of their sequence (len_k >= len_q: prefill with a prefix cache,
// context-parallel chunks); with cu_q == cu_k this is ordinary causal self-attention.
// Replaces flash_attn_varlen_func (cosmos_rl/policy/kernel/modeling_utils.py:65-173). Every wait is bounded.
#include "sm100.cuh"
#include "gemm_core.cuh"
#include "api.h"

namespace b200 {

constexpr int FA_B = 128;                         // queries per tile / keys per block
constexpr int FA_D = 128;
constexpr int FA_TILE = FA_B * FA_D * 2;          // 32 KiB
constexpr int FA_SMEM = 6 * FA_TILE + 256 + 1024; // Q x2, K x2, V x2, barriers, alignment
constexpr int FA_THREADS = 320;
constexpr float FA_LOG2E = 1.4426950408889634f;
constexpr float FA_LN2 = 0.6931471805599453f;
constexpr float FA_RESCALE_TAU = 8.0f;

struct FaParams {
  const int* cu_q;
  const int* cu_k;
  __nv_bfloat16* out;
  float* lse;
  long long ldo;      // elements between tokens of out
  int B, hq, hkv, Tq, causal;
  float scale_log2;
  uint32_t* status;
};

#define FA_WAIT1(bar, parity, code)           \
  if (!mbar_wait(bar, parity)) {              \
    atomicCAS(p.status, ST_OK, code);         \
    *abort_flag = 1;                          \
    break;                                    \
  }

__global__ void __launch_bounds__(FA_THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, FaParams p) {
  const int heads = p.hq * p.B, nblk = gridDim.x / heads;
  const int hb = blockIdx.x % heads, h = hb % p.hq, b = hb / p.hq;
  const int q0 = (nblk - 1 - (int)blockIdx.x / heads) * 2 * FA_B;   // heavy (late) query blocks first
  const int q_beg = p.cu_q[b], len_q = p.cu_q[b + 1] - q_beg;
  const int k_beg = p.cu_k[b], len_k = p.cu_k[b + 1] - k_beg;
  if (q0 >= len_q) return;
  const int shift = len_k - len_q;
  const int hk = h / (p.hq / p.hkv);
  auto key_blocks = [&](int t) -> int {           // key blocks that some query of tile t sees
    if (q0 + t * FA_B >= len_q) return 0;
    const int end = p.causal ? min(len_k, q0 + (t + 1) * FA_B + shift) : len_k;
    return end > 0 ? (end + FA_B - 1) / FA_B : 0;
  };
  const int n0 = key_blocks(0), n1 = key_blocks(1), n = max(n0, n1);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_sh = smem;                    // [2]
  uint8_t* k_sh = smem + 2 * FA_TILE;      // [2]
  uint8_t* v_sh = smem + 4 * FA_TILE;      // [2]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * FA_TILE);
  uint64_t* qfull = bars;        // [2]
  uint64_t* kfull = bars + 2;    // [2]
  uint64_t* kempty = bars + 4;   // [2]
  uint64_t* vfull = bars + 6;    // [2]
  uint64_t* vempty = bars + 8;   // [2]
  uint64_t* s_ready = bars + 10; // [2] per tile
  uint64_t* p_ready = bars + 12; // [2] per tile
  uint64_t* o_done = bars + 14;  // [2] per tile: the last product of the tile has finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&qfull[s], 1);
      mbar_init(&kfull[s], 1);
      mbar_init(&kempty[s], 1);
      mbar_init(&vfull[s], 1);
      mbar_init(&vempty[s], 1);
      mbar_init(&s_ready[s], 1);
      mbar_init(&p_ready[s], 4);
      mbar_init(&o_done[s], 1);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;   // columns: S / P of tile 0, 1 at 0, 128; O of tile 0, 1 at 256, 384

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    if (lane == 0 && n > 0) {
      auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row) {
        mbar_arrive_expect_tx(bar, FA_TILE);
        tma_load_2d(dst, tm, bar, col, row);
        tma_load_2d(dst + FA_TILE / 2, tm, bar, col + 64, row);
      };
      if (n0 > 0) load(q_sh, &tm_q, &qfull[0], h * FA_D, q_beg + q0);
      for (int j = 0; j < n && !*abort_flag; ++j) {
        const int s = j & 1;
        const uint32_t ph = ((j >> 1) & 1) ^ 1;
        const int row = k_beg + j * FA_B;
        FA_WAIT1(&kempty[s], ph, ST_TIMEOUT_EMPTY)
        load(k_sh + s * FA_TILE, &tm_k, &kfull[s], hk * FA_D, row);
        if (j == 0 && n1 > 0) load(q_sh + FA_TILE, &tm_q, &qfull[1], h * FA_D, q_beg + q0 + FA_B);
        FA_WAIT1(&vempty[s], ph, ST_TIMEOUT_EMPTY)
        load(v_sh + s * FA_TILE, &tm_v, &vfull[s], hk * FA_D, row);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (lane == 0 && n > 0) {
      constexpr uint32_t idesc_s = umma_idesc_bf16_f32(FA_B, FA_B);
      constexpr uint32_t idesc_o = umma_idesc_bf16_f32(FA_B, FA_D) | (1u << 16);   // B (= V) is MN-major
      auto mma_s = [&](int t, int j) {
        const uint32_t qs = smem_u32(q_sh + t * FA_TILE), ks = smem_u32(k_sh + (j & 1) * FA_TILE);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = (k >> 2) * (FA_TILE / 2) + (k & 3) * 32;
          umma_bf16_ss(tmem_base + t * FA_B, umma_desc_kmajor_sw128(qs + off), umma_desc_kmajor_sw128(ks + off), idesc_s,
                       k > 0 ? 1u : 0u);
        }
        tc_commit(&s_ready[t]);
      };
      auto mma_o = [&](int t, int j) {
        const uint32_t vs = smem_u32(v_sh + (j & 1) * FA_TILE);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ts(tmem_base + 256 + t * FA_D, tmem_base + t * FA_B + k * 8,
                       umma_desc_mnmajor_sw128(vs + k * 2048, FA_TILE / 2), idesc_o, (j > 0 || k > 0) ? 1u : 0u);
      };
      do {
        FA_WAIT1(&kfull[0], 0, ST_TIMEOUT_FULL)
        if (n0 > 0) {
          FA_WAIT1(&qfull[0], 0, ST_TIMEOUT_FULL)
          tc_fence_after_sync();
          mma_s(0, 0);
        }
        if (n1 > 0) {
          FA_WAIT1(&qfull[1], 0, ST_TIMEOUT_FULL)
          tc_fence_after_sync();
          mma_s(1, 0);
        }
        if (n > 2) tc_commit(&kempty[0]);   // only commits that the producer will wait for
        bool ok = true;
        for (int j = 0; j < n && ok; ++j) {
          FA_WAIT1(&vfull[j & 1], (j >> 1) & 1, ST_TIMEOUT_FULL)
          if (j + 1 < n) FA_WAIT1(&kfull[(j + 1) & 1], ((j + 1) >> 1) & 1, ST_TIMEOUT_FULL)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int nt = t ? n1 : n0;
            if (j >= nt) continue;
            if (!mbar_wait(&p_ready[t], j & 1)) {
              atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_EMPTY);
              *abort_flag = 1;
              ok = false;
              break;
            }
            tc_fence_after_sync();
            mma_o(t, j);
            if (j + 1 < nt) mma_s(t, j + 1);
            else tc_commit(&o_done[t]);
          }
          if (!ok) break;
          if (j + 2 < n) tc_commit(&vempty[j & 1]);
          if (j + 3 < n) tc_commit(&kempty[(j + 1) & 1]);
        }
      } while (false);
    }
  } else {
    // ------------------------------------------------ softmax + epilogue
    const int t = (warp - 2) >> 2;
    const int nt = t ? n1 : n0;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const uint32_t ts = tmem_base + t * FA_B + lane_addr, to = tmem_base + 256 + t * FA_D + lane_addr;
    const int q_idx = q0 + t * FA_B + row;         // position inside the sequence's queries
    const int k_limit = p.causal ? min(len_k, q_idx + shift + 1) : len_k;   // keys [0, k_limit) are visible
    const float2 c2 = make_float2(p.scale_log2, p.scale_log2);
    float m_run = -INFINITY, l_run = 0.f;
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {   // the whole warp: tcgen05.ld / st are warp-collective
      const bool w = mbar_wait(bar, parity);
      if (!w) {
        atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_FULL);
        *abort_flag = 1;
      }
      return __all_sync(0xffffffffu, w);
    };
    for (int j = 0; j < nt; ++j) {
      if (!(ok = wait(&s_ready[t], j & 1))) break;
      tc_fence_after_sync();
      uint32_t r[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(ts + c * 32, r[c]);
      tmem_ld_wait();
      const int kbase = j * FA_B;
      if (kbase + FA_B > k_limit) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i)
            if (kbase + c * 32 + i >= k_limit) r[c][i] = 0xff800000u;   // -infinity
      }
      float mx4[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mx4[c] = __uint_as_float(r[c][0]);
#pragma unroll
        for (int i = 1; i < 32; ++i) mx4[c] = fmaxf(mx4[c], __uint_as_float(r[c][i]));
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale_log2;   // scale > 0
      const bool grow = mx > m_run + FA_RESCALE_TAU || (m_run == -INFINITY && mx != -INFINITY);
      float corr = 1.f;
      if (grow) {
        corr = (m_run == -INFINITY) ? 0.f : exp2f(m_run - mx);
        m_run = mx;
        l_run *= corr;
      }
      if (j > 0 && __any_sync(0xffffffffu, grow)) {
#pragma unroll 1
        for (int c = 0; c < FA_D; c += 16) {
          uint32_t o[16];
          tmem_ld_32x32b_x16(to + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
          tmem_st_32x32b_x16(to + c, o);
        }
      }
      const float nm = (m_run == -INFINITY) ? 0.f : -m_run;
      const float2 nm2 = make_float2(nm, nm);
      float2 sum[4];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t pk[32];
#pragma unroll
        for (int c = 2 * hf; c < 2 * hf + 2; ++c) {
          sum[c] = make_float2(0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float2 x = fma2(make_float2(__uint_as_float(r[c][2 * i]), __uint_as_float(r[c][2 * i + 1])), c2, nm2);
            const float2 e = make_float2(exp2_approx(x.x), exp2_approx(x.y));
            sum[c] = add2(sum[c], e);
            pk[(c & 1) * 16 + i] = pack_bf16x2(e.x, e.y);
          }
        }
        tmem_st_32x32b_x32(ts + hf * 32, pk);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[t]);
      const float2 s2 = add2(add2(sum[0], sum[1]), add2(sum[2], sum[3]));
      l_run += s2.x + s2.y;
    }
    // ---- epilogue: O / l -> bf16, LSE
    if (ok && nt > 0) ok = wait(&o_done[t], 0);
    if (ok) {
      tc_fence_after_sync();
      const bool live = q_idx < len_q;
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      __nv_bfloat16* orow = p.out + (long long)(q_beg + q_idx) * p.ldo + h * FA_D;
#pragma unroll 1
      for (int c = 0; c < FA_D; c += 32) {
        uint32_t r[32];
        if (nt > 0) {
          tmem_ld_32x32b_x32(to + c, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
        if (live) {
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(r[8 * g + 0]) * inv, __uint_as_float(r[8 * g + 1]) * inv);
            o.y = pack_bf16x2(__uint_as_float(r[8 * g + 2]) * inv, __uint_as_float(r[8 * g + 3]) * inv);
            o.z = pack_bf16x2(__uint_as_float(r[8 * g + 4]) * inv, __uint_as_float(r[8 * g + 5]) * inv);
            o.w = pack_bf16x2(__uint_as_float(r[8 * g + 6]) * inv, __uint_as_float(r[8 * g + 7]) * inv);
            *reinterpret_cast<uint4*>(orow + c + 8 * g) = o;
          }
        }
      }
      if (live)
        p.lse[(long long)h * p.Tq + q_beg + q_idx] = l_run > 0.f ? (m_run + log2f(l_run)) * FA_LN2 : INFINITY;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace b200

// q [Tq, hq, 128], k / v [Tk, hkv, 128] bf16 with token strides ldq / ldk / ldv (elements, multiples of 8);
// out [Tq, hq, 128] with token stride ldo; lse [hq, Tq] fp32. cu_q / cu_k: int32 [B + 1] on the device.
// max_q: longest query segment (bounds the grid). Sequences need len_k >= len_q when causal.
extern "C" int b200_flash_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_q,
                              const int* cu_k, int B, int Tq, int Tk, int hq, int hkv, int d, long long ldq,
                              long long ldk, long long ldv, long long ldo, int max_q, int causal, float scale,
                              uint32_t* status, cudaStream_t stream) {
  using namespace b200;
  if (B <= 0 || Tq <= 0) return 0;
  if (d != FA_D || hkv <= 0 || hq % hkv || (ldq & 7) || (ldk & 7) || (ldv & 7) || (ldo & 7) || max_q <= 0)
    return B200_ERR_ARG;
  const long long grid = (long long)((max_q + 2 * FA_B - 1) / (2 * FA_B)) * hq * B;
  if (grid > 0x7fffffff) return B200_ERR_TOO_LARGE;
  CUtensorMap tm_q, tm_k, tm_v;
  if (make_tmap_2d(&tm_q, q, Tq, (uint64_t)hq * FA_D, ldq, FA_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_k, k, Tk, (uint64_t)hkv * FA_D, ldk, FA_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_v, v, Tk, (uint64_t)hkv * FA_D, ldv, FA_B, 64, 2)) return B200_ERR_TENSORMAP;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(flash_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FA_SMEM) != cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  FaParams p{cu_q, cu_k, (__nv_bfloat16*)out, lse, ldo, B, hq, hkv, Tq, causal, scale * FA_LOG2E, status};
  flash_fwd_kernel<<<(unsigned)grid, FA_THREADS, FA_SMEM, stream>>>(tm_q, tm_k, tm_v, p);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}
