// Varlen (packed) causal flash-attention forward on tcgen05 / TMEM / TMA for head_dim 128, GQA.
//
// CTAs take items (sequence, 256 queries, query head) one after the other, see flash_sched.cuh; an item is two tiles of 128
// queries that share every K / V tile. Calls of few tiles take the one-tile form in flash_fwd_tile.cuh. Per tile t and 128-key block j:
//     S_t  = Q_t K_j^T          tcgen05.mma M=128 (queries) N=128 (keys) K=128 (d), both operands K-major (TMA, SW128)
//     P_t  = exp2(S_t*c - m)    one thread per query row (TMEM lane) holds the whole row in registers: no shuffles, no
//                               shared memory; P goes back as bf16 over the columns of S_t
//     O_t += P_t V_j            A = P_t out of TMEM, B = V MN-major, so the [token, d] layout is used as stored
// While the softmax warps of one tile work, the tensor core runs the two products of the other. Reading P out of TMEM
// and sharing K / V between the tiles leaves 192 KB of shared-memory reads per key block for 2048 tensor-core cycles.
// The softmax chain of a tile is what bounds a long item (2400 cycles; the products of both tiles take 2048). A quarter of the
// exponentials runs on the fp32 pipe instead of the special-function unit: 3600 and 2340 tokens, 16 heads, no mask: 154 us, none
// 159, a third 153, half 171. (P handed over in halves measured nothing: 1.89 ms against 1.87 ms for one sequence of 16384
// tokens, 32 heads.) A short item is bound by what surrounds the loop, so items follow each other
// without a break: loads and the first S of the next one run under the epilogue of this one.
// O stays in TMEM for the whole item and is rescaled lazily: the running maximum only moves when it grows by more than
// 2^8, so the TMEM read-modify-write of O is rare. S_t(j+1) is issued after P_t(j) V_j by the same thread and the tensor
// core keeps that order, so "S_t(j+1) is ready" also says that P_t(j) has been read and O_t updated.
// Roles: warp 0 scheduler and TMA producer, warp 1 MMA issuer, warps 4-7 / 8-11 softmax and epilogue of tile 0 / 1. The
// first warpgroup hands registers to the other two (168 a thread at launch, then 88 and 208: 504 of 504), whose row of S
// would spill otherwise.
// Outputs O [T, hq, d] bf16 and LSE [hq, T] fp32 (natural log of the softmax denominator of the scaled scores).
// Queries are aligned to the END of the keys of their sequence (len_k >= len_q: prefill with a prefix cache,
// context-parallel chunks); with cu_q == cu_k this is ordinary causal self-attention.
// Replaces flash_attn_varlen_func (cosmos_rl/policy/kernel/modeling_utils.py:65-173). Every wait is bounded.
#include "sm100.cuh"
#include "flash_sched.cuh"
#include "gemm_core.cuh"
#include "api.h"

namespace b200 {

constexpr int FA_B = 128;                         // queries per tile / keys per block
constexpr int FA_D = 128;
constexpr int FA_TILE = FA_B * FA_D * 2;          // 32 KiB
constexpr int FA_OUT_BYTES = 8 * 4096;             // epilogue staging, 32 rows x 128 bytes a warp
constexpr int FA_SMEM = 6 * FA_TILE + FA_OUT_BYTES + 512 + 1024;   // Q x2, K x2, V x2, staging, barriers, alignment
constexpr int FA_THREADS = 384;
constexpr float FA_LOG2E = 1.4426950408889634f;
constexpr float FA_LN2 = 0.6931471805599453f;
constexpr float FA_RESCALE_TAU = 8.0f;
constexpr int FA_POLY = 4;                         // one pair of exponentials in so many runs on the fp32 pipe

struct FaParams {
  const int* cu_q;
  const int* cu_k;
  __nv_bfloat16* out;
  float* lse;
  long long ldo;      // elements between tokens of out
  int B, hq, hkv, Tq, causal;
  int levels;         // 256-query blocks of the longest sequence
  float scale_log2;
  uint32_t* status;
};

#define FA_WAIT1(bar, parity, code)           \
  if (!mbar_wait(bar, parity)) {              \
    atomicCAS(p.status, ST_OK, code);         \
    *abort_flag = 1;                          \
    break;                                    \
  }

// key blocks that some query of tile t sees
__device__ __forceinline__ int fa_key_blocks(const FlashItem& w, int t, int causal) {
  if (w.row0 + t * FA_B >= w.len_q) return 0;
  const int end = causal ? min(w.len_k, w.row0 + (t + 1) * FA_B + w.len_k - w.len_q) : w.len_k;
  return end > 0 ? (end + FA_B - 1) / FA_B : 0;
}

__global__ void __launch_bounds__(FA_THREADS, 1)
flash_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, FaParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_sh = smem;                    // [2]
  uint8_t* k_sh = smem + 2 * FA_TILE;      // [2]
  uint8_t* v_sh = smem + 4 * FA_TILE;      // [2]
  uint8_t* out_sh = smem + 6 * FA_TILE;    // [8 warps][32 rows][128 bytes]
  uint64_t* bars = reinterpret_cast<uint64_t*>(out_sh + FA_OUT_BYTES);
  uint64_t* qfull = bars;        // [2]
  uint64_t* qempty = bars + 2;   // [2]
  uint64_t* kfull = bars + 4;    // [2]
  uint64_t* kempty = bars + 6;   // [2]
  uint64_t* vfull = bars + 8;    // [2]
  uint64_t* vempty = bars + 10;  // [2]
  uint64_t* s_ready = bars + 12; // [2] per tile
  uint64_t* p_ready = bars + 14; // [2] per tile
  uint64_t* o_done = bars + 16;  // [2] per tile: the last product of the tile has finished
  uint64_t* item_full = bars + 18;   // [2] slots of the work queue
  uint64_t* item_empty = bars + 20;  // [2] read by the MMA thread and the eight softmax warps
  FlashItem* items = reinterpret_cast<FlashItem*>(bars + 22);   // [2]
  // bars + 30: 16 bytes and bars + 32: barrier of cluster launch control
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 33);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&qfull[s], 1);
      mbar_init(&qempty[s], 1);
      mbar_init(&kfull[s], 1);
      mbar_init(&kempty[s], 1);
      mbar_init(&vfull[s], 1);
      mbar_init(&vempty[s], 1);
      mbar_init(&s_ready[s], 1);
      mbar_init(&p_ready[s], 4);
      mbar_init(&o_done[s], 1);
      mbar_init(&item_full[s], 1);
      mbar_init(&item_empty[s], 9);
    }
    mbar_init(bars + 32, 1);
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

  if (warp >= 4) {
    setmaxnreg_inc<208>();
    // ------------------------------------------------ softmax + epilogue
    const int t = (warp - 4) >> 2;
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const uint32_t ts = tmem_base + t * FA_B + lane_addr, to = tmem_base + 256 + t * FA_D + lane_addr;
    uint8_t* stage = out_sh + (warp - 4) * 4096;
    const float2 c2 = make_float2(p.scale_log2, p.scale_log2);
    uint32_t ns = 0, no = 0;                        // S blocks and finished items of this tile so far
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {   // the whole warp: tcgen05.ld / st are warp-collective
      const bool w = mbar_wait(bar, parity);
      if (!w) {
        atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_FULL);
        *abort_flag = 1;
      }
      return __all_sync(0xffffffffu, w);
    };
    for (uint32_t it = 0; ok; ++it) {
      const uint32_t slot = it & 1;
      if (!(ok = wait(&item_full[slot], (it >> 1) & 1))) break;
      const FlashItem& w = items[slot];              // read where it is needed: registers are short in the loop
      if (!w.valid) break;
      const int nt = fa_key_blocks(w, t, p.causal);
      const int q_idx = w.row0 + t * FA_B + row;     // position inside the sequence's queries
      const int k_limit = p.causal ? min(w.len_k, q_idx + w.len_k - w.len_q + 1) : w.len_k;   // keys [0, k_limit) are visible
      float m_run = -INFINITY, l_run = 0.f;
      for (int j = 0; j < nt; ++j, ++ns) {
        if (!(ok = wait(&s_ready[t], ns & 1))) break;
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
              if (kbase + c * 32 + i >= k_limit) r[c][i] = 0xff800000u;   // -infinity; the scale is positive
        }
        float mx4[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          mx4[c] = fmaxf(__uint_as_float(r[c][0]), __uint_as_float(r[c][1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2) mx4[c] = max3(mx4[c], __uint_as_float(r[c][i]), __uint_as_float(r[c][i + 1]));
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
              const float2 e = i % FA_POLY == FA_POLY - 1 ? exp2_poly2(x) : make_float2(exp2_approx(x.x), exp2_approx(x.y));
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
      if (!ok) break;
      // ---- epilogue: O / l -> bf16, LSE. Rows pass through shared memory so that a warp writes whole 128-byte lines.
      if (nt > 0) {
        if (!(ok = wait(&o_done[t], no & 1))) break;
        ++no;
        tc_fence_after_sync();
      }
      const float inv = l_run > 0.f ? 1.f / l_run : 0.f;
      const int first = w.row0 + t * FA_B + quad * 32, len_q = w.len_q;   // the warp's rows
      __nv_bfloat16* dst = p.out + (long long)(w.q_beg + first) * p.ldo + w.head * FA_D;
#pragma unroll 1
      for (int c = 0; c < FA_D; c += 64) {
        uint32_t r[2][32];
        if (nt > 0) {
          tmem_ld_32x32b_x32(to + c, r[0]);
          tmem_ld_32x32b_x32(to + c + 32, r[1]);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[0][i] = r[1][i] = 0u;
        }
        __syncwarp();                                // the previous half has been read
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          const uint32_t(&v)[32] = r[g >> 2];
          const int k = (g & 3) * 8;
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(v[k + 0]) * inv, __uint_as_float(v[k + 1]) * inv);
          o.y = pack_bf16x2(__uint_as_float(v[k + 2]) * inv, __uint_as_float(v[k + 3]) * inv);
          o.z = pack_bf16x2(__uint_as_float(v[k + 4]) * inv, __uint_as_float(v[k + 5]) * inv);
          o.w = pack_bf16x2(__uint_as_float(v[k + 6]) * inv, __uint_as_float(v[k + 7]) * inv);
          *reinterpret_cast<uint4*>(stage + lane * 128 + ((g ^ (lane & 7)) << 4)) = o;
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {                // four rows a step, eight lanes each
          const int rr = 4 * i + (lane >> 3), g = lane & 7;
          const uint4 o = *reinterpret_cast<const uint4*>(stage + rr * 128 + ((g ^ (rr & 7)) << 4));
          if (first + rr < len_q) *reinterpret_cast<uint4*>(dst + rr * p.ldo + c + 8 * g) = o;
        }
      }
      tc_fence_before_sync();                        // O has been read: the next item's first product overwrites it
      if (q_idx < len_q)
        p.lse[(long long)w.head * p.Tq + w.q_beg + q_idx] = l_run > 0.f ? (m_run + log2f(l_run)) * FA_LN2 : INFINITY;
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_empty[slot]);
    }
  } else {
    setmaxnreg_dec<88>();
    if (warp == 0) {
      // ------------------------------------------------ scheduler and TMA producer (the whole warp, one elected lane issues)
      FlashWork work;
      work.list.init(p.cu_q, p.B, 2 * FA_B, p.hq, p.levels, !p.causal);
      work.init(reinterpret_cast<uint4*>(bars + 30), bars + 32);
      uint32_t kv = 0;              // key blocks so far: ring position of K and V
      uint32_t nq[2] = {0, 0};      // Q tiles so far
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        const bool w = mbar_wait(bar, parity);
        if (!w) {
          atomicCAS(p.status, ST_OK, ST_TIMEOUT_EMPTY);
          *abort_flag = 1;
        }
        return __all_sync(0xffffffffu, w);
      };
      auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row) {
        if (elect_one()) {
          mbar_arrive_expect_tx(bar, FA_TILE);
          tma_load_2d(dst, tm, bar, col, row);
          tma_load_2d(dst + FA_TILE / 2, tm, bar, col + 64, row);
        }
      };
      for (uint32_t it = 0; ok; ++it) {
        const uint32_t slot = it & 1;
        FlashItem w;
        int block = 0;
        w.head = w.b = 0;
        w.valid = work.next(w.b, block, w.head);
        if (w.valid < 0) {
          atomicCAS(p.status, ST_OK, ST_TIMEOUT_EMPTY);
          *abort_flag = 1;
          break;
        }
        w.q_beg = w.len_q = w.k_beg = w.len_k = w.row0 = 0;
        if (w.valid) {
          w.q_beg = p.cu_q[w.b];
          w.len_q = p.cu_q[w.b + 1] - w.q_beg;
          w.k_beg = p.cu_k[w.b];
          w.len_k = p.cu_k[w.b + 1] - w.k_beg;
          w.row0 = block * 2 * FA_B;
        }
        if (!(ok = wait(&item_empty[slot], ((it >> 1) & 1) ^ 1))) break;
        if (lane == 0) {
          items[slot] = w;
          mbar_arrive(&item_full[slot]);
        }
        if (!w.valid) break;
        const int n0 = fa_key_blocks(w, 0, p.causal), n1 = fa_key_blocks(w, 1, p.causal), n = max(n0, n1);
        const int hk = w.head / (p.hq / p.hkv), qrow = w.q_beg + w.row0;
        if (n0 > 0) {
          if (!(ok = wait(&qempty[0], (nq[0] & 1) ^ 1))) break;
          ++nq[0];
          load(q_sh, &tm_q, &qfull[0], w.head * FA_D, qrow);
        }
        for (int j = 0; j < n; ++j, ++kv) {
          if (j + 2 >= n) work.request();   // the answer comes while the last blocks wait for their buffers
          const uint32_t s = kv & 1, ph = ((kv >> 1) & 1) ^ 1;
          const int row = w.k_beg + j * FA_B;
          if (!(ok = wait(&kempty[s], ph))) break;
          load(k_sh + s * FA_TILE, &tm_k, &kfull[s], hk * FA_D, row);
          if (j == 0 && n1 > 0) {
            if (!(ok = wait(&qempty[1], (nq[1] & 1) ^ 1))) break;
            ++nq[1];
            load(q_sh + FA_TILE, &tm_q, &qfull[1], w.head * FA_D, qrow + FA_B);
          }
          if (!(ok = wait(&vempty[s], ph))) break;
          load(v_sh + s * FA_TILE, &tm_v, &vfull[s], hk * FA_D, row);
        }
      }
      work.finish();
      // the tensor core's last arrivals on these barriers land before the CTA's shared memory is released
      for (uint32_t i = 0; i < 2 && ok; ++i, ++kv) {
        const uint32_t s = kv & 1, ph = ((kv >> 1) & 1) ^ 1;
        ok = wait(&kempty[s], ph) && wait(&vempty[s], ph) && wait(&qempty[i], (nq[i] & 1) ^ 1);
      }
    } else if (warp == 1) {
      // ------------------------------------------------ MMA issuer
      if (elect_one()) {
        constexpr uint32_t idesc_s = umma_idesc_bf16_f32(FA_B, FA_B);
        constexpr uint32_t idesc_o = umma_idesc_bf16_f32(FA_B, FA_D) | (1u << 16);   // B (= V) is MN-major
        uint32_t kv = 0, nq[2] = {0, 0}, np[2] = {0, 0};
        auto mma_s = [&](int t, uint32_t s) {
          const uint32_t qs = smem_u32(q_sh + t * FA_TILE), ks = smem_u32(k_sh + s * FA_TILE);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const uint32_t off = (k >> 2) * (FA_TILE / 2) + (k & 3) * 32;
            umma_bf16_ss(tmem_base + t * FA_B, umma_desc_kmajor_sw128(qs + off), umma_desc_kmajor_sw128(ks + off), idesc_s,
                         k > 0 ? 1u : 0u);
          }
          tc_commit(&s_ready[t]);
        };
        auto mma_o = [&](int t, uint32_t s, bool first) {
          const uint32_t vs = smem_u32(v_sh + s * FA_TILE);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_bf16_ts(tmem_base + 256 + t * FA_D, tmem_base + t * FA_B + k * 8,
                         umma_desc_mnmajor_sw128(vs + k * 2048, FA_TILE / 2), idesc_o, (first && k == 0) ? 0u : 1u);
        };
        for (uint32_t it = 0; !*abort_flag; ++it) {
          const uint32_t slot = it & 1;
          FA_WAIT1(&item_full[slot], (it >> 1) & 1, ST_TIMEOUT_FULL)
          const FlashItem w = items[slot];
          mbar_arrive(&item_empty[slot]);
          if (!w.valid) break;
          const int n0 = fa_key_blocks(w, 0, p.causal), n1 = fa_key_blocks(w, 1, p.causal), n = max(n0, n1);
          if (n == 0) continue;
          // S of the first key block may be formed while the softmax warps still write the previous item's result: its
          // columns were last read by that item's last product, and O is not touched before P of this item is announced
          FA_WAIT1(&kfull[kv & 1], (kv >> 1) & 1, ST_TIMEOUT_FULL)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int nt = t ? n1 : n0;
            if (nt == 0) continue;
            FA_WAIT1(&qfull[t], nq[t] & 1, ST_TIMEOUT_FULL)
            ++nq[t];
            tc_fence_after_sync();
            mma_s(t, kv & 1);
            if (nt == 1) tc_commit(&qempty[t]);
          }
          if (*abort_flag) break;
          tc_commit(&kempty[kv & 1]);
          for (int j = 0; j < n && !*abort_flag; ++j, ++kv) {
            const uint32_t s = kv & 1, s1 = (kv + 1) & 1;
            FA_WAIT1(&vfull[s], (kv >> 1) & 1, ST_TIMEOUT_FULL)
            if (j + 1 < n) FA_WAIT1(&kfull[s1], ((kv + 1) >> 1) & 1, ST_TIMEOUT_FULL)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
              const int nt = t ? n1 : n0;
              if (j >= nt) continue;
              FA_WAIT1(&p_ready[t], np[t] & 1, ST_TIMEOUT_TMEM_EMPTY)
              ++np[t];
              tc_fence_after_sync();
              mma_o(t, s, j == 0);
              if (j + 1 < nt) {
                mma_s(t, s1);
                if (j + 2 == nt) tc_commit(&qempty[t]);
              } else {
                tc_commit(&o_done[t]);
              }
            }
            if (*abort_flag) break;
            tc_commit(&vempty[s]);
            if (j + 1 < n) tc_commit(&kempty[s1]);
          }
        }
      }
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

#include "flash_fwd_tile.cuh"

namespace b200 {

// One tile a CTA (flash_fwd_tile.cuh); the grid covers the longest sequence's blocks for every sequence.
template <bool POSITIVE>
static int launch_fwd_tile(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v, const FaParams& p,
                           int max_q, cudaStream_t stream) {
  auto kern = flash_fwd_tile_kernel<POSITIVE>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FT_SMEM) != cudaSuccess) return B200_ERR_LAUNCH;
    attr_set = true;
  }
  kern<<<dim3((max_q + FA_B - 1) / FA_B, p.hq, p.B), FT_THREADS, FT_SMEM, stream>>>(tm_q, tm_k, tm_v, p);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

}  // namespace b200

// q [Tq, hq, 128], k / v [Tk, hkv, 128] bf16 with token strides ldq / ldk / ldv (elements, multiples of 8);
// out [Tq, hq, 128] with token stride ldo; lse [hq, Tq] fp32. cu_q / cu_k: int32 [B + 1] on the device.
// max_q: longest query segment (bounds the grid). Sequences need len_k >= len_q when causal.
extern "C" int b200_flash_fwd(const void* q, const void* k, const void* v, void* out, float* lse, const int* cu_q,
                              const int* cu_k, int B, int Tq, int Tk, int hq, int hkv, int d, long long ldq,
                              long long ldk, long long ldv, long long ldo, int max_q, int causal, float scale,
                              uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (B <= 0 || Tq <= 0) return 0;
  if (d != FA_D || hkv <= 0 || hq % hkv || (ldq & 7) || (ldk & 7) || (ldv & 7) || (ldo & 7) || max_q <= 0)
    return B200_ERR_ARG;
  const int levels = (max_q + 2 * FA_B - 1) / (2 * FA_B);
  const long long items = flash_items(B, Tq, max_q, 2 * FA_B, hq);
  if (items > 0x7fffffff) return B200_ERR_TOO_LARGE;
  CUtensorMap tm_q, tm_k, tm_v;
  if (make_tmap_2d(&tm_q, q, Tq, (uint64_t)hq * FA_D, ldq, FA_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_k, k, Tk, (uint64_t)hkv * FA_D, ldk, FA_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_v, v, Tk, (uint64_t)hkv * FA_D, ldv, FA_B, 64, 2)) return B200_ERR_TENSORMAP;
  const FaParams p{cu_q, cu_k, (__nv_bfloat16*)out, lse, ldo, B, hq, hkv, Tq, causal, levels, scale * FA_LOG2E, status};
  // flash_fwd_kernel hides keys before the scale is applied, which takes a positive one
  if (!(scale > 0.f)) return launch_fwd_tile<false>(tm_q, tm_k, tm_v, p, max_q, stream);
  // While every tile of 128 queries has an SM of its own, the time is that of one tile's chain, and the one-tile form has the
  // shorter one: two warps a row, S of the next block under the softmax of this one, no queue before the first load. One
  // sequence of 200 tokens, 32 heads: 8.2 us, 12.0 us in the other form; 512 queries on 8192 keys, 28 heads: 100 and 126;
  // 1152 tokens, 16 heads (144 tiles): 19.7 and 23.3. Beyond one round of CTAs two tiles that share K and V win: 1300 tokens,
  // 16 heads (176 tiles): 28.4 and 27.2; 1024 tokens, 28 heads (224 tiles): 29.5 and 23.6.
  if ((long long)((max_q + FA_B - 1) / FA_B) * hq * B <= num_sms)
    return launch_fwd_tile<true>(tm_q, tm_k, tm_v, p, max_q, stream);
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(flash_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FA_SMEM) != cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  flash_fwd_kernel<<<(unsigned)items, FA_THREADS, FA_SMEM, stream>>>(tm_q, tm_k, tm_v, p);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}
