// Varlen causal flash-attention backward on tcgen05 / TMEM / TMA (head_dim 128, GQA, packed sequences).
//
// Two kernels (short sequences: one, flash_bwd_short.cuh), each owning its outputs, so nothing is accumulated through memory (no fp32 dQ buffer, no atomics, the
// same bits on every run):
//
//   dQ     one item = (sequence, 128-query block, query head); loops over the 128-key blocks it can see. CTAs take items
//          one after the other (flash_sched.cuh): loads and the first products of the next one run under the end of this
//          one.
//          S  = Q K^T          M=queries N=keys K=d        TMEM S[j&1]
//          dP = dO V^T         M=queries N=keys K=d        TMEM dP
//          dS = exp2(S c - lse) o (dP - delta)             softmax warps, bf16 into the columns of S
//          dQ += dS K          M=queries N=d K=keys        A = dS out of TMEM, B = the K tile read MN-major
//          delta = rowsum(O o dO) of its rows is formed first (O fetched under the end of the item before) and left in memory
//          for the second kernel.
//          K has three slots: a block is needed from S until dQ, and with two the load of block j + 1 starts when dQ of block
//          j - 1 is through and S of j + 1 waits for it (3600 and 2340 tokens, 16 heads, no mask: 296 us, 244 with
//          three). The result passes through the K slot that the item read last, since there is no room for staging of
//          its own. dS goes into the columns of its S, so that dP of the next block is formed as soon as this one's is in
//          registers and S two blocks ahead; the loop is then bound by the softmax warps (4096 tokens, 16 heads: 92.5 us with
//          dS over dP, 91.2).
//   dK, dV one CTA = (sequence, 128-key block, kv head); loops over the query heads of its GQA group and the
//          128-query blocks that can see the key block
//          S^T  = K Q^T        M=keys N=queries K=d        TMEM S
//          dP^T = V dO^T       M=keys N=queries K=d        TMEM dP
//          P^T, dS^T           softmax warps, bf16 into the columns of S and dP
//          dV += P^T dO        M=keys N=d K=queries        A out of TMEM, B = the dO tile read MN-major
//          dK += dS^T Q        M=keys N=d K=queries        A out of TMEM, B = the Q tile read MN-major
//
// S and dP are formed twice (7 products of 128 x 128 x 128 per tile pair instead of 5). That is the cheaper side: a
// product of two shared-memory operands reads 64 KB for 512 tensor-core cycles, which is all the 128 B per cycle that
// shared memory gives, and in the one-kernel form the transposed dS and the fp32 dQ tile go through shared memory and
// L2 as well. With P and dS taken from TMEM the five products per tile of the two accumulations need 32 KB each.
// The tensor core runs the products in the order in which the one issuing thread gives them; a product that
// overwrites the columns of an operand of the product before it (S over P or dS, dP over dS) relies on that order. In the
// dK/dV kernel the chain P, dV, S of the next block, exponentials is what is left (3100 cycles an iteration, 2048 of them
// products); S and dP changing places, with P and dS in the columns of S and the next S under dS, gave the same time.
// Roles of both: warp 0 TMA producer, warp 1 MMA issuer, warps 2..9 softmax (two per TMEM lane quadrant, 64 columns
// each). All waits are bounded; on a timeout a status code is recorded and the CTA leaves with its TMEM freed.
// Replaces flash_attn's varlen backward (cosmos_rl/policy/kernel/modeling_utils.py:65-173).
#include "sm100.cuh"
#include "flash_sched.cuh"
#include "gemm_core.cuh"
#include "api.h"

namespace b200 {

constexpr int FB_B = 128;                            // queries / keys per block
constexpr int FB_D = 128;
constexpr int FB_TILE = FB_B * FB_D * 2;             // 32 KiB, two boxes of 128 rows x 64 elements
constexpr int FB_STATS = 2 * 2 * FB_B * 4;           // dK/dV kernel: lse and delta of two query blocks
constexpr int FB_SMEM = 6 * FB_TILE + FB_STATS + 256 + 1024;          // dK/dV kernel
constexpr int FB_SMEM_DQ = 7 * FB_TILE + 512 + 2 * FB_B * 4 + 1024;   // dQ kernel: Q, dO, K x3, V x2, delta of two items
constexpr int FB_THREADS = 320;                      // TMA warp, MMA warp, 8 softmax warps
constexpr float FB_LOG2E = 1.4426950408889634f;
// One pair of exponentials in so many runs on the fp32 pipe (exp2_poly2): the two warps of a scheduler are in their exponentials
// at the same time, 1050 cycles of 1024 that the special-function unit needs for 128 x 128. us with none, a sixth, a quarter, a
// third and half of them there, 3600 and 2340 tokens, 16 heads, no mask: dQ 195, 191, 193, 193, 195; dK/dV 274, 264, 264, 266, 269.
constexpr int FB_POLY_DQ = 6, FB_POLY_KV = 4;

struct FbParams {
  const int* cu_q;
  const int* cu_k;
  const float* lse;            // [hq, Tq]
  float* delta;                // [hq, Tq]; written by the dQ kernel, read by the dK/dV kernel
  const __nv_bfloat16* out;    // [Tq, hq, d] of the forward pass
  const __nv_bfloat16* dout;
  __nv_bfloat16* dq;           // [Tq, hq, d]
  __nv_bfloat16* dk;           // [Tk, hkv, d]
  __nv_bfloat16* dv;
  long long ldo, lddo, lddq, lddk, lddv;  // token strides (elements)
  int B, hq, hkv, Tq, Tk, causal;
  int levels_q;                // 128-query blocks of the longest sequence
  float scale, scale_log2;
  uint32_t* status;
};

// Whole-warp bounded wait; on a timeout records `code`, raises the CTA's abort flag and returns false in every lane.
__device__ __forceinline__ bool fb_wait(uint64_t* bar, uint32_t parity, uint32_t code, uint32_t* status,
                                        volatile uint32_t* abort_flag) {
  const bool ok = mbar_wait(bar, parity);
  if (!ok) {
    atomicCAS(status, ST_OK, code);
    *abort_flag = 1;
  }
  return __all_sync(0xffffffffu, ok);
}

// The same for the single thread of the producer / issuer roles.
#define FB_WAIT1(bar, parity, code)           \
  if (!mbar_wait(bar, parity)) {              \
    atomicCAS(p.status, ST_OK, code);         \
    *abort_flag = 1;                          \
    break;                                    \
  }

__device__ __forceinline__ void fb_load_tile(uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row) {
  tma_load_2d(dst, tm, bar, col, row);
  tma_load_2d(dst + FB_TILE / 2, tm, bar, col + 64, row);
}

// D[128, 128] = A[128, 128] * B[128, 128]^T of two K-major shared-memory tiles
__device__ __forceinline__ void fb_mma_ss(uint32_t tmem_d, uint32_t a, uint32_t b) {
  constexpr uint32_t idesc = umma_idesc_bf16_f32(128, 128);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t off = (k >> 2) * (FB_TILE / 2) + (k & 3) * 32;
    umma_bf16_ss(tmem_d, umma_desc_kmajor_sw128(a + off), umma_desc_kmajor_sw128(b + off), idesc, k > 0 ? 1u : 0u);
  }
}

// D[128, 128] += A[128, 128] * B[128, 128] with A in TMEM (contraction elements 0..63 as bf16 pairs in columns [0, 32),
// 64..127 in columns [64, 96)) and B a shared-memory tile whose rows are the contraction index
__device__ __forceinline__ void fb_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b, bool first) {
  constexpr uint32_t idesc = umma_idesc_bf16_f32(128, 128) | (1u << 16);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    umma_bf16_ts(tmem_d, tmem_a + (k >> 2) * 64 + (k & 3) * 8, umma_desc_mnmajor_sw128(b + k * 2048, FB_TILE / 2), idesc,
                 (first && k == 0) ? 0u : 1u);
}

// 64 fp32 accumulator columns of the warp's 32 rows (+ `add`, this thread's row, one float every 128), times `mul`, as bf16
// to global memory: through 4 KB of shared memory, so that the warp writes whole 128-byte lines. `live`: rows to write.
__device__ __forceinline__ void fb_store_rows(uint32_t taddr, bool zero, float mul, uint8_t* stage, __nv_bfloat16* dst,
                                              long long ld, int live, const float* add = nullptr) {
  const int lane = threadIdx.x & 31;
  uint32_t r[2][32];
  tmem_ld_32x32b_x32(taddr, r[0]);
  tmem_ld_32x32b_x32(taddr + 32, r[1]);
  tmem_ld_wait();
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float v[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int c = 8 * g + 2 * j + u;
        v[u] = zero ? 0.f : __uint_as_float(r[c >> 5][c & 31]);
        if (add) v[u] += add[c * FB_B];
      }
      o[j] = pack_bf16x2(v[0] * mul, v[1] * mul);
    }
    *reinterpret_cast<uint4*>(stage + lane * 128 + ((g ^ (lane & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {   // four rows a step, eight lanes each
    const int rr = 4 * i + (lane >> 3), g = lane & 7;
    const uint4 o = *reinterpret_cast<const uint4*>(stage + rr * 128 + ((g ^ (rr & 7)) << 4));
    if (rr < live) *reinterpret_cast<uint4*>(dst + rr * ld + 8 * g) = o;
  }
  __syncwarp();                   // before the staging rows are written again
}

// ---------------------------------------------------------------------------------------------------------------
// dQ (and delta)
// ---------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ int fb_key_blocks(const FlashItem& w, int causal) {
  const int end = causal ? min(w.len_k, w.row0 + FB_B + w.len_k - w.len_q) : w.len_k;
  return end > 0 ? (end + FB_B - 1) / FB_B : 0;
}

__global__ void __launch_bounds__(FB_THREADS, 1)
flash_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, FbParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_sh = smem;
  uint8_t* do_sh = smem + FB_TILE;
  uint8_t* k_sh = smem + 2 * FB_TILE;                  // [3]
  uint8_t* v_sh = smem + 5 * FB_TILE;                  // [2]
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 7 * FB_TILE);
  uint64_t* q_full = bars;
  uint64_t* q_empty = bars + 1;
  uint64_t* do_full = bars + 2;
  uint64_t* do_empty = bars + 3;
  uint64_t* k_full = bars + 4;       // [3]
  uint64_t* v_full = bars + 7;       // [2]
  uint64_t* k_empty = bars + 9;      // [3]
  uint64_t* v_empty = bars + 12;     // [2]
  uint64_t* s_ready = bars + 14;     // [2]
  uint64_t* dp_ready = bars + 16;
  uint64_t* ds_ready = bars + 17;
  uint64_t* done = bars + 18;
  uint64_t* dp_free = bars + 36;     // dP has been read
  uint64_t* dlt_full = bars + 37;    // [4] delta of a quadrant's rows, from its two warps
  uint64_t* item_full = bars + 19;   // [2] slots of the work queue
  uint64_t* item_empty = bars + 21;  // [2] read by the MMA thread and the eight softmax warps
  FlashItem* items = reinterpret_cast<FlashItem*>(bars + 24);   // [2]
  // bars + 32: 16 bytes and bars + 23: barrier of cluster launch control
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 34);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* dlt_sh = reinterpret_cast<float*>(bars + 64);          // [2][128] -delta of the item's rows

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    mbar_init(q_empty, 1);
    mbar_init(do_full, 1);
    mbar_init(do_empty, 9);
    for (int s = 0; s < 3; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&s_ready[s], 1);
      mbar_init(&item_full[s], 1);
      mbar_init(&item_empty[s], 9);
    }
    for (int s = 0; s < 4; ++s) mbar_init(&dlt_full[s], 2);
    mbar_init(bars + 23, 1);
    mbar_init(dp_ready, 1);
    mbar_init(ds_ready, 8);
    mbar_init(dp_free, 8);
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // columns: S[2] (then dS) 0..255, dP 256..383, dQ 384..511
  const uint32_t tm_dp = tmem_base + 256, tm_dq = tmem_base + 384;

  if (warp == 0) {
    // ---- scheduler and TMA producer (the whole warp, one elected lane issues)
    FlashWork work;
    work.list.init(p.cu_q, p.B, FB_B, p.hq, p.levels_q, !p.causal);
    work.init(reinterpret_cast<uint4*>(bars + 32), bars + 23);
    uint32_t kv = 0, nq = 0;   // key blocks and Q tiles so far
    bool ok = true;
    auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int col, int row) {
      if (elect_one()) {
        mbar_arrive_expect_tx(bar, FB_TILE);
        fb_load_tile(dst, tm, bar, col, row);
      }
    };
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool { return fb_wait(bar, parity, ST_TIMEOUT_EMPTY, p.status, abort_flag); };
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
        w.row0 = block * FB_B;
      }
      if (!(ok = wait(&item_empty[slot], ((it >> 1) & 1) ^ 1))) break;
      if (lane == 0) {
        items[slot] = w;
        mbar_arrive(&item_full[slot]);
      }
      if (!w.valid) break;
      const int n = fb_key_blocks(w, p.causal), hk = w.head / (p.hq / p.hkv), qrow = w.q_beg + w.row0;
      for (int j = 0; j < n; ++j, ++kv) {
        if (j + 2 >= n) work.request();   // the answer comes while the last blocks wait for their buffers
        const uint32_t s = kv & 1, ph = ((kv >> 1) & 1) ^ 1, ks = kv % 3;
        const int row = w.k_beg + j * FB_B;
        if (j == 0) {
          if (!(ok = wait(q_empty, (nq & 1) ^ 1))) break;
          load(q_sh, &tm_q, q_full, w.head * FB_D, qrow);
        }
        // the third block goes where the previous item's result passes through on its way out
        if (j == 2 && it > 0 && !(ok = wait(&item_empty[slot ^ 1], ((it - 1) >> 1) & 1))) break;
        if (!(ok = wait(&k_empty[ks], (kv / 3 & 1) ^ 1))) break;
        load(k_sh + ks * FB_TILE, &tm_k, &k_full[ks], hk * FB_D, row);
        if (j == 0) {
          if (!(ok = wait(do_empty, (nq & 1) ^ 1))) break;
          load(do_sh, &tm_do, do_full, w.head * FB_D, qrow);
          ++nq;
        }
        if (!(ok = wait(&v_empty[s], ph))) break;
        load(v_sh + s * FB_TILE, &tm_v, &v_full[s], hk * FB_D, row);
      }
    }
    work.finish();
    // the tensor core's last arrivals on these barriers land before the CTA's shared memory is released
    if (ok) ok = wait(q_empty, (nq & 1) ^ 1) && wait(do_empty, (nq & 1) ^ 1);
    for (int i = 0; i < 3 && ok; ++i, ++kv)
      ok = wait(&k_empty[kv % 3], (kv / 3 & 1) ^ 1) && (i == 2 || wait(&v_empty[kv & 1], ((kv >> 1) & 1) ^ 1));
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t q_a = smem_u32(q_sh), do_a = smem_u32(do_sh);
      uint32_t kv = 0, nq = 0;
      for (uint32_t it = 0; !*abort_flag; ++it) {
        const uint32_t slot = it & 1;
        FB_WAIT1(&item_full[slot], (it >> 1) & 1, ST_TIMEOUT_FULL)
        const FlashItem w = items[slot];
        mbar_arrive(&item_empty[slot]);
        if (!w.valid) break;
        const int n = fb_key_blocks(w, p.causal);
        if (n == 0) continue;
        FB_WAIT1(q_full, nq & 1, ST_TIMEOUT_FULL)
        FB_WAIT1(&k_full[kv % 3], kv / 3 & 1, ST_TIMEOUT_FULL)
        tc_fence_after_sync();
        fb_mma_ss(tmem_base + (kv & 1) * 128, q_a, smem_u32(k_sh + kv % 3 * FB_TILE));
        tc_commit(&s_ready[kv & 1]);
        if (n == 1) tc_commit(q_empty);
        FB_WAIT1(do_full, nq & 1, ST_TIMEOUT_FULL)
        FB_WAIT1(&v_full[kv & 1], (kv >> 1) & 1, ST_TIMEOUT_FULL)
        ++nq;
        tc_fence_after_sync();
        fb_mma_ss(tm_dp, do_a, smem_u32(v_sh + (kv & 1) * FB_TILE));
        tc_commit(dp_ready);
        tc_commit(&v_empty[kv & 1]);
        if (n == 1) tc_commit(do_empty);
        if (n > 1) {
          FB_WAIT1(&k_full[(kv + 1) % 3], (kv + 1) / 3 & 1, ST_TIMEOUT_FULL)
          tc_fence_after_sync();
          fb_mma_ss(tmem_base + ((kv + 1) & 1) * 128, q_a, smem_u32(k_sh + (kv + 1) % 3 * FB_TILE));
          tc_commit(&s_ready[(kv + 1) & 1]);
          if (n == 2) tc_commit(q_empty);
        }
        for (int j = 0; j < n && !*abort_flag; ++j, ++kv) {
          const uint32_t s = kv & 1, s1 = s ^ 1, ks = kv % 3;
          if (j + 1 < n) {   // dP of the next block, once this one's is in registers
            FB_WAIT1(dp_free, kv & 1, ST_TIMEOUT_TMEM_EMPTY)
            FB_WAIT1(&v_full[s1], ((kv + 1) >> 1) & 1, ST_TIMEOUT_FULL)
            tc_fence_after_sync();
            fb_mma_ss(tm_dp, do_a, smem_u32(v_sh + s1 * FB_TILE));
            tc_commit(dp_ready);
            tc_commit(&v_empty[s1]);
            if (j + 2 == n) tc_commit(do_empty);
          }
          // dS also says that the previous item's dQ has been read, which the first product of an item overwrites
          FB_WAIT1(ds_ready, kv & 1, ST_TIMEOUT_TMEM_EMPTY)
          tc_fence_after_sync();
          fb_mma_ts(tm_dq, tmem_base + s * 128, smem_u32(k_sh + ks * FB_TILE), j == 0);
          tc_commit(&k_empty[ks]);
          if (j + 2 < n) {   // S of the block after the next, over dS of this one
            const uint32_t ks2 = (kv + 2) % 3;
            FB_WAIT1(&k_full[ks2], (kv + 2) / 3 & 1, ST_TIMEOUT_FULL)
            tc_fence_after_sync();
            fb_mma_ss(tmem_base + s * 128, q_a, smem_u32(k_sh + ks2 * FB_TILE));
            tc_commit(&s_ready[s]);
            if (j + 3 == n) tc_commit(q_empty);
          }
        }
        if (!*abort_flag) tc_commit(done);
      }
    }
  } else {
    const int quad = warp & 3;
    const int half_id = (warp - 2) >> 2;
    const int c0 = half_id * 64;                         // first key column of this warp
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const float2 c2 = make_float2(p.scale_log2, p.scale_log2);
    uint32_t kv = 0, nq = 0, finished = 0;
    bool ok = true;
    // An item's statistics: delta is rowsum(O o dO), 16 rows a warp. O (a row is one coalesced 256-byte read) and the lane's lse are
    // fetched before the result of the item before is written, dO is read from the tile that dP takes. Loads of both where the
    // sums are used, and by both warps of a quadrant, held up every item: 32 x 256 tokens, 28 heads, 92.8 us and 72.1 so (38 are
    // the bytes); 5 x 1536 tokens 147 and 133; 1 x 8192 517 and 506. (Two more warps for it: 107, 167 and 558. Their waits are
    // not free, and they had two blocks' time for 64 rows each.) Rows past the end are read at the last row and dropped: no branch
    // keeps the loads apart.
    uint2 o2[16];
    float lse = 0.f;
    bool valid = false;
    auto fetch = [&](uint32_t it) -> bool {
      if (!fb_wait(&item_full[it & 1], (it >> 1) & 1, ST_TIMEOUT_FULL, p.status, abort_flag)) return false;
      const FlashItem& w = items[it & 1];
      if (!(valid = w.valid)) return true;
      const int first = w.row0 + quad * 32 + half_id * 16, own = w.row0 + row;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const long long t = w.q_beg + min(first + i, w.len_q - 1);
        o2[i] = *reinterpret_cast<const uint2*>(p.out + t * p.ldo + w.head * FB_D + lane * 4);
      }
      lse = own < w.len_q ? p.lse[(long long)w.head * p.Tq + w.q_beg + own] : INFINITY;
      return true;
    };
    ok = fetch(0);
    for (uint32_t it = 0; ok && valid; ++it) {
      const uint32_t slot = it & 1;
      const FlashItem& w = items[slot];                  // read where it is needed: registers are short in the loop
      const int n = fb_key_blocks(w, p.causal);
      const int q_idx = w.row0 + row;
      const int k_limit = p.causal ? min(w.len_k, q_idx + w.len_k - w.len_q + 1) : w.len_k;   // keys [0, k_limit) are visible
      const float nlse = -lse * FB_LOG2E;
      // The sums of the 16 rows are reduced together (each shuffle step but the first halves the rows that a lane carries): row r
      // ends up in the lanes r and r + 16. The quadrant's two warps exchange theirs.
      float v[16];
      if (n > 0) {
        if (!(ok = fb_wait(do_full, nq & 1, ST_TIMEOUT_FULL, p.status, abort_flag))) break;
        ++nq;
      }
      // the lane's four columns: 8 of the 16 bytes of chunk (lane / 2) & 7 in the half tile lane / 16
      const uint8_t* g_row = do_sh + (lane >> 4) * (FB_TILE / 2) + (quad * 32 + half_id * 16) * 128 + (lane & 1) * 8;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const uint2 g2 = *reinterpret_cast<const uint2*>(g_row + i * 128 + ((((lane >> 1) & 7) ^ (i & 7)) << 4));
        const float2 x0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o2[i].x));
        const float2 x1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o2[i].y));
        const float2 y0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g2.x));
        const float2 y1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g2.y));
        v[i] = (x0.x * y0.x + x0.y * y0.y) + (x1.x * y1.x + x1.y * y1.y);
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 16);
#pragma unroll
      for (int d = 8; d > 0; d >>= 1) {   // lane distance d: d rows stay with each lane
        const bool hi = lane & d;
#pragma unroll
        for (int i = 0; i < d; ++i) {
          const float send = hi ? v[i] : v[i + d], keep = hi ? v[i + d] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
        }
      }
      if (lane < 16) {
        const int r = quad * 32 + half_id * 16 + lane;
        if (w.row0 + r < w.len_q && n > 0) p.delta[(long long)w.head * p.Tq + w.q_beg + w.row0 + r] = v[0];
        dlt_sh[slot * FB_B + r] = -v[0];   // two items' worth: a warp that has got to the next item's has read this one's
      }
      __syncwarp();
      if (lane == 0) {
        if (n > 0) mbar_arrive(do_empty);
        mbar_arrive(&dlt_full[quad]);
      }
      if (!(ok = fb_wait(&dlt_full[quad], it & 1, ST_TIMEOUT_FULL, p.status, abort_flag))) break;
      const float nd = dlt_sh[slot * FB_B + row];
      const float2 nl2 = make_float2(nlse, nlse), nd2 = make_float2(nd, nd);
      for (int j = 0; j < n; ++j, ++kv) {
        const uint32_t s = kv & 1;
        if (!(ok = fb_wait(&s_ready[s], (kv >> 1) & 1, ST_TIMEOUT_TMEM_FULL, p.status, abort_flag))) break;
        tc_fence_after_sync();
        float2 e[32];
        const int key0 = j * FB_B + c0;
        uint32_t rs[2][32];
        tmem_ld_32x32b_x32(tmem_base + s * 128 + lane_addr + c0, rs[0]);
        tmem_ld_32x32b_x32(tmem_base + s * 128 + lane_addr + c0 + 32, rs[1]);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t(&r)[32] = rs[i >> 4];
          const float2 x = fma2(make_float2(__uint_as_float(r[2 * (i & 15)]), __uint_as_float(r[2 * (i & 15) + 1])), c2, nl2);
          e[i] = i % FB_POLY_DQ == FB_POLY_DQ - 1 ? exp2_poly2(x) : make_float2(exp2_approx(x.x), exp2_approx(x.y));
        }
        if (key0 + 64 > k_limit) {
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (key0 + 2 * i >= k_limit) e[i].x = 0.f;
            if (key0 + 2 * i + 1 >= k_limit) e[i].y = 0.f;
          }
        }
        if (!(ok = fb_wait(dp_ready, kv & 1, ST_TIMEOUT_TMEM_FULL, p.status, abort_flag))) break;
        tc_fence_after_sync();
        uint32_t ds[32], rp[2][32];
        tmem_ld_32x32b_x32(tm_dp + lane_addr + c0, rp[0]);
        tmem_ld_32x32b_x32(tm_dp + lane_addr + c0 + 32, rp[1]);
        tmem_ld_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(dp_free);
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const uint32_t(&r)[32] = rp[i >> 4];
          const float2 v = mul2(e[i], add2(make_float2(__uint_as_float(r[2 * (i & 15)]), __uint_as_float(r[2 * (i & 15) + 1])), nd2));
          ds[i] = pack_bf16x2(v.x, v.y);
        }
        tmem_st_32x32b_x32(tmem_base + s * 128 + lane_addr + c0, ds);   // over the first half of this warp's columns of S
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(ds_ready);
      }
      if (!ok || !(ok = fetch(it + 1))) break;
      if (n > 0) {
        if (!(ok = fb_wait(done, finished & 1, ST_TIMEOUT_TMEM_FULL, p.status, abort_flag))) break;
        ++finished;
        tc_fence_after_sync();
      }
      // the rows leave through the K slot of the item's last block, or of the one before it if it has none
      uint8_t* stage = k_sh + (kv + 2) % 3 * FB_TILE + (warp - 2) * 4096;
      const int first = w.row0 + quad * 32;
      fb_store_rows(tm_dq + lane_addr + c0, n == 0, p.scale, stage,
                    p.dq + (long long)(w.q_beg + first) * p.lddq + w.head * FB_D + c0, p.lddq, w.len_q - first);
      fence_proxy_async_smem();                          // a TMA load overwrites the staging rows
      tc_fence_before_sync();                            // dQ has been read: the next item's first product overwrites it
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_empty[slot]);
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 100; ++i) __nanosleep(1000);     // copies already issued land before shared memory is released
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// rows [0, head) and [tail, T) of a gradient [T, heads, d], by the whole grid
__device__ __forceinline__ void fb_clear_outside(__nv_bfloat16* g, long long ld, int heads, int head, int tail, int T) {
  const int vec = heads * (FB_D / 4), outside = head + max(T - tail, 0);
  for (long long i = (long long)blockIdx.x * FB_THREADS + threadIdx.x; i < (long long)outside * vec;
       i += (long long)gridDim.x * FB_THREADS) {
    const int e = (int)(i % vec), k = (int)(i / vec);
    *reinterpret_cast<uint2*>(g + (long long)(k < head ? k : tail + k - head) * ld + e * 4) = make_uint2(0u, 0u);
  }
}
// tokens outside every sequence have no gradient; in a kernel all of whose CTAs run
__device__ __forceinline__ void fb_clear_all_outside(const FbParams& p) {
  const int q0 = p.cu_q[0], q1 = p.cu_q[p.B], k0 = p.cu_k[0], k1 = p.cu_k[p.B];
  if (q0 > 0 || q1 < p.Tq) fb_clear_outside(p.dq, p.lddq, p.hq, q0, q1, p.Tq);
  if (k0 > 0 || k1 < p.Tk) {
    fb_clear_outside(p.dk, p.lddk, p.hkv, k0, k1, p.Tk);
    fb_clear_outside(p.dv, p.lddv, p.hkv, k0, k1, p.Tk);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// dK, dV. SPLIT = 2: a cluster of two CTAs shares a key block, each taking half of its (head, query block) iterations; at
// the end they exchange partial sums through distributed shared memory, the first CTA finishing dK and the second dV.
// ---------------------------------------------------------------------------------------------------------------
template <int SPLIT>
__global__ void __launch_bounds__(FB_THREADS, 1)
flash_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                      const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, FbParams p) {
  const int heads = p.hkv * p.B;
  const int block = blockIdx.x / SPLIT, rank = SPLIT == 2 ? (int)cluster_ctarank() : 0;
  const int hb = block % heads, hk = hb % p.hkv, b = hb / p.hkv;
  const int kv0 = block / heads * FB_B;                 // early key blocks are seen by most queries: first
  const int q_beg = p.cu_q[b], len_q = p.cu_q[b + 1] - q_beg;
  const int k_beg = p.cu_k[b], len_k = p.cu_k[b + 1] - k_beg;
  fb_clear_all_outside(p);
  if (kv0 >= len_k) return;
  const int shift = len_k - len_q;
  const int G = p.hq / p.hkv;
  const int nqb = (len_q + FB_B - 1) / FB_B;
  int qb_first = 0;
  if (p.causal && kv0 - shift > 0) qb_first = (kv0 - shift) / FB_B;
  const int per_head = nqb > qb_first ? nqb - qb_first : 0;
  const int n_all = per_head * G, n_first = SPLIT == 2 ? (n_all + 1) / 2 : n_all;
  const int i_beg = rank ? n_first : 0, n = rank ? n_all - n_first : n_first;   // this CTA's iterations i_beg + [0, n)

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* k_sh = smem;
  uint8_t* v_sh = smem + FB_TILE;
  uint8_t* q_sh = smem + 2 * FB_TILE;                   // [2]
  uint8_t* do_sh = smem + 4 * FB_TILE;                  // [2]
  float* lse_sh = reinterpret_cast<float*>(smem + 6 * FB_TILE);   // [2][128] -lse * log2(e)
  float* dlt_sh = lse_sh + 2 * FB_B;                              // [2][128] -delta
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * FB_TILE + FB_STATS);
  uint64_t* k_full = bars;
  uint64_t* v_full = bars + 1;
  uint64_t* q_full = bars + 2;     // [2] Q tile and the statistics of its rows
  uint64_t* do_full = bars + 4;    // [2]
  uint64_t* q_empty = bars + 6;    // [2]
  uint64_t* do_empty = bars + 8;   // [2]
  uint64_t* st_empty = bars + 10;  // [2] statistics read by the softmax warps
  uint64_t* s_ready = bars + 12;
  uint64_t* dp_ready = bars + 13;
  uint64_t* p_ready = bars + 14;
  uint64_t* ds_ready = bars + 15;
  uint64_t* done = bars + 16;
  uint64_t* st_full = bars + 17;   // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 19);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&do_full[s], 1);
      mbar_init(&q_empty[s], 1);
      mbar_init(&do_empty[s], 1);
      mbar_init(&st_empty[s], 8);
      mbar_init(&st_full[s], 1);
    }
    mbar_init(s_ready, 1);
    mbar_init(dp_ready, 1);
    mbar_init(p_ready, 8);
    mbar_init(ds_ready, 8);
    mbar_init(done, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
    tma_prefetch_desc(&tm_do);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  // columns: S (then P) 0..127, dP (then dS) 128..255, dV 256..383, dK 384..511
  const uint32_t tm_s = tmem_base, tm_dp = tmem_base + 128, tm_dv = tmem_base + 256, tm_dk = tmem_base + 384;

  bool ok = true;
  if (warp == 0) {
    // the whole warp: one elected lane issues the tile loads, all lanes fetch the 128 rows' lse and delta with plain loads
    // (their addresses have no 16-byte alignment, so they cannot be a bulk copy)
    for (int i = 0; i < n && !*abort_flag; ++i) {
      const int s = i & 1;
      const uint32_t ph = ((i >> 1) & 1) ^ 1;
      const int h = hk * G + (i_beg + i) / per_head, qr = (qb_first + (i_beg + i) % per_head) * FB_B;
      float ls[4], dl[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int qi = qr + lane + 32 * j;
        const long long at = (long long)h * p.Tq + q_beg + qi;
        ls[j] = qi < len_q ? -p.lse[at] * FB_LOG2E : -INFINITY;
        dl[j] = qi < len_q ? -p.delta[at] : 0.f;
      }
      if (!fb_wait(&q_empty[s], ph, ST_TIMEOUT_EMPTY, p.status, abort_flag)) break;
      if (elect_one()) {
        if (i == 0) {
          mbar_arrive_expect_tx(k_full, FB_TILE);
          fb_load_tile(k_sh, &tm_k, k_full, hk * FB_D, k_beg + kv0);
        }
        mbar_arrive_expect_tx(&q_full[s], FB_TILE);
        fb_load_tile(q_sh + s * FB_TILE, &tm_q, &q_full[s], h * FB_D, q_beg + qr);
        if (i == 0) {
          mbar_arrive_expect_tx(v_full, FB_TILE);
          fb_load_tile(v_sh, &tm_v, v_full, hk * FB_D, k_beg + kv0);
        }
      }
      if (!fb_wait(&do_empty[s], ph, ST_TIMEOUT_EMPTY, p.status, abort_flag)) break;
      if (elect_one()) {
        mbar_arrive_expect_tx(&do_full[s], FB_TILE);
        fb_load_tile(do_sh + s * FB_TILE, &tm_do, &do_full[s], h * FB_D, q_beg + qr);
      }
      if (!fb_wait(&st_empty[s], ph, ST_TIMEOUT_EMPTY, p.status, abort_flag)) break;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        lse_sh[s * FB_B + lane + 32 * j] = ls[j];
        dlt_sh[s * FB_B + lane + 32 * j] = dl[j];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&st_full[s]);
    }
  } else if (warp == 1) {
    if (n > 0 && elect_one()) {
      const uint32_t k_a = smem_u32(k_sh), v_a = smem_u32(v_sh);
      do {
        FB_WAIT1(k_full, 0, ST_TIMEOUT_FULL)
        FB_WAIT1(&q_full[0], 0, ST_TIMEOUT_FULL)
        tc_fence_after_sync();
        fb_mma_ss(tm_s, k_a, smem_u32(q_sh));
        tc_commit(s_ready);
        FB_WAIT1(v_full, 0, ST_TIMEOUT_FULL)
        FB_WAIT1(&do_full[0], 0, ST_TIMEOUT_FULL)
        tc_fence_after_sync();
        fb_mma_ss(tm_dp, v_a, smem_u32(do_sh));
        tc_commit(dp_ready);
        for (int i = 0; i < n && !*abort_flag; ++i) {
          const int s = i & 1, s1 = s ^ 1;
          const uint32_t ph1 = ((i + 1) >> 1) & 1;
          FB_WAIT1(p_ready, i & 1, ST_TIMEOUT_TMEM_EMPTY)
          tc_fence_after_sync();
          fb_mma_ts(tm_dv, tm_s, smem_u32(do_sh + s * FB_TILE), i == 0);      // dV += P^T dO
          tc_commit(&do_empty[s]);
          if (i + 1 < n) {
            FB_WAIT1(&q_full[s1], ph1, ST_TIMEOUT_FULL)
            tc_fence_after_sync();
            fb_mma_ss(tm_s, k_a, smem_u32(q_sh + s1 * FB_TILE));              // S^T of the next block, over P^T
            tc_commit(s_ready);
          }
          FB_WAIT1(ds_ready, i & 1, ST_TIMEOUT_TMEM_EMPTY)
          tc_fence_after_sync();
          fb_mma_ts(tm_dk, tm_dp, smem_u32(q_sh + s * FB_TILE), i == 0);      // dK += dS^T Q
          tc_commit(&q_empty[s]);
          if (i + 1 < n) {
            FB_WAIT1(&do_full[s1], ph1, ST_TIMEOUT_FULL)
            tc_fence_after_sync();
            fb_mma_ss(tm_dp, v_a, smem_u32(do_sh + s1 * FB_TILE));            // dP^T of the next block, over dS^T
            tc_commit(dp_ready);
          }
        }
        if (!*abort_flag) tc_commit(done);
      } while (false);
    }
  } else {
    // TMEM lanes are keys, columns are queries: the statistics belong to columns. In the fragment layout a thread has 16
    // columns of four rows (quadrant rows lane / 4 + 0, 8, 16, 24), so it reads 16 + 16 statistics an iteration; with one
    // row a thread it would be 64 + 64, and those broadcasts took a third of the shared-memory bandwidth.
    const int quad = warp & 3;
    const int c0 = ((warp - 2) >> 2) * 64;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const int key0 = kv0 + quad * 32 + (lane >> 2);          // this thread's keys: key0 + 8 r, r = 0..3
    const int col = c0 + 2 * (lane & 3);                     // its columns: col + 8 g + {0, 1}, g = 0..7
    const float2 c2 = make_float2(p.scale_log2, p.scale_log2);
    for (int i = 0; i < n; ++i) {
      const int s = i & 1;
      const int q0 = (qb_first + (i_beg + i) % per_head) * FB_B;   // first query of the block
      if (!(ok = fb_wait(&st_full[s], (i >> 1) & 1, ST_TIMEOUT_FULL, p.status, abort_flag))) break;
      float2 nl[8];
#pragma unroll
      for (int g = 0; g < 8; ++g) nl[g] = *reinterpret_cast<const float2*>(lse_sh + s * FB_B + col + 8 * g);
      if (!(ok = fb_wait(s_ready, i & 1, ST_TIMEOUT_TMEM_FULL, p.status, abort_flag))) break;
      tc_fence_after_sync();
      float2 e[4][8];                                        // [row][column group]
      uint32_t rs[2][32];                                    // TMEM lanes 0..15 and 16..31 of the quadrant
      tmem_ld_16x256b_x8(tm_s + lane_addr + c0, rs[0]);
      tmem_ld_16x256b_x8(tm_s + lane_addr + (16u << 16) + c0, rs[1]);
      tmem_ld_wait();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const uint32_t(&r)[32] = rs[hf];
#pragma unroll
        for (int g = 0; g < 8; ++g)
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float2 x = fma2(make_float2(__uint_as_float(r[4 * g + 2 * u]), __uint_as_float(r[4 * g + 2 * u + 1])), c2, nl[g]);
            e[2 * hf + u][g] = (2 * g + u) % FB_POLY_KV == FB_POLY_KV - 1 ? exp2_poly2(x)
                                                                          : make_float2(exp2_approx(x.x), exp2_approx(x.y));
          }
      }
      // a query sees a key iff q >= key - shift (causal); queries past the end have no probabilities
      if ((p.causal && q0 + c0 < kv0 + quad * 32 + 31 - shift) || q0 + c0 + 64 > len_q) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int q_min = p.causal ? key0 + 8 * r - shift : -(1 << 30);
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const int q = q0 + col + 8 * g;
            if (q < q_min || q >= len_q) e[r][g].x = 0.f;
            if (q + 1 < q_min || q + 1 >= len_q) e[r][g].y = 0.f;
          }
        }
      }
      // both halves of the quadrant's rows have been read before any column is overwritten
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t pk[16];
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          pk[2 * g] = pack_bf16x2(e[2 * hf][g].x, e[2 * hf][g].y);
          pk[2 * g + 1] = pack_bf16x2(e[2 * hf + 1][g].x, e[2 * hf + 1][g].y);
        }
        tmem_st_16x128b_x8(tm_s + lane_addr + ((uint32_t)(16 * hf) << 16) + c0, pk);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready);
      float2 nd[8];
#pragma unroll
      for (int g = 0; g < 8; ++g) nd[g] = *reinterpret_cast<const float2*>(dlt_sh + s * FB_B + col + 8 * g);
      if (!(ok = fb_wait(dp_ready, i & 1, ST_TIMEOUT_TMEM_FULL, p.status, abort_flag))) break;
      tc_fence_after_sync();
      uint32_t ds[2][16], rp[2][32];
      tmem_ld_16x256b_x8(tm_dp + lane_addr + c0, rp[0]);
      tmem_ld_16x256b_x8(tm_dp + lane_addr + (16u << 16) + c0, rp[1]);
      tmem_ld_wait();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const uint32_t(&r)[32] = rp[hf];
#pragma unroll
        for (int g = 0; g < 8; ++g)
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const float2 v = mul2(e[2 * hf + u][g],
                                  add2(make_float2(__uint_as_float(r[4 * g + 2 * u]), __uint_as_float(r[4 * g + 2 * u + 1])), nd[g]));
            ds[hf][2 * g + u] = pack_bf16x2(v.x, v.y);
          }
      }
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) tmem_st_16x128b_x8(tm_dp + lane_addr + ((uint32_t)(16 * hf) << 16) + c0, ds[hf]);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&st_empty[s]);
        mbar_arrive(ds_ready);
      }
    }
    if (ok && n > 0) ok = fb_wait(done, 0, ST_TIMEOUT_TMEM_FULL, p.status, abort_flag);
    tc_fence_after_sync();
  }

  // ---- results of the key block; after a failed wait nothing is written
  const int quad = warp & 3, c0 = ((warp - 2) >> 2) * 64, row = quad * 32 + lane;
  const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
  __nv_bfloat16* dk_dst = p.dk + (long long)(k_beg + kv0 + quad * 32) * p.lddk + hk * FB_D + c0;
  __nv_bfloat16* dv_dst = p.dv + (long long)(k_beg + kv0 + quad * 32) * p.lddv + hk * FB_D + c0;
  uint8_t* stage = do_sh + (warp - 2) * 4096;   // the dO tiles are no longer read
  const int live = len_k - (kv0 + quad * 32);
  if constexpr (SPLIT == 2) {
    // The Q tiles' 64 KB receive the peer's partial sums as [column][row]. Both CTAs' loops have ended before either
    // writes, and every thread takes part in the cluster barriers whatever happened before.
    __syncwarp();
    cluster_sync_all();
    if (warp >= 2 && ok) {
      const uint32_t dst = mapa_shared(smem_u32(q_sh), rank ^ 1) + ((uint32_t)c0 * FB_B + row) * 4;
#pragma unroll 1
      for (int c = 0; c < 64; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x32((rank ? tm_dk : tm_dv) + lane_addr + c0 + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) st_shared_cluster(dst + (uint32_t)(c + j) * FB_B * 4, n > 0 ? __uint_as_float(r[j]) : 0.f);
      }
    }
    __syncwarp();
    cluster_sync_all();
    if (warp >= 2 && ok) {
      const float* add = reinterpret_cast<const float*>(q_sh) + c0 * FB_B + row;
      if (rank == 0) fb_store_rows(tm_dk + lane_addr + c0, n == 0, p.scale, stage, dk_dst, p.lddk, live, add);
      else fb_store_rows(tm_dv + lane_addr + c0, n == 0, 1.f, stage, dv_dst, p.lddv, live, add);
    }
  } else if (warp >= 2 && ok) {
    fb_store_rows(tm_dk + lane_addr + c0, n == 0, p.scale, stage, dk_dst, p.lddk, live);
    fb_store_rows(tm_dv + lane_addr + c0, n == 0, 1.f, stage, dv_dst, p.lddv, live);
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

#include "flash_bwd_short.cuh"

namespace b200 {

static int launch_bwd_short(const void* q, const void* k, const void* v, const FbParams& p, long long ldq, long long ldk,
                            long long ldv, cudaStream_t stream) {
  CUtensorMap tm_q, tm_k, tm_v, tm_do;
  if (make_tmap_2d(&tm_q, q, p.Tq, (uint64_t)p.hq * FB_D, ldq, FS_BQ, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_k, k, p.Tk, (uint64_t)p.hkv * FB_D, ldk, FB_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_v, v, p.Tk, (uint64_t)p.hkv * FB_D, ldv, FB_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_do, p.dout, p.Tq, (uint64_t)p.hq * FB_D, p.lddo, FS_BQ, 64, 2)) return B200_ERR_TENSORMAP;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(flash_bwd_short_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FS_SMEM) != cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  flash_bwd_short_kernel<<<(unsigned)(p.B * p.hkv), FB_THREADS, FS_SMEM, stream>>>(tm_q, tm_k, tm_v, tm_do, p);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

}  // namespace b200

// Gradients of b200_flash_fwd: dq [Tq, hq, 128], dk / dv [Tk, hkv, 128] bf16 are overwritten (rows outside every sequence
// are zeroed); delta [hq, Tq] fp32 is scratch. max_q / max_k bound the grids.
extern "C" int b200_flash_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout,
                              const float* lse, void* dq, void* dk, void* dv, float* delta, const int* cu_q,
                              const int* cu_k, int B, int Tq, int Tk, int hq, int hkv, int d, long long ldq,
                              long long ldk, long long ldv, long long ldo, long long lddo, long long lddq,
                              long long lddk, long long lddv, int max_q, int max_k, int causal, float scale,
                              uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (B <= 0 || Tq <= 0 || Tk <= 0) {   // nothing attends to anything
    auto clear = [&](void* g, long long ld, int rows, int heads) {
      return rows <= 0 || heads <= 0 ||
             cudaMemset2DAsync(g, (size_t)ld * 2, 0, (size_t)heads * FB_D * 2, (size_t)rows, stream) == cudaSuccess;
    };
    if (d != FB_D) return B200_ERR_ARG;
    return clear(dq, lddq, Tq, hq) && clear(dk, lddk, Tk, hkv) && clear(dv, lddv, Tk, hkv) ? 0 : B200_ERR_RUNTIME;
  }
  if (d != FB_D || hkv <= 0 || hq % hkv || (ldq & 7) || (ldk & 7) || (ldv & 7) || (ldo & 3) || (lddo & 7) ||
      (lddq & 7) || (lddk & 7) || (lddv & 7) || max_q <= 0 || max_k <= 0 || ((uintptr_t)out & 7) || ((uintptr_t)dq & 15) ||
      ((uintptr_t)dk & 15) || ((uintptr_t)dv & 15))
    return B200_ERR_ARG;
  const int levels_q = (max_q + FB_B - 1) / FB_B;
  const long long items_q = flash_items(B, Tq, max_q, FB_B, hq), grid_k = (long long)((max_k + FB_B - 1) / FB_B) * hkv * B;
  if (grid_k > 0x7fffffff || items_q > 0x7fffffff) return B200_ERR_TOO_LARGE;
  const FbParams p{cu_q, cu_k, lse, delta, (const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, (__nv_bfloat16*)dq,
                   (__nv_bfloat16*)dk, (__nv_bfloat16*)dv, ldo, lddo, lddq, lddk, lddv, B, hq, hkv, Tq, Tk, causal, levels_q,
                   scale, scale * FB_LOG2E, status};
  // One kernel over short sequences: it has half the prologues of the two below, which is what such calls cost, but walks
  // the G query heads of a kv head one after the other. 256 sequences of 20 tokens, 28 / 4 heads: 241 us, with the two 407;
  // one of 64 tokens, 16 / 16 heads: 10.6 and 18.4. For one or two heads a group always; for more once two fifths of the SMs
  // have a CTA (16 x 20 tokens, 28 / 4 heads: 33.6 and 40.2; 8 x 20: 33.4 and 31.3). More than 64 queries are two iterations
  // a head, which pays for one head only (8 x 128 tokens, 16 / 16 heads: 15.7 and 28.9; 32 x 128, 4 / 2 heads: 25.5 and 19.8).
  const int G = hq / hkv;
  if (max_k <= FB_B && (max_q <= FS_BQ ? G <= 2 || 5LL * B * hkv >= 2LL * num_sms : max_q <= FB_B && G == 1))
    return launch_bwd_short(q, k, v, p, ldq, ldk, ldv, stream);
  CUtensorMap tm_q, tm_k, tm_v, tm_do;
  if (make_tmap_2d(&tm_q, q, Tq, (uint64_t)hq * FB_D, ldq, FB_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_k, k, Tk, (uint64_t)hkv * FB_D, ldk, FB_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_v, v, Tk, (uint64_t)hkv * FB_D, ldv, FB_B, 64, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tm_do, dout, Tq, (uint64_t)hq * FB_D, lddo, FB_B, 64, 2)) return B200_ERR_TENSORMAP;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(flash_bwd_dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FB_SMEM_DQ) != cudaSuccess ||
        cudaFuncSetAttribute(flash_bwd_dkdv_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, FB_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(flash_bwd_dkdv_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, FB_SMEM) != cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  flash_bwd_dq_kernel<<<(unsigned)items_q, FB_THREADS, FB_SMEM_DQ, stream>>>(tm_q, tm_k, tm_v, tm_do, p);
  // Few key blocks leave SMs idle behind the one with the most queries: share each between two CTAs while there are fewer
  // than three per SM. (Seven packed sequences of 640 to 1536 tokens, 28 / 4 heads: 336 blocks, the longest 84 iterations
  // against 69 per SM on average.) A CTA costs about six iterations before and after its loop, so blocks of few iterations
  // are shared only where the longest alone takes longer than all of them with that cost twice: 8 x 600 tokens, 4 / 2 heads
  // (80 blocks of 2 to 10) 35.9 us, not shared 41.0; 8 x 129 tokens, 16 / 16 heads (256 of 1 and 2) 54.4 and 34.5; 64 x 129,
  // 4 / 2 heads 70.0 and 52.4.
  const long long longest = (long long)G * ((max_q + FB_B - 1) / FB_B);   // iterations of a block that every query sees
  const long long mean2 = causal ? longest + G : 2 * longest;             // twice the mean
  if (grid_k < 3LL * num_sms && (longest >= 12 || 2 * (6 + longest) * num_sms > grid_k * (24 + mean2))) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * grid_k));
    cfg.blockDim = dim3(FB_THREADS);
    cfg.dynamicSmemBytes = FB_SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, flash_bwd_dkdv_kernel<2>, tm_q, tm_k, tm_v, tm_do, p) != cudaSuccess) return B200_ERR_LAUNCH;
  } else {
    flash_bwd_dkdv_kernel<1><<<(unsigned)grid_k, FB_THREADS, FB_SMEM, stream>>>(tm_q, tm_k, tm_v, tm_do, p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}
