// Block-scaled fp8 (e4m3) GEMM on tcgen05:  C[M,N] = sum_kb  sa[m, kb] * sb[n / 128, kb] * (A_kb * B_kb^T)
// with A [M,K] e4m3 + one fp32 scale per 1 x 128 block (activations), B [N,K] e4m3 + one fp32 scale per
// 128 x 128 block (weights), fp32 accumulation, bf16 output. This is the scaling scheme of the reference's
// DeepSeek-style fp8 path (cosmos_rl/policy/kernel/moe/moe.py block-scaled grouped GEMM,
// cosmos_rl/utils/fp8/fp8_util.py:21-153 for dense layers).
//
// The tensor core cannot apply a different fp32 scale per 128-wide slice of K inside one accumulation, so the
// kernels accumulate in two levels: each 128-deep k-block (kind::f8f6f4 products of K = 32) goes into a TMEM buffer with
// accumulate = 0; eight promotion warps read the finished buffer, multiply by the block's scale product and add into fp32
// registers while the tensor core fills the other buffers. Two forms, the same sums in the same order:
//   one CTA, 128 x 128 tiles: four buffers, six 32 KB stages, two warps a TMEM lane quadrant with 64 columns each
//   CTA pair, 256 x 256 tiles: half the operand bytes of a product from L2 and shared memory; each CTA has two buffers of
//   its 128 rows x 256 columns, handed over by halves of 128 columns
// What bounds them, 4096 x 37888 x 3584 on pairs: 32 tiles of 28 k-blocks a pair, 896 k-blocks of 512 cycles of products; 458 752
// of the 624 000 cycles of a call the tensor pipe is busy. A k-block takes 634 cycles, 524 in a form that hands the buffers over
// and scales nothing, 541 with its TMEM loads alone and 550 with its products alone; a tile's end takes the promotion warps 1700
// more (the next tile's place and scales 535, bf16 into the slabs 600), of which the two k-blocks ahead hide part. Fewer cycles
// buy less than their share of time, for the clock falls under such calls: 777 000 cycles at 1.57 GHz became 624 000 at 1.41, ten
// calls after a pause 494 us and then 440, 544 and 488 in a loop of a second; products without hand-over are 372 and 410.
// What counted before, ten calls at a time: a form that waits for its scales, writes rows from registers and issues from one
// thread 845 us; scales multiplied when they are used 667; results through TMA stores and two issuers 613; loads in flight under
// the multiplications 539; CTA pairs 488 to 506. One issuer with 256-column products 490, one that takes the halves in turn 467,
// the next tile's scales fetched inside the loop 449: slower than 440.
// Operands arrive by TMA (128-byte swizzle, a 128-byte row = 128 fp8 elements). Persistent CTAs, bounded waits.
#include "gemm_core.cuh"
#include "gemm_2cta_launch.cuh"
#include "api.h"

namespace b200 {

constexpr int F8_BM = 128, F8_BN = 128, F8_BK = 128;
constexpr int F8_STAGES = 6;
constexpr int F8_BUFS = 4;                                   // TMEM accumulators of 128 columns: all 512
constexpr int F8_STAGE_BYTES = (F8_BM + F8_BN) * F8_BK;     // 32 KiB
constexpr int F8_OUT_BYTES = 8 * 4096;                       // one slab of 32 rows x 128 bytes a promotion warp
constexpr int F8_SMEM = F8_STAGES * F8_STAGE_BYTES + F8_OUT_BYTES + 256 + 1024;
constexpr int F8_THREADS = 384;                              // TMA warp, two MMA warps, an idle one, 8 promotion warps

struct F8Params {
  const float* sa;       // [M, ldsa]  (ldsa >= ceil(K / 128))
  const float* sb;       // [ceil(N / 128), ldsb]
  __nv_bfloat16* C;
  long long ldc;
  int M, N, K, ldsa, ldsb;
  int a_rows;            // rows of A in a box
  bool vec_scales;       // rows of both scale arrays start on 16-byte boundaries
  uint32_t* status;
};

// Scale products of one result row and one column block of 128. Those of four k-blocks are fetched four k-blocks ahead (a
// round trip to L2 is longer than one k-block) and multiplied when they are taken: a product right behind the loads waits
// for them at once, 500 cycles every four k-blocks. Rows of scales that are 16-byte aligned are read four at a time.
struct F8Scales {
  const float* a;
  const float* b;
  int num_kb;
  bool vec;
  float na[4], nb[4];
  __device__ __forceinline__ void fetch(int kb) {
    if (vec && kb + 4 <= num_kb) {
      const float4 va = *reinterpret_cast<const float4*>(a + kb), vb = *reinterpret_cast<const float4*>(b + kb);
      na[0] = va.x; na[1] = va.y; na[2] = va.z; na[3] = va.w;
      nb[0] = vb.x; nb[1] = vb.y; nb[2] = vb.z; nb[3] = vb.w;
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        na[u] = kb + u < num_kb ? a[kb + u] : 0.f;
        nb[u] = kb + u < num_kb ? b[kb + u] : 0.f;
      }
    }
  }
  // row and column block are clamped: those outside the matrix get some scale, and their results are not stored
  __device__ __forceinline__ void init(const F8Params& p, int row, int col) {
    num_kb = (p.K + F8_BK - 1) / F8_BK;
    a = p.sa + (long long)min(row, p.M - 1) * p.ldsa;
    b = p.sb + (long long)(min(col, p.N - 1) / F8_BN) * p.ldsb;
    vec = p.vec_scales;
    fetch(0);
  }
  __device__ __forceinline__ void next(int kb, float (&cur)[4]) {
#pragma unroll
    for (int u = 0; u < 4; ++u) cur[u] = na[u] * nb[u];
    fetch(kb + 4);
  }
};

// One warp's share of a tile: acc = sum over the k-blocks of scale x accumulator; `it` counts the k-blocks of all tiles.
// taddr(it): first column of the accumulator; wait / ready(it): it is complete; release(it): it has been read. The barrier of
// the next k-block is asked before the answer is needed.
// 64 columns (single CTAs): 32 at a time, the next 32 on their way out of TMEM while the present ones are multiplied. A warp
// that does one after the other takes 400 cycles a k-block.
template <class Addr, class Wait, class Ready, class Release>
__device__ __forceinline__ bool f8_promote64(float2 (&acc)[32], F8Scales& sc, uint32_t& it, Addr taddr, Wait wait, Ready ready,
                                             Release release) {
#pragma unroll
  for (int c = 0; c < 32; ++c) acc[c] = make_float2(0.f, 0.f);
  const int num_kb = sc.num_kb;
  uint32_t r[2][32];
  if (!wait(it)) return false;
  tc_fence_after_sync();
  tmem_ld_32x32b_x32(taddr(it), r[0]);
  float cur[4];
#pragma unroll 1
  for (int kb = 0; kb < num_kb; ++kb) {
    if ((kb & 3) == 0) sc.next(kb, cur);
    const float2 s = make_float2(cur[0], cur[0]);
    cur[0] = cur[1];
    cur[1] = cur[2];
    cur[2] = cur[3];
    const bool more = kb + 1 < num_kb;
    bool rdy = false;
    auto multiply = [&](float2* to, const uint32_t (&v)[32]) {
#pragma unroll
      for (int j = 0; j < 16; ++j) to[j] = fma2(s, make_float2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1])), to[j]);
    };
    tmem_ld_wait(r[0]);
    tmem_ld_32x32b_x32(taddr(it) + 32, r[1]);
    if (more) rdy = ready(it + 1);
    multiply(acc, r[0]);
    tmem_ld_wait(r[1]);
    tc_fence_before_sync();
    __syncwarp();
    release(it);
    rdy = __all_sync(0xffffffffu, rdy);
    if (rdy) {
      tc_fence_after_sync();
      tmem_ld_32x32b_x32(taddr(it + 1), r[0]);
    }
    multiply(acc + 16, r[1]);
    ++it;
    if (more && !rdy) {
      if (!wait(it)) return false;
      tc_fence_after_sync();
      tmem_ld_32x32b_x32(taddr(it), r[0]);
    }
  }
  return true;
}

// 128 columns (CTA pairs): 64 are read out of TMEM and waited for at once, and each 32 registers are loaded again as soon as
// they have been multiplied. By 32 columns as above a k-block meets four waits instead of two: 494 us, not 440, for
// 4096 x 37888 x 3584. (64 columns at once in single CTAs leave nothing to overlap: 102 us, not 97, for 1500 x 4096 x 14336.)
template <class Addr, class Wait, class Ready, class Release>
__device__ __forceinline__ bool f8_promote128(float2 (&acc)[64], F8Scales& sc, uint32_t& it, Addr taddr, Wait wait, Ready ready,
                                              Release release) {
#pragma unroll
  for (int c = 0; c < 64; ++c) acc[c] = make_float2(0.f, 0.f);
  const int num_kb = sc.num_kb;
  uint32_t r[2][32];
  auto load = [&](uint32_t t) {
    tmem_ld_32x32b_x32(t, r[0]);
    tmem_ld_32x32b_x32(t + 32, r[1]);
  };
  if (!wait(it)) return false;
  tc_fence_after_sync();
  load(taddr(it));
  float cur[4];
#pragma unroll 1
  for (int kb = 0; kb < num_kb; ++kb) {
    if ((kb & 3) == 0) sc.next(kb, cur);
    const float2 s = make_float2(cur[0], cur[0]);
    cur[0] = cur[1];
    cur[1] = cur[2];
    cur[2] = cur[3];
    const bool more = kb + 1 < num_kb;
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
      tmem_ld_wait(r[0]);
      tmem_ld_wait(r[1]);
      if (c + 2 == 4) {
        tc_fence_before_sync();
        __syncwarp();
        release(it);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          acc[16 * (c + h) + j] =
              fma2(s, make_float2(__uint_as_float(r[h][2 * j]), __uint_as_float(r[h][2 * j + 1])), acc[16 * (c + h) + j]);
        if (c + 2 < 4) tmem_ld_32x32b_x32(taddr(it) + (c + 2 + h) * 32, r[h]);
      }
    }
    bool rdy = more && ready(it + 1);
    rdy = __all_sync(0xffffffffu, rdy);
    if (rdy) {
      tc_fence_after_sync();
      load(taddr(it + 1));
    }
    ++it;
    if (more && !rdy) {
      if (!wait(it)) return false;
      tc_fence_after_sync();
      load(taddr(it));
    }
  }
  return true;
}

// 64 columns of 32 result rows, a row a thread, as bf16 into a slab of 32 rows x 128 bytes for a TMA store
__device__ __forceinline__ void f8_fill_slab(uint8_t* slab, const float2* acc) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int j = 0; j < 8; ++j)   // 128-byte swizzle: 16-byte chunk j of row r sits at chunk j ^ (r & 7)
    *reinterpret_cast<uint4*>(slab + lane * 128 + (((uint32_t)j ^ (lane & 7)) << 4)) =
        make_uint4(pack_bf16x2(acc[4 * j].x, acc[4 * j].y), pack_bf16x2(acc[4 * j + 1].x, acc[4 * j + 1].y),
                   pack_bf16x2(acc[4 * j + 2].x, acc[4 * j + 2].y), pack_bf16x2(acc[4 * j + 3].x, acc[4 * j + 3].y));
}

__global__ void __launch_bounds__(F8_THREADS, 1)
gemm_fp8_block_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmC, F8Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_sh = smem + F8_STAGES * F8_STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(out_sh + F8_OUT_BYTES);
  uint64_t* empty_bar = full_bar + F8_STAGES;
  uint64_t* pfull = empty_bar + F8_STAGES;    // [BUFS] partial accumulator ready
  uint64_t* pempty = pfull + F8_BUFS;         // [BUFS] partial accumulator consumed (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pempty + F8_BUFS);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < F8_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < F8_BUFS; ++a) {
      mbar_init(&pfull[a], 1);
      mbar_init(&pempty[a], 8);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, F8_BUFS * F8_BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int num_m = (p.M + F8_BM - 1) / F8_BM, num_n = (p.N + F8_BN - 1) / F8_BN;
  const int total = num_m * num_n;
  const int num_kb = (p.K + F8_BK - 1) / F8_BK;
  auto tile_of = [&](int i, int& m_blk, int& n_blk) {
    constexpr int G = 8;
    const int group = i / (G * num_n), first_m = group * G;
    const int gsz = min(num_m - first_m, G);
    const int r = i - group * G * num_n;
    m_blk = first_m + r % gsz;
    n_blk = r / gsz;
  };

  if (warp < 4) setmaxnreg_dec<40>();
  else setmaxnreg_inc<232>();
  if (warp == 0) {
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      for (int i = blockIdx.x; i < total && !*abort_flag; i += gridDim.x) {
        int m_blk, n_blk;
        tile_of(i, m_blk, n_blk);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_EMPTY); *abort_flag = 1; break; }
          uint8_t* sa = smem + stage * F8_STAGE_BYTES;
          mbar_arrive_expect_tx(&full_bar[stage], p.a_rows * F8_BK + F8_BN * F8_BK);
          tma_load_2d(sa, &tmA, &full_bar[stage], kb * F8_BK, m_blk * F8_BM);
          tma_load_2d(sa + F8_BM * F8_BK, &tmB, &full_bar[stage], kb * F8_BK, n_blk * F8_BN);
          if (++stage == F8_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp < 3) {
    // two issuers, a k-block each in turn: the buffers are independent, and the waits, products and commits of a k-block
    // take one thread 555 cycles, the products 256
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_e4m3_f32(F8_BM, F8_BN);
      uint32_t it = 0;
      bool ok = true;
      for (int i = blockIdx.x; i < total && ok && !*abort_flag; i += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          if ((it & 1) != warp - 1) continue;
          const uint32_t buf = it % F8_BUFS, bph = (it / F8_BUFS) & 1, stage = it % F8_STAGES, phase = (it / F8_STAGES) & 1;
          if (!mbar_wait(&pempty[buf], bph ^ 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_EMPTY); *abort_flag = 1; ok = false; break; }
          if (!mbar_wait(&full_bar[stage], phase)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_FULL); *abort_flag = 1; ok = false; break; }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * F8_STAGE_BYTES), sb = sa + F8_BM * F8_BK;
#pragma unroll
          for (int k = 0; k < F8_BK / 32; ++k)
            umma_f8_ss(tmem_base + buf * F8_BN, umma_desc_kmajor_sw128(sa + k * 32), umma_desc_kmajor_sw128(sb + k * 32),
                       idesc, k > 0 ? 1u : 0u);
          tc_commit(&empty_bar[stage]);
          tc_commit(&pfull[buf]);
        }
      }
    }
  } else if (warp >= 4) {
    // promotion warps: quadrant = warp % 4 (TMEM lanes), column half = (warp - 4) / 4
    const int quad = warp & 3, chalf = (warp - 4) >> 2;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    uint8_t* slab = out_sh + (warp - 4) * 4096;
    auto wait = [&](uint32_t it) -> bool {
      const bool w = mbar_wait(&pfull[it % F8_BUFS], (it / F8_BUFS) & 1);
      if (!w) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_FULL); *abort_flag = 1; }
      return __all_sync(0xffffffffu, w);
    };
    auto ready = [&](uint32_t it) -> bool { return mbar_try_wait(&pfull[it % F8_BUFS], (it / F8_BUFS) & 1); };
    auto release = [&](uint32_t it) { if (elect_one()) mbar_arrive(&pempty[it % F8_BUFS]); };
    auto taddr = [&](uint32_t it) -> uint32_t { return tmem_base + it % F8_BUFS * F8_BN + lane_addr + chalf * 64; };
    uint32_t it = 0;
    int m_blk = 0, n_blk = 0;
    F8Scales sc;
    if ((int)blockIdx.x < total) {
      tile_of(blockIdx.x, m_blk, n_blk);
      sc.init(p, m_blk * F8_BM + quad * 32 + lane, n_blk * F8_BN);
    }
    for (int i = blockIdx.x; i < total; i += gridDim.x) {
      float2 acc[32];
      if (!f8_promote64(acc, sc, it, taddr, wait, ready, release)) break;
      const int row0 = m_blk * F8_BM + quad * 32, col0 = n_blk * F8_BN + chalf * 64;
      if (i + (int)gridDim.x < total) {   // the next tile's first scales come under the stores
        tile_of(i + gridDim.x, m_blk, n_blk);
        sc.init(p, m_blk * F8_BM + quad * 32 + lane, n_blk * F8_BN);
      }
      // Rows leave through shared memory and a TMA store, which clips what lies outside C. (A row a thread with 16-byte
      // stores took 4300 cycles a tile, eight k-blocks' time.)
      if (elect_one()) tma_store_wait_read<0>();   // the store of the tile before has read the slab
      __syncwarp();
      f8_fill_slab(slab, acc);
      if ((p.N & 7) && row0 + lane < p.M) store_tail(p.C + (long long)(row0 + lane) * p.ldc, slab, col0, p.N, false);
      fence_proxy_async_smem();
      __syncwarp();
      if (elect_one()) {
        if (row0 < p.M && col0 < whole16(p.N, 0)) tma_store_2d(&tmC, slab, col0, row0);
        tma_store_commit();
      }
    }
    if (elect_one()) tma_store_wait<0>();
  }

  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, F8_BUFS * F8_BN);
  }
}

// ---------------------------------------------------------------------------------------------------------------
// CTA pairs on 256 x 256 tiles
// ---------------------------------------------------------------------------------------------------------------
constexpr int FP_BN = 256;                                     // tile columns; each CTA holds 128 rows of A and 128 of B
constexpr int FP_STAGES = 5;
constexpr int FP_OUT_BYTES = 8 * 2 * 4096;                     // 8 promotion warps x 2 slabs of 32 rows x 128 bytes
constexpr int FP_SMEM = FP_STAGES * F8_STAGE_BYTES + FP_OUT_BYTES + 256 + 1024;
constexpr int FP_THREADS = 384;                                // TMA warp, two MMA warps, an idle one, 8 promotion warps

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FP_THREADS, 1)
gemm_fp8_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, F8Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* out_sh = smem + FP_STAGES * F8_STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(out_sh + FP_OUT_BYTES);   // the leader's is the one in use
  uint64_t* empty_bar = full_bar + FP_STAGES;
  uint64_t* pfull = empty_bar + FP_STAGES;    // [2 buffers][2 halves] partial accumulator ready
  uint64_t* pempty = pfull + 4;               // the leader's: consumed by the half's promotion warps, four of each CTA
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pempty + 4);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < FP_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 2);   // both issuers
    }
    for (int a = 0; a < 4; ++a) {
      mbar_init(&pfull[a], 1);
      mbar_init(&pempty[a], 8);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    tma_prefetch_desc(&tmC);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers exist before anything arrives on them from the other side
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int num_m = (p.M + 2 * F8_BM - 1) / (2 * F8_BM), num_n = (p.N + FP_BN - 1) / FP_BN;
  const int total = num_m * num_n;
  const int num_kb = (p.K + F8_BK - 1) / F8_BK;
  const int pair0 = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  auto tile_of = [&](int i, int& m_blk, int& n_blk) {   // groups of 8 row blocks sweep all columns: A and B panels stay in L2
    constexpr int G = 8;
    const int group = i / (G * num_n), first_m = group * G;
    const int gsz = min(num_m - first_m, G);
    const int r = i - group * G * num_n;
    m_blk = first_m + r % gsz;
    n_blk = r / gsz;
  };

  if (warp >= 4) {
    setmaxnreg_inc<232>();
    // promotion warps: quadrant = warp % 4 (TMEM lanes), 128 columns = one scale block of B each
    const int quad = warp & 3, chalf = (warp - 4) >> 2;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const uint32_t pempty_leader = mapa_shared(smem_u32(pempty + chalf), 0);
    uint8_t* slab = out_sh + (warp - 4) * 8192;
    auto wait = [&](uint32_t it) -> bool {
      const bool w = mbar_wait(&pfull[2 * (it & 1) + chalf], (it >> 1) & 1);
      if (!w) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_FULL); *abort_flag = 1; }
      return __all_sync(0xffffffffu, w);
    };
    auto ready = [&](uint32_t it) -> bool { return mbar_try_wait(&pfull[2 * (it & 1) + chalf], (it >> 1) & 1); };
    auto release = [&](uint32_t it) { if (elect_one()) mbar_arrive_cluster(pempty_leader + (it & 1) * 16); };
    auto taddr = [&](uint32_t it) -> uint32_t { return tmem_base + (it & 1) * FP_BN + lane_addr + chalf * F8_BN; };
    const int row_in = (int)cta_rank * F8_BM + quad * 32, col_in = chalf * F8_BN;   // this warp's part of a tile
    uint32_t it = 0;
    int m_blk = 0, n_blk = 0;
    F8Scales sc;
    if (pair0 < total) {
      tile_of(pair0, m_blk, n_blk);
      sc.init(p, m_blk * 2 * F8_BM + row_in + lane, n_blk * FP_BN + col_in);
    }
    for (int i = pair0; i < total; i += pairs) {
      float2 acc[64];
      if (!f8_promote128(acc, sc, it, taddr, wait, ready, release)) break;
      const int row0 = m_blk * 2 * F8_BM + row_in, col0 = n_blk * FP_BN + col_in;
      if (i + pairs < total) {   // the next tile's first scales come under the stores
        tile_of(i + pairs, m_blk, n_blk);
        sc.init(p, m_blk * 2 * F8_BM + row_in + lane, n_blk * FP_BN + col_in);
      }
      // results: two slabs of 64 columns, handed to TMA stores, which clip rows and columns outside C
      if (elect_one()) tma_store_wait_read<0>();   // the stores of the tile before have read the slabs
      __syncwarp();
      f8_fill_slab(slab, acc);
      f8_fill_slab(slab + 4096, acc + 32);
      if ((p.N & 7) && row0 + lane < p.M) {
        store_tail(p.C + (long long)(row0 + lane) * p.ldc, slab, col0, p.N, false);
        store_tail(p.C + (long long)(row0 + lane) * p.ldc, slab + 4096, col0 + 64, p.N, false);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (elect_one()) {
        if (row0 < p.M) {
          if (col0 < whole16(p.N, 0)) tma_store_2d(&tmC, slab, col0, row0);
          if (col0 + 64 < whole16(p.N, 0)) tma_store_2d(&tmC, slab + 4096, col0 + 64, row0);
        }
        tma_store_commit();
      }
    }
    if (elect_one()) tma_store_wait<0>();
  } else {
    setmaxnreg_dec<40>();
    if (warp == 0) {
      if (elect_one()) {
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (int i = pair0; i < total && ok && !*abort_flag; i += pairs) {
          int m_blk, n_blk;
          tile_of(i, m_blk, n_blk);
          // each CTA feeds 64 rows of B to either half of the columns
          const int a_row = m_blk * 2 * F8_BM + (int)cta_rank * F8_BM, b_row = n_blk * FP_BN + (int)cta_rank * (F8_BN / 2);
          for (int kb = 0; kb < num_kb; ++kb) {
            if (!mbar_wait(&empty_bar[stage], phase ^ 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_EMPTY); *abort_flag = 1; ok = false; break; }
            uint8_t* sa = smem + stage * F8_STAGE_BYTES;
            if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * F8_STAGE_BYTES);
            const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), 0);
            tma_load_2d_pair(sa, &tmA, bar, kb * F8_BK, a_row);
            tma_load_2d_pair(sa + F8_BM * F8_BK, &tmB, bar, kb * F8_BK, b_row);
            tma_load_2d_pair(sa + (F8_BM + F8_BN / 2) * F8_BK, &tmB, bar, kb * F8_BK, b_row + F8_BN);
            if (++stage == FP_STAGES) { stage = 0; phase ^= 1; }
          }
        }
        // the leader's commits arrive on this CTA's barriers until its last product has finished: they land before it exits
        for (int s = 0; s < FP_STAGES && ok && !*abort_flag; ++s) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_EMPTY); *abort_flag = 1; break; }
          if (++stage == FP_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    } else if (warp < 3 && leader) {
      // one issuer for each half of the columns
      if (elect_one()) {
        constexpr uint32_t idesc = umma_idesc_e4m3_f32(2 * F8_BM, F8_BN);
        const uint32_t h = warp - 1;
        uint32_t stage = 0, phase = 0, it = 0;
        bool ok = true;
        for (int i = pair0; i < total && ok && !*abort_flag; i += pairs) {
          for (int kb = 0; kb < num_kb; ++kb, ++it) {
            const uint32_t buf = it & 1, bph = (it >> 1) & 1;
            if (!mbar_wait(&pempty[2 * buf + h], bph ^ 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_EMPTY); *abort_flag = 1; ok = false; break; }
            if (!mbar_wait(&full_bar[stage], phase)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_FULL); *abort_flag = 1; ok = false; break; }
            tc_fence_after_sync();
            const uint32_t sa = smem_u32(smem + stage * F8_STAGE_BYTES), sb = sa + (F8_BM + h * (F8_BN / 2)) * F8_BK;
#pragma unroll
            for (int k = 0; k < F8_BK / 32; ++k)
              umma_f8_ss_pair(tmem_base + buf * FP_BN + h * F8_BN, umma_desc_kmajor_sw128(sa + k * 32),
                              umma_desc_kmajor_sw128(sb + k * 32), idesc, k > 0 ? 1u : 0u);
            tc_commit_pair(&pfull[2 * buf + h], 3);
            tc_commit_pair(&empty_bar[stage], 3);
            if (++stage == FP_STAGES) { stage = 0; phase ^= 1; }
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
  cluster_sync_all();   // neither CTA frees TMEM or exits while the other may still signal it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

static long long f8_tiles(int M, int N, int rows, int cols) { return (long long)((M + rows - 1) / rows) * ((N + cols - 1) / cols); }

// CTA pairs of a call, 0: single CTAs, or an error code. Rounds of tiles decide: a pair does at most twice the work of a single
// CTA in its round, which takes 1.5 to 1.7 times as long, up to 1.9 times with K = 512; the line lies at 1.8, where no K loses.
// us, pairs and single CTAs (a cold L2): 8192^3 406 and 507, 1000 x 28672 x 4096 106 and 123, 129 x 37888 x 3584 42 and 49;
// 300 x 28672 x 4096 66 and 60; below the line 640 x 28672 (5 rounds and 8) 81 and 84 with K = 4096, 24.6 and 23.5 with 512. Half
// of a pair would stand idle up to 128 rows.
static int f8_pairs(int M, int N, int num_sms) {
  if (num_sms < 2 || M <= F8_BM) return 0;
  static int whole[16] = {0};
  int np = 0;
  if (const int rc = resident_pairs(gemm_fp8_pair_kernel, whole, FP_SMEM, FP_THREADS, num_sms, np)) return rc;
  auto rounds = [](long long tiles, int at_once) { return (tiles + at_once - 1) / at_once; };
  const long long pair_tiles = f8_tiles(M, N, 2 * F8_BM, FP_BN);
  if (9 * rounds(pair_tiles, np) > 5 * rounds(f8_tiles(M, N, F8_BM, F8_BN), num_sms)) return 0;
  return pair_tiles < np ? (int)pair_tiles : np;
}

}  // namespace b200

// A [M,K] e4m3 (row stride lda bytes = elements), sa [M, ldsa] fp32; B [N,K] e4m3, sb [ceil(N/128), ldsb] fp32;
// C [M,N] bf16, 16-byte aligned. K, lda, ldb multiples of 16; ldc multiple of 8.
extern "C" int b200_gemm_fp8_block(const void* A, const float* sa, const void* B, const float* sb, void* C, int M,
                                   int N, int K, long long lda, long long ldb, long long ldc, int ldsa, int ldsb,
                                   uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0 || (lda & 15) || (ldb & 15) || (ldc & 7) || (K & 15)) return B200_ERR_ARG;
  const int nkb = (K + F8_BK - 1) / F8_BK;
  if (ldsa < nkb || ldsb < nkb) return B200_ERR_ARG;
  // Boxes of A have the rows there are: a row of a box that lies outside the tensor takes longer than one that is fetched.
  // One row x 28672 x 4096: 25.3 us, 36.1 with a box of 128; 8 x 6144 x 4096: 11.4 and 15.0.
  const int a_rows = M < F8_BM ? M : F8_BM;
  CUtensorMap tmA, tmB, tmC;
  if (make_tmap_2d(&tmA, A, M, K, lda, a_rows, F8_BK, 1)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tmB, B, N, K, ldb, F8_BN, F8_BK, 1)) return B200_ERR_TENSORMAP;
  if (make_tmap_out(&tmC, C, M, N < 8 ? 8 : whole16(N, 0), ldc, 0)) return B200_ERR_TENSORMAP;
  const bool vec_scales = !((ldsa | ldsb) & 3) && !(((uintptr_t)sa | (uintptr_t)sb) & 15);
  const F8Params p{sa, sb, (__nv_bfloat16*)C, ldc, M, N, K, ldsa, ldsb, a_rows, vec_scales, status};
  const int np = f8_pairs(M, N, num_sms);
  if (np < 0) return np;
  if (np > 0) {
    if (make_tmap_2d(&tmB, B, N, K, ldb, F8_BN / 2, F8_BK, 1)) return B200_ERR_TENSORMAP;
    gemm_fp8_pair_kernel<<<2 * np, FP_THREADS, FP_SMEM, stream>>>(tmA, tmB, tmC, p);
    return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
  }
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_fp8_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F8_SMEM) != cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  const long long tiles = f8_tiles(M, N, F8_BM, F8_BN);
  const int grid = tiles < num_sms ? (int)tiles : num_sms;
  gemm_fp8_block_kernel<<<grid, F8_THREADS, F8_SMEM, stream>>>(tmA, tmB, tmC, p);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

// Whether such a call takes CTA pairs.
extern "C" int b200_gemm_fp8_block_pairs(int M, int N, int num_sms) { return b200::f8_pairs(M, N, num_sms) > 0; }
