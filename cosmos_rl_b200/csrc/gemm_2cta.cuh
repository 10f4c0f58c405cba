// Dense bf16 GEMM main loop for CTA pairs (tcgen05 cta_group::2) on sm_100a.
//
//   D[M, N] = A[M, K] * B[N, K]^T      (fp32 accumulate; operands K-major or MN-major)
//
// Two CTAs of a cluster work on one 256 x BN output tile. Each CTA streams ITS half of the operands (128 rows
// of A, BN/2 rows of B) into its own shared-memory ring with plain TMA loads (no cluster multicast), the leader
// CTA issues one tcgen05.mma (M = 256) per 16 contraction elements that reads both CTAs' shared memory, and
// each CTA keeps the fp32 accumulator of its own 128 rows in its own TMEM (two accumulators, so the epilogue
// of tile i overlaps the main loop of tile i + 1). Compared with one CTA per 128 x BN tile this halves the
// shared-memory traffic for B, which is what bounds the single-CTA kernel.
//
// Epilogue: the four epilogue warps of each CTA read their TMEM lane quadrant with tcgen05.ld, convert, write
// 32-row x 128-byte slabs into swizzled staging buffers and hand them to TMA stores (or TMA reduce-adds when
// the result is accumulated into C). TMA clips rows and columns outside C; the columns of a last, incomplete 16 bytes of C's rows
// are left to the threads (store_tail).
//
// Last round. Tiles rarely fill their last round of CTA pairs, and calls of few rows have fewer tiles than pairs. If at most
// half of the pairs would have a tile in that round, its tiles come first, each cut along the contraction into as many equal
// shares as there are pairs for. Shares go to a workspace as fp32 and are added by a small kernel behind this one, in the order
// of the contraction. The pairs of one share index walk the same blocks of A and B at the same time; shares of any size, which
// would fill every pair, do not, and read the operands from HBM again and again (1003 x 4096 x 28672: 167 us uncut, 247). A
// sum by the warp that arrives last, instead of a kernel, reads the shares one after the other (100 x 4096 x 14336: 91 us
// uncut, 42 with it, 34).
//
// Barriers (per CTA unless stated): full[s] (leader's is the one in use; loads of both CTAs complete on it),
// empty[s] (the leader's tcgen05.commit arrives on both CTAs'), tfull[a] (same), tempty[a] (leader's; the 8
// epilogue warps of the pair arrive on it). Every wait is bounded; on a timeout the kernel records a status
// code, lets the copies in flight land, frees its TMEM and returns.
#pragma once
#include "gemm_core.cuh"

namespace b200 {

constexpr int G2_BM_CTA = 128;  // accumulator rows per CTA
constexpr int G2_BM = 256;      // rows of the pair's tile
constexpr int G2_BK = 64;
constexpr int G2_THREADS = 192;

enum { G2_EPI_STORE = 0, G2_EPI_SWIGLU = 1, G2_EPI_DLOGITS = 2, G2_EPI_EXPERTS = 3, G2_EPI_LOGPROB = 4, G2_EPI_GATE_UP = 5,
       G2_EPI_DGATE_UP = 6, G2_EPI_GROUPED = 7, G2_EPI_GROUPED_GATE_UP = 8 };

// Epilogue warps of a CTA: two a TMEM lane quadrant where the epilogue computes (8192 x 18944 x 3584, backward: 1084
// us with one, 911)
__host__ __device__ constexpr int g2_epilogue_warps(int epi) {
  return epi == G2_EPI_GATE_UP || epi == G2_EPI_DGATE_UP || epi == G2_EPI_GROUPED_GATE_UP ? 8 : 4;
}
__host__ __device__ constexpr int g2_threads(int epi) { return 64 + 32 * g2_epilogue_warps(epi); }

template <int BN, int STAGES, int EPI = G2_EPI_STORE>
struct Gemm2Smem {
  static constexpr int A_BYTES = G2_BM_CTA * G2_BK * 2;
  static constexpr int B_BYTES = (BN / 2) * G2_BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGING_BYTES = g2_epilogue_warps(EPI) * 2 * 4096;  // 2 slabs of 32 rows x 128 bytes a warp
  static constexpr int BAR_BYTES = 256;
  static constexpr int TOTAL = STAGES * STAGE_BYTES + STAGING_BYTES + BAR_BYTES + 1024;
};

// G2_EPI_DLOGITS: the accumulator is a tile of logits (before the temperature) and the result is their gradient, see
// dlogit_of. Arrays of one value a row; g_ent and ent may be null.
struct DlogitsParams {
  const long long* labels;
  const float* lse;
  const float* g_lp;
  const float* g_ent;
  const float* ent;
  int v0;             // vocabulary index of column 0
  float inv_temp;
};

// Gradient of g_lp * logprob + g_ent * entropy with respect to one logit (a = the product before the temperature), without
// the label's own term.
struct DlogitsRow {
  float lse, glp, gent, ent;
  long long label;
  __device__ __forceinline__ void load(const DlogitsParams& p, long long r) {
    lse = p.lse[r];
    glp = p.g_lp[r];
    gent = p.g_ent ? p.g_ent[r] : 0.f;
    ent = p.ent ? p.ent[r] : 0.f;
    label = p.labels[r];
    if (label < 0) glp = 0.f;
  }
  __device__ __forceinline__ float of(float a, float inv_temp, bool is_label) const {
    const float x = a * inv_temp;
    const float pr = __expf(x - lse);
    float g = -glp * pr - gent * pr * (x - lse + ent);
    if (is_label) g += glp;
    return g * inv_temp;
  }
};

// G2_EPI_LOGPROB: the accumulator is a tile of logits (before the temperature), of which only four sums a row remain.
struct LogprobParams {
  const long long* labels;
  float* partial;     // [T, nsplit, 4]
  int T, V, nsplit;
  float scale_log2;   // inv_temperature * log2(e): logits are tracked in the log2 domain
};

// One row's running maximum, sum of exponentials, label logit and sum of exponential * logit over the tiles of a unit.
struct LogprobRow {
  float m, l, z, e;
  long long label;
  __device__ __forceinline__ void begin(const LogprobParams& p, long long r) {
    m = -INFINITY; l = 0.f; z = -INFINITY; e = 0.f;
    label = r < p.T ? p.labels[r] : -1;
  }
  __device__ __forceinline__ void chunk(const LogprobParams& p, int c, const float (&v)[32]) {   // columns [c, c + 32)
    if (c >= p.V) return;
    float x[32];
    float cmax = -INFINITY;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      x[i] = (c + i < p.V) ? v[i] * p.scale_log2 : -INFINITY;
      cmax = fmaxf(cmax, x[i]);
    }
    const float nm = fmaxf(m, cmax);
    const float corr = exp2f(m - nm);  // m = -inf on the first chunk -> 0
    float sl = 0.f, se = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      float pexp = exp2f(x[i] - nm);
      sl += pexp;
      se += (c + i < p.V) ? pexp * x[i] : 0.f;
    }
    l = l * corr + sl;
    e = e * corr + se;
    m = nm;
    const long long off = label - c;
    if (off >= 0 && off < 32) {
#pragma unroll
      for (int i = 0; i < 32; ++i)
        if (i == (int)off) z = x[i];
    }
  }
  __device__ __forceinline__ void store(const LogprobParams& p, long long r, int split) const {
    if (r < p.T) *reinterpret_cast<float4*>(p.partial + (r * p.nsplit + split) * 4) = make_float4(m, l, z, e);
  }
};

struct Gemm2Params {
  const void* bias;  // [N] added to every row (nullable); bf16 when bias_bf16 else fp32
  int bias_bf16;
  int out_fp32;      // element type of C (the C tensor map must agree)
  int accumulate;    // C += result (TMA reduce-add)
  int up_row0;       // G2_EPI_SWIGLU: first row of the "up" half inside B (= intermediate size)
  int group_m;       // raster: tiles of this many 256-row blocks share their B columns in time
  int a_bytes;       // bytes of A that the leader fetches a stage: all its 128 rows, or those there are
  int rest, splits;  // tiles 0 .. rest - 1 are cut into `splits` shares along the contraction (see "Last round"), 0: none
  float* ws;         // shares, [pairs][256][BN]
  void* C;           // the result and its row stride, for what the tensor map leaves out
  long long ldc;
  DlogitsParams dl;  // G2_EPI_DLOGITS
  // G2_EPI_EXPERTS: C is [experts, M, N], and expert e contracts over rows [offsets[e], offsets[e + 1]) of A and B (multiples
  // of 64; both MN-major), or over the blocks of 64 that its first filled[e] rows reach into (nullable)
  // G2_EPI_GROUPED, _GROUPED_GATE_UP: rows [offsets[e], offsets[e + 1]) of A and C belong to B[e] (multiples of 32)
  const int* offsets;
  const int* filled;
  int experts;
  LogprobParams lg;  // G2_EPI_LOGPROB
};

// tile index -> (m_blk, n_blk): groups of `G` row blocks sweep all column blocks before the next group starts, so
// the tiles in flight at any time reuse a bounded set of A and B panels out of L2.
__device__ __forceinline__ void g2_tile_coords(int i, int num_m, int num_n, int G, int& m_blk, int& n_blk) {
  const int group_size = G * num_n;
  const int group = i / group_size;
  const int first_m = group * G;
  const int gsz = min(num_m - first_m, G);
  const int r = i - group * group_size;
  m_blk = first_m + r % gsz;
  n_blk = r / gsz;
}

// What a pair works on, one unit after the other: its share of a cut tile, then whole tiles.
struct G2Unit {
  int m_blk, n_blk, batch, kb0, kb1;
  int row, row_end;   // G2_EPI_GROUPED: first row of the tile, end of the expert's
  bool cut;
};
struct G2Work {
  int pair, pairs, rest, splits, num_m, num_n, G, total, num_kb;
  __device__ __forceinline__ void init(const Gemm2Params& ep, bool may_cut, int num_m_, int num_n_, int num_kb_) {
    pair = blockIdx.x >> 1;
    pairs = gridDim.x >> 1;
    rest = may_cut ? ep.rest : 0;
    splits = ep.splits;
    num_m = num_m_;
    num_n = num_n_;
    G = ep.group_m > 0 ? ep.group_m : 8;
    total = num_m * num_n;
    num_kb = num_kb_;
  }
  __device__ __forceinline__ bool get(int it, G2Unit& u) const {
    u.cut = false;
    u.batch = 0;
    u.kb0 = 0;
    u.kb1 = num_kb;
    if (pair < rest * splits) {
      if (it == 0) {
        const int s = pair / rest;   // share s of tile t belongs to pair s * rest + t
        g2_tile_coords(pair - s * rest, num_m, num_n, G, u.m_blk, u.n_blk);
        u.cut = true;
        u.kb0 = s * num_kb / splits;
        u.kb1 = (s + 1) * num_kb / splits;
        return true;
      }
      --it;
    }
    const int tile = rest + pair + it * pairs;
    if (tile >= total) return false;
    g2_tile_coords(tile, num_m, num_n, G, u.m_blk, u.n_blk);
    return true;
  }
};

// G2_EPI_EXPERTS: all tiles of an expert's weight gradient, expert by expert
struct G2ExpertWork {
  int num_n, per_expert, total;
  const int *offsets, *filled;
  __device__ __forceinline__ void init(const Gemm2Params& ep, bool, int num_m, int num_n_, int) {
    num_n = num_n_;
    per_expert = num_m * num_n_;
    total = per_expert * ep.experts;
    offsets = ep.offsets;
    filled = ep.filled;
  }
  __device__ __forceinline__ bool get(int it, G2Unit& u) const {
    const int i = (blockIdx.x >> 1) + it * (gridDim.x >> 1);
    if (i >= total) return false;
    u.batch = i / per_expert;
    const int r = i - u.batch * per_expert;
    u.m_blk = r / num_n;
    u.n_blk = r - u.m_blk * num_n;
    u.kb0 = offsets[u.batch] / G2_BK;
    u.kb1 = offsets[u.batch + 1] / G2_BK;
    if (filled) u.kb1 = min(u.kb1, u.kb0 + (filled[u.batch] + G2_BK - 1) / G2_BK);
    u.cut = false;
    return true;
  }
};

// G2_EPI_GROUPED: the tiles of every expert's rows, which start anew with each; up to 16 row blocks of an expert run side by side,
// so that a tile of its weights comes from HBM once (columns first: 470 -> 607 us, 8 experts of 28672 x 4096, 256 rows each).
// `get` is called with rising `it` and walks on from expert to expert.
struct G2GroupedWork {
  int num_n, num_kb, experts, e, base, row, row_end;   // the expert under way, its first unit and its rows
  const int* offsets;
  __device__ __forceinline__ void init(const Gemm2Params& ep, bool, int, int num_n_, int num_kb_) {
    num_n = num_n_;
    num_kb = num_kb_;
    experts = ep.experts;
    offsets = ep.offsets;
    e = base = 0;
    row = offsets[0];
    row_end = offsets[1];
  }
  __device__ __forceinline__ bool get(int it, G2Unit& u) {
    const int i = (blockIdx.x >> 1) + it * (gridDim.x >> 1);
    int num_m = (row_end - row + G2_BM - 1) / G2_BM;
    while (i - base >= num_m * num_n) {
      if (++e >= experts) {
        e = experts - 1;
        return false;
      }
      base += num_m * num_n;
      row = row_end;
      row_end = offsets[e + 1];
      num_m = (row_end - row + G2_BM - 1) / G2_BM;
    }
    g2_tile_coords(i - base, num_m, num_n, 16, u.m_blk, u.n_blk);
    u.row = row + u.m_blk * G2_BM;
    u.row_end = row_end;
    u.batch = e;
    u.kb0 = 0;
    u.kb1 = num_kb;
    u.cut = false;
    return true;
  }
};

// G2_EPI_LOGPROB (and the form of lmhead_logprob.cu with one CTA a tile): a unit is a block of rows and one of nsplit ranges of
// column tiles, of which the first take one tile more where they cannot all be equal. The units of a CTA or pair, `first` and every
// `step` further, are walked tile by tile; the row blocks of a range run side by side, so that a tile's weights come from HBM once.
struct LogprobTiles {
  int num_m, units, len, longer;
  __device__ __forceinline__ void init(int num_m_, int num_n, int nsplit) {
    num_m = num_m_;
    units = num_m_ * nsplit;
    len = num_n / nsplit;
    longer = num_n - len * nsplit;
  }
  __device__ __forceinline__ bool get(int it, int first, int step, int& m_blk, int& n_blk, int& range) const {
    for (int i = first; i < units; i += step) {
      range = i / num_m;
      const int n = len + (range < longer);
      if (it < n) {
        m_blk = i - range * num_m;
        n_blk = range * len + min(range, longer) + it;
        return true;
      }
      it -= n;
    }
    return false;
  }
};
struct G2LogprobWork {
  LogprobTiles tiles;
  int num_kb;
  __device__ __forceinline__ void init(const Gemm2Params& ep, bool, int num_m, int num_n, int num_kb_) {
    tiles.init(num_m, num_n, ep.lg.nsplit);
    num_kb = num_kb_;
  }
  __device__ __forceinline__ bool get(int it, G2Unit& u) const {
    if (!tiles.get(it, blockIdx.x >> 1, gridDim.x >> 1, u.m_blk, u.n_blk, u.batch)) return false;
    u.kb0 = 0;
    u.kb1 = num_kb;
    u.cut = false;
    return true;
  }
};

// TAIL: the rows of C end inside 16 bytes (a test in the epilogue of all kernels took 0.6 us of 33 x 3832 x 712 in fp32, 9.9).
template <int BN, int STAGES, bool A_MN, bool B_MN, int EPI, bool TAIL>
__device__ __forceinline__ void gemm2_mainloop(const CUtensorMap* tmA, const CUtensorMap* tmB, const CUtensorMap* tmC,
                                               const CUtensorMap* tmW, int M, int N, int K, const Gemm2Params& ep,
                                               uint32_t* status) {
  using SM = Gemm2Smem<BN, STAGES, EPI>;
  constexpr int EW = g2_epilogue_warps(EPI);
  static_assert(BN == 128 || BN == 256, "BN");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + STAGES * SM::STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + SM::STAGING_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;  // [2]
  uint64_t* tempty_bar = tfull_bar + 2;      // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  uint64_t* in_full = full_bar + 16;         // [8 epilogue warps][2], G2_EPI_DGATE_UP: gates and ups of a chunk
  static_assert(EPI != G2_EPI_DGATE_UP || (2 * STAGES + 5 <= 16 && SM::BAR_BYTES >= 256), "barriers");

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();  // 0: leader of the pair
  const bool leader = cta_rank == 0;
  constexpr uint32_t TMEM_COLS = 2 * BN;  // 256 or 512: a power of two

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * EW);  // the epilogue warps of both CTAs of the pair
    }
    if constexpr (EPI == G2_EPI_DGATE_UP)
      for (int i = 0; i < 2 * EW; ++i) mbar_init(&in_full[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(tmA);
    tma_prefetch_desc(tmB);
    tma_prefetch_desc(tmC);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before anything arrives on them from the other side
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int num_m = (M + G2_BM - 1) / G2_BM;
  constexpr bool GROUPED = EPI == G2_EPI_GROUPED || EPI == G2_EPI_GROUPED_GATE_UP;
  constexpr bool GATE_UP = EPI == G2_EPI_GATE_UP || EPI == G2_EPI_GROUPED_GATE_UP;
  constexpr bool GATED = EPI == G2_EPI_SWIGLU || GATE_UP;   // half of a tile's columns are gates, half ups
  constexpr int OUT_BN = GATED ? BN / 2 : BN;  // columns of C per tile
  const int n_cols = GATED ? N / 2 : N;        // columns of C
  const int num_n = (n_cols + OUT_BN - 1) / OUT_BN;
  std::conditional_t<EPI == G2_EPI_EXPERTS, G2ExpertWork,
                     std::conditional_t<EPI == G2_EPI_LOGPROB, G2LogprobWork,
                                        std::conditional_t<GROUPED, G2GroupedWork, G2Work>>> work;
  work.init(ep, EPI == G2_EPI_STORE || EPI == G2_EPI_GATE_UP || EPI == G2_EPI_DGATE_UP, num_m, num_n, (K + G2_BK - 1) / G2_BK);
  G2Unit unit;

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (elect_one()) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int it = 0; work.get(it, unit) && ok && !*abort_flag; ++it) {
        const int n_blk = unit.n_blk;
        // rows of A that lie outside the tensor (or the expert) are not fetched: it takes longer than fetching rows that exist
        const int tile_row = GROUPED ? unit.row : unit.m_blk * G2_BM;
        const bool peer_rows = tile_row + G2_BM_CTA < (GROUPED ? unit.row_end : M);
        const int a_row0 = tile_row + (int)cta_rank * G2_BM_CTA;
        // rows of B that this CTA feeds: its half of the tile's columns; with the SwiGLU epilogue the leader
        // feeds the gate rows and the other CTA the matching up rows, so a thread sees both in its TMEM lane
        int b_row0;
        if constexpr (GATED) b_row0 = n_blk * (BN / 2) + (cta_rank ? ep.up_row0 : 0);
        else b_row0 = n_blk * BN + (int)cta_rank * (BN / 2);
        for (int kb = unit.kb0; kb < unit.kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
            atomicCAS(status, ST_OK, ST_TIMEOUT_EMPTY);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * SM::STAGE_BYTES;
          uint8_t* sb = sa + SM::A_BYTES;
          const int k = kb * G2_BK;
          if (leader) mbar_arrive_expect_tx(&full_bar[stage], 2 * SM::B_BYTES + ep.a_bytes + (peer_rows ? SM::A_BYTES : 0));
          const uint32_t bar = mapa_shared(smem_u32(&full_bar[stage]), 0);
          if (!leader && !peer_rows) {
          } else if constexpr (!A_MN) {
            tma_load_2d_pair(sa, tmA, bar, k, a_row0);
          } else {
#pragma unroll
            for (int j = 0; j < G2_BM_CTA / 64; ++j) tma_load_2d_pair(sa + j * 8192, tmA, bar, a_row0 + j * 64, k);
          }
          if constexpr (GROUPED && !B_MN) {
            tma_load_3d_pair(sb, tmB, bar, k, b_row0, unit.batch);
          } else if constexpr (GROUPED) {
#pragma unroll
            for (int j = 0; j < (BN / 2) / 64; ++j) tma_load_3d_pair(sb + j * 8192, tmB, bar, b_row0 + j * 64, k, unit.batch);
          } else if constexpr (!B_MN) {
            tma_load_2d_pair(sb, tmB, bar, k, b_row0);
          } else {
#pragma unroll
            for (int j = 0; j < (BN / 2) / 64; ++j) tma_load_2d_pair(sb + j * 8192, tmB, bar, b_row0 + j * 64, k);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      // tail: the leader's commits keep arriving on this CTA's empty barriers until its last MMA retired; the CTA
      // must not exit (and release its shared memory) before they have landed
      if (ok && !*abort_flag) {
        for (int s = 0; s < STAGES; ++s) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1)) {
            atomicCAS(status, ST_OK, ST_TIMEOUT_EMPTY);
            *abort_flag = 1;
            break;
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) --------------------------
    if (leader && elect_one()) {
      constexpr uint32_t idesc =
          umma_idesc_bf16_f32(G2_BM, BN) | (A_MN ? (1u << 15) : 0u) | (B_MN ? (1u << 16) : 0u);
      uint32_t stage = 0, phase = 0;
      uint32_t acc = 0, acc_phase = 0;
      bool ok = true;
      for (int it = 0; work.get(it, unit) && ok && !*abort_flag; ++it) {
        if (!mbar_wait(&tempty_bar[acc], acc_phase ^ 1)) {
          atomicCAS(status, ST_OK, ST_TIMEOUT_TMEM_EMPTY);
          *abort_flag = 1;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = unit.kb0; kb < unit.kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase)) {
            atomicCAS(status, ST_OK, ST_TIMEOUT_FULL);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * SM::STAGE_BYTES);
          const uint32_t sb = sa + SM::A_BYTES;
#pragma unroll
          for (int k = 0; k < G2_BK / 16; ++k) {
            uint64_t ad = A_MN ? umma_desc_mnmajor_sw128(sa + k * 2048, 8192) : umma_desc_kmajor_sw128(sa + k * 32);
            uint64_t bd = B_MN ? umma_desc_mnmajor_sw128(sb + k * 2048, 8192) : umma_desc_kmajor_sw128(sb + k * 32);
            umma_bf16_ss_pair(tmem_d, ad, bd, idesc, (kb > unit.kb0 || k > 0) ? 1u : 0u);
          }
          tc_commit_pair(&empty_bar[stage], 3);  // frees this stage in both CTAs once the MMAs retire
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        tc_commit_pair(&tfull_bar[acc], 3);  // accumulator complete, in both CTAs
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ------------------------------ epilogue (warps 2..5 of both CTAs) --------------------
    const int quad = warp & 3;  // TMEM lane quadrant this warp may access
    const int half = EW == 8 ? (warp - 2) >> 2 : 0;   // of a tile's columns, where a quadrant has two warps
    uint8_t* slab0 = staging + (quad + 4 * half) * 8192;
    const uint32_t tempty_leader0 = mapa_shared(smem_u32(&tempty_bar[0]), 0);
    const uint32_t tempty_leader1 = mapa_shared(smem_u32(&tempty_bar[1]), 0);
    uint32_t acc = 0, acc_phase = 0;
    uint32_t slab_idx = 0;
    const uint32_t sw = (uint32_t)(lane & 7);  // 128-byte swizzle: 16-byte chunk j of row r sits at chunk j ^ (r & 7)
    LogprobRow lgr;
    long long lg_row = -1;   // the row and the range that lgr is about
    int lg_split = -1;
    // G2_EPI_DGATE_UP: chunks so far, and the one whose gates and ups are fetched next (unit in_it, chunk in_i of it)
    uint32_t in_count = 0;
    int in_it = 0, in_i = 0;
    auto in_fetch = [&](uint32_t count) {   // one elected lane
      G2Unit t;
      for (; work.get(in_it, t); ++in_it, in_i = 0) {
        const int row = t.m_blk * G2_BM + (int)cta_rank * G2_BM_CTA + quad * 32, col = t.n_blk * BN + half * 128 + 32 * in_i;
        if (t.cut || row >= M || in_i == 4 || col >= n_cols) continue;
        ++in_i;
        uint64_t* bar = &in_full[2 * (warp - 2) + (count & 1)];
        uint8_t* slab = slab0 + (count & 1) * 4096;
        mbar_arrive_expect_tx(bar, 4096);
        tma_load_3d(slab, tmC, bar, col, 0, row);
        tma_load_3d(slab + 2048, tmC, bar, col, 1, row);
        return;
      }
    };
    if constexpr (EPI == G2_EPI_DGATE_UP) {
      if (elect_one()) in_fetch(0);
    }
    for (int it = 0; work.get(it, unit) && !*abort_flag; ++it) {
      const int m_blk = unit.m_blk, n_blk = unit.n_blk;
      if (!mbar_wait(&tfull_bar[acc], acc_phase)) {
        atomicCAS(status, ST_OK, ST_TIMEOUT_TMEM_FULL);
        *abort_flag = 1;
        break;
      }
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(quad * 32) << 16);
      // first row of this warp's slabs, and where the rows of C end
      const int row0 = (GROUPED ? unit.row : m_blk * G2_BM) + (int)cta_rank * G2_BM_CTA + quad * 32;
      const int row_end = GROUPED ? unit.row_end : M;
      const int col_base = n_blk * OUT_BN;
      const bool cut = EPI == G2_EPI_STORE && unit.cut;             // fp32 into the pair's part of the workspace
      const bool out_fp32 = cut || ep.out_fp32;
      DlogitsRow dlr;
      if constexpr (EPI == G2_EPI_DLOGITS) dlr.load(ep.dl, min(row0 + lane, M - 1));
      // a slab = 32 rows x 128 bytes of C: 64 bf16 or 32 fp32 columns
      const int slab_cols = out_fp32 ? 32 : 64;
      if constexpr (EPI == G2_EPI_LOGPROB) {
        if (row0 + lane != lg_row || unit.batch != lg_split) {
          if (lg_split >= 0) lgr.store(ep.lg, lg_row, lg_split);
          lg_row = row0 + lane;
          lg_split = unit.batch;
          lgr.begin(ep.lg, lg_row);
        }
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + c, r);
          tmem_ld_wait();
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          lgr.chunk(ep.lg, col_base + c, v);
        }
      } else if constexpr (GATE_UP || EPI == G2_EPI_DGATE_UP) {
        auto pair = [](uint32_t v) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v)); };
        if (unit.cut) {   // fp32 into the pair's part of the workspace; gemm2_sum_gated_kernel does the rest
          float* dst = ep.ws + ((long long)(blockIdx.x >> 1) * G2_BM + (row0 - m_blk * G2_BM) + lane) * BN;
#pragma unroll 1
          for (int c = half * (BN / 2); c < (half + 1) * (BN / 2); c += 32) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(taddr + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j += 4) *reinterpret_cast<uint4*>(dst + c + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
          }
        } else if constexpr (GATE_UP) {
          // The gate and up values as they are stored, and what the SwiGLU kernel makes of them: the same bits as its pass over them.
          const int c = half * 64, gc = col_base + c;
          if (gc < n_cols && row0 < row_end) {
            auto put = [&](const uint32_t (&v)[32], auto store) {   // 64 columns as bf16 pairs, through the next staging slab
              uint8_t* slab = slab0 + (slab_idx++ & 1) * 4096;
              if (elect_one()) tma_store_wait_read<1>();
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
            uint32_t g[32], u[32];
            fetch(c, g);
            put(g, [&](uint8_t* slab) { tma_store_3d(tmW, slab, gc, 0, row0); });
            fetch(BN / 2 + c, u);
            put(u, [&](uint8_t* slab) { tma_store_3d(tmW, slab, gc, 1, row0); });
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              float a[8], b[8];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 x = pair(g[4 * q + j]), y = pair(u[4 * q + j]);
                a[2 * j] = x.x; a[2 * j + 1] = x.y;
                b[2 * j] = y.x; b[2 * j + 1] = y.y;
              }
              swiglu_values(a, b, a);
#pragma unroll
              for (int j = 0; j < 4; ++j) g[4 * q + j] = pack_bf16x2(a[2 * j], a[2 * j + 1]);
            }
            put(g, [&](uint8_t* slab) { tma_store_2d(tmC, slab, gc, row0); });
          }
        } else if (row0 < M) {
          // The accumulators are the gradient of the product. Gates and ups come by TMA, a chunk of 32 columns ahead, into the
          // slab (two halves of 32 rows x 64 bytes) from which their gradients leave.
#pragma unroll 1
          for (int i = 0; i < 4 && col_base + half * 128 + 32 * i < n_cols; ++i, ++in_count) {
            uint8_t* slab = slab0 + (in_count & 1) * 4096;
            if (elect_one()) {
              tma_store_wait_read<0>();   // the other slab's results have left
              in_fetch(in_count + 1);
            }
            __syncwarp();
            if (!mbar_wait(&in_full[2 * (warp - 2) + (in_count & 1)], (in_count >> 1) & 1)) {
              atomicCAS(status, ST_OK, ST_TIMEOUT_FULL);
              *abort_flag = 1;
            }
            const int gc = col_base + half * 128 + 32 * i;
            uint32_t r[32];
            tmem_ld_32x32b_x32(taddr + half * 128 + 32 * i, r);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {   // 64-byte swizzle: chunk q of row r sits at chunk q ^ ((r >> 1) & 3)
              uint4* at = reinterpret_cast<uint4*>(slab + lane * 64 + ((q ^ ((lane >> 1) & 3)) << 4));
              const uint4 gv = at[0], uv = at[2048 / 16];
              const uint32_t gs[4] = {gv.x, gv.y, gv.z, gv.w}, us[4] = {uv.x, uv.y, uv.z, uv.w};
              float a[8], b[8], d[8];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float2 x = pair(gs[j]), y = pair(us[j]);
                // rounded as it was when it was stored
                const float2 z = pair(pack_bf16x2(__uint_as_float(r[8 * q + 2 * j]), __uint_as_float(r[8 * q + 2 * j + 1])));
                a[2 * j] = x.x; a[2 * j + 1] = x.y;
                b[2 * j] = y.x; b[2 * j + 1] = y.y;
                d[2 * j] = z.x; d[2 * j + 1] = z.y;
              }
              swiglu_grads(a, b, d);
              at[0] = make_uint4(pack_bf16x2(a[0], a[1]), pack_bf16x2(a[2], a[3]), pack_bf16x2(a[4], a[5]), pack_bf16x2(a[6], a[7]));
              at[2048 / 16] = make_uint4(pack_bf16x2(b[0], b[1]), pack_bf16x2(b[2], b[3]), pack_bf16x2(b[4], b[5]), pack_bf16x2(b[6], b[7]));
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (elect_one()) {
              tma_store_3d(tmW, slab, gc, 0, row0);
              tma_store_3d(tmW, slab + 2048, gc, 1, row0);
              tma_store_commit();
            }
          }
        }
      } else
      // Rows past the end hold what shared memory held, and quotients of that take the slow way: a warp that has only such rows
      // forms none (304 x 12704 x 1000 105 us with them, 28; 311 x 72 x 896 37 and 11).
#pragma unroll 1
      for (int c = EPI == G2_EPI_SWIGLU && row0 >= M ? OUT_BN : 0; c < OUT_BN; c += slab_cols) {
        uint8_t* slab = slab0 + (slab_idx & 1) * 4096;
        // the store issued two slabs ago has finished reading this buffer
        if (elect_one()) tma_store_wait_read<1>();
        __syncwarp();
        uint8_t* my_row = slab + lane * 128;
        // The slab's accumulators, all on their way before the first is used: results of short contractions are bound by the
        // epilogue (28672 x 4096 over 64 rows: 70 us, 54). Two warps a quadrant in place of a stage: 45 there, but 73 and 69
        // over 300 rows.
        uint32_t plain[2][32];
        if constexpr (EPI == G2_EPI_STORE || EPI == G2_EPI_EXPERTS || EPI == G2_EPI_GROUPED) {
          tmem_ld_32x32b_x32(taddr + c, plain[0]);
          if (!out_fp32) tmem_ld_32x32b_x32(taddr + c + 32, plain[1]);
          tmem_ld_wait();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (out_fp32 && h == 1) break;
          const int cc = c + h * 32;  // 32 accumulator columns [cc, cc + 32)
          uint32_t r[32];
          if constexpr (EPI == G2_EPI_SWIGLU || EPI == G2_EPI_DLOGITS) tmem_ld_32x32b_x32(taddr + cc, r);
          float v[32];
          if constexpr (EPI == G2_EPI_SWIGLU) {
            uint32_t u[32];
            tmem_ld_32x32b_x32(taddr + BN / 2 + cc, u);
            tmem_ld_wait();
            swiglu_values(reinterpret_cast<const float(&)[32]>(r), reinterpret_cast<const float(&)[32]>(u), v);
          } else if constexpr (EPI == G2_EPI_DLOGITS) {
            tmem_ld_wait();
            const long long off = dlr.label - (ep.dl.v0 + col_base + cc);
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = dlr.of(__uint_as_float(r[j]), ep.dl.inv_temp, (long long)j == off);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = EPI == G2_EPI_EXPERTS && unit.kb0 == unit.kb1 ? 0.f : __uint_as_float(plain[h][j]);
            if (ep.bias != nullptr && !cut) {
              const int gc = col_base + cc;
#pragma unroll
              for (int j = 0; j < 32; ++j) {
                if (gc + j < n_cols)
                  v[j] += ep.bias_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(ep.bias)[gc + j])
                                       : reinterpret_cast<const float*>(ep.bias)[gc + j];
              }
            }
          }
          if (out_fp32) {
#pragma unroll
            for (int j = 0; j < 8; ++j) {  // 8 chunks of 4 floats
              float4 o = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
              *reinterpret_cast<float4*>(my_row + ((((uint32_t)j) ^ sw) << 4)) = o;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {  // 4 chunks of 8 bf16; this half starts at chunk 4 * h
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
        const int gc = col_base + c;
        if (elect_one()) {
          if (gc < (TAIL && !cut ? whole16(n_cols, ep.out_fp32) : n_cols) && row0 < row_end) {
            if constexpr (EPI == G2_EPI_EXPERTS) {
              if (ep.accumulate) tma_reduce_add_3d(tmC, slab, gc, row0, unit.batch);
              else tma_store_3d(tmC, slab, gc, row0, unit.batch);
            } else if (cut) tma_store_2d(tmW, slab, c, (int)(blockIdx.x >> 1) * G2_BM + (row0 - m_blk * G2_BM));
            else if (ep.accumulate) tma_reduce_add_2d(tmC, slab, gc, row0);
            else tma_store_2d(tmC, slab, gc, row0);
          }
          tma_store_commit();
        }
        if constexpr (TAIL) {
          const long long at = (long long)(row0 + lane) * ep.ldc;
          if (!cut && row0 + lane < M) {
            if (ep.out_fp32) store_tail((float*)ep.C + at, slab, gc, n_cols, ep.accumulate);
            else store_tail((__nv_bfloat16*)ep.C + at, slab, gc, n_cols, ep.accumulate);
          }
        }
        ++slab_idx;
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acc ? tempty_leader1 : tempty_leader0);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if constexpr (EPI == G2_EPI_LOGPROB) {
      if (lg_split >= 0) lgr.store(ep.lg, lg_row, lg_split);
    }
    if (elect_one()) tma_store_wait<0>();
  }

  // ------------------------------ teardown ------------------------------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag && threadIdx.x == 0) {
    // let copies that were already issued land before the CTA's shared memory is released
    for (int i = 0; i < 100; ++i) __nanosleep(1000);
  }
  cluster_sync_all();  // neither CTA frees TMEM or exits while the other may still signal it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

// gate and up halves of a contiguous [rows, 2 I] tensor as [rows][2][I]: boxes of 32 rows x `cols` columns of one half
inline int make_tmap_halves(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t I, int cols, CUtensorMapSwizzle swizzle) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) { last_tmap_error() = 1 << 24; return -1; }
  cuuint64_t gdim[3] = {I, 2, rows};
  cuuint64_t gstr[2] = {I * 2, I * 4};
  cuuint32_t box[3] = {(cuuint32_t)cols, 1, 32};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode_with_context([&] {
    return enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), gdim, gstr, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) last_tmap_error() = (3 << 24) | 0x50000 | (int)r;
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Row-major [rows, cols] tensor of fp32 / bf16 for the epilogue's TMA stores: box = 32 rows x 128 bytes, 128-byte swizzle.
inline int make_tmap_out(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, int out_fp32) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (!enc) { last_tmap_error() = 1 << 24; return -1; }
  const int eb = out_fp32 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || ((ld * eb) & 15)) {
    last_tmap_error() = (2 << 24) | 0x10000;
    return -2;
  }
  cuuint64_t gdim[2] = {cols, rows};
  cuuint64_t gstr[1] = {ld * (uint64_t)eb};
  cuuint32_t box[2] = {(cuuint32_t)(128 / eb), 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_with_context([&] {
    return enc(out, out_fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
               const_cast<void*>(ptr), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  });
  if (r != CUDA_SUCCESS) last_tmap_error() = (3 << 24) | 0x10000 | (int)r;
  return r == CUDA_SUCCESS ? 0 : -3;
}

}  // namespace b200
