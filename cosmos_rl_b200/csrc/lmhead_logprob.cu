// Fused lm_head GEMM + per-token log-probability / entropy on tcgen05, without ever writing the
// [T, V] logits to memory. Replaces the eager row-loop log_softmax+gather and chunked entropy of the
// reference (cosmos_rl/utils/util.py:314-366, 899-994) and feeds the GRPO loss
// (cosmos_rl/policy/trainer/llm_trainer/grpo_trainer.py:113-353).
//
// Forward: work unit = (block of tokens, vocabulary range). The CTA or, on blocks of 256, the CTA pair that owns a unit walks its
// vocabulary tiles; each epilogue thread owns one token row and keeps an online-softmax state
// (running max, sum of exp, label logit, sum exp*logit) in registers across tiles, written once per unit
// to a [T, nsplit, 4] fp32 scratch that b200_logprob_combine reduces.
// Backward: the logits tile is recomputed on the tensor cores and the epilogue emits
// d(loss)/d(logits) in bf16 for a vocabulary chunk; the two remaining GEMMs are plain ones.
#include "gemm_2cta_launch.cuh"
#include "gemm_core.cuh"
#include "api.h"

namespace b200 {

constexpr int LP_BN = 256;
constexpr int LP_STAGES = 4;
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LN2 = 0.6931471805599453f;

// One CTA a tile of 128 rows (the pair form is an epilogue of gemm_2cta.cuh).
struct LogprobEpilogue {
  using Params = LogprobParams;
  LogprobRow st;
  int cur_m = 0, cur_range = -1;
  __device__ __forceinline__ void store(const Params& p, int row) const {
    if (cur_range >= 0) st.store(p, (long long)cur_m * GEMM_BM + row, cur_range);
  }
  __device__ __forceinline__ void tile_begin(const Params& p, const TileInfo& t, int row) {
    if (t.batch == cur_range && t.m_blk == cur_m) return;
    store(p, row);
    cur_m = t.m_blk;
    cur_range = t.batch;
    st.begin(p, (long long)cur_m * GEMM_BM + row);
  }
  __device__ __forceinline__ void chunk(const Params& p, const TileInfo& t, int, int col0, const float (&v)[32]) {
    st.chunk(p, t.n_blk * LP_BN + col0, v);
  }
  __device__ __forceinline__ void tile_end(const Params&, const TileInfo&, int) {}
  __device__ __forceinline__ void finish(const Params& p) { store(p, ((threadIdx.x >> 5) & 3) * 32 + (threadIdx.x & 31)); }
};

struct LogprobSched {
  LogprobTiles tiles;
  int num_kb;
  __device__ __forceinline__ void init(int M, int N, int K, int BN, const LogprobParams& p) {
    tiles.init((M + GEMM_BM - 1) / GEMM_BM, (N + BN - 1) / BN, p.nsplit);
    num_kb = (K + GEMM_BK - 1) / GEMM_BK;
  }
  __device__ __forceinline__ bool get(int it, TileInfo& t) const {
    if (!tiles.get(it, blockIdx.x, gridDim.x, t.m_blk, t.n_blk, t.batch)) return false;
    t.a_mn0 = t.m_blk * GEMM_BM;
    t.b_mn0 = t.n_blk * LP_BN;
    t.k0 = 0;
    t.num_kb = num_kb;
    return true;
  }
};

__global__ void __launch_bounds__(GEMM_THREADS, 1)
lmhead_logprob_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int T, int V,
                      int H, LogprobParams ep, uint32_t* status) {
  gemm_mainloop<LP_BN, LP_STAGES, LogprobEpilogue, LogprobSched>(&tmA, &tmB, T, V, H, ep, status);
}

// One warp a row.
__global__ void logprob_combine_kernel(const float* __restrict__ partial, const long long* __restrict__ labels,
                                       float* __restrict__ logprob, float* __restrict__ lse_out,
                                       float* __restrict__ entropy, int T, int nsplit) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= T) return;
  const float4* p = reinterpret_cast<const float4*>(partial) + (long long)r * nsplit;
  float M = -INFINITY, L = 0.f, E = 0.f, Z = -INFINITY;
  for (int s = lane; s < nsplit; s += 32) M = fmaxf(M, p[s].x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  for (int s = lane; s < nsplit; s += 32) {
    const float4 q = p[s];
    const float c = exp2f(q.x - M);
    L += q.y * c;
    E += q.w * c;
    Z = fmaxf(Z, q.z);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    L += __shfl_xor_sync(0xffffffffu, L, o);
    E += __shfl_xor_sync(0xffffffffu, E, o);
    Z = fmaxf(Z, __shfl_xor_sync(0xffffffffu, Z, o));
  }
  if (lane != 0) return;
  // convert from the log2 domain back to natural log
  const float lse2 = M + log2f(L);
  if (lse_out) lse_out[r] = lse2 * LN2;
  if (logprob) logprob[r] = (labels[r] >= 0) ? (Z - lse2) * LN2 : 0.f;
  if (entropy) entropy[r] = (lse2 - E / L) * LN2;
}

// ---------------------------------------------------------------------------------------------
// backward: dlogits chunk
// ---------------------------------------------------------------------------------------------
// single-CTA form, for up to 128 rows and for results off the 16-byte grid (the pair form is an epilogue of gemm_2cta.cuh)
struct DlogitsEpilogue {
  struct Params {
    DlogitsParams dl;
    __nv_bfloat16* out;
    long long ldd;
    int T, Vc;
  };
  DlogitsRow st;
  __device__ __forceinline__ void tile_begin(const Params& p, const TileInfo& t, int row) {
    const long long r = (long long)t.m_blk * GEMM_BM + row;
    if (r < p.T) st.load(p.dl, r);
  }
  __device__ __forceinline__ void chunk(const Params& p, const TileInfo& t, int row, int col0,
                                        const float (&v)[32]) {
    const long long r = (long long)t.m_blk * GEMM_BM + row;
    const int c = t.n_blk * LP_BN + col0;
    if (r >= p.T || c >= p.Vc) return;
    float o[32];
    const long long off = st.label - (long long)(p.dl.v0 + c);
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] = st.of(v[i], p.dl.inv_temp, (long long)i == off);
    __nv_bfloat16* dst = p.out + r * p.ldd + c;
    if (c + 32 <= p.Vc && ((reinterpret_cast<uintptr_t>(dst) & 15) == 0)) {
#pragma unroll
      for (int i = 0; i < 32; i += 8) {
        uint4 u;
        u.x = pack_bf16x2(o[i], o[i + 1]);
        u.y = pack_bf16x2(o[i + 2], o[i + 3]);
        u.z = pack_bf16x2(o[i + 4], o[i + 5]);
        u.w = pack_bf16x2(o[i + 6], o[i + 7]);
        *reinterpret_cast<uint4*>(dst + i) = u;
      }
    } else {
      for (int i = 0; i < 32 && c + i < p.Vc; ++i) dst[i] = __float2bfloat16(o[i]);
    }
  }
  __device__ __forceinline__ void tile_end(const Params&, const TileInfo&, int) {}
  __device__ __forceinline__ void finish(const Params&) {}
};

__global__ void __launch_bounds__(GEMM_THREADS, 1)
lmhead_dlogits_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int T, int Vc,
                      int H, DlogitsEpilogue::Params ep, uint32_t* status) {
  gemm_mainloop<LP_BN, LP_STAGES, DlogitsEpilogue, RasterSchedule>(&tmA, &tmB, T, Vc, H, ep, status);
}

}  // namespace b200

extern "C" {

int b200_lmhead_logprob_partial(const void* hidden, const void* weight, const long long* labels, float* partial,
                                int T, int V, int H, long long ldh, long long ldw, float inv_temperature,
                                int nsplit, int pairs, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (T <= 0 || V <= 0 || H <= 0 || (H & 7) || nsplit <= 0) return B200_ERR_ARG;
  const int num_n = (V + LP_BN - 1) / LP_BN, rows = pairs ? G2_BM : GEMM_BM;
  const long long units = (long long)((T + rows - 1) / rows) * nsplit;
  if (nsplit > num_n || units > INT_MAX / 2) return B200_ERR_ARG;
  const LogprobParams lg{labels, partial, T, V, nsplit, inv_temperature * LOG2E};
  CUtensorMap tmA, tmB;
  if (make_tmap_2d(&tmA, hidden, T, H, ldh, GEMM_BM, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  if (pairs) {
    using SM = Gemm2Smem<LP_BN, 6>;
    if (make_tmap_2d(&tmB, weight, V, H, ldw, LP_BN / 2, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
    auto kern = gemm2_bf16_kernel<LP_BN, 6, false, false, G2_EPI_LOGPROB>;
    static int whole[16] = {0};
    int np = 0;
    if (const int rc = resident_pairs(kern, whole, SM::TOTAL, G2_THREADS, num_sms, np)) return rc;
    Gemm2Params ep{};
    ep.a_bytes = SM::A_BYTES;
    ep.lg = lg;
    kern<<<2 * (int)(units < np ? units : np), G2_THREADS, SM::TOTAL, stream>>>(tmA, tmB, tmB, tmB, T, V, H, ep, status);
    return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
  }
  if (make_tmap_2d(&tmB, weight, V, H, ldw, LP_BN, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  using SM = GemmSmem<LP_BN, LP_STAGES>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(lmhead_logprob_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL) !=
        cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  lmhead_logprob_kernel<<<(int)(units < num_sms ? units : num_sms), GEMM_THREADS, SM::TOTAL, stream>>>(tmA, tmB, T, V, H, lg, status);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

int b200_logprob_combine(const float* partial, const long long* labels, float* logprob, float* lse, float* entropy,
                         int T, int nsplit, cudaStream_t stream) {
  if (T <= 0) return 0;
  b200::logprob_combine_kernel<<<(T + 7) / 8, 256, 0, stream>>>(partial, labels, logprob, lse, entropy, T, nsplit);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

int b200_lmhead_dlogits(const void* hidden, const void* weight, const long long* labels, const float* lse,
                        const float* g_logprob, const float* g_entropy, const float* entropy, void* dlogits, int T,
                        int V, int H, long long ldh, long long ldw, int v0, int Vc, long long ldd,
                        float inv_temperature, uint32_t* status, int num_sms, cudaStream_t stream) {
  using namespace b200;
  if (T <= 0 || Vc <= 0 || H <= 0 || (H & 7) || v0 < 0 || v0 + Vc > V) return B200_ERR_ARG;
  const __nv_bfloat16* wchunk = reinterpret_cast<const __nv_bfloat16*>(weight) + (long long)v0 * ldw;
  const DlogitsParams dl{labels, lse, g_logprob, g_entropy, entropy, v0, inv_temperature};
  // The logits are formed at the rate of the dense GEMM: CTA pairs once there are rows for their 256-row tiles (2048 x
  // 16384 x 3584: 147 us against 182 us with one CTA a tile, whose operand traffic bounds it).
  if (T > 128 && !(reinterpret_cast<uintptr_t>(dlogits) & 15) && !(ldd & 7)) {
    const Gemm2Params ep{nullptr, 0, 0, 0, 0, 8, 0, 0, 0, nullptr, nullptr, 0, dl};
    return launch_gemm2<256, 6, false, false, G2_EPI_DLOGITS>(hidden, wchunk, dlogits, T, Vc, H, ldh, ldw, ldd, ep, status,
                                                              num_sms, stream);
  }
  CUtensorMap tmA, tmB;
  if (make_tmap_2d(&tmA, hidden, T, H, ldh, GEMM_BM, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  if (make_tmap_2d(&tmB, wchunk, Vc, H, ldw, LP_BN, GEMM_BK, 2)) return B200_ERR_TENSORMAP;
  using SM = GemmSmem<LP_BN, LP_STAGES>;
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(lmhead_dlogits_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SM::TOTAL) !=
        cudaSuccess)
      return B200_ERR_LAUNCH;
    attr_set = true;
  }
  DlogitsEpilogue::Params ep{dl, (__nv_bfloat16*)dlogits, ldd, T, Vc};
  int tiles = ((T + GEMM_BM - 1) / GEMM_BM) * ((Vc + LP_BN - 1) / LP_BN);
  int grid = tiles < num_sms ? tiles : num_sms;
  lmhead_dlogits_kernel<<<grid, GEMM_THREADS, SM::TOTAL, stream>>>(tmA, tmB, T, Vc, H, ep, status);
  return cudaGetLastError() == cudaSuccess ? 0 : B200_ERR_LAUNCH;
}

}  // extern "C"
