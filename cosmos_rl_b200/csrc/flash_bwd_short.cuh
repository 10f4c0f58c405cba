// Backward of attention over short sequences, at most 128 queries and 128 keys each: one kernel with 64-query iterations (see
// flash_bwd.cu for the other form, the layouts, and why the line lies there).
//
// One CTA owns one (sequence, kv head): K and V stay in shared memory, dK and dV accumulate in TMEM over every query head of
// the GQA group and every block of 64 queries. Per (query head, 64-query block) iteration i:
//     S^T  = K Q^T                 M=keys(128) N=queries(64) K=d     TMEM S[i&1]   (64 columns)
//     dP^T = V dO^T                M=keys      N=queries     K=d     TMEM dP[i&1]  (64 columns)
//     P^T  = exp2(S^T c - lse),  dS^T = P^T o (dP^T - delta) * scale   8 softmax warps, thread = key row x 32 queries;
//                                                                      both to shared memory as bf16 [keys x queries]
//     dV  += P^T dO                M=keys N=d K=queries(64)          dO tile re-read as MN-major B
//     dK  += dS^T Q                M=keys N=d K=queries              Q  tile re-read as MN-major B
//     dQ^T = K^T dS^T              M=d N=queries K=keys              K tile as MN-major A, dS^T as MN-major B; over dP[i&1]
// All keys of a query are in this CTA, so dQ is whole after one iteration and goes out as bf16. The loads and the first two
// products of iteration i+1 run under the softmax of iteration i, the store of dQ of i-1 under the products of i. delta, the
// row sums of O o dO, is formed beside the softmax, an iteration ahead.
#pragma once

namespace b200 {

constexpr int FS_BQ = 64;                            // queries per iteration
constexpr int FS_Q_TILE = FS_BQ * FB_D * 2;          // 16 KiB
constexpr int FS_P_TILE = FB_B * FS_BQ * 2;          // 16 KiB
constexpr int FS_SMEM = 2 * FB_TILE + 4 * FS_Q_TILE + 2 * FS_P_TILE + 1024 /*lse, delta x2*/ + 256 + 1024;

#define FS_FAIL(code)                         \
  {                                           \
    atomicCAS(p.status, ST_OK, code);         \
    *abort_flag = 1;                          \
    break;                                    \
  }

__global__ void __launch_bounds__(FB_THREADS, 1)
flash_bwd_short_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do, FbParams p) {
  const int b = blockIdx.x / p.hkv, hk = blockIdx.x % p.hkv;
  const int q_beg = p.cu_q[b], len_q = p.cu_q[b + 1] - q_beg;
  const int k_beg = p.cu_k[b], len_k = p.cu_k[b + 1] - k_beg;
  const int shift = len_k - len_q;
  const int G = p.hq / p.hkv;
  fb_clear_all_outside(p);   // every CTA of this grid runs
  if (len_k <= 0) {          // queries without keys
    for (int i = threadIdx.x; i < len_q * G * (FB_D / 4); i += FB_THREADS) {
      const int e = i % (G * (FB_D / 4)), t = i / (G * (FB_D / 4));
      *reinterpret_cast<uint2*>(p.dq + (long long)(q_beg + t) * p.lddq + hk * G * FB_D + e * 4) = make_uint2(0u, 0u);
    }
    return;
  }
  const int per_head = (len_q + FS_BQ - 1) / FS_BQ;
  const int n_iter = per_head * G;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* k_sh = smem;
  uint8_t* v_sh = smem + FB_TILE;
  uint8_t* q_sh = smem + 2 * FB_TILE;                    // [2]
  uint8_t* do_sh = q_sh + 2 * FS_Q_TILE;                    // [2]
  uint8_t* pt_sh = do_sh + 2 * FS_Q_TILE;
  uint8_t* ds_sh = pt_sh + FS_P_TILE;
  float* lse_sh = reinterpret_cast<float*>(ds_sh + FS_P_TILE);   // [2][64] lse * log2(e)
  float* dlt_sh = lse_sh + 2 * FS_BQ;                             // [2][64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(lse_sh) + 1024);
  uint64_t* kv_full = bars;
  uint64_t* qdo_full = bars + 1;     // [2]
  uint64_t* qdo_empty = bars + 3;    // [2]
  uint64_t* sdp_ready = bars + 5;    // [2]
  uint64_t* pds_ready = bars + 7;
  uint64_t* mma3_done = bars + 8;
  uint64_t* dq_drained = bars + 9;   // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 11);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&qdo_full[s], 1);
      mbar_init(&qdo_empty[s], 1);
      mbar_init(&sdp_ready[s], 1);
      mbar_init(&dq_drained[s], 8);
    }
    mbar_init(pds_ready, 8);
    mbar_init(mma3_done, 1);
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
  // columns: S[2] 0..127, dP[2] (later dQ^T) 128..255, dV 256..383, dK 384..511
  const uint32_t tm_dv = tmem_base + 256, tm_dk = tmem_base + 384;

  if (warp == 0) {
    // ------------------------------------------------ TMA producer
    if (n_iter > 0 && elect_one()) {
      mbar_arrive_expect_tx(kv_full, 2 * FB_TILE);
      tma_load_2d(k_sh, &tm_k, kv_full, hk * FB_D, k_beg);
      tma_load_2d(k_sh + FB_TILE / 2, &tm_k, kv_full, hk * FB_D + 64, k_beg);
      tma_load_2d(v_sh, &tm_v, kv_full, hk * FB_D, k_beg);
      tma_load_2d(v_sh + FB_TILE / 2, &tm_v, kv_full, hk * FB_D + 64, k_beg);
      for (int i = 0; i < n_iter && !*abort_flag; ++i) {
        const int s = i & 1;
        const int h = hk * G + i / per_head, qb = i % per_head;
        if (!mbar_wait(&qdo_empty[s], ((i >> 1) & 1) ^ 1)) FS_FAIL(ST_TIMEOUT_EMPTY)
        const int row = q_beg + qb * FS_BQ;
        mbar_arrive_expect_tx(&qdo_full[s], 2 * FS_Q_TILE);
        tma_load_2d(q_sh + s * FS_Q_TILE, &tm_q, &qdo_full[s], h * FB_D, row);
        tma_load_2d(q_sh + s * FS_Q_TILE + FS_Q_TILE / 2, &tm_q, &qdo_full[s], h * FB_D + 64, row);
        tma_load_2d(do_sh + s * FS_Q_TILE, &tm_do, &qdo_full[s], h * FB_D, row);
        tma_load_2d(do_sh + s * FS_Q_TILE + FS_Q_TILE / 2, &tm_do, &qdo_full[s], h * FB_D + 64, row);
      }
      // the tensor core's last arrivals on these barriers land before the CTA's shared memory is released
      for (int i = max(n_iter - 2, 0); i < n_iter && !*abort_flag; ++i)
        if (!mbar_wait(&qdo_empty[i & 1], (i >> 1) & 1)) FS_FAIL(ST_TIMEOUT_EMPTY)
    }
  } else if (warp == 1) {
    // ------------------------------------------------ MMA issuer
    if (n_iter > 0 && elect_one()) {
      constexpr uint32_t id_s = umma_idesc_bf16_f32(128, FS_BQ);                                 // both K-major
      constexpr uint32_t id_dkv = umma_idesc_bf16_f32(128, FB_D) | (1u << 16);                   // B MN-major
      constexpr uint32_t id_dq = umma_idesc_bf16_f32(128, FS_BQ) | (1u << 15) | (1u << 16);      // A, B MN-major
      const uint32_t k_a = smem_u32(k_sh), v_a = smem_u32(v_sh), pt_a = smem_u32(pt_sh), ds_a = smem_u32(ds_sh);
      auto issue_sdp = [&](int i) -> bool {   // S^T(i), dP^T(i)
        const int s = i & 1;
        if (!mbar_wait(&qdo_full[s], (i >> 1) & 1)) return false;
        // dP[s] still holds dQ^T of iteration i-2 until the softmax warps have drained it
        if (i >= 2 && !mbar_wait(&dq_drained[s], ((i - 2) >> 1) & 1)) return false;
        tc_fence_after_sync();
        const uint32_t q_a = smem_u32(q_sh + s * FS_Q_TILE), do_a = smem_u32(do_sh + s * FS_Q_TILE);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tmem_base + s * FS_BQ, umma_desc_kmajor_sw128(k_a + (k >> 2) * (FB_TILE / 2) + (k & 3) * 32),
                       umma_desc_kmajor_sw128(q_a + (k >> 2) * (FS_Q_TILE / 2) + (k & 3) * 32), id_s, k > 0 ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tmem_base + 128 + s * FS_BQ,
                       umma_desc_kmajor_sw128(v_a + (k >> 2) * (FB_TILE / 2) + (k & 3) * 32),
                       umma_desc_kmajor_sw128(do_a + (k >> 2) * (FS_Q_TILE / 2) + (k & 3) * 32), id_s, k > 0 ? 1u : 0u);
        tc_commit(&sdp_ready[s]);
        return true;
      };
      do {
        if (!mbar_wait(kv_full, 0)) FS_FAIL(ST_TIMEOUT_FULL)
        if (!issue_sdp(0)) FS_FAIL(ST_TIMEOUT_FULL)
        for (int i = 0; i < n_iter; ++i) {
          const int s = i & 1;
          if (i + 1 < n_iter && !issue_sdp(i + 1)) FS_FAIL(ST_TIMEOUT_FULL)
          if (!mbar_wait(pds_ready, i & 1)) FS_FAIL(ST_TIMEOUT_TMEM_EMPTY)
          tc_fence_after_sync();
          const uint32_t q_a = smem_u32(q_sh + s * FS_Q_TILE), do_a = smem_u32(do_sh + s * FS_Q_TILE);
#pragma unroll
          for (int k = 0; k < 4; ++k)   // dV += P^T dO      (K = 64 queries)
            umma_bf16_ss(tm_dv, umma_desc_kmajor_sw128(pt_a + k * 32), umma_desc_mnmajor_sw128(do_a + k * 2048, FS_Q_TILE / 2),
                         id_dkv, (i > 0 || k > 0) ? 1u : 0u);
#pragma unroll
          for (int k = 0; k < 4; ++k)   // dK += dS^T Q
            umma_bf16_ss(tm_dk, umma_desc_kmajor_sw128(ds_a + k * 32), umma_desc_mnmajor_sw128(q_a + k * 2048, FS_Q_TILE / 2),
                         id_dkv, (i > 0 || k > 0) ? 1u : 0u);
#pragma unroll
          for (int k = 0; k < 8; ++k)   // dQ^T = K^T dS^T   (K = 128 keys), over dP[s]
            umma_bf16_ss(tmem_base + 128 + s * FS_BQ, umma_desc_mnmajor_sw128(k_a + k * 2048, FB_TILE / 2),
                         umma_desc_mnmajor_sw128(ds_a + k * 2048, FS_P_TILE), id_dq, k > 0 ? 1u : 0u);
          tc_commit(&qdo_empty[s]);
          tc_commit(mma3_done);
        }
      } while (false);
    }
  } else {
    // ------------------------------------------------ softmax / dS / drains (warps 2..9)
    // warp -> (TMEM lane quadrant, half of the 64 query columns). S^T / dP^T rows are keys, dQ^T rows are head-dim.
    const int quad = warp & 3;
    const int chalf = (warp - 2) >> 2;
    const int row = quad * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const int c0 = chalf * 32;                           // first query column of this warp
    const int key = row;
    const bool key_ok = key < len_k;
    const int q_min = p.causal ? key - shift : -(1 << 30);   // visible iff q >= key - shift
    const int sr = (warp - 2) * 8 + (lane >> 2);         // the query of a block whose statistics this lane brings
    bool ok = true;
    // lse and delta of query `sr` of iteration i. The warp reads O and dO of its eight queries, 256 coalesced bytes each
    // (past the end the last one again), and reduces the eight sums together: lane l ends up with query l >> 2.
    auto load_stats = [&](int i, float& l, float& dl) {
      if (i >= n_iter) return;
      const int h = hk * G + i / per_head, q0 = (i % per_head) * FS_BQ, first = q0 + (warp - 2) * 8;
      uint2 o2[8], g2[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const long long t = q_beg + min(first + u, len_q - 1);
        o2[u] = *reinterpret_cast<const uint2*>(p.out + t * p.ldo + h * FB_D + lane * 4);
        g2[u] = *reinterpret_cast<const uint2*>(p.dout + t * p.lddo + h * FB_D + lane * 4);
      }
      const bool live = q0 + sr < len_q;
      l = live ? p.lse[(long long)h * p.Tq + q_beg + q0 + sr] * FB_LOG2E : INFINITY;
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float2 x0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o2[u].x));
        const float2 x1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&o2[u].y));
        const float2 y0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g2[u].x));
        const float2 y1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&g2[u].y));
        v[u] = (x0.x * y0.x + x0.y * y0.y) + (x1.x * y1.x + x1.y * y1.y);
      }
#pragma unroll
      for (int d = 16, n = 4; n > 0; d >>= 1, n >>= 1) {   // lane distance d: n sums stay with each lane
        const bool hi = lane & d;
#pragma unroll
        for (int u = 0; u < n; ++u) {
          const float send = hi ? v[u] : v[u + n], keep = hi ? v[u + n] : v[u];
          v[u] = keep + __shfl_xor_sync(0xffffffffu, send, d);
        }
      }
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
      dl = live ? v[0] : 0.f;
    };
    auto drain_dq = [&](int j) {                         // dQ^T of iteration j: lanes = head-dim, columns = queries
      const int s = j & 1;
      const int h = hk * G + j / per_head, q0 = (j % per_head) * FS_BQ;
      uint32_t r[32];
      tmem_ld_32x32b_x32(tmem_base + 128 + s * FS_BQ + lane_addr + c0, r);
      tmem_ld_wait();
      __nv_bfloat16* dst = p.dq + (long long)(q_beg + q0 + c0) * p.lddq + h * FB_D + row;
#pragma unroll
      for (int c = 0; c < 32; ++c)
        if (q0 + c0 + c < len_q) dst[c * p.lddq] = __float2bfloat16(__uint_as_float(r[c]));
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dq_drained[s]);
    };
    float l_next = INFINITY, d_next = 0.f;
    load_stats(0, l_next, d_next);
    for (int i = 0; i < n_iter; ++i) {                   // never left early (named barrier inside)
      const int s = i & 1;
      const int q0 = (i % per_head) * FS_BQ;
      if ((lane & 3) == 0) { lse_sh[s * FS_BQ + sr] = l_next; dlt_sh[s * FS_BQ + sr] = d_next; }
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (*abort_flag) ok = false;
      load_stats(i + 1, l_next, d_next);                 // prefetch for the next iteration
      if (ok && !mbar_wait(&sdp_ready[s], (i >> 1) & 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_FULL); *abort_flag = 1; ok = false; }
      ok = __all_sync(0xffffffffu, ok);                  // tcgen05.ld below is warp-collective
      uint32_t pp[16], dd[16];
      if (ok) {
        tc_fence_after_sync();
        uint32_t rs[32], rd[32];
        tmem_ld_32x32b_x32(tmem_base + s * FS_BQ + lane_addr + c0, rs);
        tmem_ld_32x32b_x32(tmem_base + 128 + s * FS_BQ + lane_addr + c0, rd);
        tmem_ld_wait();
        const bool need_mask = !key_ok || (q0 < q_min) || (q0 + FS_BQ > len_q);
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          float pv[2], dv2[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int qc = c0 + c + u;
            float pe = exp2_approx(fmaf(__uint_as_float(rs[c + u]), p.scale_log2, -lse_sh[s * FS_BQ + qc]));
            if (need_mask && (!key_ok || q0 + qc < q_min || q0 + qc >= len_q)) pe = 0.f;
            pv[u] = pe;
            dv2[u] = pe * (__uint_as_float(rd[c + u]) - dlt_sh[s * FS_BQ + qc]) * p.scale;
          }
          pp[c >> 1] = pack_bf16x2(pv[0], pv[1]);
          dd[c >> 1] = pack_bf16x2(dv2[0], dv2[1]);
        }
        tc_fence_before_sync();
      }
      // P^T / dS^T of the previous iteration are still being read by its three MMAs until mma3_done(i-1)
      if (ok && i > 0 && !mbar_wait(mma3_done, (i - 1) & 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_FULL); *abort_flag = 1; ok = false; }
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        const int off = row * 128;
        const int chunk0 = c0 >> 3;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int sw = ((chunk0 + g) ^ (row & 7)) << 4;
          *reinterpret_cast<uint4*>(pt_sh + off + sw) = make_uint4(pp[4 * g], pp[4 * g + 1], pp[4 * g + 2], pp[4 * g + 3]);
          *reinterpret_cast<uint4*>(ds_sh + off + sw) = make_uint4(dd[4 * g], dd[4 * g + 1], dd[4 * g + 2], dd[4 * g + 3]);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(pds_ready);
        // while the tensor core runs the three MMAs of iteration i: drain dQ^T of iteration i-1
        if (i > 0) {
          tc_fence_after_sync();
          drain_dq(i - 1);
        }
      }
    }
    // ---- last dQ^T, then dK, dV of the key block
    if (n_iter > 0) {
      if (ok && !mbar_wait(mma3_done, (n_iter - 1) & 1)) { atomicCAS(p.status, ST_OK, ST_TIMEOUT_TMEM_FULL); *abort_flag = 1; ok = false; }
      ok = __all_sync(0xffffffffu, ok);
      if (ok) {
        tc_fence_after_sync();
        drain_dq(n_iter - 1);
      }
    }
    if (ok) {                                            // loads by every lane, stores by rows inside the sequence
      __nv_bfloat16* dkr = p.dk + (long long)(k_beg + key) * p.lddk + hk * FB_D;
      __nv_bfloat16* dvr = p.dv + (long long)(k_beg + key) * p.lddv + hk * FB_D;
#pragma unroll 1
      for (int c = chalf * 64; c < chalf * 64 + 64; c += 32) {
        uint32_t a[32], bb[32];
        if (n_iter > 0) {
          tmem_ld_32x32b_x32(tm_dk + lane_addr + c, a);
          tmem_ld_32x32b_x32(tm_dv + lane_addr + c, bb);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) { a[j] = 0u; bb[j] = 0u; }
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(a[8 * g + 0]), __uint_as_float(a[8 * g + 1]));
          o.y = pack_bf16x2(__uint_as_float(a[8 * g + 2]), __uint_as_float(a[8 * g + 3]));
          o.z = pack_bf16x2(__uint_as_float(a[8 * g + 4]), __uint_as_float(a[8 * g + 5]));
          o.w = pack_bf16x2(__uint_as_float(a[8 * g + 6]), __uint_as_float(a[8 * g + 7]));
          if (key_ok) *reinterpret_cast<uint4*>(dkr + c + 8 * g) = o;
          o.x = pack_bf16x2(__uint_as_float(bb[8 * g + 0]), __uint_as_float(bb[8 * g + 1]));
          o.y = pack_bf16x2(__uint_as_float(bb[8 * g + 2]), __uint_as_float(bb[8 * g + 3]));
          o.z = pack_bf16x2(__uint_as_float(bb[8 * g + 4]), __uint_as_float(bb[8 * g + 5]));
          o.w = pack_bf16x2(__uint_as_float(bb[8 * g + 6]), __uint_as_float(bb[8 * g + 7]));
          if (key_ok) *reinterpret_cast<uint4*>(dvr + c + 8 * g) = o;
        }
      }
    }
    tc_fence_before_sync();
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
