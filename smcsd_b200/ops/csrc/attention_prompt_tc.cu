// Causal attention of prompt passes over the paged cache on the 5th-generation tensor cores (tcgen05 + tensor memory).
//
// A prompt pass has its rotated queries in memory and every key and value, the new ones among them, in the cache pages.  A CTA
// takes NT tiles of 128 query rows of one KV head (consecutive tokens x the query heads that share the KV head) and walks the
// keys those rows may see in steps of 64, one K/V copy for all its rows:
//     S_t = Q_t K^T      UMMA 128 x 64 x D, two score buffers per row tile in tensor memory
//     softmax            four warps per row tile, one query row per thread: P = exp2(S - m_ref) as bf16 over the scores, in
//                        tensor memory
//     O_t += P_t V       UMMA 128 x D x 64 accumulating in tensor memory, P its left operand there, V taken MN-major from its
//                        [key][dim] tile
// m_ref moves only when the row maximum has grown by more than 2^8, as in the shared-prefix pass; probabilities are rounded to
// bf16 behind an fp32 sum, as in the mma.sync step.  Keys behind a row's position are masked on the steps that cross it.
//
// What bounds it is the exponential (16 a cycle per SM): 64 x 256 of them take 1024 cycles of the 1500 to 2100 a step takes, the two
// products 256 (D = 64) to 512 (D = 128).  Two row tiles per CTA, each with its own issuing thread, let one tile's exponentials run
// while the other waits for its scores (a product takes 400 cycles from its issue to the barrier); D = 256 has room for one
// (tensor memory: 128 score + 256 output columns).
// Microseconds on B200, mma.sync step -> this kernel: 32/8 heads of 64, 4096 tokens 453 -> 137 (0.50 PFLOP/s), 6 x 300: 43 -> 23;
// 16/4 heads of 128, 4 x 1024: 174 -> 45; 16/2 heads of 256, 3 x 1100: 250 -> 64; a single prompt of 33 to 256 tokens: the same.
// (4096 tokens without the turns below 143, with them 137; gated heads of 256 in a model, gates read at the end 128, fetched ahead 108.)
// 64 tokens x 4 heads per CTA keep the masked part of a step's work small; the longest tiles come first in the list, so that
// the last ones fill the gaps.
//
// Steps of 64 consecutive pages come by TMA, all others are gathered with 16-byte cp.async copies: keys always lie in the order
// of their positions, so that sums, and with them every bit of the result, do not depend on where the pages are.  (Descending
// runs by TMA reversed the keys of a step: the same prompt gave other bits after its first pages had come back.)  Keys past the
// last visible one repeat it, so that a zero probability never meets an undefined value.  Every mbarrier wait is bounded; a timeout raises a status bit and all roles unwind.
#include "common.cuh"
#include "tmap_host.h"

namespace smc {

constexpr int PT_BK = 64, PT_LOADERS = 4, PT_MAX_UNITS = 16;

// Row tiles of a CTA; slots of the ring, each of them K or V of a step (64 keys), next to the query tiles in 227 KB.
template <int D> struct PtCfg;
template <> struct PtCfg<64> { static constexpr int NT = 2, UNITS = 16; };
template <> struct PtCfg<128> { static constexpr int NT = 2, UNITS = 10; };
template <> struct PtCfg<256> { static constexpr int NT = 1, UNITS = 5; };

struct PromptAttnParams {
  const __nv_bfloat16* q;        // [T, Hq * D] rotated queries
  const float* gate;             // null, or fp32 [T, ld_gate]: outputs are multiplied by its sigmoid
  const __nv_bfloat16* k_pool;   // [pages + 1, Hkv * D]
  const __nv_bfloat16* v_pool;
  const int* block_table;
  const int4* tiles;             // {block-table row, position of the first token, its index in q, tokens}
  __nv_bfloat16* out;            // [T, Hq * D]
  int ld_gate, bt_stride, bt_rows, n_pages, T, Hq, Hkv;
  int pdl;
  float scale_log2;              // softmax scale * log2(e)
  int* status;
};

struct PtShared {
  uint64_t kv_full[PT_MAX_UNITS], kv_empty[PT_MAX_UNITS], q_full[2], s_full[2][2], p_full[2][2], o_done[2][2], turn[2][4];
  uint32_t tmem_slot;
  volatile int abort;
};

__device__ __forceinline__ bool pt_wait(PtShared& S, int* status, uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (S.abort) return false;
    if (clock64() - t0 > SMC_SPIN_CYCLES) {
      atomicOr(status, SMC_ERR_BARRIER_TIMEOUT);
      S.abort = 1;
      return false;
    }
  }
}

__device__ __forceinline__ uint32_t pt_pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

__device__ __forceinline__ float pt_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float pt_max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

// two fp32 operations at once
__device__ __forceinline__ uint64_t pt_pair(float a, float b) {
  uint64_t y;
  asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(a), "f"(b));
  return y;
}
__device__ __forceinline__ float2 pt_unpair(uint64_t v) {
  float2 y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(y.x), "=f"(y.y) : "l"(v));
  return y;
}
__device__ __forceinline__ uint64_t pt_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t y;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(y) : "l"(a), "l"(b), "l"(c));
  return y;
}
__device__ __forceinline__ uint64_t pt_add2(uint64_t a, uint64_t b) {
  uint64_t y;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(y) : "l"(a), "l"(b));
  return y;
}

// D[tmem] (+)= A[tmem] * B[smem]: A rows are lanes, two bf16 values of K to a column
__device__ __forceinline__ void pt_umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

template <int D>
__global__ void __launch_bounds__((5 * PtCfg<D>::NT + PT_LOADERS) * 32, 1)
attn_prompt_tc_kernel(const PromptAttnParams p, const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV) {
  constexpr int NT = PtCfg<D>::NT, UNITS = PtCfg<D>::UNITS, BK = PT_BK;
  constexpr int KPW = BK / PT_LOADERS;                // keys of a scattered step gathered by one loader warp
  constexpr int NPAN = D / 64;                        // 64-element (128-byte) panels along the head dimension
  constexpr int PANEL_Q = 128 * 128, PANEL_KV = BK * 128;
  constexpr int Q_BYTES = NPAN * PANEL_Q, KV_BYTES = NPAN * PANEL_KV;
  constexpr int CPR = D / 8;                          // 16-byte chunks per row
  // tensor memory: scores (t * 2 + buffer) * 64, outputs COL_O + t * D, probabilities behind them where there is room (32 columns
  // each), in their scores' place with D = 128
  constexpr uint32_t COL_O = NT * 128;
  constexpr bool OWN_P = COL_O + NT * D + NT * 64 <= 512;
  constexpr uint32_t COL_P = OWN_P ? COL_O + NT * D : 0, P_PITCH = OWN_P ? 32 : 64;
  extern __shared__ uint8_t pt_smem_raw[];
  __shared__ PtShared S;
  const uint32_t raw = smem_u32(pt_smem_raw);
  uint8_t* smem = pt_smem_raw + (((raw + 1023u) & ~1023u) - raw);
  uint8_t* q_s = smem;
  uint8_t* kv_s = q_s + NT * Q_BYTES;                 // [unit]: K of step 0, V of step 0, K of step 1, ...

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int MMA_WARP = 4 * NT, LOAD_WARP = 5 * NT;   // softmax, one issuer per row tile, loaders
  const int G = p.Hq / p.Hkv, TT = 128 / G;           // tokens of a row tile
  const int kvh = blockIdx.x % p.Hkv, hbase = kvh * G;

  // the list is made by the host ahead of the pass
  const int4 tile = p.tiles[blockIdx.x / p.Hkv];
  int row = tile.x, first = tile.y, tok0 = tile.z, count = min(tile.w, NT * TT);
  if (row < 0 || row >= p.bt_rows || first < 0 || tok0 < 0 || tok0 + count > p.T || first + count > p.bt_stride) {
    if (threadIdx.x == 0) atomicOr(p.status, SMC_ERR_BOUNDS);
    row = first = tok0 = count = 0;
  }
  const int keys = first + count;                     // the last token sees all of these
  // key steps of each row tile
  int n_of[2] = {0, 0};
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    const int last = min(count, (t + 1) * TT);        // tokens up to this tile's end
    if (last > t * TT) n_of[t] = (first + last + BK - 1) / BK;
  }
  const int n_steps = max(n_of[0], n_of[1]);

  if (threadIdx.x == 0) {
    for (int s = 0; s < UNITS; ++s) {
      mbar_init(&S.kv_full[s], PT_LOADERS);
      mbar_init(&S.kv_empty[s], n_of[1] > 0 ? 2 : 1);
    }
    for (int t = 0; t < NT; ++t) {
      mbar_init(&S.q_full[t], 4);
      for (int q = 0; q < 4; ++q) mbar_init(&S.turn[t][q], 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(&S.s_full[t][i], 1);
        mbar_init(&S.p_full[t][i], 4);
        mbar_init(&S.o_done[t][i], 1);
      }
    }
    S.abort = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
  }
  if (warp == MMA_WARP) {
    tmem_alloc(&S.tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = S.tmem_slot;
  // queries and pages are the previous kernels' output
  if (p.pdl) { pdl_launch_dependents(); pdl_wait_prior_grid(); }
  if (warp >= LOAD_WARP) {
    // ================================================================= loaders
    const int lw = warp - LOAD_WARP;
    const int* bt = p.block_table + (size_t)row * p.bt_stride;
    const size_t kv_row = (size_t)p.Hkv * D;
    // every loader warp reads all 64 page ids of a step (lane l: keys l and l + 32) and comes to the same decision
    // (their range is looked at when they are used: a look at the load would wait for it)
    auto page_of = [&](int step, int half) { return step < n_steps ? bt[min(step * BK + half * 32 + lane, keys - 1)] : 0; };
    auto checked = [&](int page) {
      if (page >= 0 && page <= p.n_pages) return page;
      atomicOr(p.status, SMC_ERR_BOUNDS);
      return 0;
    };
    // LAG + 1 gathered units stay in flight per warp (more would starve: the V slot of a step comes free once the next step's K
    // has been handed over); page ids are fetched PD steps ahead
    constexpr int LAG = UNITS - 2, PD = 4;
    int issued = 0;
    uint32_t gathered = 0;                            // bit (u & 31): unit u went through cp.async (arrival still owed)
    int pg[PD][2];
#pragma unroll
    for (int d = 0; d < PD; ++d) {
      pg[d][0] = page_of(d, 0);
      pg[d][1] = page_of(d, 1);
    }
    bool go = true;
    const uint64_t pol = l2_policy_evict_last();      // the other row tiles of this KV head read the same keys
    for (int j0 = 0; go && j0 < n_steps; j0 += PD) {
#pragma unroll
      for (int d = 0; d < PD; ++d) {
        const int j = j0 + d;
        if (!go || j >= n_steps) break;
        const int pa = checked(pg[d][0]), pb = checked(pg[d][1]);
        pg[d][0] = page_of(j + PD, 0);
        pg[d][1] = page_of(j + PD, 1);
        const int base = __shfl_sync(0xffffffffu, pa, 0);
        const bool run = __all_sync(0xffffffffu, pa == base + lane && pb == base + 32 + lane) && base >= 1;
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          const int u = 2 * j + kv, st = u % UNITS, use = u / UNITS;
          const bool ok = use < 1 || pt_wait(S, p.status, &S.kv_empty[st], (uint32_t)(use - 1) & 1u);
          if (!__all_sync(0xffffffffu, ok)) { go = false; break; }
          uint8_t* ptr = kv_s + (size_t)st * KV_BYTES;
          if (run) {
            if (lane == 0) {
              if (lw == 0) {
                mbar_expect_tx(&S.kv_full[st], KV_BYTES);
#pragma unroll
                for (int pan = 0; pan < NPAN; ++pan)
                  tma_load_2d(ptr + pan * PANEL_KV, kv ? &tmV : &tmK, &S.kv_full[st], kvh * D + pan * 64, base, pol);
              } else {
                mbar_arrive(&S.kv_full[st]);
              }
            }
            gathered &= ~(1u << (u & 31));
          } else {
            const uint32_t dst0 = smem_u32(ptr);
            const __nv_bfloat16* pool = kv ? p.v_pool : p.k_pool;
            const int mine = lw < 2 ? pa : pb;        // this warp's 16 keys sit in lanes (lw & 1) * 16 ..
#pragma unroll 4
            for (int idx = lane; idx < KPW * CPR; idx += 32) {
              const int kl = idx / CPR, c = idx % CPR, key = lw * KPW + kl;
              const int pgi = __shfl_sync(0xffffffffu, mine, (lw & 1) * 16 + kl);
              const uint32_t dst = dst0 + (uint32_t)((c >> 3) * PANEL_KV + key * 128 + (((c & 7) ^ (key & 7)) << 4));
              asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(pool + (size_t)pgi * kv_row + (size_t)kvh * D + c * 8) : "memory");
            }
            gathered |= 1u << (u & 31);
          }
          asm volatile("cp.async.commit_group;" ::: "memory");     // one group per unit (empty for a TMA unit)
          if (u >= LAG && ((gathered >> ((u - LAG) & 31)) & 1u)) { // gathered unit u - LAG has landed: hand it over
            asm volatile("cp.async.wait_group %0;" ::"n"(LAG) : "memory");
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.kv_full[(u - LAG) % UNITS]);
          }
          ++issued;
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_proxy_async();
    __syncwarp();
    if (lane == 0)
      for (int u = max(0, issued - LAG); u < issued; ++u)
        if ((gathered >> (u & 31)) & 1u) mbar_arrive(&S.kv_full[u % UNITS]);
    // an aborted CTA keeps its shared memory until the copies in flight have landed
    if (S.abort && lw == 0 && lane == 0)
      for (int u = max(0, issued - UNITS); u < issued; ++u)
        if (!((gathered >> (u & 31)) & 1u)) (void)mbar_wait(&S.kv_full[u % UNITS], (uint32_t)(u / UNITS) & 1u);
  } else if (warp >= MMA_WARP) {
    // ================================================================= MMA issuers (one thread per row tile)
    const int t = warp - MMA_WARP, n = NT > 1 && t ? n_of[1] : n_of[0];
    if (n > 0 && elect_one()) {
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, BK);
      constexpr uint32_t idesc_o = umma_idesc_bf16(128, D) | (1u << 16);       // B operand (V) is MN-major
      const uint32_t q_addr = smem_u32(q_s);
      const uint32_t tS = tmem_base + (uint32_t)t * 128u, tP = tmem_base + COL_P + (uint32_t)t * 2u * P_PITCH, tO = tmem_base + COL_O + t * D;
      auto wait_unit = [&](int u) { return pt_wait(S, p.status, &S.kv_full[u % UNITS], (uint32_t)(u / UNITS) & 1u); };
      auto issue_s = [&](int j) -> bool {
        if (!wait_unit(2 * j)) return false;
        // a buffer that holds probabilities as well is free once their product is done
        if (!OWN_P && j >= 2 && !pt_wait(S, p.status, &S.o_done[t][j & 1], (uint32_t)((j >> 1) - 1) & 1u)) return false;
        tc_fence_after();
        const uint32_t k_addr = smem_u32(kv_s + (size_t)(2 * j % UNITS) * KV_BYTES);
#pragma unroll
        for (int pan = 0; pan < NPAN; ++pan)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ss(tS + (uint32_t)(j & 1) * 64u, umma_desc_k_sw128(q_addr + t * Q_BYTES + pan * PANEL_Q) + 2 * k,
                         umma_desc_k_sw128(k_addr + pan * PANEL_KV) + 2 * k, idesc_s, (pan | k) ? 1u : 0u);
        umma_commit(&S.s_full[t][j & 1]);
        umma_commit(&S.kv_empty[2 * j % UNITS]);
        return true;
      };
      // scores are issued two steps ahead of the product that needs them, into the buffer whose scores became these probabilities
      bool ok = pt_wait(S, p.status, &S.q_full[t], 0) && issue_s(0);
      if (ok && n > 1) ok = issue_s(1);
      for (int j = 0; ok && j < n; ++j) {
        if (!wait_unit(2 * j + 1) || !pt_wait(S, p.status, &S.p_full[t][j & 1], (uint32_t)(j >> 1) & 1u)) { ok = false; break; }
        tc_fence_after();
        const uint32_t v_addr = smem_u32(kv_s + (size_t)((2 * j + 1) % UNITS) * KV_BYTES);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          pt_umma_ts(tO, tP + (uint32_t)(j & 1) * P_PITCH + 8 * k, umma_desc_mn_sw128(v_addr + k * 2048, PANEL_KV), idesc_o, (j | k) ? 1u : 0u);
        umma_commit(&S.o_done[t][j & 1]);             // O_t holds the sum over steps 0..j
        umma_commit(&S.kv_empty[(2 * j + 1) % UNITS]);
        if (j + 2 < n) ok = issue_s(j + 2);
      }
      // steps that only the other tile's rows see
      for (int u = 2 * n; ok && u < 2 * n_steps; ++u) {
        ok = wait_unit(u);
        if (ok) mbar_arrive(&S.kv_empty[u % UNITS]);
      }
    }
    __syncwarp();
  } else {
    // ================================================================= softmax (one query row per thread)
    const int t = warp >> 2, q = warp & 3, r = q * 32 + lane, n = NT > 1 && t ? n_of[1] : n_of[0];
    const uint32_t lane_off = ((uint32_t)(q * 32)) << 16;
    const uint32_t tO = tmem_base + COL_O + t * D + lane_off, tP = tmem_base + COL_P + (uint32_t)t * 2u * P_PITCH + lane_off;
    const int tk = t * TT + r / G;
    const bool live = r < TT * G && tk < count;
    const int pos = first + min(tk, count - 1);
    // this tile's query rows r = token * G + head, zero padded to 128, into swizzled K-major panels: a row per thread
    {
      const uint4* src = reinterpret_cast<const uint4*>(p.q + ((size_t)(tok0 + tk) * p.Hq + hbase + r % G) * D);
      uint8_t* dst = q_s + t * Q_BYTES + r * 128;
#pragma unroll
      for (int c0 = 0; c0 < CPR; c0 += 8) {
        uint4 v[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) v[c] = live ? src[c0 + c] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(dst + (c0 >> 3) * PANEL_Q + ((c ^ (r & 7)) << 4)) = v[c];
      }
    }
    fence_proxy_async();                              // generic-proxy writes before the tensor core reads them
    __syncwarp();
    if (lane == 0) mbar_arrive(&S.q_full[t]);
    const float* gate = p.gate != nullptr ? p.gate + (size_t)(tok0 + min(tk, max(count, 1) - 1)) * p.ld_gate + (size_t)(hbase + r % G) * D : nullptr;
    if (live && gate != nullptr) {                    // the row's gates on their way to L2 while the keys are walked
#pragma unroll
      for (int c = 0; c < D; c += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(gate + c));
    }
    float m_ref = -INFINITY;                          // exponent reference of the row (log2 domain)
    uint64_t sum[2] = {0ull, 0ull};                   // its running sum, in four parts
    bool alive = true;
    for (int j = 0; j < n; ++j) {
      const int nvalid = pos + 1 - j * BK;            // keys of this step the row may see (none, if not positive)
      if (!__all_sync(0xffffffffu, pt_wait(S, p.status, &S.s_full[t][j & 1], (uint32_t)(j >> 1) & 1u))) { alive = false; break; }
      tc_fence_after();
      const uint32_t ts = tmem_base + (uint32_t)(t * 2 + (j & 1)) * 64u + lane_off;
      uint32_t x[BK];
#pragma unroll
      for (int c0 = 0; c0 < BK; c0 += 16) tmem_ld_32x32b_x16(ts + c0, *reinterpret_cast<uint32_t(*)[16]>(&x[c0]));
      tmem_ld_wait();
      const bool full = __all_sync(0xffffffffu, nvalid >= BK);
      if (!full) {
#pragma unroll
        for (int i = 0; i < BK; ++i)
          if (i >= nvalid) x[i] = 0xff800000u;        // -inf: probability zero
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < BK; i += 2) mx[(i >> 1) & 3] = pt_max3(mx[(i >> 1) & 3], __uint_as_float(x[i]), __uint_as_float(x[i + 1]));
      const float top = fmaxf(pt_max3(mx[0], mx[1], mx[2]), mx[3]) * p.scale_log2;
      const bool grow = top > m_ref + 8.f;            // also true on the first step (m_ref = -inf; every row sees key 0)
      if (j >= 1 && __any_sync(0xffffffffu, grow)) {
        // rare after the first steps: PV of step j - 1 must have completed before O is rescaled in tensor memory
        if (!__all_sync(0xffffffffu, pt_wait(S, p.status, &S.o_done[t][(j - 1) & 1], (uint32_t)((j - 1) >> 1) & 1u))) { alive = false; break; }
        tc_fence_after();
        const float alpha = grow ? exp2f(m_ref - top) : 1.f;
#pragma unroll
        for (int c0 = 0; c0 < D; c0 += 16) {
          uint32_t o[16];
          tmem_ld_32x32b_x16(tO + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32b_x16(tO + c0, o);
        }
        tmem_st_wait();
        const uint64_t alpha2 = pt_pair(alpha, alpha);
        sum[0] = pt_fma2(sum[0], alpha2, 0ull);
        sum[1] = pt_fma2(sum[1], alpha2, 0ull);
      }
      if (grow) m_ref = top;
      // probabilities of step j - 2 are out of this step's place
      if (OWN_P && !__all_sync(0xffffffffu, j < 2 || pt_wait(S, p.status, &S.o_done[t][j & 1], (uint32_t)((j - 2) >> 1) & 1u))) { alive = false; break; }
      // The two warps that share a scheduler (same quarter of either tile) take turns at the exponentials, tile 0 first: one looks for its
      // maxima and moves its operands meanwhile.  Left alone they run in step, both at the exponentials and then neither.
      if (NT > 1) {
        const bool in_turn = t ? j >= n_of[0] || pt_wait(S, p.status, &S.turn[1][q], (uint32_t)j & 1u)
                               : j == 0 || n_of[1] == 0 || pt_wait(S, p.status, &S.turn[0][q], (uint32_t)(j - 1) & 1u);
        if (!__all_sync(0xffffffffu, in_turn)) { alive = false; break; }
      }
      const uint64_t mul = pt_pair(p.scale_log2, p.scale_log2), off = pt_pair(-m_ref, -m_ref);
#pragma unroll
      for (int c0 = 0; c0 < BK; c0 += 32) {
        uint32_t pk[16];
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          const float2 e = pt_unpair(pt_fma2(pt_pair(__uint_as_float(x[c0 + i]), __uint_as_float(x[c0 + i + 1])), mul, off));
          const float p0 = pt_ex2(e.x), p1 = pt_ex2(e.y);
          sum[(i >> 1) & 1] = pt_add2(sum[(i >> 1) & 1], pt_pair(p0, p1));
          pk[i >> 1] = pt_pack(p0, p1);
        }
        tmem_st_32x32b_x16(tP + (uint32_t)(j & 1) * P_PITCH + (c0 >> 1), pk);
      }
      if (NT > 1 && lane == 0) mbar_arrive(&S.turn[t ^ 1][q]);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.p_full[t][j & 1]);
    }
    // the last product is done: read the accumulated O once
    if (alive && n > 0)
      alive = __all_sync(0xffffffffu, pt_wait(S, p.status, &S.o_done[t][(n - 1) & 1], (uint32_t)((n - 1) >> 1) & 1u));
    tc_fence_after();
    if (alive && n > 0) {
      const size_t at = ((size_t)(tok0 + min(tk, count - 1)) * p.Hq + hbase + r % G) * D;
      const float2 s0 = pt_unpair(sum[0]), s1 = pt_unpair(sum[1]);
      const float inv = 1.f / ((s0.x + s0.y) + (s1.x + s1.y));
#pragma unroll
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        float4 g[8];
        tmem_ld_32x32b_x16(tO + c0, *reinterpret_cast<uint32_t(*)[16]>(&o[0]));
        tmem_ld_32x32b_x16(tO + c0 + 16, *reinterpret_cast<uint32_t(*)[16]>(&o[16]));
        if (live && gate != nullptr) {
#pragma unroll
          for (int i = 0; i < 8; ++i) g[i] = *reinterpret_cast<const float4*>(gate + c0 + 4 * i);
        }
        tmem_ld_wait();
        if (live) {
          float v[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(o[i]) * inv;
          if (gate != nullptr) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              v[4 * i] *= 1.f / (1.f + __expf(-g[i].x));
              v[4 * i + 1] *= 1.f / (1.f + __expf(-g[i].y));
              v[4 * i + 2] *= 1.f / (1.f + __expf(-g[i].z));
              v[4 * i + 3] *= 1.f / (1.f + __expf(-g[i].w));
            }
          }
          uint4* dst = reinterpret_cast<uint4*>(p.out + at + c0);
#pragma unroll
          for (int i = 0; i < 4; ++i)
            dst[i] = make_uint4(pt_pack(v[8 * i], v[8 * i + 1]), pt_pack(v[8 * i + 2], v[8 * i + 3]), pt_pack(v[8 * i + 4], v[8 * i + 5]),
                                pt_pack(v[8 * i + 6], v[8 * i + 7]));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == MMA_WARP) tmem_dealloc(tmem_base, 512);
}

template <int D>
static int launch_prompt(const PromptAttnParams& p, int n_tiles, const CUtensorMap& tmK, const CUtensorMap& tmV, cudaStream_t st) {
  constexpr int NT = PtCfg<D>::NT;
  constexpr size_t smem = (size_t)NT * (D / 64) * 16384 + (size_t)PtCfg<D>::UNITS * (D / 64) * 8192 + 1024;
  CUDA_CHECK_RET(cudaFuncSetAttribute(attn_prompt_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n_tiles * p.Hkv));
  cfg.blockDim = dim3((5 * NT + PT_LOADERS) * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = p.pdl ? 1 : 0;
  CUDA_CHECK_RET(cudaLaunchKernelEx(&cfg, attn_prompt_tc_kernel<D>, p, tmK, tmV));
  return 0;
}

}  // namespace smc

// Most tokens a tile of the list may hold (0: heads that this kernel does not take).
SMC_API int smc_attention_prompt_tokens(int Hq, int Hkv, int D) {
  if (Hkv < 1 || Hq % Hkv || Hq / Hkv > 128 || (D != 64 && D != 128 && D != 256)) return 0;
  return (D == 256 ? 1 : 2) * (128 / (Hq / Hkv));
}

// q, out [T, Hq * D] bf16; tiles [n_tiles][4] int32 {block-table row, position of the first token, its index in q, tokens}:
// consecutive tokens of one sequence that attend all keys up to their own position, all of them in the pages.
SMC_API int smc_attention_prompt_tc(const void* q, const float* gate, int ld_gate, const void* k_pool, const void* v_pool, int n_pages,
                                    const int* block_table, int bt_stride, int bt_rows, const int* tiles, int n_tiles, void* out, int T,
                                    int Hq, int Hkv, int D, float scale, int* status, int pdl, cudaStream_t st) {
  using namespace smc;
  if (n_tiles <= 0) return 0;
  if (smc_attention_prompt_tokens(Hq, Hkv, D) == 0) return -84;
  // rows of queries and outputs move in pieces of 16 bytes, a tile's numbers in one; the tensor maps look at the pools themselves
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(tiles) | reinterpret_cast<uintptr_t>(k_pool) |
       reinterpret_cast<uintptr_t>(v_pool)) & 15)
    return -86;
  if (gate != nullptr && ((ld_gate & 3) || (reinterpret_cast<uintptr_t>(gate) & 15))) return -85;
  PromptAttnParams p;
  p.q = (const __nv_bfloat16*)q; p.gate = gate; p.ld_gate = ld_gate;
  p.k_pool = (const __nv_bfloat16*)k_pool; p.v_pool = (const __nv_bfloat16*)v_pool;
  p.block_table = block_table; p.bt_stride = bt_stride; p.bt_rows = bt_rows; p.tiles = (const int4*)tiles;
  p.out = (__nv_bfloat16*)out; p.n_pages = n_pages; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.pdl = pdl;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.status = status;
  CUtensorMap tmK, tmV;
  int rc = pool_tmap(&tmK, k_pool, (long long)n_pages + 1, (long long)Hkv * D);
  if (rc == 0) rc = pool_tmap(&tmV, v_pool, (long long)n_pages + 1, (long long)Hkv * D);
  if (rc) return rc;
  if (D == 64) return launch_prompt<64>(p, n_tiles, tmK, tmV, st);
  if (D == 128) return launch_prompt<128>(p, n_tiles, tmK, tmV, st);
  return launch_prompt<256>(p, n_tiles, tmK, tmV, st);
}
