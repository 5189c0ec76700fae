// GEMM for wide batches (prompts, scored texts, large verify passes) on sm_100a:  Y[m, n] = sum_k X[m, k] * W[n, k].
//
// With a few hundred token rows the product is bound by what one SM can pull from L2 (about 64 bytes a cycle) and by the tensor
// cores, not by HBM.  A 128 x 128 tile per SM needs 32 KB for every 256 cycles of MMA, twice that rate.  Here two SMs share one tile
// (cta_group::2): 256 weight rows x BN tokens, each CTA loads its 128 weight rows and half of the tokens, so that
// 256 x 256 tiles need 64 bytes a cycle.  One CTA pair per two SMs walks the tiles (persistent); accumulators are double
// buffered in tensor memory, eight epilogue warps drain one while the MMAs fill the other.
//
//   warp 0     TMA producer of this CTA's halves (the bytes are counted on the pair leader's mbarriers)
//   warp 1     tensor memory allocation; in the leader one thread issues the MMAs
//   warps 2-9  epilogue: two warps per quarter of the 128 rows, each half of the token columns, straight from tensor memory; a
//              warp's 32 lanes are 32 neighbouring output columns, so fp32 rows leave in 128-byte pieces
//
// Epilogues are those of the weight-streaming kernel without split-K: fp32 store, residual accumulate with the bf16 copy and the
// sums of squares per 128 columns, bf16, gated units, squared relu.
//
// Every wait is bounded; on a timeout the roles of a CTA unwind, the leader waits for the copies in flight (both CTAs'), and the pair
// frees its tensor memory and returns with a status bit.
#include <string.h>

#include "common.cuh"
#include "gemm_params.cuh"

namespace smc {

constexpr int WIDE_THREADS = 320, WIDE_EPI_WARPS = 8;

template <int BN>
struct WideCfg {
  static constexpr int A_BYTES = 128 * 128;                  // this CTA's weight rows, 128 bytes of K each
  static constexpr int B_BYTES = BN / 2 * 128;               // this CTA's half of the tokens
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = 196608 / STAGE_BYTES;        // 192 KB of ring
  static constexpr int TMEM_COLS = 2 * BN <= 256 ? 256 : 512;
  static constexpr int EXCH = WIDE_EPI_WARPS * 16 * 32 * 4;          // gated units: halves traded between gate and up warps
  static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + EXCH;
};

// Sum over the lanes of 32 values per lane: lane i returns the total of v[i].  Every step halves the values a lane holds.
__device__ __forceinline__ float lanes_to_columns(float (&v)[32], int lane) {
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1) {
    const bool up = (lane & w) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float keep = up ? v[i + w] : v[i], give = up ? v[i] : v[i + w];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, w);
    }
  }
  return v[0];
}

template <int BN, int EPI, bool FP8, bool GRP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WIDE_THREADS, 1) gemm_wide_kernel(const __grid_constant__ CUtensorMap tmW,
                                                                                        const __grid_constant__ CUtensorMap tmX,
                                                                                        const GemmParams p) {
  using C = WideCfg<BN>;
  constexpr int nst = C::STAGES, HALF = BN / 2;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
  float* exch = reinterpret_cast<float*>(smem + nst * C::STAGE_BYTES);
  __shared__ uint64_t full[nst], empty[nst], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int sh_abort, sh_issued, sh_consumed;
  __shared__ float s_rstd[2][BN];
  __shared__ float s_sq[2][2][4][32];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
  const int slabs = (p.N + 255) / 256, groups = GRP ? p.grp.groups : 1;
  const int tiles = slabs * groups * p.m_tiles, nkb = p.kblocks;
  if (p.pdl) pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < nst; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * WIDE_EPI_WARPS);
    }
    sh_abort = 0;
    sh_issued = 0;
    sh_consumed = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) tmem_alloc_pair(&tmem_slot, C::TMEM_COLS);
  tc_fence_before();
  cluster_sync();                                            // the peer's barriers are initialised as well
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;

  // tile -> first weight row of its group's matrix, of the map, first token, column offsets
  auto locate = [&](int t, int& n0, int& w_row, int& m0, int& x_col, size_t& out_off) {
    const int col = t / p.m_tiles;                           // token tiles of a weight slab run at the same time
    m0 = (t - col * p.m_tiles) * BN;
    const int g = GRP ? col / slabs : 0;
    n0 = (col - g * slabs) * 256;
    w_row = GRP ? g * p.grp.w_rows + n0 : n0;
    x_col = GRP ? g * p.grp.x_cols : 0;
    out_off = GRP ? (size_t)g * p.grp.out_cols : 0;
  };

  if (warp == 0) {
    if (elect_one()) {
      constexpr int bk = FP8 ? 128 : 64;
      int n0, w_row, m0, x_col;
      size_t off;
      int issued = 0, s = 0, pre = 0;
      uint32_t ph = 0;
      // weights of the first blocks do not depend on the previous kernel
      if (pair < tiles) {
        locate(pair, n0, w_row, m0, x_col, off);
        pre = nkb < nst ? nkb : nst;
        for (int i = 0; i < pre; ++i) {
          if (rank == 0) mbar_expect_tx(&full[i], 2 * C::STAGE_BYTES);
          tma_load_2d_pair(smem + i * C::STAGE_BYTES, &tmW, dsmem_map(smem_u32(&full[i]), 0), i * bk, w_row + (int)rank * 128);
        }
      }
      if (p.pdl) pdl_wait_prior_grid();
      for (int t = pair; t < tiles && !sh_abort; t += n_pairs) {
        locate(t, n0, w_row, m0, x_col, off);
        for (int kb = 0; kb < nkb; ++kb) {
          const uint32_t bar = dsmem_map(smem_u32(&full[s]), 0);
          uint8_t* stage = smem + s * C::STAGE_BYTES;
          if (issued >= pre) {
            if (issued >= nst && (sh_abort || !mbar_wait(&empty[s], ph ^ 1u))) {
              sh_abort = 1;
              break;
            }
            if (rank == 0) mbar_expect_tx(&full[s], 2 * C::STAGE_BYTES);
            tma_load_2d_pair(stage, &tmW, bar, kb * bk, w_row + (int)rank * 128);
          }
          tma_load_2d_pair(stage + C::A_BYTES, &tmX, bar, x_col + kb * bk, m0 + (int)rank * HALF);
          sh_issued = ++issued;
          if (++s == nst) { s = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (rank == 0 && elect_one()) {
      constexpr uint32_t idesc = FP8 ? umma_idesc_e4m3(256, BN) : umma_idesc_bf16(256, BN);
      int s = 0, consumed = 0, i = 0;
      uint32_t ph = 0;
      for (int t = pair; t < tiles && !sh_abort; t += n_pairs, ++i) {
        const int buf = i & 1;
        if (i >= 2 && !mbar_wait(&acc_empty[buf], ((i >> 1) & 1) ^ 1)) {
          sh_abort = 1;
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb) {
          if (sh_abort || !mbar_wait(&full[s], ph)) {
            sh_abort = 1;
            break;
          }
          tc_fence_after();
          const uint32_t a = smem_u32(smem + s * C::STAGE_BYTES);
          const uint64_t ad = umma_desc_k_sw128(a), bd = umma_desc_k_sw128(a + C::A_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_pair_ss<FP8>(tmem_base + buf * BN, ad + 2 * k, bd + 2 * k, idesc, (kb | k) ? 1u : 0u);
          umma_commit_pair(&empty[s]);
          sh_consumed = ++consumed;
          if (++s == nst) { s = 0; ph ^= 1u; }
        }
        if (!sh_abort) umma_commit_pair(&acc_full[buf]);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2, row = q * 32 + lane;       // tensor memory lanes are open to a warp by its index mod 4
    const int et = (int)threadIdx.x - 64;
    if (p.pdl) pdl_wait_prior_grid();
    int i = 0;
    for (int t = pair; t < tiles; t += n_pairs, ++i) {
      const int buf = i & 1;
      int n0, w_row, m0, x_col;
      size_t off;
      locate(t, n0, w_row, m0, x_col, off);
      // per-token factors of this tile, while its MMAs run
      for (int c = et; c < BN; c += 32 * WIDE_EPI_WARPS) {
        const int m = m0 + c;
        float f = 1.f;
        if (m < p.M) {
          if (p.ssq_in != nullptr) {
            float ss = 0.f;
            for (int k = 0; k < p.ssq_parts; ++k) ss += p.ssq_in[(size_t)k * p.ssq_ld + (size_t)m * p.ssq_mstride];
            f = rsqrtf(ss * p.norm_inv_d + p.norm_eps);
          } else if (FP8 && p.x_scale != nullptr) {
            f = p.x_scale[(size_t)m * p.ssq_mstride];
          }
        }
        s_rstd[buf][c] = f;
      }
      named_bar(1, 32 * WIDE_EPI_WARPS);
      const bool gave_up = !mbar_wait(&acc_full[buf], (i >> 1) & 1);
      if (named_bar_or(1, 32 * WIDE_EPI_WARPS, gave_up)) {   // all or none of the epilogue warps go on
        sh_abort = 1;
        break;
      }
      tc_fence_after();
      const int n = n0 + (int)rank * 128 + row;
      const bool live_n = n < p.N;
      const uint32_t taddr = tmem_base + buf * BN + ((uint32_t)(q * 32) << 16);
      float wsc = 1.f;
      if constexpr (FP8) wsc = live_n ? p.w_scale[n] : 1.f;
#pragma unroll 1
      for (int c0 = half * HALF, it = 0; c0 < (half + 1) * HALF; c0 += 32, ++it) {
        if (m0 + c0 >= p.M) break;                           // the same for all warps of this half
        uint32_t r0[16], r1[16];
        tmem_ld_32x32b_x16(taddr + c0, r0);
        tmem_ld_32x32b_x16(taddr + c0 + 16, r1);
        const int left = p.M - m0 - c0;                      // tokens of this piece
        if constexpr (EPI == EPI_SWIGLU_BF16) {
          // quarters 0, 1 are gate channels and 2, 3 the up channels that belong to them: a gate warp finishes the first
          // sixteen tokens of a piece and hands its values of the others to its partner, which does the same the other way round
          tmem_ld_wait();
          const bool gate = q < 2;
          float* mine = exch + (half * 4 + q) * 16 * 32 + lane;
          const float* theirs = exch + (half * 4 + (q ^ 2)) * 16 * 32 + lane;
          named_bar(2 + half * 2 + (q & 1), 64);             // the partner has read the last piece
#pragma unroll
          for (int j = 0; j < 16; ++j) mine[j * 32] = __uint_as_float(gate ? r1[j] : r0[j]) * wsc;
          named_bar(2 + half * 2 + (q & 1), 64);
          const int ch = (n0 + (int)rank * 128) / 2 + (q & 1) * 32 + lane;
          __nv_bfloat16* out = reinterpret_cast<__nv_bfloat16*>(p.out) + (size_t)(m0 + c0 + (gate ? 0 : 16)) * p.ldo + ch;
          const float* f = &s_rstd[buf][c0 + (gate ? 0 : 16)];
          const int have = left - (gate ? 0 : 16);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float own = __uint_as_float(gate ? r0[j] : r1[j]) * wsc * f[j], other = theirs[j * 32] * f[j];
            const float y = gated_unit<false>(p, gate ? own : other, gate ? other : own);
            if (j < have && ch * 2 < p.N) out[(size_t)j * p.ldo] = __float2bfloat16(y);
          }
        } else if constexpr (EPI == EPI_RESID_F32) {
          float* out = reinterpret_cast<float*>(p.out) + (size_t)(m0 + c0) * p.ldo + off + n;
          float h[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) h[j] = live_n && j < left ? out[(size_t)j * p.ldo] : 0.f;
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (live_n && j < left) h[j] += __uint_as_float(j < 16 ? r0[j & 15] : r1[j & 15]) * wsc * s_rstd[buf][c0 + j];
#pragma unroll
          for (int j = 0; j < 32; ++j)
            if (live_n && j < left) out[(size_t)j * p.ldo] = h[j];
          if (p.hb_out != nullptr) {
            __nv_bfloat16* hb = p.hb_out + (size_t)(m0 + c0) * p.hb_ld + n;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (live_n && j < left) hb[(size_t)j * p.hb_ld] = __float2bfloat16(h[j]);
          }
          if (p.ssq_out != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; ++j) h[j] *= h[j];
            s_sq[it & 1][half][q][lane] = lanes_to_columns(h, lane);
            named_bar(2 + half, 128);
            if (q == 0 && lane < left && n0 + (int)rank * 128 < p.N) {
              const float(*v)[32] = s_sq[it & 1][half];
              p.ssq_out[(size_t)(n0 / 128 + rank) * p.ssq_ld + m0 + c0 + lane] = v[0][lane] + v[1][lane] + v[2][lane] + v[3][lane];
            }
          }
        } else {
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float v = __uint_as_float(j < 16 ? r0[j & 15] : r1[j & 15]) * wsc * s_rstd[buf][c0 + j];
            if constexpr (EPI == EPI_RELU2_BF16) v = v > 0.f ? v * v : 0.f;
            const size_t at = (size_t)(m0 + c0 + j) * p.ldo + off + n;
            if (live_n && j < left) {
              if constexpr (EPI == EPI_STORE_F32) reinterpret_cast<float*>(p.out)[at] = v;
              else reinterpret_cast<__nv_bfloat16*>(p.out)[at] = __float2bfloat16(v);
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(dsmem_map(smem_u32(&acc_empty[buf]), 0));
    }
  }

  __syncthreads();
  if (sh_abort && threadIdx.x == 0) {
    atomicOr(p.status, SMC_ERR_BARRIER_TIMEOUT);
    if (rank == 0)
      for (int i = sh_consumed; i < sh_issued; ++i) (void)mbar_wait(&full[i % nst], (uint32_t)(i / nst) & 1u);
  }
  tc_fence_before();
  cluster_sync();
  if (warp == 1) tmem_dealloc_pair(tmem_base, C::TMEM_COLS);
}

// ---------------------------------------------------------------- host side
template <int BN, int EPI, bool FP8, bool GRP>
static int wide(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmParams& p, cudaStream_t st) {
  using C = WideCfg<BN>;
  auto kern = gemm_wide_kernel<BN, EPI, FP8, GRP>;
  static const int pairs = [&] {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES) != cudaSuccess) return -1;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
    return sms / 2;
  }();
  if (pairs < 1) return -40;
  const long long tiles = (long long)((p.N + 255) / 256) * (GRP ? p.grp.groups : 1) * p.m_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * (tiles < pairs ? tiles : pairs)));
  cfg.blockDim = dim3(WIDE_THREADS);
  cfg.dynamicSmemBytes = C::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.pdl ? 1 : 0;
  CUDA_CHECK_RET(cudaLaunchKernelEx(&cfg, kern, tmW, tmX, p));
  return 0;
}

template <int EPI, bool FP8, bool GRP>
static int wide_bn(int bn, const CUtensorMap& w, const CUtensorMap& x, const GemmParams& p, cudaStream_t st) {
  switch (bn) {
    case 128: return wide<128, EPI, FP8, GRP>(w, x, p, st);
    case 192: return wide<192, EPI, FP8, GRP>(w, x, p, st);
    case 256: return wide<256, EPI, FP8, GRP>(w, x, p, st);
  }
  return -10;
}

int gemm_wide_launch(const CUtensorMap& w, const CUtensorMap& x, const GemmParams& p, int epi, int bn, cudaStream_t st) {
  if (p.fp8) {
    switch (epi) {
      case EPI_BF16: return wide_bn<EPI_BF16, true, false>(bn, w, x, p, st);
      case EPI_SWIGLU_BF16: return wide_bn<EPI_SWIGLU_BF16, true, false>(bn, w, x, p, st);
      case EPI_STORE_F32: return wide_bn<EPI_STORE_F32, true, false>(bn, w, x, p, st);
      case EPI_RESID_F32: return wide_bn<EPI_RESID_F32, true, false>(bn, w, x, p, st);
    }
    return -30;
  }
  if (p.grp.mode == 1) {
    switch (epi) {
      case EPI_BF16: return wide_bn<EPI_BF16, false, true>(bn, w, x, p, st);
      case EPI_STORE_F32: return wide_bn<EPI_STORE_F32, false, true>(bn, w, x, p, st);
    }
    return -33;
  }
  switch (epi) {
    case EPI_BF16: return wide_bn<EPI_BF16, false, false>(bn, w, x, p, st);
    case EPI_SWIGLU_BF16: return wide_bn<EPI_SWIGLU_BF16, false, false>(bn, w, x, p, st);
    case EPI_STORE_F32: return wide_bn<EPI_STORE_F32, false, false>(bn, w, x, p, st);
    case EPI_RESID_F32: return wide_bn<EPI_RESID_F32, false, false>(bn, w, x, p, st);
    case EPI_RELU2_BF16: return wide_bn<EPI_RELU2_BF16, false, false>(bn, w, x, p, st);
  }
  return -11;
}

// Which products take this kernel, and with how many tokens per tile.  Microseconds measured on B200, weight-streaming kernel -> this one
// (with the tile chosen below), N x K:
//   3072 x 2048    256 tokens 13 -> 11    640: 21 -> 12    1408: 36 -> 17    4096: 111 -> 41  (1.27 PFLOP/s)
//   2048 x 2048    256 tokens 12 -> 14    320: 16 -> 14     640: 28 -> 15    4096: 100 -> 34
//   2048 x 8192    320 tokens 26 -> 35    512: 26 -> 36     640: 46 -> 37    4096: 245 -> 119
//   16384 x 2048 (gated)  192 tokens 26 -> 18    640: 70 -> 40    4096: 367 -> 176 (1.56 PFLOP/s)
// Tiles of 128 tokens count the work: below 20 of them, and below 40 where K is longer than 32 blocks, split-K over a cluster keeps more SMs
// busy than one pair per tile does.  Up to 128 tokens the product is bound by reading W, which needs no pairs.
// Outputs that leave as rows of bf16 (bf16, squared relu; 64 bytes a store) cost a pair more: not where half of its 256 rows are empty (32 products of
// 128 x 64 at 1024 tokens 9.6 -> 20.7), nor where 128 x 128 tiles make one round at two CTAs per SM, more than half of it, and K is short (2048 x 256 at
// 2048 tokens 9.1 -> 10.5; at 1024, 8.3 -> 7.2), nor, with up to three blocks of K, for more rounds (8192 x 64 at 1024 tokens 15.2 -> 15.6).
// The width is the one with the least time by rounds of 74 pairs x bytes a CTA pulls per block of K (128 weight rows and half the tokens).
int gemm_wide_tile(int N, int kblocks, int M, int groups, bool rows16) {
  if (M <= 128) return 0;
  const long long slabs = (long long)((N + 255) / 256) * groups, work = slabs * ((M + 127) / 128);
  if (work < 20 || (work < 40 && kblocks > 32)) return 0;
  if (rows16) {
    const long long halves = (N + 127) / 128, tiles = halves * groups * ((M + 127) / 128);
    if (8 * 2 * ((N + 255) / 256) > 9 * halves || (tiles > 160 && (tiles <= 296 ? kblocks <= 32 : kblocks < 4))) return 0;
  }
  int best = 0;
  long long least = 0;
  for (int bn = 256; bn >= 128; bn -= 64) {
    const long long cost = (slabs * ((M + bn - 1) / bn) + 73) / 74 * (128 + bn / 2);
    if (best == 0 || cost < least) { best = bn; least = cost; }
  }
  return best;
}

}  // namespace smc

SMC_API int smc_gemm_wide_tile(int N, int kblocks, int M, int groups, int rows16) { return smc::gemm_wide_tile(N, kblocks, M, groups, rows16 != 0); }
