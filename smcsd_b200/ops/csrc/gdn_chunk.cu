// Chunk-parallel gated delta rule for prompt passes on the 5th-generation tensor cores (tcgen05 + tensor memory), in three launches.
//
// A row's tokens are taken in chunks of 64.  With gc = cumsum(g) inside the chunk, decay[i][j] = exp(gc_i - gc_j),
// L = strict_lower((K beta) K^T * decay) and Tm = (I + L)^-1 (the WY / UT transform of the delta rule), a chunk needs
//     v_w   = Tm (V beta)                 k_cum = Tm (K beta e^gc)
//     v_new = v_w - k_cum S               out   = (Q e^gc) S + lower((Q K^T) * decay) v_new
//     S    <- S e^gc_last + (K e^(gc_last - gc))^T v_new
// Only the last two lines wait for the chunk before.  gdn_prepare does the rest for all chunks at once, one CTA per (chunk, value
// head), three to an SM: operands, G = [K beta ; Q] K^T, the triangular inverse, k_cum.  It leaves 80 KB per chunk in scratch memory,
// tile images that gdn_walk fetches with bulk copies two chunks deep; gdn_gate norms and gates the outputs.  gdn_walk, one CTA per (row, value head), holds the state
// transposed (S^T [dv][dk], fp32) in tensor memory for the whole row; M = 128 throughout, the head dimension on the rows:
//     D     [dv x 64]   = (V beta)^T Tm^T - S^T k_cum^T                               (v_new^T)
//     S^T   [dv x dk]  += v_new^T (K e^(gc_last - gc))
//     out^T [dv x 64]   = S^T (Q e^gc)^T + v_new^T local^T
//   warps 0-3   state: S^T to its bf16 operand and decayed in place (one pass), D to the bf16 operand v_new^T
//   warps 4-7   outputs: tensor memory (two buffers) to the v columns that gdn_prepare has read
//   warp 8      bulk copies        warp 9  MMAs
// so that a chunk costs the chain D -> v_new -> S -> operand.  The norm over dv, the weight and silu(z) are a pass of their own over all
// SMs: on the walk's warps they took 6.6 thousand cycles a chunk, twice the chain.
// Microseconds on B200, 16 heads, one CTA for all of a (row, head) before -> prepare + walk + gate now: three rows of 996 to 1490
// tokens 509 -> 74 + 64 + 14, one of 500 beside eight single tokens 177 -> 29 + 27 + 4.
//
// Operands are bf16 tiles in the 128-byte-swizzled layouts the MMA descriptors expect; accumulation and the state are fp32.  Tm is
// obtained exactly, in fp32: forward substitution on the diagonal blocks, products for the rest.
//
// Math: Qwen3.5 / Qwen3-Next gated delta net (transformers models/qwen3_5/modeling_qwen3_5.py:
// torch_chunk_gated_delta_rule); the reference serves it through its hybrid linear-attention backend
// (smcsd/core/hybrid_multistep_backend.py:47-222).  Built for dk = dv = 128; other head sizes keep the token-serial
// kernel of gdn.cu.  Every mbarrier wait is bounded; a timeout raises a status bit and the CTA unwinds.
#include "common.cuh"

namespace smc {

constexpr int GC = 64;      // tokens per chunk
constexpr int GD = 128;     // dk == dv

struct GdnChunkParams {
  float* conv_out;            // [T][conv_dim] q | k | v channels after conv + SiLU; v becomes the outputs ahead of norm and gate
  const float* proj;          // [T][ldp] mixed | z | b | a
  float* temporal;            // [rows][Hv][dk][dv]
  const int* state_rows;
  const int* tok_off;         // optional (with tok_len): first token and token count of every row
  const int* tok_len;
  const float* dt_bias;
  const float* A_log;
  const __nv_bfloat16* gnorm_w;
  __nv_bfloat16* out;         // [T][Hv * dv]
  uint8_t* scratch;           // [slots * Hv] images of GI_BYTES, behind them [slots * Hv] totals of g
  int slots;                  // chunks there is room for
  int max_len;                // bound of the rows' lengths that the grids were made for
  int conv_dim, ldp, bs, E, Hk, Hv;
  float eps;
  int* status;
  int pdl;
  long long* trace;           // optional [10]: cycles of the first CTA of prepare (0..5, one chunk) and of walk (6..9, all its chunks)
};

// Phase clock of one thread: prepare 0 gates and operands, 1 product G, 2 L and local tiles, 3 triangular solve, 4 product k_cum, 5 its image; walk
// 6 waits for D, 7 state and v_new to their operands, 8 waits for the state, 9 outputs (their own warps).  Nothing in builds without TRACE.
template <bool TRACE>
struct GdnClock {
  long long* to;
  long long mark;
  __device__ __forceinline__ GdnClock(long long* trace, bool me) {
    if constexpr (TRACE) { to = me ? trace : nullptr; mark = clock64(); }
  }
  __device__ __forceinline__ void lap(int slot) {
    if constexpr (TRACE) {
      const long long now = clock64();
      if (to != nullptr) to[slot] += now - mark;
      mark = now;
    }
  }
};

// image of a chunk in scratch memory, also its place in a buffer of gdn_walk
constexpr int GI_VB = 0;                    // [2 panels][64 tokens][128 B]   V beta                  (MN-major A)
constexpr int GI_KC = GI_VB + 16384;        // [128 dk][128 B]                -k_cum^T                (MN-major B)
constexpr int GI_KD = GI_KC + 16384;        // [2][64][128]                   K e^(gc_last - gc)      (MN-major B)
constexpr int GI_QG = GI_KD + 16384;        // [2][64][128]                   Q e^gc                  (K-major B)
constexpr int GI_TM = GI_QG + 16384;        // [64][128 B]                    Tm                      (K-major B)
constexpr int GI_LOC = GI_TM + 8192;        // [64][128 B]                    lower((Q K^T) decay)    (K-major B)
constexpr int GI_BYTES = GI_LOC + 8192;
// shared memory of gdn_prepare
constexpr int GP_X1 = 0;                    // [2 panels][128 rows][128 B]  rows 0..63 K beta, 64..127 Q   (K-major A); then L and X, fp32 [64][64]
constexpr int GP_KT = GP_X1 + 32768;        // [2][64][128]   K                      (K-major B)
constexpr int GP_KBG = GP_KT + 16384;       // [2][64][128]   K beta e^gc            (MN-major A)
constexpr int GP_TM = GP_KBG + 16384;       // [64][128 B]    Tm                     (K-major B)
constexpr int GP_SMEM = GP_TM + 8192;
// shared memory of gdn_walk
constexpr int GW_SB = 2 * GI_BYTES;         // [2][128][128]  S^T as bf16            (K-major A)
constexpr int GW_VNT = GW_SB + 32768;       // [128][128 B]   v_new^T                (K-major A)
constexpr int GW_SMEM = GW_VNT + 16384;

// byte offset of bf16 element `e` of row `r` in a swizzled tile whose 64-element panels hold `rows` rows each
__device__ __forceinline__ uint32_t sw_off(int rows, int r, int e) {
  return (uint32_t)((e >> 6) * rows * 128 + r * 128 + ((((e & 63) >> 3) ^ (r & 7)) << 4) + (e & 7) * 2);
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// eight consecutive elements (one 16-byte chunk) of a row
__device__ __forceinline__ void store8(uint8_t* tile, int rows, int r, int e0, const float* v, float s) {
  *reinterpret_cast<uint4*>(tile + sw_off(rows, r, e0)) =
      make_uint4(pack_bf16(v[0] * s, v[1] * s), pack_bf16(v[2] * s, v[3] * s), pack_bf16(v[4] * s, v[5] * s),
                 pack_bf16(v[6] * s, v[7] * s));
}
// four of them
__device__ __forceinline__ void store4(uint8_t* tile, int rows, int r, int e0, const float4& v, float s) {
  *reinterpret_cast<uint2*>(tile + sw_off(rows, r, e0)) = make_uint2(pack_bf16(v.x * s, v.y * s), pack_bf16(v.z * s, v.w * s));
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

// Bounded wait that gives up as soon as another thread of the CTA has.
__device__ __forceinline__ bool gdn_wait(volatile int& abort, int* status, uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    for (int i = 0; i < 64; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (abort) return false;
    if (clock64() - t0 > SMC_SPIN_CYCLES) {
      atomicOr(status, SMC_ERR_BARRIER_TIMEOUT);
      abort = 1;
      return false;
    }
  }
}

// First chunk of row b: the chunks of the rows before it (called by whole warps).
__device__ __forceinline__ int chunks_before(const GdnChunkParams& p, int b) {
  if (p.tok_len == nullptr) return b * ((p.E + GC - 1) / GC);
  int n = 0;
  for (int i = threadIdx.x & 31; i < b; i += 32) n += (max(p.tok_len[i], 0) + GC - 1) / GC;
  return __reduce_add_sync(0xffffffffu, n);
}

// ---------------------------------------------------------------- every chunk by itself
template <bool TRACE>
__global__ void __launch_bounds__(128, 3) gdn_prepare_kernel(const GdnChunkParams p) {
  extern __shared__ uint8_t gdn_smem_raw[];
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ float s_beta[GC], s_gc[GC];
  const uint32_t raw = smem_u32(gdn_smem_raw);
  uint8_t* sm = gdn_smem_raw + (((raw + 1023u) & ~1023u) - raw);
  if (p.pdl) { pdl_launch_dependents(); pdl_wait_prior_grid(); }
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int b = blockIdx.z, ch = blockIdx.x, vh = blockIdx.y, kh = vh / (p.Hv / p.Hk);
  const int len = p.tok_len ? p.tok_len[b] : p.E;
  if (ch * GC >= len) return;
  const int slot = chunks_before(p, b) + ch;
  if (slot >= p.slots) {
    if (tid == 0) atomicOr(p.status, SMC_ERR_BOUNDS);
    return;
  }
  uint8_t* img = p.scratch + ((size_t)slot * p.Hv + vh) * GI_BYTES;
  const int key_dim = p.Hk * GD, value_dim = p.Hv * GD;
  const int n = min(GC, len - ch * GC);
  const size_t tc0 = (p.tok_off ? (size_t)p.tok_off[b] : (size_t)b * p.E) + (size_t)ch * GC;
  GdnClock<TRACE> clock(p.trace, tid == 0 && b == 0 && ch == 0 && vh == 0);

  if (tid == 0) {
    mbar_init(&bar, 1);
    abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(&tmem_slot, 128);
    tmem_relinquish();
  }
  // ---- gates: g_j, beta_j, gc = cumsum(g) (padding tokens: g = 0, beta = 0, all operands zero) ------------------
  if (tid < GC) {
    float g = 0.f, be = 0.f;
    if (tid < n) {
      const float* pr = p.proj + (tc0 + tid) * p.ldp + p.conv_dim + value_dim;
      const float x = pr[p.Hv + vh] + p.dt_bias[vh];
      const float sp = x > 20.f ? x : log1pf(__expf(x));
      g = -__expf(p.A_log[vh]) * sp;
      be = 1.f / (1.f + __expf(-pr[vh]));
    }
    s_beta[tid] = be;
    // inclusive scan over 64 tokens: two warps, then the second adds the first one's total
    float v = g;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    s_gc[tid] = v;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = tmem_slot, T_G = 0, T_KC = 64;
  const uint32_t lane_off = ((uint32_t)(warp * 32)) << 16;
  if (tid >= 32 && tid < GC) s_gc[tid] += s_gc[31];
  __syncthreads();
  const float gl = s_gc[GC - 1];
  if (tid == 0) reinterpret_cast<float*>(p.scratch + (size_t)p.slots * p.Hv * GI_BYTES)[(size_t)slot * p.Hv + vh] = gl;
  // ---- operands: a warp takes a token's row at a time (four elements per lane, so that rows arrive in whole lines), normalises q
  // and k; tiles of the walk leave for scratch memory
  const float qs = rsqrtf((float)GD);
#pragma unroll 1
  for (int j0 = warp * 16; j0 < warp * 16 + 16; j0 += 8) {
    float4 qv[8], kv[8], vv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const float* row = p.conv_out + (tc0 + j0 + u) * p.conv_dim + lane * 4;
      qv[u] = kv[u] = vv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (j0 + u < n) {
        qv[u] = *reinterpret_cast<const float4*>(row + kh * GD);
        kv[u] = *reinterpret_cast<const float4*>(row + key_dim + kh * GD);
        vv[u] = *reinterpret_cast<const float4*>(row + 2 * key_dim + vh * GD);
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u, e0 = lane * 4;
      const float bj = s_beta[j], gcj = s_gc[j], egc = __expf(gcj), egl = __expf(gl - gcj);
      const float qn = rsqrtf(warp_sum(qv[u].x * qv[u].x + qv[u].y * qv[u].y + qv[u].z * qv[u].z + qv[u].w * qv[u].w) + 1e-6f) * qs;
      const float kn = rsqrtf(warp_sum(kv[u].x * kv[u].x + kv[u].y * kv[u].y + kv[u].z * kv[u].z + kv[u].w * kv[u].w) + 1e-6f);
      store4(sm + GP_X1, 128, 64 + j, e0, qv[u], qn);
      store4(img + GI_QG, 64, j, e0, qv[u], qn * egc);
      store4(sm + GP_X1, 128, j, e0, kv[u], kn * bj);
      store4(sm + GP_KT, 64, j, e0, kv[u], kn);
      store4(sm + GP_KBG, 64, j, e0, kv[u], kn * bj * egc);
      store4(img + GI_KD, 64, j, e0, kv[u], kn * egl);
      store4(img + GI_VB, 64, j, e0, vv[u], bj);
    }
  }
  fence_proxy_async();
  __syncthreads();
  constexpr uint32_t idesc64 = umma_idesc_bf16(128, 64);
  const uint32_t sb = smem_u32(sm);
  clock.lap(0);
  // ---- G = [K beta ; Q] K^T ---------------------------------------------------------------------------------------
  if (tid == 0) {
#pragma unroll
    for (int pan = 0; pan < 2; ++pan)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        umma_bf16_ss(tm + T_G, umma_desc_k_sw128(sb + GP_X1 + pan * 16384) + 2 * k, umma_desc_k_sw128(sb + GP_KT + pan * 8192) + 2 * k,
                     idesc64, (pan | k) ? 1u : 0u);
    umma_commit(&bar);
  }
  bool alive = !__syncthreads_or(!gdn_wait(abort_flag, p.status, &bar, 0));
  tc_fence_after();
  clock.lap(1);
  float* Lf = reinterpret_cast<float*>(sm + GP_X1);                  // the operands of G are done with
  float* Xf = Lf + GC * GC;
  if (alive) {
    // rows 0..63: L[i][j] = G decay below the diagonal (fp32, for the solve); rows 64..127: local attention tile
    const int i = tid & 63;
    const float gci = s_gc[i];
#pragma unroll
    for (int c0 = 0; c0 < GC; c0 += 16) {
      uint32_t r[16];
      tmem_ld_32x32b_x16(tm + T_G + lane_off + c0, r);
      tmem_ld_wait();
      float f[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) {
        const int j = c0 + u;
        const float v = __uint_as_float(r[u]) * __expf(gci - s_gc[j]);
        f[u] = tid < 64 ? (j < i ? v : 0.f) : (j <= i ? v : 0.f);
      }
      if (tid < 64) {
#pragma unroll
        for (int u = 0; u < 16; u += 4)
          *reinterpret_cast<float4*>(Lf + i * GC + c0 + u) = make_float4(f[u], f[u + 1], f[u + 2], f[u + 3]);
      } else {
        store8(img + GI_LOC, 64, i, c0, f, 1.f);
        store8(img + GI_LOC, 64, i, c0 + 8, f + 8, 1.f);
      }
    }
  }
  __syncthreads();
  clock.lap(2);
  if (alive) {
    // ---- Tm = (I + L)^-1, in 32 x 32 blocks: [[A, 0], [C, B]]^-1 = [[A^-1, 0], [-B^-1 C A^-1, B^-1]] --------------
    // (1) threads 0..63 solve the two diagonal blocks by forward substitution, one column per thread (fp32, exact);
    // (2) all threads form M = C A^-1, (3) X21 = -B^-1 M; (4) Tm is written as bf16 rows.  M is parked in the unused
    // upper-right quadrant of X.
    constexpr int HB = GC / 2;
    if (tid < GC) {
      const int blk = tid >> 5, j = tid & 31, o = blk * HB;      // column j of diagonal block blk
      float x[HB];
#pragma unroll
      for (int i = 0; i < HB; ++i) {
        float a0 = (i == j) ? 1.f : 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
        const float* Li = Lf + (o + i) * GC + o;
#pragma unroll
        for (int k = 0; k + 3 < i; k += 4) {
          const float4 l4 = *reinterpret_cast<const float4*>(Li + k);
          a0 = fmaf(-l4.x, x[k], a0);
          a1 = fmaf(-l4.y, x[k + 1], a1);
          a2 = fmaf(-l4.z, x[k + 2], a2);
          a3 = fmaf(-l4.w, x[k + 3], a3);
        }
#pragma unroll
        for (int k = i & ~3; k < i; ++k) a0 = fmaf(-Li[k], x[k], a0);
        x[i] = (a0 + a1) + (a2 + a3);
      }
#pragma unroll
      for (int i = 0; i < HB; ++i) Xf[(o + i) * GC + o + j] = x[i];
    }
    __syncthreads();
    const int r = tid >> 2, c0 = (tid & 3) * 8;                  // every thread: row r, 8 columns of a 32 x 32 product
    {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const float* Cr = Lf + (HB + r) * GC;                      // row r of C = L[32.., 0..32)
#pragma unroll 8
      for (int k = 0; k < HB; ++k) {
        const float c = Cr[k];
        const float4 a0 = *reinterpret_cast<const float4*>(Xf + k * GC + c0);
        const float4 a1 = *reinterpret_cast<const float4*>(Xf + k * GC + c0 + 4);
        acc[0] = fmaf(c, a0.x, acc[0]); acc[1] = fmaf(c, a0.y, acc[1]); acc[2] = fmaf(c, a0.z, acc[2]);
        acc[3] = fmaf(c, a0.w, acc[3]); acc[4] = fmaf(c, a1.x, acc[4]); acc[5] = fmaf(c, a1.y, acc[5]);
        acc[6] = fmaf(c, a1.z, acc[6]); acc[7] = fmaf(c, a1.w, acc[7]);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) Xf[r * GC + HB + c0 + u] = acc[u];          // M[r][c0 + u], parked upper right
    }
    __syncthreads();
    {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const float* Br = Xf + (HB + r) * GC + HB;                 // row r of B^-1 (lower triangular)
#pragma unroll 8
      for (int k = 0; k < HB; ++k) {
        const float bv = Br[k];
        const float4 m0 = *reinterpret_cast<const float4*>(Xf + k * GC + HB + c0);
        const float4 m1 = *reinterpret_cast<const float4*>(Xf + k * GC + HB + c0 + 4);
        acc[0] = fmaf(bv, m0.x, acc[0]); acc[1] = fmaf(bv, m0.y, acc[1]); acc[2] = fmaf(bv, m0.z, acc[2]);
        acc[3] = fmaf(bv, m0.w, acc[3]); acc[4] = fmaf(bv, m1.x, acc[4]); acc[5] = fmaf(bv, m1.y, acc[5]);
        acc[6] = fmaf(bv, m1.z, acc[6]); acc[7] = fmaf(bv, m1.w, acc[7]);
      }
      __syncthreads();                                           // every read of M is done before it is overwritten
#pragma unroll
      for (int u = 0; u < 8; ++u) Xf[(HB + r) * GC + c0 + u] = -acc[u];       // X21
    }
    __syncthreads();
    {
      // Tm rows as bf16: thread (row i, half h) stores 32 columns; the upper-right quadrant is zero
      const int i = tid >> 1, h = tid & 1;
      float f[32];
#pragma unroll
      for (int u = 0; u < 32; ++u) f[u] = (i < HB && h == 1) ? 0.f : Xf[i * GC + h * 32 + u];
#pragma unroll
      for (int u = 0; u < 32; u += 8) {
        store8(sm + GP_TM, 64, i, h * 32 + u, f + u, 1.f);
        store8(img + GI_TM, 64, i, h * 32 + u, f + u, 1.f);
      }
    }
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  clock.lap(3);
  // ---- k_cum^T = (K beta e^gc)^T Tm^T ------------------------------------------------------------------------------
  if (alive && tid == 0) {
    tc_fence_after();
#pragma unroll
    for (int k = 0; k < 4; ++k)
      umma_bf16_ss(tm + T_KC, umma_desc_mn_sw128(sb + GP_KBG + k * 2048, 8192), umma_desc_k_sw128(sb + GP_TM) + 2 * k,
                   idesc64 | (1u << 15), k ? 1u : 0u);
    umma_commit(&bar);
  }
  alive = alive && !__syncthreads_or(!gdn_wait(abort_flag, p.status, &bar, 1));
  tc_fence_after();
  clock.lap(4);
  if (alive) {
#pragma unroll
    for (int c0 = 0; c0 < GC; c0 += 16) {
      uint32_t r[16];
      float f[16];
      tmem_ld_32x32b_x16(tm + T_KC + lane_off + c0, r);
      tmem_ld_wait();
#pragma unroll
      for (int u = 0; u < 16; ++u) f[u] = __uint_as_float(r[u]);
      store8(img + GI_KC, 128, tid, c0, f, -1.f);
      store8(img + GI_KC, 128, tid, c0 + 8, f + 8, -1.f);
    }
  }
  tc_fence_before();
  __syncthreads();
  clock.lap(5);
  if (warp == 0) tmem_dealloc(tm, 128);
}

// ---------------------------------------------------------------- chunk after chunk
constexpr int GW_COPY = 8, GW_MMA = 9, GW_THREADS = 320;

struct GdnWalkShared {
  uint64_t full[2], empty[2], sb_ready, d_done, vn_ready, s_done, o_done[2], o_empty[2];
  uint32_t tmem_slot;
  volatile int abort;
};

template <bool TRACE>
__global__ void __launch_bounds__(GW_THREADS, 1) gdn_walk_kernel(const GdnChunkParams p) {
  extern __shared__ uint8_t gdn_smem_raw[];
  __shared__ GdnWalkShared S;
  const uint32_t raw = smem_u32(gdn_smem_raw);
  uint8_t* sm = gdn_smem_raw + (((raw + 1023u) & ~1023u) - raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(&S.full[i], 1);
      mbar_init(&S.empty[i], 1);
      mbar_init(&S.o_done[i], 1);
      mbar_init(&S.o_empty[i], 4);
    }
    mbar_init(&S.sb_ready, 4);
    mbar_init(&S.d_done, 1);
    mbar_init(&S.vn_ready, 4);
    mbar_init(&S.s_done, 1);
    S.abort = 0;
    fence_barrier_init();
  }
  if (warp == GW_MMA) {
    tmem_alloc(&S.tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (p.pdl) { pdl_launch_dependents(); pdl_wait_prior_grid(); }
  const uint32_t tm = S.tmem_slot, T_S = 0, T_D = 128, T_O = 192;
  const int b = blockIdx.x, vh = blockIdx.y;
  const size_t t0 = p.tok_off ? (size_t)p.tok_off[b] : (size_t)b * p.E;
  const int len = p.tok_len ? p.tok_len[b] : p.E;
  const int slot0 = chunks_before(p, b);
  int n_chunks = len > 0 ? (len + GC - 1) / GC : 0;
  if (slot0 + n_chunks > p.slots) n_chunks = 0;              // gdn_prepare has said so
  if (len > p.max_len) {                                     // chunks behind the bound were not prepared
    if (threadIdx.x == 0) atomicOr(p.status, SMC_ERR_BOUNDS);
    n_chunks = 0;
  }
  const float* totals = reinterpret_cast<const float*>(p.scratch + (size_t)p.slots * p.Hv * GI_BYTES);
  const uint32_t lane_off = ((uint32_t)((warp & 3) * 32)) << 16;
  auto wait = [&](uint64_t* bar, int n) { return gdn_wait(S.abort, p.status, bar, (uint32_t)n & 1u); };
  auto warp_wait = [&](uint64_t* bar, int n) { return __all_sync(0xffffffffu, wait(bar, n)) != 0; };

  if (n_chunks == 0) {
  } else if (warp < 4) {
    // ================================================================= state: thread d owns row d of S^T (column d of S [dk][dv])
    float* Sg = p.temporal + (((size_t)p.state_rows[b] * p.Hv + vh) * GD) * GD;
    const uint32_t tS = tm + T_S + lane_off, tD = tm + T_D + lane_off;
    bool alive = true;
    GdnClock<TRACE> clock(p.trace, tid == 0 && b == 0 && vh == 0);
    for (int ch = 0; ch < n_chunks; ++ch) {
      const float dl = __expf(totals[(size_t)(slot0 + ch) * p.Hv + vh]);
      if (ch > 0) {
        alive = warp_wait(&S.s_done, ch - 1);
        if (!alive) break;
        tc_fence_after();
        clock.lap(8);
      }
      // S^T to its operand, and decayed by this chunk's total in place
#pragma unroll
      for (int c0 = 0; c0 < GD; c0 += 64) {
        uint32_t r[64];
        if (ch == 0) {
#pragma unroll
          for (int i = 0; i < 64; ++i) r[i] = __float_as_uint(Sg[(size_t)(c0 + i) * GD + tid]);
        } else {
#pragma unroll
          for (int i = 0; i < 64; i += 16) tmem_ld_32x32b_x16(tS + c0 + i, *reinterpret_cast<uint32_t(*)[16]>(&r[i]));
          tmem_ld_wait();
        }
#pragma unroll
        for (int i = 0; i < 64; i += 16) {
          float f[16];
          uint32_t g[16];
#pragma unroll
          for (int u = 0; u < 16; ++u) {
            f[u] = __uint_as_float(r[i + u]);
            g[u] = __float_as_uint(f[u] * dl);
          }
          store8(sm + GW_SB, 128, tid, c0 + i, f, 1.f);
          store8(sm + GW_SB, 128, tid, c0 + i + 8, f + 8, 1.f);
          tmem_st_32x32b_x16(tS + c0 + i, g);
        }
      }
      tmem_st_wait();
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.sb_ready);
      clock.lap(7);
      // v_new^T to its operand
      alive = warp_wait(&S.d_done, ch);
      if (!alive) break;
      tc_fence_after();
      clock.lap(6);
#pragma unroll
      for (int c0 = 0; c0 < GC; c0 += 32) {
        uint32_t r[32];
        float f[32];
        tmem_ld_32x32b_x16(tD + c0, *reinterpret_cast<uint32_t(*)[16]>(&r[0]));
        tmem_ld_32x32b_x16(tD + c0 + 16, *reinterpret_cast<uint32_t(*)[16]>(&r[16]));
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; ++i) f[i] = __uint_as_float(r[i]);
#pragma unroll
        for (int i = 0; i < 32; i += 8) store8(sm + GW_VNT, 128, tid, c0 + i, f + i, 1.f);
      }
      fence_proxy_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.vn_ready);
      clock.lap(7);
    }
    if (alive) alive = warp_wait(&S.s_done, n_chunks - 1);
    if (alive) {
      tc_fence_after();
      clock.lap(8);
#pragma unroll 1
      for (int c0 = 0; c0 < GD; c0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(tS + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; ++i) Sg[(size_t)(c0 + i) * GD + tid] = __uint_as_float(r[i]);
      }
    }
  } else if (warp < GW_COPY) {
    // ================================================================= outputs: thread = row of dv
    const int d = (warp & 3) * 32 + lane;
    for (int ch = 0; ch < n_chunks; ++ch) {
      const int buf = ch & 1, n = min(GC, len - ch * GC);
      if (!warp_wait(&S.o_done[buf], ch >> 1)) break;
      tc_fence_after();
      GdnClock<TRACE> clock(p.trace, d == 0 && b == 0 && vh == 0);
      float* dst = p.conv_out + (t0 + (size_t)ch * GC) * p.conv_dim + 2 * p.Hk * GD + vh * GD + d;
      uint32_t r[GC];
#pragma unroll
      for (int c0 = 0; c0 < GC; c0 += 16) tmem_ld_32x32b_x16(tm + T_O + buf * GC + c0 + lane_off, *reinterpret_cast<uint32_t(*)[16]>(&r[c0]));
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&S.o_empty[buf]);
#pragma unroll
      for (int i = 0; i < GC; ++i)
        if (i < n) dst[(size_t)i * p.conv_dim] = __uint_as_float(r[i]);
      clock.lap(9);
    }
  } else if (warp == GW_COPY) {
    // ================================================================= copies
    if (lane == 0) {
      int issued = 0;
      for (int ch = 0; ch < n_chunks; ++ch) {
        const int buf = ch & 1;
        if (ch >= 2 && !wait(&S.empty[buf], (ch >> 1) - 1)) break;
        mbar_expect_tx(&S.full[buf], GI_BYTES);
        const uint8_t* img = p.scratch + ((size_t)(slot0 + ch) * p.Hv + vh) * GI_BYTES;
        for (int at = 0; at < GI_BYTES; at += 16384) bulk_load(sm + buf * GI_BYTES + at, img + at, 16384, &S.full[buf]);
        ++issued;
      }
      // an aborted CTA keeps its shared memory until the copies in flight have landed
      if (S.abort)
        for (int ch = max(0, issued - 2); ch < issued; ++ch) (void)mbar_wait(&S.full[ch & 1], (uint32_t)(ch >> 1) & 1u);
    }
    __syncwarp();
  } else {
    // ================================================================= MMAs
    if (elect_one()) {
      constexpr uint32_t idesc64 = umma_idesc_bf16(128, 64);
      constexpr uint32_t idesc128mn = umma_idesc_bf16(128, 128) | (1u << 16);
      const uint32_t sb = smem_u32(sm), s_op = sb + GW_SB, v_op = sb + GW_VNT;
      for (int ch = 0; ch < n_chunks; ++ch) {
        const int buf = ch & 1;
        const uint32_t im = sb + buf * GI_BYTES, tO = tm + T_O + buf * GC;
        if (!wait(&S.full[buf], ch >> 1)) break;
        // D = (V beta)^T Tm^T, ahead of the state
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16_ss(tm + T_D, umma_desc_mn_sw128(im + GI_VB + k * 2048, 8192), umma_desc_k_sw128(im + GI_TM) + 2 * k, idesc64 | (1u << 15),
                       k ? 1u : 0u);
        if (!wait(&S.sb_ready, ch)) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tm + T_D, umma_desc_k_sw128(s_op + (k >> 2) * 16384) + 2 * (k & 3), umma_desc_mn_sw128(im + GI_KC + k * 2048, 8192),
                       idesc64 | (1u << 16), 1u);
        umma_commit(&S.d_done);
        if (ch >= 2 && !wait(&S.o_empty[buf], (ch >> 1) - 1)) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ss(tO, umma_desc_k_sw128(s_op + (k >> 2) * 16384) + 2 * (k & 3), umma_desc_k_sw128(im + GI_QG + (k >> 2) * 8192) + 2 * (k & 3),
                       idesc64, k ? 1u : 0u);
        if (!wait(&S.vn_ready, ch)) break;
        tc_fence_after();
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_bf16_ss(tm + T_S, umma_desc_k_sw128(v_op) + 2 * k, umma_desc_mn_sw128(im + GI_KD + k * 2048, 8192), idesc128mn, 1u);
        umma_commit(&S.s_done);                              // and all reads of the operand S^T
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_ss(tO, umma_desc_k_sw128(v_op) + 2 * k, umma_desc_k_sw128(im + GI_LOC) + 2 * k, idesc64, 1u);
        umma_commit(&S.o_done[buf]);
        umma_commit(&S.empty[buf]);
      }
    }
    __syncwarp();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == GW_MMA) tmem_dealloc(tm, 512);
}

// ---------------------------------------------------------------- gated RMSNorm: a warp per token and head, four at a time
constexpr int GG_TOKENS = 32;       // of a CTA: eight warps, four tokens each

__global__ void __launch_bounds__(256) gdn_gate_kernel(const GdnChunkParams p) {
  if (p.pdl) { pdl_launch_dependents(); pdl_wait_prior_grid(); }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.z, vh = blockIdx.y;
  const int len = p.tok_len ? p.tok_len[b] : p.E, j0 = blockIdx.x * GG_TOKENS + warp * 4;
  if (j0 >= len) return;
  const size_t t0 = (p.tok_off ? (size_t)p.tok_off[b] : (size_t)b * p.E) + j0;
  const float* op = p.conv_out + t0 * p.conv_dim + 2 * p.Hk * GD + vh * GD + lane * 4;
  const float* zp = p.proj + t0 * p.ldp + p.conv_dim + vh * GD + lane * 4;
  float4 o[4], z[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    o[u] = z[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j0 + u < len) {
      o[u] = *reinterpret_cast<const float4*>(op + (size_t)u * p.conv_dim);
      z[u] = *reinterpret_cast<const float4*>(zp + (size_t)u * p.ldp);
    }
  }
  const float w[4] = {__bfloat162float(p.gnorm_w[lane * 4]), __bfloat162float(p.gnorm_w[lane * 4 + 1]),
                      __bfloat162float(p.gnorm_w[lane * 4 + 2]), __bfloat162float(p.gnorm_w[lane * 4 + 3])};
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (j0 + u >= len) break;
    const float ss = warp_sum(o[u].x * o[u].x + o[u].y * o[u].y + o[u].z * o[u].z + o[u].w * o[u].w);
    const float rs = rsqrtf(ss / (float)GD + p.eps);
    auto fin = [&](float ov, float w, float zv) {
      const float y = __bfloat162float(__float2bfloat16(ov * rs));
      return y * w * (zv / (1.f + __expf(-zv)));
    };
    *reinterpret_cast<uint2*>(p.out + (t0 + u) * (size_t)(p.Hv * GD) + vh * GD + lane * 4) =
        make_uint2(pack_bf16(fin(o[u].x, w[0], z[u].x), fin(o[u].y, w[1], z[u].y)),
                   pack_bf16(fin(o[u].z, w[2], z[u].z), fin(o[u].w, w[3], z[u].w)));
  }
}

static int launch_gdn(void (*kern)(const GdnChunkParams), dim3 grid, int threads, size_t smem, const GdnChunkParams& p, cudaStream_t st) {
  CUDA_CHECK_RET(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = p.pdl ? 1 : 0;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  CUDA_CHECK_RET(cudaLaunchKernelEx(&cfg, kern, p));
  return 0;
}

}  // namespace smc

// Scratch bytes of smc_gdn_chunked for `slots` chunks: rows of T tokens in all take at most T / 64 + rows of them.
SMC_API long long smc_gdn_scratch_bytes(int slots, int Hv) { return (long long)slots * Hv * (smc::GI_BYTES + 4); }

// Delta rule + gated RMSNorm of prompt rows, chunk-parallel (the conv + SiLU pass must have filled conv_out).
// Rows as in smc_gdn_varlen, none longer than max_len (such a row raises SMC_ERR_BOUNDS and its state stays); dk = dv = 128 only; the v columns of conv_out are written over.  scratch: smc_gdn_scratch_bytes, 16-byte aligned.
SMC_API int smc_gdn_chunked(float* conv_out, const float* proj, int ldp, float* temporal, const int* state_rows,
                            const float* dt_bias, const float* A_log, const void* gnorm_w, void* out, int bs, int E,
                            const int* tok_off, const int* tok_len, int max_len, int Hk, int Hv, int dk, int dv, float eps,
                            void* scratch, int slots, int* status, long long* trace, int pdl, cudaStream_t st) {
  using namespace smc;
  if ((tok_off == nullptr) != (tok_len == nullptr)) return -103;
  if (tok_len == nullptr) max_len = E;
  if (bs <= 0 || max_len <= 0) return 0;
  if (dk != GD || dv != GD || Hv % Hk) return -104;
  if (scratch == nullptr || slots < 1 || (reinterpret_cast<uintptr_t>(scratch) & 15) || Hv > 65535 || bs > 65535) return -106;
  GdnChunkParams p;
  p.conv_out = conv_out; p.proj = proj; p.temporal = temporal; p.state_rows = state_rows; p.tok_off = tok_off;
  p.tok_len = tok_len; p.dt_bias = dt_bias; p.A_log = A_log; p.gnorm_w = (const __nv_bfloat16*)gnorm_w;
  p.out = (__nv_bfloat16*)out; p.scratch = (uint8_t*)scratch; p.slots = slots; p.max_len = max_len;
  p.conv_dim = 2 * Hk * dk + Hv * dv; p.ldp = ldp; p.bs = bs; p.E = E; p.Hk = Hk; p.Hv = Hv;
  p.eps = eps; p.status = status; p.pdl = pdl; p.trace = trace;
  if ((p.conv_dim % 4) != 0 || (ldp % 4) != 0 || ((reinterpret_cast<uintptr_t>(conv_out) | reinterpret_cast<uintptr_t>(proj)) & 15) ||
      (reinterpret_cast<uintptr_t>(out) & 7))
    return -105;                                                   // float4 row loads, 8-byte row stores
  const int rc = launch_gdn(trace ? gdn_prepare_kernel<true> : gdn_prepare_kernel<false>, dim3((max_len + GC - 1) / GC, Hv, bs), 128, GP_SMEM + 1024, p, st);
  if (rc) return rc;
  const int rw = launch_gdn(trace ? gdn_walk_kernel<true> : gdn_walk_kernel<false>, dim3(bs, Hv), GW_THREADS, GW_SMEM + 1024, p, st);
  return rw ? rw : launch_gdn(gdn_gate_kernel, dim3((max_len + GG_TOKENS - 1) / GG_TOKENS, Hv, bs), 256, 0, p, st);
}
