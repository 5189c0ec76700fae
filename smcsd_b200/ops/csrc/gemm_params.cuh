// What the tcgen05 GEMM kernels share: epilogues, launch parameters, links to other ranks, norms and groups.
#pragma once
#include "common.cuh"
#include "sample_core.cuh"

namespace smc {

enum { EPI_PARTIAL_F32 = 0, EPI_BF16 = 1, EPI_SWIGLU_BF16 = 2, EPI_STORE_F32 = 3, EPI_RESID_F32 = 4, EPI_RS_F32 = 5,
       EPI_SWIGLU_SPLIT = 6,     // 6: SwiGLU after a split-K reduction inside the cluster
       EPI_LMHEAD = 7,           // 7: lm_head: every slab is reduced to per-row sampling partials, logits are not stored
       EPI_RELU2_BF16 = 8,       // 8: squared relu
       EPI_RELU2_SPLIT = 9 };    // 9: squared relu after a split-K reduction inside the cluster
// Epilogues that reduce split-K inside a thread-block cluster (of one CTA, if K is not split).
__host__ __device__ constexpr bool epi_clustered(int epi) {
  return epi == EPI_STORE_F32 || epi == EPI_RESID_F32 || epi == EPI_RS_F32 || epi == EPI_SWIGLU_SPLIT || epi == EPI_RELU2_SPLIT;
}

// Tensor-parallel links of one GEMM.  Consumer side (all-gather -> GEMM): peers store their
// activation rows into this GPU's buffer and bump a counter here; the TMA producer waits for the
// counter before it fetches activations from local memory.  Producer side (GEMM -> reduce-scatter):
// the epilogue stores each reduced token row straight into the owning rank's receive buffer over
// NVLink (plain peer stores) and bumps that rank's counter.  Counters only grow; the value to wait
// for is derived from a device-resident epoch so captured graphs work unchanged on every replay.
struct TpLink {
  const unsigned long long* ag_flag;   // null: no all-gather wait
  const long long* epoch;              // device epoch, first use has epoch 1
  long long ag_uses, ag_idx, ag_inc;   // wait for ((epoch-1)*uses + idx + 1) * inc
  unsigned long long peer_base[8];     // symmetric-heap base address on every rank
  long long rs_off, rs_flag_off;       // byte offsets of the receive buffer / its counter in the heap
  int tp, rank, rows_per_rank, pad;
  int* arrive;                         // local arrival counter of this call site (self-resetting)
};

// Several products of one shape in one launch.
struct GroupLink {
  int mode;                 // 0: off, 1: batched (groups x all M rows), 2: tiled (rows of a group given by the table)
  int groups;
  int w_rows;               // weight rows between groups
  int x_cols, out_cols;     // activation / output columns between groups (batched)
  const int4* tiles;        // tiled: {group, first row, end row, -}; entries past the used ones have first == end
  int max_tiles, bn;        // tiled: table length, rows per tile (the token-tile width the table was made for)
  int act;                  // gated epilogue: 0 silu(g) * u, 1 clamped: min(g, limit) * sigmoid(slope g) * (clamp(u) + 1),
                            // 2 gelu(g) * u in the tanh form
  float limit, slope;
};

struct GemmParams {
  int N, K, M;          // weight rows (of a group), reduction length, token rows
  int kblocks;          // ceil(K / 64)
  int m_tiles;          // token tiles (grid x = weight slabs * m_tiles)
  int stages;           // 3 selects the lean build of the 128-token tile (host-side choice only)
  int splits;
  void* out;            // fp32 [splits, M, N] | bf16 [M, ldo]
  int ldo;
  int* status;
  int pdl;              // 1: wait for the previous grid only before touching activations
  TpLink tp;
  // RMSNorm folded into the GEMMs (norm weights are pre-multiplied into W):
  //   consumer side: the activation operand is the raw bf16 residual stream; every output column (token) is scaled
  //     by rstd = rsqrt(sum_p ssq_in[p, m] / norm_d + eps) in the epilogue;
  //   producer side (residual epilogue): besides h += X W^T it writes the bf16 copy of the new rows and the
  //     sum of squares of its 128 columns per token into ssq_out[n_tile, m], summed later in a fixed order.
  const float* ssq_in;
  int ssq_parts, ssq_ld, ssq_mstride;     // token of output row m is ssq column m * ssq_mstride
  float norm_inv_d, norm_eps;
  float* ssq_out;
  __nv_bfloat16* hb_out;
  int hb_ld;
  // lm_head with fused sampling / scoring (EPI_LMHEAD): out = RowPartial [M, slabs]
  SampleArgs samp;
  // FP8 operands: e4m3 bytes, value = byte * scale; w_scale per weight row, x_scale per token row (null: 1)
  int fp8;
  const float* w_scale;
  const float* x_scale;
  GroupLink grp;
  float act_a, act_b;   // gated epilogue: g / (1 + exp(-g (act_a + act_b g^2))) u, silu with 1 and 0, gelu (tanh form) with the constants below
};
constexpr float GELU_A = 1.5957691216057308f, GELU_B = 1.5957691216057308f * 0.044715f;      // 2 sqrt(2 / pi), times its cubic's factor

template <bool GRP>
__device__ __forceinline__ float gated_unit(const GemmParams& p, float g, float u) {
  if (GRP && p.grp.act == 1) {
    g = fminf(g, p.grp.limit);
    u = fminf(fmaxf(u, -p.grp.limit), p.grp.limit);
    return g / (1.0f + __expf(-p.grp.slope * g)) * (u + 1.0f);
  }
  return g / (1.0f + __expf(-g * fmaf(p.act_b * g, g, p.act_a))) * u;
}

// Launches the kernel for wide batches (gemm_wide.cu); the maps' boxes are 128 weight rows and bn / 2 token rows.
int gemm_wide_launch(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmParams& p, int epi, int bn, cudaStream_t stream);
// Token-tile width of that kernel for a product (kblocks: blocks of 128 bytes of K; rows16: plain bf16 outputs), or 0 where the
// weight-streaming kernel is the faster one.
int gemm_wide_tile(int N, int kblocks, int M, int groups, bool rows16);

}  // namespace smc
