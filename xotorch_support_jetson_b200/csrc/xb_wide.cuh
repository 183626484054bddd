// Linear of more than 128 token rows: y[T,N] (bf16) = x[T,K] W[N,K]^T with the fused prompt epilogues.
//
//   D[128 tokens x BN features] (fp32, TMEM) += A[128 x 64] (x, smem) * B[BN x 64]^T (W, smem)
//
// Same pipeline as the decode Linear (xb_gemm.cuh): one thread feeds each operand by TMA, one issues tcgen05.mma, four warps
// drain TMEM, persistent over tiles with two accumulators.  What varies is how the tiles cover the chip:
//   CG = 2  a pair of CTAs works on one tile of 2 RM rows (cta_group::2): each stages its own token rows and HALF of the
//           weight rows, with 128 rows 32 KB instead of 48 KB a k-block at BN = 256.
//   RM = 64 pairs on a tile of 128 rows, 64 a CTA.  A k-block takes as long as its operands need into the SM (64 bytes a clock), so what counts is how
//           many SMs share them: 3072 features of 373 rows are 72 tiles of 128 x 128 on 72 SMs at 32 KB a k-block, or the same 72 tiles on 72 pairs
//           at 16 KB a CTA.  Back to back, us: 373 rows x 8192 -> 3072 34.7 -> 22.1, x 3072 -> 3072 16.3 -> 12.0, 192 rows x 18944 -> 3584 76.8 -> 42.9;
//           2048 rows x 8192 -> 3072 93.9 (192 columns) -> 84.4 (256 columns on pairs of 64 rows).
//   BN      128, 192 or 256 features a tile, by what fills the SMs evenly.
// Every variant sums K in the same order, k-block by k-block into one accumulator, so a row's numbers depend neither on the tile
// it falls into nor on what else the step carries: a prompt in portions has the bits of the whole.  (K in two or four parts over a
// cluster was faster below 512 rows and gave that up.)
#pragma once
#include "xb_gemm.cuh"

template <int BN, int CG, int RM>
struct WideCfg {
  static_assert(RM == 128 || (RM == 64 && CG == 2), "token rows of a CTA");
  static constexpr int BROWS = BN / CG;                       // weight rows this CTA stages
  static constexpr int BOX = BROWS % 128 == 0 ? 128 : 64;     // rows of one TMA box (divides 128: a box stays in its weight tile)
  static constexpr int A_BYTES = RM * 64 * 2;
  static constexpr int B_BYTES = BROWS * 64 * 2;
  static constexpr int KS = RM == 64 || BN <= 128 ? 2 : 1;    // k-blocks of a stage: small tiles halve the barrier round trips (192 rows x 8192 -> 3072 28.8 -> 21.1 us; four a stage 21.6)
  static constexpr int STAGES_RAW = (216 * 1024) / (KS * (A_BYTES + B_BYTES));
  static constexpr int STAGES = STAGES_RAW > 8 ? 8 : STAGES_RAW;
  static constexpr int ACC_STAGES = 2;
  // A pair with 64 token rows a CTA keeps its rows' lower half of the columns in lanes 0-63 of tensor memory, the upper in lanes 64-127.
  static constexpr int COLS = RM == 64 ? BN / 2 : BN;         // columns a lane holds
  static constexpr int TM_RAW = ACC_STAGES * COLS;
  static constexpr int TM_COLS = TM_RAW <= 128 ? 128 : TM_RAW <= 256 ? 256 : 512;
  static constexpr int ACC_COLS = TM_COLS / ACC_STAGES;
  static constexpr int PAIRS = COLS / 32;                       // column pairs (two chunks of 16) a thread drains
  static constexpr int RING_BYTES = STAGES * KS * (A_BYTES + B_BYTES);
  static constexpr int SMEM_BYTES = RING_BYTES + 1024 + 256;
  static_assert(BROWS % BOX == 0, "tile");
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_aligned() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of this CTA's shared address `a` in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_map(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// TMA load into this CTA whose bytes are counted by a barrier of the CTA pair (`bar`: shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* m, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(m), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
template <int CG>
__device__ __forceinline__ void wide_tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  if (CG == 1) {
    tmem_alloc(dst_smem, cols);
  } else {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
}
template <int CG>
__device__ __forceinline__ void wide_tmem_dealloc(uint32_t taddr, uint32_t cols) {
  if (CG == 1) tmem_dealloc(taddr, cols);
  else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// completion of the MMAs issued so far arrives at `bar`, for a pair at the same barrier of both CTAs
template <int CG>
__device__ __forceinline__ void wide_commit(uint64_t* bar) {
  if (CG == 1) {
    tc_commit(bar);
  } else {
    const uint16_t both = 3;
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"(both) : "memory");
  }
}
template <int CG>
__device__ __forceinline__ void wide_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  if (CG == 1) {
    tc_mma_bf16(tmem_d, desc_a, desc_b, idesc, accumulate);
  } else {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
  }
}

// ---- epilogues: one thread = one token row, two chunks of 16 columns at a time ----
// The chunks of pair p: neighbours (gate beside up, interleaved rotation), or for the half-split rotation the two chunks
// whose entries turn together, half a head apart.
__device__ __forceinline__ void wide_pair_cols(const GemmArgs& g, int p, int& c0, int& c1) {
  if (g.epi == XB_EPI_QKV && g.rope_kind != 0) {
    const int per = g.head_dim >> 5, head = p / per, j = p - head * per;
    c0 = head * g.head_dim + j * 16;
    c1 = c0 + (g.head_dim >> 1);
  } else {
    c0 = p * 32;
    c1 = c0 + 16;
  }
}
__device__ __forceinline__ void wide_bias_round(const GemmArgs& g, int n0, float* x) {
#pragma unroll
  for (int j = 0; j < 16; ++j) {   // nn.Linear rounding point: bf16(acc + bias)
    float a = x[j];
    if (g.bias != nullptr) a += bf2f(g.bias[n0 + j]);
    x[j] = rbf(a);
  }
}
__device__ __forceinline__ void wide_store_plain(const GemmArgs& g, int t, int n0, float* x) {
  if (n0 >= g.b_rows) return;
  bf16* dst = reinterpret_cast<bf16*>(g.out) + (long long)t * g.ld_out + n0;
  if (g.bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (n0 + j < g.b_rows) x[j] += bf2f(g.bias[n0 + j]);
  }
  if (n0 + 16 <= g.b_rows && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
    epi_store16(dst, x);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (n0 + j < g.b_rows) dst[j] = f2bf(x[j]);
  }
}
// What the fused-QKV epilogue needs of a token row beside its sums.  A block of a prompt of a few hundred rows has one tile, so what its epilogue
// waits for adds to the Linear: the row's place in the cache (three dependent lookups) is found while the products run, the rotation factors of a
// column pair (32 neighbouring floats) arrive while the pair before is written.  Looked up where they were used, the fused projection of
// 373 rows x 3072 -> 5120 took 27 us cold, the plain one of 3072 columns 19; seven 3B layers of such a prompt 995 -> 973 us in all.
struct WideQkvRow {
  long long kv;       // element offset of (page, head 0, place in the page) in a pool
  float cs[32];       // (cos, sin) of the pair at hand
};
__device__ __forceinline__ long long wide_kv_row(const GemmArgs& g, int t, int pos) {
  const int slot = g.seq_slot[g.tok_seq[t]], block = pos / g.page_tokens;
  const int page = g.page_table[(long long)slot * g.max_pages + block];
  return ((long long)page * g.n_kv_heads * g.page_tokens + (pos - block * g.page_tokens)) * g.head_dim;
}
// the factors of the pair whose first column is n0; columns that turn in no head load nothing
__device__ __forceinline__ void wide_rope_load(const GemmArgs& g, int pos, int n0, float* cs) {
  const int hd = g.head_dim, head = hd == 128 ? n0 >> 7 : n0 >> 6, e0 = n0 - head * hd;   // head_dim is 64 or 128, a pair lies in one head
  if (head >= g.n_heads + g.n_kv_heads) return;
  const float4* src = reinterpret_cast<const float4*>(g.rope + (long long)pos * hd + (g.rope_kind != 0 ? 2 * e0 : e0));
#pragma unroll
  for (int i = 0; i < 8; ++i) *reinterpret_cast<float4*>(cs + 4 * i) = src[i];
}
// where 16 elements [e, e + 16) of fused-QKV head `head` of token row t go: q buffer or the paged cache
__device__ __forceinline__ bf16* wide_qkv_dst(const GemmArgs& g, int t, long long kv, int head, int e) {
  const int H = g.n_heads, KV = g.n_kv_heads, hd = g.head_dim;
  if (head < H) return g.q_out + ((long long)t * H + head) * hd + e;
  const bool k = head < H + KV;
  return (k ? g.k_pool : g.v_pool) + kv + (long long)(head - (k ? H : H + KV)) * g.page_tokens * hd + e;
}
// x0 / x1: fp32 sums of the columns n0.. and n1.. of token row t
__device__ __forceinline__ void wide_emit(const GemmArgs& g, int t, const WideQkvRow& r, int n0, int n1, float* x0, float* x1) {
  if (t >= g.a_rows) return;
  if (g.epi == XB_EPI_SILU) {
    // gate/up rows are interleaved in blocks of 16 features: act = bf16(bf16(silu(gate)) * up).  The exact division's branches made a tile's epilogue of
    // four warps longer than its products (373 rows x 3072 -> 2 x 8192 43.1 us, without 39.0).  __fdividef has none and is off by two units in the last place; over a
    // quarter of the denominator, which keeps it below 2^126 where __fdividef would give 0, every one of the 65536 gates that a bf16 can be rounds to the bf16 of
    // the exact quotient.
    if (n0 >= g.b_rows) return;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float gg = rbf(x0[j]), uu = rbf(x1[j]);
      x0[j] = rbf(__fdividef(0.25f * gg, fmaf(expf(-gg), 0.25f, 0.25f))) * uu;
    }
    epi_store16(reinterpret_cast<bf16*>(g.out) + (long long)t * g.ld_out + (n0 >> 1), x0);
  } else if (g.epi == XB_EPI_QKV) {
    if (n0 >= g.b_rows) return;
    const int hd = g.head_dim, half = hd >> 1, turned = g.n_heads + g.n_kv_heads;
    wide_bias_round(g, n0, x0);
    if (n1 < g.b_rows) wide_bias_round(g, n1, x1);
    const int h0 = hd == 128 ? n0 >> 7 : n0 >> 6, e0 = n0 - h0 * hd;
    if (g.rope_kind != 0) {
      if (h0 < turned) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float cc = rbf(r.cs[2 * j]), ss = rbf(r.cs[2 * j + 1]);
          const float a = x0[j], b = x1[j];
          x0[j] = __fadd_rn(rbf(__fmul_rn(a, cc)), rbf(__fmul_rn(-b, ss)));
          x1[j] = __fadd_rn(rbf(__fmul_rn(b, cc)), rbf(__fmul_rn(a, ss)));
        }
      }
      bf16* dst = wide_qkv_dst(g, t, r.kv, h0, e0);
      epi_store16(dst, x0);
      epi_store16(dst + half, x1);
    } else {
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float* x = c == 0 ? x0 : x1;
        const float* cs = r.cs + 16 * c;
        if ((c == 0 ? n0 : n1) >= g.b_rows) break;
        if (h0 < turned) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float a = x[2 * j], b = x[2 * j + 1];
            x[2 * j] = __fsub_rn(__fmul_rn(a, cs[2 * j]), __fmul_rn(b, cs[2 * j + 1]));
            x[2 * j + 1] = __fadd_rn(__fmul_rn(b, cs[2 * j]), __fmul_rn(a, cs[2 * j + 1]));
          }
        }
        epi_store16(wide_qkv_dst(g, t, r.kv, h0, e0 + 16 * c), x);
      }
    }
  } else {
    wide_store_plain(g, t, n0, x0);
    wide_store_plain(g, t, n1, x1);
  }
}

// ---- the feed-forwards of hybrid models (ACT = 1): gate and up of the same 128 features are the two halves of a 256-column tile, so the activation leaves
// from the epilogue in one piece and the matrix of gate and up rows is never written.  1800 rows x 2048 -> 2 x 8192, us: 111.5 with a kernel that read it,
// 97.6 from the epilogue (the products alone 91.2), experts 106.8 -> 95.6; 192 rows 26.9 -> 20.8, all with approximate quotients; the exact ones below cost three
// layers of bibevik-1b at 1500 rows 2 us of 1315.
// Four warps finish a tile while the next one is multiplied; with the division's branches, one an element, they took longer than that (110.7 us).  Results have the
// bits of hy_glu_vec_kernel and hy_moe_act_vec_kernel, so a row's do not hang on which of the two its step takes; the divisions are made without branches: 1 / d by one Newton step on the approximate reciprocal, which for every d from 1 to 2^126 is the correctly rounded one
// (all 126 * 2^23 of them compared), and from it a / d = q + (a - d q) / d with q = a / d rounded (Markstein 1990), correctly rounded as well.  Sixteen
// elements of which one is beyond `WIDE_NEAR` (d could leave that range, or a / d the normal numbers) take the divisions themselves.
#define WIDE_NEAR 32.f
__device__ __forceinline__ float wide_recip(float d) {
  const float r = __fdividef(1.0f, d);
  return fmaf(r, fmaf(-d, r, 1.0f), r);
}
__device__ __forceinline__ bool wide_near(const float* x) {
  float far = 0.f;
#pragma unroll
  for (int j = 0; j < 16; ++j) far = fmaxf(far, fabsf(x[j]));
  return far < WIDE_NEAR;
}
// first gate row (or up row) of the 128 features of tile tb
__device__ __forceinline__ int wide_glu_row(const GemmArgs& g, int tb, bool up) {
  const int i = tb * 128, routed = g.glu_e * g.glu_f;
  if (i >= routed) return routed + i + (up ? g.glu_sf : 0);
  const int e = i / g.glu_f;
  return e * g.glu_f + i + (up ? g.glu_f : 0);
}
// x0 / x1: fp32 sums of 16 gate and 16 up rows from n0 / n1 on, routing weight w; features f0 ..  The choice of the activation stands outside the unrolled
// loops: inside, three activations sixteen times over ran out of the instruction cache (211 us).
__device__ __forceinline__ void wide_emit_glu(const GemmArgs& g, int t, int f0, int n0, int n1, float w, bool shared, float* x0, float* x1) {
  if (t >= g.a_rows) return;
  const float limit = shared ? g.glu_limit_s : g.glu_limit;
  const bool on_input = g.glu_on_input && !shared;
#pragma unroll
  for (int j = 0; j < 16; ++j) { x0[j] = rbf(x0[j]); x1[j] = rbf(x1[j]); }   // what the Linear hands on is bf16, here as in steps of other kernels
  if (g.glu_bias != nullptr) {
#pragma unroll
    for (int j = 0; j < 16; ++j) { x0[j] += g.glu_bias[n0 + j]; x1[j] += g.glu_bias[n1 + j]; }
  }
  if (on_input) {   // (w h) W^T = w (h W^T)
#pragma unroll
    for (int j = 0; j < 16; ++j) { x0[j] *= w; x1[j] *= w; }
  }
  if (w == 0.f && !shared) {         // an expert that the token does not use
#pragma unroll
    for (int j = 0; j < 16; ++j) x0[j] = 0.f;
  } else if (g.glu_act == XB_ACT_GEGLU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) x0[j] = hy_gelu_tanh(x0[j]) * x1[j];
  } else if (g.glu_act == XB_ACT_SWIGLU) {
    if (wide_near(x0)) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float d = 1.0f + expf(-x0[j]), r = wide_recip(d), q = x0[j] * r;
        x0[j] = fmaf(fmaf(-d, q, x0[j]), r, q) * x1[j];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) x0[j] = hy_silu(x0[j]) * x1[j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) x0[j] = fminf(x0[j], limit);
    if (wide_near(x0)) {
#pragma unroll
      for (int j = 0; j < 16; ++j) x0[j] = x0[j] * wide_recip(1.0f + expf(-(1.702f * x0[j]))) * (fminf(fmaxf(x1[j], -limit), limit) + 1.0f);
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) x0[j] = hy_glu_clamp(x0[j], x1[j], limit);
    }
  }
  if (!on_input && w != 1.f) {
#pragma unroll
    for (int j = 0; j < 16; ++j) x0[j] *= w;
  }
  epi_store16(reinterpret_cast<bf16*>(g.out) + (long long)t * g.ld_out + f0, x0);
}
__device__ __forceinline__ void wide_emit_relu2(const GemmArgs& g, int t, int n0, float* x) {
  if (t >= g.a_rows || n0 >= g.b_rows) return;
#pragma unroll
  for (int j = 0; j < 16; ++j) { const float v = fmaxf(rbf(x[j]), 0.f); x[j] = v * v; }
  epi_store16(reinterpret_cast<bf16*>(g.out) + (long long)t * g.ld_out + n0, x);
}

// Roles are entered by elect.sync, not by lane == 0, and the two operands have a producer thread each: one thread doing
// everything under `lane == 0` spent 0.35 us a k-block whatever the tile (a 128 x 64 tile took as long as 128 x 256), most of
// it issuing.  4096^3, CUDA events: 256x256 pair 103 -> 94 us, 128x256 107 -> 103, 128x128 166 -> 116, 128x64 306 -> 202.
template <int BN, int CG, int RM, int ACT = 0>
__global__ void __launch_bounds__(224, 1)
xb_wide_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, GemmArgs g) {
  using Cfg = WideCfg<BN, CG, RM>;
  constexpr int STAGES = Cfg::STAGES, KS = Cfg::KS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + STAGES * KS * Cfg::A_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::RING_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = CG > 1 ? cluster_rank() : 0;
  constexpr int ROWS = RM * CG;                         // token rows of a tile
  const int a_units = (g.a_rows + ROWS - 1) / ROWS;
  const int n_units = a_units * g.b_tiles;
  const int u0 = blockIdx.x / CG, u_step = gridDim.x / CG;

  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    if (lane == 0) {
      for (int i = 0; i < STAGES; ++i) {
        mbar_init(&full_bar[i], 2);   // one arrival (with its byte count) per producer
        mbar_init(&empty_bar[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&tfull_bar[i], 1);
        mbar_init(&tempty_bar[i], 4 * CG);
      }
      fence_mbar_init();
    }
    __syncwarp();
    wide_tmem_alloc<CG>(tmem_slot, Cfg::TM_COLS);
  }
  tc_fence_before();
  __syncthreads();
  if (CG > 1) cluster_sync_aligned();   // barriers of the peer are ready too
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  if (warp == 0 || warp == 6) {
    // ===================== TMA producers: warp 0 weights, warp 6 activations =====================
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      const uint32_t pair_bar = CG == 2 ? cluster_map(smem_u32(full_bar), 0) : 0;   // a pair counts the bytes of both CTAs at the first one's barriers
      auto expect = [&](uint32_t bytes) {
        if (CG == 1) mbar_expect_tx(&full_bar[stage], bytes);
        else if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * bytes);
      };
      auto load = [&](void* dst, const CUtensorMap* m, int c0, int c1) {
        if (CG == 1) tma_load_2d(dst, m, &full_bar[stage], c0, c1);
        else tma_load_2d_pair(dst, m, pair_bar + stage * 8, c0, c1);
      };
      if (warp == 6) pdl_wait();   // weights never depend on the preceding kernel: their boxes go out at once
      for (int u = u0; u < n_units; u += u_step) {
        const int t0 = (u % a_units) * ROWS + (CG == 2 ? (int)rank * RM : 0), tb = u / a_units;
        for (int kb = 0; kb < g.k_blocks; kb += KS) {
          const int nk = KS == 1 || kb + 1 == g.k_blocks ? 1 : KS;
          mbar_wait(&empty_bar[stage], phase ^ 1);
          if (warp == 6) {
            expect(nk * Cfg::A_BYTES);
#pragma unroll
            for (int q = 0; q < KS; ++q)
              if (q < nk) load(sA + (stage * KS + q) * Cfg::A_BYTES, &tmA, (kb + q) * 64, t0);
          } else {
            expect(nk * Cfg::B_BYTES);
#pragma unroll
            for (int q = 0; q < KS; ++q) {
              if (q >= nk) break;
#pragma unroll
              for (int j = 0; j < Cfg::BROWS / Cfg::BOX; ++j) {
                int n = tb * BN + (CG == 2 ? (int)rank * Cfg::BROWS : 0) + j * Cfg::BOX;
                if (ACT != 0 && g.epi == XB_EPI_GLU) n = wide_glu_row(g, tb, CG == 2 ? rank != 0 : j != 0);
                uint8_t* dst = sB + (stage * KS + q) * Cfg::B_BYTES + j * Cfg::BOX * 128;
                if (g.w_tiled) load(dst, &tmB, 0, ((n >> 7) * g.k_blocks + kb + q) * 128 + (n & 127));
                else load(dst, &tmB, (kb + q) * 64, n);
              }
            }
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      pdl_wait();
    }
  } else if (warp == 1) {
    // ===================== MMA issuer (one elected thread, of a pair: of its first CTA) =====================
    if ((CG == 1 || rank == 0) && elect_one()) {
      constexpr uint32_t idesc = (umma_idesc_bf16(BN) & ~(0x1fu << 24)) | ((uint32_t)(ROWS >> 4) << 24);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      const uint64_t desc_a0 = umma_desc_sw128(smem_u32(sA)), desc_b0 = umma_desc_sw128(smem_u32(sB));
      for (int u = u0; u < n_units; u += u_step) {
        mbar_wait(&tempty_bar[acc], acc_phase ^ 1);   // epilogue has drained this accumulator
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * Cfg::ACC_COLS);
        for (int kb = 0; kb < g.k_blocks; kb += KS) {
          mbar_wait(&full_bar[stage], phase);
          tc_fence_after();
#pragma unroll
          for (int q = 0; q < KS; ++q) {
            if (q > 0 && kb + q >= g.k_blocks) break;
            const uint64_t da = desc_a0 + (uint64_t)((stage * KS + q) * (Cfg::A_BYTES >> 4));
            const uint64_t db = desc_b0 + (uint64_t)((stage * KS + q) * (Cfg::B_BYTES >> 4));
#pragma unroll
            for (int k = 0; k < 4; ++k)               // 4 x (K = 16) per 64-wide k-block
              wide_mma<CG>(d_tmem, da + k * 2, db + k * 2, idesc, (kb > 0 || q > 0 || k > 0) ? 1u : 0u);
          }
          wide_commit<CG>(&empty_bar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        wide_commit<CG>(&tfull_bar[acc]);
        if (++acc == Cfg::ACC_STAGES) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ===================== epilogue warps 2..5 =====================
    const int quad = warp & 3;
    const int row_in_tile = RM == 64 ? (quad & 1) * 32 + lane : quad * 32 + lane;
    const int col0 = RM == 64 ? (quad >> 1) * Cfg::COLS : 0;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
    pdl_wait();                                       // `out` may still be read by the upstream grid
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int u = u0; u < n_units; u += u_step) {
      const int tb = u / a_units, n0 = tb * BN + col0;
      const int t = (u % a_units) * ROWS + (CG == 2 ? (int)rank * RM : 0) + row_in_tile;
      const bool qkv = g.epi == XB_EPI_QKV && t < g.a_rows;
      const int pos = qkv ? g.tok_pos[t] : 0;
      WideQkvRow row;
      row.kv = qkv && n0 + Cfg::COLS > g.n_heads * g.head_dim ? wide_kv_row(g, t, pos) : 0;
      float next[32];
      int up0 = 0, gate0 = 0;
      float weight = 1.f;
      bool shared = false;
      if (ACT != 0 && g.epi == XB_EPI_GLU) {
        gate0 = wide_glu_row(g, tb, false);
        up0 = wide_glu_row(g, tb, true);
        shared = tb * 128 >= g.glu_e * g.glu_f;
        const int at = shared ? g.glu_sg_at : tb * 128 / g.glu_f;
        if (g.glu_w != nullptr && t < g.a_rows && at >= 0) weight = g.glu_w[(long long)t * g.glu_ldg + at];
      }
      if (ACT == 0 && qkv) {
        int c0, c1;
        wide_pair_cols(g, 0, c0, c1);
        wide_rope_load(g, pos, n0 + c0, next);
      }
      mbar_wait(&tfull_bar[acc], acc_phase);
      tc_fence_after();
      const uint32_t t_addr = lane_base + (uint32_t)(acc * Cfg::ACC_COLS);
#pragma unroll 1
      for (int p = 0; p < Cfg::PAIRS; ++p) {
        int c0, c1;
        if (ACT != 0 && g.epi == XB_EPI_GLU) { c0 = p * 16; c1 = 128 + p * 16; }
        else wide_pair_cols(g, p, c0, c1);
        uint32_t v0[16], v1[16];
        tmem_ld16(t_addr + c0, v0);
        tmem_ld16(t_addr + c1, v1);
        if (ACT == 0 && qkv) {
#pragma unroll
          for (int j = 0; j < 32; ++j) row.cs[j] = next[j];
          if (p + 1 < Cfg::PAIRS) {
            int d0, d1;
            wide_pair_cols(g, p + 1, d0, d1);
            wide_rope_load(g, pos, n0 + d0, next);
          }
        }
        tmem_ld_wait();
        float *x0 = reinterpret_cast<float*>(v0), *x1 = reinterpret_cast<float*>(v1);
        if (ACT == 0) {
          wide_emit(g, t, row, n0 + c0, n0 + c1, x0, x1);
        } else if (g.epi == XB_EPI_GLU) {
          wide_emit_glu(g, t, tb * 128 + c0, gate0 + c0, up0 + c0, weight, shared, x0, x1);
        } else {
          wide_emit_relu2(g, t, n0 + c0, x0);
          wide_emit_relu2(g, t, n0 + c1, x1);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 1) mbar_arrive(&tempty_bar[acc]);
        else mbar_arrive_cluster(cluster_map(smem_u32(&tempty_bar[acc]), 0));
      }
      if (++acc == Cfg::ACC_STAGES) { acc = 0; acc_phase ^= 1; }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync_aligned();                // no CTA of a pair leaves while the other still uses its memory
  if (warp == 1) {
    tc_fence_after();
    wide_tmem_dealloc<CG>(tmem_base, Cfg::TM_COLS);
  }
}

// ----------------------------------------------------------------------------- host side
struct WideVariant {
  int bn, cg, rm, cols;          // cols: columns a thread of the epilogue holds
  double us_k_block, us_ends;    // estimated time (xb_pick_wide)
  int (*run_act)(const CUtensorMap&, const CUtensorMap&, const GemmArgs&, int grid, cudaStream_t, int pdl);   // with the feed-forward activations, or nullptr
  int (*run)(const CUtensorMap&, const CUtensorMap&, const GemmArgs&, int grid, cudaStream_t, int pdl);
};

template <int BN, int CG, int RM, int ACT>
static int xb_wide_launch_t(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmArgs& g, int grid, cudaStream_t st, int pdl) {
  using Cfg = WideCfg<BN, CG, RM>;
  {
    static bool done[XB_MAX_DEVICES] = {false};
    int dev = 0;
    XB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= XB_MAX_DEVICES || !done[dev]) {
      XB_CUDA(cudaFuncSetAttribute(xb_wide_kernel<BN, CG, RM, ACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
      if (dev >= 0 && dev < XB_MAX_DEVICES) done[dev] = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(224, 1, 1);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (CG > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = CG;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  XB_CUDA(cudaLaunchKernelEx(&cfg, xb_wide_kernel<BN, CG, RM, ACT>, tmA, tmB, g));
  return 0;
}

#define XB_WIDE_VARIANT(BN, CG, RM, KB, ENDS, RUN_ACT) {BN, CG, RM, WideCfg<BN, CG, RM>::COLS, KB, ENDS, RUN_ACT, xb_wide_launch_t<BN, CG, RM, 0>}
static const WideVariant g_wide_variants[] = {
  XB_WIDE_VARIANT(256, 2, 128, 0.34, 5.3, (xb_wide_launch_t<256, 2, 128, 1>)), XB_WIDE_VARIANT(256, 1, 128, 0.38, 6.2, (xb_wide_launch_t<256, 1, 128, 1>)),
  XB_WIDE_VARIANT(192, 1, 128, 0.33, 3.4, nullptr), XB_WIDE_VARIANT(128, 1, 128, 0.26, 0.8, nullptr),
  XB_WIDE_VARIANT(256, 2, 64, 0.22, 1.6, nullptr), XB_WIDE_VARIANT(128, 2, 64, 0.165, 1.6, nullptr),
};
#undef XB_WIDE_VARIANT
enum { XB_WIDE_VARIANTS = sizeof(g_wide_variants) / sizeof(g_wide_variants[0]) };

// The variant with the least estimated time: waves x (k-blocks x time of one) + the ends.  The times (us) are fitted to a sweep of T = 150 .. 2048 over 14
// Linears of the registered models (K 2048 .. 18944, N 2048 .. 37888; back to back, weights from HBM): over the 168 shapes the choice is 0.2 % slower than
// the best variant on average, 9 % at most.  Without the pairs of 64 rows it was 18 % and 79 %.
// col_unit: columns that one thread has to hold together (a head where the rotation pairs its halves).
// act: only variants with the feed-forward activations.  *us: the estimate.
static int xb_pick_wide(int T, int N, int K, int col_unit, int num_sms, bool act = false, double* us = nullptr) {
  int best = 1;
  double best_t = 1e30;
  const int k_blocks = (K + 63) / 64;
  for (int i = 0; i < XB_WIDE_VARIANTS; ++i) {
    const WideVariant& v = g_wide_variants[i];
    if (v.cols % col_unit != 0 || (act && v.run_act == nullptr)) continue;
    const int rows = v.rm * v.cg;
    const long long units = (long long)((T + rows - 1) / rows) * ((N + v.bn - 1) / v.bn);
    const int slots = num_sms / v.cg;
    const long long waves = (units + slots - 1) / slots;
    const double t = (double)waves * k_blocks * v.us_k_block + v.us_ends;
    if (t < best_t) { best_t = t; best = i; }
  }
  if (us != nullptr) *us = best_t;
  return best;
}

static int xb_wide_plan(GemmPlan* p, const bf16* x, long long ldx, const bf16* w, int w_tiled, int T, int N, int K, int col_unit, int num_sms,
                        int force_variant) {
  int vi = force_variant > 0 ? force_variant - 1 : xb_pick_wide(T, N, K, col_unit, num_sms);
  const char* ev = getenv("XB_WIDE_VARIANT");   // pins the variant (from 1) where it does not cut a column unit (tests, A/B)
  const int pin = ev != nullptr ? atoi(ev) : 0;
  if (force_variant == 0 && pin >= 1 && pin <= XB_WIDE_VARIANTS && g_wide_variants[pin - 1].cols % col_unit == 0) vi = pin - 1;
  XB_CHECK(vi < XB_WIDE_VARIANTS, "wide Linear variant %d of %d", vi + 1, (int)XB_WIDE_VARIANTS);
  const WideVariant& v = g_wide_variants[vi];
  GemmArgs& g = p->args;
  p->wide = vi;
  p->bn = v.bn;
  g.b_tiles = (N + v.bn - 1) / v.bn;
  g.a_rows = T;
  g.b_rows = N;
  const int rows = v.rm * v.cg, units = (T + rows - 1) / rows * g.b_tiles;
  p->grid = (units < num_sms / v.cg ? units : num_sms / v.cg) * v.cg;
  const int box = (v.bn / v.cg) % 128 == 0 ? 128 : 64;
  const long long w_tiles = (N + 127) / 128;
  XB_TRY(xb_make_tmap(&p->tmA, x, T, K, ldx, v.rm));
  if (w_tiled) XB_TRY(xb_make_tmap(&p->tmB, w, w_tiles * g.k_blocks * 128, 64, 64, box));
  else XB_TRY(xb_make_tmap(&p->tmB, w, N, K, K, box));
  p->tmC = p->tmA;
  return 0;
}

// Does the activation belong into the epilogue?  Yes where the tiles that can do it are not slower than the best ones by more than the kernel
// would take that reads the finished matrix (2.5 us and 3.9 TB/s over what it reads and writes).
static bool xb_wide_act_pays(int T, int N, int K, int n_out, int num_sms) {
  double with = 0, without = 0;
  xb_pick_wide(T, N, K, 32, num_sms, true, &with);
  xb_pick_wide(T, N, K, 32, num_sms, false, &without);
  return with < without + 2.5 + 2.0 * T * ((double)N + n_out) / 3.9e6;
}

static int xb_wide_run(const GemmPlan& p, cudaStream_t st, int pdl) {
  const bool act = p.args.epi == XB_EPI_GLU || p.args.epi == XB_EPI_RELU2;
  return (act ? g_wide_variants[p.wide].run_act : g_wide_variants[p.wide].run)(p.tmA, p.tmB, p.args, p.grid, st, pdl);
}
