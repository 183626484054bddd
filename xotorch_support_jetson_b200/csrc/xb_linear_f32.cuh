// Linear of the float32 mode on the tensor cores: y[T,N] (fp32) = x[T,K] (fp32) W[N,K]^T (bf16) + bias.
//
// An fp32 number is the exact sum of three bf16 numbers (24 significant bits, eight each) and W is bf16 already, so x W^T is three
// bf16 products whose every term is exact in fp32; what rounds is the summation alone.  The sums of one k-block (64 numbers)
// are formed in TMEM, smallest piece first, and join an fp32 total in registers with one rounding per k-block: the tensor
// core never adds to a total that is large against its terms.  Error of two or three layers against 64 bits, 1 to 400 rows: 3.0e-7
// to 4.2e-7, plain FMA (16 numbers per slice) 3.9e-7 to 7.2e-7.
//
//   D[128 rows x 128 features] (TMEM) = sum over pieces  A_p[128 x 64] (smem) * B[128 x 64]^T (W, smem)
//
// Bound by the tensor cores (12 MMAs a k-block, 0.4 us) and by the 64 KB an SM takes in for them (0.55 us).  300 rows of two
// refatar-1b layers, 73 GFLOP: 7.06 ms with plain FMA on 64 x 64 tiles, 1.55 ms with this kernel (all kernels of the
// step; 1.19 ms today); one row 774 -> 506 us, so few rows take it too.  The layers' Linears of 300 rows, 37 to 50 MB of weights: 46 to 62 us, tensor pipe
// 0.5 to 0.7 busy.
// S > 1: S CTAs of a cluster share a tile, each a part of K, and add their totals in rank order through distributed shared
// memory.
#pragma once
#include "xb_wide.cuh"

struct F32Args {
  int T, N, k_blocks, a_tiles, b_tiles;
  int plane_rows;          // rows of one piece plane [3][plane_rows][K]
  const float* bias;
  float* y;
  long long ldy;
};

// x -> three planes of bf16 pieces.  Truncation keeps the first two pieces below |x| and the rests exact; numbers that are not
// finite go into the first plane alone.
__device__ __forceinline__ void f32_pieces(float x, bf16* p) {
  const uint32_t u = __float_as_uint(x);
  if ((u & 0x7f800000u) == 0x7f800000u) {
    p[0] = f2bf(x);
    p[1] = p[2] = f2bf(0.f);
    return;
  }
  const float a = __uint_as_float(u & 0xffff0000u);
  const float r = x - a;
  const float b = __uint_as_float(__float_as_uint(r) & 0xffff0000u);
  p[0] = f2bf(a);
  p[1] = f2bf(b);
  p[2] = f2bf(r - b);
}
__global__ void __launch_bounds__(256) xb_f32_pieces_kernel(const float* __restrict__ x, long long ldx, bf16* __restrict__ planes, long long plane,
                                                            int T, int K) {
  pdl_launch_dependents();
  pdl_wait();
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  const int k8 = K >> 3;
  if (i >= (long long)T * k8) return;
  const long long t = i / k8;
  const int k = (int)(i - t * k8) * 8;
  const float* src = x + t * ldx + k;
  float v[8];
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = src[j];
  }
  __align__(16) bf16 p[3][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    bf16 q[3];
    f32_pieces(v[j], q);
    p[0][j] = q[0]; p[1][j] = q[1]; p[2][j] = q[2];
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) *reinterpret_cast<uint4*>(planes + c * plane + t * K + k) = *reinterpret_cast<const uint4*>(p[c]);
}

struct F32Cfg {
  static constexpr int TILE_BYTES = 128 * 64 * 2;
  static constexpr int STAGE_BYTES = 4 * TILE_BYTES;   // three pieces of x, one box of W
  static constexpr int STAGES = 3;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

template <int S>
__global__ void __launch_bounds__(224, 1)
xb_linear_f32_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int a_box_rows, F32Args g) {
  constexpr int STAGES = F32Cfg::STAGES, TB = F32Cfg::TILE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * F32Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = S > 1 ? cluster_rank() : 0;
  const int n_units = g.a_tiles * g.b_tiles;
  const int u0 = blockIdx.x / S, u_step = S > 1 ? n_units : (int)gridDim.x;
  const int kb0 = S > 1 ? (int)(((long long)rank * g.k_blocks) / S) : 0;
  const int kb1 = S > 1 ? (int)(((long long)(rank + 1) * g.k_blocks) / S) : g.k_blocks;

  if (warp == 1) {
    if (lane == 0) {
      tma_prefetch_desc(&tmA);
      tma_prefetch_desc(&tmB);
      for (int i = 0; i < STAGES; ++i) {
        mbar_init(&full_bar[i], 2);
        mbar_init(&empty_bar[i], 1);
      }
      for (int i = 0; i < 2; ++i) {
        mbar_init(&tfull_bar[i], 1);
        mbar_init(&tempty_bar[i], 4);
      }
      fence_mbar_init();
    }
    __syncwarp();
    tmem_alloc(tmem_slot, 256);
  }
  tc_fence_before();
  __syncthreads();
  if (S > 1) cluster_sync_aligned();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  float tot[128];                                     // epilogue warps: this row's sums of the tile's 128 features
#pragma unroll
  for (int j = 0; j < 128; ++j) tot[j] = 0.f;

  // one row of 32 consecutive features of the tile -> y
  auto store32 = [&](const float* v, int t, int n0) {
    if (t >= g.T || n0 >= g.N) return;
    float* dst = g.y + (long long)t * g.ldy + n0;
    const bool whole = n0 + 32 <= g.N && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
#pragma unroll
    for (int j = 0; j < 32; j += 4) {
      float o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = v[j + i] + (g.bias != nullptr && n0 + j + i < g.N ? g.bias[n0 + j + i] : 0.f);
      if (whole) {
        *reinterpret_cast<float4*>(dst + j) = make_float4(o[0], o[1], o[2], o[3]);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (n0 + j + i < g.N) dst[j + i] = o[i];
      }
    }
  };

  if (warp == 0 || warp == 6) {
    // ===================== TMA producers: warp 0 weights, warp 6 the pieces of x =====================
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      if (warp == 6) pdl_wait();
      for (int u = u0; u < n_units; u += u_step) {
        const int ta = u % g.a_tiles, tb = u / g.a_tiles;
        for (int kb = kb0; kb < kb1; ++kb) {
          uint8_t* st = smem + stage * F32Cfg::STAGE_BYTES;
          mbar_wait(&empty_bar[stage], phase ^ 1);
          if (warp == 6) {
            mbar_expect_tx(&full_bar[stage], 3 * a_box_rows * 128);
#pragma unroll
            for (int p = 0; p < 3; ++p) tma_load_2d(st + p * TB, &tmA, &full_bar[stage], kb * 64, p * g.plane_rows + ta * 128);
          } else {
            mbar_expect_tx(&full_bar[stage], TB);
            tma_load_2d(st + 3 * TB, &tmB, &full_bar[stage], kb * 64, tb * 128);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      pdl_wait();
    }
  } else if (warp == 1) {
    // ===================== MMA issuer =====================
    if (elect_one()) {
      constexpr uint32_t idesc = umma_idesc_bf16(128);
      const uint64_t desc0 = umma_desc_sw128(smem_u32(smem));
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      for (int u = u0; u < n_units; u += u_step) {
        for (int kb = kb0; kb < kb1; ++kb) {
          mbar_wait(&tempty_bar[acc], acc_phase ^ 1);
          mbar_wait(&full_bar[stage], phase);
          tc_fence_after();
          const uint64_t d = desc0 + (uint64_t)(stage * (F32Cfg::STAGE_BYTES >> 4));
#pragma unroll
          for (int p = 2; p >= 0; --p)
#pragma unroll
            for (int k = 0; k < 4; ++k)
              tc_mma_bf16(tmem_base + acc * 128, d + p * (TB >> 4) + k * 2, d + 3 * (TB >> 4) + k * 2, idesc, (p < 2 || k > 0) ? 1u : 0u);
          tc_commit(&empty_bar[stage]);
          tc_commit(&tfull_bar[acc]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
      }
    }
  } else {
    // ===================== warps 2..5: k-block sums -> totals -> y =====================
    const int quad = warp & 3;
    const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16);
    int acc = 0;
    uint32_t acc_phase = 0;
    pdl_wait();
    for (int u = u0; u < n_units; u += u_step) {
      const int ta = u % g.a_tiles, tb = u / g.a_tiles;
      for (int kb = kb0; kb < kb1; ++kb) {
        mbar_wait(&tfull_bar[acc], acc_phase);
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 128; c += 64) {
          uint32_t v[64];
          tmem_ld16(lane_base + acc * 128 + c, v);
          tmem_ld16(lane_base + acc * 128 + c + 16, v + 16);
          tmem_ld16(lane_base + acc * 128 + c + 32, v + 32);
          tmem_ld16(lane_base + acc * 128 + c + 48, v + 48);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 64; ++j) tot[c + j] += __uint_as_float(v[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty_bar[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
      if (S == 1) {
#pragma unroll
        for (int c = 0; c < 128; c += 32) {
          store32(tot + c, ta * 128 + quad * 32 + lane, tb * 128 + c);
#pragma unroll
          for (int j = 0; j < 32; ++j) tot[c + j] = 0.f;
        }
      }
    }
  }
  __syncwarp();
  if (S > 1) {
    constexpr int OWN = 128 / S;                      // features this CTA finishes
    cluster_sync_aligned();                           // every CTA of the cluster is past its last k-block: the rings are free
    float* xch = reinterpret_cast<float*>(smem);      // [S senders][OWN features][128 rows]
    const int row = (warp & 3) * 32 + lane;
    if (warp >= 2 && warp < 6) {
#pragma unroll
      for (int d = 0; d < S; ++d) {
        const uint32_t dst = cluster_map(smem_u32(xch), d) + (uint32_t)(rank * OWN * 128 + row) * 4;
#pragma unroll
        for (int j = 0; j < OWN; ++j)
          asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)(j * 128) * 4), "f"(tot[d * OWN + j]) : "memory");
      }
    }
    __syncwarp();
    cluster_sync_aligned();
    if (warp >= 2 && warp < 6) {
      const int t = (u0 % g.a_tiles) * 128 + row, n0 = (u0 / g.a_tiles) * 128 + (int)rank * OWN;
#pragma unroll 1
      for (int c = 0; c < OWN; c += 32) {
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0.f;
#pragma unroll
        for (int s = 0; s < S; ++s) {                 // rank order
          const float* src = xch + (size_t)(s * OWN + c) * 128 + row;
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] += src[j * 128];
        }
        store32(v, t, n0 + c);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 256);
  }
}

// ----------------------------------------------------------------------------- host side
#define XB_F32_ROWS 2048   // rows of x cut into pieces at a time (the workspace is 3 planes of so many rows)

struct F32Plan {
  CUtensorMap tmA, tmB;
  F32Args args;
  int a_box_rows, split, grid;
};

static bool xb_f32_takes(const void* w, int K) { return K % 8 == 0 && K >= 16 && (reinterpret_cast<uintptr_t>(w) & 15) == 0; }

static int xb_f32_plan(F32Plan* p, const bf16* planes, int plane_rows, const bf16* w, const float* bias, float* y, long long ldy, int T, int N, int K,
                       int num_sms) {
  F32Args& g = p->args;
  g.T = T; g.N = N; g.k_blocks = (K + 63) / 64; g.a_tiles = (T + 127) / 128; g.b_tiles = (N + 127) / 128;
  g.plane_rows = plane_rows; g.bias = bias; g.y = y; g.ldy = ldy;
  const int units = g.a_tiles * g.b_tiles;
  // K in parts where the tiles alone leave SMs idle and a part keeps four k-blocks
  p->split = 1;
  if (units * 4 <= num_sms - 4 && g.k_blocks >= 16) p->split = 4;
  else if (units * 2 <= num_sms && g.k_blocks >= 8) p->split = 2;
  p->grid = p->split > 1 ? units * p->split : (units < num_sms ? units : num_sms);
  p->a_box_rows = T >= 128 ? 128 : (T + 7) / 8 * 8;   // rows behind the box keep what the stage held: only their own results depend on them
  if (p->a_box_rows > 128) p->a_box_rows = 128;
  XB_TRY(xb_make_tmap(&p->tmA, planes, 3LL * plane_rows, K, K, p->a_box_rows));
  XB_TRY(xb_make_tmap(&p->tmB, w, N, K, K, 128));
  return 0;
}

template <int S>
static int xb_f32_run_t(const F32Plan& p, cudaStream_t st, int pdl) {
  {
    static bool done[XB_MAX_DEVICES] = {false};
    int dev = 0;
    XB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= XB_MAX_DEVICES || !done[dev]) {
      XB_CUDA(cudaFuncSetAttribute(xb_linear_f32_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, F32Cfg::SMEM_BYTES));
      if (dev >= 0 && dev < XB_MAX_DEVICES) done[dev] = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.grid, 1, 1);
  cfg.blockDim = dim3(224, 1, 1);
  cfg.dynamicSmemBytes = F32Cfg::SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (pdl) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (S > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = S;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr;
  cfg.numAttrs = na;
  XB_CUDA(cudaLaunchKernelEx(&cfg, xb_linear_f32_kernel<S>, p.tmA, p.tmB, p.a_box_rows, p.args));
  return 0;
}
static int xb_f32_run(const F32Plan& p, cudaStream_t st, int pdl) {
  return p.split == 4 ? xb_f32_run_t<4>(p, st, pdl) : p.split == 2 ? xb_f32_run_t<2>(p, st, pdl) : xb_f32_run_t<1>(p, st, pdl);
}
