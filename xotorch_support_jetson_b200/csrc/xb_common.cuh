// Shared device/host helpers for the sm_100a kernels of libxb200.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda.h>
#include <stdint.h>
#include <stdio.h>
#include <string>

typedef __nv_bfloat16 bf16;

#define XB_MAX_DEVICES 64   // per-device caches (kernel attributes, built-in scratch address) are indexed by device ordinal

// ----------------------------------------------------------------------------- errors
// Thread-local message returned by xb_last_error(); no C++ exception crosses the C ABI.
extern thread_local std::string g_xb_err;
int xb_fail(int code, const char* fmt, ...);

#define XB_CUDA(expr)                                                                        \
  do {                                                                                       \
    cudaError_t _e = (expr);                                                                 \
    if (_e != cudaSuccess)                                                                   \
      return xb_fail(2, "%s:%d: %s -> %s", __FILE__, __LINE__, #expr, cudaGetErrorString(_e)); \
  } while (0)

#define XB_CHECK(cond, ...)                     \
  do {                                          \
    if (!(cond)) return xb_fail(1, __VA_ARGS__); \
  } while (0)

#define XB_TRY(expr)             \
  do {                           \
    int _r = (expr);             \
    if (_r != 0) return _r;      \
  } while (0)

// ----------------------------------------------------------------------------- bf16 helpers
__device__ __forceinline__ float bf2f(bf16 v) { return __bfloat162float(v); }
__device__ __forceinline__ bf16 f2bf(float v) { return __float2bfloat16_rn(v); }
// round an fp32 value to the nearest bf16 and return it widened again (a "rounding point")
__device__ __forceinline__ float rbf(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ float2 bf2_to_f2(uint32_t u) {
  float2 r;
  r.x = __uint_as_float(u << 16);
  r.y = __uint_as_float(u & 0xffff0000u);
  return r;
}
__device__ __forceinline__ uint32_t f2_to_bf2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// 128-bit streaming load that does not allocate in L1 (weights / KV are read once)
__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}

// ----------------------------------------------------------------------------- PTX: mbarrier / TMA / tcgen05
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool elect_one() {
  uint32_t pred = 0;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "elect.sync _|P, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(pred));
  return pred != 0;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, P;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: a pipeline bug turns into a trapped launch (reported as a CUDA error by the
// next API call) instead of a hung GPU.  ~4e9 cycles is seconds; real waits are microseconds.
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity) {
  if (mbar_try_wait(bar, parity)) return;
  long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > 4000000000LL) {
      printf("xb200: mbarrier wait timed out (block %d thread %d)\n", blockIdx.x, threadIdx.x);
      __trap();
    }
  }
}

__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(m) : "memory");
}
// 2-D tiled TMA load; c0 = innermost (K element) coordinate, c1 = row coordinate
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(m), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(void* dst, const CUtensorMap* m, uint64_t* bar, int c0, int c1,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(smem_u32(dst)), "l"(m), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "l"(policy)
      : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// whole warp: allocate `cols` (power of two >= 32) TMEM columns, base address written to *dst_smem
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
// one thread: make `bar` observe completion of all tcgen05.mma issued so far by this thread
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// D[tmem] (+)= A[smem desc] * B[smem desc]^T, bf16 x bf16 -> fp32, issued by ONE thread
__device__ __forceinline__ void tc_mma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// warp-wide: 16 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// nanosecond wall clock shared by all SMs (timeline instrumentation, XB_GEMM_TS=1)
__device__ __forceinline__ unsigned long long xb_gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
#define XB_TS_SLOTS 16

// Programmatic dependent launch: wait for the producing grid / let the consumer grid start early
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// K-major, 128-byte-swizzled shared-memory operand descriptor (rows x 64 bf16 per tile row):
// 8-row x 128 B swizzle atoms stacked every 1024 B (SBO); LBO unused for swizzled K-major.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor: A,B = bf16 (K-major), D = fp32, M = 128, N = n
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// How split-K partial sums of one output column are laid out: `slots` fp32 planes of [T][N].
// Fixed split: every column has `splits` planes.  Stream-K: the planes of a 128-column tile are
// the consecutive blocks whose item range touches the tile.
struct SplitInfo {
  int k_blocks, q, splits;
  uint32_t inv;   // ceil(2^32 / q) where x * inv >> 32 is x / q for every item x of the Linear (xb_split_inv), 0: divide
};
// x * ceil(2^32 / q) is above x * 2^32 / q by less than x * q, so the quotient is right while items * q <= 2^32; q = 1 has no 32-bit inverse
inline uint32_t xb_split_inv(int q, long long items) {
  return q < 2 || items * q > (1LL << 32) ? 0u : (uint32_t)(((1ULL << 32) + (uint64_t)q - 1) / (uint64_t)q);
}
__host__ __device__ __forceinline__ int xb_split_div(const SplitInfo& si, int x) {
  return si.inv != 0 ? (int)(((uint64_t)(uint32_t)x * si.inv) >> 32) : x / si.q;
}
__host__ __device__ __forceinline__ int xb_n_segments(const SplitInfo& si, int col) {
  if (si.q <= 0) return si.splits;
  const int at = (col >> 7) * si.k_blocks;
  return xb_split_div(si, at + si.k_blocks - 1) - xb_split_div(si, at) + 1;
}

// What a Linear left behind, whatever kernel ran it: one fp32 matrix, fp32 split-K planes, or a bf16 matrix.
struct LinOut {
  const float* f;      // fp32 [planes][T][ld] (planes summed per column, see SplitInfo), or nullptr
  const bf16* h;       // bf16 [T][ld], or nullptr
  SplitInfo si;        // si.splits == 0: one plane
  long long plane;     // floats between planes
  long long ld;
  const float* bias;   // added on read (outputs of the tcgen05 Linear; the plain kernels add it themselves), or nullptr
};

__device__ __forceinline__ float lin_at(const LinOut& o, long long row, int col) {
  const float b = o.bias != nullptr ? o.bias[col] : 0.f;
  if (o.h != nullptr) return bf2f(o.h[row * o.ld + col]) + b;
  const float* p = o.f + row * o.ld + col;
  if (o.si.splits == 0) return *p + b;
  const int n = xb_n_segments(o.si, col);
  float s = 0.f;
  int i = 0;
  for (; i + 3 < n; i += 4) {   // four planes in flight
    const float v0 = p[i * o.plane], v1 = p[(i + 1) * o.plane], v2 = p[(i + 2) * o.plane], v3 = p[(i + 3) * o.plane];
    s += (v0 + v1) + (v2 + v3);
  }
  for (; i < n; ++i) s += p[i * o.plane];
  return s + b;
}
// v[c] = o[row][col[c]] for C columns at once (col[c] < 0: not read, 0), F planes of every column in flight: a kernel of few rows waits for
// the latency of these loads, one round trip instead of one for every four planes of every column.  The planes of a column add up as
// (p0 + p1) + (p2 + p3) + ..., the last one to three one by one, whatever C and F: lin_at's order.  A token step of three bibevik-1b layers (8 rows, 36 kernels, 13
// of them waiting for such reads; 35 since): 414 -> 366 us with what changed in the latent layer's kernels beside it.
template <int C, int F>
__device__ __forceinline__ void lin_at_cols(const LinOut& o, long long row, const int (&col)[C], float (&v)[C]) {
  static_assert(F % 4 == 0, "whole groups of four planes");
  float b[C];
#pragma unroll
  for (int c = 0; c < C; ++c) b[c] = o.bias != nullptr && col[c] >= 0 ? o.bias[col[c]] : 0.f;
  if (o.h != nullptr) {
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = (col[c] >= 0 ? bf2f(o.h[row * o.ld + col[c]]) : 0.f) + b[c];
    return;
  }
  const float* p = o.f + row * o.ld;
  if (o.si.splits == 0) {
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = (col[c] >= 0 ? p[col[c]] : 0.f) + b[c];
    return;
  }
  int n[C], most = 0;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    n[c] = col[c] >= 0 ? xb_n_segments(o.si, col[c]) : 0;
    most = n[c] > most ? n[c] : most;
    v[c] = 0.f;
  }
  for (int i = 0; i < most; i += F) {
    float w[C][F];
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int j = 0; j < F; ++j) w[c][j] = i + j < n[c] ? p[(i + j) * o.plane + col[c]] : 0.f;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int j = 0; j < F; j += 4) {
        if (i + j + 3 < n[c]) {
          v[c] += (w[c][j] + w[c][j + 1]) + (w[c][j + 2] + w[c][j + 3]);
        } else {
#pragma unroll
          for (int u = 0; u < 3; ++u)
            if (i + j + u < n[c]) v[c] += w[c][j + u];
        }
      }
  }
#pragma unroll
  for (int c = 0; c < C; ++c) v[c] += b[c];
}

// ----------------------------------------------------------------------------- activations of hybrid models
__device__ __forceinline__ float hy_sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float hy_silu(float x) { return x / (1.0f + expf(-x)); }
__device__ __forceinline__ float hy_gelu_tanh(float z) {
  return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float hy_glu_clamp(float g, float u, float limit) {
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return g * hy_sigmoid(1.702f * g) * (u + 1.0f);
}
// One channel of one expert with routing weight w.  act: XB_ACT_GLU_CLAMP, XB_ACT_SWIGLU (silu(g) u) or XB_ACT_GEGLU (gelu(g) u,
// tanh form), the last two without limits.
// on_input: the weight multiplies what the expert reads, and since both projections are linear, (w h) W^T = w (h W^T):
// gate and up are scaled before the activation; otherwise the weight multiplies the activation (and so the output).
__device__ __forceinline__ float hy_expert_act(float g, float u, float w, float limit, int act, int on_input) {
  if (on_input) { g *= w; u *= w; }
  const float y = act == XB_ACT_SWIGLU ? hy_silu(g) * u : (act == XB_ACT_GEGLU ? hy_gelu_tanh(g) * u : hy_glu_clamp(g, u, limit));
  return on_input ? y : w * y;
}
