// Sampler with the row resident on chip: a cluster of CL blocks per row, each block keeps its
// 1/CL slice of the SCALED logits in shared memory, so the row is read from L2 exactly once and
// the radix-select / softmax / argmax passes run out of shared memory; per-pass results
// (histograms, sums, best candidates) are merged across the cluster through distributed shared
// memory.  Same arithmetic as xb_sample_kernel (xb_kernels.cuh), which restates
// torchtune.generation.sample as the reference calls it (sharded_inference_engine.py:208-228);
// that kernel remains the fallback for rows too long for CL x 200 KB of shared memory.
//
// One block per row spends ~14 us per pass over a 128256-entry row (a single SM pulls ~40 GB/s
// out of L2): 7 passes = 100 us for 32 rows on 32 of the 148 SMs.
#pragma once
#include "xb_kernels.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

// exchange area of one block, read by its cluster peers; two copies used alternately so that one
// cluster barrier per exchange is enough (a copy is rewritten only two exchanges later)
struct SampleXchg {
  unsigned int hist[256];
  float fhist[256];
  float f0, f1;
  int i0;
  int pad;
};

// Top-k from candidates: the row is dealt into buckets (what eight lanes, or a warp, have read); the k-th largest bucket
// maximum has k elements at or above it, so the elements from there on contain the kept set -- about k + k^2 / (2 buckets) of
// 128256, 41 for k = 35.  Only these candidates are looked at again: pivot, softmax, nucleus and draw run over them in the first
// block of the cluster.  Bound by reading the row and by three cluster barriers: 32 x 128256 logits, top-k 35, 20.7 us a call
// on inputs in turn (19.9 the kernel alone, caches flushed), against four radix passes over every element.
// The radix passes keep what they are better at; device time of 32 rows, 128256 / 32768 entries, us.  k = 35: 15 / 13 with the usual 41 candidates,
// radix 27 / 15.  Candidates are ranked all against all: 26 / 24 for 250, 43 / 40 for 500; handed on to the radix passes 32 / 20 for 300, 33 / 21 for 500.
// From k = 65 on 512 bucket maxima are ranked too: 40 / 37 for k = 200, radix 27 / 15.  A nucleus costs the radix passes four more, over mass: 57 / 41 for k = 257,
// candidates 40 / 37 for k = 200, 65 / 62 for 760 of them, 95 / 92 for 1000, handed on 84 / 71.
// Rows with more candidates than a block holds (many ties) or with a NaN are handed on as well.
#define XB_TOPK_PLAIN 64       // largest k without and with a nucleus
#define XB_TOPK_NUCLEUS 256
#define XB_CAND_PLAIN 256      // most candidates of a row without and with a nucleus
#define XB_CAND_NUCLEUS 768
#define XB_TOPK_CAND 512       // candidates a block can hold
struct SampleCand {
  float bucket[128];        // this block's bucket maxima
  float v[XB_TOPK_CAND];
  int i[XB_TOPK_CAND];
  int n;                    // > XB_TOPK_CAND: take the radix passes
};

// the first block's last steps over n <= NT candidates (v, i in shared memory, any order): the chosen index, in every thread
template <int NT>
__device__ int sample_candidates(const float* v, const int* idx, int n, int top_k, float top_p, const float* __restrict__ q_row, unsigned long long seed,
                                 int rowi, float* sorted_e, float* cum, float* s_f, int* s_i) {
  const int tid = threadIdx.x;
  if (tid == 0) { s_f[0] = -INFINITY; s_f[1] = -INFINITY; }
  __syncthreads();
  // rank of every candidate by (value down, index up): a fixed order whatever order they arrived in
  float my_v = 0.f;
  int my_i = 0, my_r = 0;
  if (tid < n) {
    int gt = 0, ge = 0;
    my_v = v[tid]; my_i = idx[tid];
    for (int b = 0; b < n; ++b) {
      const float o = v[b];
      gt += o > my_v;
      ge += o >= my_v;
      my_r += o > my_v || (o == my_v && idx[b] < my_i);
    }
    if (my_r == 0) s_f[1] = my_v;                       // largest value
    if (gt < top_k && ge >= top_k) s_f[0] = my_v;       // k-th largest value (every thread that writes has the same)
  }
  __syncthreads();
  const float pivot = s_f[0], mxv = s_f[1];
  const float my_e = tid < n && my_v >= pivot ? expf(my_v - mxv) : 0.f;
  if (tid < n) sorted_e[my_r] = my_e;
  __syncthreads();
  if (tid < 32) {               // running sums in rank order, a fixed tree
    float base = 0.f;
    for (int a = 0; a < n; a += 32) {
      float x = a + tid < n ? sorted_e[a + tid] : 0.f;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, x, o);
        if (tid >= o) x += y;
      }
      x += base;
      if (a + tid < n) cum[a + tid] = x;
      base = __shfl_sync(0xffffffffu, x, 31);
    }
    if (tid == 0) { s_f[2] = base; s_i[0] = n - 1; }
  }
  __syncthreads();
  const float sum = s_f[2];
  float p_cut = 0.f;
  if (top_p > 0.f && top_p < 1.f) {   // smallest probability of the shortest head that reaches top_p, equal ones with it
    // the lanes of the scan add up in different trees, so where weights are tiny a sum can come out an ulp below its predecessor
    // and top_p be crossed more than once: the first crossing counts
    for (int a = tid; a < n; a += NT)
      if (cum[a] >= top_p * sum && (a == 0 || cum[a - 1] < top_p * sum)) atomicMin(&s_i[0], a);
    __syncthreads();
    p_cut = sorted_e[s_i[0]];
  }
  float best = -INFINITY;
  int bi = 0x7fffffff;
  if (tid < n && my_v >= pivot && my_e >= p_cut) {
    float qv;
    if (q_row != nullptr) {
      qv = q_row[my_i];
    } else {
      const uint32_t r = mix32(seed * 0x9E3779B97F4A7C15ULL + ((unsigned long long)rowi << 32) + (unsigned)my_i);
      const float u = ((float)(r & 0xffffff) + 0.5f) * (1.0f / 16777216.0f);
      qv = -logf(u);
    }
    const float sc = (my_e / sum) / qv;
    if (sc > best || (sc == best && my_i < bi)) { best = sc; bi = my_i; }
  }
  auto better = [](float a, int ai, float b, int bj) { return a > b || (a == b && ai < bj); };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (better(ov, oi, best, bi)) { best = ov; bi = oi; }
  }
  __syncthreads();
  if ((tid & 31) == 0) { s_f[4 + (tid >> 5)] = best; s_i[tid >> 5] = bi; }
  __syncthreads();
  best = s_f[4];
  bi = s_i[0];
  for (int w = 1; w < NT / 32; ++w)
    if (better(s_f[4 + w], s_i[w], best, bi)) { best = s_f[4 + w]; bi = s_i[w]; }
  return bi;
}

template <int NT, int CL>
__global__ void __launch_bounds__(NT) xb_sample_cluster_kernel(const float* __restrict__ logits, int V, int chunk, float temp,
                                                               int top_k, float top_p, const float* __restrict__ q_noise,
                                                               unsigned long long seed, int* __restrict__ out) {
  extern __shared__ float vals[];                 // this block's slice of the row, already * 1/temp
  __shared__ SampleXchg xc[2];
  __shared__ unsigned int mh[256];
  __shared__ float mfh[256];
  __shared__ uint32_t s_prefix;
  __shared__ int s_need;
  __shared__ float s_needf;
  __shared__ float red[32];
  __shared__ float sv[NT / 32];
  __shared__ int si[NT / 32];
  __shared__ SampleCand cand;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  const int rowi = blockIdx.x / CL;
  const float* row = logits + (long long)rowi * V;
  const float inv_t = 1.0f / fmaxf(temp, 1e-5f);
  const int i0 = rank * chunk;
  const int n = V - i0 < 0 ? 0 : (V - i0 < chunk ? V - i0 : chunk);
  int xi = 0;                                     // which exchange copy the next merge uses

  // ---- load the slice once (float4 when the row allows it), scale, local max
  float mx = -INFINITY;
  bool odd = false;                               // a NaN among this thread's numbers
  if ((V & 3) == 0 && (chunk & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    const float4* r4 = reinterpret_cast<const float4*>(row + i0);
    float4* v4 = reinterpret_cast<float4*>(vals);
    const int n4 = n >> 2;
    auto put = [&](int i, float4 a) {
      a.x *= inv_t; a.y *= inv_t; a.z *= inv_t; a.w *= inv_t;
      v4[i] = a;
      odd = odd || !(a.x + a.y + a.z + a.w == a.x + a.y + a.z + a.w);
      mx = fmaxf(fmaxf(mx, fmaxf(a.x, a.y)), fmaxf(a.z, a.w));
    };
    int i = threadIdx.x;
    for (; i + 3 * NT < n4; i += 4 * NT) {   // four loads in flight per thread: the slice comes out of L2 once
      const float4 a = r4[i], b = r4[i + NT], c = r4[i + 2 * NT], d = r4[i + 3 * NT];
      put(i, a); put(i + NT, b); put(i + 2 * NT, c); put(i + 3 * NT, d);
    }
    for (; i < n4; i += NT) put(i, r4[i]);
  } else {
    for (int i = threadIdx.x; i < n; i += NT) {
      const float v = row[i0 + i] * inv_t;
      vals[i] = v;
      odd = odd || v != v;
      mx = fmaxf(mx, v);
    }
  }
  const bool use_k = top_k > 0 && top_k < V;
  const bool nucleus = top_p > 0.f && top_p < 1.f;
  if (use_k && top_k <= (nucleus ? XB_TOPK_NUCLEUS : XB_TOPK_PLAIN)) {
    // ---- candidates: everything from the k-th largest bucket maximum on
    const int lane = threadIdx.x & 31, per = top_k <= 64 ? 32 : 8;   // lanes of a bucket: 32 or 128 buckets a block
    const int nb = NT / per;
    float bm = mx;
    for (int o = 1; o < per; o <<= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, o));
    if (lane % per == 0) cand.bucket[threadIdx.x / per] = bm;
    const int any_odd = __syncthreads_or(odd);
    if (threadIdx.x == 0) cand.n = any_odd ? XB_TOPK_CAND + 1 : 0;
    cluster.sync();
    float* all = mfh;                             // [CL * nb] bucket maxima of the row (mfh | mh: 512 numbers)
    static_assert(CL * 128 <= 512, "bucket maxima of a row");
    for (int i = threadIdx.x; i < CL * nb; i += NT) {
      const float b = cluster.map_shared_rank(&cand, i / nb)->bucket[i % nb];
      if (i < 256) mfh[i] = b; else mh[i - 256] = __float_as_uint(b);
    }
    __syncthreads();
    if (threadIdx.x < CL * nb) {
      auto at = [&](int i) { return i < 256 ? all[i] : __uint_as_float(mh[i - 256]); };
      const float b = at(threadIdx.x);
      int gt = 0, ge = 0;
      for (int i = 0; i < CL * nb; ++i) {
        const float o = at(i);
        gt += o > b;
        ge += o >= b;
      }
      if (gt < top_k && ge >= top_k) s_needf = b;   // all that write write the same
    }
    __syncthreads();
    const float low = s_needf;
    if (!any_odd) {
      for (int i = threadIdx.x; i < n; i += NT) {
        const float v = vals[i];
        if (v >= low) {
          const int at = atomicAdd(&cand.n, 1);
          if (at < XB_TOPK_CAND) { cand.v[at] = v; cand.i[at] = i0 + i; }
        }
      }
    }
    cluster.sync();
    int total = 0;
    bool fits = true;
    for (int r = 0; r < CL; ++r) {
      const int c = cluster.map_shared_rank(&cand, r)->n;
      fits = fits && c <= XB_TOPK_CAND;
      total += c;
    }
    static_assert(XB_CAND_PLAIN <= NT && XB_CAND_NUCLEUS <= NT, "a thread per candidate");
    if (fits && total <= (nucleus ? XB_CAND_NUCLEUS : XB_CAND_PLAIN) && 4 * total <= chunk) {   // the same answer in every block of the cluster
      if (rank == 0) {
        float* cv = vals;                         // the slice is not needed any more
        int* ci = reinterpret_cast<int*>(vals + total);
        float* es = vals + 2 * total;
        float* cum = vals + 3 * total;
        int at = 0;
        for (int r = 0; r < CL; ++r) {
          const SampleCand* pc = cluster.map_shared_rank(&cand, r);
          const int c = pc->n;
          for (int i = threadIdx.x; i < c; i += NT) { cv[at + i] = pc->v[i]; ci[at + i] = pc->i[i]; }
          at += c;
        }
        __syncthreads();
        const int bi = sample_candidates<NT>(cv, ci, total, top_k, top_p, q_noise != nullptr ? q_noise + (long long)rowi * V : nullptr, seed, rowi, es, cum,
                                             mfh, si);
        if (threadIdx.x == 0) out[rowi] = bi == 0x7fffffff ? 0 : bi;
      }
      cluster.sync();                             // the peers' candidates outlive the first block's reads
      return;
    }
    __syncthreads();
  }
  mx = warp_max(mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m2 = red[0];
    for (int w = 1; w < NT / 32; ++w) m2 = fmaxf(m2, red[w]);
    xc[0].f0 = m2;                                // travels with the first exchange
  }
  __syncthreads();

  // ---- 1. pivot = k-th largest scaled logit: 4 radix passes over shared memory
  float mxv = -INFINITY;                          // global max = max of the kept set
  bool have_max = false;
  uint32_t pivot_key = 0;
  if (use_k) {
    uint32_t prefix = 0;
    int need = top_k;
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      SampleXchg& x = xc[xi];
      for (int i = threadIdx.x; i < 256; i += NT) x.hist[i] = 0;
      __syncthreads();
      const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
      for (int i = threadIdx.x; i < n; i += NT) {
        const uint32_t key = float_order_key(vals[i]);
        if ((key & mask) == (prefix & mask)) atomicAdd(&x.hist[(key >> shift) & 255], 1u);
      }
      cluster.sync();
      if (threadIdx.x < 256) {
        unsigned int c = 0;
#pragma unroll
        for (int r = 0; r < CL; ++r) c += cluster.map_shared_rank(&xc[xi], r)->hist[threadIdx.x];
        mh[threadIdx.x] = c;
      }
      if (!have_max && threadIdx.x == 256 % NT) {
        float m2 = -INFINITY;
        for (int r = 0; r < CL; ++r) m2 = fmaxf(m2, cluster.map_shared_rank(&xc[0], r)->f0);
        s_needf = m2;
      }
      __syncthreads();
      if (!have_max) { mxv = s_needf; have_max = true; }
      if (threadIdx.x < 32) {
        // lane l holds bins 255 - 8 l downwards: the first bin whose running count from the top reaches `need`
        int c[8], mine = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) { c[j] = (int)mh[255 - 8 * (int)threadIdx.x - j]; mine += c[j]; }
        int before = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, before, o);
          if ((int)threadIdx.x >= o) before += y;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, before >= need);
        const int who = hit != 0 ? __ffs(hit) - 1 : 31;
        if ((int)threadIdx.x == who) {
          int nn = need - (before - mine), j = 0;
          for (; j < 7 && c[j] < nn; ++j) nn -= c[j];
          s_prefix = prefix | ((uint32_t)(255 - 8 * who - j) << shift);
          s_need = nn;
        }
      }
      __syncthreads();
      prefix = s_prefix;
      need = s_need;
      xi ^= 1;
    }
    pivot_key = prefix;
  }
  const float pivot = use_k ? key_to_float(pivot_key) : -INFINITY;

  // ---- 2. softmax statistics over the kept values (>= pivot)
  if (!have_max) {                                // no top-k: the max has not been exchanged yet
    cluster.sync();
    if (threadIdx.x == 0) {
      float m2 = -INFINITY;
      for (int r = 0; r < CL; ++r) m2 = fmaxf(m2, cluster.map_shared_rank(&xc[0], r)->f0);
      s_needf = m2;
    }
    __syncthreads();
    mxv = s_needf;
    xi = 1;                                       // copy 0 was just read by the peers
    __syncthreads();
  }
  float sum = 0.f;
  for (int i = threadIdx.x; i < n; i += NT) {
    const float v = vals[i];
    if (v >= pivot) sum += expf(v - mxv);
  }
  sum = block_sum<NT>(sum, red);
  if (threadIdx.x == 0) xc[xi].f1 = sum;
  cluster.sync();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int r = 0; r < CL; ++r) t += cluster.map_shared_rank(&xc[xi], r)->f1;   // fixed order: deterministic
    s_needf = t;
  }
  __syncthreads();
  sum = s_needf;
  xi ^= 1;
  __syncthreads();

  // ---- 2b. nucleus: largest probability threshold whose upper set has mass >= top_p
  float p_cut = 0.f;
  if (top_p > 0.f && top_p < 1.f) {
    uint32_t prefix = 0;
    float needf = top_p * sum;                    // in un-normalised mass
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass;
      SampleXchg& x = xc[xi];
      for (int i = threadIdx.x; i < 256; i += NT) x.fhist[i] = 0.f;
      __syncthreads();
      const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
      for (int i = threadIdx.x; i < n; i += NT) {
        const float v = vals[i];
        if (v >= pivot) {
          const float e = expf(v - mxv);
          const uint32_t key = float_order_key(e);
          if ((key & mask) == (prefix & mask)) atomicAdd(&x.fhist[(key >> shift) & 255], e);
        }
      }
      cluster.sync();
      if (threadIdx.x < 256) {
        float c = 0.f;
#pragma unroll
        for (int r = 0; r < CL; ++r) c += cluster.map_shared_rank(&xc[xi], r)->fhist[threadIdx.x];
        mfh[threadIdx.x] = c;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        float nn = needf;
        int b = 255;
        for (; b > 0; --b) {
          if (mfh[b] >= nn) break;
          nn -= mfh[b];
        }
        s_prefix = prefix | ((uint32_t)b << shift);
        s_needf = nn;
      }
      __syncthreads();
      prefix = s_prefix;
      needf = s_needf;
      xi ^= 1;
      __syncthreads();
    }
    p_cut = key_to_float(prefix);
  }

  // ---- 3. argmax(p / q) over the kept set; ties -> lowest index
  float best = -INFINITY;
  int bi = 0x7fffffff;
  for (int i = threadIdx.x; i < n; i += NT) {
    const float v = vals[i];
    if (v < pivot) continue;
    const float e = expf(v - mxv);
    if (e < p_cut) continue;
    const int gi = i0 + i;
    float qv;
    if (q_noise != nullptr) {
      qv = q_noise[(long long)rowi * V + gi];
    } else {
      const uint32_t r = mix32(seed * 0x9E3779B97F4A7C15ULL + ((unsigned long long)rowi << 32) + (unsigned)gi);
      const float u = ((float)(r & 0xffffff) + 0.5f) * (1.0f / 16777216.0f);
      qv = -logf(u);
    }
    const float sc = (e / sum) / qv;
    if (sc > best || (sc == best && gi < bi)) { best = sc; bi = gi; }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; si[threadIdx.x >> 5] = bi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < NT / 32; ++w)
      if (sv[w] > best || (sv[w] == best && si[w] < bi)) { best = sv[w]; bi = si[w]; }
    xc[xi].f0 = best;
    xc[xi].i0 = bi;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    for (int r = 1; r < CL; ++r) {
      const SampleXchg* px = cluster.map_shared_rank(&xc[xi], r);
      const float ov = px->f0;
      const int oi = px->i0;
      if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    out[rowi] = bi == 0x7fffffff ? 0 : bi;
  }
  cluster.sync();                                 // peers' shared memory must outlive rank 0's reads
}

// First-index arg-max of a row by a cluster of CL blocks: one block reads a 128256-entry row at about 50 GB/s.
template <int NT, int CL>
__global__ void __launch_bounds__(NT) xb_argmax_cluster_kernel(const float* __restrict__ logits, int V, int chunk, int* __restrict__ out) {
  __shared__ float sv[NT / 32];
  __shared__ int si[NT / 32];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), rowi = blockIdx.x / CL;
  const float* row = logits + (long long)rowi * V;
  const int i0 = rank * chunk, i1 = i0 + chunk < V ? i0 + chunk : V;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  auto take = [&](float v, int i) { if (v > best || (v == best && i < bi)) { best = v; bi = i; } };
  if ((V & 3) == 0 && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {   // chunk is a multiple of 4
    const float4* r4 = reinterpret_cast<const float4*>(row);
#pragma unroll 4
    for (int i = (i0 >> 2) + threadIdx.x; i < (i1 >> 2); i += NT) {
      const float4 a = r4[i];
      take(a.x, 4 * i); take(a.y, 4 * i + 1); take(a.z, 4 * i + 2); take(a.w, 4 * i + 3);
    }
  } else {
    for (int i = i0 + threadIdx.x; i < i1; i += NT) take(row[i], i);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    take(ov, oi);
  }
  if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = best; si[threadIdx.x >> 5] = bi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < NT / 32; ++w) take(sv[w], si[w]);
    sv[0] = best;
    si[0] = bi;
  }
  cluster.sync();
  if (rank == 0 && threadIdx.x == 0) {
    for (int r = 1; r < CL; ++r) take(cluster.map_shared_rank(sv, r)[0], cluster.map_shared_rank(si, r)[0]);
    out[rowi] = bi == 0x7fffffff ? 0 : bi;
  }
  cluster.sync();
}
