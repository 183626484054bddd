// Row-wise kernels of hybrid prompts, four neighbouring channels per thread.
//
// The one-channel forms (hy_taps_tile_kernel, hy_hgrn_prep_kernel, hy_act_cols_kernel, hy_row_op_kernel, hy_gdelta_prep_kernel) issue 2- and
// 4-byte accesses and were bound by instructions and by loads in flight, at 0.15 to 0.35 of the copy rate.  These take
// 8- and 16-byte accesses where the operand is one bf16 or fp32 matrix (prompts; split-K planes of few rows keep the others), rows,
// columns and pitches are multiples of four and pointers are aligned (hy_quad).  Per channel the arithmetic is the same;
// sums over a row are taken in another order.
// us a launch, before -> now, 2048 rows: filter of 2048 channels fp32 -> bf16 27.9 -> 15.8, q|k|v filter of 6144 channels 59 -> 38, HGRN2
// preparation 53.5 -> 17.4, residual + norm of the stream 24.3 -> 17.4; 1800 rows: parallel block's residual + norm 27.1 -> 14.6, SiLU of
// 6144 columns 46.8 -> 15.6, general delta rule's preparation 55.6 -> 28.3.
#pragma once

__device__ __forceinline__ void hy_quad_bf(const bf16* p, float* v) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = bf2_to_f2(u.x), b = bf2_to_f2(u.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void hy_quad_f(const float* p, float* v) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
// one matrix (no planes), see hy_quad
__device__ __forceinline__ void lin_quad(const LinOut& o, long long row, int col, float* v) {
  if (o.h != nullptr) hy_quad_bf(o.h + row * o.ld + col, v);
  else hy_quad_f(o.f + row * o.ld + col, v);
  if (o.bias != nullptr) {
    float b[4];
    hy_quad_f(o.bias + col, b);
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] += b[j];
  }
}
__device__ __forceinline__ void hy_quad_st(float* p, const float* v) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void hy_quad_st(bf16* p, const float* v) {
  *reinterpret_cast<uint2*>(p) = make_uint2(f2_to_bf2(v[0], v[1]), f2_to_bf2(v[2], v[3]));
}
// can `o` be read four columns at a time from column `col` (a multiple of four) on?
static bool hy_quad(const LinOut& o, int col) {
  if (o.ld % 4 != 0 || col % 4 != 0 || (o.bias != nullptr && (reinterpret_cast<uintptr_t>(o.bias) & 15) != 0)) return false;
  if (o.h != nullptr) return (reinterpret_cast<uintptr_t>(o.h) & 7) == 0;
  return o.f != nullptr && o.si.splits == 0 && (reinterpret_cast<uintptr_t>(o.f) & 15) == 0;
}
// the same for split-K planes, each of which starts on 16 bytes
static bool hy_planes4(const LinOut& o, int col) {
  if (o.f == nullptr || o.si.splits == 0) return hy_quad(o, col);
  return o.ld % 4 == 0 && o.plane % 4 == 0 && col % 4 == 0 && (reinterpret_cast<uintptr_t>(o.f) & 15) == 0 && (reinterpret_cast<uintptr_t>(o.bias) & 15) == 0;
}
static bool hy_quad_ptr(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// hy_taps_tile_kernel with TT = 8 rows and four channels per thread; C, ld_out and tail_stride multiples of four
template <typename OT, int TAPS>
__global__ void __launch_bounds__(256) hy_taps_quad_kernel(LinOut in, int col0, int C, const float* __restrict__ w, const float* __restrict__ tail,
                                                           long long tail_stride, BatchMeta m, int identity, int act_silu, OT* __restrict__ out,
                                                           long long ld_out, int T) {
  constexpr int TT = 8;
  pdl_launch_dependents();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
  if (c >= C) return;
  // Two dependent trips: the step's metadata and the filter, then the eight rows and the rows before them together; sequence, place, rows and window one after the
  // other took four (2048 rows x 2048 channels 15.8 -> 14.3 us).  In steps that launch ahead (up to 128 rows) the first lies before the wait.
  const int r0 = blockIdx.x * TT;
  const int last_row = (r0 + TT < T ? r0 + TT : T) - 1;
  const int s_first = m.tok_seq[r0];
  const bool uniform = s_first == m.tok_seq[last_row];
  const int first_start = s_first > 0 ? m.seq_last[s_first - 1] + 1 : 0, first_pos = m.tok_pos[r0], first_pos0 = m.tok_pos[first_start];
  const float* first_tail = tail + (long long)m.seq_slot[s_first] * tail_stride;
  float wv[TAPS][4];
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int j = 0; j < TAPS; ++j) wv[j][e] = w[(long long)(c + e) * TAPS + j];
  pdl_wait();
  float win[TAPS][4];   // win[d - 1]: the input d steps back (TAPS - 1 used)
#pragma unroll
  for (int d = 0; d < TAPS; ++d)
#pragma unroll
    for (int e = 0; e < 4; ++e) win[d][e] = 0.f;
  auto window = [&](int row, int start, int pos, int pos0, const float* tl) {
#pragma unroll
    for (int d = 1; d < TAPS; ++d) {
      const int p = pos - d;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (p >= 0) {
        if (row - d >= start) lin_quad(in, row - d, col0 + c, v);
        else hy_quad_f(tl + (long long)(p - (pos0 - (TAPS - 1))) * C + c, v);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) win[d - 1][e] = v[e];
    }
  };
  float cur[TT][4];
#pragma unroll
  for (int i = 0; i < TT; ++i) lin_quad(in, r0 + i <= last_row ? r0 + i : last_row, col0 + c, cur[i]);
  window(r0, first_start, first_pos, first_pos0, first_tail);
#pragma unroll
  for (int i = 0; i < TT; ++i) {
    const int row = r0 + i;
    if (row > last_row) break;
    if (!uniform && i > 0) {
      const int s = m.tok_seq[row];
      if (m.tok_seq[row - 1] != s) {   // a sequence begins here
        const int pos = m.tok_pos[row];
        window(row, row, pos, pos, tail + (long long)m.seq_slot[s] * tail_stride);
      }
    }
    float acc[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      acc[e] = identity ? cur[i][e] : 0.f;
#pragma unroll
      for (int j = 0; j < TAPS - 1; ++j) acc[e] += wv[j][e] * win[TAPS - 2 - j][e];   // oldest first
      acc[e] += wv[TAPS - 1][e] * cur[i][e];
      if (act_silu) acc[e] = hy_silu(acc[e]);
#pragma unroll
      for (int d = TAPS - 1; d >= 2; --d) win[d - 1][e] = win[d - 2][e];
      win[0][e] = cur[i][e];
    }
    hy_quad_st(out + (long long)row * ld_out + c, acc);
  }
}

// hy_hgrn_prep_kernel; HK and HV multiples of four
__global__ void __launch_bounds__(256) hy_hgrn_prep_quad_kernel(LinOut P, int off_q, int off_f, int off_v, const float* __restrict__ lower,
                                                                float* __restrict__ c, long long ldc, int HK, int HV) {
  pdl_launch_dependents();
  pdl_wait();
  const long long t = blockIdx.x;
  const int i = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (i >= 2 * HK + HV) return;
  float v[4];
  if (i < HK) {
    lin_quad(P, t, off_q + i, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = hy_silu(v[e]);
  } else if (i < 2 * HK) {
    lin_quad(P, t, off_f + i - HK, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float lo = lower[i - HK + e];
      v[e] = lo + (1.0f - lo) * hy_sigmoid(v[e]);
    }
  } else {
    lin_quad(P, t, off_v + i - 2 * HK, v);
  }
  hy_quad_st(c + t * ldc + i, v);
}

// hy_act_cols_kernel; n a multiple of four
template <typename OT>
__global__ void __launch_bounds__(256) hy_act_cols_quad_kernel(LinOut P, int off, int n, int act, OT* __restrict__ out, long long ld_out) {
  pdl_launch_dependents();
  pdl_wait();
  const long long t = blockIdx.x;
  const int i = (blockIdx.y * 256 + threadIdx.x) * 4;
  if (i >= n) return;
  float v[4];
  lin_quad(P, t, off + i, v);
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] = act == 0 ? hy_silu(v[e]) : tanhf(v[e]);
  hy_quad_st(out + t * ld_out + i, v);
}

// hy_row_op_kernel (every form of it); D a multiple of four
template <typename AT>
__global__ void __launch_bounds__(256) hy_row_op_quad_kernel(RowOpArgs a) {
  constexpr int NT = 256;
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float row[];
  __shared__ float red[32];
  const long long t = blockIdx.x;
  const int D = a.D;
  float* x = a.x + t * D;
  const bool branch = a.m1.f != nullptr || a.m1.h != nullptr;
  const bool two = a.m2.f != nullptr || a.m2.h != nullptr;
  const bool three = a.plain_add && (a.m3.f != nullptr || a.m3.h != nullptr);
  float s2 = 0.f;
  float inv = 0.f;
  if (branch && !a.plain_add) {   // the branch's own norm
    float ss = 0.f;
    for (int i = threadIdx.x * 4; i < D; i += NT * 4) {
      float v[4], b[4];
      lin_quad(a.m1, t, i, v);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] *= a.s1;
      if (two) {
        lin_quad(a.m2, t, i, b);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] += a.s2 * b[e];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) ss += v[e] * v[e];
      hy_quad_st(row + i, v);
    }
    ss = block_sum<NT>(ss, red);
    inv = 1.0f / sqrtf(ss / (float)D + a.eps);
  }
  for (int i = threadIdx.x * 4; i < D; i += NT * 4) {
    float v[4], b[4];
    hy_quad_f(x + i, v);
    if (branch && a.plain_add) {
      float y[4];
      lin_quad(a.m1, t, i, y);
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] *= a.s1;
      if (two) {
        lin_quad(a.m2, t, i, b);
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] += a.s2 * b[e];
      }
      if (three) {
        lin_quad(a.m3, t, i, b);
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] += b[e];
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] += y[e];
    } else if (branch) {
      float w[4];
      hy_quad_f(row + i, b);   // this thread wrote them
      hy_quad_f(a.bw + i, w);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] += b[e] * inv * (w[e] + a.bw_one);
    }
    if (branch) hy_quad_st(x + i, v);
    hy_quad_st(row + i, v);
#pragma unroll
    for (int e = 0; e < 4; ++e) s2 += v[e] * v[e];
  }
  if (a.nw != nullptr) {
    s2 = block_sum<NT>(s2, red);
    const float inv2 = 1.0f / sqrtf(s2 / (float)D + a.eps);
    for (int i = threadIdx.x * 4; i < D; i += NT * 4) {
      float v[4];
      hy_quad_f(row + i, v);
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = v[e] * inv2 * hy_norm_weight(a.nw, a.nw_mode, i + e);
      hy_quad_st(a.hn + t * D + i, v);
      if (a.ha != nullptr) hy_quad_st(reinterpret_cast<AT*>(a.ha) + t * D + i, v);
    }
  }
  if (a.xa != nullptr) {
    AT* xa = reinterpret_cast<AT*>(a.xa) + t * D;
    for (int i = threadIdx.x * 4; i < D; i += NT * 4) {
      float v[4];
      hy_quad_f(row + i, v);
      hy_quad_st(xa + i, v);
    }
  }
}

// hy_gdelta_prep_kernel; n / 4 lanes per head (a power of two up to 32), grid ceil(T * H * n / 4 / 256)
__global__ void __launch_bounds__(256) hy_gdelta_prep_quad_kernel(LinOut P, int off_r, int off_k, int off_v, int off_a, LinOut Wd,
                                                                  const float* __restrict__ w0, float* __restrict__ c, long long ldc,
                                                                  float* __restrict__ ra, float* __restrict__ rk, int H, int n, int T) {
  pdl_launch_dependents();
  pdl_wait();
  const int per = n >> 2;
  const long long idx = (long long)blockIdx.x * 256 + threadIdx.x, all = (long long)T * H * per;
  const bool live = idx < all;
  const long long th = (live ? idx : all - 1) / per;
  const int i = (int)((live ? idx : all - 1) - th * per) * 4;
  const long long t = th / H, HN = (long long)H * n;
  const int h = (int)(th - t * H), b = h * n + i;
  float r[4], k[4], v[4], z[4], aa[4], w[4];
  lin_quad(P, t, off_r + b, r);
  lin_quad(P, t, off_k + b, k);
  lin_quad(P, t, off_v + b, v);
  lin_quad(P, t, off_a + b, aa);
  lin_quad(Wd, t, b, w);
  hy_quad_f(w0 + b, z);
  float sk = 0.f;
#pragma unroll
  for (int e = 0; e < 4; ++e) sk = fmaf(k[e], k[e], sk);
  for (int off = per >> 1; off > 0; off >>= 1) sk += __shfl_xor_sync(0xffffffffu, sk, off);
  const float ik = 1.0f / sqrtf(sk + 1e-6f);
  float s_ra = 0.f, s_rk = 0.f, rw[4], u[4], au[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    w[e] = expf(-0.6065306597126334f * hy_sigmoid(w[e] + z[e]));
    u[e] = k[e] * ik;
    au[e] = hy_sigmoid(aa[e]) * u[e];
    rw[e] = r[e] * w[e];
    s_ra = fmaf(r[e], au[e], s_ra);
    s_rk = fmaf(r[e], k[e], s_rk);
  }
  for (int off = per >> 1; off > 0; off >>= 1) {
    s_ra += __shfl_xor_sync(0xffffffffu, s_ra, off);
    s_rk += __shfl_xor_sync(0xffffffffu, s_rk, off);
  }
  if (!live) return;
  float* row = c + t * ldc + b;
  hy_quad_st(row, rw);
  hy_quad_st(row + HN, u);
  hy_quad_st(row + 2 * HN, w);
  hy_quad_st(row + 3 * HN, au);
  hy_quad_st(row + 4 * HN, k);
  hy_quad_st(row + 5 * HN, v);
  if (i == 0) { ra[t * H + h] = s_ra; rk[t * H + h] = s_rk; }
}

// hy_row_op_kernel for steps of few rows: a thread holds four neighbouring channels per VPT from the loads to the stores, so a row costs one trip for
// planes and stream, four barriers and the stores; sums and squares add up in the general kernel's order, bit for bit.  What waits for no kernel (weights, plane counts) is fetched ahead of the wait.  The general kernel
// reads stream and weights behind its first sum, weights again behind the second, keeps the row in shared memory, and its 1024 threads of 64 registers
// take a whole SM: the next Linear's block cannot come in beside them and starts its weights when the norm is done.
// The bound of one block an SM keeps F planes of four channels in flight (see xb_resid_norm_row_kernel).  Eight chats of three bibevik-1b layers (four such
// kernels a token) 4386 -> 4243 us; with an order of its own for the squares and two barriers it took the same.
template <int F>
__device__ __forceinline__ void lin_planes4(const LinOut& o, long long row, int col, int planes, float* v) {   // lin_at's order of planes
  float b[4] = {0.f, 0.f, 0.f, 0.f};
  if (o.bias != nullptr) hy_quad_f(o.bias + col, b);
  if (o.h != nullptr) {
    hy_quad_bf(o.h + row * o.ld + col, v);
  } else {
    const float* p = o.f + row * o.ld + col;
    v[0] = v[1] = v[2] = v[3] = 0.f;
    for (int s0 = 0; s0 < planes; s0 += F) {
      float w[F][4];
#pragma unroll
      for (int u = 0; u < F; ++u) hy_quad_f(p + (s0 + u < planes ? s0 + u : 0) * o.plane, w[u]);
#pragma unroll
      for (int u = 0; u < F; u += 4) {
        if (s0 + u + 3 < planes) {
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += (w[u][j] + w[u + 1][j]) + (w[u + 2][j] + w[u + 3][j]);
        } else {
#pragma unroll
          for (int q = 0; q < 3; ++q)
            if (s0 + u + q < planes) {
#pragma unroll
              for (int j = 0; j < 4; ++j) v[j] += w[u + q][j];
            }
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) v[j] += b[j];
}
__device__ __forceinline__ int lin_planes(const LinOut& o, int col) {
  return o.f == nullptr ? 0 : o.si.splits == 0 ? 1 : xb_n_segments(o.si, col);
}
// The sum of squares of a row of up to 2 VPT * 1024 channels in the order of hy_row_op_kernel<., 1024>: its thread i adds the channels i, i + 1024, ..; then warps,
// then their sums.  Here thread q of each half of 512 threads holds VPT pieces of the channels 4 q .. 4 q + 3 (mod 1024), the upper half carrying on where the
// lower one stops, and thread i is element i & 3 of eight neighbouring lanes.  v: zeros where the row has ended (n[it] false).
template <int VPT>
__device__ __forceinline__ float row_sum_1024(const float (&v)[VPT][4], const bool (&n)[VPT], float4* low, float* red) {
  const int q = threadIdx.x & 255;
  float s[4] = {0.f, 0.f, 0.f, 0.f};
  auto add = [&]() {
#pragma unroll
    for (int it = 0; it < VPT; ++it)
      if (n[it]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) s[j] = fmaf(v[it][j], v[it][j], s[j]);
      }
  };
  if (threadIdx.x < 256) {
    add();
    low[q] = make_float4(s[0], s[1], s[2], s[3]);
  }
  __syncthreads();
  if (threadIdx.x >= 256) {
    const float4 l = low[q];
    s[0] = l.x; s[1] = l.y; s[2] = l.z; s[3] = l.w;
    add();
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
    if ((q & 7) == 0) red[q >> 3] = (s[0] + s[2]) + (s[1] + s[3]);
  }
  __syncthreads();
  return warp_sum(red[threadIdx.x & 31]);
}

template <typename AT, int VPT, int F>
__global__ void __launch_bounds__(512, 1) hy_row_op_few_kernel(RowOpArgs a) {
  pdl_launch_dependents();
  __shared__ float4 low[256];   // used once a sum, with two barriers between
  __shared__ float red[2][32];
  const long long t = blockIdx.x;
  const int D = a.D, c0 = (threadIdx.x >> 8) * VPT * 1024 + (threadIdx.x & 255) * 4;
  const bool branch = a.m1.f != nullptr || a.m1.h != nullptr, two = a.m2.f != nullptr || a.m2.h != nullptr, three = a.m3.f != nullptr || a.m3.h != nullptr;
  float bw[VPT][4], nw[VPT][4], x[VPT][4], v[VPT][4];
  int n1[VPT], n2[VPT], n3[VPT];
  bool in[VPT];
#pragma unroll
  for (int it = 0; it < VPT; ++it) {
    const int c = c0 + it * 1024;
    in[it] = c < D;
#pragma unroll
    for (int j = 0; j < 4; ++j) bw[it][j] = nw[it][j] = x[it][j] = v[it][j] = 0.f;
    if (in[it] && branch && !a.plain_add) hy_quad_f(a.bw + c, bw[it]);
    if (in[it] && a.nw != nullptr) {
      if (a.nw_mode == 2) nw[it][0] = nw[it][1] = nw[it][2] = nw[it][3] = a.nw[0];
      else hy_quad_f(a.nw + c, nw[it]);
    }
    n1[it] = in[it] && branch ? lin_planes(a.m1, c) : 0;
    n2[it] = in[it] && two ? lin_planes(a.m2, c) : 0;
    n3[it] = in[it] && three ? lin_planes(a.m3, c) : 0;
  }
  pdl_wait();
#pragma unroll
  for (int it = 0; it < VPT; ++it) {
    const int c = c0 + it * 1024;
    if (!in[it]) break;
    hy_quad_f(a.x + t * D + c, x[it]);
    if (branch) {
      float u[4];
      lin_planes4<F>(a.m1, t, c, n1[it], u);
#pragma unroll
      for (int j = 0; j < 4; ++j) v[it][j] = a.s1 * u[j];
      if (two) {
        lin_planes4<F>(a.m2, t, c, n2[it], u);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[it][j] += a.s2 * u[j];
      }
      if (a.plain_add && three) {
        lin_planes4<F>(a.m3, t, c, n3[it], u);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[it][j] += u[j];
      }
    }
  }
  const float inv = branch && !a.plain_add ? 1.0f / sqrtf(row_sum_1024<VPT>(v, in, low, red[0]) / (float)D + a.eps) : 0.f;
#pragma unroll
  for (int it = 0; it < VPT; ++it) {
    const int c = c0 + it * 1024;
    if (!in[it]) break;
    if (branch && a.plain_add) {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[it][j] += v[it][j];
    } else if (branch) {
#pragma unroll
      for (int j = 0; j < 4; ++j) x[it][j] = fmaf(v[it][j] * inv, bw[it][j] + a.bw_one, x[it][j]);   // as hy_row_op_kernel's line comes out
    }
    if (branch) hy_quad_st(a.x + t * D + c, x[it]);
    if (a.xa != nullptr) hy_quad_st(reinterpret_cast<AT*>(a.xa) + t * D + c, x[it]);
  }
  if (a.nw == nullptr) return;
  const float inv2 = 1.0f / sqrtf(row_sum_1024<VPT>(x, in, low, red[1]) / (float)D + a.eps);
#pragma unroll
  for (int it = 0; it < VPT; ++it) {
    const int c = c0 + it * 1024;
    if (!in[it]) break;
    float h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = x[it][j] * inv2 * (a.nw_mode == 0 ? 1.0f + nw[it][j] : nw[it][j]);
    hy_quad_st(a.hn + t * D + c, h);
    if (a.ha != nullptr) hy_quad_st(reinterpret_cast<AT*>(a.ha) + t * D + c, h);
  }
}

// hy_glu_kernel, hy_moe_act_kernel and hy_logits_kernel on split-K planes or one matrix, four neighbouring columns a thread, a row a grid row (no 64-bit
// division per element), plane counts ahead of the wait and every plane of the columns in flight.  Widths multiples of four, see hy_planes4.  Eight chats of
// three bibevik-1b layers 4035 -> 3945 us.
template <typename AT>
__global__ void __launch_bounds__(128, 4) hy_glu_few_kernel(LinOut U, int F, float limit, int act, AT* __restrict__ out, long long ld_out) {
  pdl_launch_dependents();
  const int t = blockIdx.y, i = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (i >= F) return;
  const int ng = lin_planes(U, i), nu = lin_planes(U, F + i);
  pdl_wait();
  float g[4], u[4];
  lin_planes4<4>(U, t, i, ng, g);
  lin_planes4<4>(U, t, F + i, nu, u);
#pragma unroll
  for (int j = 0; j < 4; ++j) g[j] = hy_expert_act(g[j], u[j], 1.0f, limit, act, 0);
  hy_quad_st(out + t * ld_out + i, g);
}
template <typename AT>
__global__ void __launch_bounds__(128, 4) hy_moe_act_few_kernel(LinOut U, const float* __restrict__ gw, int ldg, int sg_at, int E, int f, float limit, int sf, float limit_s,
                                                                int act, int on_input, AT* __restrict__ out, long long ld_out) {
  pdl_launch_dependents();
  const int t = blockIdx.y, i = (blockIdx.x * 128 + threadIdx.x) * 4, routed = E * f;
  if (i >= routed + sf) return;
  const bool shared = i >= routed;
  const int e = shared ? 0 : i / f, cg = shared ? routed + i : e * f + i, cu = cg + (shared ? sf : f);
  const int ng = lin_planes(U, cg), nu = lin_planes(U, cu);
  pdl_wait();
  const float w = shared ? hy_shared_weight(gw + (long long)t * ldg, sg_at) : gw[(long long)t * ldg + e];
  float g[4] = {0.f, 0.f, 0.f, 0.f}, u[4];
  if (shared || w != 0.f) {
    lin_planes4<4>(U, t, cg, ng, g);
    lin_planes4<4>(U, t, cu, nu, u);
#pragma unroll
    for (int j = 0; j < 4; ++j) g[j] = hy_expert_act(g[j], u[j], w, shared ? limit_s : limit, act, shared ? 0 : on_input);
  }
  hy_quad_st(out + t * ld_out + i, g);
}
__global__ void __launch_bounds__(256, 4) hy_logits_few_kernel(LinOut y, float cap, float* __restrict__ out, int V) {
  pdl_launch_dependents();
  const int t = blockIdx.y, i = (blockIdx.x * 256 + threadIdx.x) * 4;
  if (i >= V) return;
  const int n = lin_planes(y, i);
  pdl_wait();
  float v[4];
  lin_planes4<4>(y, t, i, n, v);
  if (cap > 0.f) {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = cap * tanhf(v[j] / cap);
  }
  hy_quad_st(out + (long long)t * V + i, v);
}
