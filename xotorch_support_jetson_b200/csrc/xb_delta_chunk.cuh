// The delta rules of prompts, sixteen tokens at a time (gated delta rule, general delta rule; see hy_recur_kernel for the steps).
//
// Token by token every step waits for a chain of dot product, shuffles and update: 0.36 us a step whatever the width.  Here
// the sixteen tokens of a chunk read the state S_0 they start from side by side, and what the earlier tokens of the chunk have
// written enters through small matrices that are the same for every value column:
//
//   gated delta rule    S_i = g_i S_(i-1) + k_i u_i,  u_i = beta_i (v_i - g_i a_i),  a_i = k_i . S_(i-1),  G_i = g_1 .. g_i
//     a_i = G_(i-1) k_i.S_0 + sum_(j<i) D_ij (k_i.k_j) u_j,  b_i = the same with q_i,  D_ij = g_(j+1) .. g_(i-1) (a product: any decay, zero
//     included),  o_i = g_i b_i + (q_i.k_i) u_i,  S_16 = G_16 S_0 + sum_j g_(j+1) .. g_16 k_j u_j
//   general delta rule  S_i = w_i*S_(i-1) - (au)_i a_i + k_i v_i,  a_i = u_i . S_(i-1),  P_i = w_1*..*w_i per channel (w >= e^-0.61, so P_16
//     >= 6e-5 and dividing by it is harmless)
//     a_i = (u_i P_(i-1)).S_0 + sum_(j<i) ((u_i P_(i-1)).(k_j / P_j)) v_j - ((u_i P_(i-1)).((au)_j / P_j)) a_j,  b_i = the same with (r w)_i,
//     o_i = b_i - (r_i.(au)_i) a_i + (r_i.k_i) v_i,  S_16 = P_16*(S_0 + sum_j (k_j / P_j) v_j - ((au)_j / P_j) a_j)
//
// All fp32.  hy_chunk_prep_kernel makes a block of numbers per (chunk, head), hy_chunk_kernel walks the chunks of a sequence: sixteen lanes
// share two value columns (lane `sub` holds the rows of the 16-byte pieces sub, sub + 16, .. of each, in pairs for the packed two-wide
// FMA), the 2 x 16 dot products of a chunk are reduced together by halving exchanges, after which lane i owns token i, and only the
// triangular solve goes token by token.  Bound by instruction issue (about a thousand a chunk and warp, one warp a scheduler) and by that
// solve.
// 2048 tokens, 16 heads of 128 x 128 (gated): 741 -> 212 us and 41 us of preparation; 450 and 1350 tokens, 32 heads of 64 x 64
// (general): 777 -> 218 and 84 us, with launch bounds that leave the walk its registers and the preparation four blocks an SM 206 and 80
// (gated 211 and 40).  Errors against 64 bits as token by token (3.4e-7 and 2.9e-7 after 2047 tokens).
#pragma once

#define HY_CT 16          // tokens of a chunk = lanes that share a column
#define HY_CHUNK_VP 18    // pitch of the chunk's 16 x 16 values in shared memory
#define HY_CHUNK_BYTES ((size_t)192 << 20)   // most the prepared blocks may take (bibevik-1b: 4500 tokens, refatar-1b: 10000); steps beyond that go in parts
// Tokens of the step's longest sequence from which the chunks are used: the longest one sets the time of either form while the chip has room
// for all of them.  A layer in bf16, token by token -> chunks: gated, 32 tokens 257 -> 245 us,
// two of 64 417 -> 388; general, 32 tokens 241 -> 236, 33 237 -> 239, two of 64 363 -> 359, six of 100 493 -> 430.
// Where sequences fill the chip token by token is as fast or faster, hence a limit on the blocks of the walk per SM that run abreast.  A bf16 step of
// one layer (128 blocks a sequence), token by token -> chunks, us, gated / general: 2 x 200 tokens 410 -> 373 / 382 -> 333, 4 x 500 782 -> 717 / 782 -> 696, 10 x
// 500 1470 -> 1412 / 1465 -> 1471, 14 x 500 1877 -> 1895 / 2245 -> 2023, 20 x 200 1164 -> 1188 / 1200 -> 1219; below 200 tokens 4 x 100 388 -> 380 / 347 -> 340,
// 6 x 100 423 -> 434 / 386 -> 389, 10 x 100 510 -> 510 / 461 -> 474, 64 x 40 (gated) 913 -> 995.  One of 1000 beside 60 of one: 981 -> 769 / 1074 -> 791.
__host__ __device__ constexpr int hy_chunk_abreast(int mode, long long longest_chunks) { return longest_chunks < 13 ? 4 : mode == HY_REC_GDELTA ? 16 : 11; }
__host__ __device__ constexpr int hy_chunk_min(int mode) { return mode == HY_REC_GDELTA ? 96 : 32; }
__host__ __device__ constexpr int hy_chunk_vectors(int mode) { return mode == HY_REC_GDELTA ? 4 : 2; }
// floats of one (chunk, head): the row vectors [vectors][16][dkp], for the general rule P_16 [dkp], the matrices [16][16], sixteen numbers per token
__host__ __device__ constexpr int hy_chunk_mats(int mode, int dkp) { return hy_chunk_vectors(mode) * HY_CT * dkp + (mode == HY_REC_GDELTA ? dkp : 0); }
__host__ __device__ constexpr int hy_chunk_scal(int mode, int dkp) { return hy_chunk_mats(mode, dkp) + hy_chunk_vectors(mode) * HY_CT * HY_CT; }
__host__ __device__ constexpr int hy_chunk_block(int mode, int dkp) { return hy_chunk_scal(mode, dkp) + 6 * HY_CT; }

// Where the blocks of a step lie.  per = 0, all of them at once: chunk c of sequence s at entry start_row / 16 + s + c (no two sequences share
// one), grid T / 16 + n_seqs.  per > 0, the chunks [c0, c0 + per) of every sequence: entry s * per + c - c0, grid n_seqs * per.
struct ChunkPart {
  int c0, per;
};
// grid (entries, H), 256 threads; dynamic shared memory: the row vectors (general rule: and the decays) at pitch dkp + 4
template <int MODE>
__global__ void __launch_bounds__(256, 4) hy_chunk_prep_kernel(RecurIn in, float* __restrict__ ws, BatchMeta m, ChunkPart part, int n_seqs, int H, int dk,
                                                            int dkp) {
  extern __shared__ __align__(16) float cps[];
  __shared__ float gs[HY_CT];
  pdl_launch_dependents();
  pdl_wait();
  int s = 0, start = 0, len = 0, c = -1;
  if (part.per > 0) {
    s = blockIdx.x / part.per;
    c = part.c0 + (int)blockIdx.x - s * part.per;
    start = s > 0 ? m.seq_last[s - 1] + 1 : 0;
    len = m.seq_last[s] - start + 1;
    if (c * HY_CT >= len) return;
  } else {
    for (; s < n_seqs; ++s) {
      start = s > 0 ? m.seq_last[s - 1] + 1 : 0;
      len = m.seq_last[s] - start + 1;
      c = (int)blockIdx.x - (start / HY_CT + s);
      if (c < 0) return;
      if (c * HY_CT < len) break;
    }
    if (s == n_seqs) return;
  }
  const int h = blockIdx.y, g = h / (H / in.q_heads), tid = threadIdx.x;
  const int nt = len - c * HY_CT < HY_CT ? len - c * HY_CT : HY_CT;
  const long long row0 = start + c * HY_CT;
  float* blk = ws + ((long long)blockIdx.x * H + h) * hy_chunk_block(MODE, dkp);
  float* mats = blk + hy_chunk_mats(MODE, dkp);
  float* scal = blk + hy_chunk_scal(MODE, dkp);
  const int pitch = dkp + 4;
  if (MODE == HY_REC_DELTA) {
    for (int x = tid; x < HY_CT * dkp; x += 256) {
      const int t = x / dkp, r = x - t * dkp;
      const bool have = t < nt && r < dk;
      const float* src = in.c + (row0 + t) * in.ldc + (long long)g * dk + r;
      const float k = have ? src[in.koff] : 0.f, q = have ? src[in.qoff] : 0.f;
      cps[t * pitch + r] = k;
      cps[(HY_CT + t) * pitch + r] = q;
      blk[x] = k;
      blk[HY_CT * dkp + x] = q;
    }
    if (tid < HY_CT) gs[tid] = tid < nt ? in.decay[(row0 + tid) * H + h] : 1.f;
    __syncthreads();
    const int i = tid & 15, j = tid >> 4;   // matrices lie column by column: lane i of the walk reads its row without bank conflicts
    float kk = 0.f, qk = 0.f;
    if (j < i) {
      const float *ki = cps + i * pitch, *qi = cps + (HY_CT + i) * pitch, *kj = cps + j * pitch;
      float kb = 0.f, qb = 0.f;
      for (int r = 0; r < dkp; r += 4) {
        const float4 a = *reinterpret_cast<const float4*>(ki + r), b = *reinterpret_cast<const float4*>(qi + r), x = *reinterpret_cast<const float4*>(kj + r);
        kk = fmaf(a.x, x.x, kk); kb = fmaf(a.y, x.y, kb); kk = fmaf(a.z, x.z, kk); kb = fmaf(a.w, x.w, kb);
        qk = fmaf(b.x, x.x, qk); qb = fmaf(b.y, x.y, qb); qk = fmaf(b.z, x.z, qk); qb = fmaf(b.w, x.w, qb);
      }
      float d = 1.f;
      for (int l = j + 1; l < i; ++l) d *= gs[l];
      kk = (kk + kb) * d;
      qk = (qk + qb) * d;
    }
    mats[tid] = kk;
    mats[HY_CT * HY_CT + tid] = qk;
    if (tid < HY_CT) {   // per token: beta, g, q.k, G before it, decay behind it up to the chunk's end; the whole chunk's decay
      float before = 1.f, behind = 1.f, all = 1.f;
      for (int l = 0; l < HY_CT; ++l) {
        if (l < tid) before *= gs[l];
        if (l > tid) behind *= gs[l];
        all *= gs[l];
      }
      const bool have = tid < nt;
      scal[tid] = have ? in.beta[(row0 + tid) * H + h] : 0.f;
      scal[HY_CT + tid] = gs[tid];
      scal[2 * HY_CT + tid] = have ? in.qk[(row0 + tid) * in.q_heads + g] : 0.f;
      scal[3 * HY_CT + tid] = before;
      scal[4 * HY_CT + tid] = behind;
      scal[5 * HY_CT + tid] = all;
    }
  } else {
    float* wv = cps + 4 * HY_CT * pitch;
    const int n4 = HY_CT * dkp;
#pragma unroll 4
    for (int x = tid; x < n4; x += 256) {   // u, r*w, k, a*u, w as they are
      const int t = x / dkp, r = x - t * dkp;
      const bool have = t < nt && r < dk;
      const float* src = in.c + (row0 + t) * in.ldc + (long long)g * dk + r;
      cps[t * pitch + r] = have ? src[in.koff] : 0.f;
      cps[(HY_CT + t) * pitch + r] = have ? src[in.qoff] : 0.f;
      cps[(2 * HY_CT + t) * pitch + r] = have ? src[in.xoff[2]] : 0.f;
      cps[(3 * HY_CT + t) * pitch + r] = have ? src[in.xoff[1]] : 0.f;
      wv[t * pitch + r] = have ? src[in.xoff[0]] : 1.f;
    }
    __syncthreads();
    for (int r = tid; r < dkp; r += 256) {
      float P = 1.f;
#pragma unroll
      for (int t = 0; t < HY_CT; ++t) {
        float* x = cps + t * pitch + r;
        x[0] *= P;                          // before this token's decay
        x[HY_CT * pitch] *= P;
        P *= wv[t * pitch + r];
        const float ip = 1.0f / P;
        x[2 * HY_CT * pitch] *= ip;
        x[3 * HY_CT * pitch] *= ip;
      }
      blk[4 * HY_CT * dkp + r] = P;
    }
    __syncthreads();
    for (int x = tid; x < 4 * n4; x += 256) {
      const int t = x / dkp, r = x - t * dkp;
      blk[x] = cps[t * pitch + r];
    }
    const int i = tid & 15, j = tid >> 4;   // matrices lie column by column: lane i of the walk reads its row without bank conflicts
    float o[4] = {0.f, 0.f, 0.f, 0.f};   // u.k, u.e, q.k, q.e
    if (j < i) {
      const float *ui = cps + i * pitch, *qi = cps + (HY_CT + i) * pitch, *kj = cps + (2 * HY_CT + j) * pitch, *ej = cps + (3 * HY_CT + j) * pitch;
      for (int r = 0; r < dkp; r += 4) {
        const float4 a = *reinterpret_cast<const float4*>(ui + r), b = *reinterpret_cast<const float4*>(qi + r);
        const float4 x = *reinterpret_cast<const float4*>(kj + r), y = *reinterpret_cast<const float4*>(ej + r);
        o[0] = fmaf(a.x, x.x, fmaf(a.y, x.y, fmaf(a.z, x.z, fmaf(a.w, x.w, o[0]))));
        o[1] = fmaf(a.x, y.x, fmaf(a.y, y.y, fmaf(a.z, y.z, fmaf(a.w, y.w, o[1]))));
        o[2] = fmaf(b.x, x.x, fmaf(b.y, x.y, fmaf(b.z, x.z, fmaf(b.w, x.w, o[2]))));
        o[3] = fmaf(b.x, y.x, fmaf(b.y, y.y, fmaf(b.z, y.z, fmaf(b.w, y.w, o[3]))));
      }
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) mats[x * HY_CT * HY_CT + tid] = o[x];
    if (tid < HY_CT) {
      const bool have = tid < nt;
      scal[tid] = have ? in.beta[(row0 + tid) * H + h] : 0.f;            // r.(a*u)
      scal[HY_CT + tid] = have ? in.decay[(row0 + tid) * H + h] : 0.f;   // r.k
#pragma unroll
      for (int x = 2; x < 6; ++x) scal[x * HY_CT + tid] = 0.f;
    }
  }
}

// v[16 tokens][2 columns], a part of every sum in each of sixteen lanes -> lane i: token i's two sums
__device__ __forceinline__ void hy_chunk_reduce(float (&v)[HY_CT][2], int sub) {
#pragma unroll
  for (int off = 8; off >= 1; off >>= 1) {
    const bool up = (sub & off) != 0;
#pragma unroll
    for (int t = 0; t < off; ++t)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float lo = v[t][c], hi = v[t + off][c];
        v[t][c] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, off);
      }
  }
}

// grid (n_seqs, H, ceil(dv / 16)), 128 threads (16 value columns); dynamic shared memory 2 * (block + 16 x 18 values) floats
template <int NCH, int MODE>
__global__ void __launch_bounds__(128, 1) hy_chunk_kernel(RecurIn in, const float* __restrict__ ws, float* __restrict__ state, long long state_stride,
                                                       float* __restrict__ o, long long ldo, BatchMeta m, ChunkPart part, int H, int dk, int dv) {
  pdl_wait();   // no early trigger, as in hy_recur_kernel
  extern __shared__ __align__(16) float cks[];
  constexpr int DKP = 64 * NCH, BLK = hy_chunk_block(MODE, DKP), NB = BLK + HY_CT * HY_CHUNK_VP, RP = HY_CT * DKP;
  const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, sub = lane & 15;
  const int j0 = blockIdx.z * 16, jl = warp * 4 + (lane >> 4) * 2, col = j0 + jl;   // this lane's columns col, col + 1
  const SeqSpan sp = seq_span(m, s);
  // this launch's chunks [c0, c1); chunk c at entry e0 + c
  const int all = (sp.len + HY_CT - 1) / HY_CT, c0 = part.c0, c1 = part.per > 0 && c0 + part.per < all ? c0 + part.per : all;
  const int e0 = part.per > 0 ? s * part.per - c0 : sp.start / HY_CT + s;
  if (c0 >= c1) return;
  const float* cv = in.c + in.voff + (long long)h * dv + j0;
  const int ncv = dv - j0 < 16 ? dv - j0 : 16;
  auto stage = [&](int c, float* buf) {
    const float* src = ws + ((long long)(e0 + c) * H + h) * BLK;
    for (int i = tid; i < BLK / 4; i += 128) hy_cp16(buf + 4 * i, src + 4 * i);
    for (int i = tid; i < HY_CT * 16; i += 128) {
      const int t = c * HY_CT + (i >> 4), x = i & 15;
      if (t < sp.len && x < ncv) hy_cp4(buf + BLK + (i >> 4) * HY_CHUNK_VP + x, cv + (sp.start + t) * in.ldc + x);
      else buf[BLK + (i >> 4) * HY_CHUNK_VP + x] = 0.f;
    }
    hy_cp_commit();
  };
  hy_f2 S[2][2 * NCH];
  float* st[2];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const bool live = col + c < dv, have = live && (sp.pos0 > 0 || c0 > 0);   // the part before left its state there
    st[c] = state + (long long)sp.slot * state_stride + ((long long)h * dv + (live ? col + c : 0)) * dk;
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const int r = (ch * 16 + sub) * 4;
      float x[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) x[e] = have && r + e < dk ? st[c][r + e] : 0.f;
      S[c][2 * ch] = hy_f2_pack(x[0], x[1]);
      S[c][2 * ch + 1] = hy_f2_pack(x[2], x[3]);
    }
  }
  auto row4 = [&](const float* p, int ch, hy_f2& a, hy_f2& b) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + (ch * 16 + sub) * 4);
    a = v.x;
    b = v.y;
  };
  // dot products of sixteen row vectors with the two columns; lane i is left with token i's
  auto dots = [&](const float* rows, float (&out)[2]) {
    float v[HY_CT][2];
#pragma unroll
    for (int t = 0; t < HY_CT; ++t) {
      hy_f2 acc[2] = {0ull, 0ull};
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        hy_f2 a, b;
        row4(rows + t * DKP, ch, a, b);
#pragma unroll
        for (int c = 0; c < 2; ++c) acc[c] = hy_f2_fma(b, S[c][2 * ch + 1], hy_f2_fma(a, S[c][2 * ch], acc[c]));
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float2 f = hy_f2_unpack(acc[c]);
        v[t][c] = f.x + f.y;
      }
    }
    hy_chunk_reduce(v, sub);
    out[0] = v[0][0];
    out[1] = v[0][1];
  };
  stage(c0, cks + (c0 & 1) * NB);
  for (int c = c0; c < c1; ++c) {
    const float* buf = cks + (c & 1) * NB;
    if (c + 1 < c1) { stage(c + 1, cks + ((c + 1) & 1) * NB); hy_cp_wait<1>(); }
    else hy_cp_wait<0>();
    __syncthreads();
    const float* mats = buf + hy_chunk_mats(MODE, DKP);
    const float* scal = buf + hy_chunk_scal(MODE, DKP);
    const float* V = buf + BLK + jl;
    float pa[2], pb[2], ov[2];
    dots(buf, pa);
    dots(buf + RP, pb);
    const float2 v2 = *reinterpret_cast<const float2*>(V + sub * HY_CHUNK_VP);
    const float v[2] = {v2.x, v2.y};
    float coef[HY_CT][2];          // what every token writes into the two columns (the same in all sixteen lanes)
    if (MODE == HY_REC_DELTA) {
      const float be = scal[sub], gd = scal[HY_CT + sub], qk = scal[2 * HY_CT + sub], before = scal[3 * HY_CT + sub];
      pa[0] *= before; pa[1] *= before; pb[0] *= before; pb[1] *= before;
      float u[2];
#pragma unroll
      for (int j = 0; j < HY_CT; ++j) {
        const float kk = mats[j * HY_CT + sub], qq = mats[HY_CT * HY_CT + j * HY_CT + sub], behind = scal[4 * HY_CT + j];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          u[x] = be * (v[x] - gd * pa[x]);   // final in lane j
          const float uj = __shfl_sync(0xffffffffu, u[x], j, 16);
          pa[x] = j < sub ? fmaf(kk, uj, pa[x]) : pa[x];
          pb[x] = j < sub ? fmaf(qq, uj, pb[x]) : pb[x];
          coef[j][x] = behind * uj;
        }
      }
#pragma unroll
      for (int x = 0; x < 2; ++x) ov[x] = fmaf(qk, be * (v[x] - gd * pa[x]), gd * pb[x]);
      const float all = scal[5 * HY_CT];
      const hy_f2 all2 = hy_f2_pack(all, all);
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int p = 0; p < 2 * NCH; ++p) S[x][p] = hy_f2_mul(all2, S[x][p]);
#pragma unroll
      for (int j = 0; j < HY_CT; ++j)
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
          hy_f2 a, b;
          row4(buf + j * DKP, ch, a, b);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const hy_f2 w = hy_f2_pack(coef[j][x], coef[j][x]);
            S[x][2 * ch] = hy_f2_fma(a, w, S[x][2 * ch]);
            S[x][2 * ch + 1] = hy_f2_fma(b, w, S[x][2 * ch + 1]);
          }
        }
    } else {
      constexpr int M = HY_CT * HY_CT;
#pragma unroll
      for (int j = 0; j < HY_CT; ++j) {
        const float2 vj = *reinterpret_cast<const float2*>(V + j * HY_CHUNK_VP);
        const float uk = mats[j * HY_CT + sub], qk = mats[2 * M + j * HY_CT + sub];
        pa[0] = j < sub ? fmaf(uk, vj.x, pa[0]) : pa[0]; pa[1] = j < sub ? fmaf(uk, vj.y, pa[1]) : pa[1];
        pb[0] = j < sub ? fmaf(qk, vj.x, pb[0]) : pb[0]; pb[1] = j < sub ? fmaf(qk, vj.y, pb[1]) : pb[1];
      }
#pragma unroll
      for (int j = 0; j < HY_CT; ++j) {
        const float ue = mats[M + j * HY_CT + sub], qe = mats[3 * M + j * HY_CT + sub];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const float aj = __shfl_sync(0xffffffffu, pa[x], j, 16);   // final in lane j
          pa[x] = j < sub ? fmaf(-ue, aj, pa[x]) : pa[x];
          pb[x] = j < sub ? fmaf(-qe, aj, pb[x]) : pb[x];
          coef[j][x] = aj;
        }
      }
      const float ra = scal[sub], rk = scal[HY_CT + sub];
#pragma unroll
      for (int x = 0; x < 2; ++x) ov[x] = fmaf(rk, v[x], fmaf(-ra, pa[x], pb[x]));
#pragma unroll
      for (int j = 0; j < HY_CT; ++j) {
        const float2 vj = *reinterpret_cast<const float2*>(V + j * HY_CHUNK_VP);
        const hy_f2 kv[2] = {hy_f2_pack(vj.x, vj.x), hy_f2_pack(vj.y, vj.y)};
        const hy_f2 ea[2] = {hy_f2_pack(-coef[j][0], -coef[j][0]), hy_f2_pack(-coef[j][1], -coef[j][1])};
#pragma unroll
        for (int ch = 0; ch < NCH; ++ch) {
          hy_f2 ka, kb, a, b;
          row4(buf + 2 * RP + j * DKP, ch, ka, kb);
          row4(buf + 3 * RP + j * DKP, ch, a, b);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            S[x][2 * ch] = hy_f2_fma(a, ea[x], hy_f2_fma(ka, kv[x], S[x][2 * ch]));
            S[x][2 * ch + 1] = hy_f2_fma(b, ea[x], hy_f2_fma(kb, kv[x], S[x][2 * ch + 1]));
          }
        }
      }
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        hy_f2 a, b;
        row4(buf + 4 * RP, ch, a, b);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          S[x][2 * ch] = hy_f2_mul(a, S[x][2 * ch]);
          S[x][2 * ch + 1] = hy_f2_mul(b, S[x][2 * ch + 1]);
        }
      }
    }
    const int t = c * HY_CT + sub;
    if (t < sp.len) {
      float* dst = o + (long long)(sp.start + t) * ldo + (long long)h * dv + col;
      if (col < dv) dst[0] = ov[0];
      if (col + 1 < dv) dst[1] = ov[1];
    }
    __syncthreads();   // the buffer is refilled by the next iteration's copies
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    if (col + c >= dv) continue;
#pragma unroll
    for (int ch = 0; ch < NCH; ++ch) {
      const int r = (ch * 16 + sub) * 4;
      const float2 a = hy_f2_unpack(S[c][2 * ch]), b = hy_f2_unpack(S[c][2 * ch + 1]);
      const float x[4] = {a.x, a.y, b.x, b.y};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (r + e < dk) st[c][r + e] = x[e];
    }
  }
}
