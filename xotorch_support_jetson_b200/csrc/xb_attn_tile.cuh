// Softmax attention of float32 prompts by tiles of queries.  Included by xb_hybrid_kernels.cuh, ahead of the other kernel.
//
// hy_attn_window_kernel gives every (token, query head) a block that reads all of its keys and values: 300 tokens x 32 heads of 64 pull 0.7 GB
// through L2 and are bound by that (268 us).  Here a block takes 32 query rows of one key head -- 32 / R consecutive tokens of a sequence x
// its R query heads -- against 32 keys at a time from shared memory, so that a key row is read once for 32 queries.  All sums are fp32 FMA:
// what bounds it is their issue and the shared-memory reads that feed them.  Half a warp owns two query rows from scores to output.
// That layer 268 -> 49 us with the caches flushed, two float32 layers on a prompt of 300 rows 1196 -> 959 in all.
//
// Key tiles start at multiples of 32 positions whatever the queries, and keys that a query does not see change none of its sums, whatever they hold: a
// query's result depends on its own position and context alone.  Which sequences go by tiles: hy_at_takes.
#pragma once

#define HY_AT_ROWS 32
#define HY_AT_KEYS 32
#define HY_AT_MIN_LEN 64

// Whether the rows of a sequence (len new ones behind ctx) go by tiles.  A tile walks all keys of its rows by itself, so a sequence takes about as long as
// its last tile however few it has; the other kernel has a block for every (token, head) and takes as long as there is work.  Both grow with the context,
// so the line lies at a number of tiles, each counted by the share of the last one's keys that an average one sees: a half without a context, all of them
// behind a long one.  Tiles against (token, head), us of the kernel: latents of 320 / 256 channels, 16 heads, 64 rows without a context (32 tiles that count
// 16) 38 against 23, 96 rows (24) 45 against 48, 64 rows behind 256 (29) 97 against 154, behind 4096 985 against 1573; 4 heads behind 4096, 128 rows (16)
// 999 against 905, 192 rows (24) 1013 against 1357; 32 heads over 8, 64 rows (32) 16 against 24.  Below 64 rows it was not measured, those stay.
// The choice hangs on the sequence and the layer alone.  from > 1: from so many rows on, whatever the tiles.
__host__ __device__ __forceinline__ bool hy_at_takes(int len, int ctx, int H, int G, int window, int from) {
  if (from > 1) return len >= from;
  const int tq = HY_AT_ROWS / (H / G), seen = ctx < window ? ctx : window;
  const long long tiles = (long long)((len + tq - 1) / tq) * G;
  return len >= HY_AT_MIN_LEN && tiles * (2LL * seen + len) > 32LL * (seen + len);
}

__device__ __forceinline__ void hy_at_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

struct AttnTile {
  int H, G, dk, dv;          // query heads, key heads, key and value channels (rows of the pools: dk / dv floats)
  int v_in_k;                // 1: a value is the head of its key row (v_pool unused)
  int window, keep_first;
  float scale, out_scale;
  int tiles;                 // blocks of a sequence: grid (sequences x tiles, G)
  int from;                  // see hy_at_takes
};
// queries + two stages of keys (and values) + weights; 64 floats behind the last row, which wide value reads may touch
static size_t hy_at_smem(const AttnTile& a, int nv) {
  return ((size_t)HY_AT_ROWS * (a.dk + 4) + 2 * HY_AT_KEYS * ((size_t)a.dk + 4 + (a.v_in_k ? 0 : 64 * nv)) + HY_AT_ROWS * (HY_AT_KEYS + 4) + 64) * sizeof(float);
}

// NV: 64-channel groups of a value row (dv <= 64 NV).  sigmoid(gate column) and out_scale as in hy_attn_window_kernel.
template <int NV, typename AT>
__global__ void __launch_bounds__(256) hy_attn_tile_kernel(LinOut P, int off_q, int off_gate, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                                                           BatchMeta m, AttnTile a, AT* __restrict__ out, long long ld_out) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ __align__(16) float at_smem[];
  const int R = a.H / a.G, TQ = HY_AT_ROWS / R, dk = a.dk, dv = a.dv, KP = dk + 4, VP = a.v_in_k ? KP : 64 * NV;
  const int s = blockIdx.x / a.tiles, i0 = (blockIdx.x - s * a.tiles) * TQ, g = blockIdx.y;
  const int first = s > 0 ? m.seq_last[s - 1] + 1 : 0, len = m.seq_last[s] + 1 - first;
  if (i0 >= len) return;
  const int ctx = m.tok_pos[first];
  if (!hy_at_takes(len, ctx, a.H, a.G, a.window, a.from)) return;
  const int n_tok = min(TQ, len - i0), pos0 = ctx + i0, pos_last = pos0 + n_tok - 1;
  const int* pages = m.page_table + (long long)m.seq_slot[s] * m.max_pages;
  float* sQ = at_smem;
  float* sK = sQ + HY_AT_ROWS * KP;
  float* sV = sK + 2 * HY_AT_KEYS * KP;
  float* sP = sV + (a.v_in_k ? 0 : 2 * HY_AT_KEYS * VP);
  const int tid = threadIdx.x, hw = tid >> 4, l16 = tid & 15;
  for (int i = tid; i < HY_AT_ROWS * dk; i += 256) {
    const int r = i / dk, d = i - r * dk, t = r / R;
    sQ[r * KP + d] = t < n_tok && r < TQ * R ? lin_at(P, first + i0 + t, off_q + (g * R + r - t * R) * dk + d) * a.scale : 0.f;
  }
  // the two rows of this half-warp: position (-1: no such row), newest first key of the window
  int pos[2], row[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = hw * 2 + u, t = r / R;
    row[u] = t < n_tok && r < TQ * R ? t : -1;
    pos[u] = row[u] >= 0 ? pos0 + t : -1;
  }
  auto fetch = [&](int kt, int stage) {   // eight threads a key; keys behind the last query are not read
    const int j = tid >> 3, key = kt * HY_AT_KEYS + j;
    float* kd = sK + (stage * HY_AT_KEYS + j) * KP;
    float* vd = sV + (stage * HY_AT_KEYS + j) * VP;
    if (key <= pos_last) {
      const long long kr = ((long long)pages[key / m.page_tokens] * a.G + g) * m.page_tokens + key % m.page_tokens;
      for (int c = (tid & 7) * 4; c < dk; c += 32) hy_at_copy16(kd + c, k_pool + kr * dk + c);
      if (!a.v_in_k)
        for (int c = (tid & 7) * 4; c < dv; c += 32) hy_at_copy16(vd + c, v_pool + kr * dv + c);
    } else {   // zero rows: their weights are 0
      for (int c = (tid & 7) * 4; c < dk; c += 32) *reinterpret_cast<float4*>(kd + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!a.v_in_k)
        for (int c = (tid & 7) * 4; c < dv; c += 32) *reinterpret_cast<float4*>(vd + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int last = pos_last / HY_AT_KEYS, lo = max(0, pos0 - a.window + 1);   // lo: oldest key of the tile's windows
  auto next = [&](int kt) {   // the next tile that some query sees: kept first keys, then the windows
    ++kt;
    return kt * HY_AT_KEYS >= a.keep_first && kt < lo / HY_AT_KEYS ? lo / HY_AT_KEYS : kt;
  };
  float mx[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float4 acc[2][NV];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[u][v] = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* q0 = sQ + hw * 2 * KP;
  // oldest and newest position of the warp's rows: tiles that all of them see whole need no mask
  const int first_pos = __reduce_min_sync(0xffffffffu, min(row[0] < 0 ? 0x7fffffff : pos[0], row[1] < 0 ? 0x7fffffff : pos[1]));
  const int last_pos = __reduce_max_sync(0xffffffffu, max(pos[0], pos[1]));
  int kt = next(-1), stage = 0;
  fetch(kt, 0);
  while (kt <= last) {
    const int kn = next(kt);
    if (kn <= last) fetch(kn, stage ^ 1);
    else asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    // ---- scores of two rows against keys l16 and l16 + 16
    const float* k0 = sK + (stage * HY_AT_KEYS + l16) * KP;
    float sc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 4
    for (int c = 0; c < dk; c += 4) {
      const float4 qa = *reinterpret_cast<const float4*>(q0 + c), qb = *reinterpret_cast<const float4*>(q0 + KP + c);
      const float4 ka = *reinterpret_cast<const float4*>(k0 + c), kb = *reinterpret_cast<const float4*>(k0 + 16 * KP + c);
      sc[0][0] = fmaf(qa.x, ka.x, sc[0][0]); sc[0][0] = fmaf(qa.y, ka.y, sc[0][0]); sc[0][0] = fmaf(qa.z, ka.z, sc[0][0]); sc[0][0] = fmaf(qa.w, ka.w, sc[0][0]);
      sc[0][1] = fmaf(qa.x, kb.x, sc[0][1]); sc[0][1] = fmaf(qa.y, kb.y, sc[0][1]); sc[0][1] = fmaf(qa.z, kb.z, sc[0][1]); sc[0][1] = fmaf(qa.w, kb.w, sc[0][1]);
      sc[1][0] = fmaf(qb.x, ka.x, sc[1][0]); sc[1][0] = fmaf(qb.y, ka.y, sc[1][0]); sc[1][0] = fmaf(qb.z, ka.z, sc[1][0]); sc[1][0] = fmaf(qb.w, ka.w, sc[1][0]);
      sc[1][1] = fmaf(qb.x, kb.x, sc[1][1]); sc[1][1] = fmaf(qb.y, kb.y, sc[1][1]); sc[1][1] = fmaf(qb.z, kb.z, sc[1][1]); sc[1][1] = fmaf(qb.w, kb.w, sc[1][1]);
    }
    const int k_lo = kt * HY_AT_KEYS, k_hi = k_lo + HY_AT_KEYS - 1;
    const bool whole = k_hi <= first_pos && (last_pos - k_lo < a.window || k_hi < a.keep_first);
    uint32_t seen[2] = {0u, 0u};   // else: the keys of the tile that a row sees
    if (!whole) {
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int j = k_lo + l16 + 16 * h;
          const bool sees = j <= pos[u] && (pos[u] - j < a.window || j < a.keep_first);
          if (!sees) sc[u][h] = -INFINITY;
          seen[u] |= ((__ballot_sync(0xffffffffu, sees) >> (threadIdx.x & 16)) & 0xffffu) << (16 * h);
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float t = fmaxf(sc[u][0], sc[u][1]);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, o));
      const float nm = fmaxf(mx[u], t), ref = nm == -INFINITY ? 0.f : nm;   // (no key seen yet: every weight below is 0)
      const float corr = expf(mx[u] - ref), p0 = expf(sc[u][0] - ref), p1 = expf(sc[u][1] - ref);
      mx[u] = nm;
      l[u] = l[u] * corr + (p0 + p1);
      float* sp = sP + (hw * 2 + u) * (HY_AT_KEYS + 4) + l16;
      sp[0] = p0;
      sp[16] = p1;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        acc[u][v].x *= corr; acc[u][v].y *= corr; acc[u][v].z *= corr; acc[u][v].w *= corr;
      }
    }
    __syncwarp();   // a row's weights are its half-warp's own
    // ---- weighted values: channels 4 l16 .. of each group of 64.  In a tile that some row does not see whole, the values of its masked keys enter as 0:
    // their weights are 0, but 0 x inf and 0 x NaN are not
    const float* vs = (a.v_in_k ? sK : sV) + stage * HY_AT_KEYS * VP + l16 * 4;
    const float* pr = sP + hw * 2 * (HY_AT_KEYS + 4);
    auto add_values = [&](auto mask) {
      constexpr bool MASK = decltype(mask)::value;
      const int n = MASK ? min(HY_AT_KEYS, last_pos + 1 - k_lo) : HY_AT_KEYS;
#pragma unroll(MASK ? 1 : 2)
      for (int j = 0; j < n; j += 4) {
        const float4 pa = *reinterpret_cast<const float4*>(pr + j), pb = *reinterpret_cast<const float4*>(pr + HY_AT_KEYS + 4 + j);
        const float pja[4] = {pa.x, pa.y, pa.z, pa.w}, pjb[4] = {pb.x, pb.y, pb.z, pb.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool sa = !MASK || (seen[0] >> (j + i) & 1), sb = !MASK || (seen[1] >> (j + i) & 1);
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            const float4 x = *reinterpret_cast<const float4*>(vs + (j + i) * VP + v * 64);
            const float4 xa = sa ? x : make_float4(0.f, 0.f, 0.f, 0.f), xb = sb ? x : make_float4(0.f, 0.f, 0.f, 0.f);
            acc[0][v].x = fmaf(pja[i], xa.x, acc[0][v].x); acc[0][v].y = fmaf(pja[i], xa.y, acc[0][v].y);
            acc[0][v].z = fmaf(pja[i], xa.z, acc[0][v].z); acc[0][v].w = fmaf(pja[i], xa.w, acc[0][v].w);
            acc[1][v].x = fmaf(pjb[i], xb.x, acc[1][v].x); acc[1][v].y = fmaf(pjb[i], xb.y, acc[1][v].y);
            acc[1][v].z = fmaf(pjb[i], xb.z, acc[1][v].z); acc[1][v].w = fmaf(pjb[i], xb.w, acc[1][v].w);
          }
        }
      }
    };
    if (whole) add_values(std::false_type());
    else add_values(std::true_type());
    __syncthreads();   // the stage may be filled again
    kt = kn;
    stage ^= 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    float L = l[u];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) L += __shfl_xor_sync(0xffffffffu, L, o);
    if (row[u] < 0) continue;
    const long long t = first + i0 + row[u];
    const int h = g * R + hw * 2 + u - row[u] * R;
    const float inv = a.out_scale / L;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const float x[4] = {acc[u][v].x, acc[u][v].y, acc[u][v].z, acc[u][v].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int d = v * 64 + l16 * 4 + i;
        if (d >= dv) break;
        float y = x[i] * inv;
        if (off_gate >= 0) y *= hy_sigmoid(lin_at(P, t, off_gate + h * dv + d));
        act_store<AT>(out + t * ld_out + (long long)h * dv + d, y);
      }
    }
  }
}
