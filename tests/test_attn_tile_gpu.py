"""Attention of float32 prompts by tiles of queries (hy_attn_tile_kernel) against the kernel of one block per (token, head): window with kept
first keys and gate, and the latent form whose values are the heads of its key rows; query tiles and key tiles (32 positions) that end
inside a sequence, sequences on both sides of the least length it takes, portions behind a context; and the rule that chooses between the two."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(kind, heads, kv_heads, dim, vdim):
  from xotorch_support_jetson_b200 import synth
  if kind == "latent":
    hf = {"architecture": "Bibevik", "width": 64, "vocab": 97, "embedding": {"scale": 8.0}, "norm": {"eps": 1e-6}, "layers": [
      {"type": "latent_attention", "mixer": {"heads": heads, "dim": 24, "rot_dim": 16, "vdim": 40, "kv_rank": vdim, "scale": 40 ** -0.5,
                                             "rot": {"base": 10000.0, "dims": 16}}, "mlp": {"kind": "dense", "ff": 64, "limit": 2.0}}]}
    return hf, synth.random_bibevik_state(hf, seed=2)
  hf = {"architecture": "Refatar", "width": 64, "vocab": 97, "norm": {"eps": 1e-5}, "layers": [
    {"type": "parallel", "mixer": {"left": {"heads": heads, "kv_heads": kv_heads, "dim": dim, "vdim": vdim, "scale": dim ** -0.5, "mask": {"size": 70, "keep_first": 3}},
                                   "right": {"heads": 2, "dim": 32, "vdim": 64}, "left_scale": 1.0, "right_scale": 1.0}, "mlp": None}]}
  return hf, synth.random_refatar_state(hf, seed=2)


# (context, rows) of each sequence: 63 / 64 rows about the least length, one row into a tile, a window that leaves tiles out
STEPS = [[(0, 64)], [(0, 63), (0, 65), (0, 97)], [(0, 200), (0, 5)], [(130, 64), (0, 161)]]


@pytest.mark.parametrize("kind,heads,kv_heads,dim,vdim", [("window", 4, 2, 32, 48), ("window", 6, 2, 64, 64), ("window", 32, 1, 20, 132), ("window", 3, 3, 128, 200),
                                                         ("latent", 2, 1, 0, 48), ("latent", 16, 1, 0, 256)])
def test_tiles_of_queries_match_single_queries(built_lib, monkeypatch, kind, heads, kv_heads, dim, vdim):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf, state = _model(kind, heads, kv_heads, dim, vdim)
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  g = torch.Generator().manual_seed(heads + vdim)
  ids = torch.randint(0, 97, (2048,), generator=g).to("cuda", torch.int32)
  rows = {}
  for tile in ("64", "0"):   # by tiles from 64 rows on; never
    monkeypatch.setenv("XB_HY_ATTN_TILE", tile)
    st = StageRuntime(Shard("tile-test", 0, 0, 1), cfg, max_batch_tokens=256, max_seqs=3, max_tokens_per_seq=320, page_tokens=16, dtype="float32")
    st.load_state(state)
    rows[tile] = []
    for step in STEPS:
      for i, (c, _) in enumerate(step):
        st.release_slot(i)
        if c:
          st.forward([i], [c], [0], tokens=ids[:c])
      n = [q for _, q in step]
      out = torch.empty((sum(n), 64), device="cuda")
      st.forward(list(range(len(step))), n, [c for c, _ in step], tokens=ids[300:300 + sum(n)], taps=[out])
      torch.cuda.synchronize()
      rows[tile].append(out)
    st.close()
  for a, b in zip(rows["64"], rows["0"]):
    assert not torch.equal(a, b)   # two kernels
    # the same sums in another order: fp32 roundings of at most 200 terms on either side, through one layer
    assert torch.isfinite(a).all()
    assert (a - b).abs().max() <= 2e-5 * b.abs().max()


def _takes(n, ctx, heads, kv_heads, window):
  """Whether n rows behind ctx go by tiles of 32 / (heads / kv_heads) tokens: 64 rows and more of a sequence whose tiles number above 16, each counted by the
  share of the last one's keys that an average one sees."""
  tq, seen = 32 // (heads // kv_heads), min(ctx, window)
  return n >= 64 and -(-n // tq) * kv_heads * (2 * seen + n) > 32 * (seen + n)


# rows on both sides of the line, alone, behind a context and beside sequences that go the other way
@pytest.mark.parametrize("kind,heads,kv_heads,dim,vdim,step", [
  ("window", 32, 8, 32, 48, [(0, 63), (0, 64)]), ("window", 8, 8, 32, 48, [(0, 128), (0, 129), (200, 64), (200, 96)]),
  ("window", 4, 2, 32, 48, [(0, 256), (0, 257), (300, 161)]), ("latent", 16, 1, 0, 48, [(0, 64), (0, 65), (33, 63), (33, 64)]),
  ("latent", 2, 1, 0, 48, [(300, 336), (300, 352), (0, 64)])])
def test_which_rows_go_by_tiles(built_lib, monkeypatch, kind, heads, kv_heads, dim, vdim, step):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf, state = _model(kind, heads, kv_heads, dim, vdim)
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  g = torch.Generator().manual_seed(heads)
  ids = [torch.randint(0, 97, (c + n,), generator=g).to("cuda", torch.int32) for c, n in step]
  rows = {}
  for tile in ("64", "1", "0"):
    monkeypatch.setenv("XB_HY_ATTN_TILE", tile)
    st = StageRuntime(Shard("rule-test", 0, 0, 1), cfg, max_batch_tokens=1024, max_seqs=8, max_tokens_per_seq=768, page_tokens=16, dtype="float32")
    st.load_state(state)
    for i, (c, _) in enumerate(step):
      for slot in (i, 4 + i):
        for a in range(0, c, 16):   # the context by the same kernel on every route
          st.forward([slot], [min(c, a + 16) - a], [a], tokens=ids[i][a:min(c, a + 16)])
    out = torch.empty((sum(n for _, n in step), 64), device="cuda")
    st.forward(list(range(len(step))), [n for _, n in step], [c for c, _ in step], tokens=torch.cat([t[c:] for t, (c, _) in zip(ids, step)]), taps=[out])
    alone = []
    for i, (c, n) in enumerate(step):
      one = torch.empty((n, 64), device="cuda")
      st.forward([4 + i], [n], [c], tokens=ids[i][c:], taps=[one])
      alone.append(one)
    torch.cuda.synchronize()
    rows[tile] = list(out.split([n for _, n in step])), alone
    st.close()
  took = [_takes(n, c, heads, kv_heads, 70 if kind == "window" else 1 << 30) for c, n in step]
  assert True in took and False in took
  for i, t in enumerate(took):
    for form in (0, 1):   # beside the others, alone
      assert torch.equal(rows["1"][form][i], rows["64" if t else "0"][form][i]), (step[i], t)
    if step[i][1] >= 64:
      assert not torch.equal(rows["64"][1][i], rows["0"][1][i])
