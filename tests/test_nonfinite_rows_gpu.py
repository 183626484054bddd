"""A token whose row is not finite spoils the queries that see it and no others: earlier tokens of its prompt, later ones that its window has left
behind, and other sequences answer as if it were an ordinary one.  Attention of hybrid models by tiles of queries (hy_attn_tile_kernel) and by
(token, head) (hy_attn_window_kernel)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BAD = 96   # the vocabulary's last id: its embedding row is not finite


def _window(keep_first, size, heads=4, kv_heads=2):
  from xotorch_support_jetson_b200 import synth
  hf = {"architecture": "Refatar", "width": 64, "vocab": 97, "norm": {"eps": 1e-5}, "layers": [
    {"type": "parallel", "mixer": {"left": {"heads": heads, "kv_heads": kv_heads, "dim": 32, "vdim": 48, "scale": 32 ** -0.5, "mask": {"size": size, "keep_first": keep_first}},
                                   "right": {"heads": 2, "dim": 32, "vdim": 64}, "left_scale": 1.0, "right_scale": 1.0}, "mlp": None}]}
  return hf, synth.random_refatar_state(hf, seed=2)


def _latent(heads=8, window=25):
  from xotorch_support_jetson_b200 import synth
  hf = {"architecture": "Rurutar", "width": 64, "vocab": 97, "embedding": {"scale": 0.6}, "norm": {"eps": 1e-5}, "logit_softcap": 9.0, "layers": [
    {"type": "latent_attention", "mlp": None, "mixer": {"heads": heads, "dim": 12, "rot_dim": 8, "vdim": 20, "kv_rank": 24, "q_rank": 40, "scale": 20 ** -0.5,
                                                        "mask": {"size": window}, "rot": {"base": 500.0, "dims": 8}}}]}
  return hf, synth.random_rurutar_state(hf, seed=2)


def _stage(hf, state, dtype="float32"):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  state = dict(state)
  state["embed"] = state["embed"].clone()
  state["embed"][BAD] = float("nan") if hf["architecture"] == "Rurutar" else float("inf")   # (a tanh norm makes an infinity finite)
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  st = StageRuntime(Shard("nonfinite-test", 0, 0, 1), cfg, max_batch_tokens=256, max_seqs=3, max_tokens_per_seq=320, page_tokens=16, dtype=dtype)
  st.load_state(state)
  return st


def _ids(n, seed, bad=()):
  t = torch.randint(0, BAD, (n,), generator=torch.Generator().manual_seed(seed))
  t[list(bad)] = BAD
  return t.to("cuda", torch.int32)


def _rows(st, slot, ids, pos=0):
  out = torch.empty((ids.numel(), 64), device="cuda")
  st.forward([slot], [ids.numel()], [pos], tokens=ids, taps=[out])
  torch.cuda.synchronize()
  return out


# 150 rows; the bad token late (earlier rows of its query and key tile), and early (rows whose window has left it, beside kept first keys or not)
@pytest.mark.parametrize("bad", [149, 100, 2])
@pytest.mark.parametrize("model", ["window", "window_one_head", "latent"])
def test_only_the_queries_that_see_it(built_lib, monkeypatch, model, bad):
  hf, state = {"window": lambda: _window(3, 70), "window_one_head": lambda: _window(0, 40, 2, 2), "latent": _latent}[model]()
  rows = {}
  for tile in ("64", "0"):
    monkeypatch.setenv("XB_HY_ATTN_TILE", tile)
    st = _stage(hf, state)
    rows[tile] = _rows(st, 0, _ids(150, 7, [bad]))
    rows[tile, "plain"] = _rows(st, 1, _ids(150, 7))
    st.close()
  a, b = rows["64"], rows["0"]
  assert not torch.equal(rows["64", "plain"], rows["0", "plain"])   # two kernels
  fine = torch.isfinite(b).all(1)
  assert fine[:bad].all() and not fine[bad]
  if model == "latent":
    assert fine[bad + 25:].all()   # (the other model's recurrence carries it on)
  assert torch.equal(torch.isfinite(a).all(1), fine)
  assert (a - b)[fine].abs().max() <= 2e-5 * b[fine].abs().max()
  # rows before it: the same bits as without it
  assert torch.equal(a[:bad], rows["64", "plain"][:bad])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("model", ["window", "latent"])
def test_another_sequence_in_the_first_row_of_the_pool(built_lib, monkeypatch, model, dtype):
  """37 keys end inside a round of four: what fills the round up must not be the pool's first row, another sequence's."""
  monkeypatch.setenv("XB_HY_TC_ATTN", "0")
  monkeypatch.setenv("XB_HY_LAT_MMA", "0")
  hf, state = {"window": lambda: _window(3, 70), "latent": _latent}[model]()
  got = []
  for bad in ([], [0]):
    st = _stage(hf, state, dtype)
    _rows(st, 0, _ids(5, 1, bad))   # pages are handed out from the first on
    ids = _ids(38, 2)
    got.append(torch.cat([_rows(st, 1, ids[:37]), _rows(st, 1, ids[37:], 37)]))
    st.close()
  assert torch.isfinite(got[0]).all()
  assert torch.equal(got[0], got[1])
