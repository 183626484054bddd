"""Per-(token, head) attention of float32 prompts: the warps of a block are chosen by the step's longest context, and a row's sums must
not depend on that choice; nor do those of rows that go by tiles of queries."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(kind):
  from xotorch_support_jetson_b200 import synth
  if kind == "latent":
    hf = {"architecture": "Bibevik", "width": 64, "vocab": 97, "embedding": {"scale": 8.0}, "norm": {"eps": 1e-6}, "layers": [
      {"type": "latent_attention", "mixer": {"heads": 2, "dim": 24, "rot_dim": 16, "vdim": 40, "kv_rank": 48, "scale": 40 ** -0.5,
                                             "rot": {"base": 10000.0, "dims": 16}}, "mlp": {"kind": "dense", "ff": 64, "limit": 2.0}}]}
    return hf, synth.random_bibevik_state(hf, seed=2)
  hf = {"architecture": "Refatar", "width": 64, "vocab": 97, "norm": {"eps": 1e-5}, "layers": [
    {"type": "parallel", "mixer": {"left": {"heads": 4, "kv_heads": 2, "dim": 32, "vdim": 48, "scale": 32 ** -0.5, "mask": {"size": 900, "keep_first": 3}},
                                   "right": {"heads": 2, "dim": 32, "vdim": 64}, "left_scale": 1.0, "right_scale": 1.0}, "mlp": None}]}
  return hf, synth.random_refatar_state(hf, seed=2)


def _stage(kind, rows):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf, state = _model(kind)
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  st = StageRuntime(Shard("warps-test", 0, 0, 1), cfg, max_batch_tokens=rows, max_seqs=3, max_tokens_per_seq=512, dtype="float32")
  st.load_state(state)
  return st


@pytest.mark.parametrize("route", ["0", "64"])   # never by tiles; by tiles from 64 rows on
@pytest.mark.parametrize("kind", ["latent", "window"])
@pytest.mark.parametrize("mine,other", [(100, 300), (150, 340), (70, 400)])   # 3 to 5 tiles of keys alone, 10 to 13 beside the other one
def test_a_prompt_beside_a_longer_one(built_lib, monkeypatch, kind, mine, other, route):
  monkeypatch.setenv("XB_HY_ATTN_TILE", route)
  st = _stage(kind, mine + other)
  g = torch.Generator().manual_seed(mine + other)
  ids = [torch.randint(0, 97, (n,), generator=g).to("cuda", torch.int32) for n in (mine, other)]
  alone, both = torch.empty((mine, 64), device="cuda"), torch.empty((mine + other, 64), device="cuda")
  st.forward([0], [mine], [0], tokens=ids[0], taps=[alone])
  st.forward([1, 2], [mine, other], [0, 0], tokens=torch.cat(ids), taps=[both])
  torch.cuda.synchronize()
  assert torch.isfinite(both).all()
  assert torch.equal(alone, both[:mine])
  st.close()


@pytest.mark.parametrize("kind", ["latent", "window"])
@pytest.mark.parametrize("ctx,mine,other", [(40, 60, 300), (100, 50, 340), (290, 63, 400)])
def test_a_few_rows_behind_a_context_beside_a_prompt(built_lib, kind, ctx, mine, other):
  """On the default route: rows that stay with the kernel of one block per (token, head), behind a context, alone and beside a prompt."""
  st = _stage(kind, mine + other)
  g = torch.Generator().manual_seed(ctx + other)
  ids = [torch.randint(0, 97, (n,), generator=g).to("cuda", torch.int32) for n in (ctx + mine, other)]
  alone, both = torch.empty((mine, 64), device="cuda"), torch.empty((mine + other, 64), device="cuda")
  for slot in (0, 1):
    for a in range(0, ctx, 32):
      b = min(ctx, a + 32)
      st.forward([slot], [b - a], [a], tokens=ids[0][a:b])
  st.forward([0], [mine], [ctx], tokens=ids[0][ctx:], taps=[alone])
  st.forward([1, 2], [mine, other], [ctx, 0], tokens=torch.cat([ids[0][ctx:], ids[1]]), taps=[both])
  torch.cuda.synchronize()
  assert torch.isfinite(both).all()
  assert torch.equal(alone, both[:mine])
  st.close()
