"""A prompt's numbers do not depend on what else its step carries: above 128 rows every Linear sums in one order, so a prompt in
portions, or beside other prompts, gives the bits of the prompt alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stage(kind, max_rows, sizes=None):
  from oracle import torch_oracle as O
  from xotorch_support_jetson_b200 import models
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  from xotorch_support_jetson_b200.synth import random_hf_state
  # long enough sums (1024 and 2816) and few enough tiles that splitting K over blocks would look worthwhile at 129 to 512 rows
  if sizes is not None:   # (heads, kv heads, head dim, feed-forward)
    H, KV, hd, ff = sizes
    mid, hf = ("llama-3.2-tiny", dict(models.model_cards["llama-3.2-tiny"]["hf_config"], hidden_size=640, num_attention_heads=H, num_key_value_heads=KV,
                                      head_dim=hd, intermediate_size=ff, num_hidden_layers=2)) if kind == "interleaved" else \
              ("qwen-2.5-odd", models._qwen(640, H, KV, ff, 2, vocab=1536, max_pos=4096))
  elif kind == "interleaved":
    mid, hf = "llama-3.2-tiny", dict(models.model_cards["llama-3.2-tiny"]["hf_config"], hidden_size=1024, num_attention_heads=16, num_key_value_heads=4,
                                     head_dim=64, intermediate_size=2816, num_hidden_layers=2)
  else:
    mid, hf = "qwen-2.5-hd128", models._qwen(1024, 8, 2, 2816, 2, vocab=1536, max_pos=4096)
  cfg = O.model_config_from_hf(hf)
  st = StageRuntime(Shard(mid, 0, 1, 2), cfg, device=0, max_batch_tokens=max_rows, max_seqs=4, max_tokens_per_seq=2048)
  st.load_state(random_hf_state(hf, seed=11, std=0.05, norm_jitter=0.1))
  return st, cfg


def _rows(st, cfg, slots, lens, starts, tokens):
  """Hidden rows behind the first layer and behind the last one."""
  taps = [torch.empty((sum(lens), cfg["embed_dim"]), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
  st.forward(slots, lens, starts, tokens=tokens, taps=taps)
  return torch.stack(taps, 1)


@pytest.mark.parametrize("kind", ["interleaved", "half-split"])
@pytest.mark.parametrize("portions", [[129, 271, 384, 512, 104 + 129], [512, 513, 129], [300, 700, 256]])
def test_portions_have_the_bits_of_the_whole(built_lib, kind, portions):
  n = sum(portions)
  st, cfg = _stage(kind, n)
  ids = torch.randint(1, cfg["vocab_size"], (n,), generator=torch.Generator().manual_seed(n)).to("cuda", torch.int32)
  whole = _rows(st, cfg, [0], [n], [0], ids)
  parts, a = [], 0
  for p in portions:
    parts.append(_rows(st, cfg, [1], [p], [a], ids[a:a + p].contiguous()))
    a += p
  torch.cuda.synchronize()
  assert torch.isfinite(whole.float()).all()
  assert torch.equal(whole, torch.cat(parts))
  st.close()


@pytest.mark.parametrize("kind", ["interleaved", "half-split"])
@pytest.mark.parametrize("lens", [[300, 260], [129, 5, 500], [200, 180, 1]])
def test_neighbours_do_not_change_a_prompt(built_lib, kind, lens):
  st, cfg = _stage(kind, sum(lens))
  g = torch.Generator().manual_seed(sum(lens))
  ids = [torch.randint(1, cfg["vocab_size"], (n,), generator=g).to("cuda", torch.int32) for n in lens]
  together = _rows(st, cfg, list(range(len(lens))), lens, [0] * len(lens), torch.cat(ids)).split(lens)
  for i, n in enumerate(lens):
    if n > 128:   # (up to 128 rows take the decode Linear, which sums in an order of its own)
      assert torch.equal(together[i], _rows(st, cfg, [3], [n], [0], ids[i])), (i, n)
      st.release_slot(3)
  torch.cuda.synchronize()
  st.close()


@pytest.mark.parametrize("kind", ["interleaved", "half-split"])
@pytest.mark.parametrize("sizes", [(10, 2, 64, 992), (5, 1, 128, 1120)])   # 896 q/k/v, 640 o and down, 1984 or 2240 gate/up features: ends inside every tile
@pytest.mark.parametrize("n", [129, 257, 300])
def test_every_tile_has_the_same_bits(built_lib, monkeypatch, kind, sizes, n):
  """CTA pairs and tiles of 256, 192 and 128 features on tile-major weights, with the rotation, cache-append and SiLU epilogues: the whole
  forward and a token step that reads the cached keys and values."""
  outs = []
  for variant in range(1, 5):
    monkeypatch.setenv("XB_WIDE_VARIANT", str(variant))
    st, cfg = _stage(kind, n, sizes)
    ids = torch.randint(1, cfg["vocab_size"], (n + 1,), generator=torch.Generator().manual_seed(n)).to("cuda", torch.int32)
    rows = _rows(st, cfg, [0], [n], [0], ids[:n].contiguous())
    step = _rows(st, cfg, [0], [1], [n], ids[n:].contiguous())
    outs.append(torch.cat([rows, step]).cpu())
    st.close()
  assert torch.isfinite(outs[0].float()).all()
  for o in outs[1:]:
    assert torch.equal(outs[0], o)
