"""Residual + norm of a decode step at every width where its kernel changes (512, 768 and 1024 threads, one or two groups of four columns a thread): a token
step against the same row at the end of a prompt, and a pipeline cut against the uncut model."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (512, 8192): 32 split-K planes a column, where a round fetches 12; (3584, 18944): 7 where it fetches 6
@pytest.mark.parametrize("D,I", [(648, 512), (2048, 512), (2056, 512), (3072, 512), (3080, 512), (4096, 512), (4104, 512), (8192, 512), (512, 8192), (2056, 16384), (3584, 18944)])
@pytest.mark.parametrize("kind", ["interleaved", "half-split"])
def test_token_step_against_prompt_and_cut(built_lib, D, I, kind):
  from oracle import torch_oracle as O
  from xotorch_support_jetson_b200 import models
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  from xotorch_support_jetson_b200.synth import random_hf_state
  if kind == "interleaved":
    mid, hf = "llama-3.2-tiny", dict(models.model_cards["llama-3.2-tiny"]["hf_config"], hidden_size=D, num_attention_heads=8, num_key_value_heads=2, head_dim=64,
                                     intermediate_size=I, num_hidden_layers=2)
  else:   # with biases
    if D % 128:
      pytest.skip("heads of 128 fill the width")
    mid, hf = "qwen-2.5-widths", models._qwen(D, D // 128, D // 128, I, 2, vocab=1536, max_pos=4096)
  cfg = O.model_config_from_hf(hf)
  state = random_hf_state(hf, seed=3, std=0.05, norm_jitter=0.1)
  n = 140
  ids = torch.randint(1, cfg["vocab_size"], (n,), generator=torch.Generator().manual_seed(D)).to("cuda", torch.int32)

  def stage(a, b):
    st = StageRuntime(Shard(mid, a, b, 2), cfg, device=0, max_batch_tokens=256, max_seqs=2, max_tokens_per_seq=256)
    st.load_state(state)
    return st

  whole = stage(0, 1)
  prompt = whole.forward([0], [n], [0], tokens=ids).clone()
  whole.forward([1], [n - 1], [0], tokens=ids[:-1].contiguous())
  step = whole.forward([1], [1], [n - 1], tokens=ids[-1:].contiguous()).clone()
  whole.close()
  first, second = stage(0, 0), stage(1, 1)
  second.forward([0], [n - 1], [0], hidden=first.forward([0], [n - 1], [0], tokens=ids[:-1].contiguous()))
  cut = second.forward([0], [1], [n - 1], hidden=first.forward([0], [1], [n - 1], tokens=ids[-1:].contiguous()))
  torch.cuda.synchronize()
  assert torch.isfinite(step).all()
  # two layers of bf16 activations whose sums are taken in two orders: a few roundings of 2^-8 each
  assert ((step - prompt).norm() / prompt.norm()).item() < 0.02
  assert torch.equal(step, cut)
  first.close()
  second.close()
