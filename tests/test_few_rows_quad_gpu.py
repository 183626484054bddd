"""Gated feed-forwards, experts and logits of hybrid steps of few rows, four columns a thread, against the kernels that take one, bit for bit: on split-K planes
(bf16; some columns with more of them than a round fetches) and plain matrices (float32), with vocabularies and widths that do and do not divide by four."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


# rows of 1024 channels: narrower ones take, with the switch, another kernel for residual + norm as well
@pytest.mark.parametrize("model,change", [("bibevik-tiny", {}), ("bibevik-tiny", {"vocab": 386}), ("bibevik-tiny", {"ff": 66}), ("bibevik-tiny", {"width": 4096}),
                                          ("pufivik-tiny", {}), ("vusenex-tiny", {}), ("rurutar-tiny", {}), ("rurutar-tiny", {"width": 4096}), ("sizolorn-tiny", {})])
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("rows", [1, 5, 64])
def test_four_columns_equal_one(built_lib, monkeypatch, model, change, dtype, rows):
  import inspect

  from xotorch_support_jetson_b200 import model_config, synth
  from xotorch_support_jetson_b200.models import model_cards
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf = copy.deepcopy(model_cards[model]["hf_config"])
  hf["width"] = change.get("width", 1024)   # 4096: 64 k-blocks over few tiles, a dozen planes and more a column
  if "vocab" in change:
    hf["vocab"] = change["vocab"]
  if "ff" in change:
    for lay in hf["layers"]:
      if lay["mlp"] and lay["mlp"]["kind"] == "dense":
        lay["mlp"]["ff"] = change["ff"]
  make = getattr(synth, f"random_{model.split('-')[0]}_state")
  w = make(hf, seed=4, **({"device": "cuda"} if "device" in inspect.signature(make).parameters else {}))
  cfg = model_config.hybrid_model_config(hf)
  model_config.resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in w.items()})
  ids = torch.randint(0, hf["vocab"], (2, rows), generator=torch.Generator().manual_seed(rows)).to("cuda", torch.int32)
  outs = []
  for quad in ("1", "0"):
    monkeypatch.setenv("XB_HY_QUAD", quad)
    st = StageRuntime(Shard("quad-test", 0, cfg["num_layers"] - 1, cfg["num_layers"]), cfg, max_batch_tokens=64, max_seqs=rows, max_tokens_per_seq=8, dtype=dtype)
    st.load_state(w)
    outs.append(torch.stack([st.forward(list(range(rows)), [1] * rows, [s] * rows, tokens=ids[s].contiguous()).clone() for s in range(2)]).cpu())
    st.close()
  assert torch.isfinite(outs[0]).all()
  assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("n", [65535, 65536])
def test_logits_of_more_rows_than_a_grid_has(built_lib, n):
  """A program may ask for the logits of any number of rows, the same one several times."""
  from xotorch_support_jetson_b200 import model_config, synth
  from xotorch_support_jetson_b200.models import model_cards
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf = copy.deepcopy(model_cards["bibevik-tiny"]["hf_config"])
  hf["vocab"], hf["layers"] = 64, hf["layers"][:1]
  w = synth.random_bibevik_state(hf, seed=4)
  cfg = model_config.hybrid_model_config(hf)
  model_config.resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in w.items()})
  st = StageRuntime(Shard("rows-test", 0, 0, 1), cfg, max_batch_tokens=64, max_seqs=1, max_tokens_per_seq=8, dtype="bfloat16", max_logit_rows=n)
  st.load_state(w)
  ids = torch.randint(0, hf["vocab"], (4,), generator=torch.Generator().manual_seed(1)).to("cuda", torch.int32)
  got = st.forward([0], [4], [0], tokens=ids, want_rows=[i % 4 for i in range(n)]).clone()
  assert torch.isfinite(got).all() and torch.equal(got, got[:4].repeat((n + 3) // 4, 1)[:n])
  st.close()
