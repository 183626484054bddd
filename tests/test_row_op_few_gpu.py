"""Residual + norms of hybrid steps of few rows, four channels a thread (hy_row_op_few_kernel), against the general kernel, bit for bit: at widths around
its limits, with split-K planes (bf16; fewer and more of them than a round fetches) and plain matrices (float32), the sandwich form and the plain sum with a
Linear's input."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu


def _steps(model, width, dtype, rows, ff):
  from xotorch_support_jetson_b200 import model_config, synth
  from xotorch_support_jetson_b200.models import model_cards
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf = dict(copy.deepcopy(model_cards[model]["hf_config"]), width=width)
  hf["layers"] = hf["layers"][:2]
  if ff is not None:
    hf["layers"][0]["mlp"]["ff"] = ff
  cfg = model_config.hybrid_model_config(hf)
  w = getattr(synth, f"random_{model.split('-')[0]}_state")(hf, seed=5, device="cuda")
  model_config.resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in w.items()})
  st = StageRuntime(Shard("x", 0, 1, 2), cfg, max_batch_tokens=64, max_seqs=rows, max_tokens_per_seq=16, dtype=dtype)
  st.load_state(w)
  g = torch.Generator().manual_seed(width)
  outs = []
  for s in range(3):
    ids = torch.randint(1, hf["vocab"], (rows,), generator=g).to("cuda", torch.int32)
    stream = torch.empty((rows, width), dtype=torch.float32, device="cuda")
    outs += [st.forward(list(range(rows)), [1] * rows, [s] * rows, tokens=ids, taps=[None, stream]).clone(), stream]
  torch.cuda.synchronize()
  st.close()
  return [o.cpu() for o in outs]


@pytest.mark.parametrize("model", ["refatar-tiny", "bibevik-tiny"])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,rows,ff", [(1024, 1, None), (1032, 5, None), (1536, 64, None), (2048, 3, None), (2056, 2, None), (4096, 1, None), (4104, 2, None),
                                           (1024, 4, 8192), (2056, 3, 8192)])   # 8192 features over 8 and 17 tiles: some twenty and ten planes a column
def test_few_rows_have_the_bits_of_the_general_kernel(built_lib, monkeypatch, model, dtype, width, rows, ff):
  got = _steps(model, width, dtype, rows, ff)
  monkeypatch.setenv("XB_HY_QUAD", "0")
  for a, b in zip(got, _steps(model, width, dtype, rows, ff)):
    assert torch.isfinite(a).all()
    assert torch.equal(a, b)
