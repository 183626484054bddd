"""The float32 mode's Linears on the tensor cores (fp32 rows as three exact bf16 pieces) against the plain FMA kernels on the same
model and tokens, and both against the float64 oracle."""
import pytest
import torch

import bibevik_oracle
import refatar_oracle

pytestmark = pytest.mark.gpu

_ORACLE = {"refatar-tiny": lambda cfg, w, ids: refatar_oracle.forward(cfg, w, ids), "bibevik-tiny": lambda cfg, w, ids: bibevik_oracle.forward(cfg, w, ids)[0]}


def _logits(mid, hf, state, ids, monkeypatch, tensor_cores):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  monkeypatch.setenv("XB_HY_TC", "1" if tensor_cores else "0")
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  nl, n = cfg["num_layers"], len(ids)
  st = StageRuntime(Shard(mid, 0, nl - 1, nl), cfg, max_batch_tokens=n, max_seqs=2, max_tokens_per_seq=n + 8, dtype="float32", max_logit_rows=n)
  st.load_state(state)
  rows = sorted({0, n // 2, n - 1})
  out = st.forward([0], [n], [0], tokens=torch.tensor(ids, dtype=torch.int32, device="cuda"), want_rows=rows).cpu()
  torch.cuda.synchronize()
  st.close()
  return rows, out.double()


@pytest.mark.parametrize("mid", ["refatar-tiny", "bibevik-tiny"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 127, 128, 129, 300, 2049])   # edges of the row box, of the 128-row tile and of the 2048-row workspace
def test_pieces_on_tensor_cores_equal_plain_fma(built_lib, monkeypatch, mid, n):
  from xotorch_support_jetson_b200.models import model_cards
  from xotorch_support_jetson_b200 import synth
  hf = model_cards[mid]["hf_config"]
  state = {"refatar-tiny": synth.random_refatar_state, "bibevik-tiny": synth.random_bibevik_state}[mid](hf, seed=3)
  ids = torch.randint(0, hf["vocab"], (n,), generator=torch.Generator().manual_seed(n)).tolist()
  rows, tc = _logits(mid, hf, state, ids, monkeypatch, True)
  _, plain = _logits(mid, hf, state, ids, monkeypatch, False)
  # the two differ by the order of fp32 sums of up to 512 terms through 4 or 5 layers: a few 1e-6 of the logits' size
  assert (tc - plain).norm() <= 1e-5 * plain.norm()
  if n <= 300:
    ref = _ORACLE[mid](hf, state, ids)[rows].double()
    assert (tc - ref).norm() <= max(1.5 * float((plain - ref).norm()), 1e-6 * float(ref.norm()))


@pytest.mark.parametrize("n", [1, 300])
def test_infinite_weights_answer_as_plain_fma(built_lib, monkeypatch, n):
  """One infinite weight per logit: the product is an infinity of the activation's sign, whatever its low bits."""
  from xotorch_support_jetson_b200 import synth
  from xotorch_support_jetson_b200.models import model_cards
  hf = model_cards["bibevik-tiny"]["hf_config"]
  state = synth.random_bibevik_state(hf, seed=3)
  V, D = state["head"].shape
  state["head"][torch.arange(V), torch.arange(V) % D] = float("inf")
  ids = torch.randint(0, hf["vocab"], (n,), generator=torch.Generator().manual_seed(n)).to(torch.int32)
  rows, tc = _logits("bibevik-tiny", hf, state, ids.tolist(), monkeypatch, True)
  _, plain = _logits("bibevik-tiny", hf, state, ids.tolist(), monkeypatch, False)
  assert torch.isinf(plain).any()
  assert torch.equal(torch.isnan(tc), torch.isnan(plain))
  assert torch.equal(tc.sign()[torch.isinf(plain)], plain.sign()[torch.isinf(plain)]) and torch.equal(torch.isinf(tc), torch.isinf(plain))
