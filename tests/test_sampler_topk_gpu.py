"""The sampler's candidate path (top-k up to 256, one look at the row) and the clustered arg-max against the one-block-per-row
kernels and the restated reference sampler, where the candidates are few, many, tied or not numbers."""
import json
import tempfile
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu


def _stage(V):
  from xotorch_support_jetson_b200 import model_config as mc
  from xotorch_support_jetson_b200.models import model_cards
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf = dict(model_cards["llama-3.2-tiny"]["hf_config"], vocab_size=V)
  with tempfile.TemporaryDirectory() as td:
    (Path(td) / "config.json").write_text(json.dumps(hf))
    cfg = mc.load_model_config(Path(td) / "config.json")
  nl = cfg["num_layers"]
  return StageRuntime(Shard("llama-3.2-tiny", 0, nl - 1, nl), cfg, device=0, max_batch_tokens=16, max_seqs=8, max_tokens_per_seq=32)


def _rows(V, g):
  """Rows of the kinds a sampler meets: spread, rounded to bf16 (ties), few distinct values, constant, masked to a few entries."""
  x = torch.randn(6, V, generator=g) * 3
  x[1] = x[1].to(torch.bfloat16).float()
  x[2] = torch.randint(0, 5, (V,), generator=g).float()
  x[3] = 1.5
  x[4, torch.randperm(V, generator=g)[: V - 9]] = -float("inf")
  x[5] = torch.finfo(torch.float32).min
  x[5, V // 2] = 0.0
  return x


@pytest.mark.parametrize("V", [128256, 152064, 4097, 1000])
@pytest.mark.parametrize("top_k", [1, 2, 35, 64, 65, 256, 257])
def test_candidates_equal_radix_passes(built_lib, monkeypatch, V, top_k):
  from oracle import torch_oracle as O
  st = _stage(V)
  g = torch.Generator().manual_seed(V + top_k)
  logits, q = _rows(V, g), torch.empty(6, V).exponential_(1, generator=g)
  ref = O.sample(logits.clone(), temperature=0.7, top_k=top_k, q=q).reshape(-1).to(torch.int64)
  for top_p in (0.0, 0.6):
    got = {}
    for cluster in ("1", "0"):
      monkeypatch.setenv("XB_SAMPLE_CLUSTER", cluster)
      got[cluster] = st.sample(logits.cuda(), temp=0.7, top_k=top_k, top_p=top_p, q=q.cuda()).cpu().to(torch.int64)
      noise = st.sample(logits.cuda(), temp=0.7, top_k=top_k, top_p=top_p, seed=11).cpu().to(torch.int64)
      got[cluster] = torch.cat([got[cluster], noise])
    assert torch.equal(got["1"], got["0"]), (V, top_k, top_p, got)
    if top_p == 0.0:
      assert torch.equal(got["1"][:6], ref)
  bad = logits.clone()
  bad[0, V // 3] = float("nan")
  bad[1, V - 1] = float("inf")
  got = []
  for cluster in ("1", "0"):
    monkeypatch.setenv("XB_SAMPLE_CLUSTER", cluster)
    got.append(st.sample(bad.cuda(), temp=0.7, top_k=top_k, q=q.cuda()).cpu())
  # (top-k 1 of a row with a NaN: the pivot is the NaN itself, and the two kernels' radix passes answer differently)
  assert torch.equal(got[0][top_k == 1:], got[1][top_k == 1:])
  st.close()


@pytest.mark.parametrize("V", [4095, 4096, 4097, 50257, 128256])
@pytest.mark.parametrize("rows", [1, 7])
def test_argmax_is_the_first_largest(built_lib, V, rows):
  st = _stage(V)
  g = torch.Generator().manual_seed(V)
  x = torch.randn(rows, V, generator=g).to(torch.bfloat16).float()
  x[0, [3, V // 2, V - 1]] = 9.0
  x[-1] = x[-1].clamp(max=1.0)
  got = st.sample(x.cuda(), temp=0.0).cpu()
  for r in range(rows):
    assert got[r].item() == int((x[r] == x[r].max()).nonzero()[0])
  st.close()
