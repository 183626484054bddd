"""The sampler's candidate path (top-k up to 256, one look at the row) and the clustered arg-max against the one-block-per-row
kernels and the restated reference sampler, where the candidates are few, many, tied or not numbers."""
import json
import tempfile
from pathlib import Path

import numpy as np
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


def _running_sums(e):
  """The sampler's running sums of up to 32 weights: lanes of a shuffle scan, each with a tree of its own."""
  x = np.zeros(32, np.float32)
  x[: len(e)] = e
  for o in (1, 2, 4, 8, 16):
    x = (x + np.concatenate([np.zeros(o, np.float32), x[:-o]])).astype(np.float32)
  return x


def _crossed_twice(rng, weights):
  """30 logits, a top_p that their running sums reach at two ranks, and these ranks: sums of tiny weights dip by an ulp."""
  while True:
    v = np.concatenate([np.sort(rng.standard_normal(12) * 2)[::-1], np.full(18, -17.0) - 0.3 * np.arange(18)]).astype(np.float32)
    v[:12] -= v[0]
    c = _running_sums(weights(v))
    for j in range(1, 40):
      top_p = np.float32(1.0 - j * 2.0 ** -24)
      t = np.float32(top_p * c[31])
      at = [a for a in range(30) if c[a] >= t and (a == 0 or c[a - 1] < t)]
      if len(at) > 1:
        return v, float(top_p), at


def test_nucleus_ends_at_the_first_crossing(built_lib):
  """Where rounding lets the running sums cross top_p more than once, the head up to the first crossing is kept, in every call."""
  V = 4096
  st = _stage(V)
  rng = np.random.default_rng(5)
  for _ in range(20):
    v, top_p, at = _crossed_twice(rng, lambda x: torch.exp(torch.from_numpy(x).cuda()).cpu().numpy())
    logits, q = torch.full((8, V), -200.0), torch.ones(8, V)
    logits[:, torch.arange(30) * 128] = torch.from_numpy(v)   # one per bucket of the candidate search: exactly these are candidates
    q[:, 128 * at[-1]] = 1e-30                                # chosen if it is kept: it lies behind the first crossing
    for _ in range(5):
      assert (st.sample(logits.cuda(), temp=1.0, top_k=30, top_p=top_p, q=q.cuda()) == 0).all(), (top_p, at)
  st.close()


@pytest.mark.parametrize("top_p", [0.0, 0.9])
@pytest.mark.parametrize("top_k", [35, 64, 65, 256])
def test_ties_around_the_candidate_limits(built_lib, monkeypatch, top_k, top_p):
  """As many tied largest entries as the candidates of a row and of a block may be, and one more and less."""
  V = 32768
  st = _stage(V)
  g = torch.Generator().manual_seed(top_k)
  counts = [255, 256, 257, 511, 513, 767, 768, 769, 1023, 1024, 1025, 1500, 2049]
  x = torch.randn(len(counts), V, generator=g)
  for r, n in enumerate(counts):
    x[r, torch.randperm(V, generator=g)[:n]] = 9.0
  x = torch.cat([x, x])
  x[len(counts):, : V // 4 - 600] = -3.0   # the same with most of the ties in three of the four blocks
  q = torch.empty_like(x).exponential_(1, generator=g).cuda()
  got = []
  for cluster in ("1", "0"):
    monkeypatch.setenv("XB_SAMPLE_CLUSTER", cluster)
    got.append(st.sample(x.cuda(), temp=0.7, top_k=top_k, top_p=top_p, q=q).cpu())
  assert torch.equal(got[0], got[1])
  st.close()
