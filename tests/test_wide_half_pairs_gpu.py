"""Prompt Linears on CTA pairs of 64 token rows each (tiles of 128 rows x 128 or 256 features): every edge of their tiles."""
import pytest
import torch

from test_prompt_portions_gpu import _rows, _stage

pytestmark = pytest.mark.gpu
PAIRS_64 = (5, 6)   # 256 and 128 features


@pytest.mark.parametrize("variant", PAIRS_64)
@pytest.mark.parametrize("T,N,K", [(129, 512, 1024), (192, 128, 64), (193, 1000, 328), (257, 200, 2048), (700, 640, 1088), (2100, 3200, 192)])
def test_linear_matches_fp64(built_lib, variant, T, N, K):
  """One row past a CTA's half and past a tile, features that end inside a half and inside a chunk of 16, odd numbers of k-blocks, several tiles a pair."""
  from xotorch_support_jetson_b200.stage import debug_linear
  g = torch.Generator(device="cuda").manual_seed(T + N + K)
  x = (torch.randn(T, K, device="cuda", generator=g) * 0.5).to(torch.bfloat16)
  w = (torch.randn(N, K, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
  y = debug_linear(x, w, use_tensor_cores=True, force_splits=variant)
  ref = x.double() @ w.double().t()
  torch.cuda.synchronize()
  # one bf16 rounding of a sum that is off by at most K fp32 roundings of its largest partial sum
  bound = ref.abs() * 2 ** -8 + K * 2 ** -24 * (x.double().abs() @ w.double().abs().t())
  assert ((y.double() - ref).abs() <= bound).all()
  assert torch.equal(y, debug_linear(x, w, use_tensor_cores=True, force_splits=2))   # one order of sums in every tile shape


@pytest.mark.parametrize("kind", ["interleaved", "half-split"])
@pytest.mark.parametrize("sizes", [(10, 2, 64, 992), (5, 1, 128, 1120)])   # features of every site end inside a tile
@pytest.mark.parametrize("n", [129, 193, 300])
def test_engine_epilogues_have_the_same_bits(built_lib, monkeypatch, kind, sizes, n):
  """Rotation, cache append and SiLU from both lane halves; where a head of 128 may not be cut, 128 features fall back to another tile."""
  outs = []
  for variant in (2, *PAIRS_64):
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
