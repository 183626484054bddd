"""Feed-forwards of hybrid prompts with the activation in the up Linear's epilogue against the kernels of their own, bit for bit, and against the oracles in 64 bits:
every activation, biases, experts with routing weights on output and input, a shared expert with and without a gate and with a limit of its own, widths of one and several
128-feature halves, rows around a tile's end, gates beyond the range in which the epilogue divides by a reciprocal."""
import copy
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu

# (model, layer index, feed-forward of that layer)
_FF = {
  "relu2": ("refatar-tiny", 0, None),
  "clamped": ("bibevik-tiny", 0, {"kind": "dense", "ff": 384, "limit": 1.5}),
  "geglu": ("rurutar-tiny", 0, {"kind": "dense", "ff": 384}),
  "experts, shared": ("bibevik-tiny", 1, {"kind": "moe", "expert": {"ff": 128, "limit": 2.0}, "shared": {"ff": 256, "limit": 0.5},
                                          "router": {"experts": 8, "top": 2, "scale": 1.5, "groups": {"count": 4, "keep": 2}}}),
  "experts, no shared": ("bibevik-tiny", 1, {"kind": "moe", "expert": {"ff": 256, "limit": 2.0},
                                             "router": {"experts": 4, "top": 1, "scale": 1.0, "groups": {"count": 2, "keep": 1}}}),
  "experts, gated shared": ("rurutar-tiny", 1, {"kind": "moe", "expert": {"ff": 128}, "router": {"experts": 6, "top": 2}, "shared": {"ff": 256}}),
  "swiglu experts": ("pufivik-tiny", 0, {"kind": "moe", "expert": {"ff": 128}, "router": {"experts": 6, "top": 2}}),
}


def _one_layer(mid, at, ff):
  from xotorch_support_jetson_b200 import synth
  from xotorch_support_jetson_b200.models import model_cards
  hf = copy.deepcopy(model_cards[mid]["hf_config"])
  hf["layers"] = [hf["layers"][at]]
  hf["layers"][0].pop("weights_of", None)
  if ff is not None:
    hf["layers"][0]["mlp"] = ff
  return mid.split("-")[0], hf, getattr(synth, f"random_{mid.split('-')[0]}_state")(hf, seed=7)


def _stream(hf, state, n, dtype):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  nl = cfg["num_layers"]
  st = StageRuntime(Shard("ff-test", 0, nl - 1, nl), cfg, max_batch_tokens=n, max_seqs=1, max_tokens_per_seq=n + 8, dtype=dtype)
  st.load_state(state)
  ids = torch.randint(0, hf["vocab"], (n,), generator=torch.Generator().manual_seed(n)).to("cuda", torch.int32)
  out = torch.empty((n, cfg["embed_dim"]), device="cuda")
  st.forward([0], [n], [0], tokens=ids, taps=[None] * (nl - 1) + [out])
  torch.cuda.synchronize()
  launches = st.counters()["launches"]
  st.close()
  return out.double().cpu(), launches


@pytest.mark.parametrize("name", sorted(_FF))
@pytest.mark.parametrize("n", [129, 256, 300])
@pytest.mark.parametrize("gain", [1, 60])   # gates of a few units, and of up to some hundreds
def test_epilogue_equals_kernel(built_lib, monkeypatch, name, n, gain):
  _, hf, state = _one_layer(*_FF[name])
  for k in state:
    if k.startswith("l0.mlp.") and (k.endswith("gate") or k.endswith("up")):
      state[k] = state[k] * gain
  got = {}
  for on in ("0", "1"):
    monkeypatch.setenv("XB_HY_ACT", on)
    got[on] = _stream(hf, state, n, "bfloat16")
  (a, la), (b, lb) = got["0"], got["1"]
  assert torch.isfinite(b).all() and lb == la - 1        # a kernel less
  assert torch.equal(a, b)


@pytest.mark.parametrize("name", sorted(_FF))
def test_epilogue_against_64_bits(built_lib, monkeypatch, name):
  family, hf, state = _one_layer(*_FF[name])
  n = 140
  monkeypatch.setenv("XB_HY_ACT", "1")
  out, _ = _stream(hf, state, n, "bfloat16")
  O = importlib.import_module(f"{family}_oracle")
  ids = torch.randint(0, hf["vocab"], (n,), generator=torch.Generator().manual_seed(n)).tolist()
  state = {k: v.to(torch.bfloat16) for k, v in state.items()}
  if family == "bibevik":
    ref = O.forward(hf, state, ids)[1][-1]
  elif family == "rurutar":
    ref = torch.as_tensor(O.forward(state, hf, ids, want_layers=True)[1][-1])
  else:
    ref = O.forward(hf, state, ids, return_layers=True)[1][-1]
  rows = (out - torch.as_tensor(ref).double()).norm(dim=1) / torch.as_tensor(ref).double().norm(dim=1)
  # a chain of bf16 roundings (2^-9 each) from norm to norm: their spread is a few of them in every row; a router that ties sends single rows to another expert
  assert rows.quantile(0.9) < 0.02


def test_rows_at_which_the_choice_flips(built_lib, monkeypatch):
  """160 -> 2 x 2048 by the estimate: a kernel of its own up to 512 rows, the epilogue from 513 on."""
  _, hf, state = _one_layer("rurutar-tiny", 0, {"kind": "dense", "ff": 2048})
  for n in (512, 513):
    monkeypatch.delenv("XB_HY_ACT", raising=False)
    own, launches = _stream(hf, state, n, "bfloat16")
    monkeypatch.setenv("XB_HY_ACT", "0")
    kernel, more = _stream(hf, state, n, "bfloat16")
    assert more - launches == n - 512
    assert torch.equal(own, kernel)


def test_layers_that_share_weights_keep_their_limits(built_lib, monkeypatch):
  """Two layers over one set of weights, each with a limit of its own: a launch takes its layer's."""
  from xotorch_support_jetson_b200 import synth
  from xotorch_support_jetson_b200.models import model_cards
  hf = copy.deepcopy(model_cards["bibevik-tiny"]["hf_config"])
  lay = next(l for l in hf["layers"] if l["type"] == "latent_attention")
  lay.pop("weights_of", None)
  hf["layers"] = [dict(lay, mlp={"kind": "dense", "ff": 384, "limit": 0.05}), dict(lay, mlp={"kind": "dense", "ff": 384, "limit": 2.0}, weights_of=0)]
  state = synth.random_bibevik_state(hf, seed=8)
  got = {}
  for on in ("0", "1"):
    monkeypatch.setenv("XB_HY_ACT", on)
    got[on], _ = _stream(hf, state, 300, "bfloat16")
  assert torch.equal(got["0"], got["1"])
