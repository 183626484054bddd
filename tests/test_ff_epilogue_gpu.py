"""Feed-forwards of hybrid prompts with the activation in the up Linear's epilogue against the kernels of their own: every activation, experts with routing weights on output and input, a shared expert, widths of one and several 128-feature halves, rows around a tile's end."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu

# (model, layer index, feed-forward of that layer)
_FF = {
  "relu2": ("refatar-tiny", 0, None),
  "clamped": ("bibevik-tiny", 0, {"kind": "dense", "ff": 384, "limit": 1.5}),
  "experts, shared": ("bibevik-tiny", 1, {"kind": "moe", "expert": {"ff": 128, "limit": 2.0}, "shared": {"ff": 256, "limit": 2.0},
                                          "router": {"experts": 8, "top": 2, "scale": 1.5, "groups": {"count": 4, "keep": 2}}}),
  "experts, no shared": ("bibevik-tiny", 1, {"kind": "moe", "expert": {"ff": 256, "limit": 2.0},
                                             "router": {"experts": 4, "top": 1, "scale": 1.0, "groups": {"count": 2, "keep": 1}}}),
  "swiglu experts": ("pufivik-tiny", None, 128),
}


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
def test_epilogue_equals_kernel(built_lib, monkeypatch, name, n):
  from xotorch_support_jetson_b200 import synth
  from xotorch_support_jetson_b200.models import model_cards
  mid, at, ff = _FF[name]
  hf = copy.deepcopy(model_cards[mid]["hf_config"])
  if at is not None:
    hf["layers"] = [hf["layers"][at]]
    hf["layers"][0].pop("weights_of", None)
    if ff is not None:
      hf["layers"][0]["mlp"] = ff
  else:   # the first expert layer, experts of `ff` features
    hf["layers"] = [next(l for l in hf["layers"] if (l["mlp"] or {}).get("kind") == "moe")]
    hf["layers"][0]["mlp"]["expert"]["ff"] = ff
  state = getattr(synth, f"random_{mid.split('-')[0]}_state")(hf, seed=7)
  got = {}
  for on in ("0", "1"):
    monkeypatch.setenv("XB_HY_ACT", on)
    got[on] = _stream(hf, state, n, "bfloat16")
  (a, la), (b, lb) = got["0"], got["1"]
  assert torch.isfinite(b).all() and lb == la - 1        # a kernel less
  if name == "relu2":
    assert torch.equal(a, b)
  # the sigmoids differ by a few 1e-7, so one activation in some 1e4 rounds to a neighbouring bf16 (2^-8): 4e-5 of a row, a few times that behind a layer
  assert ((a - b).norm() / a.norm()).item() < 2e-4


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
  assert ((got["0"] - got["1"]).norm() / got["0"].norm()).item() < 2e-4   # as above
