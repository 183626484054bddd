"""Prompts above 64 rows take the four-channel row kernels, portions of up to 64 rows the one-channel ones: both must leave the same
stream, at row counts around the eight-row tiles, with sequences that end inside a tile, and for widths that are and are not
multiples of four (the latter keep the one-channel kernels)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stream(hf, state, lens, portion, dtype):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  nl, D = cfg["num_layers"], cfg["embed_dim"]
  st = StageRuntime(Shard("quad-test", 0, nl - 1, nl), cfg, max_batch_tokens=sum(lens), max_seqs=len(lens), max_tokens_per_seq=max(lens) + 8, dtype=dtype)
  st.load_state(state)
  g = torch.Generator().manual_seed(sum(lens))
  ids = [torch.randint(0, hf["vocab"], (n,), generator=g).to("cuda", torch.int32) for n in lens]
  rows = [torch.empty((n, D), device="cuda") for n in lens]
  if portion:
    for i, n in enumerate(lens):
      for a in range(0, n, portion):
        b = min(n, a + portion)
        st.forward([i], [b - a], [a], tokens=ids[i][a:b].contiguous(), taps=[None] * (nl - 1) + [rows[i][a:b]])
  else:
    whole = torch.empty((sum(lens), D), device="cuda")
    st.forward(list(range(len(lens))), lens, [0] * len(lens), tokens=torch.cat(ids), taps=[None] * (nl - 1) + [whole])
    rows = list(whole.split(lens))
  torch.cuda.synchronize()
  out = torch.cat(rows).double().cpu()
  st.close()
  return out


@pytest.mark.parametrize("lens", [[65], [71], [72], [73], [30, 50, 41], [129, 3, 64]])
@pytest.mark.parametrize("mid,dk", [("refatar-tiny", 32), ("refatar-tiny", 34), ("bibevik-tiny", 32), ("bibevik-tiny", 30)])
def test_whole_prompts_equal_portions(built_lib, mid, dk, lens):
  import copy
  from xotorch_support_jetson_b200 import synth
  from xotorch_support_jetson_b200.models import model_cards
  hf = copy.deepcopy(model_cards[mid]["hf_config"])
  for lay in hf["layers"]:
    if lay["type"] in ("delta", "general_delta"):
      lay["mixer"]["dim"] = dk
  state = {"refatar-tiny": synth.random_refatar_state, "bibevik-tiny": synth.random_bibevik_state}[mid](hf, seed=5)
  a, b = (_stream(hf, state, lens, portion, "float32") for portion in (0, 32))
  # fp32 sums of rows and products in another order through 4 or 5 layers
  assert (a - b).norm() <= 1e-5 * b.norm()


@pytest.mark.parametrize("lens", [[129], [150, 30, 41], [1, 200, 7]])   # more than 128 rows: the projections come back as one bf16 matrix
@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("mid", ["refatar-tiny", "bibevik-tiny"])
def test_four_channels_equal_one(built_lib, monkeypatch, mid, dtype, lens):
  """The same rows with the four-channel kernels and with the one-channel ones, one layer of the model at a time."""
  import copy
  from xotorch_support_jetson_b200 import synth
  from xotorch_support_jetson_b200.models import model_cards
  for i in range(3):
    hf = copy.deepcopy(model_cards[mid]["hf_config"])
    hf["layers"] = [hf["layers"][i]]
    state = {"refatar-tiny": synth.random_refatar_state, "bibevik-tiny": synth.random_bibevik_state}[mid](hf, seed=5)
    out = []
    for quad in ("1", "0"):
      monkeypatch.setenv("XB_HY_QUAD", quad)
      out.append(_stream(hf, state, lens, 0, dtype))
    # Row sums in another order, fp32.  In bf16 a last bit of them turns the rounding of a few activations: far below one bf16 step of the row
    assert (out[0] - out[1]).norm() <= (2 ** -9 if dtype == "bfloat16" else 2e-6) * out[1].norm(), i
