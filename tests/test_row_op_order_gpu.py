"""The order in which residual + norm of hybrid models adds the squares of a row is part of its result: every later rounding follows from it.  Prompts whose
branch is one bf16 matrix take one kernel, with and without the four-channel kernels."""
import copy

import pytest
import torch

from test_quad_kernels_gpu import _stream

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [128, 1032, 2048])
@pytest.mark.parametrize("lens", [[129], [150, 30, 41]])
def test_prompts_of_one_branch_have_one_order(built_lib, monkeypatch, width, lens):
  """Entries of the stream are +-1/2 and mixer and token side add nothing, so every sum of squares but that of the feed-forward's output is exact in any
  order and the switch changes nothing else."""
  from xotorch_support_jetson_b200 import synth
  from xotorch_support_jetson_b200.models import model_cards
  hf = copy.deepcopy(model_cards["refatar-tiny"]["hf_config"])
  hf["width"] = width
  hf["layers"] = [hf["layers"][0]]
  state = synth.random_refatar_state(hf, seed=5)
  state["embed"] = torch.where(state["embed"] < 0, -0.5, 0.5).to(state["embed"].dtype)
  for name in ("l0.mix.o", "l0.side.proj"):
    state[name] = torch.zeros_like(state[name])
  out = []
  for quad in ("1", "0"):
    monkeypatch.setenv("XB_HY_QUAD", quad)
    out.append(_stream(hf, state, lens, 0, "bfloat16"))
  assert (out[0].abs() != 0.5).any()          # the feed-forward's output is there
  assert torch.equal(out[0], out[1])
