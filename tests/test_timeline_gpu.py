"""Timeline stamps of the decode Linears (XB_GEMM_TS=1): every block that works writes every stamp of the producers, also one with fewer
k-blocks than its ring has stages, and prompt Linears, which write none, take up no record."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_every_block_stamps_its_producers(built_lib, monkeypatch):
  from oracle import torch_oracle as O
  from xotorch_support_jetson_b200 import models
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  from xotorch_support_jetson_b200.synth import random_hf_state
  monkeypatch.setenv("XB_GEMM_TS", "1")
  hf = models.model_cards["llama-3.2-tiny"]["hf_config"]
  cfg = O.model_config_from_hf(hf)
  nl = cfg["num_layers"]
  st = StageRuntime(Shard("llama-3.2-tiny", 0, nl - 1, nl), cfg, device=0, max_batch_tokens=256, max_seqs=2, max_tokens_per_seq=256)
  st.load_state(random_hf_state(hf, seed=1))
  ids = torch.randint(1, cfg["vocab_size"], (200,), generator=torch.Generator().manual_seed(1)).to("cuda", torch.int32)
  st.timeline()
  st.forward([0], [200], [0], tokens=ids)
  assert st.timeline().shape[0] == 1        # the head, of one row
  st.forward([0], [1], [200], tokens=ids[:1])
  ts = st.timeline()
  assert ts.shape[0] == 4 * nl + 1
  for launch in ts:
    act = launch[:, 0] > 0
    assert act.any()
    # boxes of weights, dependency, first MMA, last MMA, end of the weights
    assert (launch[act][:, [1, 2, 3, 4, 9]] >= launch[act][:, :1]).all()
    assert (launch[act][:, 1] <= launch[act][:, 9]).all()
  st.close()
