"""SiLU in the epilogue of a prompt's gate/up Linear against the kernel of steps of up to 128 rows, which divides exactly: every finite bf16 a gate can be."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1, 5])
def test_every_gate_has_the_exact_quotient(built_lib, monkeypatch, variant):
  from oracle import torch_oracle as O
  from xotorch_support_jetson_b200 import models
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  from xotorch_support_jetson_b200.synth import random_hf_state
  D, I = 1024, 64
  hf = dict(models.model_cards["llama-3.2-tiny"]["hf_config"], hidden_size=D, num_attention_heads=16, num_key_value_heads=4, head_dim=64, intermediate_size=I,
            num_hidden_layers=3)
  state = random_hf_state(hf, seed=11, std=0.05)
  layer = "model.layers.1."
  # Row t of the stream is 64 at channel t and the norm makes a one of it: the gate of feature f is the weight [f, t], and the sums are exact.
  state[layer + "self_attn.o_proj.weight"].zero_()
  state[layer + "post_attention_layernorm.weight"].fill_(1 / 32)
  gates = torch.arange(D * I, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).reshape(I, D).clone()
  gates[~torch.isfinite(gates)] = 0
  state[layer + "mlp.gate_proj.weight"] = gates
  state[layer + "mlp.up_proj.weight"] = torch.ones(I, D, dtype=torch.bfloat16)
  down = torch.zeros(D, I, dtype=torch.bfloat16)
  down[:I] = down[512:512 + I] = torch.eye(I)      # twice: one copy lies clear of the row's own channel
  state[layer + "mlp.down_proj.weight"] = down
  if variant:
    monkeypatch.setenv("XB_WIDE_VARIANT", str(variant))
  st = StageRuntime(Shard("llama-3.2-tiny", 1, 1, 3), O.model_config_from_hf(hf), device=0, max_batch_tokens=D, max_seqs=2, max_tokens_per_seq=D)
  st.load_state({k: v for k, v in state.items() if k.startswith(layer)})
  rows = (64 * torch.eye(D)).to("cuda", torch.bfloat16)
  prompt = st.forward([0], [D], [0], hidden=rows).clone()
  few = torch.cat([st.forward([1], [128], [a], hidden=rows[a:a + 128].contiguous()).clone() for a in range(0, D, 128)])
  torch.cuda.synchronize()
  st.close()
  assert torch.isfinite(few).all()
  act = torch.cat([few[:512, 512:512 + I], few[512:, :I]]).float().cpu()
  gate = gates.t().double()   # the few rows do compute SiLU, within two bf16 roundings; below -88.7, where e^-x leaves fp32, 89 e^-88.7 = 3e-37 becomes 0
  bad = (act.double() - gate * torch.sigmoid(gate)).abs() > 2 ** -7 * (gate * torch.sigmoid(gate)).abs() + 3e-37
  assert not bad.any(), (int(bad.sum()), gate[bad][:8], act[bad][:8])
  assert int((prompt != few).sum()) == 0
