"""Latent attention in steps of few rows (a row a block: hy_latent_absorb_row_kernel, the read-out's early weights) against the same rows in a wider step, at
sizes around what a thread fetches ahead (64 rows of keys' weights, 512 latent columns, 128 value channels) and at a latent width that takes the older kernel.  In
float32 a row has the same bits in both: its sums do not hang on how many rows the step has."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,rank,vdim", [(64, 256, 128), (24, 48, 40), (72, 264, 136), (8, 16, 8), (130, 512, 64), (24, 44, 40), (24, 45, 40)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_few_rows_equal_many(built_lib, dim, rank, vdim, dtype):
  from xotorch_support_jetson_b200 import model_config, synth
  from xotorch_support_jetson_b200.models import model_cards
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  hf = dict(model_cards["bibevik-tiny"]["hf_config"])
  lay = next(l for l in hf["layers"] if l["type"] == "latent_attention")
  hf["layers"] = [dict(lay, mixer=dict(lay["mixer"], dim=dim, kv_rank=rank, vdim=vdim, scale=(dim + lay["mixer"]["rot_dim"]) ** -0.5), mlp=None)]
  hf["layers"][0].pop("weights_of", None)
  cfg = model_config.hybrid_model_config(hf)
  w = synth.random_bibevik_state(hf, seed=9)
  model_config.resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in w.items()})
  n = 20                                     # rows of the wide step: more than the 16 that take the row kernels
  ids = torch.randint(0, hf["vocab"], (n, 9), generator=torch.Generator().manual_seed(rank)).to("cuda", torch.int32)

  def run(groups):
    st = StageRuntime(Shard("latent-test", 0, 0, 1), cfg, max_batch_tokens=256, max_seqs=n, max_tokens_per_seq=16, dtype=dtype)
    st.load_state(w)
    st.forward(list(range(n)), [8] * n, [0] * n, tokens=ids[:, :8].reshape(-1).contiguous())
    rows = []
    for g in groups:
      out = torch.empty((len(g), cfg["embed_dim"]), device="cuda")
      st.forward(list(g), [1] * len(g), [8] * len(g), tokens=ids[g[0]:g[-1] + 1, 8].contiguous(), taps=[out])
      rows.append(out)
    torch.cuda.synchronize()
    st.close()
    return torch.cat(rows).double().cpu()

  many = run([range(n)])
  few = run([range(0, 1), range(1, 4), range(4, 20)])
  assert torch.isfinite(few).all()
  if dtype == "float32":
    assert torch.equal(few, many)
  # bf16 steps share their keys out by the step's rows: fp32 sums in another order, after which a rounding (2^-9) of any of the layer's activations may fall the other way
  assert ((few - many).norm(dim=1) / many.norm(dim=1)).max() < 2 ** -7
