"""Latent attention on the tensor cores at the edges of its tiles: latents that fill their value columns and latents that do not, cache rows
that are no multiple of sixteen, heads that do not divide a tile's rows, prompts that end one key before, at and behind a tile of 32 keys."""
import pytest
import torch

from test_bibevik_gpu import TOL, bf16_round, config, glu, latent, logits, rel, stage, toks, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["4", "2"])
@pytest.mark.parametrize("rank,heads", [(128, 5), (256, 16), (112, 3), (272, 1)])
def test_prompts_of_tile_edges(built_lib, monkeypatch, rank, heads, form):
  monkeypatch.setenv("XB_HY_LAT_MMA", form)
  cfg = config([(latent(heads=heads, dim=16, rot_dim=8, vdim=16, kv_rank=rank, scale=0.5), glu(64))], width=64, vocab=50)
  w = weights(cfg, seed=rank + heads)
  lens = [31, 33, 1, 97]
  ids = [toks(n + 32, 50, seed=n) for n in lens]
  refs = [logits(cfg, w, i, rounding=bf16_round) for i in ids]
  st = stage(cfg, w, "bfloat16", page=16)
  flat = lambda rows: torch.tensor([t for r in rows for t in r], dtype=torch.int32, device="cuda")
  new = sum(lens)
  got = st.forward([0, 1, 2, 3], lens, [0] * 4, tokens=flat([i[:n] for i, n in zip(ids, lens)]), want_rows=list(range(new))).cpu().double()
  at = 0
  for ref, n in zip(refs, lens):
    assert rel(got[at:at + n], ref[:n]) < TOL["bfloat16"]
    at += n
  got = st.forward([0, 1, 2, 3], [32] * 4, lens, tokens=flat([i[n:] for i, n in zip(ids, lens)]), want_rows=list(range(128))).cpu().double()   # on top of the cached rows
  for k, (ref, n) in enumerate(zip(refs, lens)):
    assert rel(got[32 * k:32 * k + 32], ref[n:]) < TOL["bfloat16"]
  st.close()
