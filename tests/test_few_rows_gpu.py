"""Steps of one to a few dozen single tokens on the hybrid engine, at sizes where the row kernels of such steps change what they do: a
stream wider than one pass of a block, branches of many split-K planes, a norm over more channels than a block has threads, delta heads of
more channels than a lane holds, latents and value rows beyond what is fetched ahead of the attention, shares of keys that short
sequences leave empty."""
import pytest
import torch

from test_bibevik_gpu import TOL, bf16_round, config, experts, gdelta, glu, latent, lightning, logits, rel, stage, toks, weights

pytestmark = pytest.mark.gpu

MODELS = {
  "wide": config([(lightning(heads=8, dim=16, vdim=264), glu(1536)), (gdelta(heads=2, dim=96, rank=8), None),
                  (latent(heads=3, dim=40, rot_dim=12, vdim=72, kv_rank=320, dims=8), experts())], width=1152, vocab=90),
  "narrow": config([(gdelta(heads=9, dim=64, rank=16), glu(72)), (latent(heads=16, dim=24, rot_dim=8, vdim=8, kv_rank=48), glu(64)),
                    (lightning(heads=1, dim=8, vdim=40), None)], width=1024, vocab=90),
}
CONTEXTS = [150, 1, 33, 2, 64, 31, 5, 95, 17]


@pytest.mark.parametrize("n_seqs", [1, 9, 18])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_single_token_steps_against_the_oracle(built_lib, name, dtype, n_seqs):
  cfg = MODELS[name]
  w = weights(cfg, seed=31)
  ctx = [CONTEXTS[i % len(CONTEXTS)] for i in range(n_seqs)]
  ids = [toks(c + 2, cfg["vocab"], seed=40 + c) for c in ctx]
  refs = {c: logits(cfg, w, toks(c + 2, cfg["vocab"], seed=40 + c), rounding=bf16_round if dtype == "bfloat16" else None) for c in set(ctx)}
  st = stage(cfg, w, dtype, page=16, seqs=n_seqs, cap=2048)
  flat = lambda rows: torch.tensor([t for r in rows for t in r], dtype=torch.int32, device="cuda")
  st.forward(list(range(n_seqs)), ctx, [0] * n_seqs, tokens=flat([r[:c] for r, c in zip(ids, ctx)]), want_rows=[])
  for step in range(2):
    call = dict(tokens=flat([[r[c + step]] for r, c in zip(ids, ctx)]))
    got = st.forward(list(range(n_seqs)), [1] * n_seqs, [c + step for c in ctx], **call).cpu().double()
    ref = torch.stack([refs[c][c + step] for c in ctx])
    assert rel(got, ref) < TOL[dtype]
    for g, r in zip(got, ref):
      assert rel(g[None], r[None]) < 2 * TOL[dtype]   # one row: the batch's bound with room for its smaller sample
  st.close()
