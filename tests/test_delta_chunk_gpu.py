"""The delta rules by chunks of sixteen tokens against the same rules token by token (float32 engine): lengths around a chunk's and the
rule's edges, key and value sizes around the kernel's tiles, shared key heads, unequal sequences, prompts that go on from a
cached state, and decays near zero and one."""
import pytest
import torch

pytestmark = pytest.mark.gpu

_MLP = {"kind": "dense", "ff": 64}


def _model(kind, dk, dv, heads, kv):
  from xotorch_support_jetson_b200 import synth
  if kind == "delta":
    hf = {"architecture": "Refatar", "width": 64, "vocab": 97, "norm": {"eps": 1e-5},
          "layers": [{"type": "delta", "mixer": {"heads": heads, "kv_heads": kv, "dim": dk, "vdim": dv, "conv": 2}, "mlp": None}]}
    state = synth.random_refatar_state(hf, seed=dk + dv)
    state["l0.mix.A_log"] = torch.linspace(-6.0, 4.5, heads)   # decays from about one down to exp(-90 softplus): zero within a few tokens
  else:
    hf = {"architecture": "Bibevik", "width": 64, "vocab": 97, "embedding": {"scale": 8.0}, "norm": {"eps": 1e-6},
          "layers": [{"type": "general_delta", "mixer": {"heads": heads, "dim": dk, "rank": 8}, "mlp": None}]}
    state = synth.random_bibevik_state(hf, seed=dk)
    state["l0.mix.w0"] = torch.linspace(-9.0, 9.0, heads * dk)   # decays over their whole range
  return hf, state


def _run(hf, state, lens, monkeypatch, by_steps):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  monkeypatch.setenv("XB_HY_LPC", "16" if by_steps else "0")
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  st = StageRuntime(Shard("delta-test", 0, 0, 1), cfg, max_batch_tokens=sum(lens), max_seqs=len(lens), max_tokens_per_seq=2 * max(lens) + 8, dtype="float32")
  st.load_state(state)
  g = torch.Generator().manual_seed(sum(lens))
  outs = []
  for start in (0, 1):   # twice the same lengths: the second half goes on from the cached state
    ids = torch.randint(0, 97, (sum(lens),), generator=g).to("cuda", torch.int32)
    tap = torch.empty((sum(lens), 64), device="cuda")
    st.forward(list(range(len(lens))), lens, [start * n for n in lens], tokens=ids, taps=[tap])
    outs.append(tap.double().cpu())
  torch.cuda.synchronize()
  st.close()
  return torch.cat(outs)


@pytest.mark.parametrize("lens", [[96], [97], [111], [112], [113], [32, 300], [100, 96, 130]])
@pytest.mark.parametrize("kind,dk,dv,heads,kv", [("delta", 32, 48, 4, 2), ("delta", 64, 16, 3, 1), ("delta", 65, 17, 2, 2), ("delta", 128, 33, 4, 4),
                                                 ("delta", 200, 40, 2, 1), ("general", 32, 32, 3, 3), ("general", 64, 64, 2, 2), ("general", 72, 72, 2, 2),
                                                 ("general", 130, 130, 1, 1)])
def test_chunks_equal_steps(built_lib, monkeypatch, kind, dk, dv, heads, kv, lens):
  hf, state = _model(kind, dk, dv, heads, kv)
  a, b = (_run(hf, state, lens, monkeypatch, steps) for steps in (False, True))
  assert torch.isfinite(a).all()
  # both sum dk + 16 fp32 products in another order; read-out norm and output projection carry that on: a few 1e-6 of a row
  err = (a - b).norm(dim=1) / b.norm(dim=1)
  assert err.max() < 2e-5, err.max()


def _stage(hf, state, rows, seqs, per_seq):
  from xotorch_support_jetson_b200.model_config import hybrid_model_config, resolve_tensor_sizes
  from xotorch_support_jetson_b200.shard import Shard
  from xotorch_support_jetson_b200.stage import StageRuntime
  cfg = hybrid_model_config(hf)
  resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in state.items()})
  st = StageRuntime(Shard("delta-test", 0, 0, 1), cfg, max_batch_tokens=rows, max_seqs=seqs, max_tokens_per_seq=per_seq, dtype="float32")
  st.load_state(state)
  return st


def _calls(st, calls):
  """Stream rows of calls (slots, lengths, starts); the ids depend on slot and position alone."""
  outs = []
  for slots, lens, starts in calls:
    ids = [torch.randint(0, 97, (2048,), generator=torch.Generator().manual_seed(s))[a:a + n] for s, n, a in zip(slots, lens, starts)]
    tap = torch.empty((sum(lens), 64), device="cuda")
    st.forward(slots, lens, starts, tokens=torch.cat(ids).to("cuda", torch.int32), taps=[tap])
    outs.append(tap.cpu())
  torch.cuda.synchronize()
  return torch.cat(outs)


def _by_steps(monkeypatch, hf, state, calls, rows, seqs, per_seq):
  monkeypatch.setenv("XB_HY_LPC", "16")
  st = _stage(hf, state, rows, seqs, per_seq)
  out = _calls(st, calls)
  st.close()
  monkeypatch.setenv("XB_HY_LPC", "0")
  return out


_MIXES = [
  [[31]], [[32]], [[33]], [[95]], [[1, 32]],                            # where the rules change over
  [[1, 400, 3, 2, 15, 17, 300]], [[5, 4, 3, 2, 1, 100]],                # several sequences that begin inside the same sixteen rows
  [[100, 40, 200], [1, 300, 17]], [[200, 97], [3, 1], [16, 112]],       # continuations of other lengths
]


@pytest.mark.parametrize("lens", _MIXES)
@pytest.mark.parametrize("kind,dk,dv,heads,kv", [("delta", 64, 33, 3, 1), ("delta", 128, 16, 2, 2), ("general", 64, 64, 2, 2), ("general", 72, 72, 2, 2)])
def test_mixed_lengths_equal_steps(built_lib, monkeypatch, kind, dk, dv, heads, kv, lens):
  hf, state = _model(kind, dk, dv, heads, kv)
  calls, at = [], [0] * len(lens[0])
  for part in lens:
    calls.append((list(range(len(part))), part, list(at[: len(part)])))
    at = [a + n for a, n in zip(at, part)] + at[len(part):]
  rows, seqs, per = max(sum(p) for p in lens), len(lens[0]), max(at) + 8
  ref = _by_steps(monkeypatch, hf, state, calls, rows, seqs, per).double()
  st = _stage(hf, state, rows, seqs, per)
  got = _calls(st, calls).double()
  st.close()
  assert torch.isfinite(got).all()
  err = (got - ref).norm(dim=1) / ref.norm(dim=1)
  assert err.max() < 2e-5, err.max()   # as above


@pytest.mark.parametrize("kind", ["delta", "general"])
def test_short_neighbours_do_not_change_a_long_prompt(built_lib, kind):
  hf, state = _model(kind, 64, 64, 2, 2)
  st = _stage(hf, state, 430, 24, 512)
  alone = _calls(st, [([0], [400], [0])])
  beside = _calls(st, [(list(range(1, 23)) + [0], [1] * 22 + [400], [0] * 23)])[22:]
  st.close()
  assert torch.equal(alone, beside)


# a chunk's block of 32 general or 64 gated heads of 256 channels is 2.3 MB: the workspace holds 88 or 89 of them
@pytest.mark.parametrize("kind,dv,lens,first", [("general", 256, [1700], [1408]), ("general", 256, [900, 30, 800], [448, 30, 464]), ("general", 256, [20] * 10 + [1400], None),
                                                ("delta", 16, [1500], [1424]), ("delta", 16, [700, 900], [688, 704])])
def test_steps_beyond_the_workspace(built_lib, monkeypatch, kind, dv, lens, first):
  heads = 32 if kind == "general" else 64
  hf, state = _model(kind, 256, dv, heads, heads)
  n, rows, per = len(lens), sum(lens), max(lens) + 8
  whole = [(list(range(n)), lens, [0] * n)]
  ref = _by_steps(monkeypatch, hf, state, whole, rows, n, per).double()
  st = _stage(hf, state, rows, n, per)
  got = _calls(st, whole)
  err = (got.double() - ref).norm(dim=1) / ref.norm(dim=1)
  assert torch.isfinite(got).all() and err.max() < 2e-5, err.max()   # as above
  if first is not None:   # the same rows in two steps that the workspace holds: the state passes in fp32, so the bits are the same
    rest = [(s, a - b, b) for s, (a, b) in enumerate(zip(lens, first)) if a > b]
    parts = _calls(st, [(list(range(n)), first, [0] * n), ([s for s, _, _ in rest], [k for _, k, _ in rest], [b for _, _, b in rest])])
    heads, tails = parts[: sum(first)].split(first), dict(zip([s for s, _, _ in rest], parts[sum(first):].split([k for _, k, _ in rest])))
    again = torch.cat([torch.cat([heads[s], tails[s]]) if s in tails else heads[s] for s in range(n)])
    assert torch.equal(got, again)
  st.close()


def test_workspaces_follow_the_caches(built_lib):
  """Reserving the caches anew frees the workspaces first and makes them again: the same bits from another place."""
  hf, state = _model("delta", 64, 64, 2, 2)
  st = _stage(hf, state, 300, 3, 512)
  calls = [([0, 1], [200, 97], [0, 0]), ([0, 1], [1, 1], [200, 97])]
  first = _calls(st, calls)
  from xotorch_support_jetson_b200 import _cabi
  _cabi.check(st.lib.xb_kv_reserve(st._h, 3, 512, st.page_tokens))
  assert torch.equal(first, _calls(st, calls))
  st.close()
