"""What users of this framework have it compute, at the sizes they do it at: the work whose speed is looked after.

A case is a dict of plain values.  ``listed`` names the fixed ones, ``draw`` makes more of the same ranges, ``prepare`` builds
what a program holds before the call (engine with its weights, inputs on the device), ``run`` is one pass through the public
calls, ``work`` the bytes and operations a pass cannot do without, ``tolerance`` how far a correct result may be off and
``exact`` the result in 64 bits by plain torch.

Four kinds:

``stage``   a layer range of a Llama-shaped model as one pipeline stage holds it (the whole model where the range is all of
            it): decode steps and prompts, hidden rows or token ids in, hidden rows or logits out.
``sample``  one sampler call on the logits of a step.
``prompt``  prompts through layers of a hybrid model, logits of the last rows and the stream behind the layers out.
``chat``    short prompts and the decode steps behind them on a hybrid model, logits of every step out.

Hybrid cases with experts put that layer first: the router then reads the embedding, and a rounding in an earlier layer
cannot send a token to another expert.  Sequences of a "ragged" case have lengths from a half to one and a half of the mean.
"""
import json
import math
import tempfile
from pathlib import Path

import torch

from xotorch_support_jetson_b200 import model_config
from xotorch_support_jetson_b200.models import model_cards
from xotorch_support_jetson_b200.shard import Shard
from xotorch_support_jetson_b200.stage import StageRuntime
from xotorch_support_jetson_b200.synth import random_bibevik_state, random_refatar_state

F64 = torch.float64
DEVICE = "cuda"
_STREAM = []
CHUNK = 8192                     # token rows per call while a context is filled
STAGE_LAYERS = {"llama-3.2-1b": 16, "llama-3.2-3b": 7, "llama-3.1-8b": 4, "qwen-2.5-7b": 7}


def listed():
  return [
    # one user's reply on the smallest model, token by token: the call that is made most often
    dict(name="token-1b", kind="stage", model="llama-3.2-1b", layers=16, last=True, seqs=1, context=600, new=1, ragged=False),
    # the same in an eighth of the 8B model, a stage of an 8-GPU ring
    dict(name="token-8b-stage", kind="stage", model="llama-3.1-8b", layers=4, last=False, seqs=1, context=2048, new=1, ragged=False),
    # eight users at once on a quarter of the 3B model
    dict(name="tokens8-3b-stage", kind="stage", model="llama-3.2-3b", layers=7, last=False, seqs=8, context=700, new=1, ragged=True),
    # the serving batch of 32 on the last stage of the 8B model, logits out
    dict(name="tokens32-8b-last", kind="stage", model="llama-3.1-8b", layers=4, last=True, seqs=32, context=2048, new=1, ragged=True),
    # several short questions that arrive together
    dict(name="prompts-3b-short", kind="stage", model="llama-3.2-3b", layers=7, last=False, seqs=5, context=0, new=75, ragged=True),
    # one prompt of a few paragraphs, a model with q/k/v bias and half-split rotation
    dict(name="prompt-qwen-733", kind="stage", model="qwen-2.5-7b", layers=7, last=False, seqs=1, context=0, new=733, ragged=False),
    # a full batch of long prompts
    dict(name="prompts-8b-2048", kind="stage", model="llama-3.1-8b", layers=4, last=False, seqs=4, context=0, new=2048, ragged=False),
    # the sampler as the plugin calls it for the batch of 32: temperature, top-k, noise of the caller's generator
    dict(name="sample-32", kind="sample", rows=32, vocab=128256, temp=0.6, top_k=35, top_p=0.0),
    # a long prompt on each hybrid design: delta rule, then window attention beside HGRN2
    dict(name="prompt-refatar-2048", kind="prompt", model="refatar-1b", picks="0 1", dtype="bfloat16", seqs=1, new=2048, ragged=False),
    # two requests of odd lengths: latent attention with experts, general delta rule, lightning attention
    dict(name="prompts-bibevik-900", kind="prompt", model="bibevik-1b", picks="1 0 2", dtype="bfloat16", seqs=2, new=900, ragged=True),
    # eight chats: a question of a line and the first words of the reply
    dict(name="chat8-bibevik", kind="chat", model="bibevik-1b", picks="1 0 2", dtype="bfloat16", seqs=8, new=24, steps=12),
    # the float32 mode, which serves as the reference for the bf16 one
    dict(name="prompt-refatar-f32", kind="prompt", model="refatar-1b", picks="0 1", dtype="float32", seqs=1, new=300, ragged=False),
  ]


def _log_int(rng, lo, hi):
  return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
  kind = rng.choice(["stage", "stage", "stage", "stage", "sample", "prompt", "chat"])
  if kind == "stage":
    model = rng.choice(sorted(STAGE_LAYERS))
    layers = STAGE_LAYERS[model]
    last = model == "llama-3.2-1b" or rng.random() < 0.3
    if rng.random() < 0.5:      # decode step
      seqs = _log_int(rng, 1, 32)
      case = dict(seqs=seqs, context=_log_int(rng, 16, min(4096, 65536 // seqs)), new=1)
    else:                       # prompts, at times the next portion of prompts that have begun
      rows = _log_int(rng, 9, 4096)
      seqs = _log_int(rng, 1, max(1, min(8, rows // 8)))
      case = dict(seqs=seqs, context=rng.choice([0, 0, 0, rng.randrange(1, 1024)]), new=max(2, rows // seqs))
    return dict(case, kind=kind, model=model, layers=layers, last=last, ragged=rng.random() < 0.5)
  if kind == "sample":
    return dict(kind=kind, rows=_log_int(rng, 1, 64), vocab=rng.choice([32768, 128256, 151936, 152064, rng.randrange(1000, 152064)]),
                temp=rng.choice([0.0, 0.6, 0.6, 1.0]), top_k=rng.choice([0, 1, 35, 35, 200]), top_p=rng.choice([0.0, 0.0, 0.9]))
  model, picks = rng.choice([("refatar-1b", "0 1"), ("bibevik-1b", "1 0 2")])
  dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
  if kind == "chat":
    return dict(kind=kind, model=model, picks=picks, dtype=dtype, seqs=_log_int(rng, 1, 32), new=rng.randrange(1, 48), steps=rng.randrange(4, 16))
  seqs = _log_int(rng, 1, 6)
  return dict(kind=kind, model=model, picks=picks, dtype=dtype, seqs=seqs, new=max(2, _log_int(rng, 9, 2500 if dtype == "bfloat16" else 400) // seqs),
              ragged=rng.random() < 0.5)


# ----------------------------------------------------------------------------- sizes
def _lengths(n, mean, ragged):
  """Lengths of n sequences, the same for every seed."""
  if not ragged or n == 1 or mean <= 1:
    return [mean] * n
  return [max(1, int(mean * (0.5 + i / (n - 1)))) for i in range(n)]


def _batch(case):
  """(context lengths, new rows) of a stage case; a ragged decode step is ragged in its context."""
  if case["new"] == 1:
    return _lengths(case["seqs"], case["context"], case["ragged"]), [1] * case["seqs"]
  return [case["context"]] * case["seqs"], _lengths(case["seqs"], case["new"], case["ragged"])


def _read_config(hf):
  with tempfile.TemporaryDirectory() as td:
    (Path(td) / "config.json").write_text(json.dumps(hf))
    return model_config.load_model_config(Path(td) / "config.json")


def _hybrid_hf(case):
  hf = dict(model_cards[case["model"]]["hf_config"])
  hf["layers"] = [hf["layers"][int(i)] for i in case["picks"].split()]
  return hf


def _hf_dims(hf):
  H = hf["num_attention_heads"]
  return hf["hidden_size"], H, hf["num_key_value_heads"], hf.get("head_dim", hf["hidden_size"] // H), hf["intermediate_size"], hf["vocab_size"]


def _first_layer(case, hf):
  """A range of all layers starts at 0, one that ends the model at its tail, any other sits in the middle."""
  n = hf["num_hidden_layers"]
  return n - case["layers"] if case["last"] else 1


# ----------------------------------------------------------------------------- inputs
def _randn(seed, salt, *shape, std=1.0, dtype=torch.bfloat16):
  g = torch.Generator(device=DEVICE).manual_seed(seed * 1000003 + salt)
  return (torch.randn(*shape, generator=g, device=DEVICE) * std).to(dtype)


def _ids(seed, salt, n, vocab):
  g = torch.Generator(device=DEVICE).manual_seed(seed * 1000003 + salt)
  return torch.randint(0, vocab, (n,), generator=g, device=DEVICE, dtype=torch.int32)


def _layer_weights(hf, seed, l):
  """Weights of one layer by HF leaf name: Linears N(0, 0.02^2), norms 1 + N(0, 0.1^2), Qwen biases N(0, 0.02^2)."""
  D, H, KV, hd, I, _ = _hf_dims(hf)
  shapes = {"self_attn.q_proj.weight": (H * hd, D), "self_attn.k_proj.weight": (KV * hd, D), "self_attn.v_proj.weight": (KV * hd, D),
            "self_attn.o_proj.weight": (D, H * hd), "mlp.gate_proj.weight": (I, D), "mlp.up_proj.weight": (I, D), "mlp.down_proj.weight": (D, I)}
  if hf["model_type"] == "qwen2":
    shapes.update({"self_attn.q_proj.bias": (H * hd,), "self_attn.k_proj.bias": (KV * hd,), "self_attn.v_proj.bias": (KV * hd,)})
  w = {n: _randn(seed, 100 * (l + 1) + j, *s, std=0.02) for j, (n, s) in enumerate(sorted(shapes.items()))}
  for j, n in enumerate(("input_layernorm.weight", "post_attention_layernorm.weight")):
    w[n] = (1.0 + _randn(seed, 100 * (l + 1) + 50 + j, D, std=0.1, dtype=torch.float32)).to(torch.bfloat16)
  return w


def _stage_ends(case, hf, seed):
  """Embedding, final norm and head, where the range holds them."""
  D, V = hf["hidden_size"], hf["vocab_size"]
  w = {}
  if _first_layer(case, hf) == 0 or (case["last"] and hf["tie_word_embeddings"]):
    w["model.embed_tokens.weight"] = _randn(seed, 1, V, D, std=0.02)
  if case["last"]:
    w["model.norm.weight"] = (1.0 + _randn(seed, 2, D, std=0.1, dtype=torch.float32)).to(torch.bfloat16)
    if not hf["tie_word_embeddings"]:
      w["lm_head.weight"] = _randn(seed, 3, V, D, std=0.02)
  return w


def _stage_rows(case, hf, seed, i, n):
  """The n rows of sequence i, context first: token ids of a first stage, hidden rows of any other."""
  if _first_layer(case, hf) == 0:
    return _ids(seed, 20 + i, n, hf["vocab_size"])
  return _randn(seed, 20 + i, n, hf["hidden_size"])


def _sample_inputs(case, seed):
  """Logits as a bf16 head leaves them, and the noise of the caller's generator."""
  logits = (_randn(seed, 5, case["rows"], case["vocab"], std=2.0)).float()
  g = torch.Generator(device=DEVICE).manual_seed(seed * 1000003 + 6)
  return logits, torch.empty_like(logits).exponential_(1, generator=g)


def _hybrid_state(case, hf, seed):
  make = {"refatar-1b": random_refatar_state, "bibevik-1b": random_bibevik_state}[case["model"]]
  return make(hf, seed=seed, device=DEVICE)


# ----------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
  state = {"sample": _prepare_sample, "stage": _prepare_stage}.get(case["kind"], _prepare_hybrid)(case, seed)
  state["kind"] = case["kind"]
  state["stream"] = _serving_stream()
  torch.cuda.synchronize()
  return state


def _serving_stream():
  """The one stream a GPU's engine serves on; not the default one, so that decode steps replay CUDA graphs.  All states share it:
  passes of one program follow one another."""
  if not _STREAM:
    _STREAM.append(torch.cuda.Stream())
  return _STREAM[0]


def _prepare_stage(case, seed):
  hf = model_cards[case["model"]]["hf_config"]
  first, n_layers = _first_layer(case, hf), hf["num_hidden_layers"]
  ctx, new = _batch(case)
  total = [c + q for c, q in zip(ctx, new)]
  st = StageRuntime(Shard(case["model"], first, first + case["layers"] - 1, n_layers), _read_config(hf), max_batch_tokens=max(CHUNK, sum(new)),
                    max_seqs=case["seqs"], max_tokens_per_seq=max(total) + 64)
  weights = _stage_ends(case, hf, seed)
  for l in range(first, first + case["layers"]):
    weights.update({f"model.layers.{l}.{k}": v for k, v in _layer_weights(hf, seed, l).items()})
  st.load_state(weights)
  del weights
  rows = [_stage_rows(case, hf, seed, i, n) for i, n in enumerate(total)]
  key = "tokens" if first == 0 else "hidden"
  for i, c in enumerate(ctx):                 # the context, portion by portion
    for a in range(0, c, CHUNK):
      b = min(c, a + CHUNK)
      st.forward([i], [b - a], [a], **{key: rows[i][a:b].contiguous()})
  call = dict(slot_ids=list(range(case["seqs"])), q_lens=new, positions=ctx, **{key: torch.cat([r[c:] for r, c in zip(rows, ctx)]).contiguous()})
  return dict(st=st, call=call)


def _prepare_sample(case, seed):
  hf = model_cards["llama-3.2-tiny"]["hf_config"]
  st = StageRuntime(Shard("llama-3.2-tiny", 0, hf["num_hidden_layers"] - 1, hf["num_hidden_layers"]), _read_config(hf), max_batch_tokens=64,
                    max_seqs=64, max_tokens_per_seq=64)
  logits, noise = _sample_inputs(case, seed)
  return dict(st=st, logits=logits, call=dict(temp=case["temp"], top_k=case["top_k"], top_p=case["top_p"], q=noise))


def _prepare_hybrid(case, seed):
  hf = _hybrid_hf(case)
  cfg = model_config.hybrid_model_config(hf)
  weights = _hybrid_state(case, hf, seed)
  model_config.resolve_tensor_sizes(cfg, {k: tuple(v.shape) for k, v in weights.items()})
  n, steps = cfg["num_layers"], case.get("steps", 0)
  lens = _lengths(case["seqs"], case["new"], case.get("ragged", False))
  st = StageRuntime(Shard(case["model"], 0, n - 1, n), cfg, max_batch_tokens=sum(lens), max_seqs=case["seqs"], max_tokens_per_seq=max(lens) + steps + 8,
                    dtype=case["dtype"])
  st.load_state(weights)
  ids = [_ids(seed, 20 + i, m + steps, hf["vocab"]) for i, m in enumerate(lens)]
  parts = [(lens, [0] * len(lens), torch.cat([t[:m] for t, m in zip(ids, lens)]).contiguous())]
  for s in range(steps):
    parts.append(([1] * len(lens), [m + s for m in lens], torch.stack([t[m + s] for t, m in zip(ids, lens)]).contiguous()))
  return dict(st=st, slots=list(range(len(lens))), parts=parts, rows=sum(lens), layers=n, width=hf["width"])


def run(state):
  st = state["st"]
  with torch.cuda.stream(state["stream"]):
    if state["kind"] == "sample":
      return st.sample(state["logits"], **state["call"])
    if state["kind"] == "stage":
      return st.forward(**state["call"])
    if state["kind"] == "chat":
      return [st.forward(state["slots"], q, pos, tokens=ids) for q, pos, ids in state["parts"]]
    q, pos, ids = state["parts"][0]
    stream = torch.empty((state["rows"], state["width"]), dtype=torch.float32, device=ids.device)
    logits = st.forward(state["slots"], q, pos, tokens=ids, taps=[None] * (state["layers"] - 1) + [stream])
    return logits, stream


# ----------------------------------------------------------------------------- what a pass cannot do without
def _seen(context, new, window=None):
  """Keys that the new queries of one sequence see, summed over the queries."""
  if window is None:
    return new * context + new * (new + 1) // 2
  return sum(min(window, context + i + 1) for i in range(new))


def _hybrid_layer_work(lc, rows, lens, steps):
  """(weights every token uses, weights read at all, operations beside the Linears) of one hybrid layer; an expert layer multiplies with the chosen
  experts only."""
  m, seen = lc["mixer"], sum(_seen(0, n + steps) for n in lens)
  D = lc["width"]
  if lc["type"] == "delta":
    H, G, dk, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    w, ops = D * (2 * G * dk + 3 * H * dv + 2 * H), 6 * rows * H * dk * dv
  elif lc["type"] == "parallel":
    le, ri = m["left"], m["right"]
    seen = sum(_seen(0, n + steps, le["mask"]["size"]) for n in lens)
    w = D * (le["heads"] * (le["dim"] + 2 * le["vdim"]) + le["kv_heads"] * (le["dim"] + le["vdim"]) + ri["heads"] * (2 * ri["dim"] + 2 * ri["vdim"]))
    ops = 2 * seen * le["heads"] * (le["dim"] + le["vdim"]) + 4 * rows * ri["heads"] * ri["dim"] * ri["vdim"]
  elif lc["type"] == "latent_attention":
    H, dn, dr, dv, R = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
    w, ops = D * (H * (dn + dr) + R + dr + H * dv) + R * H * (dn + dv), 2 * seen * H * (dn + dr + dv)
  elif lc["type"] == "general_delta":
    H, n = m["heads"], m["dim"]
    w, ops = D * (6 * H * n + m.get("rank", 16)) + H * n * m.get("rank", 16), 6 * rows * H * n * n
  else:
    H, n, dv = m["heads"], m["dim"], m["vdim"]
    w, ops = D * H * (2 * n + 3 * dv), 4 * rows * H * n * dv
  f = lc["mlp"]
  if f["kind"] == "dense":
    ff = (3 if "limit" in f else 2) * D * f["ff"]
    return w + ff, w + ff, ops
  rt, F, S = f["router"], f["expert"]["ff"], (f.get("shared") or {"ff": 0})["ff"]
  used = w + D * rt["experts"] + 3 * D * (rt["top"] * F + S)
  return used, used + 3 * D * F * (min(rt["experts"], rows * rt["top"]) - rt["top"]), ops


def work(case):
  if case["kind"] == "sample":
    return {"bytes": 4 * case["rows"] * (case["vocab"] * (1 if case["temp"] <= 0 else 2) + 1), "flops": 0}
  if case["kind"] == "stage":
    hf = model_cards[case["model"]]["hf_config"]
    D, H, KV, hd, I, V = _hf_dims(hf)
    ctx, new = _batch(case)
    rows = sum(new)
    layer = D * hd * (2 * H + 2 * KV) + 3 * D * I
    seen = sum(_seen(c, q) for c, q in zip(ctx, new))
    flops = case["layers"] * (2 * rows * layer + 4 * seen * H * hd)
    kv_rows = sum(ctx) + rows                 # old rows read, new rows written
    nbytes = case["layers"] * 2 * (layer + 2 * kv_rows * KV * hd)
    nbytes += rows * 4 if _first_layer(case, hf) == 0 else rows * D * 2
    if case["last"]:
      flops += 2 * case["seqs"] * V * D
      nbytes += 2 * V * D + 4 * case["seqs"] * V
    else:
      nbytes += rows * D * 2
    return {"bytes": nbytes, "flops": flops}
  hf = _hybrid_hf(case)
  es = 2 if case["dtype"] == "bfloat16" else 4
  lens, steps = _lengths(case["seqs"], case["new"], case.get("ragged", False)), case.get("steps", 0)
  D, V = hf["width"], hf["vocab"]
  rows = sum(lens)
  calls = [rows] + [len(lens)] * steps
  nbytes = flops = 0
  for lc in hf["layers"]:
    used, _, ops = _hybrid_layer_work(dict(lc, width=D), rows + steps * len(lens), lens, steps)
    flops += 2 * used * sum(calls) + ops
    for c in calls:
      nbytes += es * _hybrid_layer_work(dict(lc, width=D), c, lens, steps)[1]
  flops += 2 * V * D * len(lens) * len(calls)
  nbytes += len(calls) * (es * V * D + 4 * V * len(lens)) + (4 * rows * D if not steps else 0)
  return {"bytes": nbytes, "flops": flops}


# ----------------------------------------------------------------------------- accuracy
def tolerance(case):
  if case["kind"] == "sample":
    return "exact"
  # Sums in another order (other split of the Linears, prompts in other portions) move the rows behind 4 to 7 layers by 0.9 to 1.6
  # per cent and the logits of 16 layers by 2.0 per cent (largest single value 0.09): in bf16 every later rounding starts anew.
  if case["kind"] == "stage":
    return {"rel": 0.03, "max": 0.35}
  # The hybrid stream is fp32: 0.6 per cent off the 64-bit result in bf16 (the first tokens of a chat 1.4), 7e-7 in float32.
  return {"rel": 1e-5, "max": 2e-4} if case["dtype"] == "float32" else {"rel": 0.025, "max": 0.4}


# ----------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
  if case["kind"] == "sample":
    return _exact_sample(case, seed)
  if case["kind"] == "stage":
    if work(case)["flops"] + _context_flops(case) > 3e14:
      return None
    return _exact_stage(case, seed)
  return _exact_hybrid(case, seed)


def _rms(x, eps):
  return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
  return x * torch.sigmoid(x)


def _exact_sample(case, seed):
  """torchtune's sampling rule with a nucleus: keep the top_k largest, of those the most likely that reach top_p together,
  then the largest probability over noise."""
  logits, noise = (t.to(F64) for t in _sample_inputs(case, seed))
  if case["temp"] <= 0:
    return logits.argmax(-1).to(torch.int32)
  z = logits / max(case["temp"], 1e-5)
  if 0 < case["top_k"] < case["vocab"]:
    z = torch.where(z < z.topk(case["top_k"], dim=-1).values[:, -1:], -math.inf, z)
  p = torch.softmax(z, dim=-1)
  if 0 < case["top_p"] < 1:
    s = p.sort(dim=-1, descending=True).values
    cut = s.gather(1, (s.cumsum(-1) < case["top_p"]).sum(-1, keepdim=True).clamp(max=case["vocab"] - 1))
    p = torch.where(p < cut, 0.0, p)
  return (p / noise).argmax(-1).to(torch.int32)


def _context_flops(case):
  hf = model_cards[case["model"]]["hf_config"]
  D, H, KV, hd, I, _ = _hf_dims(hf)
  return case["layers"] * sum(_batch(case)[0]) * 2 * (D * hd * (2 * H + 2 * KV) + 3 * D * I)


def _rope_angles(hf, n, hd):
  """(cos, sin) [n, hd/2] of the model's table, which is kept in bf16 (Llama: frequencies rescaled by 32 as the reference does)."""
  f = 1.0 / (hf["rope_theta"] ** (torch.arange(0, hd, 2).float() / hd))
  if hf["model_type"] == "llama":
    out = []
    for x in f:
      wave = 2 * math.pi / x
      s = (8192 / wave - 1) / 3
      out.append(x if wave < 8192 / 4 else x / 32 if wave > 8192 else (1 - s) * x / 32 + s * x)
    f = torch.tensor(out, dtype=f.dtype)
  a = torch.arange(n).float()[:, None] * f[None, :]
  return torch.cos(a).to(torch.bfloat16).to(DEVICE, F64), torch.sin(a).to(torch.bfloat16).to(DEVICE, F64)


def _causal(q, k, v, scale, window=None, keep=0):
  """Softmax attention of one sequence: q [n, H, dk] are the last n positions, k [m, G, dk], v [m, G, dv]."""
  n, H, m, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
  i, j = torch.arange(m - n, m, device=q.device)[:, None], torch.arange(m, device=q.device)[None, :]
  hide = j > i if window is None else (j > i) | ((i - j >= window) & (j >= keep))
  out = torch.empty(n, H, v.shape[2], dtype=q.dtype, device=q.device)
  for g in range(G):
    h = slice(g * (H // G), (g + 1) * (H // G))
    s = torch.einsum("nhd,md->hnm", q[:, h], k[:, g]).mul_(scale).masked_fill_(hide, -math.inf)
    out[:, h] = torch.einsum("hnm,md->nhd", torch.softmax(s, dim=-1), v[:, g])
  return out


def _by_rows(f, x, rows=8192):
  return torch.cat([f(x[a:a + rows]) for a in range(0, x.shape[0], rows)])


def _exact_stage(case, seed):
  hf = model_cards[case["model"]]["hf_config"]
  D, H, KV, hd, _, _ = _hf_dims(hf)
  first, eps = _first_layer(case, hf), hf["rms_norm_eps"]
  ctx, new = _batch(case)
  total = [c + q for c, q in zip(ctx, new)]
  ends = {k: v.to(F64) for k, v in _stage_ends(case, hf, seed).items()}
  rows = [_stage_rows(case, hf, seed, i, n) for i, n in enumerate(total)]
  x = torch.cat([ends["model.embed_tokens.weight"][r.long()] if first == 0 else r.to(F64) for r in rows])
  cos, sin = _rope_angles(hf, max(total), hd)
  start = [sum(total[:i]) for i in range(len(total))]
  new_rows = torch.cat([torch.arange(s + c, s + n) for s, c, n in zip(start, ctx, total)]).to(DEVICE)

  def turn(t, pos):             # pairs (i, i + hd/2): the layout of HF weights
    a, b, c, s = t[..., :hd // 2], t[..., hd // 2:], cos[pos][:, None], sin[pos][:, None]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)

  for l in range(first, first + case["layers"]):
    w = {k: v.to(F64) for k, v in _layer_weights(hf, seed, l).items()}
    final = l + 1 == first + case["layers"]   # of the last layer only the new rows are wanted

    def proj(t, name):
      y = t @ w[f"self_attn.{name}_proj.weight"].T
      return y + w[f"self_attn.{name}_proj.bias"] if f"self_attn.{name}_proj.bias" in w else y

    h = _rms(x, eps) * w["input_layernorm.weight"]
    att = []
    for s, c, n in zip(start, ctx, total):
      t, q0 = h[s:s + n], c if final else 0
      pos = torch.arange(n, device=DEVICE)
      k, v = turn(proj(t, "k").view(n, KV, hd), pos), proj(t, "v").view(n, KV, hd)
      q = turn(proj(t[q0:], "q").view(n - q0, H, hd), pos[q0:])
      att.append(_causal(q, k, v, hd ** -0.5).reshape(n - q0, H * hd) @ w["self_attn.o_proj.weight"].T)
    x = (x[new_rows] if final else x) + torch.cat(att)
    gate, up, down = (w[f"mlp.{n}_proj.weight"] for n in ("gate", "up", "down"))
    x = x + _by_rows(lambda t: (_silu(t @ gate.T) * (t @ up.T)) @ down.T, _rms(x, eps) * w["post_attention_layernorm.weight"])
  if not case["last"]:
    return x
  at = torch.tensor([sum(new[:i + 1]) - 1 for i in range(len(new))], device=DEVICE)
  head = ends["lm_head.weight" if "lm_head.weight" in ends else "model.embed_tokens.weight"]
  return (_rms(x[at], eps) * ends["model.norm.weight"]) @ head.T


def _scan(step, state, n):
  """Outputs of n steps of a recurrence: step(state, t) -> (state, output)."""
  out = []
  for t in range(n):
    state, o = step(state, t)
    out.append(o)
  return torch.stack(out)


def _taps(h, w):
  """Causal filter per channel; the last column of w weighs the current row."""
  out = torch.zeros_like(h)
  for j in range(w.shape[1]):
    back = w.shape[1] - 1 - j
    if back < h.shape[0]:
      out[back:] += h[:h.shape[0] - back] * w[:, j]
  return out


def _delta_layer(w, m, h, eps):
  T, (H, G, dk, dv) = h.shape[0], (m[k] for k in ("heads", "kv_heads", "dim", "vdim"))
  q, k, v = (_silu(_taps(h @ w[n].T, w[n + ".conv"])).view(T, c, d) for n, c, d in (("q", G, dk), ("k", G, dk), ("v", H, dv)))
  q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
  q, k = (t.repeat_interleave(H // G, 1) for t in (q * dk ** -0.5, k))
  beta = torch.sigmoid(h @ w["b"].T)
  keep = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(h @ w["a"].T + w["dt_bias"]))

  def step(S, t):
    S = keep[t][:, None, None] * S
    S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - (k[t][:, None] @ S)[:, 0]))[:, None]
    return S, (q[t][:, None] @ S)[:, 0]

  o = _scan(step, torch.zeros(H, dk, dv, dtype=F64, device=h.device), T)
  return (_rms(o, eps) * w["norm"] * _silu(h @ w["g"].T).view(T, H, dv)).reshape(T, H * dv) @ w["o"].T


def _parallel_layer(w, m, h, eps):
  T, le, ri = h.shape[0], m["left"], m["right"]
  q, k, v = ((h @ w[f"left.{n}"].T + w[f"left.{n}.b"]).view(T, c, d) for n, c, d in
             (("q", le["heads"], le["dim"]), ("k", le["kv_heads"], le["dim"]), ("v", le["kv_heads"], le["vdim"])))
  o = _causal(q, k, v, le["scale"], le["mask"]["size"], le["mask"]["keep_first"]).reshape(T, -1)
  left = (o * torch.sigmoid(h @ w["left.g"].T)) @ w["left.o"].T
  H, dk, dv = ri["heads"], ri["dim"], ri["vdim"]
  q, v = _silu(h @ w["right.q"].T).view(T, H, dk), (h @ w["right.v"].T).view(T, H, dv)
  f = (w["right.lower"] + (1 - w["right.lower"]) * torch.sigmoid(h @ w["right.f"].T + w["right.f.b"])).view(T, H, dk)

  def step(S, t):
    S = f[t][:, :, None] * S + (1 - f[t])[:, :, None] * v[t][:, None]
    return S, (q[t][:, None] @ S)[:, 0]

  o = _scan(step, torch.zeros(H, dk, dv, dtype=F64, device=h.device), T)
  return m["left_scale"] * left + m["right_scale"] * ((_rms(o, eps) * w["right.norm"]).reshape(T, H * dv) @ w["right.o"].T)


def _latent_layer(w, m, h, eps):
  T, (H, dn, dr, dv, R) = h.shape[0], (m[k] for k in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
  turned = m["rot"]["dims"]
  a = torch.arange(T, device=h.device, dtype=F64)[:, None] * m["rot"]["base"] ** (-2.0 * torch.arange(turned // 2, device=h.device, dtype=F64) / turned)

  def turn(t):                  # neighbouring entries are a pair
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    out = t.clone()
    out[..., 0:turned:2] = t[..., 0:turned:2] * c - t[..., 1:turned:2] * s
    out[..., 1:turned:2] = t[..., 1:turned:2] * c + t[..., 0:turned:2] * s
    return out

  q, down = (h @ w["q"].T).view(T, H, dn + dr), h @ w["dkv"].T
  c = _rms(down[:, :R], eps) * w["dkv.norm"]
  q = torch.cat([q[..., :dn], turn(q[..., dn:])], dim=-1)
  k = torch.cat([(c @ w["uk"].T).view(T, H, dn), turn(down[:, None, R:]).expand(T, H, dr)], dim=-1)
  return _causal(q, k, (c @ w["uv"].T).view(T, H, dv), m["scale"]).reshape(T, H * dv) @ w["o"].T


def _general_delta_layer(w, m, h, eps):
  T, H, n = h.shape[0], m["heads"], m["dim"]
  r, k, v = ((h @ w[x].T).view(T, H, n) for x in ("r", "k", "v"))
  d = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(h @ w["w1"].T) @ w["w2"].T + w["w0"])).view(T, H, n)
  u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
  au = torch.sigmoid(h @ w["a"].T + w["a.b"]).view(T, H, n) * u

  def step(S, t):
    S = d[t][:, :, None] * S - au[t][:, :, None] * (u[t][:, None] @ S) + k[t][:, :, None] * v[t][:, None]
    return S, (r[t][:, None] @ S)[:, 0]

  o = _scan(step, torch.zeros(H, n, n, dtype=F64, device=h.device), T)
  return (_rms(o, eps).reshape(T, H * n) * w["norm"] * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def _lightning_layer(w, m, h, eps):
  T, H, n, dv = h.shape[0], m["heads"], m["dim"], m["vdim"]
  q, k, v = (_silu(h @ w[x].T).view(T, H, d) for x, d in (("q", n), ("k", n), ("v", dv)))
  decay = torch.tensor(m["decay"], dtype=F64, device=h.device)[:, None, None]

  def step(S, t):
    S = decay * S + k[t][:, :, None] * v[t][:, None]
    return S, (q[t][:, None] @ S)[:, 0]

  o = _scan(step, torch.zeros(H, n, dv, dtype=F64, device=h.device), T)
  return (_rms(o.reshape(T, H * dv), eps) * w["norm"] * torch.sigmoid(h @ w["g"].T)) @ w["o"].T


def _glu(w, p, h, limit):
  bias = lambda n: w.get(p + n + ".b", 0.0)  # noqa: E731
  g = torch.clamp(h @ w[p + "gate"].T + bias("gate"), max=limit)
  u = torch.clamp(h @ w[p + "up"].T + bias("up"), min=-limit, max=limit)
  return (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w[p + "down"].T + bias("down")


def _feed_forward(w, f, h, rounded):
  """rounded: the rows as the serving type holds them, which is what the router reads: a choice between two experts that are
  nearly equal follows them."""
  if f["kind"] == "dense":
    return _glu(w, "", h, f["limit"]) if "limit" in f else torch.relu(h @ w["up"].T) ** 2 @ w["down"].T
  rt = f["router"]
  s = torch.sigmoid(rounded @ w["router"].T)
  T, E, n = s.shape[0], rt["experts"], rt["groups"]["count"]
  worth = s.view(T, n, E // n).topk(min(2, E // n), dim=-1).values.sum(-1)
  open_ = torch.zeros(T, n, dtype=torch.bool, device=h.device).scatter_(1, worth.topk(rt["groups"]["keep"], dim=-1).indices, True)
  pick = s.masked_fill(~open_.repeat_interleave(E // n, 1), -1.0).topk(rt["top"], dim=-1).indices
  weight = torch.zeros_like(s).scatter_(1, pick, s.gather(1, pick) * rt["scale"])
  y = _glu(w, "shared.", h, f["shared"]["limit"]) if f.get("shared") else 0.0
  for e in range(E):
    y = y + weight[:, e:e + 1] * _glu(w, f"e{e}.", h, f["expert"]["limit"])
  return y


_MIXERS = {"delta": _delta_layer, "parallel": _parallel_layer, "latent_attention": _latent_layer, "general_delta": _general_delta_layer,
           "lightning": _lightning_layer}


def _exact_sequence(hf, w, ids, serving):
  """Stream behind the layers and normed stream of one sequence from its first token on."""
  eps, tok = hf["norm"]["eps"], ids.long()
  sub = lambda p: {k[len(p):]: v for k, v in w.items() if k.startswith(p)}  # noqa: E731
  refatar = hf["architecture"] == "Refatar"
  x = w["embed"][tok] * (1.0 if refatar else hf["embedding"]["scale"])
  for i, lc in enumerate(hf["layers"]):
    p, mix = f"l{i}.", lambda t: _MIXERS[lc["type"]](sub(f"l{i}.mix."), lc["mixer"], t, eps)  # noqa: B023
    if refatar:                 # each sublayer: norm, filter, branch, norm; then the token's own input
      h = _rms(x, eps) * (1 + w[p + "norm1"])
      x = x + _rms(mix(h + _taps(h, w[p + "canon1"])), eps) * (1 + w[p + "norm1b"])
      h = _rms(x, eps) * (1 + w[p + "norm2"])
      x = x + _rms(_feed_forward(sub(p + "mlp."), lc["mlp"], h + _taps(h, w[p + "canon2"]), None), eps) * (1 + w[p + "norm2b"])
      n = hf["token_side"]["dim"]
      z = torch.nn.functional.gelu(x @ w[p + "side.gate"].T, approximate="tanh") * w["side.embed"][tok][:, i * n:(i + 1) * n]
      x = x + _rms(z @ w[p + "side.proj"].T, eps) * w[p + "side.norm"]
    else:                       # both sublayers read one norm
      h = _rms(x, eps) * w[p + "norm1"]
      x = x + mix(h) + _feed_forward(sub(p + "mlp."), lc["mlp"], h, h.to(serving).to(F64))
  g = w["final.norm"]
  return x, _rms(x, eps) * (1 + g if refatar else g)


def _exact_hybrid(case, seed):
  hf = _hybrid_hf(case)
  w = {k: v.to(F64) for k, v in _hybrid_state(case, hf, seed).items()}
  lens, steps = _lengths(case["seqs"], case["new"], case.get("ragged", False)), case.get("steps", 0)
  cap = hf.get("logit_softcap")
  streams, heads = [], []
  for i, n in enumerate(lens):
    x, h = _exact_sequence(hf, w, _ids(seed, 20 + i, n + steps, hf["vocab"]), getattr(torch, case["dtype"]))
    z = h[n - 1:] @ w["head"].T
    streams.append(x)
    heads.append(cap * torch.tanh(z / cap) if cap else z)
  if steps:
    return [torch.stack([z[s] for z in heads]) for s in range(steps + 1)]
  return torch.cat(heads), torch.cat(streams)
