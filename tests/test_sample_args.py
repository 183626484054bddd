"""StageRuntime.sample hands bare addresses to the library, which reads n * vocab numbers behind them: buffers that hold less, or other things than
it takes them for, have to be refused on the host.  (No GPU: the library is a stand-in that records its calls.)"""
from types import SimpleNamespace

import pytest
import torch

VOCAB = 64


class OnGpu(torch.Tensor):
  """A host tensor that says it is a CUDA one."""
  is_cuda = property(lambda self: True)


def gpu(*shape, dtype=torch.float32):
  return torch.zeros(*shape, dtype=dtype).as_subclass(OnGpu)


@pytest.fixture
def stage(monkeypatch):
  from xotorch_support_jetson_b200.stage import StageRuntime
  st = StageRuntime.__new__(StageRuntime)
  st.calls = []
  st._h, st.vocab, st.device = None, VOCAB, torch.device("cpu")
  st.lib = SimpleNamespace(xb_sample=lambda *a: st.calls.append(a) or 0)
  monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: SimpleNamespace(cuda_stream=0))
  return st


@pytest.mark.parametrize("logits,q,out", [
  ((3, VOCAB - 1), None, None), ((VOCAB,), None, None),                                                  # rows shorter than the vocabulary, a row without its batch
  ((3, VOCAB), gpu(3, VOCAB - 1), None), ((3, VOCAB), gpu(2, VOCAB), None),                              # too little noise
  ((3, VOCAB), gpu(3, VOCAB, dtype=torch.float64), None), ((3, VOCAB), gpu(VOCAB, 3).t(), None),         # noise of another type, of another layout
  ((3, VOCAB), torch.zeros(3, VOCAB, device="meta"), None),                                              # noise on another device
  ((3, VOCAB), None, gpu(2, dtype=torch.int32)), ((3, VOCAB), None, gpu(3, dtype=torch.int64)), ((3, VOCAB), None, gpu(6, dtype=torch.int32)[::2]),   # places for the tokens
])
def test_buffers_that_do_not_hold_the_rows_are_refused(stage, logits, q, out):
  with pytest.raises(ValueError):
    stage.sample(gpu(*logits), temp=0.6, q=q, out=out)
  assert stage.calls == []


@pytest.mark.parametrize("temp", [0.0, 0.6])
def test_buffers_that_hold_the_rows_are_taken(stage, temp):
  tok = stage.sample(gpu(3, VOCAB), temp=temp, q=gpu(3, VOCAB))
  assert tok.shape == (3,) and tok.dtype == torch.int32
  tok = gpu(5, dtype=torch.int32)
  assert stage.sample(gpu(3, VOCAB), temp=temp, out=tok[1:4]).data_ptr() == tok[1:].data_ptr()
  assert len(stage.calls) == 2 and [c[2] for c in stage.calls] == [3, 3]
