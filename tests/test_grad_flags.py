"""The gradient-buffer flags of weights around the compiled backward calls: a call that raises or
declines leaves them as they were, one that is covered leaves them set. The compiled path is a
stand-in."""
import types

import pytest
import torch

from t5x_b200.ops import functional as F
from t5x_b200.ops import native


def _weights(n):
  out = []
  for i in range(n):
    w = torch.nn.Parameter(torch.zeros(8, 8))
    w.bf16, w.main_grad, w.grad_ready = w.detach().bfloat16(), torch.zeros(8, 8), i == 1
    out.append(w)
  return out


def _host(result):
  def call(*args):
    if isinstance(result, Exception):
      raise result
    return result
  return types.SimpleNamespace(multi_linear_bwd=call, gated_in_bwd=call)


def _flags(ws):
  return [w.grad_ready for w in ws]


@pytest.mark.parametrize("twice", [False, True])
def test_projections(monkeypatch, twice):
  ws = _weights(3)
  if twice:
    ws[2] = ws[0]
  x, dys, needs = torch.zeros(4, 8), [torch.zeros(4, 8)] * 3, (True, True, True, True)
  before = _flags(ws)
  monkeypatch.setattr(native, "host", lambda: _host(torch.OutOfMemoryError("no room")))
  with pytest.raises(torch.OutOfMemoryError):
    F._host_linear_bwd(dys, x, ws, needs)
  assert _flags(ws) == before
  monkeypatch.setattr(native, "host", lambda: _host(None))
  assert F._host_linear_bwd(dys, x, ws, needs) == (False, None) and _flags(ws) == before
  monkeypatch.setattr(native, "host", lambda: _host((x,)))
  assert F._host_linear_bwd(dys, x, ws, needs) == (True, x) and all(_flags(ws))


def test_gated_projections(monkeypatch):
  ws = _weights(2)
  ctx = types.SimpleNamespace(saved_tensors=(torch.zeros(4, 8), *ws, torch.zeros(4, 16)),
                              needs_input_grad=(True, True, True))
  monkeypatch.setattr(native, "host", lambda: _host(torch.OutOfMemoryError("no room")))
  with pytest.raises(torch.OutOfMemoryError):
    F._GatedGeluMlpInFn.backward(ctx, torch.zeros(4, 8))
  assert _flags(ws) == [False, True]
  monkeypatch.setattr(native, "host", lambda: _host((None,)))
  F._GatedGeluMlpInFn.backward(ctx, torch.zeros(4, 8))
  assert all(_flags(ws))
