"""A second backward pass over a kept graph gives the gradients of the first: what the gated products save is
overwritten only where no other pass reads it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _parameter(g, *shape, buffer):
  p = torch.nn.Parameter((torch.randn(*shape, device="cuda", generator=g) * shape[-2] ** -0.5).bfloat16().float())
  p.bf16 = p.detach().bfloat16()
  if buffer:
    p.main_grad = torch.full_like(p, 7.0)
    p.grad_ready = False
  return p


def _setup(kind, buffer):
  """(input, parameters, function of the input)"""
  from t5x_b200.models.t5 import layers
  from t5x_b200.ops import blocks
  from t5x_b200.ops import functional as F
  g = torch.Generator(device="cuda").manual_seed(5)
  if kind == "experts":
    x = torch.randn(3, 40, 64, device="cuda", generator=g).bfloat16()
    w = [_parameter(g, 3, 64, 136, buffer=buffer) for _ in range(2)]
    return x, w, lambda x: F.batched_gated_mlp_in(x, *w)
  x = torch.randn(2, 40, 64, device="cuda", generator=g).bfloat16()
  if kind.startswith("dense"):
    w = [_parameter(g, 64, 136, buffer=buffer) for _ in range(2)]
    return x, w, lambda x: F.gated_gelu_mlp_in(x, *w)
  norm = layers.LayerNorm(64, dtype="bfloat16", device="cuda")
  mlp = layers.MlpBlock(64, 136, ("gelu", "linear"), 0.0, "bfloat16", device="cuda")
  w = [mlp.wi_0.kernel, mlp.wi_1.kernel, mlp.wo.kernel, norm.scale]
  for p in w:
    p.bf16, p.main_grad, p.grad_ready = p.detach().bfloat16(), torch.full_like(p, 7.0), False

  def call(x):
    y = blocks.gated_mlp(x, norm, mlp, layers.LayerNorm, layers.MlpBlock, layers.DenseGeneral)
    assert y is not None
    return y

  return x, w, call


@pytest.mark.parametrize("kind,buffer", [("experts", False), ("experts", True), ("dense", False), ("dense", True),
                                         ("dense_general", True), ("block", True)])
def test_second_backward(kind, buffer, monkeypatch):
  from t5x_b200.ops import native
  if kind == "dense_general":  # the path for calls that the compiled one does not cover
    monkeypatch.setattr(native, "host", lambda: None)
  x, params, call = _setup(kind, buffer)
  x.requires_grad_()
  y = call(x)
  dy = torch.randn(y.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(6)).bfloat16()

  def grads(keep):
    x.grad = None
    for p in params:
      p.grad, p.grad_ready = None, False
    y.backward(dy, retain_graph=keep)
    return [x.grad] + [p.main_grad.clone() if buffer else p.grad for p in params]

  first, second, last = grads(True), grads(True), grads(False)
  for a, b, c in zip(first, second, last):
    assert bool(a.any())
    # (the norm's scale gets its gradient by atomic adds: fp32 sums of 80 rows in another order)
    assert float((a - b).norm() / a.norm()) < 80 * 2.0 ** -24 and float((a - c).norm() / a.norm()) < 80 * 2.0 ** -24
