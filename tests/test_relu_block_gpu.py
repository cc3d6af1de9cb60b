"""ReLU and its gradient inside the products around it: against float64 at the edges of tiles, and a model whose MLPs
take them against the same op by op."""
import pytest
import torch

from test_blocks_gpu import _model, _pass, _tokens

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (257, 264, 72), (1000, 1000, 128), (2050, 3072, 768)])
def test_product_with_relu(m, n, k):
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(m)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
  a, w, act = rnd(m, k), rnd(k, n), rnd(m, n).relu()
  act[::3, ::5] = 0.0
  act[1, 1:40] = float("nan")
  a[0, 0] = float("nan")
  for positive in (None, act):
    out = torch.full((m, n), 7.0, device="cuda").bfloat16()
    native._check(native.lib().t5x_gemm_relu(a.data_ptr(), w.data_ptr(), out.data_ptr(), native.ptr(positive), m, n,
                                             k, k, n, n, n, 1, native.stream_ptr()), "gemm_relu")
    native.check_status()
    want = a.double() @ w.double()
    want = want.relu() if positive is None else want * ~(positive <= 0)
    if positive is None:
      assert bool(out[0].isnan().all())  # as torch's
    else:
      assert not bool(out[positive == 0].any())
    assert float((out[1:].double() - want[1:]).norm() / want[1:].norm()) < 2.0 ** -8  # one rounding to bf16


def test_same_as_op_by_op(monkeypatch):
  from t5x_b200.ops import blocks
  enc, dec = _tokens(40, 128, 1), _tokens(40, 130, 2)
  results, taken = [], []
  for on in (True, False):
    def call(*a, _fn=blocks.relu_mlp, **k):
      y = _fn(*a, **k) if on else None
      taken.append(y is not None)
      return y
    with monkeypatch.context() as m:
      m.setattr(blocks, "relu_mlp", call)
      results.append(_pass(_model(act=("relu",), mlp=1024), enc, dec))
  assert taken == [True] * 12 + [False] * 12  # four layers, two passes and one without gradients
  (h1, y1, g1), (h2, y2, g2) = results
  assert torch.equal(h1, h2) and torch.equal(y1, y2)
  assert [n for n in g1 if g1[n] is None] == [n for n in g2 if g2[n] is None]
  for n in (n for n in g1 if g1[n] is not None):  # up to the order of atomic adds
    assert float((g1[n].float() - g2[n].float()).norm() / g2[n].float().norm()) < 1e-3, n


def test_pair_mode_between_the_passes():
  """The forward pass through the products with ReLU, the backward pass after CTA pairs were switched off."""
  from t5x_b200.ops import blocks, native
  grads = []
  for mode in (1, 0):
    module = _model(act=("relu",), mlp=1024)
    mlp, norm = module.encoder.layers_0.mlp, module.encoder.layers_0.pre_mlp_layer_norm
    for p in module.parameters():
      p.grad_ready = False
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(5000, 256, device="cuda", generator=g).bfloat16().requires_grad_()
    dy = torch.randn(5000, 256, device="cuda", generator=g).bfloat16()
    y = blocks.relu_mlp(x, norm, mlp, type(norm), type(mlp), type(mlp.wi))
    assert y is not None
    native.gemm_set_pair_mode(mode)
    try:
      y.backward(dy)
    finally:
      native.gemm_set_pair_mode(1)
    native.check_status()
    grads.append([x.grad] + [p.main_grad for p in (mlp.wi.kernel, mlp.wo.kernel, norm.scale)])
  # dg is rounded to bf16 either way; other tiles add in another order
  for a, b in zip(*grads):
    assert float((a.float() - b.float()).norm() / b.float().norm()) < 2.0 ** -8
