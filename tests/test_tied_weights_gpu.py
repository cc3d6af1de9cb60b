"""Projections that share one weight (and so one gradient buffer): the gradient is the sum of both, on the
first pass and on passes that add to it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _parameter(g, *shape):
  p = torch.nn.Parameter((torch.randn(*shape, device="cuda", generator=g) * shape[0] ** -0.5).bfloat16().float())
  p.bf16, p.main_grad, p.grad_ready = p.detach().bfloat16(), torch.full_like(p, 7.0), False
  return p


@pytest.mark.parametrize("rows,k,n", [(40, 64, 64), (700, 256, 512)])
@pytest.mark.parametrize("kind", ["pair", "first_and_last", "gated"])
def test_tied_products(kind, rows, k, n):
  """Against float64. A gradient adds 2 passes x 2 products of `rows` terms in fp32; what goes into them
  has been rounded to bf16 (the gated product's pre-activations and their gradients: 3 x 2^-8)."""
  from t5x_b200.ops import functional as F
  g = torch.Generator(device="cuda").manual_seed(rows)
  a, b = _parameter(g, k, n), _parameter(g, k, n)
  weights = {"pair": [a, a], "first_and_last": [a, b, a], "gated": [a, a]}[kind]
  x = torch.randn(rows, k, device="cuda", generator=g).bfloat16()
  dys = [torch.randn(rows, n, device="cuda", generator=g).bfloat16() for _ in weights]
  xd = x.double()
  ref = {p: p.detach().double().requires_grad_() for p in (a, b)}
  for _ in range(2):
    if kind == "gated":
      F.gated_gelu_mlp_in(x, *weights).backward(dys[0])
      h = xd @ ref[a]
      (torch.nn.functional.gelu(h, approximate="tanh") * h).backward(dys[0].double())
    else:
      outs = F.multi_linear(x, weights)
      torch.autograd.backward(outs, dys)
      torch.autograd.backward([xd @ ref[w] for w in weights], [d.double() for d in dys])
  for p in set(weights):
    err = float((p.main_grad.double() - ref[p].grad).norm() / ref[p].grad.norm())
    assert err < (3 * 2.0 ** -8 if kind == "gated" else 4 * rows * 2.0 ** -24)


def test_tied_key_and_value_of_a_layer():
  """The compiled block against the same layer op by op, over two passes that add up."""
  from t5x_b200.models.t5 import network
  grads = []
  for compiled in (True, False):
    torch.manual_seed(0)
    cfg = network.T5Config(vocab_size=512, dtype="bfloat16", emb_dim=256, num_heads=4, head_dim=64,
                           num_encoder_layers=1, num_decoder_layers=1, mlp_dim=512,
                           mlp_activations=("gelu", "linear"), dropout_rate=0.0)
    layer = network.EncoderLayer(cfg, device="cuda")
    layer.attention.value.kernel = layer.attention.key.kernel
    for p in layer.parameters():
      p.bf16, p.main_grad, p.grad_ready = p.detach().bfloat16(), torch.full_like(p, 7.0), False
    x = torch.randn(3, 50, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).bfloat16()
    if not compiled:
      layer.attention.register_forward_hook(lambda *a: None)  # (a module with hooks runs op by op)
    y = [layer(x, bias_table=None, key_mask=None) for _ in range(2)]
    for t in y:
      t.float().square().sum().backward()
    grads.append(layer.attention.key.kernel.main_grad)
  assert float((grads[0] - grads[1]).norm() / grads[1].norm()) < 2 ** -8
