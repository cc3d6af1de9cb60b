"""The experts' gated MLP in batched launches, and the router's weight gradient, at tile edges."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e,n,d,ff", [(1, 1, 64, 64), (3, 130, 72, 136), (8, 320, 256, 512), (2, 700, 768, 2048)])
@pytest.mark.parametrize("buffers", [True, False])
def test_gated_experts(e, n, d, ff, buffers):
  """Against float64: forward one rounding to bf16 after fp32 sums (2^-9, a factor of two for the
  sums and the activation); gradients pass two more bf16 tensors (3 x 2^-8 of the norm)."""
  from t5x_b200.ops import functional as F
  g = torch.Generator(device="cuda").manual_seed(n)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  x = rnd(e, n, d).bfloat16().requires_grad_()
  w = [torch.nn.Parameter((rnd(e, d, ff) * d ** -0.5).bfloat16().float()) for _ in range(2)]
  for p in w:
    p.bf16 = p.detach().bfloat16()
    if buffers:
      p.main_grad = torch.full_like(p, 9.0)
      p.grad_ready = False
  dy = rnd(e, n, ff).bfloat16()
  y = F.batched_gated_mlp_in(x, *w)
  y.backward(dy)
  xd, wd = x.detach().double().requires_grad_(), [p.detach().double().requires_grad_() for p in w]
  want = torch.nn.functional.gelu(xd @ wd[0], approximate="tanh") * (xd @ wd[1])
  want.backward(dy.double())
  assert float((y.double() - want).abs().max() / want.abs().max()) < 2 * 2.0 ** -9
  for got, ref in [(x.grad, xd.grad)] + [(p.main_grad if buffers else p.grad, q.grad) for p, q in zip(w, wd)]:
    assert float((got.double() - ref).norm() / ref.norm()) < 3 * 2.0 ** -8


@pytest.mark.parametrize("t,d,e", [(1, 64, 2), (127, 250, 8), (128, 258, 9), (129, 1024, 16), (5000, 768, 8),
                                   (300, 33, 64), (300001, 64, 2), (90001, 701, 3), (200001, 700, 2)])
def test_router_weight_gradient(t, d, e):
  """fp32 sums over the tokens: below t 2^-24 of the sum of magnitudes, whatever the order."""
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(t)
  x = torch.randn(t, d, device="cuda", generator=g).bfloat16()
  w = torch.randn(d, e, device="cuda", generator=g) * d ** -0.5
  k, capacity = 1, max(4, t)
  fwd = native.moe_router_fwd(x, w, k, capacity)
  dgate = torch.randn(t, k, device="cuda", generator=g)
  coef = torch.zeros(2, device="cuda")
  dx, dw = native.moe_router_bwd(x, w, k, capacity, fwd, dgate, coef)
  native.check_status()
  p = torch.softmax(x.double() @ w.double(), -1)
  onehot = torch.nn.functional.one_hot(fwd["index"].long()[:, 0], e).double()
  chosen = (p * onehot).sum(-1, keepdim=True)
  dl = dgate.double() * chosen * (onehot - p)
  ref, size = x.double().t() @ dl, x.double().abs().t() @ dl.abs()
  # the logits' gradients themselves are fp32 values of a few operations (2^-18 of a magnitude)
  assert bool(((dw.double() - ref).abs() <= (t * 2.0 ** -24 + 2.0 ** -15) * size + 1e-12).all())
  again = native.moe_router_bwd(x, w, k, capacity, fwd, dgate, coef)[1]
  assert torch.equal(dw, again)


def test_gated_gelu_far_from_zero():
  """gelu itself, from -8 to 8, with a gate of 1. On the negative side 1 + tanh is a difference of two numbers
  near 1, and the fast `tanhf` is good to 2^-11 of its value: beside the rounding to bf16 (half a unit of its
  8 bits, 2^-8 of the result) that leaves |x| / 2 times as much, for the gradient times the inner derivative
  and a square more."""
  from t5x_b200.ops import functional as F
  from t5x_b200.ops import native
  x = torch.linspace(-8, 8, 1 << 15, device="cuda").bfloat16().unique()
  x = x[:x.numel() // 248 * 248]
  rows = torch.zeros(x.numel() // 62, 64, device="cuda")
  rows[:, :62], rows[:, 63] = x.view(-1, 62), 1
  w0, w1 = torch.eye(64, device="cuda"), torch.zeros(64, 64, device="cuda")
  w0[63], w1[63] = 0, 1
  with torch.no_grad():
    got = F.batched_gated_mlp_in(rows.bfloat16()[None], w0[None], w1[None])[0, :, :62].reshape(-1)
  xd = x.double().requires_grad_()
  want = torch.nn.functional.gelu(xd, approximate="tanh")
  slope, = torch.autograd.grad(want.sum(), xd)
  want, xd = want.detach(), xd.detach()
  tanh_part = 2.0 ** -11 * (1 + xd.abs() / 2)
  assert bool(((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + tanh_part).all())
  h = torch.cat([x, torch.ones_like(x)])[None].contiguous()
  native.gated_gelu_bwd_(torch.ones(1, x.numel(), device="cuda").bfloat16(), h)
  d_x, d_gate = h[0, :x.numel()].double(), h[0, x.numel():].double()
  inner = 0.8 * (1 + 3 * 0.044715 * xd * xd)
  assert bool(((d_x - slope).abs() <= 2.0 ** -8 * slope.abs() + tanh_part * (1 + 2 * inner)).all())
  assert bool(((d_gate - want).abs() <= 2.0 ** -8 * want.abs() + tanh_part).all())


@pytest.mark.parametrize("spread", [0.3, 1.0, 3.0])
def test_gated_experts_lose_nothing_to_separate_ops(spread):
  """The activation in the epilogue, on sums that have not been rounded, against products, activation and
  gate as separate ops with a rounding to bf16 after each: no further from float64, the negative side of the
  activation taken by itself too."""
  from t5x_b200.ops import functional as F
  g = torch.Generator(device="cuda").manual_seed(9)
  x = torch.randn(2, 300, 128, device="cuda", generator=g).bfloat16()
  w = [(torch.randn(2, 128, 512, device="cuda", generator=g) * spread * 128 ** -0.5).bfloat16().float()
       for _ in range(2)]
  with torch.no_grad():
    got = F.batched_gated_mlp_in(x, *w)
    h = [F.batched_linear(x, p, torch.bfloat16) for p in w]
    apart = torch.nn.functional.gelu(h[0], approximate="tanh") * h[1]
  hd = [x.double() @ p.double() for p in w]
  want = torch.nn.functional.gelu(hd[0], approximate="tanh") * hd[1]
  for part in (hd[0] < 100, hd[0] < 0, hd[0] < -1, hd[0] < -3):
    if int(part.sum()) > 100:
      assert float((got.double() - want)[part].norm()) < float((apart.double() - want)[part].norm())


@pytest.mark.parametrize("kind", ["experts", "dense", "dense_general"])
def test_pre_activations_are_kept_for_a_backward_pass_only(kind, monkeypatch):
  """The same result bit by bit with and without gradients; without them nothing but the result is
  allocated."""
  from t5x_b200.ops import functional as F
  from t5x_b200.ops import native
  if kind == "dense_general":  # the path for calls that the compiled one does not cover
    monkeypatch.setattr(native, "host", lambda: None)
  g = torch.Generator(device="cuda").manual_seed(3)
  lead = (2,) if kind == "experts" else ()
  x = torch.randn(*lead, 640, 64, device="cuda", generator=g).bfloat16()
  w = [torch.nn.Parameter(torch.randn(*lead, 64, 512, device="cuda", generator=g) * 0.1) for _ in range(2)]
  for p in w:
    p.bf16 = p.detach().bfloat16()
  call = F.batched_gated_mlp_in if kind == "experts" else F.gated_gelu_mlp_in
  y = call(x, *w)
  with torch.no_grad():
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    z = call(x, *w)
    assert torch.cuda.max_memory_allocated() - before == z.numel() * 2
  assert y.requires_grad and torch.equal(y, z)


def test_gradient_that_is_not_aligned_is_refused():
  """A contiguous gradient that starts between two 16-byte boundaries: an error, as from the products."""
  from t5x_b200.ops import functional as F
  from t5x_b200.ops import native
  x = torch.randn(2, 16, 64, device="cuda").bfloat16().requires_grad_()
  w = [torch.nn.Parameter(torch.randn(2, 64, 64, device="cuda")) for _ in range(2)]
  y = F.batched_gated_mlp_in(x, *w)
  dg = torch.randn(y.numel() + 1, device="cuda").bfloat16()[1:].view(y.shape)
  with pytest.raises(native.NativeError, match="aligned"):
    y.backward(dg)
  torch.cuda.synchronize()
