"""The gradient of a gated GELU inside the product that it follows, at the edges of its tiles, against the product and
the pass over memory that it takes the place of (which rounds dg in between)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _fused(dy, w, h):
  from t5x_b200.ops import native
  m, n = h.shape[0], h.shape[1] // 2
  native._check(native.lib().t5x_gemm_gated_grad(
      dy.data_ptr(), w.data_ptr(), h.data_ptr(), h.data_ptr() + 2 * n, m, n, dy.shape[1], dy.stride(0), w.stride(0),
      h.stride(0), 0, native.stream_ptr()), "gemm_gated_grad")
  native.check_status()


@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (257, 288, 72), (500, 480, 128), (1000, 2048, 768),
                                   (4099, 3584, 1472), (64, 32, 64)])
def test_gated_grad(m, n, k):
  g = torch.Generator(device="cuda").manual_seed(m)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
  dy, w, h = rnd(m, k), rnd(n, k), rnd(m, 2 * n)  # w: [n, k], the second kernel of the block
  w *= k ** -0.5
  x0, x1 = (t.double().requires_grad_() for t in (h[:, :n], h[:, n:]))
  dg = dy.double() @ w.double().t()
  want = torch.autograd.grad(torch.nn.functional.gelu(x0, approximate="tanh") * x1, (x0, x1), dg)
  guard = torch.full((m + 3, 2 * n), 5.0, device="cuda", dtype=torch.bfloat16)
  guard[:m] = h
  _fused(dy, w, guard[:m])
  assert bool((guard[m:] == 5.0).all())
  for got, x in zip((guard[:m, :n], guard[:m, n:]), want):
    # one rounding to bf16 of the result; tanh to some 5e-4 (its fast form), of values below one
    assert float((got.double() - x).norm() / x.norm()) < 2.0 ** -8


def test_choice():
  """Both sides of the rule, where the tiles' last wave or last rows are nearly empty."""
  from t5x_b200.ops import native
  covers = native.lib().t5x_gemm_gated_grad_covers
  for m, n in ((300, 10240), (384, 10240), (4864, 1024), (1700, 2816), (512, 5120), (1280, 2048), (256, 65536 * 8 + 8)):
    assert not covers(m, n), (m, n)
  for m, n in ((512, 10240), (768, 5120), (1000, 2816), (3000, 1024), (8192, 1024), (65536, 2048), (32768, 10240)):
    assert covers(m, n), (m, n)
  assert native.lib().t5x_gemm_relu_covers(384, 10240) and not native.lib().t5x_gemm_relu_covers(384, 1024)


@pytest.mark.parametrize("m,d,ff", [(2048, 256, 2048), (384, 128, 10240), (257, 128, 512)])
def test_block(m, d, ff):
  """The backward pass of a gated block by either route, against float64."""
  from t5x_b200.ops import native
  host = native.host()
  g = torch.Generator(device="cuda").manual_seed(m)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  x, dy, scale = rnd(m, d).bfloat16(), rnd(m, d).bfloat16(), 1 + 0.1 * rnd(d)
  w = [(rnd(d, ff) * d ** -0.5).bfloat16(), (rnd(d, ff) * d ** -0.5).bfloat16(), (rnd(ff, d) * ff ** -0.5).bfloat16()]
  y, *saved = host.mlp_block(x, scale, 1e-6, w, True)
  grads, dscale = [torch.full(t.shape, 7.0, device="cuda") for t in w], torch.zeros(d, device="cuda")
  dx = host.mlp_block_bwd(dy, x, scale, w, saved, grads, [False] * 3, dscale)
  native.check_status()
  leaves = [t.double().requires_grad_() for t in (x, scale, *w)]
  x2, s2, w0, w1, wo = leaves
  h = x2 * torch.rsqrt(x2.pow(2).mean(-1, keepdim=True) + 1e-6) * s2
  want = torch.autograd.grad(x2 + (torch.nn.functional.gelu(h @ w0, approximate="tanh") * (h @ w1)) @ wo, leaves,
                             dy.double())
  # a chain of four results in bf16 (h, the pre-activations, g, their gradients), each off by up to 2^-9
  for got, ref in zip((dx, dscale, *grads), want):
    assert float((got.double() - ref).norm() / ref.norm()) < 4 * 2.0 ** -8
