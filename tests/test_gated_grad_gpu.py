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
