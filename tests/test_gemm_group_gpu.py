"""Several products in one launch (`native.gemm_shared`, `native.gemm_sum`) at tile edges, odd and unequal
widths, both operand orientations and both tile kernels, against float64 and against separate launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mat(rows, cols, transposed, seed):
  g = torch.Generator(device="cuda").manual_seed(seed)
  if transposed:
    return torch.randn(cols, rows, device="cuda", generator=g).bfloat16().t()
  return torch.randn(rows, cols, device="cuda", generator=g).bfloat16()


SHAPES = [(1, 64, (128, 128, 128)), (130, 72, (8, 264)), (257, 200, (256, 512, 264)),
          (700, 768, (768, 768, 768)), (2600, 128, (384, 384, 384)), (5000, 1024, (1024, 256)),
          (300, 96, (520,))]


@pytest.mark.parametrize("M,K,widths", SHAPES)
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True), (True, False)])
def test_shared_input_equals_separate_launches(M, K, widths, ta, tb):
  from t5x_b200.ops import native
  if ta and M % 8:
    pytest.skip("rows of a transposed operand are multiples of 8 elements")
  a = _mat(M, K, ta, 1)
  b = [_mat(K, n, tb, 2 + i) for i, n in enumerate(widths)]
  out = native.gemm_shared(a, b)
  native.check_status()
  for o, w in zip(out, b):
    assert torch.equal(o, native.gemm(a, w))


@pytest.mark.parametrize("M,N,widths", [(1, 128, (64, 64)), (130, 72, (8, 264)), (257, 264, (200, 64, 136)),
                                        (700, 768, (768, 768, 768)), (5000, 1472, (384, 384, 384)),
                                        (4096, 1024, (2816, 2816)), (300, 96, (520,))])
@pytest.mark.parametrize("ta,tb", [(False, False), (False, True)])
def test_sum_of_products(M, N, widths, ta, tb):
  """fp32 sums over all products, one rounding to bf16 (2^-9 of a value), with a factor of two for the
  fp32 sums."""
  from t5x_b200.ops import native
  a = [_mat(M, k, ta, 1 + i) for i, k in enumerate(widths)]
  b = [_mat(k, N, tb, 5 + i) for i, k in enumerate(widths)]
  out = native.gemm_sum(a, b)
  native.check_status()
  ref = sum(x.double() @ y.double() for x, y in zip(a, b))
  assert float((out.double() - ref).abs().max() / ref.abs().max()) < 2 * 2.0 ** -9
  assert torch.equal(out, native.gemm_sum(a, b))


@pytest.mark.parametrize("M,tokens,widths", [(256, 4096, (256, 512)), (768, 12216, (768, 768, 768)),
                                             (520, 1000, (264, 256, 272)), (64, 300, (64, 128)),
                                             (1472, 8192, (384, 384, 384))])
@pytest.mark.parametrize("pieces", [0, 1, 3])
@pytest.mark.parametrize("accumulate", [False, True])
def test_weight_gradients_of_a_shared_input(M, tokens, widths, pieces, accumulate):
  """fp32 sums over the tokens: the error of a sum of n products in any order stays below
  n 2^-24 times the sum of their magnitudes."""
  from t5x_b200.ops import native
  x = _mat(M, tokens, True, 1)
  dy = [_mat(tokens, n, False, 2 + i) for i, n in enumerate(widths)]
  out = [torch.full((M, n), 3.0, device="cuda") for n in widths]
  native.gemm_shared(x, dy, out=out, accumulate=accumulate, pieces=pieces)
  native.check_status()
  for o, d in zip(out, dy):
    ref = x.double() @ d.double() + (3.0 if accumulate else 0.0)
    size = x.double().abs() @ d.double().abs() + 3.0
    assert bool(((o.double() - ref).abs() <= tokens * 2.0 ** -24 * size).all())


def test_too_many_products_are_refused():
  from t5x_b200.ops import native
  a, b = _mat(64, 64, False, 1), [_mat(64, 64, False, 2)] * 4
  with pytest.raises(native.NativeError):
    native.gemm_shared(a, b)
  with pytest.raises(native.NativeError):
    native.gemm_sum([a] * 4, b)
