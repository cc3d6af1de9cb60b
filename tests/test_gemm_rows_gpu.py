"""The few-row GEMM with its norm, residual and gated-GELU forms at 1 to 64 rows, K and N down to
one step, and the decode step built from it. The bf16 output rounds to 2^-9 relative; the
normalised operand is rounded to bf16 in both forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 16, 16), (4, 768, 768), (8, 32, 144), (16, 48, 2048),
                                   (17, 64, 1024), (33, 16, 1040), (64, 80, 512)])
@pytest.mark.parametrize("norm", [False, True])
def test_gemm_rows(M, N, K, norm):
  from t5x_b200.ops import native
  assert native.gemm_rows_ok(M, N, K) and native.gemm_rows_ok(M, N, K, gated=True)
  g = torch.Generator(device="cuda").manual_seed(M * N + K)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  a = (rnd(M, K + 8) * 3).bfloat16()[:, :K]
  b, b2 = ((rnd(K, N + 8) * K ** -0.5).bfloat16()[:, :N] for _ in range(2))
  scale = 1 + 0.1 * rnd(K) if norm else None
  h = a.double()
  if norm:
    h = native.rmsnorm_fwd(a.contiguous(), scale, 1e-6)[0].double()
  res = rnd(M, N).bfloat16()
  tol = dict(rtol=2 ** -7, atol=2 ** -7)
  y = native.gemm_rows(a, b, norm_scale=scale, residual=res)
  torch.testing.assert_close(y.double(), h @ b.double() + res.double(), **tol)
  z = native.gemm_rows(a, b, norm_scale=scale, out_dtype=torch.float32, alpha=0.5)
  # one operand in a few thousand may round the other way where the norm's sum order differs
  torch.testing.assert_close(z.double(), 0.5 * (h @ b.double()), rtol=1e-3, atol=4e-3)
  y = native.gemm_rows(a, b, b2=b2, norm_scale=scale)
  gelu = torch.nn.functional.gelu(h @ b.double(), approximate="tanh")
  torch.testing.assert_close(y.double(), gelu * (h @ b2.double()), rtol=2 ** -6, atol=2 ** -5)


def test_refuses_what_it_does_not_cover():
  from t5x_b200.ops import native
  for m, n, k in [(0, 16, 16), (65, 16, 16), (4, 24, 16), (4, 16, 24), (64, 16, 2048)]:
    assert not native.gemm_rows_ok(m, n, k)
  a = torch.zeros(4, 32, device="cuda", dtype=torch.bfloat16)
  with pytest.raises(native.NativeError):
    native.gemm_rows(a, torch.zeros(32, 24, device="cuda", dtype=torch.bfloat16))


@pytest.mark.parametrize("batch,beams", [(1, 1), (3, 4), (16, 4)])
def test_decode_step_agrees_with_the_other_kernels(batch, beams):
  """The same search with and without the few-row products: the same logits up to bf16."""
  from t5x_b200 import decoding_fast, trainer
  from t5x_b200.models.t5 import network
  torch.manual_seed(0)
  cfg = network.T5Config(vocab_size=256, dtype="bfloat16", emb_dim=256, num_heads=4, head_dim=64,
                         num_encoder_layers=1, num_decoder_layers=2, mlp_dim=512,
                         mlp_activations=("gelu", "linear"), dropout_rate=0.0)
  module = network.Transformer(cfg, device="cuda")
  for p in module.parameters():
    p.bf16 = p.detach().bfloat16()
  enc = torch.randint(2, 256, (batch, 19), device="cuda")
  logits = []
  for few in (True, False):
    d = decoding_fast.GraphBeamDecoder(module, batch, beams, 12, 1, use_graph=False)
    assert d.few_rows == (batch * beams <= decoding_fast.FEW_ROWS)
    d.few_rows = few
    with torch.no_grad():
      d._encode(enc)
      d._reset()
      logits.append(d._model_step())
  scale = logits[1].abs().max()
  assert float((logits[0] - logits[1]).abs().max() / scale) < 0.03


@pytest.mark.parametrize("b,lk,h", [(1, 1, 1), (2, 31, 3), (3, 33, 2), (2, 64, 4), (1, 129, 2)])
def test_cross_layout(b, lk, h):
  """A rearrangement: equal to the tensor-op statement bit by bit, the padding zero."""
  from t5x_b200 import decoding_fast
  k, v = (torch.randn(b, lk, h, 64, device="cuda").bfloat16() for _ in range(2))
  kp, vt = decoding_fast.cross_kv_layout(k, v)
  kc, vc = decoding_fast.cross_kv_layout(k.cpu(), v.cpu())
  assert torch.equal(kp.cpu(), kc) and torch.equal(vt.cpu(), vc)
  again = decoding_fast.cross_kv_layout(v, k, out=(kp, vt))
  assert again[0] is kp and torch.equal(kp[:, :, :lk], v.transpose(1, 2))


@pytest.mark.parametrize("m,k,n,splits,transposed,with_res", [
    (256, 2048, 2048, 4, False, True), (37, 128, 384, 2, True, False),
    (200, 1024, 256, 8, False, True), (128, 192, 128, 1, False, False), (1, 64, 128, 1, True, True),
    (300, 512, 640, 2, True, True)])
def test_skinny_with_half_width_tiles(m, k, n, splits, transposed, with_res):
  """The cluster split-K GEMM with 128 x 64 tiles: every cluster size, rings that are not filled
  and rings that wrap, both weight layouts, row tails. fp32 accumulation, one rounding to bf16
  (2^-9 of a value), with a factor of two for the fp32 sums."""
  from t5x_b200.ops import native
  torch.manual_seed(m + k + n)
  a = torch.randn(m, k, device="cuda").bfloat16()
  w = (torch.randn(n, k, device="cuda") * 0.05).bfloat16().t() if transposed else \
      (torch.randn(k, n, device="cuda") * 0.05).bfloat16()
  res = torch.randn(m, n, device="cuda").bfloat16() if with_res else None
  out = native.gemm_skinny(a, w, residual=res, splits=splits, tile_n=64)
  native.check_status()
  ref = a.double() @ w.double() + (0 if res is None else res.double())
  assert float((out.double() - ref).abs().max() / ref.abs().max()) < 2 * 2.0 ** -9
  assert torch.equal(out, native.gemm_skinny(a, w, residual=res, splits=splits, tile_n=64))
