"""Epilogues of the bf16 GEMMs at the edges of their tiles: column ranges that end inside a warp's
half of a tile or before it, rows that end inside a warp, residuals on and off the 16-byte path,
and the cross-entropy epilogues, which fold 128 columns into one partial. Bounds: the operands are
exact in both forms, the fp32 sums of K products differ by their order (K * 2^-24 of the sum of
magnitudes, far below the bf16 rounding of the output, 2^-9 relative)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 64), (40, 96, 64), (129, 136, 72), (256, 264, 128), (300, 392, 64), (513, 640, 192)]


def _operands(M, N, K, seed):
  g = torch.Generator(device="cuda").manual_seed(seed)
  a = torch.randn(M, K, device="cuda", generator=g).bfloat16()
  b = (torch.randn(K, N, device="cuda", generator=g) * K ** -0.5).bfloat16()
  return a, b, g


@pytest.mark.parametrize("pair", [0, 2])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_residual_and_accumulate(M, N, K, pair):
  from t5x_b200.ops import native
  a, b, g = _operands(M, N, K, M + N)
  want = a.double() @ b.double()
  wide = torch.randn(M, N + 4, device="cuda", generator=g).bfloat16()
  native.gemm_set_pair_mode(pair)
  try:
    for res in (wide[:, :N].contiguous(), wide[:, :N], wide[:, 1:N + 1]):
      y = native.gemm(a, b, residual=res)
      torch.testing.assert_close(y.double(), want + res.double(), rtol=2 ** -8, atol=2 ** -8)
    acc = torch.randn(M, N, device="cuda", generator=g)
    out = acc.clone()
    native.gemm(a, b, out=out, accumulate=True)
    torch.testing.assert_close(out.double(), want + acc.double(), rtol=1e-5, atol=1e-5)
  finally:
    native.gemm_set_pair_mode(1)
  native.check_status()


def _views(M, N, dtype):
  """(name, make): [M, N] and [3, M, N] outputs whose rows, start or batches lie on and off 16 bytes."""
  unit = 8 if dtype == torch.bfloat16 else 4
  ld = -(-N // unit) * unit

  def of(batch, ld, step, start):
    flat = torch.randn(max(batch, 1) * max(step, M * ld) + start + 64, device="cuda").to(dtype)
    return flat.as_strided((M, N) if batch == 0 else (batch, M, N),
                           (ld, 1) if batch == 0 else (step, ld, 1), start)
  return [("whole", of(0, ld, 0, 0)), ("rows apart", of(0, ld + unit, 0, 0)),
          ("odd rows", of(0, ld + 1, 0, 0)), ("odd start", of(0, ld, 0, 1)),
          ("batches", of(3, ld, M * ld + unit, 0)), ("odd batches", of(3, ld, M * ld + 1, 0))]


@pytest.mark.parametrize("pair", [0, 2])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M,N,K", SHAPES + [(70, 100, 64)])
def test_store_and_add_at_any_alignment(M, N, K, dtype, pair):
  """C = and C += in both output types. A bf16 result is rounded once: 2^-9 relative, with a factor
  of two; the fp32 sums of K products as above."""
  from t5x_b200.ops import native
  native.gemm_set_pair_mode(pair)
  rtol = 2 ** -8 if dtype == torch.bfloat16 else 1e-5
  try:
    for name, out in _views(M, N, dtype):
      batch = out.shape[0] if out.dim() == 3 else 1
      ops = [_operands(M, -(-N // 8) * 8, K, M + N + i) for i in range(batch)]
      a, b = (torch.stack([o[i] for o in ops]) for i in (0, 1))
      if out.dim() == 2:
        a, b = a[0], b[0]
      b = b[..., :N]
      want = a.double() @ b.double()
      old = out.clone()
      native.gemm(a, b, out=out, accumulate=True)
      torch.testing.assert_close(out.double(), want + old.double(), rtol=rtol, atol=2e-5, msg=lambda m: name + m)
      native.gemm(a, b, out=out)
      torch.testing.assert_close(out.double(), want, rtol=rtol, atol=2e-5, msg=lambda m: name + m)
      if dtype == torch.bfloat16:
        y = native.gemm(a, b, residual=out)  # the same views as a residual
        torch.testing.assert_close(y.double(), want + out.double(), rtol=rtol, atol=2e-5)
  finally:
    native.gemm_set_pair_mode(1)
  native.check_status()


@pytest.mark.parametrize("pair", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (37, 129, 64), (256, 128, 64), (300, 1000, 128),
                                   (515, 2184, 64)])
def test_cross_entropy(M, N, K, pair):
  from t5x_b200.ops import native
  ldb = -(-N // 8) * 8
  a, b, g = _operands(M, ldb, K, 3 * M + N)
  b = b[:, :N]
  t = torch.randint(0, N, (M,), device="cuda", generator=g)
  t[0], t[-1] = 0, N - 1
  x = (a.double() @ b.double()) * 0.5
  native.gemm_set_pair_mode(pair)
  try:
    stats, _, arg = native.gemm_ce_stats(a, b, t, alpha=0.5)
    lse = stats[:, 0] + torch.log(stats[:, 1])
    want_lse = torch.logsumexp(x, -1)
    torch.testing.assert_close(lse.double(), want_lse, rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(stats[:, 2].double(), x.gather(1, t[:, None])[:, 0], rtol=1e-5,
                               atol=1e-5)
    torch.testing.assert_close(stats[:, 3].double(), x.sum(-1), rtol=1e-4, atol=1e-3)
    top = x.gather(1, arg.long()[:, None])[:, 0]
    assert bool((top >= x.max(-1).values - 1e-5).all())
    scale = torch.rand(M, device="cuda", generator=g)
    scale[M // 2] = 0.0
    d = native.gemm_ce_grad(a, b, t, want_lse.float(), scale, 1e-3, 0.9, 0.1 / (N - 1), alpha=0.5)
    soft = torch.full_like(x, 0.1 / (N - 1)).scatter_(1, t[:, None], 0.9)
    want = scale.double()[:, None] * ((1 + 2e-3 * want_lse)[:, None] *
                                      torch.exp(x - want_lse[:, None]) - soft)
    torch.testing.assert_close(d.double(), want, rtol=2 ** -8, atol=1e-5)
    assert not bool(d[M // 2].any())
  finally:
    native.gemm_set_pair_mode(1)
  native.check_status()


@pytest.mark.parametrize("batch,M,N,K", [(1, 768, 768, 4264), (1, 1472, 384, 8200),
                                         (1, 256, 256, 40000), (3, 256, 520, 13000),
                                         (1, 704, 304, 6000), (1, 2048, 2600, 8000)])
@pytest.mark.parametrize("ta", [0, 1])
def test_weight_gradient_with_a_split_last_wave(batch, M, N, K, ta):
  """fp32 outputs whose last wave of tiles is cut along K, the pieces added atomically (also with
  whole tiles before them, batches, and K off the block size). The tensor core
  adds 16 products at a time and truncates: at most one unit in the last place of an accumulator
  of up to 5 sqrt(K) per step, K / 16 steps."""
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(K)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
  a = rnd(batch, K, M).transpose(1, 2) if ta else rnd(batch, M, K)
  b = rnd(batch, K, N)
  if batch == 1:
    a, b = a[0], b[0]
  want = a.double() @ b.double()
  tol = K / 16 * 2 ** -23 * 5 * K ** 0.5
  wide = torch.zeros(*want.shape[:-1], N + 8, device="cuda")  # rows apart: whole tiles
  for pieces in (0, 2, 7):
    out = torch.full(want.shape, 3.0, device="cuda")
    native.gemm_wgrad(a, b, out=out, pieces=pieces)
    assert float((out - want).abs().max()) < tol
    native.gemm_wgrad(a, b, out=out, accumulate=True, pieces=pieces)
    assert float((out - 2 * want).abs().max()) < 2 * tol
    native.gemm_wgrad(a, b, out=wide[..., :N], pieces=pieces)
    assert float((wide[..., :N] - want).abs().max()) < tol and not bool(wide[..., N:].any())
  native.check_status()


@pytest.mark.parametrize("M,N,K", [(256, 384, 2560), (256, 384, 2048), (256, 384, 4672), (512, 768, 8200)])
def test_forward_products_keep_whole_tiles(M, N, K):
  """fp32 logits are the same bit by bit on every call, and equal those of an output whose rows lie
  apart, which is never cut: no product is cut along K unless its caller asks for it."""
  from t5x_b200.ops import native
  a, b, _ = _operands(M, N, K, K)
  wide = torch.empty(M, N + 8, device="cuda")
  native.gemm(a, b, out=wide[:, :N])
  for _ in range(10):
    assert torch.equal(native.gemm(a, b, out_dtype=torch.float32), wide[:, :N])
  native.check_status()


@pytest.mark.parametrize("M,N,K,cut", [(1024, 2816, 2048, False), (768, 2304, 2048, False),
                                       (3072, 768, 2048, False), (2048, 2048, 12216, False),
                                       (768, 768, 12216, True), (256, 256, 65536, True)])
def test_weight_gradients_are_cut_where_it_pays(M, N, K, cut):
  """Where the fill and the adds cost more than the last wave gives, the tiles stay whole (the sums
  are then those of whole tiles, bit by bit); long products with few tiles are cut."""
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(M + K)
  a, b = (torch.randn(K, n, device="cuda", generator=g).bfloat16() for n in (M, N))
  whole = native.gemm_wgrad(a.t(), b, pieces=1)
  assert torch.equal(native.gemm_wgrad(a.t(), b), whole) != cut
  native.check_status()


def test_phase_trace_stays_inside_its_buffer():
  """8 int64 per SM are enough for every traced GEMM, also for the 256 CTAs of a cluster product."""
  import ctypes
  from t5x_b200.ops import native
  sms = torch.cuda.get_device_properties(0).multi_processor_count
  buf = torch.zeros(4 * sms * 8, dtype=torch.int64, device="cuda")
  a = torch.randn(256, 2048, device="cuda").bfloat16()
  b = torch.randn(2048, 2048, device="cuda").bfloat16()
  set_trace = native.lib().t5x_gemm_set_trace
  set_trace.argtypes = [ctypes.c_void_p]
  for product in (lambda: native.gemm_skinny(a, b, splits=4), lambda: native.gemm_skinny(a, b, splits=8),
                  lambda: native.gemm(a[:128], b)):
    buf.zero_()
    set_trace(buf.data_ptr())
    try:
      product()
    finally:
      set_trace(None)
    t = buf.view(4 * sms, 8).cpu()
    assert bool((t[0] > 0).any()) and not bool(t[sms:].any())
  native.check_status()


@pytest.mark.parametrize("N", [128, 136, 200])
def test_cross_entropy_of_infinite_logits(N):
  """Rows whose logits overflow: all -inf (nothing to sum: the columns that pad a tile to 32 do not
  count either), one of them finite, one +inf."""
  from t5x_b200.ops import native
  big = 2.0 ** 100
  a = torch.zeros(4, 64, device="cuda", dtype=torch.bfloat16)
  b = torch.zeros(64, N, device="cuda", dtype=torch.bfloat16)
  a[0, 0] = a[1, 0] = a[2, 1] = big
  b[0], b[1, N - 1] = -big, big  # row 0: all -inf; row 2: the last +inf, zeros otherwise
  a[1, 2], b[0, 5], b[2, 5] = 1.0, 0.0, 3.0  # row 1: 3 in column 5
  b[0, 5] = 0.0
  a[0, 3], b[3, 5] = big, -big  # row 0, column 5: -inf as well
  t = torch.zeros(4, dtype=torch.long, device="cuda")
  x = a.double() @ b.double()
  x[x < -1e39], x[x > 1e39] = -float("inf"), float("inf")
  assert bool((x[0] == -float("inf")).all()) and x[1, 5] == 3.0
  stats, _, arg = native.gemm_ce_stats(a, b, t)
  lse = stats[:, 0] + torch.log(stats[:, 1])
  assert stats[0, 1] == 0 and lse[0] == -float("inf")
  torch.testing.assert_close(lse[[1, 3]].double(), torch.logsumexp(x[[1, 3]], -1))
  assert arg[1] == 5 and not bool(torch.isfinite(lse[2]))
  native.check_status()
