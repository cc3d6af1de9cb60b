"""The forward kernel for few heads of 64 channels: the bits of the kernel for many heads over every kind of mask, sizes
at the edges of its blocks of 128 queries and keys, projections side by side in one buffer; some against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(lq, lk, bias, kind, side_by_side=False, b=3, h=5):
  from t5x_b200.ops import attention as A
  g = torch.Generator(device="cuda").manual_seed(lq * 7 + lk)
  if side_by_side:
    q, k, v = torch.randn(b, lq, 3, h, 64, device="cuda", generator=g).bfloat16().unbind(2)
    q = q.mul_(0.3)
  else:
    q = (torch.randn(b, lq, h, 64, device="cuda", generator=g) * 0.3).bfloat16()
    k, v = (torch.randn(b, lk, h, 64, device="cuda", generator=g).bfloat16() for _ in range(2))
  table = torch.randn(h, 32, device="cuda", generator=g) if bias else None
  km = qs = ks = None
  if "padded" in kind or "unseen" in kind:
    km = torch.arange(lk, device="cuda")[None] < torch.tensor([lk, max(1, lk // 3), lk // 2 + 1], device="cuda")[:, None]
    if "unseen" in kind:
      km[2] = False  # an example in which no query sees a key: uniform rows
  if "packed" in kind:
    qs, ks = ((torch.arange(l, device="cuda") * 3 // l + 1)[None].expand(b, l).contiguous() for l in (lq, lk))
  causal = "causal" in kind
  return q, k, v, A.prepare(lq, lk, h, q.device, table, not causal, 32, 128, km, causal, qs, ks, 0, None), table


def _run(entry, q, k, v, prep):
  from t5x_b200.ops import attention as A, native
  rel_bias, buckets, km, qs, ks, mode, off, rel_off = prep
  b, lq, h, _ = q.shape
  o = torch.full((b, lq, h, 64), 7.0, device="cuda").bfloat16()
  lse = torch.full((b, h, lq), 7.0, device="cuda")
  p, (nb, nrel) = native.ptr, A._bias_sizes(rel_bias, buckets)
  rc = getattr(native.lib(), entry)(
      *(t.data_ptr() for t in (q, k, v, o, lse)), b, h, lq, k.shape[1], *(s for t in (q, k, v, o) for s in A._sbh(t)),
      p(rel_bias), p(buckets), nb, nrel, rel_off, p(km), p(qs), p(ks), mode, off, native.stream_ptr())
  native._check(rc, entry)
  native.check_status()
  return o, lse


@pytest.mark.parametrize("kind", ["none", "padded", "unseen", "causal", "causal padded", "packed", "causal packed padded"])
@pytest.mark.parametrize("lq,lk", [(1, 1), (9, 37), (64, 65), (127, 128), (129, 129), (114, 512), (256, 256), (255, 400),
                                   (300, 511), (512, 512), (200, 90)])
def test_bits_of_the_kernel_for_many_heads(lq, lk, kind):
  for bias in (False, True):
    for side_by_side in (False, True) if lq == lk else (False,):
      *ops, _ = _operands(lq, lk, bias, kind, side_by_side)
      few, many = _run("t5x_attention_fwd_few", *ops), _run("t5x_attention_fwd", *ops)
      assert torch.equal(few[0], many[0]) and torch.equal(few[1], many[1]), (bias, side_by_side)


@pytest.mark.parametrize("lq,lk,kind", [(9, 37, "padded"), (129, 200, "unseen"), (256, 512, "none"), (100, 100, "causal")])
def test_against_float64(lq, lk, kind):
  from t5x_b200.ops import reference as ref
  q, k, v, prep, table = _operands(lq, lk, True, kind)
  o, lse = _run("t5x_attention_fwd_few", q, k, v, prep)
  rel = torch.arange(lk, device="cuda")[None] - torch.arange(lq, device="cuda")[:, None]
  s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double())
  s = s + table.double()[:, ref.relative_position_bucket(rel, kind != "causal", 32, 128)][None]
  if prep[2] is not None:
    s = torch.where(prep[2].bool()[:, None, None], s, -1e10)
  if kind == "causal":
    s = torch.where(rel <= 0, s, -1e10)
  want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.double())
  # the probabilities and the result are each rounded to bf16 once; log-sum-exps are 32-bit
  assert float((o.double() - want).norm() / want.norm()) < 2 * 2.0 ** -8
  assert float(((lse.double() - torch.logsumexp(s, -1)).abs() / (1 + s.amax(-1).abs())).max()) < 1e-5


def test_choice():
  from t5x_b200.ops import attention as A
  sms = A._sms()
  assert A.forward_kernel(114, 512, 64, heads=sms) == "few" and A.forward_kernel(256, 64, 64, heads=1) == "few"
  assert A.forward_kernel(114, 512, 64, heads=sms + 1) == "classic"
  assert A.forward_kernel(257, 64, 64, heads=1) == "classic" and A.forward_kernel(64, 513, 64, heads=1) == "classic"
  assert A.forward_kernel(64, 64, 64, True, heads=1) == "classic" and A.forward_kernel(64, 64, 128, heads=1) == "stream"


@pytest.mark.parametrize("compiled", [True, False])
def test_the_choice_makes_no_difference(compiled, monkeypatch):
  """Examples together, which go to the kernel for many heads, and one by one, which do not."""
  from t5x_b200.ops import attention as A, native
  if not compiled:
    monkeypatch.setattr(native, "host", lambda: None)
  g = torch.Generator(device="cuda").manual_seed(0)
  b = A._sms() // 6 + 1
  q, k, v = (torch.randn(b, 130, 6, 64, device="cuda", generator=g).bfloat16() for _ in range(3))
  table = torch.randn(6, 32, device="cuda", generator=g)
  with torch.no_grad():
    whole = A.flash_attention(q, k, v, bias_table=table, bidirectional=True)
    parts = [A.flash_attention(q[i:i + 1], k[i:i + 1], v[i:i + 1], bias_table=table, bidirectional=True)
             for i in range(b)]
  assert torch.equal(whole, torch.cat(parts))
