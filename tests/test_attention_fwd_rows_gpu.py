"""The forward kernel for heads of 64 at the edges of its tiles of 128 queries, pairs of tiles, blocks of 64 keys
and of its two ranges of keys, under every kind of mask, against float64; and the log-sum-exp that it leaves for
the backward pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask", ["none", "padded", "unseen", "causal", "packed", "prefix"])
@pytest.mark.parametrize("lq,lk,bias", [(1, 1, True), (33, 64, True), (128, 65, False), (129, 31, True),
                                        (64, 512, True), (256, 256, True), (257, 257, True), (385, 512, False),
                                        (100, 513, True), (600, 600, True), (130, 2048, True),
                                        (40, 1000, False)])
def test_against_float64(lq, lk, bias, mask):
  from t5x_b200.ops import attention as A, native, reference as ref
  if mask in ("causal", "packed", "prefix") and lq != lk:
    pytest.skip("self-attention")
  g = torch.Generator(device="cuda").manual_seed(lq * 3 + lk)
  b, h = 3, 2
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  q = (rnd(b, lq, h, 64) * 0.3).bfloat16()
  k, v = rnd(b, lk, h, 64).bfloat16(), rnd(b, lk, h, 64).bfloat16()
  table = rnd(h, 32) if bias else None
  pos = torch.arange(lk, device="cuda")
  kw, allowed, both = {}, torch.ones(b, lq, lk, dtype=torch.bool, device="cuda"), True
  if mask in ("padded", "unseen"):
    km = torch.ones(b, lk, dtype=torch.bool, device="cuda")
    km[1, max(1, lk // 3):] = False
    if mask == "unseen":
      km[2] = False  # an example in which no query sees a key: uniform rows
    allowed, kw = allowed & km[:, None], dict(key_mask=km)
  elif mask != "none":
    both = False
    allowed, kw = allowed & (pos[None] <= pos[:, None]), dict(causal=True)
    if mask == "packed":
      seg = (pos // 70 + 1)[None].expand(b, lk).contiguous()
      allowed = allowed & (seg[:, :, None] == seg[:, None])
      kw.update(q_segment_ids=seg, kv_segment_ids=seg)
    if mask == "prefix":
      inside = pos[None] < torch.tensor([lk // 3, 0, lk], device="cuda")[:, None]
      prefix = ref.PrefixLMMask(inside, torch.ones_like(inside), None)
      allowed, kw = prefix.bool()[:, 0], dict(prefix_lm=prefix)
  assert A.forward_kernel(lq, lk, 64, mask == "prefix") == "classic"
  prep = A.prepare(lq, lk, h, q.device, table, both, 32, 128, kw.get("key_mask"), kw.get("causal", False),
                   kw.get("q_segment_ids"), kw.get("kv_segment_ids"), 0, kw.get("prefix_lm"))
  rel_bias, buckets, km8, qs, ks, mode, off, rel_off = prep
  o = torch.full_like(q, 7.0)
  lse = torch.full((b, h, lq), 7.0, device="cuda")
  p, (nb, nrel) = native.ptr, A._bias_sizes(rel_bias, buckets)
  native._check(native.lib().t5x_attention_fwd(
      *(t.data_ptr() for t in (q, k, v, o, lse)), b, h, lq, lk, *(s for t in (q, k, v, o) for s in A._sbh(t)),
      p(rel_bias), p(buckets), nb, nrel, rel_off, p(km8), p(qs), p(ks), mode, off, native.stream_ptr()), "fwd")
  native.check_status()
  s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double())
  if bias:
    rel = pos[None] - torch.arange(lq, device="cuda")[:, None]
    s = s + table.double()[:, ref.relative_position_bucket(rel, both, 32, 128)][None]
  s = torch.where(allowed[:, None], s, -1e10)
  want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.double())
  # the probabilities and the result are each rounded to bf16 once; log-sum-exps are 32-bit
  assert float((o.double() - want).norm() / want.norm()) < 2 * 2.0 ** -8
  assert float(((lse.double() - torch.logsumexp(s, -1)).abs() / (1 + s.amax(-1).abs())).max()) < 1e-5


@pytest.mark.parametrize("kind", ["causal", "causal masked", "causal packed", "causal packed masked"])
@pytest.mark.parametrize("lq,lk,bias", [(300, 460, True), (460, 300, True), (130, 700, False), (64, 40, True),
                                        (600, 1100, True), (1100, 600, True), (513, 140, False)])
def test_causal_of_other_lengths(lq, lk, bias, kind):
  """More or fewer queries than keys: the last query sees the last key, and the first ones may see none."""
  from t5x_b200.ops import attention as A, native, reference as ref
  g = torch.Generator(device="cuda").manual_seed(lq * 5 + lk)
  b, h = 3, 2
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  q = (rnd(b, lq, h, 64) * 0.3).bfloat16()
  k, v = rnd(b, lk, h, 64).bfloat16(), rnd(b, lk, h, 64).bfloat16()
  table = rnd(h, 32) if bias else None
  qpos, kpos = torch.arange(lq, device="cuda"), torch.arange(lk, device="cuda")
  allowed = (kpos[None] <= qpos[:, None] + lk - lq).expand(b, lq, lk)
  km = qs = ks = None
  if "masked" in kind:
    km = torch.ones(b, lk, dtype=torch.bool, device="cuda")
    km[1, :30], km[2, lk // 2:] = False, False
    allowed = allowed & km[:, None]
  if "packed" in kind:
    qs, ks = ((p * 4 // p.numel()).int()[None].expand(b, -1).contiguous() for p in (qpos, kpos))
    allowed = allowed & (qs[:, :, None] == ks[:, None])
  rel_bias, buckets, km8, qc, kc, mode, off, rel_off = A.prepare(lq, lk, h, q.device, table, False, 32, 128, km, True,
                                                                 qs, ks, 0, None)
  s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double())
  if bias:
    s = s + table.double()[:, ref.relative_position_bucket(kpos[None] - qpos[:, None], False, 32, 128)][None]
  s = torch.where(allowed[:, None], s, -1e10)
  want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.double())
  p, (nb, nrel) = native.ptr, A._bias_sizes(rel_bias, buckets)
  entries = ["t5x_attention_fwd"] + (["t5x_attention_fwd_few"] if max(lq, lk) <= 512 else [])
  for entry in entries:
    o = torch.full_like(q, 7.0)
    lse = torch.full((b, h, lq), 7.0, device="cuda")
    native._check(getattr(native.lib(), entry)(
        *(t.data_ptr() for t in (q, k, v, o, lse)), b, h, lq, lk, *(s for t in (q, k, v, o) for s in A._sbh(t)),
        p(rel_bias), p(buckets), nb, nrel, rel_off, p(km8), p(qc), p(kc), mode, off, native.stream_ptr()), entry)
    native.check_status()
    assert float((o.double() - want).norm() / want.norm()) < 2 * 2.0 ** -8, entry
    assert float(((lse.double() - torch.logsumexp(s, -1)).abs() / (1 + s.amax(-1).abs())).max()) < 1e-5, entry
