"""The backward kernel that keeps dQ of a head in TMEM, at the edges of its units of 64 queries and blocks of
128 keys, under every kind of mask, against float64 (the entry point is called as it is: by itself the choice
of the kernel goes by the number of heads)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(q, k, v, o, do, lse, table, lq, lk, key_mask, qs, ks, mode, outs=None):
  from t5x_b200.ops import attention as A, native
  b, h = q.shape[0], q.shape[2]
  dq, dk, dv = outs or (torch.full_like(t, 7.0) for t in (q, k, v))
  buckets = d_table = None
  if table is not None:
    buckets = A._rel_buckets(lq, lk, 0, mode == 0, 32, 128, q.device)
    d_table = torch.zeros_like(table)
  nb, nrel = A._bias_sizes(table, buckets)
  wide = [torch.zeros_like(t, dtype=torch.float32) if lq > 512 else None for t in (k, v)]
  p = native.ptr
  native._check(native.lib().t5x_attention_bwd_head(
      *(t.data_ptr() for t in (q, k, v, o, do, lse, dq, dk, dv)), *map(p, wide), b, h, lq, lk,
      *(s for t in (q, k, v, o, do, dq, dk) for s in A._sbh(t)), p(table), p(buckets), p(d_table), nb, nrel,
      lq - 1, p(key_mask), p(qs), p(ks), mode, lk - lq if mode else 0, native.stream_ptr()), "head")
  native.check_status()
  if lq > 512:
    dk, dv = wide
  return dq, dk, dv, d_table


@pytest.mark.parametrize("mask", ["none", "padded", "unseen", "causal", "packed", "prefix"])
@pytest.mark.parametrize("lq,lk,bias", [(1, 1, True), (31, 129, False), (64, 128, True), (65, 257, True),
                                        (129, 129, True), (200, 200, False), (512, 512, True),
                                        (511, 640, True), (130, 1100, False), (513, 130, True),
                                        (1000, 1000, True), (1100, 300, False)])
def test_against_float64(lq, lk, bias, mask):
  from t5x_b200.ops import attention as A, reference as ref
  if mask in ("causal", "packed", "prefix") and lq != lk:
    pytest.skip("self-attention")
  g = torch.Generator(device="cuda").manual_seed(lq + lk)
  b, h = 3, 2
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  q = (rnd(b, lq, h, 64) * 0.3).bfloat16()
  k, v, do = rnd(b, lk, h, 64).bfloat16(), rnd(b, lk, h, 64).bfloat16(), rnd(b, lq, h, 64).bfloat16()
  table = rnd(h, 32) if bias else None
  pos = torch.arange(lk, device="cuda")
  km = seg = None
  mode, kw, allowed = 0, {}, torch.ones(b, lq, lk, dtype=torch.bool, device="cuda")
  if mask in ("padded", "unseen"):
    km = torch.ones(b, lk, dtype=torch.bool, device="cuda")
    km[1, max(1, lk // 3):] = False
    if mask == "unseen":
      km[2] = False  # an example in which no query sees a key: uniform rows
    allowed = allowed & km[:, None]
    kw = dict(key_mask=km)
  elif mask != "none":
    mode, allowed = 1, allowed & (pos[None] <= pos[:, None])
    kw = dict(causal=True)
    if mask == "packed":
      seg = (pos // 70 + 1).int()[None].expand(b, lk).contiguous()
      allowed = allowed & (seg[:, :, None] == seg[:, None])
      kw = dict(causal=True, q_segment_ids=seg, kv_segment_ids=seg)
    if mask == "prefix":
      inside = pos[None] < torch.tensor([lk // 3, 0, lk], device="cuda")[:, None]
      prefix = ref.PrefixLMMask(inside, torch.ones_like(inside), None)
      mode, allowed, kw = 2, prefix.bool()[:, 0], dict(prefix_lm=prefix)
  prep = A.prepare(lq, lk, h, q.device, table, mode == 0, 32, 128, kw.get("key_mask"),
                   kw.get("causal", False), seg, seg, 0, kw.get("prefix_lm"))
  q2, k2, v2 = (t.double().requires_grad_() for t in (q, k, v))
  s = torch.einsum("bqhd,bkhd->bhqk", q2, k2)
  leaves = [q2, k2, v2]
  if bias:
    t2 = table.double().requires_grad_()
    leaves.append(t2)
    rel = pos[None] - torch.arange(lq, device="cuda")[:, None]
    s = s + t2[:, ref.relative_position_bucket(rel, mode == 0, 32, 128)][None]
  # the mask is an addition to the scores: it hides them, and hands on their gradients
  s = s + torch.where(allowed[:, None], 0.0, -1e10 - s.detach())
  probs = torch.softmax(s, -1)
  want = torch.autograd.grad(torch.einsum("bhqk,bkhd->bqhd", probs, v2), leaves, do.double())
  o = torch.einsum("bhqk,bkhd->bqhd", probs, v2).detach().bfloat16()
  lse = torch.logsumexp(s, -1).detach().float().contiguous()
  got = _call(q, k, v, o, do, lse, table, lq, lk, prep[2], prep[3], prep[4], mode)
  # P, dS and the results are each rounded to bf16 once, and rowsum(dO * O) takes a rounded O. (Of a single
  # key dq, dk and dbias are zero; dS is then the rounding of two equal 32-bit sums of 64 products, up to
  # 64 * 2^-24 * |dO| |v| or 1e-4 with norms of 8.)
  for name, a, w in zip(("dq", "dk", "dv", "dbias"), got, want):
    assert float((a.double() - w).norm() / (w.norm() + 1e-2)) < 4 * 2.0 ** -8, name


def _prefix(lq, kind):
  """A prefix-LM mask of three examples: whole, padded (a padding query sees nothing), padded within its prefix."""
  from t5x_b200.ops import reference as ref
  pos = torch.arange(lq, device="cuda")
  inside = pos[None] < torch.tensor([lq // 3, lq // 2, lq], device="cuda")[:, None]
  valid = pos[None] < torch.tensor([lq, lq - lq // 4, lq // 2], device="cuda")[:, None]
  seg = (pos * 3 // lq + 1).int()[None].expand(3, lq).contiguous() if "packed" in kind else None
  return ref.PrefixLMMask(inside, valid, seg)


@pytest.mark.parametrize("kind", ["causal", "causal masked", "causal packed", "causal packed masked", "prefix",
                                  "prefix packed", "holes"])
@pytest.mark.parametrize("lq,lk,bias", [(300, 300, True), (512, 512, True), (512, 512, False), (700, 700, True),
                                        (1100, 1100, True), (300, 460, True), (460, 300, True), (130, 700, False),
                                        (600, 1100, True), (1100, 600, True), (513, 140, False)])
def test_passed_over_blocks_and_offsets(lq, lk, bias, kind):
  """Blocks of keys or queries that are passed over, and those that must not be: queries that do not see themselves,
  prefixes, leading hidden blocks and holes; causal attention of more or fewer queries than keys."""
  from t5x_b200.ops import attention as A, reference as ref
  if "prefix" in kind and lq != lk:
    pytest.skip("self-attention")
  g = torch.Generator(device="cuda").manual_seed(lq * 5 + lk)
  b, h, outs = 3, 2, None
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  if lq == lk and lq <= 512:  # projections and their gradients side by side
    q, k, v = rnd(b, lq, 3, h, 64).bfloat16().unbind(2)
    q.mul_(0.3)
    outs = torch.full((b, lq, 3, h, 64), 7.0, device="cuda").bfloat16().unbind(2)
  else:
    q = (rnd(b, lq, h, 64) * 0.3).bfloat16()
    k, v = rnd(b, lk, h, 64).bfloat16(), rnd(b, lk, h, 64).bfloat16()
  do = rnd(b, lq, h, 64).bfloat16()
  table = rnd(h, 32) if bias else None
  qpos, kpos = torch.arange(lq, device="cuda"), torch.arange(lk, device="cuda")
  allowed = torch.ones(b, lq, lk, dtype=torch.bool, device="cuda")
  km = qs = ks = prefix = None
  if "prefix" in kind:
    prefix = _prefix(lq, kind)
    allowed = prefix.bool()[:, 0]
  elif "causal" in kind:
    allowed = allowed & (kpos[None] <= qpos[:, None] + lk - lq)
  if "masked" in kind or kind == "holes":
    km = torch.ones(b, lk, dtype=torch.bool, device="cuda")
    km[1, :140] = False
    km[2, 120:260] = False
    km[2, lk - 1] = True
    allowed = allowed & km[:, None]
  if "packed" in kind and prefix is None:
    qs, ks = ((p * 4 // p.numel()).int()[None].expand(b, -1).contiguous() for p in (qpos, kpos))
    allowed = allowed & (qs[:, :, None] == ks[:, None])
  prep = A.prepare(lq, lk, h, q.device, table, "causal" not in kind and prefix is None, 32, 128, km, "causal" in kind,
                   qs, ks, 0, prefix)
  q2, k2, v2, do2 = (t.double() for t in (q, k, v, do))
  bucket = ref.relative_position_bucket(kpos[None] - qpos[:, None], prep[5] == 0, 32, 128)
  s = torch.einsum("bqhd,bkhd->bhqk", q2, k2)
  if bias:
    s = s + table.double()[:, bucket][None]
  s = torch.where(allowed[:, None], s, -1e10)
  probs = torch.softmax(s, -1)
  o = torch.einsum("bhqk,bkhd->bqhd", probs, v2).bfloat16()
  lse = torch.logsumexp(s, -1).float().contiguous()
  # the gradients as the inputs give them, with rowsum(dO * O) of the rounded O: where all keys of a row share a
  # bucket, dbias is what that sum is off by
  ds = probs * (torch.einsum("bqhd,bkhd->bhqk", do2, v2) - (do2 * o.double()).sum(-1).transpose(1, 2)[..., None])
  want = [torch.einsum("bhqk,bkhd->bqhd", ds, k2), torch.einsum("bhqk,bqhd->bkhd", ds, q2),
          torch.einsum("bhqk,bqhd->bkhd", probs, do2)]
  if bias:
    want.append(torch.zeros(h, 32, dtype=torch.float64, device="cuda").index_add_(
        1, bucket.flatten(), ds.sum(0).flatten(1)))
  got = _call(q, k, v, o, do, lse, table, lq, lk, *prep[2:5], prep[5], outs)
  for name, a, w in zip(("dq", "dk", "dv", "dbias"), got, want):  # P, dS and the results rounded once, as above
    assert float((a.double() - w).norm() / (w.norm() + 1e-2)) < 4 * 2.0 ** -8, name


def test_both_kernels_are_reached():
  from t5x_b200.ops import native
  covers = native.lib().t5x_attention_bwd_head_covers
  assert covers(128, 12, 512, 512, 64, 32) and covers(8, 6, 64, 64, 64, 32) and covers(64, 12, 114, 512, 64, 0)
  assert not covers(1, 12, 512, 512, 64, 32)  # too few CTAs
  assert covers(16, 12, 1024, 1024, 64, 32) == 2 and not covers(16, 12, 1024, 1300, 64, 32)
  assert not covers(128, 12, 512, 512, 128, 32) and not covers(128, 12, 512, 700, 64, 32)
  assert not covers(128, 12, 512, 512, 64, 300)
  # without a bias the kernel by key blocks is the faster one for longer
  assert covers(8, 6, 1024, 1024, 64, 32) == 2 and not covers(8, 6, 1024, 1024, 64, 0)
  assert covers(50, 6, 1024, 1024, 64, 32) == 2 and not covers(50, 6, 1024, 1024, 64, 0)
  assert not covers(1, 6, 1100, 300, 64, 32) and not covers(1, 6, 1100, 300, 64, 0)
  assert covers(24, 6, 600, 600, 64, 0) == 2 and not covers(12, 6, 600, 600, 64, 0)


@pytest.mark.parametrize("compiled", [True, False])
def test_the_choice_makes_no_difference(compiled, monkeypatch):
  """A batch that goes to the kernel in parts of 512 queries, projections side by side in one buffer, against its
  examples one by one, which do not."""
  from t5x_b200.ops import attention as A, native
  if not compiled:
    monkeypatch.setattr(native, "host", lambda: None)
  b, l, h = 16, 1024, 12
  covers = native.lib().t5x_attention_bwd_head_covers
  assert covers(b, h, l, l, 64, 32) == 2 and not covers(1, h, l, l, 64, 32)
  g = torch.Generator(device="cuda").manual_seed(0)
  qkv = torch.randn(b, l, 3, h, 64, device="cuda", generator=g).mul_(0.3).bfloat16()
  do = torch.randn(b, l, h, 64, device="cuda", generator=g).bfloat16()
  seg = (torch.arange(l, device="cuda") // 300)[None].expand(b, l).contiguous()
  grads = []
  for rows in ([slice(0, b)], [slice(i, i + 1) for i in range(b)]):
    table = torch.nn.Parameter(torch.linspace(-1, 1, h * 32, device="cuda").view(h, 32))
    parts = []
    for r in rows:
      q, k, v = (qkv[r, :, i].detach().requires_grad_() for i in range(3))
      o = A.flash_attention(q, k, v, bias_table=table, bidirectional=False, causal=True,
                            q_segment_ids=seg[r], kv_segment_ids=seg[r])
      parts.append(torch.autograd.grad(o, (q, k, v, table), do[r]))
    native.check_status()
    grads.append([torch.cat([p[i] for p in parts]) for i in range(3)] + [sum(p[3] for p in parts)])
  for x, y in zip(*grads):  # sums in another order, results rounded to bf16
    assert float((x.float() - y.float()).norm() / y.float().norm()) < 2.0 ** -8
