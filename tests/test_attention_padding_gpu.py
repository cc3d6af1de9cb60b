"""Attention over batches with padding: whole blocks of hidden keys (which the kernels pass over), blocks with
one visible key, hidden blocks in the middle, and an example without any visible key (whose rows are
uniform over all keys), against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mask(kind, b, lk):
  m = torch.ones(b, lk, dtype=torch.bool, device="cuda")
  if kind == "tail":
    for i, n in enumerate((lk, max(1, lk // 2), 1, min(lk, 129))):
      m[i, n:] = False
  elif kind == "middle":
    m[1, lk // 4:3 * lk // 4] = False
    m[2, :lk - 1] = False
  elif kind == "none":
    m[1] = False
    m[2, 1:] = False
  return m


@pytest.mark.parametrize("kind", ["tail", "middle", "none"])
@pytest.mark.parametrize("lq,lk,d,bias", [(130, 512, 64, True), (64, 385, 64, False), (200, 700, 64, True),
                                          (600, 600, 64, True), (140, 520, 128, True), (128, 256, 128, False)])
def test_hidden_blocks(kind, lq, lk, d, bias):
  from t5x_b200.ops import attention, native, reference
  g = torch.Generator(device="cuda").manual_seed(lq + lk)
  b, h = 4, 2
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  q = (rnd(b, lq, h, d) * d ** -0.5).bfloat16().requires_grad_()
  k, v = (rnd(b, lk, h, d).bfloat16().requires_grad_() for _ in range(2))
  do = rnd(b, lq, h, d).bfloat16()
  table = torch.nn.Parameter(rnd(h, 32) * 0.5) if bias else None
  mask = _mask(kind, b, lk)
  leaves = [q, k, v] + ([table] if bias else [])
  o = attention.flash_attention(q, k, v, bias_table=table, key_mask=mask)
  grads = torch.autograd.grad(o, leaves, do)
  native.check_status()
  q2, k2, v2 = (t.detach().double().requires_grad_() for t in (q, k, v))
  s = torch.einsum("bqhd,bkhd->bhqk", q2, k2)
  ref_leaves = [q2, k2, v2]
  if bias:
    t2 = table.detach().double().requires_grad_()
    ref_leaves.append(t2)
    rel = torch.arange(lk, device="cuda")[None] - torch.arange(lq, device="cuda")[:, None]
    s = s + t2[:, reference.relative_position_bucket(rel, True, 32, 128)][None]
  # hidden keys take the value -1e10 whatever their score: a row without visible keys is uniform
  s = torch.where(mask[:, None, None, :], s, s * 0 - 1e10)
  want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v2)
  ref = torch.autograd.grad(want, ref_leaves, do.double())
  # probabilities and their gradients are rounded to bf16 once, as is the result
  assert float((o.double() - want).norm() / want.norm()) < 2 * 2.0 ** -8
  seen = mask.any(1)
  for i, (x, y) in enumerate(zip(grads, ref)):
    if i == 3 and kind == "none":
      continue  # (the kernel hands the bias dS of every position, also where no key is visible)
    x, y = (x, y) if i == 3 else (x[seen], y[seen])
    assert float((x.double() - y).norm() / y.norm()) < 3 * 2.0 ** -8
  hidden = ~mask & seen[:, None]
  assert not grads[1][hidden].any() and not grads[2][hidden].any()
  # what padding holds does not reach anything
  with torch.no_grad():
    k3, v3 = k.clone(), v.clone()
    k3[hidden], v3[hidden] = 3.0, -2.0
    assert torch.equal(attention.flash_attention(q, k3, v3, bias_table=table, key_mask=mask), o)


@pytest.mark.parametrize("mode", ["causal", "causal_padded", "causal_packed", "prefix", "prefix_padded",
                                  "prefix_packed"])
@pytest.mark.parametrize("l,d", [(129, 64), (384, 64), (700, 64), (300, 128), (520, 128)])
def test_hidden_query_blocks(mode, l, d):
  """Causal and prefix-LM self-attention over several blocks: those that nothing in a tile sees are passed
  over, but not where a padding query sees no key at all (its row is uniform over all of them)."""
  from t5x_b200.ops import attention, native, reference
  g = torch.Generator(device="cuda").manual_seed(l + d)
  b, h = 3, 2
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  q = (rnd(b, l, h, d) * d ** -0.5).bfloat16().requires_grad_()
  k, v = (rnd(b, l, h, d).bfloat16().requires_grad_() for _ in range(2))
  do = rnd(b, l, h, d).bfloat16()
  table = torch.nn.Parameter(rnd(h, 32) * 0.5)
  pos = torch.arange(l, device="cuda")
  valid = torch.ones(b, l, dtype=torch.bool, device="cuda")
  if mode.endswith("padded"):
    valid[1, l // 2:] = False
    valid[2, 3:] = False
    if not mode.startswith("prefix"):
      valid[2, 0] = False  # the first queries see nothing
  seg = (pos // 100 + 1)[None].expand(b, l).contiguous() if mode.endswith("packed") else None
  mask = (pos[None] <= pos[:, None])[None].expand(b, l, l)
  if mode.startswith("prefix"):
    inside = torch.zeros(b, l, dtype=torch.bool, device="cuda")
    inside[0, :l // 3], inside[1, :l // 4], inside[2, :1] = True, True, True
    prefix = reference.PrefixLMMask(inside, valid, seg)
    mask = prefix.bool()[:, 0]
    kw = dict(prefix_lm=prefix)
  elif mode.endswith("packed"):
    mask = mask & (seg[:, :, None] == seg[:, None, :])
    kw = dict(causal=True, q_segment_ids=seg, kv_segment_ids=seg)
  else:
    mask = mask & valid[:, None, :]
    kw = dict(causal=True, key_mask=valid if mode.endswith("padded") else None)
  o = attention.flash_attention(q, k, v, bias_table=table, bidirectional=False, **kw)
  grads = torch.autograd.grad(o, [q, k, v, table], do)
  native.check_status()
  q2, k2, v2, t2 = (t.detach().double().requires_grad_() for t in (q, k, v, table))
  rel = pos[None] - pos[:, None]
  s = torch.einsum("bqhd,bkhd->bhqk", q2, k2) + \
      t2[:, reference.relative_position_bucket(rel, False, 32, 128)][None]
  s = torch.where(mask[:, None], s, s * 0 - 1e10)
  want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v2)
  ref = torch.autograd.grad(want, [q2, k2, v2, t2], do.double())
  # probabilities and their gradients are rounded to bf16 once, as is the result
  assert float((o.double() - want).norm() / want.norm()) < 2 * 2.0 ** -8
  # (the kernel hands q, k and the bias the dS of rows that see nothing as if they were not masked)
  seen = mask.any(-1).all(-1)
  if bool(seen.all()):
    assert float((grads[3].double() - ref[3]).norm() / ref[3].norm()) < 3 * 2.0 ** -8
  grads, ref = grads[:3], ref[:3]
  for i, (x, y) in enumerate(zip(grads, ref)):
    x, y = (x, y) if i == 2 else (x[seen], y[seen])
    if y.numel():
      assert float((x.double() - y).norm() / y.norm()) < 3 * 2.0 ** -8


@pytest.mark.parametrize("lk,offset", [(1024, 0), (1024, 8), (1040, 0), (5200, 0), (5200, 5), (5121, 0)])
@pytest.mark.parametrize("d", [64, 128])
def test_last_visible_key(lk, offset, d):
  """The last visible key at the edges of the 16 bytes that a thread reads of the mask, of the blocks of 128
  keys and of the part read first; rows of the mask that are and are not aligned."""
  from t5x_b200.ops import attention, native
  g = torch.Generator(device="cuda").manual_seed(lk)
  ends = [1, 15, 16, 17, 128, 129, lk // 2, lk - 1, lk] + [n for n in (5119, 5120, 5121) if n < lk]
  b, lq = len(ends), 130
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  q = (rnd(b, lq, 1, d) * d ** -0.5).bfloat16()
  k, v = (rnd(b, lk, 1, d).bfloat16() for _ in range(2))
  mask = torch.zeros(offset + b * lk, dtype=torch.bool, device="cuda")[offset:].view(b, lk)
  mask.copy_(torch.arange(lk, device="cuda")[None] < torch.tensor(ends, device="cuda")[:, None])
  mask[:, ::3] = False  # holes; of the first examples nothing or one key is left
  with torch.no_grad():
    o = attention.flash_attention(q, k, v, key_mask=mask)
  native.check_status()
  s = torch.einsum("bqhd,bkhd->bhqk", q.double(), k.double())
  s = torch.where(mask[:, None, None, :], s, s * 0 - 1e10)
  want = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), v.double())
  # probabilities and result are each rounded to bf16 once
  for x, y in zip(o.double(), want):
    assert float((x - y).norm() / y.norm()) < 2 * 2.0 ** -8
