"""The compiled host path and the general Python path run the same kernels on the same operands, so
their results are equal bit by bit (weight gradients: up to the order of atomic adds). Which calls ran
compiled is counted. Forms that the compiled path declines (strided activations and residuals) or is
not asked for (weights partly frozen or without a gradient buffer) give the same answers through
the general path."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _param(*shape, main_grad=True, seed=0):
  g = torch.Generator(device="cuda").manual_seed(seed)
  p = torch.nn.Parameter(torch.randn(*shape, device="cuda", generator=g) * shape[0] ** -0.5)
  p.bf16 = p.detach().bfloat16()
  if main_grad:
    p.main_grad = torch.full_like(p, 5.0)
    p.grad_ready = False
  return p


class _Spy:
  """The compiled path, with how often each function covered a call and how often it declined."""

  def __init__(self, host):
    self.covered, self.declined = {}, {}
    for name in host.NAMES:
      setattr(self, name, self._watch(name, getattr(host, name)))

  def _watch(self, name, fn):
    def call(*args):
      out = fn(*args)
      side = self.declined if out is None else self.covered
      side[name] = side.get(name, 0) + 1
      return out
    return call


def _spy(monkeypatch, host):
  from t5x_b200.ops import native
  spy = _Spy(native.host()) if host else None
  monkeypatch.setattr(native, "host", lambda: spy)
  return spy


def _run(host, case, monkeypatch):
  from t5x_b200.ops import functional as F
  with monkeypatch.context() as m:
    spy = _spy(m, host)
    return _passes(F, case) + (spy,)


def _passes(F, case):
  g = torch.Generator(device="cuda").manual_seed(3)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
  x = rnd(3, 50, 256).requires_grad_()
  xin, mg = x, case != "no_buffer"
  if case == "strided":
    xin = x.transpose(0, 1)
  w = [_param(256, 128 * (i + 2), main_grad=mg, seed=i) for i in range(3)]
  if case == "three_dim":
    w = [_param(256, 4, 32, main_grad=mg, seed=i) for i in range(3)]
  wo, w0, w1, ln = (_param(w[0].numel() // 256, 256, main_grad=mg, seed=7), _param(256, 512, main_grad=mg, seed=8),
                    _param(256, 512, main_grad=mg, seed=9), _param(256, main_grad=mg, seed=10))
  if case == "frozen":
    w[1].requires_grad_(False)
  outs = []
  for _ in range(2):  # the second pass adds to the gradient buffers
    r, h = F.residual_rmsnorm(xin, ln)
    q, k, v = F.multi_linear(h, w)
    y = F.linear(q, wo, residual=r)
    m = F.gated_gelu_mlp_in(F.rmsnorm(y, ln), w0, w1)
    (m.float().square().sum() + k.float().sum() + v.float().sum()).backward()
    outs += [q, k, v, y, m]
  params = w + [wo, w0, w1, ln]
  grads = [p.grad if p.grad is not None else getattr(p, "main_grad", None) for p in params]
  with torch.no_grad():
    outs += [F.linear(F.rmsnorm(xin, ln), w[0])]
  return [o.detach() for o in outs] + [x.grad], [g_ for g_ in grads if g_ is not None]


@pytest.mark.parametrize("case", ["plain", "strided", "three_dim", "frozen", "no_buffer"])
def test_same_as_the_general_path(case, monkeypatch):
  a, ga, spy = _run(True, case, monkeypatch)
  b, gb, _ = _run(False, case, monkeypatch)
  every = {"linear", "multi_linear", "multi_linear_bwd", "gated_in", "gated_in_bwd", "rmsnorm",
           "rmsnorm_bwd"}
  # the calls it declines; everything else ran compiled
  declined = {"rmsnorm", "linear"} if case == "strided" else set()
  assert set(spy.declined) == declined, (spy.covered, spy.declined)
  if case in ("plain", "three_dim"):
    assert set(spy.covered) == every
  elif case == "no_buffer":
    assert set(spy.covered) == every - {"multi_linear_bwd", "gated_in_bwd"}
  assert len(ga) == len(gb)
  for x, y in zip(a, b):
    assert torch.equal(x, y)
  for x, y in zip(ga, gb):
    torch.testing.assert_close(x, y, rtol=1e-5, atol=1e-4 * float(y.abs().max()))


@pytest.mark.parametrize("lq,lk,d,packed,segments", [(130, 70, 64, False, False), (96, 96, 64, True, True),
                                                     (600, 600, 128, False, True)])
def test_attention_same_as_the_general_path(lq, lk, d, packed, segments, monkeypatch):
  from t5x_b200.ops import attention as attn
  g = torch.Generator(device="cuda").manual_seed(lq)
  if packed:
    qkv = torch.randn(2, lq, 3, 2, d, device="cuda", generator=g).bfloat16().requires_grad_()
    q, k, v, leaves = qkv[:, :, 0], qkv[:, :, 1], qkv[:, :, 2], [qkv]
  else:
    leaves = [torch.randn(2, l, 2, d, device="cuda", generator=g).bfloat16().requires_grad_()
              for l in (lq, lk, lk)]
    q, k, v = leaves
  do = torch.randn(2, lq, 2, d, device="cuda", generator=g).bfloat16()
  seg = lambda n: (torch.arange(n, device="cuda") // 40)[None].expand(2, n) if segments else None
  mask = torch.rand(2, lk, device="cuda", generator=g) > 0.2
  res = []
  for host in (True, False):
    with monkeypatch.context() as m:
      spy = _spy(m, host)
      table = torch.nn.Parameter(torch.linspace(-1, 1, 64, device="cuda").view(2, 32))
      o = attn.flash_attention(q, k, v, bias_table=table, key_mask=mask, q_segment_ids=seg(lq),
                               kv_segment_ids=seg(lk))
      res.append([o.detach(), *torch.autograd.grad(o, leaves + [table], do)])
    if host:
      assert spy.covered == {"attention": 1, "attention_bwd": 1} and not spy.declined
  for x, y in zip(*res):
    # dq and the bias gradient are sums of atomic adds, rounded to bf16
    assert float((x - y).float().norm() / y.float().norm()) < 2 ** -8


def test_no_grad_calls_build_no_node():
  """Without gradients the forward runs directly; recording, forward-mode and function
  transforms still go through autograd."""
  from t5x_b200.ops import functional as F
  w = _param(64, 64)
  x = torch.randn(8, 64, device="cuda").bfloat16()
  with torch.no_grad():
    y = F.linear(x, w)
  assert not y.requires_grad
  assert F.linear(x, w).grad_fn is not None and torch.equal(F.linear(x, w), y)
  with torch.no_grad(), torch.autograd.forward_ad.dual_level():
    with pytest.raises(RuntimeError):
      F.linear(torch.autograd.forward_ad.make_dual(x, x), w)
