"""A layer's blocks as one call against the same layer op by op: equal outputs, gradients equal up to the
order of atomic adds; and what must not take the compiled path does not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(act=("gelu", "linear"), d=256, heads=4, hd=64, mlp=512, buffers=True, seed=0):
  from t5x_b200.models.t5 import network
  torch.manual_seed(seed)
  cfg = network.T5Config(vocab_size=512, dtype="bfloat16", emb_dim=d, num_heads=heads, head_dim=hd,
                         num_encoder_layers=2, num_decoder_layers=2, mlp_dim=mlp, mlp_activations=act,
                         dropout_rate=0.0)
  module = network.Transformer(cfg, device="cuda")
  for p in module.parameters():
    p.bf16 = p.detach().bfloat16()
    if buffers:
      p.main_grad = torch.full_like(p, 7.0)
      p.grad_ready = False
  return module


def _tokens(b, l, seed):
  g = torch.Generator().manual_seed(seed)
  t = torch.randint(2, 512, (b, l), generator=g)
  t[0, l - l // 4:] = 0
  return t.cuda()


def _count(monkeypatch, on):
  """Counts the calls that take the compiled path; with `on` False none does."""
  from t5x_b200.ops import blocks
  taken = []
  for name in ("attention", "gated_mlp"):
    def call(*a, _fn=getattr(blocks, name), _name=name, **k):
      y = _fn(*a, **k) if on else None
      if y is not None:
        taken.append(_name)
      return y
    monkeypatch.setattr(blocks, name, call)
  return taken


def _pass(module, enc, dec, segments=None, passes=2):
  for p in module.parameters():
    p.grad, p.grad_ready = None, False
  kw = dict(enable_dropout=False, return_hidden=True)
  if segments is not None:
    kw.update(encoder_segment_ids=segments, decoder_segment_ids=segments[:, :dec.shape[1]])
  for i in range(passes):  # the second adds to the gradient buffers
    h = module(enc, dec, dec, **kw)
    (h.float() * torch.linspace(-1, 1, h.numel(), device="cuda").view(h.shape)).sum().backward()
  grads = {n: (p.main_grad.clone() if getattr(p, "grad_ready", False) else p.grad)
           for n, p in module.named_parameters()}
  with torch.no_grad():
    y = module(enc, dec, dec, **kw)
  return h.detach(), y, grads


CASES = {
    "plain": dict(), "one_token": dict(lengths=(1, 1)), "long": dict(lengths=(530, 70)),
    "heads_of_128": dict(hd=128, heads=2), "segments": dict(segments=True), "relu": dict(act=("relu",)),
    "narrow_heads": dict(heads=1), "frozen": dict(frozen=True), "no_buffers": dict(buffers=False),
}


@pytest.mark.parametrize("case", CASES)
def test_same_as_op_by_op(case, monkeypatch):
  kw = dict(CASES[case])
  le, ld = kw.pop("lengths", (37, 21))
  segments, frozen = kw.pop("segments", False), kw.pop("frozen", False)
  enc, dec = _tokens(3, le, 1), _tokens(3, ld, 2)
  seg = torch.arange(le, device="cuda")[None].expand(3, le) // 10 if segments else None
  results = []
  for on in (True, False):
    module = _model(**kw)
    if frozen:
      module.encoder.layers_0.attention.key.kernel.requires_grad_(False)
      module.decoder.layers_1.mlp.wo.kernel.requires_grad_(False)
    with monkeypatch.context() as m:
      taken = _count(m, on)
      results.append(_pass(module, enc, dec, seg))
    attn, mlp = taken.count("attention"), taken.count("gated_mlp")
    passes, no_grad = 2, 1
    if not on:
      assert not taken
    elif case == "relu":
      assert (attn, mlp) == (6 * 3, 0)
    elif case == "no_buffers":
      assert (attn, mlp) == (6 * no_grad, 4 * no_grad)
    elif case == "frozen":
      assert (attn, mlp) == (5 * passes + 6 * no_grad, 3 * passes + 4 * no_grad)
    else:
      assert (attn, mlp) == (6 * 3, 4 * 3)
  (h0, y0, g0), (h1, y1, g1) = results
  assert torch.equal(h0, h1) and torch.equal(y0, y1) and torch.equal(h0, y0)
  assert g0.keys() == g1.keys()
  for n in g0:
    if g1[n] is None:
      assert g0[n] is None
      continue
    # sums in fp32 of atomic adds in another order; dq is such a sum rounded to bf16
    assert float((g0[n] - g1[n]).norm() / g1[n].norm().clamp(min=1e-20)) < 2 ** -8, n


def test_hooks_transforms_and_recomputation(monkeypatch):
  enc, dec = _tokens(2, 20, 3), _tokens(2, 12, 4)
  module = _model()
  run = lambda: module(enc, dec, dec, enable_dropout=False, return_hidden=True)
  want = run().detach()
  seen = []
  handles = [m.register_forward_hook(lambda mod, a, out, n=n: seen.append(n))
             for n, m in module.named_modules() if n.endswith(("attention.out", "mlp", "mlp.wo"))]
  with monkeypatch.context() as m:
    taken = _count(m, True)
    assert torch.equal(run(), want)
    assert len(seen) == 6 + 4 + 4 and not taken  # every hook ran
  for h in handles:
    h.remove()
  # saved tensors pass through the hooks of whoever asked for them
  packed = []
  with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t, lambda t: t):
    out = run()
  assert torch.equal(out, want) and len(packed) > 50
  layer, x = module.encoder.layers_0, torch.randn(2, 20, 256, device="cuda").bfloat16().requires_grad_()
  call = lambda t: layer(t, bias_table=module.encoder.relpos_bias.rel_embedding, key_mask=enc > 0)
  grads = []
  for fn in (call, lambda t: torch.utils.checkpoint.checkpoint(call, t, use_reentrant=False)):
    for p in module.parameters():
      p.grad_ready = False
    x.grad = None
    fn(x).float().square().sum().backward()
    grads.append((x.grad.clone(), layer.mlp.wo.kernel.main_grad.clone()))
  for a, b in zip(*grads):
    assert float((a - b).float().norm() / b.float().norm()) < 2 ** -8
  # forward mode has no rule for these ops and says so, as op by op
  with torch.no_grad(), torch.autograd.forward_ad.dual_level():
    with pytest.raises(RuntimeError):
      call(torch.autograd.forward_ad.make_dual(x.detach(), x.detach()))
  # weights that are put in the module's place for one call
  other = {n: p.detach() * 0.5 for n, p in layer.named_parameters()}
  kw = dict(bias_table=module.encoder.relpos_bias.rel_embedding, key_mask=enc > 0)
  with torch.no_grad():
    a = torch.func.functional_call(layer, other, (x,), kw)
    with monkeypatch.context() as m:
      _count(m, False)
      b = torch.func.functional_call(layer, other, (x,), kw)
    assert torch.equal(a, b) and not torch.equal(a, call(x))


def test_gradient_flags_after_an_exception(monkeypatch):
  from t5x_b200.ops import native
  module = _model()
  enc, dec = _tokens(2, 20, 3), _tokens(2, 12, 4)
  loss = module(enc, dec, dec, enable_dropout=False, return_hidden=True).float().sum()
  host = native.host()

  class Broken:
    def __getattr__(self, name):
      if name == "mlp_block_bwd":
        def fail(*a):
          raise native.NativeError("no")
        return fail
      return getattr(host, name)

  monkeypatch.setattr(native, "host", lambda: Broken())
  with pytest.raises(native.NativeError):
    loss.backward()
  mlp = module.decoder.layers_1.mlp
  assert not any(p.grad_ready for p in (mlp.wi_0.kernel, mlp.wi_1.kernel, mlp.wo.kernel))


def test_a_gradient_buffer_that_goes_between_the_passes():
  module = _model()
  enc, dec = _tokens(2, 20, 3), _tokens(2, 12, 4)
  wo = module.decoder.layers_0.mlp.wo.kernel
  grads = []
  for drop in (False, True):
    for p in module.parameters():
      p.grad, p.grad_ready = None, False
    loss = module(enc, dec, dec, enable_dropout=False, return_hidden=True).float().square().sum()
    if drop:
      del wo.main_grad
    loss.backward()
    grads.append(wo.main_grad.clone() if not drop else wo.grad.clone())
  assert float((grads[0] - grads[1]).norm() / grads[0].norm()) < 2 ** -8


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("heads", [2, 6])
@pytest.mark.parametrize("cross", [False, True])
def test_weights_of_another_head_count_are_refused(cross, heads, grad):
  """Weights of 2 or 6 heads in the place of a layer's 4: the bias table was checked for 4."""
  from torch.func import functional_call
  model, other = _model(heads=4), _model(heads=heads)
  if cross:
    layer, prefix = model.decoder.layers_0, "encoder_decoder_attention."
  else:
    layer, prefix = model.encoder.layers_0, "attention."
  source = other.decoder.layers_0 if cross else other.encoder.layers_0
  swapped = {n: p for n, p in source.named_parameters() if n.startswith(prefix)}
  x = torch.randn(2, 9, 256, device="cuda").bfloat16()
  table = (model.decoder if cross else model.encoder).relpos_bias.rel_embedding
  kw = dict(bias_table=table, decoder_key_mask=None, encoder_key_mask=None) if cross else \
      dict(bias_table=table, key_mask=None)
  args = (x, x) if cross else (x,)
  with torch.set_grad_enabled(grad):
    layer(*args, **kw)
    with pytest.raises(RuntimeError, match="shape"):
      functional_call(layer, swapped, args, kw)
