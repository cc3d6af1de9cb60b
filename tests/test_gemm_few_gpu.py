"""The product for a handful of rows equals, bit by bit, the kernels for more rows: every cluster size,
rings that hold all of K and rings that wrap, row counts at the edges of the 8-row groups and 32-lane
quarters."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rows(m, k, seed):
  g = torch.Generator(device="cuda").manual_seed(seed)
  return torch.randn(m, k, device="cuda", generator=g).bfloat16()


def _weights(k, width, n, seed):
  g = torch.Generator(device="cuda").manual_seed(seed)
  return [(torch.randn(k, width, device="cuda", generator=g) * k ** -0.5).bfloat16() for _ in range(n)]


@pytest.mark.parametrize("m", [1, 4, 8, 9, 31, 33, 64])
@pytest.mark.parametrize("k,n,splits", [(64, 128, 1), (192, 128, 1), (768, 768, 4), (768, 384, 2),
                                        (2048, 768, 8), (5120, 2048, 4), (512, 512, 8), (4096, 256, 2)])
@pytest.mark.parametrize("with_res", [False, True])
def test_slices_of_a_cluster(m, k, n, splits, with_res):
  from t5x_b200.ops import native
  a, (w,) = _rows(m, k, m), _weights(k, n, 1, k)
  res = _rows(m, n, 5) if with_res else None
  out = native.gemm_few(a, [w], residual=res, splits=splits)
  native.check_status()
  if splits == 1:
    want = native.gemm(a, w, residual=res)
  else:
    want = native.gemm_skinny(a, w, residual=res, splits=splits)
  assert torch.equal(out, want)


@pytest.mark.parametrize("m", [1, 8, 17, 40, 64])
@pytest.mark.parametrize("k,width", [(64, 64), (512, 384), (768, 768), (1024, 1088), (1472, 384), (2048, 2048)])
@pytest.mark.parametrize("kind", ["one", "three", "gated"])
def test_whole_sums(m, k, width, kind):
  from t5x_b200.ops import native
  a, w = _rows(m, k, 3), _weights(k, width, {"one": 1, "three": 3, "gated": 2}[kind], 7)
  out = native.gemm_few(a, w, gated=kind == "gated")
  native.check_status()
  if kind == "gated":
    assert torch.equal(out, native.gemm(a, w[0], b2=w[1]))
  else:
    assert torch.equal(out, torch.cat([native.gemm(a, v) for v in w], dim=1))


def test_strided_operands_and_what_is_not_covered():
  from t5x_b200.ops import native
  big = _rows(6, 2048, 1)
  a = big[:, 512:1280]
  wide = _weights(768, 1024, 1, 2)[0]
  w = wide[:, 256:640]
  res = _rows(6, 1024, 3)[:, 100:484]
  assert torch.equal(native.gemm_few(a, [w], residual=res, splits=2),
                     native.gemm_skinny(a, w, residual=res, splits=2))
  assert native.gemm_few(_rows(65, 768, 1), [wide]) is None          # too many rows
  assert native.gemm_few(a, [wide.t()[:768, :768].t().contiguous().t()]) is None  # other orientation
  assert native.gemm_few(a, [w, wide[:, :256]]) is None              # unequal widths
  assert native.gemm_few(big[:, 1:769], [w]) is None                 # misaligned
  assert native.gemm_few(_rows(2, 96, 1), _weights(96, 64, 1, 1)) is None
  with pytest.raises(native.NativeError):
    native._check(native.lib().t5x_gemm_few_bf16(a.data_ptr(), None, a.data_ptr(), None, 70, 768, 1, 384,
                                                 2048, 1024, 384, 0, 1, 0, 0), "gemm_few")


@pytest.mark.parametrize("chain", [1, 2])
def test_chained_products(chain):
  """A row of dependent products under programmatic launches gives what it gives one by one."""
  from t5x_b200.ops import native
  ws = _weights(768, 768, 12, 5)
  scale = torch.ones(768, device="cuda")

  def run():
    x = _rows(4, 768, 9)
    for i, w in enumerate(ws):
      h = native.gemm_few(native.rmsnorm_fwd(x, scale, 1e-6)[0], [w], splits=4)
      x = native.gemm_few(h, [w], residual=x, splits=4)
    return x

  want = run()
  for _ in range(3):
    with native.chained_launches(chain):
      got = run()
    native.check_status()
    assert torch.equal(got, want)


@pytest.mark.parametrize("batch", [3, 40])
def test_a_captured_step_reads_the_weights_as_they_are(batch):
  """A decoder that was built before the module's weights changed in place decodes with the new ones."""
  from t5x_b200 import decoding_fast
  from t5x_b200.models.t5 import network
  torch.manual_seed(batch)
  cfg = network.T5Config(vocab_size=256, dtype="bfloat16", emb_dim=128, num_heads=2, head_dim=64,
                         num_encoder_layers=1, num_decoder_layers=2, mlp_dim=256,
                         mlp_activations=("gelu", "linear"), dropout_rate=0.0)
  module = network.Transformer(cfg, device="cuda")
  for p in module.parameters():
    p.bf16 = p.detach().bfloat16()
  enc = torch.randint(2, 256, (batch, 19), device="cuda")
  make = lambda: decoding_fast.GraphBeamDecoder(module, batch, 2, 8, 1)
  old = make()
  before = old.decode(enc)[1]
  with torch.no_grad():
    for p in module.parameters():
      p.copy_(torch.randn_like(p) * 0.1 + p)
      p.bf16.copy_(p)
  seqs, scores = old.decode(enc)
  want_seqs, want = make().decode(enc)
  assert torch.equal(seqs, want_seqs) and torch.equal(scores, want) and not torch.equal(scores, before)


@pytest.mark.parametrize("batch", [2, 70])
@pytest.mark.parametrize("what", ["fused", "logits", "embedding", "norm", "parameter", "data"])
def test_weights_put_in_the_place_of_others(what, batch):
  """Working copies that are made anew between two searches (q/k/v moved side by side, a copy gathered from
  other ranks), or parameters and norms replaced: the next search reads them, as a new decoder does."""
  from t5x_b200 import decoding_fast
  from t5x_b200.models.t5 import network
  torch.manual_seed(batch)
  cfg = network.T5Config(vocab_size=256, dtype="bfloat16", emb_dim=128, num_heads=2, head_dim=64,
                         num_encoder_layers=1, num_decoder_layers=2, mlp_dim=256,
                         mlp_activations=("gelu", "linear"), dropout_rate=0.0)
  module = network.Transformer(cfg, device="cuda")
  for p in module.parameters():
    p.bf16 = p.detach().bfloat16()
  enc = torch.randint(2, 256, (batch, 19), device="cuda")
  make = lambda: decoding_fast.GraphBeamDecoder(module, batch, 2, 8, 1)
  old = make()
  before = old.decode(enc)[1]
  assert not old._weights_moved()
  graph = old.graph
  assert torch.equal(old.decode(enc)[1], before) and old.graph is graph
  layer = module.decoder.layers_1
  if what == "fused":
    attn = layer.self_attention
    wide = torch.cat([m.kernel.bf16 for m in (attn.query, attn.key, attn.value)], dim=1)
    for i, m in enumerate((attn.query, attn.key, attn.value)):
      m.kernel.bf16 = wide[:, 128 * i:128 * (i + 1)]
    wide.mul_(1.5)  # (the optimizer writes the new copies)
  elif what == "logits":
    module.decoder.logits_dense.kernel.bf16 = module.decoder.logits_dense.kernel.bf16 * 2
  elif what == "embedding":
    module.token_embedder.embedding.bf16 = module.token_embedder.embedding.bf16 * 2
  elif what == "norm":
    module.decoder.decoder_norm.scale = torch.nn.Parameter(module.decoder.decoder_norm.scale.detach() * 2)
  elif what == "parameter":
    new = torch.nn.Parameter(layer.mlp.wo.kernel.detach() * 2)
    new.bf16 = new.detach().bfloat16()
    layer.mlp.wo.kernel = new
  else:
    layer.mlp.wi_0.kernel.bf16.data = layer.mlp.wi_0.kernel.bf16 * 2
  seqs, scores = old.decode(enc)
  want_seqs, want = make().decode(enc)
  assert torch.equal(seqs, want_seqs) and torch.equal(scores, want) and not torch.equal(scores, before)
