"""Kernels of the decode step for few rows, and a greedy decode of few sentences against the same
sentences in a larger batch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emb,heads,mlp", [(256, 4, 512), (256, 32, 1024), (768, 12, 2048)])
@pytest.mark.parametrize("few", [1, 4, 9])
def test_a_sentence_does_not_depend_on_its_batch(emb, heads, mlp, few):
  """The products of a step add up in one order whatever the number of rows (up to one tile of 128),
  and so does the attention in both of its forms (32 heads: wide for few rows, narrow for 80). So
  the logits of a sentence are the same bit by bit alone and in a batch of 80, and no near-tie
  between two tokens is decided by who else is decoded."""
  from t5x_b200 import decoding_fast
  from t5x_b200.models.t5 import network
  torch.manual_seed(emb + heads)
  cfg = network.T5Config(vocab_size=512, dtype="bfloat16", emb_dim=emb, num_heads=heads, head_dim=64,
                         num_encoder_layers=1, num_decoder_layers=3, mlp_dim=mlp,
                         mlp_activations=("gelu", "linear"), dropout_rate=0.0)
  module = network.Transformer(cfg, device="cuda")
  for p in module.parameters():
    p.bf16 = p.detach().bfloat16()
  enc = torch.randint(2, 512, (80, 19), device="cuda")
  steps = []
  tokens = torch.zeros(80, 1, 41, dtype=torch.long, device="cuda")
  tokens[:, :, 1:] = torch.randint(2, 512, (80, 1, 40), device="cuda")
  for n in (few, 80):
    d = decoding_fast.GraphBeamDecoder(module, n, 1, 40, 1, use_graph=False)
    with torch.no_grad():
      d._encode(enc[:n])
      d._reset()
      d.live_seqs.copy_(tokens[:n])
      logits = []
      for t in range(40):
        d.cur.fill_(t)
        logits.append(d._model_step()[:few].clone())
    steps.append(torch.stack(logits))
  assert torch.equal(steps[0], steps[1])


@pytest.mark.parametrize("batch,beams", [(1, 1), (5, 1), (7, 2), (16, 4)])
def test_steps_launched_one_by_one(batch, beams):
  """Without a captured graph a step follows the search's kernels on the stream: its first kernel starts a
  chain of its own, so that no kernel of the step reads the position, the ancestry or the caches before
  they are written. Chained and not, the search is the same bit by bit, whenever it is run."""
  from t5x_b200 import decoding_fast
  from t5x_b200.models.t5 import network
  from t5x_b200.ops import native
  torch.manual_seed(batch)
  cfg = network.T5Config(vocab_size=512, dtype="bfloat16", emb_dim=256, num_heads=4, head_dim=64,
                         num_encoder_layers=1, num_decoder_layers=2, mlp_dim=512,
                         mlp_activations=("gelu", "linear"), dropout_rate=0.0)
  module = network.Transformer(cfg, device="cuda")
  for p in module.parameters():
    p.bf16 = (p.detach() * (20 if p.dim() == 2 and p.shape[1] == 512 else 1)).bfloat16()
  enc = torch.randint(2, 512, (batch, 23), device="cuda")
  plain = decoding_fast.GraphBeamDecoder(module, batch, beams, 40, 1, use_graph=False)
  plain.chain_level = 0
  want = plain.decode(enc)
  chained = decoding_fast.GraphBeamDecoder(module, batch, beams, 40, 1, use_graph=False)
  assert chained.chain_level == 2
  for _ in range(4):
    got = chained.decode(enc)
    native.check_status()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("rows,beams,heads", [(1, 1, 1), (6, 2, 5), (64, 4, 37), (64, 4, 38), (80, 1, 32)])
def test_self_attention_in_a_chain_and_by_itself(rows, beams, heads):
  """The wide and the narrow form (more than 16 items an SM), each in a chain of launches and by itself: the
  same sums in the same order, against float64 too (probabilities in fp32, one rounding to bf16)."""
  from t5x_b200 import decoding_fast
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(rows + heads)
  n = 67
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  qkv = rnd(rows, 3, heads, 64).bfloat16()
  history = [rnd(rows // beams, beams, heads, n, 64).bfloat16() for _ in range(2)]
  anc = torch.randint(0, beams, (rows // beams, beams, n), device="cuda", generator=g, dtype=torch.int32)
  bias = rnd(heads, n)
  for cur in (0, 3, 4, 31, 32, 33, 66):
    at = torch.tensor([cur], dtype=torch.int32, device="cuda")
    results = []
    for level in (0, 2):
      ck, cv = (t.clone() for t in history)
      out = torch.empty(rows, heads, 64, dtype=torch.bfloat16, device="cuda")
      torch.cuda.synchronize()  # (a chain starts where all before it has completed)
      with native.chained_launches(level):
        decoding_fast.decode_self_attention(qkv[:, 0], qkv[:, 1], qkv[:, 2], ck, cv, anc, bias, at, out, beams)
      results.append((out, ck, cv))
    for a, b in zip(*results):
      assert torch.equal(a, b)
    out, ck, cv = (t.double() for t in results[0])
    slot = anc.long().clone()
    slot[:, :, cur] = torch.arange(beams, device="cuda")  # the new key and value lie in the row's own slot
    pick = lambda c: c.transpose(2, 3).gather(1, slot[..., None, None].expand(-1, -1, -1, heads, 64))
    k, v = (pick(c)[:, :, :cur + 1].flatten(0, 1) for c in (ck, cv))
    s = torch.einsum("rhd,rthd->rht", qkv[:, 0].double(), k) + bias[:, :cur + 1].double()
    want = torch.einsum("rht,rthd->rhd", torch.softmax(s, -1), v)
    assert float((out - want).norm() / want.norm()) < 2.0 ** -8


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
