"""Embedding gradient: chunks of 1 to 128 tokens, remainders, ids that repeat within and across
chunks, ids outside a vocabulary slice, a table off the 16-byte grid. fp32 sums of at most
`tokens` bf16 terms: the bound is tokens * 2^-24 of their magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,d,vocab,offset", [
    (1, 8, 5, 0), (15, 24, 3, 0), (17, 1032, 7, 1), (8191, 64, 40, 0), (8192, 520, 1000, 0),
    (8333, 8, 2, 1), (600, 64, 30, 0), (1187, 1032, 9, 1), (4740, 32, 700, 0), (75800, 16, 50, 0)])
def test_embedding_bwd(tokens, d, vocab, offset):
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(tokens)
  ids = torch.randint(0, vocab, (tokens,), device="cuda", generator=g)
  ids[tokens // 2:] = ids[0].item()  # a hot id
  dout = torch.randn(tokens, d, device="cuda", generator=g).bfloat16()
  start = 1 if vocab > 3 else 0
  rows = vocab - start - (1 if vocab > 4 else 0)
  buf = torch.randn(rows * d + 4, device="cuda", generator=g)
  table = buf[offset:offset + rows * d].view(rows, d)
  want = table.double().clone()
  own = (ids >= start) & (ids < start + rows)
  want.index_add_(0, (ids - start)[own], dout.double()[own])
  native.embedding_bwd_(ids, dout, table, vocab_start=start)
  torch.testing.assert_close(table.double(), want, rtol=0, atol=tokens * 2 ** -24 * 8 + 1e-6)
