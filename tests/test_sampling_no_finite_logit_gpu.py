"""Sampling from rows without a finite logit: the token is one of the vocabulary, and the other rows are what they are
without these."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [7, 1000, 5000])
@pytest.mark.parametrize("temperature,topk,topp", [(0.0, 0, 0.0), (1.0, 0, 0.0), (0.7, 3, 0.0), (1.0, 0, 0.5)])
def test_rows_without_finite_logits(vocab, temperature, topk, topp):
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(vocab)
  x = torch.randn(6, vocab, device="cuda", generator=g) * 2
  kw = dict(temperature=temperature, topk=topk, topp=topp, rescale_log_probs=False, seed=5, stream_id=1)
  want, want_lp = native.sample_tokens(x.clone(), **kw)
  x[1] = float("nan")
  x[4] = float("-inf")
  tok, lp = native.sample_tokens(x, **kw)
  native.check_status()
  assert int(tok.min()) >= 0 and int(tok.max()) < vocab
  rows = [0, 2, 3, 5]
  assert torch.equal(tok[rows], want[rows]) and torch.equal(lp[rows], want_lp[rows])
