"""The beam step's choice of candidates: logits with many equal entries (more than there is room for: every thread then
keeps its own), hidden ones, chunks that hold fewer than are asked for, against a sort that puts the lower index
first; and examples that hold fewer."""
import pytest
import torch

from tests.test_beam_sampling_gpu import _State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beams", [1, 2, 4, 8])
@pytest.mark.parametrize("kind", ["steps", "equal", "hidden", "peak_at_the_end"])
@pytest.mark.parametrize("vocab", [20, 255, 4096, 8200])
def test_candidates(beams, kind, vocab):
  g = torch.Generator(device="cuda").manual_seed(vocab + beams)
  b, eos, k2 = 3, 1, 2 * beams
  x = torch.randn(b * beams, vocab, device="cuda", generator=g) * 3
  if kind == "steps":  # a hundred equal entries of each height
    x = (x * 2).round() / 2
  elif kind == "equal":
    x.zero_()
  elif kind == "hidden":
    x[:, k2 + 1:] = float("-inf")
  else:
    x[:, -1] += 50.0
  st = _State(b, beams, 6, eos, 0.6, torch.device("cuda"))
  live = torch.randn(b, beams, device="cuda", generator=g).sort(-1).values
  st.d.live_lp.copy_(live)
  st.d._beam_step(x.clone())
  s = st.snapshot()
  lp = torch.log_softmax(x.double(), -1).view(b, beams, vocab) + live[:, :, None].double()
  # heights of one beam are compared as they are: the order inside a row is that of its logits
  flat = lp.view(b, -1)
  order = torch.sort(flat.float(), stable=True, dim=-1, descending=True).indices[:, :k2]
  for i in range(b):
    picks = [int(j) % vocab for j in order[i] if int(j) % vocab != eos][:beams]
    assert s["live_seqs"][i, :, 1].tolist() == picks[::-1], (kind, i)
  got = s["live_lp"].double()
  want = torch.stack([flat[i][[int(j) for j in order[i] if int(j) % vocab != eos][:beams][::-1]] for i in range(b)])
  # 32-bit sums of up to 4096 exponentials, and their logarithm
  torch.testing.assert_close(got, want, rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("beams,vocab", [(1, 37), (4, 300), (4, 9001), (8, 20000)])
@pytest.mark.parametrize("eos", [1, 0])
def test_examples_without_enough_candidates(beams, vocab, eos):
  """An example of NaNs, one with a single finite logit per row and one with none: parents stay among the beams and
  tokens in the vocabulary, and the other examples are what they are by themselves."""
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(vocab)
  dev, b, steps = torch.device("cuda"), 5, 4
  st, alone = _State(b, beams, steps + 2, eos, 0.6, dev), _State(2, beams, steps + 2, eos, 0.6, dev)
  for _ in range(steps):
    x = torch.randn(b, beams, vocab, device="cuda", generator=g) * 3
    x[1] = float("nan")
    x[2, :, 1:] = float("-inf")
    x[3] = float("-inf")
    st.d._beam_step(x.view(b * beams, vocab).clone())
    alone.d._beam_step(x[[0, 4]].view(2 * beams, vocab).clone())
    s, a = st.snapshot(), alone.snapshot()
    for n in ("anc", "live_seqs", "fin_seqs"):
      assert int(s[n].min()) >= 0 and int(s[n].max()) < (beams if n == "anc" else vocab), n
    for n in ("live_seqs", "anc", "fin_seqs", "live_lp", "fin_scores", "fin_flags"):
      assert torch.equal(s[n][[0, 4]], a[n]), n
  assert int(s["cur"]) == steps
  native.check_status()
