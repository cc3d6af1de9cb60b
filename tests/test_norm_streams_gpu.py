"""Norms' backward passes on several streams at once: each call's partial sums of the scale gradient are its
own."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [512, 1472, 4096])
@pytest.mark.parametrize("path", ["compiled", "general"])
def test_scale_gradients_on_two_streams(d, path, monkeypatch):
  """Against the same calls one after the other (the sums run in one order: equal bit by bit)."""
  from t5x_b200.ops import functional as F
  from t5x_b200.ops import native
  if path == "general":
    monkeypatch.setattr(native, "host", lambda: None)
  g = torch.Generator(device="cuda").manual_seed(d)
  rows, calls = 6000, 6
  data = []
  for _ in range(2):
    x, dy = (torch.randn(rows, d, device="cuda", generator=g).bfloat16() for _ in range(2))
    scale = torch.randn(d, device="cuda", generator=g)
    data.append((x, dy, scale, native.rmsnorm_fwd(x, scale, 1e-6)[1]))

  def work(i):
    x, dy, scale, rstd = data[i]
    out = []
    for _ in range(calls):
      dscale = torch.zeros(d, device="cuda")
      out.append((F._rmsnorm_bwd(dy, x, scale, rstd, None, dscale), dscale))
    return out

  want = [work(0)[0], work(1)[0]]
  torch.cuda.synchronize()
  streams = [torch.cuda.Stream(), torch.cuda.Stream()]
  got = []
  for _ in range(3):
    for i, s in enumerate(streams):
      with torch.cuda.stream(s):
        got.append((i, work(i)))
  torch.cuda.synchronize()
  for i, results in got:
    for dx, dscale in results:
      assert torch.equal(dx, want[i][0]) and torch.equal(dscale, want[i][1])
