"""Decode cross attention over hidden chunks of 32 keys, which are not read: holes, padding, an example without any
visible key (its rows are uniform over all keys), against float64; what the hidden keys hold does not matter."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beams", [1, 4])
@pytest.mark.parametrize("lk", [33, 96, 256, 257, 416, 512, 1000])
@pytest.mark.parametrize("chained", [0, 1])
def test_hidden_chunks(beams, lk, chained):
  from t5x_b200 import decoding_fast
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(lk)
  b, h = 4, 3
  q = (torch.randn(b * beams, h, 64, device="cuda", generator=g) * 0.3).bfloat16()
  k, v = (torch.randn(b, lk, h, 64, device="cuda", generator=g).bfloat16() for _ in range(2))
  mask = torch.ones(b, lk, dtype=torch.uint8, device="cuda")
  mask[0, lk // 3:] = 0
  mask[1, :lk - 1] = 0
  mask[2] = 0
  mask[3, 32:64] = 0
  outs = []
  for fill in (False, True):
    if fill:
      seen = mask.bool().any(1)
      k, v = k.clone(), v.clone()
      k[(mask == 0) & seen[:, None]], v[(mask == 0) & seen[:, None]] = 3.0, -2.0
    kp, vt = decoding_fast.cross_kv_layout(k, v)
    out = torch.empty_like(q)
    torch.cuda.synchronize()
    native.lib().t5x_set_chained_launches(chained)
    try:
      decoding_fast.decode_cross_attention_mma(q, kp, vt, mask, out, beams, lk)
    finally:
      native.lib().t5x_set_chained_launches(0)
    native.check_status()
    outs.append(out)
  assert torch.equal(*outs)
  s = torch.einsum("bjhd,bthd->bhjt", q.double().view(b, beams, h, 64), k.double())
  s = torch.where((mask == 0)[:, None, None], -1e10, s)
  want = torch.einsum("bhjt,bthd->bjhd", torch.softmax(s, -1), v.double()).reshape(outs[0].shape)
  # probabilities and result are each rounded to bf16 once
  assert float((outs[0].double() - want).norm() / want.norm()) < 2 * 2.0 ** -8


@pytest.mark.parametrize("beams", [1, 2, 4, 8])
@pytest.mark.parametrize("lk", [256, 288, 384, 385, 513, 769])
def test_both_forms_give_the_same_bits(beams, lk):
  """On either side of the lines between the form that looks for hidden chunks and the one that does not, which
  chained launches take."""
  from t5x_b200 import decoding_fast
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(lk)
  b, h = 3, 5
  q = (torch.randn(b * beams, h, 64, device="cuda", generator=g) * 0.3).bfloat16()
  k, v = (torch.randn(b, lk, h, 64, device="cuda", generator=g).bfloat16() for _ in range(2))
  mask = torch.ones(b, lk, dtype=torch.uint8, device="cuda")
  mask[0, lk // 2:], mask[1, 40:200] = 0, 0
  kp, vt = decoding_fast.cross_kv_layout(k, v)
  for m in (mask, None):
    outs = []
    for chained in (0, 1):
      outs.append(torch.empty_like(q))
      torch.cuda.synchronize()
      native.lib().t5x_set_chained_launches(chained)
      try:
        decoding_fast.decode_cross_attention_mma(q, kp, vt, m, outs[-1], beams, lk)
      finally:
        native.lib().t5x_set_chained_launches(0)
      native.check_status()
    assert torch.equal(*outs)
