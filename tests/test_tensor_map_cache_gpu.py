"""The cache of tensor maps is cleared when it is full (65536 maps): by another thread, or between two maps of
one call. A call's maps are its own copies, so its result does not change."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _fill(stop, count, address):
  """Encodes map after map without a launch: products whose second operand is refused (misaligned)."""
  from t5x_b200.ops import native
  l, v = native.lib(), native.c_void_p
  torch.cuda.set_device(0)
  while not stop.is_set() and count[0] < 4 * 65536:
    for _ in range(256):
      address += 16  # (each call's first operand is a map of its own)
      rc = l.t5x_gemm_bf16(v(address), v(8), None, v(1 << 20), 64, 64, 64, 1, 64, 64, 64, 0, 0, 0, 0, 0, 0, 0,
                           0, None, 0, 0, None, None, 0, native.c_float(1.0), 0, None)
      assert rc != 0
    count[0] += 256


def test_results_while_the_cache_is_cleared():
  from t5x_b200.ops import attention, native
  g = torch.Generator(device="cuda").manual_seed(0)
  pool = torch.randn(64, 3, 2, 160, 2, 64, device="cuda", generator=g).bfloat16()
  a = torch.randn(32, 128, 256, device="cuda", generator=g).bfloat16()
  w = torch.randn(256, 256, device="cuda", generator=g).bfloat16()

  def results(i):
    q, k, v = pool[i % 64]
    with torch.no_grad():
      o = attention.flash_attention(q * 0.125, k, v)
    return o, native.gemm(a[i % 32], w), native.gemm_skinny(a[i % 32], w)

  want = [results(i) for i in range(64)]
  native.check_status()
  stop, count = threading.Event(), [0]
  room = torch.empty(16 << 20, dtype=torch.uint8, device="cuda")  # 4 x 65536 maps, 16 bytes apart
  thread = threading.Thread(target=_fill, args=(stop, count, room.data_ptr()))
  thread.start()
  try:
    i = 0
    while thread.is_alive():
      for x, y in zip(results(i), want[i % 64]):
        assert torch.equal(x, y)
      i += 1
  finally:
    stop.set()
    thread.join()
  native.check_status()
  assert count[0] >= 3 * 65536 and i > 10
