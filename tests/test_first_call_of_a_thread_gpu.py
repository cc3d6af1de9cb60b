"""A thread whose first touch of the device is a product of this library (autograd's worker in the first
backward pass of a process), each call in a process of its own."""
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SETUP = """
import torch
from t5x_b200.ops import functional as F
x = torch.randn(16, 64, device="cuda").bfloat16()
w = torch.nn.Parameter(torch.randn(64, 64, device="cuda"))
w.bf16, w.main_grad, w.grad_ready = w.detach().bfloat16(), torch.zeros_like(w), False
"""
BACKWARD = """
y = F.linear(x, w)
y.backward(torch.ones_like(y))
want = x.double().t() @ torch.ones(16, 64, device="cuda").double()
assert float((w.main_grad.double() - want).abs().max()) < 16 * 2.0 ** -24 * 64
"""
FORWARD = """
import threading
out = []
def work():
  with torch.no_grad():
    out.append(F.linear(x, w))
torch.cuda.synchronize()
t = threading.Thread(target=work); t.start(); t.join()
want = x.double() @ w.bf16.double()
assert float((out[0].double() - want).norm() / want.norm()) < 2.0 ** -8
"""


@pytest.mark.parametrize("call", [BACKWARD, FORWARD], ids=["backward", "thread"])
def test_first_call(call):
  done = subprocess.run([sys.executable, "-c", SETUP + call], capture_output=True, text=True, timeout=300)
  assert done.returncode == 0, done.stderr[-2000:]
