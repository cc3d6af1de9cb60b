import gc
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def pytest_configure(config):
  config.addinivalue_line("markers", "gpu: needs a CUDA device (run on a B200 box)")


@pytest.fixture(autouse=True)
def _reset_parallel_state():
  from t5x_b200.parallel import state as pstate
  pstate.reset()
  yield
  pstate.reset()


@pytest.fixture(autouse=True, scope="module")
def _no_garbage_of_other_modules():
  """Decoders and optimizers of earlier tests hold device memory in reference cycles; freed in the middle of
  a test that measures what is allocated, they change its figure."""
  gc.collect()
  yield
