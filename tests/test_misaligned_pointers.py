"""Kernels that access 8 or 16 bytes at a time refuse pointers that are not aligned so, before any launch. The
addresses here are made up: on the device such a call would be a misaligned access."""
import ctypes

import pytest

A = 1 << 20  # aligned


def _calls(lib):
  norm_tail = (4, 64, ctypes.c_float(1e-6), ctypes.c_void_p(0))
  return {
      "rmsnorm_fwd": (lib.t5x_rmsnorm_fwd, [A] * 4, [0, 1, 2], norm_tail),
      "rmsnorm_bwd": (lib.t5x_rmsnorm_bwd, [A] * 8, [0, 1, 2, 4, 5, 7], (4, 64, 0)),
      "gated_gelu_bwd": (lib.t5x_gated_gelu_bwd, [A] * 2, [0, 1], (4, 64, 128, 64, 0, 0)),
      "embedding_fwd": (lib.t5x_embedding_fwd, [A] * 3, [1, 2], (4, 64, 0, 8, 0)),
      "embedding_bwd": (lib.t5x_embedding_bwd, [A] * 3, [1], (4, 64, 0, 8, 0)),
      "cast": (lib.t5x_cast_f32_bf16, [A] * 2, [0, 1], (4, 64, 64, 64, 0)),
      "f32_to_bf16_residual": (lib.t5x_f32_to_bf16_residual, [A] * 3, [0, 1, 2], (64, 0)),
      "f32_to_bf16_residual_clear": (lib.t5x_f32_to_bf16_residual_clear, [A] * 3, [0, 1, 2], (64, 0)),
      "finish_residual_rmsnorm": (lib.t5x_finish_residual_rmsnorm, [A] * 5, [0, 1, 2, 3, 4], norm_tail),
  }


NAMES = ["rmsnorm_fwd", "rmsnorm_bwd", "gated_gelu_bwd", "embedding_fwd", "embedding_bwd", "cast",
         "f32_to_bf16_residual", "f32_to_bf16_residual_clear", "finish_residual_rmsnorm"]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("off", [2, 4])
def test_refused(name, off):
  from t5x_b200.ops import native
  call, pointers, checked, tail = _calls(native.lib())[name]
  for i in checked:
    moved = list(pointers)
    moved[i] += off
    assert call(*map(ctypes.c_void_p, moved), *tail) != 0
    assert "aligned" in native.lib().t5x_last_error().decode()
