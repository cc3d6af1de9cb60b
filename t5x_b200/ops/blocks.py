"""Residual blocks of a T5 layer (norm, projections, attention or MLP, residual) as one call.

What bounds it: a pass of a small model, or over one sentence, waits for the host. Op by op a block
is five to eight module calls, four or five autograd nodes and as many calls into the library, 20 to
40 us each on the host for kernels of 3 to 8 us. Here a block is one autograd node whose forward and
backward are one compiled call each (csrc/host/host_ops.cpp); without gradients it is the call alone.
The kernels and their order are those of the op by op path, but that of wide enough MLPs the products do the
activation and its gradient themselves. (One sentence scored by T5.1.1 small,
8 + 8 layers: 3.83 ms op by op, 1.97 so, with the cheaper `_owns` of models/base.py; a training step of
one small layer pair 3.48, 2.71.)

Covered is the plain case, everything else takes the op by op path in the layer: bf16 activations on
one GPU (no model axis), no dropout, no decode cache, modules of this package's own classes that
carry no hooks, and either no gradients at all or weights that all have fp32 gradient buffers.
"""
from __future__ import annotations

from typing import Optional

import torch
from torch.nn.modules import module as _module_lib

from t5x_b200.ops import attention as attn_ops
from t5x_b200.ops import functional as F
from t5x_b200.ops import native
from t5x_b200.parallel import state as pstate


def _unhooked(m) -> bool:
  return not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or
              "forward" in m.__dict__)


def _no_global_hooks() -> bool:
  return not (_module_lib._global_forward_hooks or _module_lib._global_forward_pre_hooks or
              _module_lib._global_backward_hooks or _module_lib._global_backward_pre_hooks)


def _kernels(parent, names, dense_cls):
  """The kernels of the projections of `parent`, or None where one is not plain."""
  out = []
  for n in names:
    m = parent._modules.get(n)
    if type(m) is not dense_cls or m.dtype is not torch.bfloat16 or not _unhooked(m):
      return None
    out.append(m._parameters["kernel"])
  return out


def _host_for(x):
  """(the compiled path if blocks may run through it for activations x, else None; whether gradients are
  recorded)."""
  if not (x.is_cuda and x.dtype is torch.bfloat16) or pstate.get().model_size != 1 or \
      F._transformed() or not _no_global_hooks():
    return None, False
  return native.host(), torch.is_grad_enabled()


def _usable_grad(p) -> Optional[torch.Tensor]:
  g = getattr(p, "main_grad", None)
  return g if (p.requires_grad and g is not None and g.dtype is torch.float32 and g.is_contiguous() and
               g.shape == p.shape and g.device == p.device) else None


def _norm_ok(norm, norm_cls) -> bool:
  return type(norm) is norm_cls and norm.dtype is torch.bfloat16 and _unhooked(norm)


def attention(x, kv, norm, attn, norm_cls, attn_cls, dense_cls, *, bias_table=None, bidirectional=True,
              num_buckets=32, max_distance=128, key_mask=None, causal=False, q_segment_ids=None,
              kv_segment_ids=None) -> Optional[torch.Tensor]:
  """x + attention(norm(x)) through the compiled path, or None where it is not covered. `kv`: what the
  keys and values of cross attention are projected from."""
  host, recording = _host_for(x)
  if (host is None or type(attn) is not attn_cls or not _unhooked(attn) or not _norm_ok(norm, norm_cls) or
      attn.dtype is not torch.bfloat16 or attn.scale_attn_logits or attn.head_dim not in (64, 128) or
      x.dim() != 3 or x.shape[1] > attn_ops.BWD_MAX_LQ):
    return None
  params = _kernels(attn, ("query", "key", "value", "out"), dense_cls)
  if params is None:
    return None
  scale = norm._parameters["scale"]
  weights = [F.compute_weight(p, torch.bfloat16) for p in params]
  if not host.attention_block_ok(x, kv, scale, weights, attn.local_heads, attn.head_dim):
    return None
  lq, lk = x.shape[1], (x if kv is None else kv).shape[1]
  masks = attn_ops.prepare(lq, lk, attn.local_heads, x.device, bias_table, bidirectional, num_buckets,
                           max_distance, key_mask, causal, q_segment_ids, kv_segment_ids)
  kernel = attn_ops.KERNELS[attn_ops.forward_kernel(lq, lk, attn.head_dim, masks[5] == 2,
                                                    x.shape[0] * attn.local_heads)]
  if not recording:
    return host.attention_block(x, kv, scale, norm.epsilon, weights, attn.local_heads, attn.head_dim, *masks,
                                kernel)[0]
  grads = [_usable_grad(p) for p in params]
  if any(g is None for g in grads) or _usable_grad(scale) is None or \
      not host.attention_grads_ok(x, kv, weights, grads):
    return None
  return _AttentionBlockFn.apply(x, kv, scale, *params, masks[0], norm.epsilon, attn.local_heads,
                                 attn.head_dim, masks[1:], kernel)


def gated_mlp(x, norm, mlp, norm_cls, mlp_cls, dense_cls) -> Optional[torch.Tensor]:
  """x + mlp(norm(x)) for the gated-GELU MLP, or None where it is not covered."""
  host, recording = _host_for(x)
  if (host is None or type(mlp) is not mlp_cls or mlp.activations != ("gelu", "linear") or
      not _unhooked(mlp) or not _norm_ok(norm, norm_cls) or mlp.dtype is not torch.bfloat16):
    return None
  params = _kernels(mlp, ("wi_0", "wi_1", "wo"), dense_cls)
  if params is None:
    return None
  scale = norm._parameters["scale"]
  weights = [F.compute_weight(p, torch.bfloat16) for p in params]
  if not host.mlp_block_ok(x, scale, weights):
    return None
  if not recording:
    return host.mlp_block(x, scale, norm.epsilon, weights, False)[0]
  grads = [_usable_grad(p) for p in params]
  if any(g is None for g in grads) or _usable_grad(scale) is None or \
      not host.mlp_grads_ok(x, weights, grads):
    return None
  return _GatedMlpBlockFn.apply(x, scale, *params, norm.epsilon)


def relu_mlp(x, norm, mlp, norm_cls, mlp_cls, dense_cls) -> Optional[torch.Tensor]:
  """x + mlp(norm(x)) for the MLP of one ReLU, or None where it is not covered."""
  host, recording = _host_for(x)
  if (host is None or type(mlp) is not mlp_cls or mlp.activations != ("relu",) or
      not _unhooked(mlp) or not _norm_ok(norm, norm_cls) or mlp.dtype is not torch.bfloat16):
    return None
  params = _kernels(mlp, ("wi", "wo"), dense_cls)
  if params is None:
    return None
  scale = norm._parameters["scale"]
  weights = [F.compute_weight(p, torch.bfloat16) for p in params]
  if not host.relu_block_ok(x, scale, weights):
    return None
  if not recording:
    return host.relu_block(x, scale, norm.epsilon, weights, False)[0]
  grads = [_usable_grad(p) for p in params]
  if any(g is None for g in grads) or _usable_grad(scale) is None or \
      not host.relu_grads_ok(x, weights, grads):
    return None
  return _ReluMlpBlockFn.apply(x, scale, *params, norm.epsilon)


class _Buffers:
  """Where a backward pass writes the gradients of `params` (weights first, `extra` small ones after
  them that are added to): their fp32 buffers, or, where a buffer has gone since the forward pass, a
  new tensor that is handed to autograd. On an exception the flags are as they were."""

  def __init__(self, params, extra):
    self.params = list(params) + list(extra)
    self.flags, self.out, self.returned = [], [], []
    for i, p in enumerate(self.params):
      g = _usable_grad(p)
      ready = False
      if g is None:
        g = torch.zeros(p.shape, dtype=torch.float32, device=p.device)
        self.returned.append(g)
      else:
        self.returned.append(None)
        ready = bool(getattr(p, "grad_ready", False))
        p.grad_ready = True
        if i >= len(params) and not ready:
          g.zero_()
      self.flags.append(ready)
      self.out.append(g)

  def weights(self, n):
    return self.out[:n], self.flags[:n]

  def results(self):
    return [None if g is None else g.to(p.dtype) for g, p in zip(self.returned, self.params)]


class _AttentionBlockFn(torch.autograd.Function):

  @staticmethod
  def forward(ctx, x, kv, scale, wq, wk, wv, wo, rel_bias, eps, heads, head_dim, masks, kernel):
    weights = [F.compute_weight(w, torch.bfloat16) for w in (wq, wk, wv, wo)]
    y, *saved = native.host().attention_block(x, kv, scale, eps, weights, heads, head_dim, rel_bias, *masks,
                                              kernel)
    ctx.save_for_backward(x, kv, scale, wq, wk, wv, wo, rel_bias, *masks[:4], *saved)
    ctx.modes = masks[4:]
    return y

  @staticmethod
  def backward(ctx, dy):
    x, kv, scale, wq, wk, wv, wo, rel_bias, *rest = ctx.saved_tensors
    params = [wq, wk, wv, wo]
    want_bias = rel_bias is not None and ctx.needs_input_grad[7]
    flags = [bool(getattr(p, "grad_ready", False)) for p in params + [scale, rel_bias]
             if p is not None]
    done = False
    try:
      buf = _Buffers(params, [scale, rel_bias] if want_bias else [scale])
      grads, accumulate = buf.weights(4)
      dx, dkv = native.host().attention_block_bwd(
          dy.contiguous(), x, kv, scale, [F.compute_weight(w, torch.bfloat16) for w in params], rest[4:],
          grads, accumulate, buf.out[4], buf.out[5] if want_bias else None, bool(ctx.needs_input_grad[1]),
          rel_bias, *rest[:4], *ctx.modes)
      done = True
    finally:
      if not done:
        F._restore_grad_flags([p for p in params + [scale, rel_bias] if p is not None], flags)
    dw = buf.results()
    return (dx, dkv, dw[4], *dw[:4], dw[5] if want_bias else None, None, None, None, None, None)


class _GatedMlpBlockFn(torch.autograd.Function):

  @staticmethod
  def forward(ctx, x, scale, w0, w1, wo, eps):
    weights = [F.compute_weight(w, torch.bfloat16) for w in (w0, w1, wo)]
    y, *saved = native.host().mlp_block(x, scale, eps, weights, True)
    ctx.save_for_backward(x, scale, w0, w1, wo, *saved)
    return y

  @staticmethod
  def backward(ctx, dy):
    x, scale, w0, w1, wo, *saved = ctx.saved_tensors
    saved[3] = F.to_overwrite(saved[3])  # the pre-activations become their gradients
    params = [w0, w1, wo]
    flags = [bool(getattr(p, "grad_ready", False)) for p in params + [scale]]
    done = False
    try:
      buf = _Buffers(params, [scale])
      grads, accumulate = buf.weights(3)
      dx = native.host().mlp_block_bwd(dy.contiguous(), x, scale,
                                       [F.compute_weight(w, torch.bfloat16) for w in params], saved, grads,
                                       accumulate, buf.out[3])
      done = True
    finally:
      if not done:
        F._restore_grad_flags(params + [scale], flags)
    dw = buf.results()
    return (dx, dw[3], *dw[:3], None)


class _ReluMlpBlockFn(torch.autograd.Function):

  @staticmethod
  def forward(ctx, x, scale, wi, wo, eps):
    weights = [F.compute_weight(w, torch.bfloat16) for w in (wi, wo)]
    y, *saved = native.host().relu_block(x, scale, eps, weights, True)
    ctx.save_for_backward(x, scale, wi, wo, *saved)
    return y

  @staticmethod
  def backward(ctx, dy):
    x, scale, wi, wo, *saved = ctx.saved_tensors
    params = [wi, wo]
    flags = [bool(getattr(p, "grad_ready", False)) for p in params + [scale]]
    done = False
    try:
      buf = _Buffers(params, [scale])
      grads, accumulate = buf.weights(2)
      dx = native.host().relu_block_bwd(dy.contiguous(), x, scale,
                                        [F.compute_weight(w, torch.bfloat16) for w in params], saved, grads,
                                        accumulate, buf.out[2])
      done = True
    finally:
      if not done:
        F._restore_grad_flags(params + [scale], flags)
    dw = buf.results()
    return (dx, dw[2], *dw[:2], None)
