"""Flash attention with in-kernel T5 relative-position bias (CUDA path of `functional.attention`).

The kernels read the [heads, buckets] bias table itself and the bucket of every relative offset,
`bucket[(k - q) + Lq - 1]`, which comes from the oracle's own bucket function (so bucket
boundaries are bit-identical); they build the masks from per-token metadata and never
materialise [b, h, q, k] scores. The backward kernel folds the bias gradient into the buckets
and adds it to the table's gradient, in `main_grad` when the table has one. (With the table
expanded per offset by tensor ops, each layer paid an indexing kernel forward and five kernels
backward, 27 to 57 us a layer for the sort-based index backward alone.)
"""
from __future__ import annotations

import functools
import os
from typing import Optional

import torch

from t5x_b200.ops import native
from t5x_b200.ops import reference as ref

c_void_p, c_int, c_ll = native.c_void_p, native.c_int, native.c_ll
for _name in ("t5x_attention_fwd", "t5x_attention_fwd_few"):
  native.register_signature(_name, [c_void_p] * 5 + [c_int] * 4 + [c_ll] * 12 +
                            [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p,
                             c_int, c_int, c_void_p])
native.register_signature("t5x_attention_bwd", [c_void_p] * 10 + [c_int] * 5 + [c_ll] * 18 +
                          [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p,
                           c_void_p, c_int, c_int, c_void_p])

native.register_signature("t5x_attention_fwd_stream", [c_void_p] * 5 + [c_int] * 5 + [c_ll] * 12 +
                          [c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p, c_void_p,
                           c_int, c_int, c_void_p])

native.register_signature("t5x_attention_bwd_head", [c_void_p] * 11 + [c_int] * 4 + [c_ll] * 21 +
                          [c_void_p, c_void_p, c_void_p, c_int, c_int, c_int, c_void_p, c_void_p,
                           c_void_p, c_int, c_int, c_void_p])
native.register_signature("t5x_attention_bwd_head_covers", [c_int] * 6)

# The forward kernel for head_dim 64 keeps the bias by relative position of all keys in shared memory, that for few
# heads the scores of all keys in TMEM.
CLASSIC_MAX_LK, FEW_MAX_LQ, FEW_MAX_LK = 2048, 256, 512
KERNELS = {"stream": 0, "classic": 1, "few": 2}  # as csrc/host/host_ops.cpp has them
# The backward kernel keeps bias-gradient bins for the whole query range in shared memory.
BWD_MAX_LQ = 4096


@functools.lru_cache(maxsize=None)
def _sms() -> int:
  return torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count


def forward_kernel(Lq: int, Lk: int, D: int, prefix_lm: bool = False, heads: int = 0) -> str:
  """'classic' (csrc/attention_fwd_rows_sm100.cu: head_dim 64, up to 2048 keys), 'few'
  (csrc/attention_fwd_few_sm100.cu: `heads`, those of all examples together, leave SMs idle, and the queries
  are one or two of its blocks) or 'stream' (any length, head_dim 64 or 128). `T5X_B200_ATTN_FWD=stream`
  forces the streaming kernel everywhere.

  'few' has a CTA per head, 'classic' two per SM, whose waits fill one another. us, few / classic, key mask and bias:
  128 x 128 queries x keys, 6 heads 7.2 / 8.4, 148 7.1 / 9.1, 156 (a second wave) 13.1 / 10.0; 114 x 512, 6 heads
  12.1 / 16.8, 148 13.2 / 17.3, 156 23.8 / 18.7; 256 x 256, 148 heads 14.3 / 17.8; 257 x 257, three blocks in
  turn against two CTAs, 6 heads 24.1 / 14.0, 148 25.1 / 21.4. Both give the same bits."""
  classic_ok = D == 64 and Lk <= CLASSIC_MAX_LK
  want = os.environ.get("T5X_B200_ATTN_FWD", "classic")
  if not (classic_ok and want == "classic"):
    return "stream"
  few = 0 < heads <= _sms() and Lq <= FEW_MAX_LQ and Lk <= FEW_MAX_LK and not prefix_lm
  return "few" if few else "classic"


def _strides_ok(t: torch.Tensor) -> bool:
  return (t.dim() == 4 and t.stride(3) == 1 and t.stride(0) % 8 == 0 and t.stride(1) % 8 == 0 and
          t.stride(2) % 8 == 0 and t.data_ptr() % 16 == 0)


def flash_supported(q, k, v, explicit_bias, extra_mask) -> bool:
  """True when the sm_100a flash kernels cover this call."""
  prefix_lm = isinstance(extra_mask, ref.PrefixLMMask)
  if prefix_lm and q.shape[1] != k.shape[1]:
    return False
  return (explicit_bias is None and (extra_mask is None or prefix_lm) and
          q.shape[-1] in (64, 128) and q.shape[1] <= BWD_MAX_LQ and q.dtype == torch.bfloat16 and
          k.dtype == torch.bfloat16 and v.dtype == torch.bfloat16)


def _sbh(t):
  return t.stride(0), t.stride(1), t.stride(2)


def _packed_qkv(q, k, v) -> bool:
  """True when q, k, v [B, L, H, D] are the three column blocks of one [B * L, 3 * H * D]
  projection output (a fused q/k/v GEMM): their gradients are then written as the column
  blocks of one buffer too, so that the projection's backward is a single GEMM over it."""
  if q.shape != k.shape or q.shape != v.shape:
    return False
  b, l, h, d = q.shape
  row = 3 * h * d
  want = (l * row, row, d, 1)
  step = h * d * q.element_size()
  return (q.stride() == want and k.stride() == want and v.stride() == want and
          k.data_ptr() == q.data_ptr() + step and v.data_ptr() == q.data_ptr() + 2 * step)


def _bias_sizes(rel_bias, buckets):
  """(number of buckets, number of relative offsets)."""
  return (0, 0) if rel_bias is None else (rel_bias.shape[1], buckets.shape[0])


class _FlashAttentionFn(torch.autograd.Function):

  @staticmethod
  def forward(ctx, q, k, v, rel_bias, buckets, key_mask, q_seg, kv_seg, causal, causal_off,
              rel_off):
    ctx.cfg = (causal, causal_off, rel_off)
    host = native.host()
    if host is not None:
      kernel = forward_kernel(q.shape[1], k.shape[1], q.shape[3], int(causal) == 2, q.shape[0] * q.shape[2])
      done = host.attention(q, k, v, rel_bias, buckets, key_mask, q_seg, kv_seg, int(causal),
                            causal_off, rel_off, KERNELS[kernel])
      if done is not None:
        ctx.save_for_backward(q, k, v, *done, rel_bias, buckets, key_mask, q_seg, kv_seg)
        return done[0]
    q = q if _strides_ok(q) else q.contiguous()
    k = k if _strides_ok(k) else k.contiguous()
    v = v if _strides_ok(v) else v.contiguous()
    B, Lq, H, D = q.shape
    Lk = k.shape[1]
    o = torch.empty((B, Lq, H, D), dtype=torch.bfloat16, device=q.device)
    lse = torch.empty((B, H, Lq), dtype=torch.float32, device=q.device)
    nb, nrel = _bias_sizes(rel_bias, buckets)
    tail = (*_sbh(q), *_sbh(k), *_sbh(v), *_sbh(o), native.ptr(rel_bias), native.ptr(buckets), nb,
            nrel, rel_off, native.ptr(key_mask), native.ptr(q_seg), native.ptr(kv_seg),
            int(causal), causal_off, native.stream_ptr())
    kernel = forward_kernel(Lq, Lk, D, int(causal) == 2, B * H)
    if kernel != "stream":
      fwd = native.lib().t5x_attention_fwd_few if kernel == "few" else native.lib().t5x_attention_fwd
      rc = fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, H, Lq, Lk, *tail)
    else:
      rc = native.lib().t5x_attention_fwd_stream(q.data_ptr(), k.data_ptr(), v.data_ptr(),
                                                 o.data_ptr(), lse.data_ptr(), B, H, Lq, Lk, D,
                                                 *tail)
    native._check(rc, "attention_fwd")
    ctx.save_for_backward(q, k, v, o, lse, rel_bias, buckets, key_mask, q_seg, kv_seg)
    return o

  @staticmethod
  def backward(ctx, do):
    q, k, v, o, lse, rel_bias, buckets, key_mask, q_seg, kv_seg = ctx.saved_tensors
    causal, causal_off, rel_off = ctx.cfg
    d_rel = ret_rel = None  # the buffer the kernel adds to, and what autograd gets
    if rel_bias is not None and ctx.needs_input_grad[3]:
      mg = getattr(rel_bias, "main_grad", None)
      if (mg is not None and mg.dtype == torch.float32 and mg.is_contiguous() and
          mg.shape == rel_bias.shape and mg.device == rel_bias.device):
        if not getattr(rel_bias, "grad_ready", False):
          mg.zero_()
          rel_bias.grad_ready = True
        d_rel = mg
      else:
        d_rel = ret_rel = torch.zeros_like(rel_bias)
    packed = _packed_qkv(q, k, v)
    host = native.host()
    if host is not None:
      done = host.attention_bwd(do, q, k, v, o, lse, rel_bias, buckets, key_mask, q_seg, kv_seg,
                                d_rel, int(causal), causal_off, rel_off, packed)
      if done is not None:
        return (*done, ret_rel, None, None, None, None, None, None, None)
    B, Lq, H, D = q.shape
    Lk = k.shape[1]
    do = do if _strides_ok(do) else do.contiguous()
    nb, nrel = _bias_sizes(rel_bias, buckets)
    head = native.lib().t5x_attention_bwd_head_covers(B, H, Lq, Lk, D, nb)
    if packed:
      dqkv = torch.empty((B, Lq, 3, H, D), dtype=torch.bfloat16, device=q.device)
      dq, dk, dv = dqkv[:, :, 0], dqkv[:, :, 1], dqkv[:, :, 2]
    else:
      dk = torch.empty((B, Lk, H, D), dtype=torch.bfloat16, device=q.device)
      dv = torch.empty((B, Lk, H, D), dtype=torch.bfloat16, device=q.device)
    tail = (native.ptr(rel_bias), native.ptr(buckets), native.ptr(d_rel), nb, nrel, rel_off,
            native.ptr(key_mask), native.ptr(q_seg), native.ptr(kv_seg), int(causal), causal_off,
            native.stream_ptr())
    if head:
      if not packed:
        dq = torch.empty((B, Lq, H, D), dtype=torch.bfloat16, device=q.device)
      # what parts of the queries add to
      wide = [torch.zeros((B, Lk, H, D), dtype=torch.float32, device=q.device) if head == 2 else None
              for _ in range(2)]
      rc = native.lib().t5x_attention_bwd_head(
          q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(),
          dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), *map(native.ptr, wide), B, H, Lq, Lk, *_sbh(q),
          *_sbh(k), *_sbh(v), *_sbh(o), *_sbh(do), *_sbh(dq), *_sbh(dk), *tail)
      native._check(rc, "attention_bwd")
      if head == 2:
        dk.copy_(wide[0])
        dv.copy_(wide[1])
      return dq, dk, dv, ret_rel, None, None, None, None, None, None, None
    dq32 = torch.zeros((B, Lq, H, D), dtype=torch.float32, device=q.device)
    delta = torch.empty((B, H, Lq), dtype=torch.float32, device=q.device)
    rc = native.lib().t5x_attention_bwd(
        q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(),
        delta.data_ptr(), dq32.data_ptr(), dk.data_ptr(), dv.data_ptr(), B, H, Lq, Lk, D,
        *_sbh(q), *_sbh(k), *_sbh(v), *_sbh(o), *_sbh(do), *_sbh(dk), *tail)
    native._check(rc, "attention_bwd")
    if packed:
      dq.copy_(dq32)
    else:
      dq = dq32.to(torch.bfloat16)
    return dq, dk, dv, ret_rel, None, None, None, None, None, None, None


_BUCKET_CACHE: dict = {}


def _rel_buckets(Lq, Lk, q_offset, bidirectional, num_buckets, max_distance, device):
  """Bucket index for every relative offset of an [Lq, Lk] attention: entry t stands for
  (k - q_pos) = t - (Lq - 1) - q_offset. Cached: it depends on the shapes only."""
  key = (Lq, Lk, q_offset, bool(bidirectional), num_buckets, max_distance, str(device))
  b = _BUCKET_CACHE.get(key)
  if b is None:
    rel = torch.arange(Lq + Lk - 1, device=device) - (Lq - 1) - q_offset
    b = ref.relative_position_bucket(rel, bidirectional, num_buckets, max_distance).to(torch.int32)
    if len(_BUCKET_CACHE) > 256:
      _BUCKET_CACHE.clear()
    _BUCKET_CACHE[key] = b
  return b


def _byte_mask(mask: torch.Tensor) -> torch.Tensor:
  """`mask` as contiguous uint8. Where nothing is kept for a backward pass a boolean one is read as
  it is (its bytes are 0 and 1), not copied."""
  if mask.dtype == torch.bool and not torch.is_grad_enabled():
    return mask.contiguous().view(torch.uint8)
  return mask.to(torch.uint8).contiguous()


def flash_attention(q, k, v, *, bias_table: Optional[torch.Tensor] = None,
                    bidirectional: bool = True, num_buckets: int = 32, max_distance: int = 128,
                    key_mask: Optional[torch.Tensor] = None, causal: bool = False,
                    q_segment_ids=None, kv_segment_ids=None, q_offset: int = 0,
                    prefix_lm: Optional["ref.PrefixLMMask"] = None) -> torch.Tensor:
  """q [B,Lq,H,D], k/v [B,Lk,H,D] bf16 -> [B,Lq,H,D], D = 64 or 128. `prefix_lm`: prefix-LM visibility in factored form; it replaces `causal`,
  `key_mask` and the segment ids (which it contains)."""
  B, Lq, H, D = q.shape
  Lk = k.shape[1]
  from t5x_b200.ops import functional
  return functional._apply(_FlashAttentionFn, q, k, v,
                           *prepare(Lq, Lk, H, q.device, bias_table, bidirectional, num_buckets,
                                    max_distance, key_mask, causal, q_segment_ids, kv_segment_ids,
                                    q_offset, prefix_lm))


def prepare(Lq, Lk, H, device, bias_table, bidirectional, num_buckets, max_distance, key_mask, causal,
            q_segment_ids, kv_segment_ids, q_offset=0, prefix_lm=None):
  """What the kernels take beside q, k and v: (bias table, buckets, key mask, query codes, key codes,
  mask mode, its offset, offset of the relative positions)."""
  rel_bias = buckets = None
  if bias_table is not None:
    # an fp32 parameter goes in as it is, so that its gradient buffer is found in backward
    rel_bias = bias_table.float().contiguous()
    if rel_bias.device != device:  # the kernels read it by its address
      raise ValueError(f"bias table on {rel_bias.device}, queries on {device}")
    if rel_bias.shape[0] < H or rel_bias.shape[1] < num_buckets:
      raise ValueError(f"bias table {tuple(rel_bias.shape)}: {H} heads and {num_buckets} buckets are "
                       "indexed")
    buckets = _rel_buckets(Lq, Lk, q_offset, bidirectional, num_buckets, max_distance, device)
  km = _byte_mask(key_mask) if key_mask is not None else None
  qs = q_segment_ids.to(torch.int32).contiguous() if q_segment_ids is not None else None
  ks = kv_segment_ids.to(torch.int32).contiguous() if kv_segment_ids is not None else None
  if qs is None or ks is None:
    qs = ks = None
  mode = int(bool(causal))
  if prefix_lm is not None:
    qs, ks = prefix_lm.token_codes()
    valid = _byte_mask(prefix_lm.valid)
    km = valid if km is None else km & valid
    mode = 2
  return rel_bias, buckets, km, qs, ks, mode, (Lk - Lq) if mode else 0, Lq - 1
