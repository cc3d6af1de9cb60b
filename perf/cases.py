"""Performance cases: what users of this framework run, through its public entry points.

A case is one pass of a model of this repository's own sizes over a synthetic batch:

* job "train":  `trainer.train_with_lr` (forward, backward, Adafactor); returns the loss, the
  updated fp32 weights and, for the smallest stacks, the gradients;
* job "grads":  `trainer.accumulate_grads_microbatched` (forward and backward: what gradient
  accumulation and fine-tuning loops call); returns the loss and every gradient;
* job "score":  `model.score_batch` (forward only: evaluation and re-ranking); returns
  sequence and token log-likelihoods;
* job "decode": `model.predict_batch_with_aux` (encoder, then beam search step by step);
  returns the tokens and their score.

Layer counts are cut where a full stack would only repeat the same layers.
"""
import math

import torch
import torch.nn.functional as TF

# name: (emb, heads, head_dim, mlp, mlp activation, logits tied to the embedding, vocabulary)
SIZES = {
    "small": (512, 6, 64, 1024, "gated", False, 32128),        # T5.1.1 / mT5 small
    "base": (768, 12, 64, 2048, "gated", False, 32128),        # T5.1.1 base
    "large": (1024, 16, 64, 2816, "gated", False, 32128),      # T5.1.1 large
    "xl": (2048, 32, 64, 5120, "gated", False, 32128),         # T5.1.1 XL
    "xxl": (4096, 64, 64, 10240, "gated", False, 32128),       # T5.1.1 XXL
    "base_1_0": (768, 12, 64, 3072, "relu", True, 32128),      # T5.1.0 base
    "3b_1_0": (1024, 32, 128, 16384, "relu", True, 32128),     # T5.1.0 3B (heads of 128)
    "byt5_small": (1472, 6, 64, 3584, "gated", False, 384),    # ByT5 small (byte vocabulary)
    "lm_base": (768, 12, 64, 2048, "gated", True, 32128),      # decoder-only base
    "switch_base": (768, 12, 64, 2048, "gated", False, 32128),  # Switch base, 8 experts
}
EXPERTS, CAPACITY_FACTOR, AUX_FACTOR, ROUTER_Z_FACTOR = 8, 1.25, 1e-2, 1e-3
Z_LOSS = 1e-4
LEARNING_RATE = 0.01  # constant * rsqrt_decay after 10000 warm-up steps
# Training goes on from this step with these second moments: at step 0 the update of a vector is
# the sign of its gradient, which says nothing about how well a small gradient was computed.
STEP, SECOND_MOMENT = 1000, 1.0
EOS = 1


def _case(job, size, layers, batch, inputs, targets, **kw):
  case = {"job": job, "size": size, "layers": layers, "batch": batch, "inputs": inputs,
          "targets": targets, "packed": False, "dropout": 0.0, "beams": 0}
  case.update(kw)
  return case


def listed():
  cases = [
      # a first run on a laptop-sized config: one small layer pair, short text; launches count
      ("train_small", _case("train", "small", 1, 8, 64, 32)),
      # span-corruption pre-training of T5.1.1 base at its own lengths (512 -> 114)
      ("train_base", _case("train", "base", 2, 128, 512, 114)),
      # one microbatch of the XXL pre-training benchmark (32 sequences)
      ("train_xxl", _case("train", "xxl", 1, 32, 512, 114)),
      # Switch base pre-training: every other feed-forward block is 8 experts
      ("train_switch", _case("train", "switch_base", 2, 64, 512, 114)),
      # fine-tuning of a T5.1.0 checkpoint on packed examples with dropout, odd lengths
      ("grads_packed_1_0", _case("grads", "base_1_0", 2, 24, 509, 131, packed=True, dropout=0.1)),
      # byte-level pre-training: long sequences, tiny vocabulary
      ("grads_bytes", _case("grads", "byt5_small", 2, 16, 1024, 189)),
      # prefix language model, decoder only: bidirectional over the inputs, causal after them
      ("grads_prefix_lm", _case("grads", "lm_base", 2, 16, 768, 256)),
      # summarisation-like fine-tuning of the 3B model: heads of 128, wide feed-forward
      ("grads_3b", _case("grads", "3b_1_0", 1, 8, 1024, 256)),
      # evaluation of a large model: log-likelihoods of given targets
      ("score_xl", _case("score", "xl", 2, 64, 512, 64)),
      # one sentence through the whole small model: latency of a single request
      ("score_one", _case("score", "small", 8, 1, 37, 9)),
      # greedy translation of a few sentences with the whole base model
      ("decode_greedy", _case("decode", "base", 12, 4, 128, 32, beams=1)),
      # beam search over a full batch with XL layers
      ("decode_beam4", _case("decode", "xl", 6, 64, 512, 64, beams=4)),
  ]
  return [dict(name=n, **c) for n, c in cases]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  """A case of the same kinds with sizes spread over the same ranges."""
  limit = _weight(dict(listed()[2]))
  while True:
    job = rng.choice(["train", "train", "grads", "grads", "score", "decode"])
    packed, dropout, beams = False, 0.0, 0
    if job == "decode":
      size = rng.choice(["small", "base", "large", "xl"])
      layers = rng.randint(2, 6 if size == "xl" else 12)
      batch, beams = _log_int(rng, 1, 64), rng.choice([1, 2, 4])
      inputs, targets = _log_int(rng, 17, 512), _log_int(rng, 16, 64)
      if targets * layers > 64 * 6:
        continue
    else:
      size = rng.choice(["small", "base", "large", "xl", "xxl", "base_1_0", "3b_1_0",
                         "byt5_small"] + (["lm_base", "switch_base"] if job != "score" else []))
      layers = 1 if size in ("xxl", "3b_1_0") else 2
      batch = _log_int(rng, 1, 128)
      inputs, targets = _log_int(rng, 37, 1024), _log_int(rng, 9, 256)
      if job == "grads" and size not in ("lm_base", "switch_base"):
        packed = rng.random() < 0.3
        dropout = rng.choice([0.0, 0.0, 0.1])
    case = _case(job, size, layers, batch, inputs, targets, packed=packed, dropout=dropout,
                 beams=beams)
    if size == "switch_base" and batch * min(inputs, targets) < 64:
      continue
    if _weight(case) <= limit:
      return case


# ------------------------------------------------------------------------------------------------
# Work
# ------------------------------------------------------------------------------------------------
def _counts(case):
  """(flops of a forward pass, parameters, weights read by one decode step)."""
  d, h, hd, ff, act, tied, vocab = SIZES[case["size"]]
  b, li, lt, n = case["batch"], case["inputs"], case["targets"], case["layers"]
  inner, mats = h * hd, (3 if act == "gated" else 2)
  attn_w, mlp_w = 4 * d * inner, mats * d * ff
  lm = case["size"] == "lm_base"
  if lm:
    t = b * (li + lt)
    weights = n * (attn_w + mlp_w)
    flops = 2.0 * t * (weights + d * vocab) + n * 4.0 * t * (li + lt) / 2 * inner
    return flops, weights + d * vocab, 0
  te, td = b * li, b * lt
  flops = 2.0 * n * (te * (attn_w + mlp_w) + td * (attn_w + 2 * d * inner + mlp_w) +
                     te * 2 * d * inner)
  flops += 2.0 * td * d * vocab
  flops += 4.0 * n * inner * (te * li + td * lt / 2 + td * li)
  params = n * (3 * attn_w + 2 * mlp_w) + d * vocab * (1 if tied else 2)
  if case["size"] == "switch_base":
    params += 2 * (n // 2) * (EXPERTS - 1) * mlp_w
  step = n * (2 * attn_w - 2 * d * inner + mlp_w) + d * vocab
  return flops, params, step


def work(case):
  d, h, hd, ff, act, tied, vocab = SIZES[case["size"]]
  flops, params, step = _counts(case)
  b, li, lt, n = case["batch"], case["inputs"], case["targets"], case["layers"]
  tokens = 16.0 * b * (li + lt)
  if case["job"] == "train":
    # master weights read and written, bf16 copies read and written, gradients written
    return {"bytes": params * 16.0 + tokens, "flops": 3 * flops}
  if case["job"] == "grads":
    return {"bytes": params * 6.0 + tokens, "flops": 3 * flops}
  if case["job"] == "score":
    return {"bytes": params * 2.0 + tokens, "flops": flops}
  # decode: every step reads the decoder weights, the self-attention cache so far and the
  # cross-attention keys and values of every example
  rows = b * case["beams"]
  kv = 2.0 * 2 * n * h * hd
  per_step = step * 2.0 + kv * (b * li + rows * lt / 2)
  flops += 2.0 * lt * rows * step - 2.0 * b * lt * step
  return {"bytes": lt * per_step + params * 2.0, "flops": max(flops, 0.0)}


def _weight(case):
  w = work(case)
  extra = 5e9 * case["targets"] * case["layers"] if case["job"] == "decode" else 0
  return max(w["bytes"], w["flops"] / 50, extra / 50)


# ------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------
def _names_and_shapes(case):
  """Every parameter's name and shape in the checkpoint layout of the T5 family."""
  d, h, hd, ff, act, tied, vocab = SIZES[case["size"]]
  inner, out = h * hd, []
  mats = ["wi_0", "wi_1"] if act == "gated" else ["wi"]

  def attention(prefix):
    out.extend((f"{prefix}/{m}/kernel", (d, inner)) for m in ("query", "key", "value"))
    out.append((f"{prefix}/out/kernel", (inner, d)))

  def mlp(prefix, sparse):
    if sparse:
      out.append((f"{prefix}/router/router_weights/w/kernel", (d, EXPERTS)))
      out.extend((f"{prefix}/expert/{m}/kernel", (EXPERTS, d, ff)) for m in mats)
      out.append((f"{prefix}/expert/wo/kernel", (EXPERTS, ff, d)))
    else:
      out.extend((f"{prefix}/{m}/kernel", (d, ff)) for m in mats)
      out.append((f"{prefix}/wo/kernel", (ff, d)))

  lm, moe = case["size"] == "lm_base", case["size"] == "switch_base"
  out.append(("decoder/token_embedder/embedding" if lm else "token_embedder/embedding", (vocab, d)))
  for stack in (("decoder",) if lm else ("encoder", "decoder")):
    out.append((f"{stack}/relpos_bias/rel_embedding", (h, 32)))
    for i in range(case["layers"]):
      p = f"{stack}/layers_{i}"
      if stack == "encoder":
        out.append((f"{p}/pre_attention_layer_norm/scale", (d,)))
        attention(f"{p}/attention")
      else:
        out.append((f"{p}/pre_self_attention_layer_norm/scale", (d,)))
        attention(f"{p}/self_attention")
        if not lm:
          out.append((f"{p}/pre_cross_attention_layer_norm/scale", (d,)))
          attention(f"{p}/encoder_decoder_attention")
      out.append((f"{p}/pre_mlp_layer_norm/scale", (d,)))
      mlp(f"{p}/mlp", moe and i % 2 == 1)
    out.append((f"{stack}/{stack}_norm/scale", (d,)))
  if not tied:
    out.append(("decoder/logits_dense/kernel", (d, vocab)))
  return out


def _successors(vocab, seed):
  """next[t]: a random cycle over the ordinary tokens; token 0 starts somewhere on it."""
  g = torch.Generator().manual_seed(seed * 7 + 3)
  cycle = torch.randperm(vocab - 2, generator=g) + 2
  nxt = torch.zeros(vocab, dtype=torch.long)
  nxt[cycle] = torch.roll(cycle, -1)
  nxt[0] = cycle[0]
  return nxt.cuda()


def _weights(case, seed):
  """fp32 weights with the initialisers' statistics (values a bf16 checkpoint can hold)."""
  d, h, hd, ff, act, tied, vocab = SIZES[case["size"]]
  g = torch.Generator(device="cuda").manual_seed(seed * 1000 + 17)
  w = {}
  for name, shape in _names_and_shapes(case):
    x = torch.randn(shape, generator=g, device="cuda")
    if name.endswith("scale"):
      x = 1.0 + 0.1 * x
    elif name.endswith("rel_embedding"):
      x.mul_(0.5)
    elif not name.endswith("embedding"):
      x.mul_(shape[-2] ** -0.5 * (hd ** -0.5 if "/query/" in name else 1.0))
    w[name] = x
  if case["size"] == "switch_base":
    # a trained router sends a token by what it is: its direction is part of the embedding
    emb = w["token_embedder/embedding"]
    u = torch.linalg.qr(torch.randn(d, EXPERTS, generator=g, device="cuda"))[0]
    emb.add_(12.0 * u.t()[torch.arange(vocab, device="cuda") % EXPERTS])
    for name in w:
      if name.endswith("router_weights/w/kernel"):
        w[name] = 0.4 * u + 0.02 * d ** -0.5 * w[name]
  if case["job"] == "decode":
    # as in a trained model some token stands out at every step: each has a successor, far above
    # the rest of the vocabulary together with which it shares the probability; the
    # end-of-sequence token does not come up before the last step
    emb, nxt = w["token_embedder/embedding"], _successors(vocab, seed)
    logits = torch.zeros(vocab, d, device="cuda")
    src = torch.cat([torch.arange(1, device="cuda"), torch.arange(2, vocab, device="cuda")])
    logits.index_add_(0, nxt[src], emb[src])
    w["decoder/logits_dense/kernel"] = (logits.t() * (10.0 / d)).contiguous()
  return {k: v.bfloat16().float() for k, v in w.items()}


def _lengths(b, full, g):
  n = (full * (0.6 + 0.4 * torch.rand(b, generator=g, device="cuda"))).ceil().long()
  n[0] = full
  return n.clamp(1, full)


def _tokens(b, l, lengths, vocab, g):
  """Zipf-like ids (the most frequent one is about 2 % of them), zero after each row's length."""
  u = torch.rand(b, l, generator=g, device="cuda", dtype=torch.float64)
  ids = (2 + (vocab - 2) ** (u ** 0.7) - 1).long().clamp(2, vocab - 1)
  return torch.where(torch.arange(l, device="cuda")[None] < lengths[:, None], ids, 0)


def _segments(b, l, lengths, parts):
  """Segment ids 1..parts over each row's real tokens, and positions inside the segments."""
  pos = torch.arange(l, device="cuda")[None]
  size = (lengths[:, None] + parts - 1) // parts
  seg = torch.where(pos < lengths[:, None], pos // size + 1, 0)
  return seg, torch.where(seg > 0, pos - (seg - 1) * size, 0)


def _batch(case, seed):
  vocab = SIZES[case["size"]][-1]
  b, li, lt = case["batch"], case["inputs"], case["targets"]
  g = torch.Generator(device="cuda").manual_seed(seed * 1000 + 29)
  n_in, n_tg = _lengths(b, li, g), _lengths(b, lt, g)
  if case["size"] == "lm_base":
    l = li + lt
    pos = torch.arange(l, device="cuda")[None]
    target = _tokens(b, l, n_in + n_tg, vocab, g)
    return {"decoder_target_tokens": target,
            "decoder_input_tokens": TF.pad(target, (1, 0))[:, :l].contiguous(),
            "decoder_causal_attention": (pos <= n_in[:, None]).long(),
            "decoder_loss_weights": ((pos >= n_in[:, None]) & (target > 0)).float()}
  batch = {"encoder_input_tokens": _tokens(b, li, n_in, vocab, g)}
  if case["job"] == "decode":
    batch["decoder_input_tokens"] = torch.zeros(b, lt, dtype=torch.long, device="cuda")
    return batch
  target = _tokens(b, lt, n_tg, vocab, g)
  shifted = TF.pad(target, (1, 0))[:, :lt]
  if case["packed"]:
    batch["encoder_segment_ids"], batch["encoder_positions"] = _segments(b, li, n_in, 3)
    seg, pos = _segments(b, lt, n_tg, 3)
    batch["decoder_segment_ids"], batch["decoder_positions"] = seg, pos
    shifted = torch.where(pos > 0, shifted, 0)
  batch.update(decoder_target_tokens=target, decoder_input_tokens=shifted.contiguous(),
               decoder_loss_weights=(target > 0).float())
  return batch


def prepare(case, seed):
  from t5x_b200 import adafactor, models, train_state as train_state_lib, trainer
  from t5x_b200.data import vocabularies
  from t5x_b200.parallel import state as parallel_state
  from t5x_b200.utils import tree as tree_utils
  d, h, hd, ff, act, tied, vocab = SIZES[case["size"]]
  if parallel_state.get().device.type != "cuda":
    torch.cuda.set_device(0)
    parallel_state.setup_mesh(1)
  dev = torch.device("cuda", torch.cuda.current_device())
  common = dict(vocab_size=vocab, dtype="bfloat16", emb_dim=d, num_heads=h, head_dim=hd, mlp_dim=ff,
                mlp_activations=("gelu", "linear") if act == "gated" else ("relu",),
                dropout_rate=case["dropout"], logits_via_embedding=tied)
  stacks = dict(num_encoder_layers=case["layers"], num_decoder_layers=case["layers"])
  tokens = vocabularies.PassThroughVocabulary(vocab)
  rules = adafactor.standard_logical_factor_rules()
  if case["size"] == "switch_base":
    from t5x_b200.contrib.moe import adafactor_utils, models as moe_models, network
    opt = adafactor.Adafactor(decay_rate=0.8, step_offset=0,
                              logical_factor_rules=adafactor_utils.logical_factor_rules())
    module = network.Transformer(network.MoeT5Config(
        num_experts=EXPERTS, num_selected_experts=1, train_capacity_factor=CAPACITY_FACTOR,
        sparse_layout="every_other", **stacks, **common), device=dev)
    model = moe_models.MoeEncoderDecoderModel(
        module, tokens, tokens, opt, z_loss=Z_LOSS, aux_loss_factor=AUX_FACTOR,
        router_z_loss_factor=ROUTER_Z_FACTOR)
  elif case["size"] == "lm_base":
    from t5x_b200.models.decoder_only import network
    opt = adafactor.Adafactor(decay_rate=0.8, step_offset=0, logical_factor_rules=rules)
    module = network.DecoderWrapper(network.TransformerConfig(num_layers=case["layers"], **common),
                                    device=dev)
    model = models.DecoderOnlyModel(module, tokens, opt, z_loss=Z_LOSS,
                                    inputs_bidirectional_attention=True)
  else:
    from t5x_b200.models.t5 import network
    opt = adafactor.Adafactor(decay_rate=0.8, step_offset=0, logical_factor_rules=rules)
    module = network.Transformer(network.T5Config(**stacks, **common), device=dev)
    model = models.EncoderDecoderModel(module, tokens, tokens, opt, z_loss=Z_LOSS)
  variables = model.get_initial_variables(
      None, {"decoder_input_tokens": (case["batch"], case["targets"])})
  flat = tree_utils.flatten_dict(variables["params"])
  weights = _weights(case, seed)
  if set(flat) != set(weights):
    raise ValueError(f"parameter names differ: {sorted(set(flat) ^ set(weights))[:6]}")
  with torch.no_grad():
    for name, value in weights.items():
      flat[name].copy_(value)
  del weights
  state = {"case": dict(case), "model": model, "batch": _batch(case, seed), "flat": flat,
           "params": variables["params"]}
  if case["job"] in ("train", "grads"):
    train_state = train_state_lib.FlaxOptimTrainState.create(model.optimizer_def, variables)
    for name, slot in tree_utils.flatten_dict(train_state.param_states).items():
      if name.rsplit("/", 1)[-1] in ("v", "v_row", "v_col"):
        slot.fill_(SECOND_MOMENT)
    state["train_state"] = train_state.replace_step(STEP)
    trainer.attach_compute_buffers(state["train_state"].params)
  else:
    trainer.attach_compute_buffers(variables["params"], main_grad=False)
  return state


def run(state):
  from t5x_b200 import trainer
  from t5x_b200.utils import tree as tree_utils
  case, model, batch = state["case"], state["model"], state["batch"]
  if case["job"] == "decode":
    tokens, aux = model.predict_batch_with_aux(state["params"], batch, num_decodes=case["beams"])
    return {"tokens": tokens, "scores": aux["scores"]}
  if case["job"] == "score":
    sequence, detail = model.score_batch(state["params"], batch, return_intermediates=True)
    return {"sequence": sequence, "tokens": detail["decoder"]["token_scores"][0]}
  # the step's seed draws the dropout masks (no masks without dropout)
  rng = 1234 if case["dropout"] else None
  if case["job"] == "grads":
    grads, metrics, _ = trainer.accumulate_grads_microbatched(model, state["train_state"], batch,
                                                              rng, None)
    return {"loss": metrics["loss"].total, "grads": tree_utils.flatten_dict(grads)}
  state["train_state"], metrics = trainer.train_with_lr(state["train_state"], batch, LEARNING_RATE,
                                                        rng, model, None)
  out = {"loss": metrics["loss"].total, "params": state["flat"]}
  if len(state["flat"]) <= 31:
    out["grads"] = {k: p.main_grad for k, p in state["flat"].items()}
  return out


# ------------------------------------------------------------------------------------------------
# The same in 64 bits
# ------------------------------------------------------------------------------------------------
def _bucket(rel, bidirectional, buckets=32, far=128):
  """The T5 bucket of key position minus query position."""
  base = torch.zeros_like(rel)
  n = -rel
  if bidirectional:
    buckets //= 2
    base, n = (n < 0).long() * buckets, n.abs()
  else:
    n = n.clamp(min=0)
  exact_below = buckets // 2
  eps = torch.finfo(torch.float32).eps
  large = exact_below + (torch.log(n.float() / exact_below + eps) / math.log(far / exact_below) *
                         (buckets - exact_below)).long()
  return base + torch.where(n < exact_below, n, large.clamp(max=buckets - 1))


def _norm(x, scale):
  return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * scale


class _Model64:
  """The network of a case over 64-bit weights `w`."""

  def __init__(self, case, w):
    self.case, self.w = case, w
    (self.d, self.h, self.hd, self.ff, self.act, self.tied, self.vocab) = SIZES[case["size"]]
    self.router_losses = []

  def bias(self, stack, lq, lk, bidirectional):
    rel = torch.arange(lk, device="cuda")[None] - torch.arange(lq, device="cuda")[:, None]
    return self.w[f"{stack}/relpos_bias/rel_embedding"][:, _bucket(rel, bidirectional)]

  def attention(self, p, x, kv, bias, mask):
    b, lq, lk = x.shape[0], x.shape[1], kv.shape[1]
    q = (x @ self.w[f"{p}/query/kernel"]).view(b, lq, self.h, self.hd).transpose(1, 2)
    k = (kv @ self.w[f"{p}/key/kernel"]).view(b, lk, self.h, self.hd).transpose(1, 2)
    v = (kv @ self.w[f"{p}/value/kernel"]).view(b, lk, self.h, self.hd).transpose(1, 2)
    s = q @ k.transpose(2, 3)
    if bias is not None:
      s = s + bias[None]
    o = torch.softmax(s.masked_fill(~mask, -1e10), -1) @ v
    return o.transpose(1, 2).reshape(b, lq, -1) @ self.w[f"{p}/out/kernel"]

  def mlp(self, p, x):
    if f"{p}/router/router_weights/w/kernel" in self.w:
      return self.experts(p, x)
    return self.feed_forward(x, [self.w[f"{p}/{m}/kernel"] for m in
                                 (("wi_0", "wi_1") if self.act == "gated" else ("wi",))],
                             self.w[f"{p}/wo/kernel"])

  def feed_forward(self, x, wi, wo):
    if self.act == "gated":
      return (TF.gelu(x @ wi[0], approximate="tanh") * (x @ wi[1])) @ wo
    return torch.relu(x @ wi[0]) @ wo

  def experts(self, p, x):
    t = x.reshape(-1, self.d)
    n = t.shape[0]
    capacity = max(4, math.ceil(CAPACITY_FACTOR * n / EXPERTS))
    logits = t @ self.w[f"{p}/router/router_weights/w/kernel"]
    probs = torch.softmax(logits, -1)
    choice = probs.argmax(-1)
    used = TF.one_hot(choice, EXPERTS).to(probs.dtype)
    aux = (used.mean(0) * probs.mean(0)).mean() * EXPERTS ** 2
    z = torch.logsumexp(logits, -1).square().mean()
    self.router_losses.append((aux, z))
    y = torch.zeros_like(t)
    for e in range(EXPERTS):
      rows = (choice == e).nonzero()[:capacity, 0]
      out = self.feed_forward(t[rows], [self.w[f"{p}/expert/wi_{i}/kernel"][e] for i in (0, 1)],
                              self.w[f"{p}/expert/wo/kernel"][e])
      y = y.index_add(0, rows, out * probs[rows, e][:, None])
    return y.view(x.shape)

  def stack(self, name, x, mask, bidirectional, cross=None, cross_mask=None):
    l = x.shape[1]
    bias = self.bias(name, l, l, bidirectional)
    first, attn = (("pre_attention_layer_norm", "attention") if name == "encoder" else
                   ("pre_self_attention_layer_norm", "self_attention"))
    for i in range(self.case["layers"]):
      p = f"{name}/layers_{i}"
      y = _norm(x, self.w[f"{p}/{first}/scale"])
      x = x + self.attention(f"{p}/{attn}", y, y, bias, mask)
      if cross is not None:
        y = _norm(x, self.w[f"{p}/pre_cross_attention_layer_norm/scale"])
        x = x + self.attention(f"{p}/encoder_decoder_attention", y, cross, None, cross_mask)
      x = x + self.mlp(f"{p}/mlp", _norm(x, self.w[f"{p}/pre_mlp_layer_norm/scale"]))
    return _norm(x, self.w[f"{name}/{name}_norm/scale"])

  def logits(self, batch):
    dec_in = batch["decoder_input_tokens"]
    b, l = dec_in.shape
    causal = torch.ones(l, l, dtype=torch.bool, device="cuda").tril()[None, None]
    if self.case["size"] == "lm_base":
      emb = self.w["decoder/token_embedder/embedding"]
      inside = batch["decoder_causal_attention"] > 0
      real = batch["decoder_target_tokens"] > 0
      mask = (causal | (inside[:, None, :, None] & inside[:, None, None, :])) & \
          real[:, None, :, None] & real[:, None, None, :]
      x = self.stack("decoder", emb[dec_in], mask, False)
    else:
      emb = self.w["token_embedder/embedding"]
      ids = batch["encoder_input_tokens"]
      enc_mask = (ids > 0)[:, None, None, :]
      cross_mask, dec_mask = enc_mask, causal
      if "decoder_target_tokens" in batch:
        dec_mask = causal & (batch["decoder_target_tokens"] > 0)[:, None, None, :]
      if "encoder_segment_ids" in batch:
        es, ds = batch["encoder_segment_ids"], batch["decoder_segment_ids"]
        enc_mask = enc_mask & (es[:, None, :, None] == es[:, None, None, :])
        cross_mask = cross_mask & (ds[:, None, :, None] == es[:, None, None, :])
        dec_mask = dec_mask & (ds[:, None, :, None] == ds[:, None, None, :])
      enc = self.stack("encoder", emb[ids], enc_mask, True)
      x = self.stack("decoder", emb[dec_in], dec_mask, False, enc, cross_mask)
    if self.tied:
      return (x * self.d ** -0.5) @ emb.t()
    return x @ self.w["decoder/logits_dense/kernel"]


def _adafactor(name, p, g):
  """One Adafactor update from STEP with every second moment at SECOND_MOMENT."""
  decay = 1.0 - (STEP + 1.0) ** -0.8
  ema = lambda m: decay * SECOND_MOMENT + (1.0 - decay) * m
  gsq = g * g + 1e-30
  if p.dim() >= 2 and "rel_embedding" not in name and "router_weights" not in name:
    row, col = ema(gsq.mean(-1, keepdim=True)), ema(gsq.mean(-2, keepdim=True))
    v = row * col / row.mean(-2, keepdim=True)
  else:
    v = ema(gsq)
  dims = (-2, -1) if p.dim() >= 2 else (-1,)  # experts are updated one by one
  y = g * v.rsqrt()
  y = y / y.square().mean(dims, keepdim=True).sqrt().clamp(min=1.0)
  scale = p.square().mean(dims, keepdim=True).sqrt().clamp(min=1e-3)
  return p - LEARNING_RATE * scale * y


def exact(case, seed):
  if case["dropout"]:
    return None  # the masks are the framework's own
  w = {k: v.double() for k, v in _weights(case, seed).items()}
  batch = _batch(case, seed)
  net = _Model64(case, w)
  if case["job"] == "decode":
    if case["batch"] * case["inputs"] > 40000:
      return None
    # the path is known: each token's successor; its score is the sum of log-probabilities
    nxt, path = _successors(net.vocab, seed), [0]
    for _ in range(case["targets"]):
      path.append(int(nxt[path[-1]]))
    ids = torch.tensor(path, device="cuda")[None].expand(case["batch"], -1)
    batch["decoder_input_tokens"] = ids[:, :-1]
    with torch.no_grad():
      lp = torch.log_softmax(net.logits(batch), -1)
    return {"tokens": ids[:, 1:].contiguous(),
            "scores": lp.gather(2, ids[:, 1:, None])[..., 0].sum(-1)}
  target, weight = batch["decoder_target_tokens"], batch["decoder_loss_weights"].double()
  if case["job"] == "score":
    with torch.no_grad():
      lp = torch.log_softmax(net.logits(batch), -1).gather(2, target[..., None])[..., 0] * weight
    return {"sequence": lp.sum(-1), "tokens": lp}
  for v in w.values():
    v.requires_grad_(True)
  logits = net.logits(batch)
  lse = torch.logsumexp(logits, -1)
  token = lse - logits.gather(2, target[..., None])[..., 0] + Z_LOSS * lse.square()
  loss = (token * weight).sum()
  if net.router_losses:
    loss = loss + AUX_FACTOR * torch.stack([a for a, _ in net.router_losses]).mean() + \
        ROUTER_Z_FACTOR * torch.stack([z for _, z in net.router_losses]).mean()
  grads = dict(zip(w, torch.autograd.grad(loss, list(w.values()))))
  out = {"loss": loss.detach()}
  if case["job"] == "grads":
    out["grads"] = grads
    return out
  with torch.no_grad():
    out["params"] = {k: _adafactor(k, w[k].detach(), g) for k, g in grads.items()}
  if len(w) <= 31:
    out["grads"] = grads
  return out


def tolerance(case):
  # bf16 activations and matrix operands with 32-bit sums. Measured against 64 bits: gradients
  # 0.002 to 0.012 (the key projections are the noisiest), token log-likelihoods 0.0005 to 0.001,
  # sums of log-probabilities 0.01; tokens are the same unless two are nearly tied. A single
  # gradient may be further off: a frequent token's row of the embedding gradient is an order of
  # magnitude above the table's root mean square, and its small elements carry the row's error.
  if case["job"] == "decode":
    return {"rel": 3e-2, "max": 0.2, "differ": 2e-3}
  if case["job"] == "score":
    return {"rel": 4e-3, "max": 0.1}
  return {"rel": 3e-2, "max": 0.99}
