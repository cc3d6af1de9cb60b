"""The grouped Adafactor step against the one-parameter-at-a-time kernels: the same arithmetic in
the same order except for the order of atomic adds, so results agree to a few fp32 roundings. Sizes
cover tile remainders, column counts off the 16-byte grid, vectors, stacked parameters, both
orders of the factored dimensions, more parameters than one launch takes, and a sliced bf16 copy."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _params(count):
  shapes = {"a/kernel": (64, 512), "b/kernel": (65, 1028), "c/kernel": (3, 5), "d/scale": (777,),
            "e/rel_embedding": (6, 32), "f/kernel": (2, 33, 70), "g/kernel": (1, 4096)}
  axes = {"a/kernel": ("embed", "mlp"), "b/kernel": ("mlp", "embed"), "c/kernel": ("embed", "mlp"),
          "d/scale": ("embed",), "e/rel_embedding": ("heads", "relpos_buckets"),
          "f/kernel": ("layers", "embed", "mlp"), "g/kernel": ("embed", "mlp")}
  for i in range(count):
    shapes[f"x{i}/kernel"], axes[f"x{i}/kernel"] = (8, 16 + i), ("embed", "mlp")
  g = torch.Generator(device="cuda").manual_seed(count)
  ps = {k: torch.randn(s, device="cuda", generator=g) for k, s in shapes.items()}
  gs = {k: torch.randn(s, device="cuda", generator=g) * 10 ** ((i % 5) - 2)
        for i, (k, s) in enumerate(shapes.items())}
  gs["c/kernel"].zero_()
  return ps, gs, axes


@pytest.mark.parametrize("count,kwargs", [
    (0, {}), (70, dict(weight_decay_rate=0.01)), (3, dict(beta1=0.9, clipping_threshold=None)),
    (3, dict(multiply_by_parameter_scale=False, skip_nan_updates=True))])
def test_group_matches_single(count, kwargs):
  from t5x_b200 import adafactor
  from t5x_b200.utils import tree as tree_utils
  ps, gs, axes = _params(count)
  if kwargs.get("skip_nan_updates"):
    gs["a/kernel"][3, 7] = float("nan")
  results = []
  for grouped in (False, True):
    opt = adafactor.Adafactor(learning_rate=0.1, decay_rate=0.8, step_offset=0,
                              logical_factor_rules=adafactor.standard_logical_factor_rules(),
                              **kwargs)
    params = {k: v.clone() for k, v in ps.items()}
    tree = tree_utils.unflatten_dict(params)
    opt.set_param_axes(tree_utils.unflatten_dict(axes))
    for k, p in params.items():
      p.bf16 = torch.zeros(p.shape, device="cuda", dtype=torch.bfloat16)
    wide = torch.zeros(64, 600, device="cuda", dtype=torch.bfloat16)
    params["a/kernel"].bf16 = wide[:, 8:520]
    state = opt.init_state(tree)
    flat = tree_utils.flatten_dict(state.param_states, is_leaf=adafactor._is_state_leaf)
    for step in range(3):
      items = [(params[k], flat[k], gs[k] * (step + 1), k) for k in params]
      if grouped:
        opt.apply_param_gradients(step, opt.hyper_params, items)
      else:
        for p, s, g, k in items:
          opt.apply_param_gradient(step, opt.hyper_params, p, s, g, k)
    results.append((params, flat))
  (p0, s0), (p1, s1) = results
  for k in p0:
    torch.testing.assert_close(p1[k], p0[k], rtol=2e-5, atol=1e-6, equal_nan=True)
    torch.testing.assert_close(p1[k].bf16, p1[k].bfloat16(), rtol=0, atol=0, equal_nan=True)
    for name in s0[k]:
      torch.testing.assert_close(s1[k][name], s0[k][name], rtol=1e-5, atol=1e-30, equal_nan=True)


@pytest.mark.parametrize("rows,cols,batch", [(256, 512, 1), (1, 7, 1), (33, 1030, 3)])
def test_scratch_is_as_large_as_stated(rows, cols, batch):
  """Nothing is written beyond `scratch_floats()`, and two runs agree bit by bit: the sums that meet
  by atomic adds do so in fp64."""
  from t5x_b200.ops import native
  g = torch.Generator(device="cuda").manual_seed(rows)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
  p0, grad = rnd(batch, rows, cols), rnd(batch, rows, cols)
  vec = rnd(77)
  results = []
  for _ in range(2):
    p, v0, v1 = p0.clone(), torch.ones(batch, rows, device="cuda"), torch.ones(batch, cols, device="cuda")
    q, full = vec.clone(), torch.ones(77, device="cuda")
    items = native.AdafactorItems()
    items.add(p, grad, v0, v1, None, None, 0, 0, batch, rows, cols, True, True)
    items.add(q, vec, full, None, None, None, 0, 0, 1, 1, 77, False, True)
    n = items.scratch_floats()
    scratch = torch.full((n + 64,), 7.0, device="cuda")
    native.adafactor_group_(items, scratch, lr=0.01, decay=0.8, eps1=1e-30, eps2=1e-3,
                            clip_threshold=1.0, weight_decay=0.0, beta1=0.0, max_param_scale=0.0,
                            flags=native.AF_CLIP)
    assert bool((scratch[n:] == 7.0).all())
    results.append((p, v0, v1, q, full))
  for a, b in zip(*results):
    assert torch.equal(a, b) and bool(torch.isfinite(a).all())


def test_scratch_belongs_to_one_stream(monkeypatch):
  """Updates on two streams share no scratch, and a buffer that grows is replaced on its own
  stream only."""
  from t5x_b200 import adafactor
  dev = torch.device("cuda", torch.cuda.current_device())
  monkeypatch.setattr(adafactor, "_SCRATCH", {})
  here = adafactor._scratch(dev, 1000).data_ptr()
  side = torch.cuda.Stream()
  with torch.cuda.stream(side):
    there = adafactor._scratch(dev, 1000).data_ptr()
    grown = adafactor._scratch(dev, 1 << 20)
  assert len({here, there, grown.data_ptr()}) == 3
  assert adafactor._scratch(dev, 1000).data_ptr() == here
