"""The layered engine's row-wise kernels by the size of a row (csrc/layer_ops.cuh, recurrent_out_kernel): norms with 1, 2, 4 and 8 groups of 1024 channels per
thread, the recurrences' output with 2, 4 and 8 channels of a head per lane and with any number of them, against the oracles."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import gugidra, maxengine, pyconfig, zakelorn
from oracle import gugidra_ref, zakelorn_ref

pytestmark = pytest.mark.gpu

# float32: sums of up to 8192 products of one sign at random, 2^-24 sqrt(8192) = 5e-6 of their size each, a few of them one after the other; bfloat16: the
# bound of the designs' own tests (some ten roundings of 2^-9 along a row)
TOL = {"float32": 3e-5, "bfloat16": 3e-2}
TOKENS = [5, 0, 60, 7, 33]


def error(dtype, got, want):
  got, want = got.cpu().numpy().astype(np.float64), np.asarray(want)
  if dtype == "float32":
    return np.abs(got - want).max() / np.abs(want).max()
  return np.sqrt(((got - want) ** 2).mean() / (want**2).mean())


def logits(model, tensors, dtype):
  cfg = pyconfig.from_model_dict(model, dtype=dtype, per_device_batch_size=2, max_target_length=32, pagedattn_tokens_per_page=8, pagedattn_num_pages=12)
  engine = maxengine.MaxEngine(cfg)
  engine.load_params({k: torch.from_numpy(np.asarray(v)).to(torch.bfloat16) for k, v in tensors.items()})
  engine.init_decode_state()
  return torch.cat([engine.step([(0, TOKENS[:4], [0, 1, 2, 3])]), engine.step([(0, TOKENS[4:], [0])])])


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width", [1024, 1028, 2048, 2052, 4096, 4100, 8192])
def test_norms_of_a_row(width, dtype):
  """Widths at both ends of each number of groups; the loop adds the embedding and a vector to the row in front of its second time."""
  layers = [gugidra.gla_layer(1, 8, 8, mlp=gugidra.dense_ff(16, 2.0)), gugidra.gla_layer(1, 8, 8)]
  model = gugidra.model_dict(width, 61, layers, eps=1e-5, embed_scale=1.7, loop={"start": 0, "stop": 1, "times": 2})
  t = gugidra_ref.random_model(model, seed=width)
  assert error(dtype, logits(model, t, dtype), gugidra_ref.logits_of(model, t, TOKENS)) < TOL[dtype]
  layer = zakelorn.parallel_layer(zakelorn.attention_part(1, 1, 8, window=4, keep_first=1), zakelorn.lightning_part(1, 8, 8), 0.9, 1.2, zakelorn.dense_ff(16))
  model = zakelorn.model_dict(width, 61, [layer], eps=1e-5, embed_scale=3.0)
  t = zakelorn_ref.random_model(model, seed=width)
  assert error(dtype, logits(model, t, dtype), zakelorn_ref.forward(model, t, TOKENS)) < TOL[dtype]


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("vdim", [30, 64, 65, 128, 129, 250, 256, 257, 320])
def test_output_of_a_recurrence(vdim, dtype):
  model = gugidra.model_dict(64, 61, [gugidra.gla_layer(9, 8, vdim)], eps=1e-5, embed_scale=1.7)  # (nine heads: one more than warps)
  t = gugidra_ref.random_model(model, seed=vdim)
  assert error(dtype, logits(model, t, dtype), gugidra_ref.logits_of(model, t, TOKENS)) < TOL[dtype]


@pytest.mark.parametrize("heads,kv,dim,rot", [(4, 2, 64, 32), (2, 1, 16, 16), (8, 4, 256, 256), (16, 4, 128, 0), (16, 16, 64, 64), (3, 1, 96, 48), (4, 2, 64, 12), (2, 2, 48, 24), (32, 8, 128, 64),
                                                (16, 8, 256, 256), (33, 11, 64, 64)])
@pytest.mark.parametrize("rows", [1, 300])
def test_rotated_keys_and_values(heads, kv, dim, rot, rows):
  """Keys (of unit RMS, then rotated) and values of a first layer, appended behind 37 tokens: heads of 64, 128 and 256 channels eight channels per thread, in one
  round of the CTA (512 pieces of eight channels) and in two (768, 1024; 440 leave a warp with queries, keys and values), the others, and where fewer channels turn than that, channel by channel."""
  part = zakelorn.attention_part(heads, kv, dim, rot_dims=rot)
  model = zakelorn.model_dict(256, 320, [zakelorn.parallel_layer(part, zakelorn.lightning_part(2, 64), mlp=zakelorn.dense_ff(256))])
  cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=2, max_target_length=400, pagedattn_tokens_per_page=24, pagedattn_num_pages=40, max_step_rows=400)
  tensors = zakelorn.random_tensors(cfg, seed=3)
  engine = maxengine.MaxEngine(cfg)
  engine.load_params(tensors)
  state = engine.init_decode_state()
  toks = np.random.Generator(np.random.PCG64(5)).integers(0, 320, size=37 + rows).tolist()
  engine.step([(1, toks[:37], [])])
  engine.step([(1, toks[37:], [])])
  pages = torch.as_tensor(engine.page_state.page_map[1], device="cuda").long()
  f64 = lambda t: t.to("cuda", torch.float64)
  x = f64(tensors["embed"].cuda()[toks])
  pos = torch.arange(37 + rows, device="cuda", dtype=torch.float64)
  for name, pool in (("k", "key_pages"), ("v", "value_pages")):
    got = f64(state["cache"][pool][0][:, pages].flatten(1, 2)[:, : 37 + rows]).permute(1, 0, 2)
    want = (x @ f64(tensors["l0.mix.left." + name]).T).reshape(37 + rows, kv, dim)
    if name == "k":
      want = want / torch.sqrt(want.square().mean(-1, keepdim=True) + cfg.normalization_layer_epsilon)
    if name == "k" and rot:
      ang = pos[:, None] * 10000.0 ** (-torch.arange(0, rot, 2, device="cuda", dtype=torch.float64) / rot)[None]
      a, b = want[..., 0:rot:2].clone(), want[..., 1:rot:2].clone()
      co, si = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
      want[..., 0:rot:2], want[..., 1:rot:2] = a * co - b * si, b * co + a * si
    # the projection rounded to bf16 and its rotation again: at most 2^-8 (bf16's unit roundoff) of each value or turned pair, twice
    off = (got - want).square().sum((1, 2)).sqrt() / want.square().sum((1, 2)).sqrt()
    assert float(off.max()) < 2.0**-7


@pytest.mark.parametrize("rows", [1, 70])
@pytest.mark.parametrize("design,heads,kv,dim,rot", [("zakelorn", 4, 2, 64, 32), ("zakelorn", 48, 8, 128, 64), ("zakelorn", 20, 4, 256, 256), ("gugidra", 4, 2, 64, 64), ("gugidra", 8, 2, 96, 32),
                                                     ("gugidra", 48, 8, 128, 128)])
def test_rotated_queries(design, heads, kv, dim, rot, rows):
  """Logits behind 37 tokens against the float32 engine, whose queries come from the kernels of a channel per lane: with norms (zakelorn) and without (gugidra, whose layers call the other
  kernel's instance), in one round of the CTA and in two (queries of more than 4096 channels).  The attention alone feeds the layer, so that a head's query of its own shows in every row."""
  if design == "zakelorn":
    mod, layer = zakelorn, zakelorn.parallel_layer(zakelorn.attention_part(heads, kv, dim, rot_dims=rot), zakelorn.lightning_part(2, 64), 1.0, 0.0, mlp=zakelorn.dense_ff(256))
    model = zakelorn.model_dict(256, 320, [layer])
  else:
    mod, layer = gugidra, gugidra.parallel_layer(heads, kv, dim, 2, 32, 64, mlp=gugidra.dense_ff(256), rot_dims=rot, right_scale=0.0)
    model = gugidra.model_dict(256, 320, [layer])
  toks = np.random.Generator(np.random.PCG64(6)).integers(0, 320, size=37 + rows).tolist()
  out = {}
  for dtype in ("float32", "bfloat16"):
    cfg = pyconfig.from_model_dict(model, dtype=dtype, per_device_batch_size=2, max_target_length=128, pagedattn_tokens_per_page=16, pagedattn_num_pages=20, max_step_rows=80)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(mod.random_tensors(cfg, seed=3))
    engine.init_decode_state()
    engine.step([(0, toks[:37], [])])
    out[dtype] = engine.step([(0, toks[37:], list(range(rows)))]).double()
  # the designs' own bound, over all logits and (twice) in each row
  off = (out["bfloat16"] - out["float32"]).square().mean(1).sqrt() / out["float32"].square().mean().sqrt()
  assert float(off.square().mean().sqrt()) < TOL["bfloat16"] and float(off.max()) < 2 * TOL["bfloat16"]
