"""The pair GEMM (csrc/gemm_wide.cuh) behind steps of more than 256 rows: the bfloat16 engine against the float32 engine, whose projections
are fp32 FMA kernels, with the same weights.  Rows at the edges of the 256-row tiles, output widths that leave the last tile of columns
part empty, and every epilogue that the designs use (bias, clamped and tanh gates, silu columns, gelu, bf16 and fp32 outputs)."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import gugidra, kifusun, ligidra, maxengine, pyconfig, zakelorn

pytestmark = pytest.mark.gpu


def _model(name, width):
  ff = 3 * width // 2
  if name == "kifusun":
    return kifusun, kifusun.model_dict(width, 320, [kifusun.attention_layer(4, 2, 64, 64, 96, ff=ff, bias_max=96.0)] * 2)
  if name == "gugidra":
    return gugidra, gugidra.model_dict(width, 384, [gugidra.parallel_layer(4, 2, 32, 2, 32, 64, mlp=gugidra.dense_ff(ff)), gugidra.gla_layer(4, 32, 64, mlp=gugidra.dense_ff(ff))])
  if name == "ligidra":
    layers = [ligidra.attention_layer(4, 2, 64, window=64, pool=16, mlp=ligidra.moe_ff(4, 4, 128, shared_ff=ff)),
              ligidra.delta_layer(4, 2, 32, 64, mlp=ligidra.moe_ff(4, 4, 128, shared_ff=ff))]
    return ligidra, ligidra.model_dict(width, 384, layers, side_dim=64)
  ffs = [zakelorn.dense_ff(ff), zakelorn.moe_ff(5, 4, 128, identity=1, groups=2, keep=2)]  # unequal experts, slots beyond their ranges
  layers = [zakelorn.parallel_layer(zakelorn.attention_part(4, 2, 64, window=64, keep_first=4), zakelorn.lightning_part(4, 64), mlp=f) for f in ffs]
  return zakelorn, zakelorn.model_dict(width, 384, layers)


def _repeating(name):
  """Models whose every result is the same in steps of any length, but for kifusun's behind the first attention (its key splits go by the number
  of query tiles).  zakelorn's windows are longer than the sequence and its decayed sums, whose chunks go by the run, are left out; 768 rows reach the grouped
  pair GEMM with experts of their own number of rows each, 256 do not."""
  if name == "kifusun":
    return _model(name, 256)
  if name == "gugidra":
    ffs = [gugidra.dense_ff(384), gugidra.moe_ff(5, 1, 128, shared_ff=256)]
    return gugidra, gugidra.model_dict(256, 384, [gugidra.parallel_layer(4, 2, 64, 2, 32, 64, mlp=ffs[0]), gugidra.gla_layer(4, 32, 64, mlp=ffs[1]),
                                                  gugidra.parallel_layer(4, 2, 64, 2, 32, 64, mlp=ffs[1])])
  ffs = [zakelorn.moe_ff(5, 1, 128, identity=1, shared_ff=256), zakelorn.dense_ff(384), zakelorn.moe_ff(3, 1, 64)]
  layers = [zakelorn.parallel_layer(zakelorn.attention_part(4, 2, 64, window=1024, keep_first=4), zakelorn.lightning_part(4, 64), right_scale=0.0, mlp=f) for f in ffs]
  return zakelorn, zakelorn.model_dict(256, 384, layers)


@pytest.mark.parametrize("name", ["kifusun", "gugidra", "zakelorn"])
def test_long_steps_repeat_short_ones(name):
  """A row's bits do not depend on how many rows its step has: 768 rows at once against three steps of 256.  Every layer's keys, and the logits of
  every row."""
  design, model = _repeating(name)
  toks = np.random.Generator(np.random.PCG64(1)).integers(0, model["vocab"], size=768).tolist()
  out = []
  for rows in (768, 256):
    cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=2, max_target_length=800, pagedattn_tokens_per_page=16,
                                   pagedattn_num_pages=60, max_step_rows=rows)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(design.random_tensors(cfg, seed=3))
    state = engine.init_decode_state()
    logits = engine.step([(0, toks, list(range(768)))])
    pages = torch.as_tensor(engine.page_state.page_map[0][:48], device="cuda").long()
    keys = [t[:, pages].clone() for t in state["cache"]["key_pages"]]
    out.append(keys[:1] if name == "kifusun" else keys + [t.clone() for t in state["cache"]["recurrent_state"]] * (name == "gugidra") + [logits])
  assert all(torch.isfinite(t).all() for t in out[0]) and all(torch.equal(a, b) for a, b in zip(*out))


def _blocks_per_stage(rows, n, k):
  """K blocks of a stage for this product of a layered design: plan_rows, wide_tile_columns and wide_group (csrc/host_util.cuh) over again."""
  tiles, kb, parts = -(-n // 128), k // 64, 1
  if 2 * tiles <= 148:
    while parts * 2 <= min(8, kb) and tiles * 2 * parts * 2 <= 148 + 148 // 4:
      parts *= 2
  pairs, row_tiles = torch.cuda.get_device_properties(0).multi_processor_count // 2, -(-rows // 256)
  cost = lambda bn: -(-row_tiles * -(-n // bn) // pairs) * (128 + bn)
  columns = min(range(256, 32, -32), key=cost)  # (of equal costs the widest)
  return 2 if columns <= 128 and kb % (2 * parts) == 0 else 1


@pytest.mark.parametrize("rows", [257, 288, 545, 767])
@pytest.mark.parametrize("width,ff,blocks", [(256, 448, 1), (256, 256, 1), (1024, 1024, 2)])
def test_part_empty_row_tile_repeats_a_whole_one(rows, width, ff, blocks):
  """The last row tile's warps with 32, some and no rows, and feed-forwards with one k block per stage, of an odd number of them (7) and of four, and with two
  (four and eight parts of two blocks and more): bit for bit what the same rows are among 768."""
  assert all(_blocks_per_stage(r, n, k) == blocks for r in (rows, 768) for n, k in ((2 * ff, width), (width, ff)))
  layers = [gugidra.parallel_layer(4, 2, 64, 2, 32, 64, mlp=gugidra.dense_ff(ff)), gugidra.gla_layer(4, 32, 64, mlp=gugidra.dense_ff(ff))]
  model = gugidra.model_dict(width, 384, layers)
  toks = np.random.Generator(np.random.PCG64(4)).integers(0, model["vocab"], size=768).tolist()
  out = []
  for n in (rows, 768):
    cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=2, max_target_length=800, pagedattn_tokens_per_page=16,
                                   pagedattn_num_pages=60, max_step_rows=768)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(gugidra.random_tensors(cfg, seed=3))
    engine.init_decode_state()
    out.append(engine.step([(0, toks[:n], list(range(rows)))]).clone())
  assert torch.isfinite(out[0]).all() and torch.equal(out[0], out[1])


def test_unequal_experts_against_float32():
  """Experts of 0, 1, 255, 256 and 257 rows on the grouped pair GEMM, and slots of an identity expert behind the last range: the token says which
  expert its row takes."""
  counts, ff, width = [0, 1, 255, 256, 257, 100], 128, 256  # (the last: the identity expert)
  rows, experts = sum(counts), len(counts) - 1
  assert rows >= 128 * experts and ff % 64 == 0 and width % 64 == 0  # (takes_wide_grouped)
  layer = zakelorn.parallel_layer(zakelorn.attention_part(4, 2, 64, window=64, keep_first=4), zakelorn.lightning_part(4, 64),
                                  mlp=zakelorn.moe_ff(experts, 1, ff, identity=1, shared_ff=64))
  model = zakelorn.model_dict(width, 384, [layer] * 2)
  toks = np.concatenate([np.full(n, e) + 6 * np.arange(n) % 384 // 6 * 6 for e, n in enumerate(counts)]) % 384
  expert_of = toks % 6
  assert np.bincount(expert_of, minlength=6).tolist() == counts
  toks = np.random.Generator(np.random.PCG64(2)).permutation(toks).tolist()
  out = {}
  for dtype in ("float32", "bfloat16"):
    cfg = pyconfig.from_model_dict(model, dtype=dtype, per_device_batch_size=2, max_target_length=rows + 8, pagedattn_tokens_per_page=16,
                                   pagedattn_num_pages=rows // 16 + 4, max_step_rows=1024)
    tensors = zakelorn.random_tensors(cfg, seed=3)
    embed = next(t for n, t in tensors.items() if "embed" in n and t.shape == (384, width))
    embed[:, :6] = 30.0 * torch.nn.functional.one_hot(torch.arange(384) % 6, 6)  # the stream's first channels name the token's expert
    for n, t in tensors.items():
      if n.endswith("mlp.router"):
        t.zero_()
        t[:, :6] = torch.eye(6)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(tensors)
    engine.init_decode_state()
    out[dtype] = engine.step([(0, toks, list(range(rows)))]).double()
  # bf16 operands (2^-9 each) through two layers, no row's experts near a tie
  off = (out["bfloat16"] - out["float32"]).square().mean(1).sqrt() / out["float32"].square().mean().sqrt()
  assert float(off.max()) < 4e-2


@pytest.mark.parametrize("name", ["kifusun", "gugidra", "ligidra", "zakelorn"])
@pytest.mark.parametrize("width,rows", [(256, 257), (384, 512), (256, 769), (1024, 389)])
def test_long_steps_against_float32(name, width, rows):
  """(1024 wide: the up-projection, for one, has two k blocks per stage.)"""
  assert _blocks_per_stage(rows, 3 * width, width) == (2 if width == 1024 else 1)
  design, model = _model(name, width)
  toks = np.random.Generator(np.random.PCG64(rows)).integers(0, model["vocab"], size=rows).tolist()
  out = {}
  for dtype in ("float32", "bfloat16"):
    cfg = pyconfig.from_model_dict(model, dtype=dtype, per_device_batch_size=2, max_target_length=rows + 8, pagedattn_tokens_per_page=16,
                                   pagedattn_num_pages=rows // 16 + 4, max_step_rows=1024)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(design.random_tensors(cfg, seed=3))
    engine.init_decode_state()
    out[dtype] = engine.step([(0, toks, list(range(rows)))]).double()
  got, want = out["bfloat16"], out["float32"]
  # bf16 operands (2^-9 each) through two layers: the designs' own tests allow 3e-2 of the rms over all logits.  A wrong tile part is 32 rows or
  # 16 columns off by their own size; single rows may be far off all the same (the mLSTM divides by |n . q|, which comes near 0)
  off = lambda dim: ((got - want).square().mean(dim) / want.square().mean()).sqrt()
  assert float(((got - want).square().mean() / want.square().mean()).sqrt()) < 3e-2
  assert int((off(1) > 0.15).sum()) < 8 and float(off(0).max()) < 0.15
