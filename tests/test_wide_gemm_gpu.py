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
  ffs = [zakelorn.dense_ff(ff), zakelorn.moe_ff(5, 4, 96, identity=1, groups=2, keep=2)]  # unequal experts, slots beyond their ranges
  layers = [zakelorn.parallel_layer(zakelorn.attention_part(4, 2, 64, window=64, keep_first=4), zakelorn.lightning_part(4, 64), mlp=f) for f in ffs]
  return zakelorn, zakelorn.model_dict(width, 384, layers)


@pytest.mark.parametrize("name", ["kifusun", "gugidra", "zakelorn"])
def test_long_steps_repeat_short_ones(name):
  """A row's bits do not depend on how many rows its step has: 768 rows at once against three steps of 256."""
  design, model = _model(name, 256)
  toks = np.random.Generator(np.random.PCG64(1)).integers(0, model["vocab"], size=768).tolist()
  out = []
  for rows in (768, 256):
    cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=2, max_target_length=800, pagedattn_tokens_per_page=16,
                                   pagedattn_num_pages=60, max_step_rows=rows)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(design.random_tensors(cfg, seed=3))
    state = engine.init_decode_state()
    engine.step([(0, toks, [])])
    out.append([t.clone() for t in state["cache"]["key_pages"][:1]])
  assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("name", ["kifusun", "gugidra", "ligidra", "zakelorn"])
@pytest.mark.parametrize("width,rows", [(256, 257), (384, 512), (256, 769)])
def test_long_steps_against_float32(name, width, rows):
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
