"""The tcgen05 softmax attention of long runs (csrc/softmax_flash.cuh) against the mma.sync kernel of shorter ones: without windows the same bits."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import ginodra, gugidra, ligidra, maxengine, pyconfig, zakelorn

pytestmark = pytest.mark.gpu

GROUP = 256  # rows per step, whatever they are made of: the projections' plans go by it


def _model(name, dim):
  if name == "gugidra":
    return gugidra, gugidra.model_dict(256, 320, [gugidra.parallel_layer(4, 2, dim, 2, 32, 64, mlp=gugidra.dense_ff(256))] * 2)
  if name == "ginodra":  # distance penalties, gates
    return ginodra, ginodra.model_dict(256, 320, [ginodra.attention_layer(4, 4, dim, mlp=ginodra.dense_ff(256))] * 2)
  if name == "ligidra":  # capped scores, sinks
    return ligidra, ligidra.model_dict(256, 320, [ligidra.attention_layer(4, 1, dim, softcap=20.0, mlp=ligidra.moe_ff(4, 4, 64, shared_ff=64))] * 2, side_dim=64)
  # sinks, gates per channel (the right part, whose chunks go by the run, is left out)
  layers = [zakelorn.parallel_layer(zakelorn.attention_part(4, 2, dim, window=1024, keep_first=4), zakelorn.lightning_part(4, 64), right_scale=0.0, mlp=zakelorn.dense_ff(256))] * 2
  return zakelorn, zakelorn.model_dict(256, 320, layers)


@pytest.mark.parametrize("name,dim,page", [("gugidra", 64, 16), ("gugidra", 128, 64), ("gugidra", 256, 8), ("ginodra", 64, 128), ("ginodra", 128, 24), ("ligidra", 64, 64),
                                           ("ligidra", 256, 40), ("zakelorn", 64, 32), ("zakelorn", 128, 8)])
def test_long_runs_repeat_short_ones(name, dim, page):
  """Runs of 256 and 150 rows against runs of 85: the second layer's keys of a sequence of 662 tokens.  The long runs begin and end inside pages
  and key tiles."""
  design, model = _model(name, dim)
  toks = np.random.Generator(np.random.PCG64(1)).integers(0, model["vocab"], size=1024).tolist()
  out = []
  for long_runs in (True, False):
    cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=3, max_target_length=960, pagedattn_tokens_per_page=page,
                                   pagedattn_num_pages=3 * (960 // page + 1) + 2, max_step_rows=GROUP)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(design.random_tensors(cfg, seed=3))
    state = engine.init_decode_state()
    at = [0, 0, 0]
    while at[0] < 662:
      n = min(85, 662 - at[0])
      if long_runs:
        n = min(256, 662 - at[0])
      counts = [n, (GROUP - n) // 2, GROUP - n - (GROUP - n) // 2] if not long_runs else [n, GROUP - n, 0]
      engine.step([(s, toks[at[s] : at[s] + c], []) for s, c in enumerate(counts) if c])
      at = [a + c for a, c in zip(at, counts)]
    pages = torch.as_tensor(engine.page_state.page_map[0], device="cuda").long()
    keys = state["cache"]["key_pages"][1][:, pages].flatten(1, 2)
    out.append(keys[:, :662].clone())
  assert torch.isfinite(out[0]).all() and torch.equal(out[0], out[1])


@pytest.mark.parametrize("name,dim,page", [("gugidra", 64, 16), ("gugidra", 128, 24), ("gugidra", 256, 64), ("ginodra", 64, 8), ("ligidra", 128, 40), ("zakelorn", 64, 64)])
@pytest.mark.parametrize("portions", [(700,), (257, 512), (512, 257, 129), (3, 690, 300)])
def test_runs_of_several_tiles(name, dim, page, portions):
  """Runs of one to three CTAs' rows, alone and side by side, at the start of a sequence and behind the 200 tokens that it holds, against runs of 85."""
  design, model = _model(name, dim)
  rng = np.random.Generator(np.random.PCG64(sum(portions)))
  held = [0, 200, 37][: len(portions)]
  toks = [rng.integers(0, model["vocab"], size=h + n).tolist() for h, n in zip(held, portions)]
  out = []
  for long_runs in (True, False):
    cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=7, max_target_length=960, pagedattn_tokens_per_page=page,
                                   pagedattn_num_pages=7 * (960 // page + 1) + 2, max_step_rows=1024)
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(design.random_tensors(cfg, seed=3))
    state = engine.init_decode_state()
    at = [0] * len(portions)
    for end, most in ((held, 85), ([h + n for h, n in zip(held, portions)], 960 if long_runs else 85)):
      while at != end:
        part = [min(b - a, most) for a, b in zip(at, end)]
        entries = [(s, toks[s][a : a + n], []) for s, (a, n) in enumerate(zip(at, part)) if n]
        if sum(part) <= 256:  # (more rows in every step, in short runs: the products' plans are then the same)
          for s in range(3, 7):
            engine.release_pages(s)
            entries.append((s, toks[0][:85] if len(toks[0]) >= 85 else toks[1][:85], []))
        rows = sum(len(e[1]) for e in entries)
        assert rows > 256 and (rows >= 128 * len(entries)) == (max(part) > 85)  # (takes_paged_flash)
        engine.step(entries)
        at = [a + n for a, n in zip(at, part)]
    keys = []
    for s, n in enumerate(at):
      pages = torch.as_tensor(engine.page_state.page_map[s], device="cuda").long()
      keys.append(state["cache"]["key_pages"][1][:, pages].flatten(1, 2)[:, :n].clone())
    out.append(keys)
  for a, b in zip(*out):
    assert torch.isfinite(a).all() and torch.equal(a, b)
