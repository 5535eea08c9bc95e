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
