"""Mixed batches of the windowed sigmoid attention: single tokens on the decode kernel, prompts' tiles on the other (csrc/window_attention_decode.cuh,
window_attention_mma.cuh), against every sequence in a step of its own."""

import numpy as np
import pytest

from maxtext_indextts2_b200 import kifusun, maxengine, pyconfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,dim,window", [(4, 2, 64, 96), (16, 4, 128, 40), (8, 8, 32, 300)])
def test_mixed_batch_against_each_alone(heads, kv_heads, dim, window):
  """Portions of 33 (a last tile of one row), 2, 40 and 1 tokens among single tokens of sequences that are shorter and longer than the window."""
  model = kifusun.model_dict(256, 320, [kifusun.attention_layer(heads, kv_heads, dim, dim, window, ff=256, bias_max=float(window))] * 2)
  cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=12, max_target_length=256, pagedattn_tokens_per_page=16,
                                 pagedattn_num_pages=12 * 17 + 2, max_step_rows=256)
  rng = np.random.Generator(np.random.PCG64(1))
  seen = [0, 5, 0, 120, 30, 1, 97, 60, 15, 16, 17, 130]
  new = [33, 1, 2, 1, 40, 1, 1, 1, 1, 1, 1, 1]
  toks = [rng.integers(0, 320, size=a + b).tolist() for a, b in zip(seen, new)]
  out = []
  tensors = None
  for together in (True, False):
    engine = maxengine.MaxEngine(cfg)
    tensors = tensors or kifusun.random_tensors(cfg, seed=3)
    engine.load_params(tensors)
    engine.init_decode_state()
    for s, a in enumerate(seen):
      if a:
        engine.step([(s, toks[s][:a], [])])
    entries = [(s, toks[s][a:], list(range(n))) for s, (a, n) in enumerate(zip(seen, new))]
    out.append([engine.step(entries).double()] if together else [engine.step([x]).double() for x in entries])
  got, want = out[0][0], np.concatenate([x.cpu().numpy() for x in out[1]])
  # bf16 weights and values (2^-9 each) through two layers, added up in another order
  off = np.sqrt(np.square(got.cpu().numpy() - want).mean(1) / np.square(want).mean())
  assert off.max() < 2e-2
