"""Decayed sums of long portions as states and outputs in two launches (csrc/decayed_sums.cuh) against the kernel that walks a run's chunks in turn:
the same products in the same order, so the same bits."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import maxengine, pyconfig, zakelorn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,vdim,n", [(2, 64, 64, 300), (1, 128, 128, 1000), (2, 64, 32, 257), (4, 200, 56, 319), (8, 8, 8, 449), (1, 256, 128, 640)])
def test_split_repeats_the_walk_of_chunks(heads, dim, vdim, n):
  """A prompt alone (two launches) and beside fifteen single tokens (runs too short on average for them), from an empty state and from one that holds a
  portion; ends before, at and behind a chunk's edge."""
  layer = zakelorn.parallel_layer(zakelorn.attention_part(4, 2, 32, window=64, keep_first=4), zakelorn.lightning_part(heads, dim, vdim), 0.0, 1.0, zakelorn.dense_ff(256))
  model = zakelorn.model_dict(128, 384, [layer])
  cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=16, max_target_length=2200, pagedattn_tokens_per_page=16,
                                 pagedattn_num_pages=400, max_step_rows=1100)
  tensors = zakelorn.random_tensors(cfg, seed=3)
  rng = np.random.Generator(np.random.PCG64(n))
  first, second = (rng.integers(0, 384, size=n).tolist() for _ in range(2))
  got = []
  for beside in ([], [(s, [7 + s], []) for s in range(1, 16)]):
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(tensors)
    state = engine.init_decode_state()
    logits = [engine.step([(0, toks, list(range(n)))] + beside).clone() for toks in (first, second)]
    got.append(logits + [t[0].clone() for t in state["cache"]["recurrent_state"]])
  assert all(torch.equal(a, b) for a, b in zip(*got))


def test_split_of_many_heads():
  """Heads enough for 16 value columns per CTA."""
  test_split_repeats_the_walk_of_chunks(40, 16, 64, 300)


@pytest.mark.parametrize("heads", [37, 38])
def test_split_at_the_edge_of_the_rule_on_columns(heads):
  """148 and 152 CTAs of eight value columns on 148 SMs: eight columns per CTA, then sixteen."""
  test_split_repeats_the_walk_of_chunks(heads, 16, 32, 300)
