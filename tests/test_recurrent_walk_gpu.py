"""The recurrences' walks (csrc/recurrent_mixers.cuh) where CTAs of one head share state, and the walk of long runs against the one of short ones."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import gugidra as g
from maxtext_indextts2_b200 import maxengine, pyconfig

pytestmark = pytest.mark.gpu


def tokens(n, seed):
  return np.random.Generator(np.random.PCG64(seed)).integers(0, 320, size=n).tolist()


def test_many_slots_decode_like_each_alone():
  """A decode step of more (slot, head, column block) CTAs than run at once: every CTA of a head reads the mLSTM's normaliser and running
  maximum of the state, whichever of them is done first."""
  cfg = g.model_dict(256, 320, [g.parallel_layer(4, 2, 64, 8, 64, 128)])
  config = lambda slots: pyconfig.from_model_dict(cfg, dtype="float32", per_device_batch_size=slots, max_target_length=64, pagedattn_tokens_per_page=16,
                                                  pagedattn_num_pages=4 * slots + 2)
  tensors = g.random_tensors(config(1), seed=2)
  many, one = (maxengine.MaxEngine(config(n)) for n in (64, 1))
  for e in (many, one):
    e.load_params(tensors)
    e.init_decode_state()
  prompt, then = tokens(9, 5), tokens(64, 6)
  many.step([(s, prompt, []) for s in range(64)])
  got = many.step([(s, [then[s]], [0]) for s in range(64)])
  for s in range(0, 64, 9):
    one.release_pages(0)
    one.step([(0, prompt, [])])
    want = one.step([(0, [then[s]], [0])])
    assert float((got[s] - want[0]).abs().max() / want[0].abs().max()) < 3e-5  # (fp32 sums in another order, as in the design's own tests)


def test_long_walk_repeats_short_portions():
  """Runs of 16 tokens and more (one reduction per chunk of tokens) leave the bits that the token-by-token walk of portions of 10 leaves."""
  for kind in ("gla", "parallel"):
    layer = g.gla_layer(4, 64, 64) if kind == "gla" else g.parallel_layer(4, 2, 32, 2, 128, 64)
    cfg = g.model_dict(256, 320, [layer])
    config = pyconfig.from_model_dict(cfg, dtype="float32", per_device_batch_size=1, max_target_length=128, pagedattn_tokens_per_page=16, pagedattn_num_pages=10)
    tensors, toks, states = g.random_tensors(config, seed=4), tokens(90, 5), []
    for portion in (90, 10):
      engine = maxengine.MaxEngine(config)
      engine.load_params(tensors)
      state = engine.init_decode_state()
      for at in range(0, 90, portion):
        logits = engine.step([(0, toks[at : at + portion], [portion - 1])])
      states.append([t.clone() for t in state["cache"]["recurrent_state"]] + [logits])
    assert all(torch.equal(a, b) for a, b in zip(*states))


def columns_per_thread(runs, heads, dim, vdim):
  """What csrc/layered.cu (launch_rec_scan, launch_rec_walk) takes on this GPU for runs of 16 tokens and more; 0: the walk token by token."""
  sms, ctas = torch.cuda.get_device_properties(0).multi_processor_count, lambda cols: runs * heads * -(-vdim // cols)
  if ctas(16) >= 2 * sms or dim < 64 or runs * heads * vdim * 8 >= 512 * sms:
    return 0
  return 1 if ctas(8) <= sms else 2


@pytest.mark.parametrize("kind,heads,dim,vdim,columns", [
    ("gla", 24, 64, 128, 0), ("gla", 2, 256, 40, 1), ("gla", 3, 100, 72, 1), ("mlstm", 20, 128, 128, 0), ("mlstm", 2, 200, 20, 1), ("mlstm", 1, 64, 8, 1),
    ("gla", 12, 64, 128, 2), ("gla", 16, 128, 40, 2), ("gla", 12, 256, 72, 2), ("mlstm", 16, 64, 40, 2), ("mlstm", 12, 128, 128, 2), ("mlstm", 12, 200, 72, 2)])
def test_walk_of_two_long_runs(kind, heads, dim, vdim, columns):
  """Two runs of a step, ends before, at and behind a chunk of 16 tokens, one and two columns per thread, channels and columns that fill neither slices nor
  CTAs: the bits of portions of ten tokens, which are walked token by token -- the states' and, by the logits of every position, the read-outs'."""
  assert columns_per_thread(2, heads, dim, vdim) == columns
  layer = g.gla_layer(heads, dim, vdim) if kind == "gla" else g.parallel_layer(4, 2, 32, heads, dim, vdim)
  cfg = g.model_dict(256, 320, [layer])
  config = pyconfig.from_model_dict(cfg, dtype="float32", per_device_batch_size=2, max_target_length=128, pagedattn_tokens_per_page=16, pagedattn_num_pages=20)
  tensors, toks, states = g.random_tensors(config, seed=4), [tokens(n, 5) for n in (79, 64)], []
  for portion in (47, 10):  # 47 + 32, 47 + 17 against tens
    engine = maxengine.MaxEngine(config)
    engine.load_params(tensors)
    state = engine.init_decode_state()
    logits = ([], [])
    for at in range(0, 79, portion):
      parts = [(slot, t[at : at + portion], list(range(len(t[at : at + portion])))) for slot, t in enumerate(toks) if t[at : at + portion]]
      out = engine.step(parts).split([len(p[1]) for p in parts])
      for (slot, _, _), rows in zip(parts, out):
        logits[slot].append(rows)
    if not columns:  # (the tens behind 70 are one run, for which the walk token by token cuts a column into more slices: read-outs added up in another order)
      logits[0][-1] = logits[0][-1][: 23 if portion == 47 else 0]
    states.append([t[:2].clone() for t in state["cache"]["recurrent_state"]] + [torch.cat(rows) for rows in logits])
  assert all(torch.equal(a, b) for a, b in zip(*states))
