"""Calls of a layered engine on streams of their own: a prompt returns when it is enqueued, and what the other streams do next finds it done."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import gugidra as g
from maxtext_indextts2_b200 import maxengine, pyconfig

pytestmark = pytest.mark.gpu


def test_streams_take_turns():
  """Long prompts with a key each, inserted, decoded and freed on other streams than they were prefilled on: tokens, logits and states of one stream."""
  layers = [g.parallel_layer(4, 2, 64, 2, 64, 128, mlp=g.dense_ff(512, 2.0)), g.gla_layer(4, 64, 128)]
  cfg = pyconfig.from_model_dict(g.model_dict(256, 320, layers), dtype="bfloat16", per_device_batch_size=3, max_target_length=2100, pagedattn_tokens_per_page=16,
                                 pagedattn_num_pages=420, max_step_rows=2048, decode_sampling_strategy="weighted", return_log_prob=True)
  tensors, rng = g.random_tensors(cfg, seed=4), np.random.Generator(np.random.PCG64(1))
  prompts = [rng.integers(0, 320, size=n) for n in (2000, 1500, 900, 1700, 30)]
  runs = []
  for several in (False, True):
    engine = maxengine.MaxEngine(cfg)
    params = engine.load_params(tensors)
    state = engine.init_decode_state()
    streams, turn, got = [torch.cuda.Stream() for _ in range(4)] if several else [torch.cuda.current_stream()], 0, []

    def elsewhere():
      nonlocal turn
      turn += 1
      return torch.cuda.stream(streams[turn % len(streams)])

    torch.cuda.synchronize()
    for i, prompt in enumerate(prompts):
      slot = i % 3
      with elsewhere():
        prefix, first = engine.prefill(params=params, padded_tokens=prompt, true_length=len(prompt), slot=slot, rng=100 + i)
      with elsewhere():
        engine.insert(prefix, state, slot)
      with elsewhere():
        _, result = engine.generate(params, state, rng=200 + i)
      with elsewhere():
        logits = engine.step([((slot + 1) % 3, [3, 4, 5], [0, 1, 2])])
      if i >= 2:
        with elsewhere():
          engine.release_pages((slot + 2) % 3)
      got += [prefix, first.data, first.log_prob, result.data, result.log_prob, logits]  # (read at the end only)
    torch.cuda.synchronize()
    got = [t["tokens"] if isinstance(t, dict) else t for t in got] + [state["logits"]] + [t[:3] for t in state["cache"]["recurrent_state"]]
    runs.append([t.clone() for t in got])
  assert all(torch.equal(a, b) for a, b in zip(*runs))
