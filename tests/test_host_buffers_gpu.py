"""Decode steps whose kernels read the tokens and write the result in pinned host memory, beside steps that copy (pageable buffers): any mix of them."""

import pytest
import torch

from maxtext_indextts2_b200 import maxengine
from tests.helpers import make_params, random_tokens, small_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sampling", [dict(), dict(decode_sampling_strategy="nucleus", decode_sampling_nucleus_p=0.7)], ids=["greedy", "nucleus"])
@pytest.mark.parametrize("sync", [True, False])  # the call waits for the step, or its caller does
def test_buffers_change_from_step_to_step(sampling, sync):
  cfg = small_config(per_device_batch_size=3, max_prefill_predict_length=16, max_target_length=64, return_log_prob=True, **sampling)
  params, prompts, runs = make_params(cfg), random_tokens((3, 16), cfg.vocab_size, seed=8), []
  for mixed in (False, True):
    engine = maxengine.MaxEngine(cfg)
    dparams = engine.load_params(params)
    state = engine.init_decode_state()
    for slot, n in enumerate((16, 4, 9)):
      prefix, _ = engine.prefill(params=dparams, padded_tokens=prompts[slot], true_length=n)
      state = engine.insert(prefix, state, slot)
    tokens, got = state["tokens"].cpu(), []
    pinned = torch.zeros(4, 64, dtype=torch.int32).pin_memory()
    for step in range(24):  # (more pairs of buffers than graphs are kept)
      at = step % 21  # buffers at any multiple of four bytes
      block = pinned if mixed and step % 5 != 4 else torch.zeros(4, 64, dtype=torch.int32)
      result, given, log_prob = block[0, at : at + 9].view(3, 3), block[1, at : at + 3].view(3, 1), block[2, at : at + 3].view(3, 1).view(torch.float32)
      given.copy_(tokens)
      lp = log_prob if step % 3 else None
      state, _ = engine.generate_to_host(dparams, state, result, host_tokens=given if step % 4 else None, host_log_prob=lp, sync=sync)
      if not sync:
        torch.cuda.current_stream().synchronize()
      tokens = result[:, :1].clone()
      got.append((result.clone(), None if lp is None else lp.clone()))
      torch.testing.assert_close(state["tokens"].cpu().view(-1), tokens.view(-1), rtol=0, atol=0)
    runs.append(got)
  for (a, la), (b, lb) in zip(*runs):
    assert torch.equal(a, b) and (la is None or torch.equal(la, lb))
