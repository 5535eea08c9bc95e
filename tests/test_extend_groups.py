"""Pages for all sequences of a mixed batch at once (page_manager._extend_pages_for_groups) against one sequence after the other."""

import dataclasses
import random

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import layered_engine
from maxtext_indextts2_b200 import page_manager as pm


def test_groups_at_once_against_in_turn():
  rng = random.Random(1)
  failures = 0
  for _ in range(300):
    groups, tpp, per_group = rng.randint(1, 6), rng.choice((1, 4, 8)), rng.randint(1, 6)
    state = pm.initialize_page_state(rng.randint(2, 25), groups, per_group)
    for _ in range(6):
      gs = rng.sample(range(groups), rng.randint(1, groups))
      lengths = [int(state.sequence_lengths[g]) + rng.randint(1, 3 * tpp) for g in gs]
      want, failed = state, -1
      for i, (g, n) in enumerate(zip(gs, lengths)):
        want = pm._extend_pages_for_group(want, g, n, tpp, per_group)
        if int(want.sequence_lengths[g]) != n:
          failed = i
          break
      got, at = pm._extend_pages_for_groups(state, np.asarray(gs), np.asarray(lengths), tpp, per_group)
      assert at == failed
      if failed >= 0:
        failures += 1
        assert got is state
        state = pm._release_pages_for_group(state, gs[0])
        continue
      for f in dataclasses.fields(want):
        a, b = getattr(want, f.name), getattr(got, f.name)
        assert a.dtype == b.dtype and np.array_equal(a, b), f.name
      state = got
  assert failures > 50


def test_token_arrays():
  for tokens in ([3, 4, 5], (3, 4, 5), np.array([3, 4, 5]), np.array([3, 4, 5], np.int16), [3.7, 4.0, 5.2], np.array([3.0, 4.0, 5.0]), [np.int64(3), 4, 5],
                 torch.tensor([3, 4, 5]), torch.tensor([3.0, 4.0, 5.0], dtype=torch.bfloat16), [torch.tensor(3), 4, 5]):
    a = layered_engine._token_array(tokens)
    assert a.dtype == np.int32 and a.tolist() == [3, 4, 5]


def test_token_arrays_of_odd_forms():
  """Whatever a loop of int() over the tokens takes, and its refusals."""
  for tokens in (torch.tensor([3.0, 4.0, 5.0], requires_grad=True), ["3", "4", "5"], np.array([3, 4, 5], np.uint64), np.array([3, 4, 5], np.int32)[::1],
                 np.array([3, 0, 4, 0, 5])[::2], np.array([3, 4, 5], object)):
    a = layered_engine._token_array(tokens)
    assert a.dtype == np.int32 and a.tolist() == [3, 4, 5]
  for tokens in ([2**40], [-(2**31) - 1], [2**63], [2**70], [2**70, 3], [1e30], [float("nan")], [[1], [2]], [None], np.array([2**31])):
    with pytest.raises(Exception) as old:
      torch.tensor([int(t) for t in tokens], dtype=torch.int32)
    with pytest.raises(type(old.value)):
      layered_engine._token_array(tokens)
