"""A step of more rows than max_step_rows: the descriptors of every slice reach the device as they were written, however late the stream gets to the
copies.  The stream is a queue here that runs when somebody waits for it, as one that still holds other work does."""

import types

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import layered_engine
from maxtext_indextts2_b200 import page_manager as pm


class _Stream:
  def __init__(self):
    self.queue = []

  def synchronize(self):
    while self.queue:
      self.queue.pop(0)()


class _Event:
  def __init__(self, stream):
    self.stream, self.left = stream, None

  def record(self, stream=None):
    self.left = stream.queue[-1] if stream.queue else None

  def synchronize(self):
    while self.left in self.stream.queue:
      self.stream.queue.pop(0)()


class _DeviceBuffer:
  def __init__(self, stream, n):
    self.stream, self.now = stream, np.zeros(n, np.int32)

  def copy_(self, src, non_blocking=False):
    self.stream.queue.append(lambda: self.now.__setitem__(slice(None), src.numpy()))

  def data_ptr(self):
    return 0


@pytest.mark.parametrize("rows", [8, 16])
def test_slices_of_a_busy_stream(monkeypatch, rows):
  stream = _Stream()
  monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: stream)
  e = object.__new__(layered_engine.LayeredEngine)
  e.config = types.SimpleNamespace(vocab_size=7, per_device_batch_size=3, pagedattn_num_pages=40, pagedattn_tokens_per_page=4, max_target_length=60,
                                   pagedattn_max_pages_per_group=16)
  e.device, e._max_rows = torch.device("cpu"), rows
  e.page_manager = pm.PageManager(e.config)
  e.page_state = pm.initialize_page_state(40, 3, 16)
  e._require_params = lambda params: None
  e._upload_page_map = lambda: None
  e._desc_host = torch.zeros(6 * rows + 16, dtype=torch.int32)
  e._desc_dev = _DeviceBuffer(stream, 6 * rows + 16)
  e._desc_read = _Event(stream)
  seen = []

  def run(n, token_ptr, group_ptr, pos_ptr, n_want, want_ptr, logits, n_tiles, tiles_ptr, graph=False, n_runs=0, runs_ptr=None):
    assert (group_ptr, pos_ptr, want_ptr, tiles_ptr, runs_ptr) == (4 * rows, 8 * rows, 12 * rows, 16 * rows, 4 * (5 * rows + 8))
    d = e._desc_dev
    stream.queue.append(lambda: seen.append((d.now[:n].copy(), d.now[rows : rows + n].copy(), d.now[2 * rows : 2 * rows + n].copy(),
                                             d.now[3 * rows : 3 * rows + n_want].copy(), d.now[4 * rows : 4 * rows + n_tiles + 1].copy(),
                                             d.now[5 * rows + 8 : 5 * rows + 8 + n_runs + 1].copy())))

  e._run = run
  lengths, toks, at = (21, 1, 17), list(range(100, 139)), 0
  entries = []
  for slot, n in enumerate(lengths):
    entries.append((slot, toks[at : at + n], [0, n - 1]))
    at += n
  e.step(entries)
  assert [len(s[0]) for s in seen] == [min(rows, 39 - lo) for lo in range(0, 39, rows)]
  tok, grp, pos = (np.concatenate([s[i] for s in seen]).tolist() for i in range(3))
  assert tok == toks and grp == [0] * 21 + [1] + [2] * 17 and pos == [*range(21), 0, *range(17)]
  assert [lo + int(w) for lo, s in zip(range(0, 39, rows), seen) for w in s[3]] == [0, 20, 21, 21, 22, 38]
  for lo, s in zip(range(0, 39, rows), seen):
    hi = min(lo + rows, 39)
    starts = [max(a, lo) - lo for a, b in ((0, 21), (21, 22), (22, 39)) if max(a, lo) < min(b, hi)]
    assert s[5].tolist() == starts + [hi - lo] and set(starts) <= set(s[4].tolist()) and s[4][-1] == hi - lo
