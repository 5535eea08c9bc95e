"""Steps that return before their kernels are done (a prompt of the layered engine): what the host writes for the next one reaches the device as it was
written, and another stream does not run ahead of them.  The streams are queues here that run when somebody waits for them."""

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

  def wait_event(self, event):
    self.queue.append(event.synchronize)


class _OrderedStream(_Stream):
  """Waits for what an event stood for when it was called, as a stream of the device does (the event may be recorded again before the wait is reached)."""

  def wait_event(self, event):
    stream, item = event.stream, event.item

    def wait():
      while item in stream.queue:
        stream.queue.pop(0)()

    self.queue.append(wait)


class _Event:
  def __init__(self):
    self.stream, self.left = None, None

  def record(self, stream):
    self.stream, self.left = stream, object()
    mark = self.left
    stream.queue.append(lambda: mark)
    self.item = stream.queue[-1]

  def synchronize(self):
    while self.stream is not None and self.item in self.stream.queue:
      self.stream.queue.pop(0)()


class _DeviceBuffer:
  def __init__(self, now, *shape):
    self.now_stream, self.now = now, np.zeros(shape, np.int32)

  def __getitem__(self, rows):
    return self

  def copy_(self, src, non_blocking=False):
    assert non_blocking
    self.now_stream[0].queue.append(lambda: self.now.__setitem__(slice(None), src.numpy()))

  def data_ptr(self):
    return 0


def _engine(monkeypatch, rows=40):
  now = [_Stream()]
  monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: now[0])
  e = object.__new__(layered_engine.LayeredEngine)
  e.config = types.SimpleNamespace(vocab_size=7, per_device_batch_size=3, pagedattn_num_pages=40, pagedattn_tokens_per_page=4, max_target_length=60,
                                   pagedattn_max_pages_per_group=16)
  e.device, e._max_rows = torch.device("cpu"), rows
  e.page_manager = pm.PageManager(e.config)
  e.page_state = pm.initialize_page_state(40, 3, 16)
  e._require_params = lambda params: None
  e._desc_host, e._map_host = torch.zeros(6 * rows + 16, dtype=torch.int32), torch.zeros(3, 16, dtype=torch.int32)
  e._desc_dev, e._page_map_dev = _DeviceBuffer(now, 6 * rows + 16), _DeviceBuffer(now, 3, 16)
  e._desc_read, e._map_read, e._step_done = _Event(), _Event(), _Event()
  e._uploaded_map = None
  seen = []

  def run(n, token_ptr, group_ptr, pos_ptr, n_want, want_ptr, logits, n_tiles, tiles_ptr, graph=False, n_runs=0, runs_ptr=None):
    now[0].queue.append(lambda: seen.append((e._desc_dev.now[:n].tolist(), int(e._desc_dev.now[rows]), e._page_map_dev.now.copy())))

  e._run = run
  return e, now, seen


@pytest.mark.parametrize("rows", [40, 8])
def test_back_to_back_prompts(monkeypatch, rows):
  e, now, seen = _engine(monkeypatch, rows)
  maps = []
  for slot, first in ((0, 100), (2, 200), (1, 300)):
    e._step([(slot, np.arange(first, first + 8), [7])], wait=False)
    maps.append(e.page_state.page_map.copy())
  now[0].synchronize()
  assert [s[0] for s in seen] == [list(range(f, f + 8)) for f in (100, 200, 300)] and [s[1] for s in seen] == [0, 2, 1]
  assert all((s[2] == m).all() for s, m in zip(seen, maps))
  e.step([(0, [5], [0]), (1, [6, 7], [])])  # (a step that waits, behind those)
  assert seen[-1][0] == [5, 6, 7] and (seen[-1][2] == e.page_state.page_map).all()


def test_another_stream_waits(monkeypatch):
  e, now, seen = _engine(monkeypatch)
  e._step([(0, [1, 2, 3], [2])], wait=False)
  first, now[0] = now[0], _Stream()
  e.step([(1, [4, 5], [1])])
  assert [s[0] for s in seen] == [[1, 2, 3], [4, 5]] and not first.queue
  e._step([(2, [6], [])], wait=False)
  e._step([(0, [7], [])], wait=False)  # (the same stream: nothing to wait for but the buffers)
  assert not any(getattr(q, "__func__", None) is _Event.synchronize for q in now[0].queue)
  now[0].synchronize()
  assert [s[0] for s in seen[2:]] == [[6], [7]]


def test_a_third_stream_waits_too(monkeypatch):
  """A stream that has waited for a prompt (here to free a slot) does not stand for the others."""
  e, now, seen = _engine(monkeypatch)
  now[0] = _OrderedStream()
  e._states, e._active, e._next_pos = [], torch.ones(3, 1, dtype=torch.int32), torch.ones(3, 1, dtype=torch.int32)
  e._step([(0, [1, 2, 3], [2])], wait=False)
  first, now[0] = now[0], _OrderedStream()
  e.release_pages(1)
  now[0] = _OrderedStream()
  e.step([(2, [4, 5], [1])])
  assert [s[0] for s in seen] == [[1, 2, 3], [4, 5]] and not first.queue


def _serving(monkeypatch):
  """An engine whose keys and draws leave a mark when their stream runs them."""
  e, now, seen = _engine(monkeypatch)
  now[0] = _OrderedStream()
  i32 = torch.int32
  e._params = e._state = {}
  e.config.return_log_prob = True
  e._states, e._uploaded_map = [], None
  e._active, e._next_pos, e._generated, e._tokens = (torch.zeros(3, 1, dtype=i32) for _ in range(4))
  e._first_token, e._first_log_prob, e._log_prob = torch.zeros(1, dtype=i32), torch.zeros(1), torch.zeros(3, 1)
  e._result, e._logits, e._slot_ids = torch.zeros(3, 3, dtype=i32), torch.zeros(3, 1, 7), torch.arange(3, dtype=i32)
  e._decode_groups, e._decode_tiles, e.use_cuda_graph = torch.zeros(3, dtype=i32), torch.arange(4, dtype=i32), False
  marks = []
  e._seed = lambda rng: rng is not None and now[0].queue.append(lambda: marks.append(("key", rng)))
  e._sample = lambda logits, rows, *rest: now[0].queue.append(lambda: marks.append(("draw", rows)))
  return e, now, marks


def test_insert_on_another_stream_follows_the_draw(monkeypatch):
  e, now, marks = _serving(monkeypatch)
  prefix, _ = e.prefill(padded_tokens=[1, 2, 3], true_length=3, slot=1)
  now[0] = _OrderedStream()
  e.insert(prefix, e._state, 1)
  now[0].synchronize()
  assert marks == [("draw", 1)]


@pytest.mark.parametrize("call", ["prefill", "generate"])
def test_keys_follow_the_draws_before_them(monkeypatch, call):
  e, now, marks = _serving(monkeypatch)
  e.prefill(padded_tokens=[1, 2, 3], true_length=3, slot=1, rng=5)
  now[0] = _OrderedStream()
  if call == "prefill":
    e.prefill(padded_tokens=[4], true_length=1, slot=2, rng=6)
  else:
    e.generate(e._params, e._state, rng=6)
  now[0].synchronize()
  assert marks == [("key", 5), ("draw", 1), ("key", 6), ("draw", 1 if call == "prefill" else 3)]


def test_a_step_follows_a_decode_step(monkeypatch):
  """A decode step whose page map is still on its way, a step on another stream (which uploads none), and a decode step that grows a page."""
  e, now, marks = _serving(monkeypatch)
  maps, run = [], e._run
  e._run = lambda *args, **kw: now[0].queue.append(lambda: maps.append(e._page_map_dev.now.copy()))
  e.step([(0, [1, 2, 3], []), (1, [4], [])])
  first, want = now[0], [e.page_state.page_map]
  e.generate(e._params, e._state)
  e.generate(e._params, e._state)  # (slot 0 grows a page)
  want += [maps[0], e.page_state.page_map]
  now[0] = _OrderedStream()
  e.step([(1, [5], [])])
  want.append(e.page_state.page_map)
  now[0] = first
  for _ in range(4):
    e.generate(e._params, e._state)
    want.append(e.page_state.page_map)
  first.synchronize()
  assert len(maps) == len(want) and all((a == b).all() for a, b in zip(maps, want))


def test_a_step_of_no_rows_uploads_for_the_next_stream(monkeypatch):
  e, now, marks = _serving(monkeypatch)
  maps = []
  e._run = lambda *args, **kw: now[0].queue.append(lambda: maps.append(e._page_map_dev.now.copy()))
  first = now[0]
  e.prefill(padded_tokens=[1, 2, 3], true_length=3, slot=1)
  e.release_pages(1)
  now[0] = _OrderedStream()
  assert e.step([]).shape == (0, 7)
  now[0] = first
  e.generate(e._params, e._state)
  first.synchronize()
  assert (maps[-1] == e.page_state.page_map).all() and maps[-1].sum() == 0


def test_a_prompt_follows_its_slot_s_release(monkeypatch):
  e, now, marks = _serving(monkeypatch)
  e.step([(1, [1, 2], [])])
  e._states = [(torch.zeros(3, 2),)]
  monkeypatch.setattr(torch, "_foreach_zero_", lambda ts: now[0].queue.append(lambda: marks.append("zero")))
  e.prefill(padded_tokens=[1, 2, 3], true_length=3, slot=1)
  first, now[0] = now[0], _OrderedStream()
  e.release_pages(1)
  now[0] = first
  e.prefill(padded_tokens=[4, 5], true_length=2, slot=1)
  first.synchronize()
  assert marks == ["zero", "zero", ("draw", 1), "zero", "zero", "zero", "zero", ("draw", 1)]


def test_an_engine_gives_nothing_up_under_a_prompt(monkeypatch):
  """Dropped engines and replaced weights: the buffers of a prompt that returned early are in use until its stream is done."""
  e, now, seen = _engine(monkeypatch)
  e._handle, first = None, now[0]
  e._step([(0, [1, 2, 3], [2])], wait=False)
  with pytest.raises(AttributeError):  # (no weights here: what comes after the wait)
    e._create(types.SimpleNamespace(float32=False))
  assert not first.queue and len(seen) == 1
  e._step([(1, [4], [])], wait=False)
  e.__del__()
  assert not first.queue and len(seen) == 2


def test_tokens_of_mixed_forms(monkeypatch):
  """Entries given as lists, arrays and tensors keep their order."""
  e, now, seen = _engine(monkeypatch)
  e.step([(0, [1, 2], [0]), (2, np.array([3, 4, 5], np.int64), []), (1, [6], [0])])
  e.step([(0, torch.tensor([7, 8]), [1]), (1, (9,), [0]), (2, [True, 2.0], [])])
  assert [s[0] for s in seen] == [[1, 2, 3, 4, 5, 6], [7, 8, 9, 1, 2]]
