"""Prompts of more than 256 tokens: one pass over all rows (csrc/gemm_wide.cuh, csrc/prefill_flash.cuh) against the same prompt in portions of
at most 200 tokens, which run the 256-row kernels.  Lengths at the edges of the 128- and 256-row tiles, every head size, sliding windows
that start and end inside a tile, unfolded norm scales, a paged and an 8-bit engine (their prompts go through a staging plane)."""

import pytest
import torch

from maxtext_indextts2_b200 import _lib, maxengine, pyconfig

pytestmark = pytest.mark.gpu


def _config(block, dim, **kw):
  base = dict(base_num_decoder_layers=2, base_emb_dim=192, base_num_query_heads=6, base_num_kv_heads=2, head_dim=dim, base_mlp_dim=320, vocab_size=512,
              per_device_batch_size=2, max_prefill_predict_length=832, max_target_length=900, weight_dtype="bfloat16", scan_layers=False,
              attention="dot_product", materialize_logits=True, use_chunked_prefill=True)
  if block == "gemma3":
    base.update(model_name="gemma3-4b", sliding_window_size=150)
  base.update(kw)
  return pyconfig.initialize(None, **base)


CASES = [("llama2", 64, {}), ("llama2", 128, {}), ("llama2", 64, dict(fold_norm_scales=False)), ("llama2", 64, dict(attn_logits_soft_cap=5.0)),
         ("llama2", 64, dict(quantize_kvcache=True, kv_quant_axis="dkv")),
         ("llama2", 64, dict(attention="paged", pagedattn_num_pages=120, pagedattn_tokens_per_page=16)),
         ("gemma3", 64, {}), ("gemma3", 128, {}), ("gemma3", 256, {}), ("gemma3", 256, dict(sliding_window_size=64))]


@pytest.mark.parametrize("block,dim,kw", CASES)
def test_one_pass_against_portions(block, dim, kw):
  cfg = _config(block, dim, **kw)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  for n in (257, 384, 513, 831):
    toks = torch.randint(0, cfg.vocab_size, (n,), generator=torch.Generator().manual_seed(n))
    whole, _ = engine.prefill(params=params, padded_tokens=toks, true_length=n, slot=0)
    prefix, done = None, 0
    while done < n:
      m = min(200, n - done)
      before = maxengine.ExistingPrefix(cache=prefix["cache"], common_prefix_tokens=toks[:done]) if done else None
      prefix, _ = engine.prefill(params=params, padded_tokens=toks[done : done + m], true_length=m, existing_prefix=before, slot=0)
      done += m
    for name in ("key", "value"):
      got, want = whole["cache"][name].double(), prefix["cache"][name].double()  # [L, heads, n, D]
      assert got.shape == want.shape
      # bf16 activations through at most two layers: 2^-9 for each of about ten roundings
      err = ((got - want).square().mean((0, 1, 3)) / want.square().mean()).sqrt()
      assert float(err.max()) < 4e-2, (n, name, int(err.argmax()))
    a, b = whole["logits"].double(), prefix["logits"].double()
    assert float((a - b).norm() / b.norm()) < 4e-2, n


@pytest.mark.parametrize("dim,kw", [(64, {}), (128, {"sliding_window_size": 256}), (256, {}), (256, {"sliding_window_size": 256}), (256, {"sliding_window_size": 300})])
def test_gemma3_pass_repeats_steps(dim, kw):
  """The gemma3 block in one pass leaves the bits of its 256-token steps: windows that no, some and all positions fill, a length at which a group of
  positions holds some of either kind, and a remainder behind the pass."""
  cfg = _config("gemma3", dim, **kw)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  toks = torch.randint(0, cfg.vocab_size, (831,), generator=torch.Generator().manual_seed(2))
  whole, _ = engine.prefill(params=params, padded_tokens=toks, true_length=831, slot=0)
  prefix = None
  for at in range(0, 831, 256):
    m = min(256, 831 - at)
    before = maxengine.ExistingPrefix(cache=prefix["cache"], common_prefix_tokens=toks[:at]) if at else None
    prefix, _ = engine.prefill(params=params, padded_tokens=toks[at : at + m], true_length=m, existing_prefix=before, slot=0)
  for name in ("key", "value"):
    assert torch.equal(whole["cache"][name], prefix["cache"][name])


@pytest.mark.parametrize("dim,n", [(64, 641), (128, 767), (256, 640), (256, 641), (256, 767)])
def test_gemma3_rows_behind_the_last_256(dim, n):
  """129 to 255 rows behind the last multiple of 256 go with the pass, up to 128 are a step of their own: the bits of the 256-token steps either way."""
  cfg = _config("gemma3", dim)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  toks = torch.randint(0, cfg.vocab_size, (n,), generator=torch.Generator().manual_seed(n))
  whole, _ = engine.prefill(params=params, padded_tokens=toks, true_length=n, slot=0)
  prefix = None
  for at in range(0, n, 256):
    m = min(256, n - at)
    before = maxengine.ExistingPrefix(cache=prefix["cache"], common_prefix_tokens=toks[:at]) if at else None
    prefix, _ = engine.prefill(params=params, padded_tokens=toks[at : at + m], true_length=m, existing_prefix=before, slot=0)
  for name in ("key", "value"):
    assert torch.equal(whole["cache"][name], prefix["cache"][name])
  assert torch.equal(whole["logits"], prefix["logits"])


@pytest.mark.parametrize("heads,kv_heads,window,sizes", [(4, 4, 700, (2304,)), (4, 2, 1024, (2304,)), (8, 1, 300, (1280,)), (5, 1, 64, (768, 512)), (4, 2, 500, (512, 1536))])
def test_gemma3_items_of_many_positions(heads, kv_heads, window, sizes):
  """Wide heads: items of 4 to 32 positions (four groups of 8 columns), more positions than one item takes, windows that end inside an item, behind a
  prefix that begins inside a group; the bits of the 256-token steps in every layer's keys and values, and in the logits."""
  cfg = _config("gemma3", 256, base_num_query_heads=heads, base_num_kv_heads=kv_heads, sliding_window_size=window, max_prefill_predict_length=2400, max_target_length=2500,
                base_num_decoder_layers=7)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  n = sum(sizes)
  toks = torch.randint(0, cfg.vocab_size, (n,), generator=torch.Generator().manual_seed(n))

  def portions(sizes):
    prefix, done = None, 0
    for m in sizes:
      before = maxengine.ExistingPrefix(cache=prefix["cache"], common_prefix_tokens=toks[:done]) if done else None
      prefix, _ = engine.prefill(params=params, padded_tokens=toks[done : done + m], true_length=m, existing_prefix=before, slot=0)
      done += m
    return prefix

  got, want = portions(sizes), portions([256] * (n // 256) + [n % 256] * (n % 256 > 0))
  for name in ("key", "value"):
    assert torch.equal(got["cache"][name], want["cache"][name])
  assert torch.equal(got["logits"], want["logits"])


@pytest.mark.parametrize("block,dim,kw", [("llama2", 64, {}), ("llama2", 128, {}), ("gemma3", 256, {}), ("llama2", 64, dict(quantize_kvcache=True, kv_quant_axis="dkv"))])
def test_several_passes_and_a_prefix(block, dim, kw):
  """A prompt of more rows than a pass takes (4096), and passes behind prefixes that end inside a tile, against portions of 200."""
  cfg = _config(block, dim, max_prefill_predict_length=5000, max_target_length=5100, **kw)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  n = 4096 + 401
  toks = torch.randint(0, cfg.vocab_size, (n,), generator=torch.Generator().manual_seed(n))

  def portions(*sizes):
    prefix, done = None, 0
    for m in sizes:
      before = maxengine.ExistingPrefix(cache=prefix["cache"], common_prefix_tokens=toks[:done]) if done else None
      prefix, _ = engine.prefill(params=params, padded_tokens=toks[done : done + m], true_length=m, existing_prefix=before, slot=0)
      done += m
    return prefix

  want = portions(*[200] * 22, n - 4400)
  for sizes in ((n,), (99, 4397 - 1000, 1001), (1300, n - 1300)):
    assert sum(sizes) == n
    got = portions(*sizes)
    for name in ("key", "value"):
      a, b = got["cache"][name].double(), want["cache"][name].double()  # [L, heads, n, D]
      # bf16 activations through at most two layers: 2^-9 for each of about ten roundings
      err = ((a - b).square().mean((0, 1, 3)) / b.square().mean()).sqrt()
      assert float(err.max()) < 4e-2, (sizes, name, int(err.argmax()))
    a, b = got["logits"].double(), want["logits"].double()
    assert float((a - b).norm() / b.norm()) < 4e-2, sizes


@pytest.mark.parametrize("block,dim,chunk", [("llama2", 64, 64), ("llama2", 128, 200), ("gemma3", 256, 100)])
def test_prefill_chunk_size_bounds_a_step(block, dim, chunk):
  """A prefill_chunk_size below its default of 256 is the most rows of a prompt that a step takes: the bits of the prompt in portions of that size."""
  cfg = _config(block, dim, prefill_chunk_size=chunk)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  toks = torch.randint(0, cfg.vocab_size, (700,), generator=torch.Generator().manual_seed(3))
  whole, _ = engine.prefill(params=params, padded_tokens=toks, true_length=700, slot=0)
  prefix = None
  for at in range(0, 700, chunk):
    m = min(chunk, 700 - at)
    before = maxengine.ExistingPrefix(cache=prefix["cache"], common_prefix_tokens=toks[:at]) if at else None
    prefix, _ = engine.prefill(params=params, padded_tokens=toks[at : at + m], true_length=m, existing_prefix=before, slot=0)
  for name in ("key", "value"):
    assert torch.equal(whole["cache"][name], prefix["cache"][name])
  assert torch.equal(whole["logits"], prefix["logits"])


def test_chunk_entry_is_the_same_prefill():
  """mtx_prefill_chunk (at most max_rows positions) leaves what MaxEngine.prefill leaves of the same prompt, and refuses longer ones."""
  cfg = _config("llama2", 64)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  toks = torch.randint(0, cfg.vocab_size, (200,), generator=torch.Generator().manual_seed(3))
  prefix, _ = engine.prefill(params=params, padded_tokens=toks, true_length=200)
  plane = engine._staging
  engine._k[:, plane].zero_()
  dev = toks.to(device="cuda", dtype=torch.int32)
  first, logits = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(cfg.vocab_size, device="cuda")
  call = lambda n, at, last: engine.lib.mtx_prefill_chunk(engine._handle, dev.data_ptr() + 4 * at, n, at, plane, last, first.data_ptr(), logits.data_ptr(), None, None)
  assert call(120, 0, 0) == _lib.MTX_OK and call(80, 120, 1) == _lib.MTX_OK
  torch.cuda.synchronize()
  assert int(first) == int(prefix["tokens"])
  torch.testing.assert_close(logits, prefix["logits"].reshape(-1), rtol=4e-2, atol=4e-2 * float(logits.abs().max()))  # (two steps against one)
  assert call(257, 0, 0) == _lib.MTX_ERR_ARG and call(0, 0, 0) == _lib.MTX_ERR_ARG
