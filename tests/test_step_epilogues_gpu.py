"""What the decode steps' projections do with their sums (csrc/gemm_rows.cuh): rotated queries, appended keys and values, in bfloat16 and in 8 bits."""

import ctypes

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import _lib, maxengine, pyconfig

pytestmark = pytest.mark.gpu


def _ptr(t):
  return ctypes.c_void_p(t.data_ptr())


def _qkv(rows, E, Hq, Hkv, D, scratch_offset):
  """Queries, keys and values of `rows` random rows through mtx_qkv_rope_append, its scratch so many bytes behind an allocation's start."""
  lib = _lib.load()
  g = torch.Generator(device="cuda").manual_seed(rows + E)
  rn = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
  x, w = rn(256, E), rn((Hq + 2 * Hkv) * D, E) / E**0.5
  T = 40
  pos, row = (torch.randint(0, hi, (rows,), generator=g, device="cuda").to(torch.int32) for hi in (3000, T))
  plane = torch.arange(rows, device="cuda", dtype=torch.int32)
  k, v = (torch.zeros(rows, Hkv, T, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
  q = torch.zeros(rows, Hq * D, dtype=torch.bfloat16, device="cuda")
  scratch = torch.empty(lib.mtx_qkv_rope_append_scratch_bytes(rows, D) + 256, dtype=torch.uint8, device="cuda")[scratch_offset:]
  stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
  _lib.check(lib.mtx_qkv_rope_append(_ptr(x), _ptr(w), _ptr(pos), _ptr(plane), _ptr(row), _ptr(q), _ptr(k), _ptr(v), rows, E, Hq, Hkv, D, T, 1.0, 10000.0, _ptr(scratch), stream))
  torch.cuda.synchronize()
  return q, k, v


@pytest.mark.parametrize("rows,E,Hq,Hkv,D", [(5, 256, 4, 2, 64), (65, 512, 4, 2, 64), (200, 512, 8, 8, 128), (256, 64, 20, 4, 64)])
def test_scratch_of_eight_byte_alignment(rows, E, Hq, Hkv, D):
  """The table of angles in the caller's scratch holds pairs of floats: any address that suits them will do, in every plan of the projection."""
  assert all(torch.equal(a, b) for a, b in zip(_qkv(rows, E, Hq, Hkv, D, 0), _qkv(rows, E, Hq, Hkv, D, 8)))


def _appended(rows, heads, kv_heads, emb, **kw):
  """(keys, values) and, of an 8-bit cache, their scales that a decode step appends in its first layer: [slot, kv head, dim] / [slot, kv head]."""
  cfg = pyconfig.initialize(None, base_num_decoder_layers=1, base_emb_dim=emb, base_num_query_heads=heads, base_num_kv_heads=kv_heads, head_dim=64, base_mlp_dim=256, vocab_size=640,
                            per_device_batch_size=rows, max_prefill_predict_length=48, max_target_length=80, weight_dtype="bfloat16", scan_layers=False, attention="dot_product",
                            materialize_logits=True, decode_sampling_strategy="greedy", **kw)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  lengths = np.random.Generator(np.random.PCG64(rows)).integers(1, 49, size=rows)
  state = engine.fill_synthetic_context(lengths, np.full(rows, 7), seed=3)
  state["tokens"].copy_(torch.randint(0, 640, (rows, 1), generator=torch.Generator().manual_seed(4), dtype=torch.int32))
  state, _ = engine.generate(params, state)
  at = lambda name: state["cache"][name][0][:rows, :, 48 + 7].clone()  # (a bfloat16 cache has a plane more)
  return [at(n) for n in ("key", "value")] + ([at(n + "_scale").float() for n in ("key", "value")] if "quantize_kvcache" in kw else [])


@pytest.mark.parametrize("dtype", ["int8", "fp8"])
@pytest.mark.parametrize("rows,heads,kv_heads,emb", [(65, 6, 2, 320), (97, 3, 1, 640), (128, 20, 4, 1280), (129, 4, 4, 64), (200, 20, 4, 1280), (256, 3, 1, 640)])
def test_8_bit_rows_are_the_bfloat16_rows_quantised(rows, heads, kv_heads, emb, dtype):
  """Byte for byte: the projection's plan is the same for both caches, and so are its sums and its roundings.  K cut in 2, 4 and 8 parts and left whole (emb 64), an odd
  number of heads, rows at the edges of the 128-row blocks."""
  plain = _appended(rows, heads, kv_heads, emb)
  got = _appended(rows, heads, kv_heads, emb, quantize_kvcache=True, kv_quant_axis="dkv", kv_quant_dtype=dtype)
  for x, q, scale in zip((t.float() for t in plain), got[:2], got[2:]):
    assert torch.equal(scale, x.abs().amax(-1))
    y = x * torch.div(torch.full_like(scale, 448.0 if dtype == "fp8" else 127.5), scale)[..., None]  # (a number / a tensor is a product with its reciprocal)
    want = y.to(torch.float8_e4m3fn).view(torch.uint8) if dtype == "fp8" else (y.round().clamp(-128, 127) + 128).to(torch.uint8)
    assert torch.equal(q.view(torch.uint8), want)
