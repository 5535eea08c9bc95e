"""Decode steps of 65 to 256 slots whose gated up-projection has columns enough for the pair GEMM (norm scales folded into the weights) against the same steps on
the row-major GEMM (norm scales left alone): row counts at the edges of the 32-row warps and the 128-row halves of its tile, and the caches whose rows the
split-K projections finish."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import maxengine, pyconfig

pytestmark = pytest.mark.gpu

CACHES = {"bf16": {}, "int8": dict(quantize_kvcache=True, kv_quant_axis="dkv"), "fp8": dict(quantize_kvcache=True, kv_quant_dtype="fp8", kv_quant_axis="dkv"),
          "tokens": dict(quantize_kvcache=True, kv_quant_axis="heads_and_dkv"), "paged": dict(attention="paged", pagedattn_tokens_per_page=16)}


@pytest.mark.parametrize("cache,dim,rows", [("bf16", 64, 65), ("bf16", 128, 97), ("bf16", 64, 256), ("int8", 64, 128), ("int8", 64, 129), ("int8", 64, 200), ("fp8", 64, 255),
                                            ("tokens", 64, 40), ("tokens", 64, 161), ("paged", 64, 66), ("paged", 128, 224)])
def test_step_against_row_major_gemm(cache, dim, rows):
  out = []
  for fold in (True, False):
    kw = dict(attention="dot_product")
    kw.update(CACHES[cache])
    if cache == "paged":
      kw["pagedattn_num_pages"] = 6 * rows + 1
    cfg = pyconfig.initialize(None, base_num_decoder_layers=2, base_emb_dim=320, base_num_query_heads=6, base_num_kv_heads=2, head_dim=dim, base_mlp_dim=4864, vocab_size=640,
                              per_device_batch_size=rows, max_prefill_predict_length=48, max_target_length=80, weight_dtype="bfloat16", scan_layers=False,
                              materialize_logits=True, return_log_prob=True, decode_sampling_strategy="greedy", fold_norm_scales=fold, **kw)
    assert 2 * (2 * cfg.mlp_dim // 128) > 148  # (its K stays whole: enqueue_step's wide_up)
    engine = maxengine.MaxEngine(cfg)
    params = engine.load_params(on_device_init=True, norm_jitter=0.1)
    lengths = np.random.Generator(np.random.PCG64(rows)).integers(1, 49, size=rows)
    state = engine.fill_synthetic_context(lengths, np.full(rows, 7), seed=3)
    state["tokens"].copy_(torch.randint(0, 640, (rows, 1), generator=torch.Generator().manual_seed(4), dtype=torch.int32))
    state, _ = engine.generate(params, state)
    out.append(state["logits"].double().clone())
  got, want = out
  assert got.shape[0] == rows and torch.isfinite(got).all()
  # bf16 activations through two layers, 2^-9 for each of about ten roundings (and one step of an 8-bit cache's scale in the step's own keys); a row of its own is
  # off by its whole size
  off = (got - want).square().sum(-1).sqrt() / want.square().sum(-1).sqrt()
  assert float(off.max()) < 4e-2
