"""Decode steps whose gated up-projection may take the pair GEMM (takes_wide_up in csrc/host_util.cuh; norm scales folded into the weights): bit for bit what the
row-major GEMM gives, and close to the steps with the norm scales left alone.  Row counts at the edges of the 32-row warps and the 128-row halves of its tile, and the
caches whose rows the split-K projections finish."""

import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from maxtext_indextts2_b200 import maxengine, pyconfig

pytestmark = pytest.mark.gpu

CACHES = {"bf16": {}, "int8": dict(quantize_kvcache=True, kv_quant_axis="dkv"), "fp8": dict(quantize_kvcache=True, kv_quant_dtype="fp8", kv_quant_axis="dkv"),
          "tokens": dict(quantize_kvcache=True, kv_quant_axis="heads_and_dkv"), "paged": dict(attention="paged", pagedattn_tokens_per_page=16)}


def _step(cache, dim, rows, mlp=4864, fold=True, graph=True, emb=768):
  """The state behind one generated token per slot, and the names of the kernels that ran."""
  kw = dict(attention="dot_product")
  kw.update(CACHES[cache])
  if cache == "paged":
    kw["pagedattn_num_pages"] = 6 * rows + 1
  cfg = pyconfig.initialize(None, base_num_decoder_layers=2, base_emb_dim=emb, base_num_query_heads=6, base_num_kv_heads=2, head_dim=dim, base_mlp_dim=mlp, vocab_size=640,
                            per_device_batch_size=rows, max_prefill_predict_length=48, max_target_length=80, weight_dtype="bfloat16", scan_layers=False,
                            materialize_logits=True, return_log_prob=True, decode_sampling_strategy="greedy", fold_norm_scales=fold, **kw)
  engine = maxengine.MaxEngine(cfg, use_cuda_graph=graph)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  lengths = np.random.Generator(np.random.PCG64(rows)).integers(1, 49, size=rows)
  state = engine.fill_synthetic_context(lengths, np.full(rows, 7), seed=3)
  state["tokens"].copy_(torch.randint(0, 640, (rows, 1), generator=torch.Generator().manual_seed(4), dtype=torch.int32))
  with profile(activities=[ProfilerActivity.CUDA], acc_events=True) as p:
    state, _ = engine.generate(params, state)
    torch.cuda.synchronize()
  got = {k: v.clone() for k, v in state["cache"].items() if torch.is_tensor(v)}
  return dict(got, logits=state["logits"].clone()), {e.name for e in p.events()}


@pytest.mark.parametrize("cache,dim,rows,emb,mlp,wide", [
    ("bf16", 64, 65, 768, 4864, True), ("bf16", 128, 97, 768, 4864, True), ("bf16", 64, 256, 768, 4864, True), ("int8", 64, 129, 768, 4864, True), ("int8", 64, 200, 768, 4864, True),
    ("fp8", 64, 255, 768, 4864, True), ("tokens", 64, 161, 768, 4864, True), ("paged", 64, 66, 768, 4864, True), ("paged", 128, 224, 768, 4864, True),
    ("bf16", 64, 200, 768, 9472, True),  # 148 tiles of 128 columns, more than 128 rows
    ("bf16", 64, 70, 768, 9472, False), ("tokens", 64, 64, 768, 4864, False), ("tokens", 64, 1, 768, 4864, False),  # (a full wave; rows that fill a quarter of a tile)
    ("bf16", 64, 200, 704, 4864, False), ("bf16", 64, 200, 832, 4864, True),  # (narrow layers)
    ("bf16", 64, 74, 768, 9728, False), ("bf16", 64, 74, 2048, 9728, True)])  # (152 tiles: a second wave, a short and a long K)
def test_up_projection_has_the_same_bits_on_either_gemm(cache, dim, rows, emb, mlp, wide, monkeypatch):
  """Logits and caches of a step on the GEMM that the rule picks and on the row-major one (MTX_ROWS_WIDE_UP=0)."""
  got, names = _step(cache, dim, rows, mlp, graph=False, emb=emb)
  monkeypatch.setenv("MTX_ROWS_WIDE_UP", "0")
  want, plain = _step(cache, dim, rows, mlp, graph=False, emb=emb)
  is_wide = lambda names: any("gemm_wide_kernel" in n for n in names)
  assert any("gemm_rows_kernel" in n for n in plain) and is_wide(names) == wide and not is_wide(plain)
  assert got.keys() == want.keys() and torch.isfinite(got["logits"]).all()
  assert all(torch.equal(got[k], want[k]) for k in want)


@pytest.mark.parametrize("cache,dim,rows", [("bf16", 64, 65), ("bf16", 128, 97), ("bf16", 64, 256), ("int8", 64, 128), ("int8", 64, 129), ("int8", 64, 200), ("fp8", 64, 255),
                                            ("tokens", 64, 40), ("tokens", 64, 161), ("paged", 64, 66), ("paged", 128, 224)])
def test_step_against_row_major_gemm(cache, dim, rows):
  """Norm scales folded into the weights (fused into the products around them) against norm scales left alone (the row-major GEMM, norms of their own)."""
  got, want = (_step(cache, dim, rows, fold=fold)[0]["logits"].double() for fold in (True, False))
  assert got.shape[0] == rows and torch.isfinite(got).all()
  # bf16 activations through two layers, 2^-9 for each of about ten roundings (and one step of an 8-bit cache's scale in the step's own keys); a row of its own is
  # off by its whole size
  off = (got - want).square().sum(-1).sqrt() / want.square().sum(-1).sqrt()
  assert float(off.max()) < 4e-2
