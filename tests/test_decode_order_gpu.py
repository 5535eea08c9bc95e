"""Decode steps on the per-kernel attention: a slot's bits do not depend on where its length puts it in the sorted work list (step_kernels.cuh, attn_item)."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import maxengine, pyconfig

pytestmark = pytest.mark.gpu


def _config(kind, batch):
  kw = dict(base_num_decoder_layers=2, base_emb_dim=128, base_num_query_heads=4, base_num_kv_heads=2, head_dim=64, base_mlp_dim=256, vocab_size=512,
            per_device_batch_size=batch, max_prefill_predict_length=1024, max_target_length=1024 + 192, weight_dtype="bfloat16", scan_layers=False,
            attention="dot_product", materialize_logits=True)
  if kind == "gemma3":
    kw.update(model_name="gemma3-4b", head_dim=256, sliding_window_size=200)
  elif kind != "bf16":
    kw.update(quantize_kvcache=True, kv_quant_dtype=kind, kv_quant_axis="dkv")
  return pyconfig.initialize(None, **kw)


@pytest.mark.parametrize("kind,batch", [("bf16", 65), ("bf16", 256), ("int8", 200), ("fp8", 97), ("gemma3", 3), ("gemma3", 80)])
def test_slots_in_another_order(kind, batch):
  cfg = _config(kind, batch)
  rng = np.random.Generator(np.random.PCG64(batch))
  prompts, grown = rng.integers(1, 1025, size=batch), rng.integers(100, 192, size=batch)
  prompts[: batch // 2] = prompts[0]  # equal lengths among them
  tokens, order = torch.as_tensor(rng.integers(0, 512, size=(batch, 1)), dtype=torch.int32), rng.permutation(batch)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  out, cache = [], None
  for slots in (np.arange(batch), order):
    state = engine.fill_synthetic_context(prompts[slots], grown[slots])
    if cache is None:
      cache = {k: v.clone() for k, v in state["cache"].items() if torch.is_tensor(v) and v.dim() > 2}
      assert cache
    else:
      for k, v in cache.items():
        state["cache"][k][:, :batch].copy_(v[:, torch.as_tensor(order, device=v.device)])  # (a dense cache has a plane for prompts behind the slots')
    state["tokens"].copy_(tokens[slots])
    state, _ = engine.generate(params, state)
    out.append(state["logits"].clone())
  assert torch.equal(out[0][torch.as_tensor(order, device="cuda")], out[1])
