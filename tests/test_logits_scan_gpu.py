"""The persistent step's scan of a logits tile (csrc/step_persistent.cuh, pk_logits_scan): 2 to 32 threads per row by the number of rows, a vocabulary that
ends inside a tile, a log-softmax whose values spread over many octaves."""

import pytest
import torch

from maxtext_indextts2_b200 import maxengine, pyconfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 4, 5, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("softcap", [0.0, 20.0])
def test_token_and_log_prob_of_the_rows(rows, softcap):
  cfg = pyconfig.initialize(None, base_num_decoder_layers=1, base_emb_dim=128, base_num_query_heads=4, base_num_kv_heads=2, head_dim=64, base_mlp_dim=256, vocab_size=1096,
                            per_device_batch_size=rows, max_prefill_predict_length=64, max_target_length=128, weight_dtype="bfloat16", scan_layers=False,
                            attention="dot_product", materialize_logits=True, return_log_prob=True, final_logits_soft_cap=softcap)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  state = engine.fill_synthetic_context([40] * rows, [10] * rows)
  for _ in range(3):
    state, result = engine.generate(params, state)
    logits = state["logits"][:, 0].double()
    assert torch.equal(result.data[:, 0].cpu().long(), torch.as_tensor(logits.cpu().numpy().argmax(axis=-1)))  # (the lowest index of equal values)
    want = torch.log_softmax(logits, dim=-1).amax(dim=-1)
    # 1096 exponentials by ex2.approx (2^-22 each) and fp32 sums: 1e-6 of the sum; the logarithm of it beside values of up to 10
    assert float((result.log_prob.reshape(-1).double() - want).abs().max()) < 2e-5
