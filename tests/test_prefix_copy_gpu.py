"""mtx_copy_prefix: the rows that a prefill left in its plane, every layer and head, keys and values."""

import pytest
import torch

from maxtext_indextts2_b200 import _lib, maxengine, pyconfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,kw", [(64, {}), (128, {}), (256, dict(model_name="gemma3-4b", sliding_window_size=64)), (64, dict(quantize_kvcache=True, kv_quant_axis="dkv")),
                                    (64, dict(attention="paged", pagedattn_num_pages=60, pagedattn_tokens_per_page=16))])
def test_rows_of_a_prefix(dim, kw):
  cfg = pyconfig.initialize(None, **{**dict(base_num_decoder_layers=3, base_emb_dim=128, base_num_query_heads=6, base_num_kv_heads=3, head_dim=dim, base_mlp_dim=256,
                                            vocab_size=512, per_device_batch_size=2, max_prefill_predict_length=600, max_target_length=640, weight_dtype="bfloat16",
                                            scan_layers=False, attention="dot_product"), **kw})
  engine = maxengine.MaxEngine(cfg)
  engine.load_params(on_device_init=True)
  engine.init_decode_state()
  g = torch.Generator(device="cuda").manual_seed(1)
  for t in (engine._k, engine._v):
    t.copy_(torch.randn(t.shape, device="cuda", generator=g))
  copy = lambda n, slot, k, v: engine.lib.mtx_copy_prefix(engine._handle, n, slot, k, v, None)
  for n in (1, 7, 257, 600):  # less than a block's piece, an odd number, several pieces, all
    out = [torch.zeros(3, 3, n, dim, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    assert copy(n, engine._staging, out[0].data_ptr(), out[1].data_ptr()) == _lib.MTX_OK
    torch.cuda.synchronize()
    for got, cache in zip(out, (engine._k, engine._v)):
      assert torch.equal(got, cache[:, engine._staging, :, :n])
  k = out[0].data_ptr()
  assert copy(601, engine._staging, k, k) == _lib.MTX_ERR_ARG and copy(0, engine._staging, k, k) == _lib.MTX_ERR_ARG
  assert copy(1, -1, k, k) == _lib.MTX_ERR_ARG and copy(1, engine._staging, None, k) == _lib.MTX_ERR_ARG and copy(1, engine._staging, k + 2, k) == _lib.MTX_ERR_ARG
