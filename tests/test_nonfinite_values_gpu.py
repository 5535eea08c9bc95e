"""Prompts with a value row that holds no finite numbers: the positions that do not see it keep their bits, those that see it do not."""

import pytest
import torch

from maxtext_indextts2_b200 import maxengine, pyconfig

pytestmark = pytest.mark.gpu


def _decoder(block, dim, heads, kv_heads, **kw):
  base = dict(base_num_decoder_layers=2, base_emb_dim=192, base_num_query_heads=heads, base_num_kv_heads=kv_heads, head_dim=dim, base_mlp_dim=320, vocab_size=512,
              per_device_batch_size=2, max_prefill_predict_length=832, max_target_length=900, weight_dtype="bfloat16", scan_layers=False,
              attention="dot_product", materialize_logits=True)
  if block == "gemma3":
    base.update(model_name="gemma3-4b", sliding_window_size=150)
  base.update(kw)
  return pyconfig.initialize(None, **base)


DECODERS = [("llama2", 64, 6, 2, {}), ("llama2", 128, 4, 4, {}), ("gemma3", 256, 8, 4, {}), ("gemma3", 256, 6, 2, {}), ("gemma3", 256, 8, 2, dict(sliding_window_size=64)), ("gemma3", 256, 8, 4, dict(sliding_window_size=400))]


@pytest.mark.parametrize("kind", ["nan", "inf"])
@pytest.mark.parametrize("block,dim,heads,kv_heads,kw", DECODERS)
def test_decoder_prompts(block, dim, heads, kv_heads, kw, kind):
  """The second layer's keys of a prompt with a token at `bad` whose embedding is NaN, or one of whose values in the first layer is infinite: of
  that layer's attention only positions at and behind it (as far as the window goes) see it."""
  cfg = _decoder(block, dim, heads, kv_heads, **kw)
  engine = maxengine.MaxEngine(cfg)
  params = engine.load_params(on_device_init=True, norm_jitter=0.1)
  engine.init_decode_state()
  embedding, wqkv = params.tensors["embedding"], params.tensors["wqkv"]
  embedding[:, 5] = 0.0  # (the only token with a 5th channel: its products with 3e38 overflow)
  embedding[511, 5] = 8.0
  spoil = (lambda on: embedding[511, :4].fill_(float("nan") if on else 0.5)) if kind == "nan" else (lambda on: wqkv[0, -1, 5].fill_(3e38 if on else 0.0))
  window = kw.get("sliding_window_size", 150) if block == "gemma3" else 10**6
  for n, bad in ((831, 300), (831, 511), (200, 77), (512, 256)):
    if block == "llama2" and n <= 256:  # (prefill_attn_kernel: within 64 positions)
      continue
    toks = torch.randint(0, 511, (n,), generator=torch.Generator().manual_seed(n))
    toks[bad] = 511
    keys = []
    for on in (False, True):
      spoil(on)
      prefix, _ = engine.prefill(params=params, padded_tokens=toks, true_length=n, slot=0)
      keys.append(prefix["cache"]["key"][1].clone())  # [heads, n, D]
    clean, got = keys
    assert torch.isfinite(clean).all()
    end = min(n, bad + window)
    assert torch.equal(got[:, :bad], clean[:, :bad]), (n, bad)
    assert torch.equal(got[:, end:], clean[:, end:]), (n, bad)
    assert not torch.isfinite(got[:, bad:end]).any(), (n, bad)
