"""Prompts with a value row that holds no finite numbers: the positions that do not see it keep their bits, those that see it do not."""

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import ginodra, gugidra, ligidra, maxengine, pyconfig

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


def _layered(name, dim):
  if name == "gugidra":  # (the values are the keys before their rotation)
    return gugidra, gugidra.model_dict(256, 320, [gugidra.parallel_layer(4, 2, dim, 2, 32, 64, mlp=gugidra.dense_ff(256))] * 2)
  if name == "ginodra":
    return ginodra, ginodra.model_dict(256, 320, [ginodra.attention_layer(4, 4, dim, mlp=ginodra.dense_ff(256))] * 2)
  return ligidra, ligidra.model_dict(256, 320, [ligidra.attention_layer(4, 1, dim, softcap=20.0, mlp=ligidra.moe_ff(4, 4, 64, shared_ff=64))] * 2, side_dim=64)


@pytest.mark.parametrize("kind", ["nan", "inf"])
@pytest.mark.parametrize("name,dim,page", [("gugidra", 64, 16), ("gugidra", 256, 8), ("ginodra", 128, 24), ("ligidra", 64, 64), ("ligidra", 256, 40)])
def test_layered_portions(name, dim, page, kind):
  """The same for the logits of every token of portions of 700 and 260 tokens, in pages of many sizes."""
  design, model = _layered(name, dim)
  cfg = pyconfig.from_model_dict(model, dtype="bfloat16", per_device_batch_size=2, max_target_length=720, pagedattn_tokens_per_page=page,
                                 pagedattn_num_pages=2 * (720 // page + 1) + 2, max_step_rows=960)
  tensors = design.random_tensors(cfg, seed=3)
  embed = next(t for n, t in tensors.items() if "embed" in n and t.shape == (320, 256))
  value = next(t for n, t in tensors.items() if n.startswith("l0.") and n.endswith("left.k" if name == "gugidra" else ".v"))
  embed[:, 5] = 0.0
  embed[319, 5] = 8.0
  rng = np.random.Generator(np.random.PCG64(dim))
  toks = [rng.integers(0, 319, size=n).tolist() for n in (700, 260)]
  bad = (300, 255)
  for t, b in zip(toks, bad):
    t[b] = 319
  out = []
  for on in (False, True):
    if kind == "nan":
      embed[319, :4] = float("nan") if on else 0.5
    else:
      value[-1, 5] = 3e38 if on else 0.0
    engine = maxengine.MaxEngine(cfg)
    engine.load_params(tensors)
    engine.init_decode_state()
    out.append(engine.step([(s, t, list(range(len(t)))) for s, t in enumerate(toks)])[:, :319])  # (the head may be the embedding)
  clean, got = out
  assert torch.isfinite(clean).all()
  for lo, n, b in ((0, 700, 300), (700, 260, 255)):
    assert torch.equal(got[lo : lo + b], clean[lo : lo + b])
    assert not torch.isfinite(got[lo + b : lo + n]).all(1).any()
