"""What is timed when this framework is made faster: its engines' calls, as a serving program makes them.

Two engines answer ``MaxEngine(config)``.  The decoder engine runs the text-to-semantic GPT (`llama` below; IndexTTS2-scale: 24 layers of
width 1280 over a vocabulary of 264,192 text and audio tokens) and the gemma3 block; the layered engine runs the designs that list
their layers one by one, here kifusun (windowed sigmoid attention, heads mixed), gugidra (softmax attention beside mLSTM, gated linear
attention, routed experts) and zakelorn (windowed attention with kept first tokens beside decayed sums, routed and identity experts).

A pass is one call of the serving loop: `generate` (one token for every slot, the loop holding its tokens on the host), `prefill` (one
prompt; with `insert` the prefix is put into a slot, as every request does), or `mixed` (continuous batching: one prompt portion
beside the other slots' tokens).  Weights are random with the initialisers' distributions, contexts random-normal, lengths ragged.
Models are cut to a few layers where a layer is what counts; the flagship runs whole.
"""

import math

import numpy as np
import torch

from maxtext_indextts2_b200 import gugidra, kifusun, maxengine, pyconfig, zakelorn

TTS = dict(layers=24, emb=1280, heads=20, kv_heads=4, dim=64, mlp=5120, vocab=264192)
TINY = dict(layers=4, emb=256, heads=4, kv_heads=2, dim=64, mlp=1024, vocab=264192)
GEMMA = dict(layers=6, emb=2560, heads=8, kv_heads=4, dim=256, mlp=10240, vocab=262144, window=1024)
GEMMA_128 = dict(layers=6, emb=2048, heads=16, kv_heads=4, dim=128, mlp=8192, vocab=32768, window=1024)
GEMMA_64 = dict(layers=6, emb=1024, heads=16, kv_heads=8, dim=64, mlp=4096, vocab=32768, window=512)
BIG = dict(emb=2048, heads=16, kv_heads=4, dim=128, mlp=8192, window=1024, vocab=32768)
WIDE = dict(emb=2560, heads=8, kv_heads=4, dim=256, mlp=10240, window=1024, vocab=32768)
SMALL = dict(emb=1024, heads=16, kv_heads=8, dim=64, mlp=4096, window=512, vocab=32768)
LAYERED = ("kifusun", "gugidra", "zakelorn")
DECODER = ("llama", "gemma3")
PAGE = 64  # tokens per page of the layered engine's pools
GROW = 8192  # tokens a slot of a paged engine may grow by while it is measured


def listed():
  return [
      # the smallest call: the command line's tiny model, one user; launches and latency
      dict(name="generate tiny 1", model="llama", call="generate", batch=1, prompt=64, ring=64, kv="bf16", sampling="greedy", **TINY),
      # the flagship serving step: 64 utterances at once
      dict(name="generate tts 64", model="llama", call="generate", batch=64, prompt=1024, ring=512, kv="bf16", sampling="greedy", **TTS),
      # a throughput server's step: more slots than one tensor-core tile has rows, an odd number, an 8-bit cache
      dict(name="generate tts 200 int8", model="llama", call="generate", batch=200, prompt=1536, ring=512, kv="int8", sampling="greedy", **TTS),
      # a latency server's step over the paged cache, drawn from the nucleus, with the log-probability that a caller scores by
      dict(name="generate tts 23 paged", model="llama", call="generate", batch=23, prompt=777, ring=256, kv="paged", sampling="nucleus", **TTS),
      # text and reference audio of a long prompt
      dict(name="prefill tts 4000", model="llama", call="prefill", batch=4, prompt=4096, length=4000, kv="bf16", sampling="greedy", **TTS),
      # an ordinary prompt, its length as it comes, put into a slot
      dict(name="insert tts 389", model="llama", call="insert", batch=8, prompt=1024, length=389, kv="bf16", sampling="greedy", **TTS),
      # the block of the model that the expanded vocabulary is made for: five windowed layers and a global one
      dict(name="prefill gemma3 3001", model="gemma3", call="prefill", batch=4, prompt=4096, length=3001, kv="bf16", sampling="greedy", **GEMMA),
      dict(name="generate gemma3 48", model="gemma3", call="generate", batch=48, prompt=1024, ring=512, kv="bf16", sampling="greedy", **GEMMA),
      # a layered design under continuous batching: a portion of a prompt beside single tokens
      dict(name="mixed kifusun 500+31", model="kifusun", call="mixed", batch=32, prompt=1024, length=500, layers=2, **BIG),
      # layered designs with recurrences and routed experts: a long prompt, a decode step, a shorter prompt of an odd length
      dict(name="prefill gugidra 4096", model="gugidra", call="prefill", batch=4, prompt=4096, length=4096, layers=4, **BIG),
      dict(name="generate zakelorn 64", model="zakelorn", call="generate", batch=64, prompt=2048, length=2048, layers=4, **BIG),
      dict(name="prefill zakelorn 1777", model="zakelorn", call="prefill", batch=4, prompt=2048, length=1777, layers=4, **SMALL),
  ]


def _spread(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  """One more case: a model, a call, sizes spread over what the listed ones span."""
  model = rng.choice(("llama", "llama", "gemma3") + LAYERED)
  if model in DECODER:
    size = dict(rng.choice((TTS, TTS, TINY)) if model == "llama" else rng.choice((GEMMA, GEMMA_128, GEMMA_64)))
    if model == "llama":
      size["layers"] = rng.randint(2, size["layers"])
    call = rng.choice(("generate", "generate", "prefill", "insert"))
    if call == "generate":
      kv = rng.choice(("bf16", "int8", "fp8", "paged")) if model == "llama" else "bf16"
      batch = _spread(rng, 1, 200 if kv in ("int8", "fp8") else 128 if model == "llama" else 64)
      if batch > 64:
        size["layers"] = min(size["layers"], 12)
      return dict(model=model, call=call, batch=batch, prompt=rng.randint(64, 1536), ring=rng.randint(64, 512), kv=kv,
                  sampling=rng.choice(("greedy", "greedy", "weighted", "topk", "nucleus")), **size)
    length = _spread(rng, 20, 4000 if model == "llama" else 3001)
    return dict(model=model, call=call, batch=rng.randint(1, 8), prompt=length + rng.randint(0, 90), length=length, kv="bf16", sampling="greedy", **size)
  size = dict(rng.choice((BIG, WIDE, SMALL)))
  call = rng.choice({"kifusun": ("generate", "prefill", "mixed"), "gugidra": ("prefill",), "zakelorn": ("generate", "prefill")}[model])
  layers = rng.randint(1, 2 if size["emb"] == WIDE["emb"] else 4)
  if call == "prefill":
    length = _spread(rng, 20, 4096)
    return dict(model=model, call=call, batch=rng.randint(1, 8), prompt=length + rng.randint(0, 90), length=length, layers=layers, **size)
  if call == "mixed":
    length = _spread(rng, 20, 1000)
    return dict(model=model, call=call, batch=rng.randint(2, 48), prompt=max(length, rng.randint(64, 2000)), length=length, layers=layers, **size)
  length = _spread(rng, 64, 2048)
  return dict(model=model, call=call, batch=_spread(rng, 1, 64), prompt=length, length=length, layers=layers, **size)


# -- configurations, weights, inputs ------------------------------------------------------------------------------------------


def _decoder_config(c):
  kw = dict(base_num_decoder_layers=c["layers"], base_emb_dim=c["emb"], base_num_query_heads=c["heads"], base_num_kv_heads=c["kv_heads"],
            head_dim=c["dim"], base_mlp_dim=c["mlp"], vocab_size=c["vocab"], per_device_batch_size=c["batch"], weight_dtype="bfloat16",
            scan_layers=False, attention="dot_product", max_prefill_predict_length=c["prompt"], max_target_length=c["prompt"] + c.get("ring", 64),
            decode_sampling_strategy=c["sampling"], materialize_logits=True, return_log_prob=True)
  if c["model"] == "gemma3":
    kw.update(model_name="gemma3-4b", sliding_window_size=c["window"])
  if c["sampling"] == "topk":
    kw.update(decode_sampling_top_k=64)
  if c["sampling"] == "nucleus":
    kw.update(decode_sampling_nucleus_p=0.9)
  if c["kv"] in ("int8", "fp8"):
    kw.update(quantize_kvcache=True, kv_quant_dtype=c["kv"], kv_quant_axis="dkv")
  if c["kv"] == "paged":
    total = c["prompt"] + c["ring"] + GROW // 2
    kw.update(attention="paged", max_target_length=total, pagedattn_tokens_per_page=32, pagedattn_num_pages=c["batch"] * ((total + 31) // 32) + 1)
  return pyconfig.initialize(None, **kw)


def _rn(g, shape, std, mean=0.0):
  return torch.randn(shape, generator=g, device="cuda").mul_(std).add_(mean).to(torch.bfloat16)


def _decoder_weights(c, seed):
  """The parameter tree by the checkpoint's names, as the initialisers draw it (norm scales a little off one, as trained ones are)."""
  g = torch.Generator(device="cuda").manual_seed(seed)
  E, H, G, D, M, V = c["emb"], c["heads"], c["kv_heads"], c["dim"], c["mlp"], c["vocab"]
  scale = lambda n: {"scale": _rn(g, (n,), 0.1, 1.0)}
  dec = {"decoder_norm": scale(E)}
  for i in range(c["layers"]):
    attn = {"query": {"kernel": _rn(g, (E, H, D), E**-0.5 * D**-0.5)}, "key": {"kernel": _rn(g, (E, G, D), E**-0.5)},
            "value": {"kernel": _rn(g, (E, G, D), E**-0.5)}, "out": {"kernel": _rn(g, (H, D, E), (H * D) ** -0.5)}}
    mlp = {"mlp_layer_norm": scale(E), "wi_0": {"kernel": _rn(g, (E, M), E**-0.5)}, "wi_1": {"kernel": _rn(g, (E, M), E**-0.5)},
           "wo": {"kernel": _rn(g, (M, E), M**-0.5)}}
    if c["model"] == "gemma3":
      attn.update(query_norm=scale(D), key_norm=scale(D))
      dec[f"layers_{i}"] = {"pre_self_attention_norm": scale(E), "self_attention": attn, "post_self_attention_norm": scale(E), "mlp": mlp,
                            "post_ffw_norm": scale(E)}
    else:
      dec[f"layers_{i}"] = {"pre_self_attention_layer_norm": scale(E), "self_attention": attn, "mlp": mlp}
  if c["model"] != "gemma3":  # (gemma3 reads its embedding table)
    dec["logits_dense"] = {"kernel": _rn(g, (E, V), E**-0.5)}
  return {"params": {"token_embedder": {"embedding": _rn(g, (V, E), 1.0)}, "decoder": dec}}


def _layered_model(c):
  H, G, d, F, W, L = c["heads"], c["kv_heads"], c["dim"], c["mlp"], c["window"], c["layers"]
  if c["model"] == "kifusun":
    layers = [kifusun.attention_layer(H, G, d, d, W, ff=F, bias_max=float(W)) for _ in range(L)]
    return kifusun.model_dict(c["emb"], c["vocab"], layers)
  if c["model"] == "gugidra":
    ffs = [gugidra.dense_ff(F), gugidra.moe_ff(16, 4, F // 8, groups=4, keep=2, shared_ff=F // 2)]
    layers = [gugidra.parallel_layer(H, G, d, H // 2, d // 2, d, mlp=ffs[(i // 2) % 2]) if i % 2 == 0 else gugidra.gla_layer(H, d // 2, d, mlp=ffs[((i + 1) // 2) % 2])
              for i in range(L)]
    return gugidra.model_dict(c["emb"], c["vocab"], layers)
  r = min(d, 128)
  ffs = [zakelorn.dense_ff(F * 3 // 2), zakelorn.moe_ff(16, 4, F // 8, identity=4, groups=4, keep=3, shared_ff=F // 2)]
  layers = [zakelorn.parallel_layer(zakelorn.attention_part(H, G, d, window=W, keep_first=4, rot_dims=d // 2), zakelorn.lightning_part(H * d // r, r), 0.8, 1.1, ffs[i % 2])
            for i in range(L)]
  return zakelorn.model_dict(c["emb"], c["vocab"], layers, embed_scale=c["emb"] ** 0.5)


_DESIGN = {"kifusun": kifusun, "gugidra": gugidra, "zakelorn": zakelorn}


def _layered_config(c):
  B, n = c["batch"], c["prompt"]
  if c["call"] == "prefill":
    total, pages = n + 64, (n + PAGE - 1) // PAGE + B + 2
  else:
    total = n + GROW
    pages = B * ((total + PAGE - 1) // PAGE) + 2
  return pyconfig.from_model_dict(_layered_model(c), dtype="bfloat16", per_device_batch_size=B, max_target_length=total, pagedattn_tokens_per_page=PAGE,
                                  pagedattn_num_pages=pages, max_step_rows=max(n, B) if c["call"] == "prefill" else c["length"] + B)


def _lengths(c, seed):
  """Ragged contexts: (prompt tokens, generated tokens) per slot.  The ring of generated tokens is full or nearly so, as on a
  server that has run for a while, so that a pass costs the same however many came before it."""
  rng = np.random.Generator(np.random.PCG64(seed))
  P, R, B = c["prompt"], c["ring"], c["batch"]
  return rng.integers(max(1, P // 8), P + 1, size=B), rng.integers(max(1, R - R // 4), R, size=B)


def _tokens(c, seed, n):
  return torch.randint(0, c["vocab"], (n,), generator=torch.Generator().manual_seed(seed + 1), dtype=torch.int32)


def prepare(case, seed):
  """An engine with its weights, its slots' contexts where tokens are generated, and the pass's tokens on the host."""
  c = case
  if c["model"] in DECODER:
    engine = maxengine.MaxEngine(_decoder_config(c))
    params = engine.load_params(_decoder_weights(c, seed))
  else:
    cfg = _layered_config(c)
    engine = maxengine.MaxEngine(cfg)
    params = engine.load_params(_DESIGN[c["model"]].random_tensors(cfg, seed=seed, device="cuda"))
  s = dict(case=c, engine=engine, params=params)
  B = c["batch"]
  if c["call"] in ("prefill", "insert"):
    s["decode"] = engine.init_decode_state(rng=seed)
    s["tokens"] = torch.zeros(c["prompt"], dtype=torch.int32)
    s["tokens"][: c["length"]] = _tokens(c, seed, c["length"])
    return s
  if c["model"] in DECODER:
    s["decode"] = engine.fill_synthetic_context(*_lengths(c, seed), seed=seed)
  else:
    s["decode"] = engine.fill_synthetic_context(_contexts(c, seed), seed=seed)
  if c["call"] == "mixed":
    s["entries"] = _entries(c, seed)
  else:
    s["tokens"] = _tokens(c, seed, B).reshape(B, 1).pin_memory()
    s["result"] = torch.zeros(B, 3, dtype=torch.int32).pin_memory()
    s["log_prob"] = torch.zeros(B, 1, dtype=torch.float32).pin_memory() if c["model"] in DECODER else None
  return s


def _contexts(c, seed):
  rng = np.random.Generator(np.random.PCG64(seed))
  return [int(x) for x in rng.integers(max(1, c["prompt"] // 2), c["prompt"] + 1, size=c["batch"])]


def _entries(c, seed):
  """Slot 0 is a new request whose portion of `length` tokens is read; every other slot goes on by one token."""
  t = _tokens(c, seed, c["length"] + c["batch"]).tolist()
  n = c["length"]
  return [(0, t[:n], [n - 1])] + [(b, [t[n + b]], [0]) for b in range(1, c["batch"])]


def run(state):
  s, c, engine = state, state["case"], state["engine"]
  if c["call"] == "generate":
    s["decode"], out = engine.generate_to_host(s["params"], s["decode"], s["result"], s["tokens"], s["log_prob"])
    return {"logits": s["decode"]["logits"], "result": out.data, "log_prob": out.log_prob}
  if c["call"] == "mixed":
    engine.release_pages(0)
    return {"logits": engine.step(s["entries"])}
  prefix, out = engine.prefill(params=s["params"], padded_tokens=s["tokens"], true_length=c["length"], slot=0)
  if c["model"] in DECODER:
    got = {"logits": prefix["logits"], "result": out.data, "log_prob": out.log_prob, "key": prefix["cache"]["key"], "value": prefix["cache"]["value"]}
    if c["call"] == "insert":
      s["decode"] = engine.insert(prefix, s["decode"], c["batch"] - 1)
      got["slot_tokens"], got["slot_pos"] = s["decode"]["tokens"], s["decode"]["next_pos"]
    return got
  cache = s["decode"]["cache"]
  return {"logits": prefix["logits"], "result": out.data, "key_pages": cache["key_pages"], "value_pages": cache["value_pages"], "state": cache["recurrent_state"]}


# -- what a pass cannot do without ----------------------------------------------------------------------------------------------


def _seen(n, window, start=0):
  """Keys seen by the positions start .. start + n - 1 together."""
  i = np.arange(start, start + n, dtype=np.float64) + 1
  return float(np.minimum(i, window).sum() if window else i.sum())


def work(case):
  c = case
  E, H, G, D, M, V, L, B = (c[k] for k in ("emb", "heads", "kv_heads", "dim", "mlp", "vocab", "layers", "batch"))
  if c["model"] in DECODER:
    layer = E * (2 * H + 2 * G) * D + 3 * E * M
    kv_row = 2 * G * D * (1 if c["kv"] in ("int8", "fp8") else 2) + (8 * G if c["kv"] in ("int8", "fp8") else 0)
    local = lambda i: c["window"] if c["model"] == "gemma3" and i % 6 != 5 else 0
    if c["call"] == "generate":
      p, r = _lengths(c, 0)
      hidden = [max(0, c["prompt"] - local(i)) if local(i) else 0 for i in range(L)]  # cache rows before a layer's window
      ctx = [float(np.maximum(0, p - hidden[i]).sum() + r.sum()) for i in range(L)]
      return {"bytes": 2.0 * (L * layer + E * V + B * E) + sum(ctx) * kv_row + 4.0 * B * V, "flops": 2.0 * B * (L * layer + E * V) + 4.0 * sum(ctx) * H * D}
    n = c["length"]
    copies = 2 if c["call"] == "insert" else 1  # (the prefix that the caller holds, and the slot's rows)
    return {"bytes": 2.0 * (L * layer + E * V + n * E) + copies * float(n) * L * kv_row + 4.0 * V,
            "flops": 2.0 * (n * L * layer + E * V) + 4.0 * H * D * sum(_seen(n, local(i)) for i in range(L))}
  rows = B if c["call"] == "generate" else c["length"] + (B - 1 if c["call"] == "mixed" else 0)
  wanted = 1 if c["call"] == "prefill" else B
  W = 0 if c["model"] == "gugidra" else c["window"]
  weights, flops, moved = 0.0, 0.0, 0.0
  for i in range(L):
    attends, state = c["model"] != "gugidra" or i % 2 == 0, 0
    mats = E * (2 * H + 2 * G) * D if attends else 0
    if c["model"] == "gugidra":
      rh = H if i % 2 else H // 2
      state = rh * (D // 2) * D
      mats = (E * (2 * H + G) * D if attends else 0) + E * rh * (D + 3 * D)
      routed = ((i + 1) // 2 if i % 2 else i // 2) % 2 == 1
    if c["model"] == "zakelorn":
      r = min(D, 128)
      state = H * D * r
      mats += E * H * D + 5 * E * H * D  # the gate of the attention, the recurrence's five
      routed = i % 2 == 1
    if c["model"] == "kifusun" or not routed:
      ff_all = ff_row = 3 * E * M
    else:
      ff_row = 4 * 3 * E * (M // 8) + 3 * E * (M // 2)
      ff_all = min(16, 4 * rows) * 3 * E * (M // 8) + 3 * E * (M // 2)
    weights += 2.0 * (mats + ff_all)
    flops += 2.0 * rows * (mats + ff_row) + 4.0 * rows * state
    moved += 8.0 * state * (1 if c["call"] == "prefill" else B)
    if attends:
      ctx = 0.75 * c["prompt"]
      seen = _seen(c["length"], W) if c["call"] != "generate" else 0.0
      others = 0 if c["call"] == "prefill" else (B - 1 if c["call"] == "mixed" else B)
      seen += others * (min(ctx, W) if W else ctx)
      flops += 4.0 * H * D * seen
      moved += 4.0 * G * D * (rows + others * (min(ctx, W) if W else ctx))
  return {"bytes": weights + moved + 2.0 * (E * V + rows * E) + 4.0 * wanted * V, "flops": flops + 2.0 * wanted * E * V}


def tolerance(case):
  """bf16 operands and stores between the layers, fp32 sums: the error of a layer grows through those after it (routed experts: a
  near-tie of two experts moves a row).  Tokens are the largest of logits that are themselves rounded: each may differ, a third of the
  result's whole numbers; the others may not."""
  c = case
  if c["model"] == "llama":
    return {"rel": 0.08, "differ": 0.34}
  if c["model"] == "gemma3":
    return {"rel": 0.05, "differ": 0.34}
  if c["model"] == "kifusun":
    return {"rel": 0.035, "differ": 0.34}
  return {"rel": 0.1, "differ": 0.34}


# -- the same in 64 bits ----------------------------------------------------------------------------------------------------------


def _f(x):
  return x.to(device="cuda", dtype=torch.float64)


def _rms(x, eps):
  return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _softmax_rows(q, k, v, mask, scale=1.0, sink=None):
  """q [n, H, d], k [m, G, d], v [m, G, dv], mask [n, m] -> [n, H, dv]."""
  H, G = q.shape[1], k.shape[1]
  out = torch.empty(q.shape[0], H, v.shape[2], dtype=torch.float64, device="cuda")
  for h in range(H):
    g = h * G // H
    for a in range(0, q.shape[0], 1024):
      s = (q[a : a + 1024, h] @ k[:, g].T) * scale
      s.masked_fill_(~mask[a : a + 1024], -math.inf)
      top = s.amax(dim=1, keepdim=True)
      if sink is not None:
        top = torch.clamp(top, min=float(sink[h]))
      p = torch.exp(s - top)
      total = p.sum(dim=1, keepdim=True)
      if sink is not None:
        total = total + torch.exp(sink[h] - top)
      out[a : a + 1024, h] = (p / total) @ v[:, g]
  return out


def _half_turn(x, pos, base):
  """x [n, heads, d]: channel i is paired with i + d / 2, the angle pos / base^(2 i / d)."""
  half = x.shape[-1] // 2
  ang = pos.to(torch.float64)[:, None] * (float(base) ** (-2.0 * torch.arange(half, dtype=torch.float64, device="cuda") / x.shape[-1]))[None, :]
  co, si = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
  a, b = x[..., :half], x[..., half:]
  return torch.cat((a * co - b * si, b * co + a * si), dim=-1)


def _exact_decoder(c, seed):
  w = _decoder_weights(c, seed)["params"]
  s = prepare(c, seed) if c["call"] == "generate" else None
  gem = c["model"] == "gemma3"
  E, H, G, D, P, L = c["emb"], c["heads"], c["kv_heads"], c["dim"], c["prompt"], c["layers"]
  eps = 1e-6 if gem else 1e-5
  norm = lambda x, p: _rms(x, eps) * _f(p["scale"])
  if s is None:
    tok = _tokens(c, seed, c["length"]).cuda()
    pos = torch.arange(c["length"], device="cuda")
  else:
    tok = s["tokens"].reshape(-1).cuda()
    p_len, r_len = _lengths(c, seed)
    pos = torch.as_tensor(p_len + r_len, device="cuda")
    cache = s["decode"]["cache"]
    R, at = c["ring"], int(r_len.max())
  x = _f(w["token_embedder"]["embedding"][tok.long()])
  keys, values = [], []
  for l in range(L):
    lw = w["decoder"][f"layers_{l}"]
    sa, mlp = lw["self_attention"], lw["mlp"]
    window = c["window"] if gem and l % 6 != 5 else 0
    n = norm(x, lw["pre_self_attention_norm" if gem else "pre_self_attention_layer_norm"])
    q, k, v = (torch.einsum("te,ehd->thd", n, _f(sa[name]["kernel"])) for name in ("query", "key", "value"))
    base = 10000.0
    if gem:
      q, k = norm(q, sa["query_norm"]), norm(k, sa["key_norm"])
      base = 10000.0 if window else 1000000.0
    q, k = _half_turn(q, pos, base), _half_turn(k, pos, base)
    if gem:
      q = q * D**-0.5
    if s is None:
      i = torch.arange(x.shape[0], device="cuda")
      mask = i[None, :] <= i[:, None]
      if window:
        mask &= i[None, :] > i[:, None] - window
      o = _softmax_rows(q, k, v, mask)
      keys.append(k.permute(1, 0, 2))
      values.append(v.permute(1, 0, 2))
    else:
      o = torch.empty_like(q)
      for b in range(c["batch"]):
        n0, n1 = int(p_len[b]), int(r_len[b])
        if c["kv"] == "paged":
          pages = torch.as_tensor(s["engine"].page_state.page_map[b]).long().cuda()
          rows = [_f(cache[name][l][:, pages[: (n0 + n1 + 31) // 32]]).reshape(G, -1, D)[:, : n0 + n1].permute(1, 0, 2) for name in ("key_pages", "value_pages")]
        else:
          # a windowed layer sees the last `window` cache rows of the prompt's segment and of the ring
          lo = max(0, P - window) if window else 0
          ring = (at - n1 + torch.arange(n1, device="cuda")) % R
          if window:
            ring = ring[ring >= R - window]
          idx = torch.cat((torch.arange(lo, max(lo, n0), device="cuda"), P + ring))
          rows = []
          for name in ("key", "value"):
            u = cache[name][l, b][:, idx]
            if c["kv"] == "bf16":
              u = _f(u)
            else:
              sc = _f(cache[name + "_scale"][l, b][:, idx])[..., None]
              u = _f(u.view(torch.float8_e4m3fn).float()) * (sc / 448.0) if c["kv"] == "fp8" else (_f(u) - 128.0) * (sc / 127.5)
            rows.append(u.permute(1, 0, 2))
        kk, vv = torch.cat((rows[0], k[b : b + 1])), torch.cat((rows[1], v[b : b + 1]))
        sc = torch.einsum("gjd,sgd->gjs", q[b].reshape(G, H // G, D), kk)
        o[b] = torch.einsum("gjs,sgd->gjd", torch.softmax(sc, dim=-1), vv).reshape(H, D)
    y = o.reshape(-1, H * D) @ _f(sa["out"]["kernel"]).reshape(H * D, E)
    x = x + (norm(y, lw["post_self_attention_norm"]) if gem else y)
    n = norm(x, mlp["mlp_layer_norm"])
    a = n @ _f(mlp["wi_0"]["kernel"])
    a = torch.nn.functional.gelu(a, approximate="tanh") if gem else a * torch.sigmoid(a)
    y = (a * (n @ _f(mlp["wi_1"]["kernel"]))) @ _f(mlp["wo"]["kernel"])
    x = x + (norm(y, lw["post_ffw_norm"]) if gem else y)
  y = norm(x if s is not None else x[-1:], w["decoder"]["decoder_norm"])
  logits = torch.empty(y.shape[0], c["vocab"], dtype=torch.float64, device="cuda")
  for lo in range(0, c["vocab"], 32768):
    if gem:
      logits[:, lo : lo + 32768] = y @ _f(w["token_embedder"]["embedding"][lo : lo + 32768]).T / math.sqrt(E)
    else:
      logits[:, lo : lo + 32768] = y @ _f(w["decoder"]["logits_dense"]["kernel"][:, lo : lo + 32768])
  out = {"logits": logits[:, None, :], "result": None, "log_prob": None}
  if s is None:
    out.update(key=torch.stack(keys), value=torch.stack(values))
    if c["call"] == "insert":
      out.update(slot_tokens=None, slot_pos=None)
  return out


def _pair_turn(x, pos, dims, base):
  """x [n, heads, d]: the pairs (2 i, 2 i + 1), i < dims / 2, turn by pos * base^(-2 i / dims)."""
  ang = pos.to(torch.float64)[:, None] * (float(base) ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims))[None, :]
  co, si = torch.cos(ang)[:, None, :], torch.sin(ang)[:, None, :]
  a, b = x[..., 0:dims:2], x[..., 1:dims:2]
  out = x.clone()
  out[..., 0:dims:2], out[..., 1:dims:2] = a * co - b * si, b * co + a * si
  return out


def _sums(q, k, v, decay, S, put=None, kept=None):
  """S <- decay S + put k v^T, o = S^T q, token by token; q, k [n, H, d], v [n, H, dv], decay [n, H, d], S [H, d, dv]; `kept` collects
  (a second sum over the keys alone) for the mLSTM's denominator."""
  out = torch.empty(v.shape, dtype=torch.float64, device="cuda")
  w = k if put is None else k * put[..., None]
  for t in range(q.shape[0]):
    S = decay[t][:, :, None] * S + w[t][:, :, None] * v[t][:, None, :]
    out[t] = torch.einsum("hdc,hd->hc", S, q[t])
    if kept is not None:
      kept[0] = decay[t] * kept[0] + w[t]
      kept[1][t] = (kept[0] * q[t]).sum(dim=-1)
  return out, S


def _gated_ff(h, t, p, act):
  return act(h @ t[p + "gate"].T, h @ t[p + "up"].T) @ t[p + "down"].T


def _experts(h, t, p, chosen, weight, experts, act):
  y = torch.zeros_like(h)
  for e in range(experts):
    r, i = torch.nonzero(chosen == e, as_tuple=True)
    if r.numel():
      y.index_add_(0, r, weight[r, i][:, None] * _gated_ff(h[r], t, f"{p}e{e}.", act))
  return y


def _kept_groups(choice, groups, keep, best):
  n, m = choice.shape
  by = choice.reshape(n, groups, m // groups)
  score = by.amax(dim=-1) if best else by.topk(2, dim=-1).values.sum(dim=-1)
  ok = torch.zeros(n, groups, dtype=torch.bool, device="cuda").scatter_(1, score.topk(keep, dim=1).indices, True)
  return by.masked_fill(~ok[:, :, None], -math.inf).reshape(n, m)


def _clamped(g, u):
  g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
  return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _gugidra(model, t, tokens, pos, past):
  """One sequence from `past` (per layer: S, n, m, k, v); updates it; the final hidden rows."""
  eps = model["norm"]["eps"]
  wn = lambda y, w: _rms(y, eps) * (1.0 + w)
  x = t["embed"][tokens]
  for i, l in enumerate(model["layers"]):
    m, st = l["mixer"], past[i]
    h, n = wn(x, t[f"l{i}.norm1"]), x.shape[0]
    heads = lambda name, H: (h @ t[name].T).reshape(n, H, -1)
    if l["type"] == "gla":
      p, H, d = f"l{i}.mix.", m["heads"], m["dim"]
      z = (h @ t[p + "a1"].T) @ t[p + "a2"].T + t[p + "a2.b"]
      a = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).reshape(n, H, d)
      o, st["S"] = _sums(heads(p + "q", H) * d**-0.5, heads(p + "k", H), heads(p + "v", H), a, st["S"])
      o = (_rms(o, eps) * t[p + "norm"]).reshape(n, -1)
      y = (o * torch.nn.functional.silu(h @ t[p + "g"].T)) @ t[p + "o"].T
    else:
      p, a = f"l{i}.mix.left.", m["left"]
      H, G, d = a["heads"], a["kv_heads"], a["dim"]
      q = (h @ t[p + "q"].T + t[p + "q.b"]).reshape(n, H, d)
      k = (h @ t[p + "k"].T + t[p + "k.b"]).reshape(n, G, d)
      st["v"] = torch.cat((st["v"], k))
      st["k"] = torch.cat((st["k"], _pair_turn(k, pos, a["rot"]["dims"], a["rot"]["base"])))
      mask = torch.arange(st["k"].shape[0], device="cuda")[None, :] <= pos[:, None]
      o = _softmax_rows(_pair_turn(q, pos, a["rot"]["dims"], a["rot"]["base"]), st["k"], st["v"], mask, a["scale"])
      y = m["left_scale"] * (o.reshape(n, -1) @ t[p + "o"].T + t[p + "o.b"])
      p, r = f"l{i}.mix.right.", m["right"]
      H, d, cap = r["heads"], r["dim"], r["gate_cap"]
      ig = cap * torch.tanh((h @ t[p + "i"].T + t[p + "i.b"]) / cap)
      fg = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ t[p + "f"].T + t[p + "f.b"]) / cap))
      igc, fgc, top = ig.cpu(), fg.cpu(), st["m"].cpu()
      tops = torch.empty(n + 1, H, dtype=torch.float64)
      tops[0] = top
      for j in range(n):
        tops[j + 1] = torch.maximum(fgc[j] + tops[j], igc[j])
      tops = tops.cuda()
      keep, put = torch.exp(fg + tops[:-1] - tops[1:]), torch.exp(ig - tops[1:])
      kept = [st["n"], torch.empty(n, H, dtype=torch.float64, device="cuda")]
      o, st["S"] = _sums(heads(p + "q", H) * d**-0.5, heads(p + "k", H), heads(p + "v", H), keep[..., None].expand(n, H, d), st["S"], put, kept)
      st["n"], st["m"] = kept[0], tops[-1]
      o = o / (torch.maximum(kept[1].abs(), torch.exp(-tops[1:])) + 1e-6)[..., None]
      y = y + m["right_scale"] * ((_rms(o, eps).reshape(n, -1) * t[p + "norm"] * torch.sigmoid(h @ t[p + "g"].T)) @ t[p + "o"].T)
    x = x + wn(y, t[f"l{i}.norm1b"])
    f, p = l["mlp"], f"l{i}.mlp."
    h = wn(x, t[f"l{i}.norm2"])
    if f["kind"] == "dense":
      y = _gated_ff(h, t, p, _clamped)
    else:
      r = f["router"]
      score = torch.sigmoid(h @ t[p + "router"].T)
      chosen = _kept_groups(score + t[p + "correction"], r["groups"]["count"], r["groups"]["keep"], False).topk(r["top"], dim=1).indices
      weight = score.gather(1, chosen)
      y = _experts(h, t, p, chosen, weight / weight.sum(dim=1, keepdim=True), r["experts"], _clamped) + _gated_ff(h, t, p + "shared.", _clamped)
    x = x + wn(y, t[f"l{i}.norm2b"])
  return wn(x, t["final.norm"])


def _zakelorn(model, t, tokens, pos, past):
  eps = model["norm"]["eps"]
  ln = lambda y, name: torch.nn.functional.layer_norm(y, y.shape[-1:], t[name], t[name + ".b"], eps)
  x = t["embed"][tokens] * model["embedding"]["scale"]
  silu = torch.nn.functional.silu
  gate = lambda g, u: silu(g) * u
  n = x.shape[0]
  for i, l in enumerate(model["layers"]):
    m, st = l["mixer"], past[i]
    a, p = m["left"], f"l{i}.mix.left."
    H, G = a["heads"], a["kv_heads"]
    turn = lambda y: _rms(_pair_turn(y, pos, a["rot"]["dims"], a["rot"]["base"]), eps)
    q, k = turn((x @ t[p + "q"].T).reshape(n, H, -1)), turn((x @ t[p + "k"].T).reshape(n, G, -1))
    st["k"], st["v"] = torch.cat((st["k"], k)), torch.cat((st["v"], (x @ t[p + "v"].T).reshape(n, G, -1)))
    j = torch.arange(st["k"].shape[0], device="cuda")[None, :]
    mask = (j <= pos[:, None]) & ((j > pos[:, None] - a["mask"]["size"]) | (j < a["mask"]["keep_first"]))
    o = _softmax_rows(q, st["k"], st["v"], mask, a["scale"], t[p + "sink"]).reshape(n, -1)
    y = m["left_scale"] * ((o * torch.sigmoid(x @ t[p + "g"].T)) @ t[p + "o"].T)
    r, p = m["right"], f"l{i}.mix.right."
    H, d = r["heads"], r["dim"]
    q, k, v = (silu(x @ t[p + name].T).reshape(n, H, -1) for name in "qkv")
    decay = torch.tensor(r["decay"], dtype=torch.float64, device="cuda")[None, :, None].expand(n, H, d)
    o, st["S"] = _sums(q, k, v, decay, st["S"])
    y = y + m["right_scale"] * ((_rms(o.reshape(n, -1), eps) * t[p + "norm"] * torch.sigmoid(x @ t[p + "g"].T)) @ t[p + "o"].T)
    x = x + ln(y, f"l{i}.norm1") * t[f"l{i}.ls1"]
    f, p = l["mlp"], f"l{i}.mlp."
    if f["kind"] == "dense":
      y = torch.nn.functional.gelu(x @ t[p + "up"].T, approximate="tanh") @ t[p + "down"].T
    else:
      r = f["router"]
      score = torch.softmax(x @ t[p + "router"].T, dim=-1)
      chosen = _kept_groups(score + t[p + "correction"], r["groups"]["count"], r["groups"]["keep"], True).topk(r["top"], dim=1).indices
      weight = score.gather(1, chosen)
      y = _experts(x, t, p, chosen, weight, r["experts"], gate) + (weight * (chosen >= r["experts"])).sum(dim=1, keepdim=True) * x
      y = y + torch.sigmoid(x @ t[p + "shared.sg"].T) * _gated_ff(x, t, p + "shared.", gate)
    x = x + ln(y, f"l{i}.norm2") * t[f"l{i}.ls2"]
  return ln(x, "final.norm")


def _kifusun(model, t, tokens, pos, past):
  eps = model["norm"]["eps"]
  x = t["embed"][tokens] * model["embedding"]["scale"]
  n, first = x.shape[0], None
  for i, l in enumerate(model["layers"]):
    m, st, p = l["mixer"], past[i], f"l{i}.mix."
    H, G, W = m["heads"], m["kv_heads"], m["mask"]["size"]
    q = _rms((x @ t[p + "q"].T + t[p + "q.b"]).reshape(n, H, -1), eps) * t[p + "q.norm"]
    k = _rms((x @ t[p + "k"].T + t[p + "k.b"]).reshape(n, G, -1), eps) * t[p + "k.norm"]
    v = (x @ t[p + "v"].T + t[p + "v.b"]).reshape(n, G, -1)
    if i == 0:
      first = v
    else:
      v = (1.0 - t[p + "vmix"]) * v + t[p + "vmix"] * first
    st["k"], st["v"] = torch.cat((st["k"], k)), torch.cat((st["v"], v))
    rel, rows = t[p + "rel"], t[p + "rel"].shape[0]
    half = rows // 2
    dist = np.arange(W)
    far = np.maximum(dist, half).astype(np.float32) / np.float32(half)
    steps = np.floor(np.log(far) / np.float32(math.log(m["bias_max"] / half)) * np.float32(rows - half)).astype(np.int64)
    bucket = torch.as_tensor(np.where(dist < half, dist, np.minimum(rows - 1, half + steps)), device="cuda")
    o = torch.empty(n, H, v.shape[2], dtype=torch.float64, device="cuda")
    for a in range(0, n, 256):
      b = min(n, a + 256)
      lo, hi = max(0, int(pos[a]) - W + 1), int(pos[b - 1]) + 1
      kk, vv = (y[lo:hi].repeat_interleave(H // G, dim=1) for y in (st["k"], st["v"]))
      d = pos[a:b, None] - torch.arange(lo, hi, device="cuda")[None, :]
      seen = (d >= 0) & (d < W)
      s = torch.einsum("ihd,jhd->hij", q[a:b], kk) * m["scale"]
      s = m["softcap"] * torch.tanh(s / m["softcap"]) + rel[bucket[d.clamp(0, W - 1)]].permute(2, 0, 1)
      w = torch.sigmoid(s + t[p + "pb"][:, None, None]) * seen
      o[a:b] = torch.einsum("hij,jhd->ihd", torch.einsum("hg,gij->hij", t[p + "talk"], w), vv)
    x = x + _rms(o.reshape(n, -1) @ t[p + "o"].T, eps) * t[f"l{i}.norm1"]
    gelu = lambda g, u: torch.nn.functional.gelu(g, approximate="tanh") * u
    x = x + _rms(_gated_ff(x, t, f"l{i}.mlp.", gelu), eps) * t[f"l{i}.norm2"]
  return _rms(x, eps) * t["final.norm"]


def _exact_layered(c, seed):
  cfg, model = _layered_config(c), _layered_model(c)
  t = {k: _f(v) for k, v in _DESIGN[c["model"]].random_tensors(cfg, seed=seed, device="cuda").items()}
  forward = {"kifusun": _kifusun, "gugidra": _gugidra, "zakelorn": _zakelorn}[c["model"]]
  head = t["embed"] if c["model"] == "zakelorn" else t["head"]
  zeros = lambda *shape: torch.zeros(shape, dtype=torch.float64, device="cuda")

  def empty():
    past = []
    for l in model["layers"]:
      m = l["mixer"]
      a = m if c["model"] == "kifusun" else m.get("left")
      r = None if c["model"] == "kifusun" else m.get("right", m)
      past.append({"k": zeros(0, a["kv_heads"], a["dim"]) if a else None, "v": zeros(0, a["kv_heads"], a["vdim"]) if a else None,
                   "S": zeros(r["heads"], r["dim"], r["vdim"]) if r else None, "n": zeros(r["heads"], r["dim"]) if r else None, "m": zeros(r["heads"]) if r else None})
    return past

  def logits_of(y):
    z = y @ head.T
    return 30.0 * torch.tanh(z / 30.0) if c["model"] == "gugidra" else z

  if c["call"] == "prefill":
    n, past = c["length"], empty()
    y = forward(model, t, _tokens(c, seed, n).cuda().long(), torch.arange(n, device="cuda"), past)
    pages, slots = int(cfg.pagedattn_num_pages), c["batch"] + 1

    def pool(rows):  # pages 1, 2, .. in order
      p = zeros(rows.shape[1], pages * PAGE, rows.shape[2])
      p[:, PAGE : PAGE + n] = rows.permute(1, 0, 2)
      return p.reshape(rows.shape[1], pages, PAGE, rows.shape[2])

    def slot(x):
      p = zeros(slots, *x.shape)
      p[0] = x
      return p

    state = []
    for l, st in zip(model["layers"], past):
      if st["S"] is not None:
        state.append(slot(st["S"].transpose(1, 2)))
        if l["type"] == "parallel" and c["model"] == "gugidra":
          state += [slot(st["n"]), slot(st["m"])]
    return {"logits": logits_of(y[-1:])[None], "result": None, "key_pages": [pool(st["k"]) for st in past if st["k"] is not None],
            "value_pages": [pool(st["v"]) for st in past if st["v"] is not None], "state": state}

  s = prepare(c, seed)
  ctx, cache, maps = _contexts(c, seed), s["decode"]["cache"], s["engine"].page_state.page_map

  def held(b):
    past, i_pool, i_state = empty(), 0, 0
    pages = torch.as_tensor(maps[b]).long().cuda()[: (ctx[b] + PAGE - 1) // PAGE]
    for l, st in zip(model["layers"], past):
      if st["k"] is not None:
        for name, pools in (("k", "key_pages"), ("v", "value_pages")):
          rows = _f(cache[pools][i_pool][:, pages])
          st[name] = rows.reshape(rows.shape[0], -1, rows.shape[3])[:, : ctx[b]].permute(1, 0, 2)
        i_pool += 1
      if st["S"] is not None:
        st["S"] = _f(cache["recurrent_state"][i_state][b]).transpose(1, 2)
        i_state += 1
        if l["type"] == "parallel" and c["model"] == "gugidra":
          st["n"], st["m"] = _f(cache["recurrent_state"][i_state][b]), _f(cache["recurrent_state"][i_state + 1][b])
          i_state += 2
    return past

  rows = []
  if c["call"] == "mixed":
    for b, tokens, _ in s["entries"]:
      start = 0 if b == 0 else ctx[b]
      pos = torch.arange(start, start + len(tokens), device="cuda")
      rows.append(forward(model, t, torch.tensor(tokens, device="cuda"), pos, empty() if b == 0 else held(b))[-1:])
    return {"logits": logits_of(torch.cat(rows))}
  for b in range(c["batch"]):
    rows.append(forward(model, t, s["tokens"][b].cuda().long(), torch.tensor([ctx[b]], device="cuda"), held(b)))
  return {"logits": logits_of(torch.cat(rows))[:, None, :], "result": None, "log_prob": None}


def exact(case, seed):
  """The pass in float64 with plain torch: from the same weights (as bf16 holds them), tokens and cached rows."""
  return _exact_decoder(case, seed) if case["model"] in DECODER else _exact_layered(case, seed)
