"""Workloads that a user of this package has it do, for timing and for comparing results.

  listed()          the named workloads
  draw(rng)         one more of the same ranges
  prepare(case, s)  inputs, weights and compiled handles on the GPU, made from the seed `s`
  run(state)        one pass through the public entry points
  work(case)        bytes and floating-point operations the pass cannot do without
  tolerance(case)   how far another correct implementation may be off

Six kinds of work (`op`): attention forward, attention with a per-key score (H2O, RoCo, SnapKV, Corm), KeyFormer, the
KV-cache eviction that follows a score, the bandwidth ops around attention, and a whole decoder layer.
"""
import math

import torch

from deepgengraph_b200 import attention, layer, native_ops
from deepgengraph_b200.compile import compile as compile_module
from deepgengraph_b200.kernels import KERNEL_ZOO

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
SCORE_OPS = ("h2o", "roco", "snapkv", "corm")


def attn(name, batch, q_len, kv_len, heads, kv_heads, head_dim, dtype, window=-1, softcap=0.0, layout="dense"):
  case = dict(op="attn", batch=batch, q_len=q_len, kv_len=kv_len, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
              dtype=dtype, window=window, softcap=softcap, layout=layout)
  return dict(case, name=name) if name else case


def score(name, op, batch, q_len, kv_len, heads, kv_heads, dtype):
  case = dict(op=op, batch=batch, q_len=q_len, kv_len=kv_len, heads=heads, kv_heads=kv_heads, head_dim=128, dtype=dtype)
  return dict(case, name=name) if name else case


def keyformer(name, batch, seq, heads, dtype, tau, seeded):
  case = dict(op="kf", batch=batch, q_len=seq, kv_len=seq, heads=heads, kv_heads=heads, head_dim=128, dtype=dtype, tau=tau,
              seeded=seeded)
  return dict(case, name=name) if name else case


def evict(name, kind, batch, seq, heads, head_dim, dtype, budget, recent):
  case = dict(op="evict", kind=kind, batch=batch, seq=seq, heads=heads, head_dim=head_dim, dtype=dtype, budget=budget,
              recent=recent)
  return dict(case, name=name) if name else case


def ops(name, tokens, hidden, heads, kv_heads, head_dim, intermediate, act, dtype):
  case = dict(op="ops", tokens=tokens, hidden=hidden, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
              intermediate=intermediate, act=act, dtype=dtype)
  return dict(case, name=name) if name else case


def decoder_layer(name, batch, seq):
  case = dict(op="layer", batch=batch, seq=seq, dtype="bf16")
  return dict(case, name=name) if name else case


def listed():
  return [
      # one generated token for four sequences against the compact cache that an eviction leaves (budget 512): the
      # smallest call of a generation loop, views of the [B, 2, budget, H, D] cache
      attn("decode_evicted_cache", 4, 1, 512, 32, 32, 128, "fp16", layout="cache"),
      # one generated token for eight sequences with a long un-evicted cache, grouped-query heads
      attn("decode_gqa_8k", 8, 1, 8192, 32, 8, 128, "bf16"),
      # a short prompt: the causal core module at batch 1, 32 heads, 1024 tokens
      attn("prefill_1k", 1, 1024, 1024, 32, 32, 128, "fp16"),
      # the headline workload: causal prefill at batch 4, 32 heads, 4096 tokens
      attn("prefill_4k_b4", 4, 4096, 4096, 32, 32, 128, "bf16"),
      # the next chunk of a prompt whose beginning is in the cache, odd lengths, grouped-query heads
      attn("prefill_chunk_ragged", 2, 777, 3001, 32, 8, 128, "bf16"),
      # Gemma-2-style attention: head_dim 256, sliding window, soft-capped logits, read as views of the QKV projection
      attn("gemma2_8k_window", 1, 8192, 8192, 16, 8, 256, "bf16", window=4096, softcap=50.0, layout="qkv"),
      # accumulated attention score for KV eviction, batch 2, 32 heads, 4096 tokens
      score("h2o_4k_b2", "h2o", 2, 4096, 4096, 32, 32, "bf16"),
      # score and squared score of one prompt of odd length
      score("roco_1501", "roco", 1, 1501, 1501, 32, 32, "fp16"),
      # second softmax over logits with Gumbel noise handed over as a tensor, batch 2, 32 heads, 2048 tokens
      keyformer("keyformer_2k_b2", 2, 2048, 32, "bf16", 1.0, False),
      # selection and gather of 512 keys per head out of 4096
      evict("evict_512_of_4k", "topk", 2, 4096, 32, 128, "bf16", 512, 0),
      # norm, rotary embedding, residual norm and gated activation of one decoding step of eight sequences (Llama-7B)
      ops("layer_ops_decode", 8, 4096, 32, 32, 128, 11008, "silu", "fp16"),
      # a whole Gemma-2-style decoder layer over a prompt of 4096 tokens
      decoder_layer("gemma2_layer_4k", 1, 4096),
  ]


def _log(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw(rng):
  kind = rng.choice(["prefill", "prefill", "chunk", "decode", "decode", "score", "score", "kf", "evict", "ops", "ops", "layer"])
  dtype = rng.choice(["bf16", "fp16"])
  heads = rng.choice([8, 12, 16, 32, 40])
  kv_heads = heads // rng.choice([1, 1, 2, 4])
  if kind in ("prefill", "chunk", "decode"):
    head_dim = rng.choice([128, 128, 128, 256])
    softcap = rng.choice([0.0, 0.0, 50.0])
    if kind == "prefill":
      seq = _log(rng, 64, 8192)
      window = rng.choice([-1, -1, max(16, seq // 3)])
      return attn(None, _log(rng, 1, 8), seq, seq, heads, kv_heads, head_dim, dtype, window, softcap,
                  rng.choice(["dense", "qkv"]))
    if kind == "chunk":
      kv_len = _log(rng, 256, 8192)
      return attn(None, _log(rng, 1, 4), _log(rng, 16, kv_len // 2), kv_len, heads, kv_heads, head_dim, dtype, -1, softcap)
    return attn(None, _log(rng, 1, 16), rng.choice([1, 1, 1, 4]), _log(rng, 128, 16384), heads, kv_heads, head_dim, dtype, -1,
                softcap, rng.choice(["dense", "cache"]))
  if kind == "score":
    op = rng.choice(SCORE_OPS)
    seq = _log(rng, 128, 4096)
    return score(None, op, _log(rng, 1, 4), seq, seq, heads, kv_heads if op in ("h2o", "roco") else heads, dtype)
  if kind == "kf":
    seeded = rng.choice([False, False, True])
    seq = _log(rng, 128, 2048)
    return keyformer(None, _log(rng, 1, 2), seq if seeded else (seq + 3) // 4 * 4, heads, dtype, rng.choice([1.0, 1.5]), seeded)
  if kind == "evict":
    seq = _log(rng, 512, 8192)
    budget = _log(rng, 32, seq // 2)
    which = rng.choice(["topk", "roco"])
    return evict(None, which, _log(rng, 1, 4), seq, heads, 128, dtype, budget, rng.choice([16, 32, 128]) if which == "roco" else 0)
  if kind == "ops":
    hidden, h, hk, d, inter = rng.choice([(4096, 32, 32, 128, 11008), (3584, 16, 8, 256, 14336), (2048, 16, 16, 128, 5504)])
    return ops(None, _log(rng, 1, 8192), hidden, h, hk, d, inter, rng.choice(["silu", "gelu"]),
               rng.choice(["bf16", "fp16", "fp16", "fp32"]))
  return decoder_layer(None, 1, _log(rng, 128, 4096))


def draw(rng):
  """One more case; never more work than the largest listed case of its kind."""
  limit = {}
  for c in listed():
    w, kind = work(c), "score" if c["op"] in SCORE_OPS else c["op"]
    old = limit.get(kind, {"bytes": 0.0, "flops": 0.0})
    limit[kind] = {k: max(old[k], w[k]) for k in w}
  limit["ops"] = {"bytes": 1.3e9, "flops": 1e12}
  limit["evict"] = {"bytes": 4 * limit["evict"]["bytes"], "flops": 1e12}
  while True:
    c = _draw(rng)
    w, most = work(c), limit["score" if c["op"] in SCORE_OPS else c["op"]]
    if all(w[k] <= most[k] for k in w):
      return c


def _generator(seed):
  return torch.Generator(device="cuda").manual_seed(int(seed))


def _qkv(case, g):
  dtype = DTYPES[case["dtype"]]
  B, Sq, Skv, H, Hk, D = (case[k] for k in ("batch", "q_len", "kv_len", "heads", "kv_heads", "head_dim"))

  def randn(*shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32).to(dtype)

  layout = case.get("layout", "dense")
  if layout == "qkv":      # column ranges of the fused projection's output
    qkv = randn(B, Sq, (H + 2 * Hk) * D)
    return (qkv[:, :, :H * D].unflatten(-1, (H, D)), qkv[:, :, H * D:(H + Hk) * D].unflatten(-1, (Hk, D)),
            qkv[:, :, (H + Hk) * D:].unflatten(-1, (Hk, D)))
  if layout == "cache":    # planes of a [B, 2, kv_len, Hk, D] cache
    cache = randn(B, 2, Skv, Hk, D)
    return randn(B, Sq, H, D), cache[:, 0], cache[:, 1]
  return randn(B, Sq, H, D), randn(B, Skv, Hk, D), randn(B, Skv, Hk, D)


def _zoo(name, inputs, outputs, **kw):
  """The compiled handle of a core module, as a program that switched from the reference's dispatch holds it."""
  return compile_module(KERNEL_ZOO[name](**kw), list(inputs), list(inputs.values()), outputs, system="b200")


def prepare(case, seed):
  g, op = _generator(seed), case["op"]
  if op == "attn":
    q, k, v = _qkv(case, g)
    return dict(op=op, q=q, k=k, v=v, window=case["window"], softcap=case["softcap"])
  if op in SCORE_OPS:
    q, k, v = _qkv(case, g)
    state = dict(op=op, q=q, k=k, v=v)
    if case["heads"] == case["kv_heads"] and op != "corm":
      outputs = {"h2o": ["out", "h2o_score"], "roco": ["out", "roco_score", "roco_sq_score"], "snapkv": ["out", "snapkv_score"]}
      state["f"] = _zoo(op, dict(q=q, k=k, v=v), outputs[op], kv_head_num=case["heads"], head_num=case["heads"])
    return state
  if op == "kf":
    q, k, v = _qkv(case, g)
    if case["seeded"]:
      return dict(op=op, q=q, k=k, v=v, tau=case["tau"], seed=int(seed))
    u = torch.rand((case["batch"], case["heads"], case["q_len"], case["kv_len"]), generator=g, device="cuda")
    noise = u.clamp_min_(1e-10).log_().neg_()          # -log(noise) is Gumbel(0, 1)
    f = _zoo("kf", dict(q=q, k=k, v=v, exp_rand=noise), ["out", "kf_score"], tau=case["tau"], kv_head_num=case["heads"],
             head_num=case["heads"])
    return dict(op=op, q=q, k=k, v=v, exp_rand=noise, f=f)
  if op == "evict":
    B, S, H, D = case["batch"], case["seq"], case["heads"], case["head_dim"]
    p = torch.randn((B, H, 64, S), generator=g, device="cuda").mul_(2.0).softmax(dim=-1)
    kv = [torch.randn((B, S, H, D), generator=g, device="cuda").to(DTYPES[case["dtype"]]) for _ in range(2)]
    return dict(op=op, kind=case["kind"], score=p.sum(2), score_sq=p.square().sum(2), k=kv[0], v=kv[1], q_len=64,
                budget=case["budget"], recent=case["recent"])
  if op == "ops":
    T, h, D, inter, dtype = case["tokens"], case["hidden"], case["head_dim"], case["intermediate"], DTYPES[case["dtype"]]

    def randn(*shape, scale=1.0, shift=0.0):
      return (torch.randn(shape, generator=g, device="cuda") * scale + shift).to(dtype)

    nq, nk = case["heads"] * D, case["kv_heads"] * D
    return dict(op=op, x=randn(T, h), norm=torch.empty((T, h), dtype=dtype, device="cuda"), w1=randn(h, scale=0.02, shift=1.0),
                w2=randn(h, scale=0.02, shift=1.0), qkv=randn(T, nq + 2 * nk), nq=nq, nk=nk, head_dim=D,
                positions=torch.randint(0, 8192, (T,), generator=g, device="cuda", dtype=torch.int32), attn_out=randn(T, h),
                residual=randn(T, h), gate_up=randn(T, 2 * inter), act=torch.empty((T, inter), dtype=dtype, device="cuda"),
                gate=native_ops.silu_and_mul if case["act"] == "silu" else native_ops.gelu_tanh_and_mul)
  cfg = layer.Gemma2LayerConfig()

  def weight(*shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16) * 0.02

  w = dict(ln1=1 + weight(cfg.hidden), qkv=weight((cfg.heads + 2 * cfg.kv_heads) * cfg.head_dim, cfg.hidden),
           o=weight(cfg.hidden, cfg.heads * cfg.head_dim), ln2=1 + weight(cfg.hidden),
           gate_up=weight(2 * cfg.intermediate, cfg.hidden), down=weight(cfg.hidden, cfg.intermediate))
  x = torch.randn((case["batch"], case["seq"], cfg.hidden), generator=g, device="cuda", dtype=torch.bfloat16)
  return dict(op=op, cfg=cfg, w=w, x=x)


def run(s):
  op = s["op"]
  if op == "attn":
    return attention.attn_fwd(s["q"], s["k"], s["v"], causal=True, window=s["window"], softcap=s["softcap"])
  if op == "corm":
    return attention.attn_corm_fwd(s["q"], s["k"], s["v"])
  if op in SCORE_OPS:
    if "f" in s:
      return s["f"](s["q"], s["k"], s["v"])
    return attention.attn_score_fwd(s["q"], s["k"], s["v"], want_sq=op == "roco")     # grouped-query heads
  if op == "kf":
    if "f" in s:
      return s["f"](s["q"], s["k"], s["v"], s["exp_rand"])
    return attention.attn_kf_fwd(s["q"], s["k"], s["v"], tau=s["tau"], seed=s["seed"])
  if op == "evict":
    if s["kind"] == "topk":
      return attention.kv_evict_topk(s["score"], s["k"], s["v"], s["budget"], return_indices=True)
    return attention.kv_evict_roco(s["score"], s["score_sq"], s["k"], s["v"], s["q_len"], s["budget"], s["recent"],
                                   return_indices=True)
  if op == "ops":
    nq, nk, qkv = s["nq"], s["nk"], s["qkv"]
    native_ops.rms_norm(s["norm"], s["x"], s["w1"], 1e-6)
    native_ops.rotary_embedding_online(s["positions"], qkv[:, :nq], qkv[:, nq:nq + nk], s["head_dim"], 10000.0)
    native_ops.fused_add_rms_norm(s["attn_out"], s["residual"], s["w2"], 1e-6)
    s["gate"](s["act"], s["gate_up"])
    return s["norm"], qkv, s["attn_out"], s["residual"], s["act"]
  return layer.gemma2_layer(s["x"], s["w"], s["cfg"])


def _pairs(q_len, kv_len, window=-1):
  """Visible (query, key) pairs of one head under the causal mask and, if positive, the sliding window."""
  first = kv_len - q_len + 1                           # keys that query 0 sees without a window
  if window <= 0 or window >= kv_len:
    return q_len * (first + kv_len) / 2.0
  short = max(0, min(q_len, window - first))           # queries that see fewer keys than the window
  return short * (2 * first + short - 1) / 2.0 + (q_len - short) * float(window)


def _attention_work(case):
  B, Sq, Skv, H, Hk, D = (case[k] for k in ("batch", "q_len", "kv_len", "heads", "kv_heads", "head_dim"))
  pairs = B * H * _pairs(Sq, Skv, case.get("window", -1))
  return 2.0 * B * D * (2 * Sq * H + 2 * Skv * Hk), 4.0 * pairs * D, pairs


def work(case):
  op = case["op"]
  if op == "attn":
    nbytes, flops, _ = _attention_work(case)
  elif op in SCORE_OPS:
    nbytes, flops, _ = _attention_work(case)
    keys = case["batch"] * case["kv_heads"] * case["kv_len"]
    nbytes += keys * {"h2o": 4, "snapkv": 4, "roco": 8, "corm": 1}[op]
  elif op == "kf":
    nbytes, flops, pairs = _attention_work(case)
    nbytes += 4.0 * case["batch"] * case["heads"] * case["kv_len"] + (0.0 if case["seeded"] else 4.0 * pairs)
  elif op == "evict":
    B, S, H, keep = case["batch"], case["seq"], case["heads"], case["budget"] + case["recent"]
    nbytes = 4.0 * B * H * S * (2 if case["kind"] == "roco" else 1) + 4.0 * B * H * keep
    nbytes += 4.0 * B * H * keep * case["head_dim"] * SIZE[case["dtype"]]
    flops = 0.0
  elif op == "ops":
    T, h, sz = case["tokens"], case["hidden"], SIZE[case["dtype"]]
    rope = 2.0 * (case["heads"] + case["kv_heads"]) * case["head_dim"]
    nbytes = T * sz * (6.0 * h + rope + 3.0 * case["intermediate"]) + 2.0 * h * sz + 4.0 * T
    flops = T * (10.0 * h + 3.0 * rope + 10.0 * case["intermediate"])
  else:
    cfg, T = layer.Gemma2LayerConfig(), case["batch"] * case["seq"]
    weights = cfg.hidden * ((2 * cfg.heads + 2 * cfg.kv_heads) * cfg.head_dim + 3 * cfg.intermediate)
    nbytes = 2.0 * (weights + 2 * T * cfg.hidden)
    flops = 2.0 * T * weights + 4.0 * cfg.head_dim * case["batch"] * cfg.heads * _pairs(case["seq"], case["seq"], cfg.window)
  return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
  """The 16-bit types round the probabilities and the results (2^-9 and 2^-12 relative at most); the fp32 operators are
  sums of a few thousand terms.  The eviction picks and copies."""
  if case["op"] == "evict":
    return "exact"
  rel = {"bf16": 1e-2, "fp16": 2e-3, "fp32": 1e-5}[case["dtype"]]
  return {"rel": rel, "differ": 1e-3} if case["op"] == "corm" else {"rel": rel}
