"""Timed cases of the framework's main paths: a training step through `TrainEngine.train_step`, a prompt through `MaxEngine.prefill`, one
token for every slot through `MaxEngine.generate`.

Model sizes are those of the catalog (`maxtext_b200/configs/models`) and of the serving benchmark with fewer layers, so that a state is built in about
a second; every layer does the same work. Weights, tokens and cached keys are drawn from the seed alone. `exact` computes the same in 64 bits with
plain torch operations.
"""
from __future__ import annotations

import math
import os

import torch

from maxtext_b200.config import pyconfig
from maxtext_b200.inference.maxengine import MaxEngine
from maxtext_b200.train.engine import TrainEngine

# width, query heads, key / value heads, head width, feed-forward width, vocabulary, tied table, norms on q and k, rotary base
ARCHS = {
    "small": dict(width=512, heads=4, kv_heads=2, head_dim=128, ff=1024, vocab=4096, tied=False, qk_norm=False, theta=10000.0, eps=1e-5),
    "plain_1b": dict(width=2048, heads=16, kv_heads=8, head_dim=128, ff=5504, vocab=65536, tied=False, qk_norm=False, theta=10000.0, eps=1e-5),
    "qk_norm_1.7b": dict(width=2048, heads=16, kv_heads=8, head_dim=128, ff=6144, vocab=151936, tied=True, qk_norm=True, theta=1000000.0, eps=1e-6),
    "plain_8b": dict(width=4096, heads=32, kv_heads=8, head_dim=128, ff=14336, vocab=32000, tied=False, qk_norm=False, theta=500000.0, eps=1e-5),
    "latent_moe_16b": dict(width=2048, heads=16, nope=128, rope=64, v_dim=128, kv_rank=512, ff=10944, experts=64, top=6, expert_ff=1408, shared=2,
                           vocab=102400, tied=False, theta=10000.0, eps=1e-6),
}


def listed():
  return [
      # the smallest step: what a first run, a test or a hyper-parameter sweep of small models does; launches count
      dict(name="train_small", kind="train", arch="small", layers=2, batch=2, seq=512, packed=False, fp8=False),
      # the layers of the headline pre-training job: long rows, two per GPU
      dict(name="train_8b_long", kind="train", arch="plain_8b", layers=2, batch=2, seq=8192, packed=False, fp8=False),
      # fine-tuning on packed documents of odd lengths, rows whose length is no multiple of any tile, norms on q and k, tied table
      dict(name="train_packed", kind="train", arch="qk_norm_1.7b", layers=2, batch=3, seq=1999, packed=True, fp8=False),
      # linear layers on the 8-bit path
      dict(name="train_8b_fp8", kind="train", arch="plain_8b", layers=2, batch=1, seq=4096, packed=False, fp8=True),
      # latent attention, one dense layer and one of 64 routed and two shared experts
      dict(name="train_latent_moe", kind="train", arch="latent_moe_16b", layers=2, batch=1, seq=4096, packed=False, fp8=False),
      # a short chat prompt: time to the first token
      dict(name="prefill_short", kind="prefill", arch="plain_1b", layers=12, prompt=333),
      # a long document
      dict(name="prefill_long", kind="prefill", arch="plain_8b", layers=8, prompt=7777),
      # one user: latency of a token
      dict(name="decode_one", kind="decode", arch="plain_8b", layers=8, slots=1, context=1000),
      # a server in use: slots at unequal lengths
      dict(name="decode_mixed", kind="decode", arch="qk_norm_1.7b", layers=8, slots=45, context=1500),
      # a full server
      dict(name="decode_full", kind="decode", arch="plain_1b", layers=12, slots=128, context=2048),
  ]


def _log_int(rng, lo, hi):
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
  kind = rng.choice(["train", "train", "prefill", "decode", "decode"])
  if kind == "train":
    arch = rng.choice(["small", "plain_1b", "qk_norm_1.7b", "plain_8b", "latent_moe_16b"])
    most = 16384 if arch in ("small", "plain_8b") else 8192
    batch = rng.randint(1, 4)
    seq = min(_log_int(rng, 256, 8192), most // batch)
    if rng.random() < 0.5:
      seq = max(256, seq // 128 * 128)
    return dict(kind=kind, arch=arch, layers=2 if arch != "small" else rng.randint(2, 4), batch=batch, seq=seq, packed=rng.random() < 0.3,
                fp8=arch == "plain_8b" and rng.random() < 0.3)
  arch = rng.choice(["plain_1b", "qk_norm_1.7b", "plain_8b"])
  layers = 12 if arch == "plain_1b" else 8
  if kind == "prefill":
    return dict(kind=kind, arch=arch, layers=layers, prompt=_log_int(rng, 16, 8000))
  return dict(kind=kind, arch=arch, layers=layers, slots=_log_int(rng, 1, 128), context=_log_int(rng, 64, 2048))


# ------------------------------------------------------------------------------------------ inputs
def _generator(seed, part):
  g = torch.Generator(device="cuda")
  g.manual_seed((int(seed) * 1000003 + part) % (2 ** 62))
  return g


def _shapes(case):
  """name -> (shape [out, in], standard deviation; 0: a norm scale around one), in a fixed order."""
  a = ARCHS[case["arch"]]
  D, H, latent = a["width"], a["heads"], "kv_rank" in a
  out = {"token_embedder/embedding": ((a["vocab"], D), 1.0 if latent else 0.02 if a["tied"] else 0.5)}
  for i in range(case["layers"]):
    dense = not latent or i == 0
    p = f"layers_{i}/" if not latent else "dense_layers_0/" if dense else f"moe_layers_{i - 1}/"
    s = p + "self_attention/"
    out[p + "pre_self_attention_layer_norm/scale"] = ((D,), 0)
    if latent:
      out[s + "query/kernel"] = ((H * (a["nope"] + a["rope"]), D), 0.02)
      out[s + "wkv_a/kernel"] = ((a["kv_rank"] + a["rope"], D), 0.02)
      out[s + "kv_norm/scale"] = ((a["kv_rank"],), 0)
      out[s + "wkv_b/kernel"] = ((H * (a["nope"] + a["v_dim"]), a["kv_rank"]), 0.04)
      out[s + "out/kernel"] = ((D, H * a["v_dim"]), 0.02)
    else:
      d, G = a["head_dim"], a["kv_heads"]
      # the factor head_dim ** -0.5 is part of the query weights of models without norms on q and k
      out[s + "query/kernel"] = ((H * d, D), 0.02 * (1.0 if a["qk_norm"] else d ** -0.5))
      out[s + "key/kernel"] = ((G * d, D), 0.02)
      out[s + "value/kernel"] = ((G * d, D), 0.02)
      out[s + "out/kernel"] = ((D, H * d), 0.02)
      if a["qk_norm"]:
        out[s + "query_norm/scale"] = ((d,), 0)
        out[s + "key_norm/scale"] = ((d,), 0)
    out[p + "post_self_attention_layer_norm/scale"] = ((D,), 0)
    if dense:
      m = p + "mlp/"
      ff = a["ff"]
    else:
      m, ff = p + "DeepSeekMoeBlock_0/shared_experts/", a["shared"] * a["expert_ff"]
      r = p + "DeepSeekMoeBlock_0/MoeBlock_0/"
      out[r + "gate/kernel"] = ((a["experts"], D), 0.02)
      out[r + "wi_0"] = ((a["experts"], a["expert_ff"], D), 0.02)
      out[r + "wi_1"] = ((a["experts"], a["expert_ff"], D), 0.02)
      out[r + "wo"] = ((a["experts"], D, a["expert_ff"]), 0.02)
    out[m + "wi_0/kernel"] = ((ff, D), 0.02)
    out[m + "wi_1/kernel"] = ((ff, D), 0.02)
    out[m + "wo/kernel"] = ((D, ff), 0.02)
  out["decoder/decoder_norm/scale"] = ((D,), 0)
  if not a["tied"]:
    out["decoder/logits_dense/kernel"] = ((a["vocab"], D), 0.02)
  return out


def _weights(case, seed):
  """name -> fp32 tensor whose values bf16 holds (a server's weights; a training job's at a restart from them). Routers are peaked, as trained
  ones are: every token id has experts of its own, towards whose router rows its embedding leans."""
  a = ARCHS[case["arch"]]
  out = {}
  for n, (name, (shape, std)) in enumerate(_shapes(case).items()):
    t = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
    t.normal_(0.0, std or 0.1, generator=_generator(seed, n))
    out[name] = t.float() if std else (1.0 + t).to(torch.bfloat16).float()
  if "experts" in a:
    g, emb = _generator(seed, 900), out["token_embedder/embedding"]
    for i in range(1, case["layers"]):
      gate = out[f"moe_layers_{i - 1}/DeepSeekMoeBlock_0/MoeBlock_0/gate/kernel"]
      unit = gate / gate.norm(dim=1, keepdim=True)
      own = torch.rand(a["vocab"], a["experts"], device="cuda", generator=g).topk(a["top"], dim=1).indices
      emb += 6.0 * torch.zeros(a["vocab"], a["experts"], device="cuda").scatter_(1, own, 1.0) @ unit
    out["token_embedder/embedding"] = emb.to(torch.bfloat16).float()
  return out


def _batch(case, seed):
  """Host arrays of one batch: rows of random tokens, or rows of packed documents with lengths of their own and padding at the end."""
  a = ARCHS[case["arch"]]
  g = torch.Generator().manual_seed(int(seed) * 7 + 3)
  B, S = case["batch"], case["seq"]
  tok = torch.randint(1, a["vocab"], (B, S + 1), generator=g, dtype=torch.int32)
  pos = torch.arange(S, dtype=torch.int32)[None].repeat(B, 1)
  seg = torch.ones(B, S, dtype=torch.int32)
  if case["packed"]:
    for b in range(B):
      at, n = 0, 1
      while at < S:
        length = int(torch.randint(max(1, S // 16), max(2, S // 3), (1,), generator=g))
        last = at + length >= S and n > 1
        seg[b, at: at + length] = 0 if last else n
        m = min(S, at + length) - at
        pos[b, at: at + m] = torch.arange(m, dtype=torch.int32)
        at, n = at + length, n + 1
  return dict(inputs=tok[:, :-1].contiguous(), targets=tok[:, 1:].contiguous(), inputs_position=pos, targets_position=pos.clone(),
              inputs_segmentation=seg, targets_segmentation=seg.clone())


def _lengths(case, seed):
  """Tokens that each slot holds already: all equal for one slot or a full server, spread over a factor of eight otherwise."""
  n, c = case["slots"], case["context"]
  if n in (1, 128):
    return torch.full((n,), c, dtype=torch.long, device="cuda")
  return (c // 8 + torch.rand(n, device="cuda", generator=_generator(seed, 950)) * (c - c // 8)).long().clamp_min(1)


def _cached(case, seed, layer, which):
  """What slots hold of one layer: keys (0) or values (1), bf16 [slots, context, key heads, head width]."""
  a = ARCHS[case["arch"]]
  t = torch.empty(case["slots"], case["context"], a["kv_heads"], a["head_dim"], dtype=torch.bfloat16, device="cuda")
  return t.normal_(0.0, 1.0, generator=_generator(seed, 1000 + 2 * layer + which))


def _last_tokens(case, seed):
  return torch.randint(1, ARCHS[case["arch"]]["vocab"], (case["slots"],), device="cuda", generator=_generator(seed, 951))


def _prompt(case, seed):
  return torch.randint(1, ARCHS[case["arch"]]["vocab"], (case["prompt"],), generator=torch.Generator().manual_seed(int(seed) * 7 + 5))


# ------------------------------------------------------------------------------------------ the framework's calls
def _config(case, **more):
  a = ARCHS[case["arch"]]
  keys = dict(base_emb_dim=a["width"], base_num_query_heads=a["heads"], base_num_decoder_layers=case["layers"], base_mlp_dim=a["ff"], vocab_size=a["vocab"],
              logits_via_embedding=a["tied"], normalize_embedding_logits=False, normalization_layer_epsilon=a["eps"], rope_max_timescale=int(a["theta"]),
              enable_dropout=False, mlp_activations=["silu", "linear"])
  if "kv_rank" in a:
    keys.update(decoder_block="deepseek", attention_type="mla", base_num_kv_heads=a["heads"], first_num_dense_layers=1, q_lora_rank=0,
                kv_lora_rank=a["kv_rank"], qk_nope_head_dim=a["nope"], qk_rope_head_dim=a["rope"], v_head_dim=a["v_dim"], rope_type="default",
                num_experts=a["experts"], num_experts_per_tok=a["top"], base_moe_mlp_dim=a["expert_ff"],
                shared_experts=a["shared"], routed_bias=False, routed_scaling_factor=1.0, routed_score_func="softmax")
  else:
    keys.update(decoder_block="qwen3" if a["qk_norm"] else "llama2", base_num_kv_heads=a["kv_heads"], head_dim=a["head_dim"], use_qk_norm=a["qk_norm"])
  keys.update(dtype="bfloat16", hardware="gpu", enable_checkpointing=False, log_config=False, dataset_type="synthetic")
  keys.update(more)
  return pyconfig.initialize(["cases", os.path.join(pyconfig.CONFIG_ROOT, "base.yml")], num_devices=1, **keys)


def _load(store, weights):
  for name, w in weights.items():
    store.load_full(name, w)
  store.sync_compute_from_master()


class _Server(MaxEngine):
  """Keeps the logits that a step samples from."""

  logits = None

  def _sample(self, logits):
    self.logits = logits
    return super()._sample(logits)


def prepare(case, seed):
  dev = torch.device("cuda", torch.cuda.current_device())
  if case["kind"] == "train":
    cfg = _config(case, weight_dtype="float32", max_target_length=case["seq"], per_device_batch_size=float(case["batch"]), remat_policy="full",
                  steps=100000, learning_rate=3e-5, packing_in_synthetic=case["packed"], quantization="fp8" if case["fp8"] else "")
    eng = TrainEngine(cfg, None, dev, init=False)
    _load(eng.store, _weights(case, seed))
    return dict(case=case, engine=eng, batch={k: v.pin_memory() for k, v in _batch(case, seed).items()})
  longest = (case["prompt"] if case["kind"] == "prefill" else case["context"]) + 64
  cfg = _config(case, weight_dtype="bfloat16", max_target_length=longest, max_prefill_predict_length=longest - 1, cuda_graphs=True,
                decode_sampling_strategy="greedy", per_device_batch_size=float(case.get("slots", 1)))
  eng = _Server(cfg, device=dev)
  _load(eng.model.store, _weights(case, seed))
  if case["kind"] == "prefill":
    return dict(case=case, engine=eng, tokens=_prompt(case, seed))
  state = eng.init_decode_state(case["slots"])
  for i, per_layer in enumerate(state.caches):
    for which, name in enumerate(("k", "v")):
      getattr(per_layer[0], name)[:, : case["context"]] = _cached(case, seed, i, which)
  lengths, tokens = _lengths(case, seed), _last_tokens(case, seed)
  state.next_pos.copy_(lengths)
  state.tokens.copy_(tokens)
  state.active.fill_(True)
  eng.generate(state)                                     # a server has stepped before: its step is captured once per state
  return dict(case=case, engine=eng, state=state, lengths=lengths, tokens=tokens)


def run(state):
  eng, kind = state["engine"], state["case"]["kind"]
  if kind == "train":
    metrics = eng.train_step(state["batch"])
    out = dict(loss=metrics["learning/lm_loss"], weights=eng.store.master)
    # gradients through 8-bit operands (a step of 2 ** -4) differ by several percent between any two orders of the sums in front of them
    return out if state["case"]["fp8"] else dict(out, grads={k: p.main_grad for k, p in eng.store.params.items()})
  if kind == "prefill":
    prefix, _ = eng.prefill(state["tokens"], int(state["tokens"].numel()))
    n = prefix.length
    return dict(logits=prefix.logits, chosen=prefix.logits.gather(1, prefix.first_token[:, None]),
                keys=[c[0].k[:, :n] for c in prefix.caches], values=[c[0].v[:, :n] for c in prefix.caches])
  # every pass answers the same request: the slots stand where the requests left them
  s = state["state"]
  s.next_pos.copy_(state["lengths"])
  s.tokens.copy_(state["tokens"])
  s, result = eng.generate(s)
  return dict(logits=eng.logits, chosen=eng.logits.gather(1, result.data[:, :1]), lengths=s.next_pos, keys=[c[0].k for c in s.caches],
              values=[c[0].v for c in s.caches])


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _pairs(case):
  """Pairs of a query and a key that it sees."""
  if case["kind"] == "decode":
    c = case["context"]
    return case["slots"] * (c + 1 if case["slots"] in (1, 128) else (c + c // 8) // 2 + 1)
  if case["kind"] == "prefill":
    return case["prompt"] * (case["prompt"] + 1) // 2
  if not case["packed"]:
    return case["batch"] * case["seq"] * (case["seq"] + 1) // 2
  total = 0
  for row in _batch(case, 1)["inputs_segmentation"]:
    for n in torch.bincount(row[row > 0].long()).tolist():
      total += n * (n + 1) // 2
  return total


def work(case):
  a = ARCHS[case["arch"]]
  L, D, latent = case["layers"], a["width"], "kv_rank" in a
  tokens = {"train": lambda: case["batch"] * case["seq"], "prefill": lambda: case["prompt"], "decode": lambda: case["slots"]}[case["kind"]]()
  stored = sum(math.prod(shape) for shape, _ in _shapes(case).values())
  per_token = 0                                           # weights that one token meets in the layers
  for name, (shape, std) in _shapes(case).items():
    if std and "layers" in name:
      per_token += math.prod(shape) // a["experts"] * a["top"] if len(shape) == 3 else math.prod(shape)
  width = a["heads"] * (a["nope"] + a["rope"] + a["v_dim"] if latent else 2 * a["head_dim"])
  attention = 2 * _pairs(case) * width * L
  if case["kind"] == "train":
    # three products per weight and token (forward, input gradient, weight gradient); five of the size of attention's two in its passes
    head = a["vocab"] * D
    flops = 6 * tokens * (per_token + head) + attention * 7 // 2
    return dict(bytes=stored * (4 + 2 + 3 * 8) + tokens * 20, flops=flops)
  kv = 2 * a["kv_heads"] * a["head_dim"] * 2 * L          # bytes of a token in the cache
  rows = 1 if case["kind"] == "prefill" else tokens
  head = a["vocab"] * D
  read = 2 * (stored - (0 if a["tied"] else head)) + 2 * tokens * D
  cache = tokens * kv + (_pairs(case) * kv if case["kind"] == "decode" else 0)
  return dict(bytes=read + cache + 4 * rows * a["vocab"], flops=2 * tokens * per_token + 2 * rows * head + attention)


def tolerance(case):
  # bf16 between layers: 0.008 - 0.026 against 64 bits, and 0.014 between two orders of the sums in one product of a decode step. Single gradients
  # of router and expert weights, which few tokens reach, differ by up to 0.73 of the root mean square
  return {"rel": 0.03, "max": 0.9}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _norm(x, scale, eps):
  return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * scale


def _rotate(x, pos, theta):
  """x [B, S, heads, width], pos [B, S]: lane i turns together with lane i + width / 2."""
  d = x.shape[-1]
  inv = (1.0 / theta ** (2.0 * torch.arange(d // 2, dtype=torch.float64, device=x.device) / d)).float()
  ang = (pos.float()[:, :, None, None] * inv).double()
  sin, cos = torch.sin(ang), torch.cos(ang)
  a, b = x[..., : d // 2], x[..., d // 2:]
  return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _attend(q, k, v, seg):
  """Causal attention inside segments, one (row, head) at a time: q [B, S, H, d], k, v [B, S, G, d]."""
  from torch.utils.checkpoint import checkpoint

  def head(qh, kh, vh, sg):
    n = qh.shape[0]
    ok = torch.ones(n, n, dtype=torch.bool, device=qh.device).tril_()
    if sg is not None:
      ok &= (sg[:, None] == sg[None]) & (sg[:, None] != 0)
    w = torch.softmax((qh @ kh.T).masked_fill(~ok, -1e300), -1)
    return w.masked_fill(~ok, 0.0) @ vh
  group = q.shape[2] // k.shape[2]
  rows = []
  for b in range(q.shape[0]):
    sg = seg[b] if seg is not None else None
    rows.append(torch.stack([checkpoint(head, q[b, :, h], k[b, :, h // group], v[b, :, h // group], sg, use_reentrant=False)
                             for h in range(q.shape[2])], 1))
  return torch.stack(rows)


def _layer(a, W, i, x, pos, seg, attend):
  """One layer on x [B, S, D]; `attend(i, q, k, v)` is the attention itself."""
  B, S, D = x.shape
  H, latent = a["heads"], "kv_rank" in a
  dense = not latent or i == 0
  p = f"layers_{i}/" if not latent else "dense_layers_0/" if dense else f"moe_layers_{i - 1}/"
  s = p + "self_attention/"
  h = _norm(x, W[p + "pre_self_attention_layer_norm/scale"], a["eps"])
  q = (h @ W[s + "query/kernel"].T).view(B, S, H, -1)
  if latent:
    n, r = a["nope"], a["rope"]
    q = torch.cat([q[..., :n], _rotate(q[..., n:], pos, a["theta"])], -1) * (n + r) ** -0.5
    kva = h @ W[s + "wkv_a/kernel"].T
    kr = _rotate(kva[..., a["kv_rank"]:].view(B, S, 1, r), pos, a["theta"])
    kv = (_norm(kva[..., : a["kv_rank"]], W[s + "kv_norm/scale"], a["eps"]) @ W[s + "wkv_b/kernel"].T).view(B, S, H, -1)
    k, v = torch.cat([kv[..., :n], kr.expand(B, S, H, r)], -1), kv[..., n:]
  else:
    k, v = ((h @ W[s + f"{m}/kernel"].T).view(B, S, a["kv_heads"], -1) for m in ("key", "value"))
    if a["qk_norm"]:
      q, k = _norm(q, W[s + "query_norm/scale"], a["eps"]), _norm(k, W[s + "key_norm/scale"], a["eps"])
    q, k = _rotate(q, pos, a["theta"]), _rotate(k, pos, a["theta"])
    if a["qk_norm"]:
      q = q * a["head_dim"] ** -0.5
  x = x + attend(i, q, k, v).reshape(B, S, -1) @ W[s + "out/kernel"].T
  h = _norm(x, W[p + "post_self_attention_layer_norm/scale"], a["eps"]).view(B * S, D)
  m = p + ("mlp/" if dense else "DeepSeekMoeBlock_0/shared_experts/")
  y = (torch.nn.functional.silu(h @ W[m + "wi_0/kernel"].T) * (h @ W[m + "wi_1/kernel"].T)) @ W[m + "wo/kernel"].T
  if not dense:
    r = p + "DeepSeekMoeBlock_0/MoeBlock_0/"
    prob, chosen = torch.softmax(h @ W[r + "gate/kernel"].T, -1).topk(a["top"], -1)
    parts = []
    for e in range(a["experts"]):
      t, j = torch.where(chosen == e)
      u = h[t]
      z = (torch.nn.functional.silu(u @ W[r + "wi_0"][e].T) * (u @ W[r + "wi_1"][e].T)) @ W[r + "wo"][e].T
      parts.append((t, z * prob[t, j][:, None]))
    y = y.index_add(0, torch.cat([t for t, _ in parts]), torch.cat([z for _, z in parts]))
  return x + y.view(B, S, D)


def exact(case, seed):
  a = ARCHS[case["arch"]]
  W = {k: v.double() for k, v in _weights(case, seed).items()}
  table = W["token_embedder/embedding"]
  head = table if a["tied"] else W["decoder/logits_dense/kernel"]
  if case["kind"] == "train":
    for v in W.values():
      v.requires_grad_(True)
    batch = {k: v.cuda() for k, v in _batch(case, seed).items()}
    seg = batch["inputs_segmentation"] if case["packed"] else None
    x = table[batch["inputs"].long()]
    for i in range(case["layers"]):
      x = _layer(a, W, i, x, batch["inputs_position"], seg, lambda i, q, k, v: _attend(q, k, v, seg))
    x = _norm(x, W["decoder/decoder_norm/scale"], a["eps"]).view(-1, a["width"])
    target, counts = batch["targets"].view(-1).long(), (batch["targets_segmentation"].view(-1) != 0).double()
    leaf, total = x.detach().requires_grad_(True), 0.0
    for at in range(0, leaf.shape[0], 2048):              # the logits of all rows at once would not fit beside the rest
      part = (torch.nn.functional.cross_entropy(leaf[at: at + 2048] @ head.T, target[at: at + 2048], reduction="none") * counts[at: at + 2048]).sum()
      part.backward()
      total += part.detach()
    x.backward(leaf.grad)
    out = dict(loss=total / counts.sum(), weights=None)
    return out if case["fp8"] else dict(out, grads={k: w.grad for k, w in W.items()})
  with torch.no_grad():
    if case["kind"] == "prefill":
      x, kept = table[_prompt(case, seed).cuda()][None], []
      pos = torch.arange(case["prompt"], device="cuda")[None]

      def attend(i, q, k, v):
        kept.append((k, v))
        return _attend(q, k, v, None)
      for i in range(case["layers"]):
        x = _layer(a, W, i, x, pos, None, attend)
      logits = _norm(x[:, -1], W["decoder/decoder_norm/scale"], a["eps"]) @ head.T
      return dict(logits=logits, chosen=logits.amax(1, keepdim=True), keys=[k for k, _ in kept], values=[v for _, v in kept])
    lengths = _lengths(case, seed)
    x = table[_last_tokens(case, seed)][:, None]

    def attend(i, q, k, v):
      ck, cv = (_cached(case, seed, i, which) for which in (0, 1))
      out = []
      for b in range(case["slots"]):
        n = int(lengths[b])
        kb, vb = torch.cat([ck[b, :n].double(), k[b]]), torch.cat([cv[b, :n].double(), v[b]])
        qb = q[b, 0].view(a["kv_heads"], -1, a["head_dim"])
        w = torch.softmax(torch.einsum("gjd,ngd->gjn", qb, kb), -1)
        out.append(torch.einsum("gjn,ngd->gjd", w, vb).reshape(1, a["heads"], -1))
      return torch.stack(out)
    for i in range(case["layers"]):
      x = _layer(a, W, i, x, lengths[:, None], None, attend)
    logits = _norm(x[:, 0], W["decoder/decoder_norm/scale"], a["eps"]) @ head.T
    return dict(logits=logits, chosen=logits.amax(1, keepdim=True), lengths=None, keys=[], values=[])
