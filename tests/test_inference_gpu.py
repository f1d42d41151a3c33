"""Decode on the GPU: the kernel path (split-KV decode attention, no host sync) against the CPU reference engine, and the
CUDA-graph replay against eager decoding."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ARGS = ["base_emb_dim=256", "base_num_query_heads=4", "base_num_kv_heads=2", "head_dim=64", "base_mlp_dim=512", "base_num_decoder_layers=3",
        "vocab_size=512", "max_target_length=160", "max_prefill_predict_length=64", "per_device_batch_size=3", "weight_init=normal"]


def _run(cfg, device, steps=12, weights=None):
  from maxtext_b200.inference.maxengine import MaxEngine
  eng = MaxEngine(cfg, device=device)
  eng.load_params(seed=3)
  if weights is not None:              # the initialiser draws from the device's own generator: share one set of weights
    eng.model.store.master.copy_(weights.to(device))
    eng.model.store.sync_compute_from_master()
  state = eng.init_decode_state(3)
  g = torch.Generator().manual_seed(0)
  for s, n in enumerate((5, 17, 40)):
    toks = torch.randint(1, cfg.vocab_size, (n,), generator=g)
    p, _ = eng.prefill(toks, n)
    state = eng.insert(p, state, s)
  out = []
  for _ in range(steps):
    state, res = eng.generate(state)
    out.append(res.data[:, 0].cpu())
  return torch.stack(out), eng


def test_gpu_decode_matches_cpu_reference_and_graph_replay():
  from helpers import tiny_config
  cpu_cfg = tiny_config(extra=ARGS + ["dtype=float32", "hardware=cpu"])
  want, cpu_eng = _run(cpu_cfg, "cpu")
  w = cpu_eng.model.store.master.clone()
  gpu_cfg = tiny_config(extra=ARGS + ["dtype=bfloat16", "hardware=gpu"])
  got, eng = _run(gpu_cfg, "cuda", weights=w)
  # bf16 vs fp32 can flip a near-tie; the first tokens of every slot must agree and most of the rest
  assert torch.equal(got[0], want[0])
  assert (got == want).float().mean() > 0.8
  graph_cfg = tiny_config(extra=ARGS + ["dtype=bfloat16", "hardware=gpu", "cuda_graphs=true"])
  got_g, eng_g = _run(graph_cfg, "cuda", weights=w)
  assert any(v is not False for v in eng_g._graphs.values()), "graph capture fell back to eager"
  assert torch.equal(got_g, got)


def test_sampling_kernel_matches_the_pytorch_definition():
  """Greedy is the arg-max; top-k and nucleus draws stay inside the support PyTorch's masks give; the empirical frequencies of
  many rows with the same logits follow softmax(kept / temperature); the same uniform numbers give the same tokens."""
  import torch
  from maxtext_b200.inference import inference_utils as U
  from maxtext_b200.ops import backend
  E = backend.ext(required=True)
  torch.manual_seed(0)
  big = torch.randn(64, 128256, device="cuda") * 3
  assert torch.equal(U.sampling(big, "greedy"), big.argmax(-1))
  assert torch.equal(U.sampling(big.bfloat16(), "greedy"), big.bfloat16().float().argmax(-1))
  g = torch.Generator(device="cuda").manual_seed(5)
  tk = U.sampling(big, "topk", topk=40, temperature=0.8, generator=g)
  kth = big.topk(40, -1).values[:, -1]
  assert (big.gather(1, tk[:, None])[:, 0] >= kth).all()
  g.manual_seed(5)
  assert torch.equal(tk, U.sampling(big, "topk", topk=40, temperature=0.8, generator=g))          # reproducible under a seed
  keep = torch.isfinite(U._mask_nucleus(big.float(), 0.6))
  g.manual_seed(6)
  nu = U.sampling(big, "nucleus", nucleus_p=0.6, generator=g)
  assert keep.gather(1, nu[:, None]).all()
  keep_c = torch.isfinite(U._mask_nucleus(U._mask_topk(big.float(), 50), 0.9))
  co = U.sampling(big, "composite", topk=50, nucleus_p=0.9, temperature=1.3, generator=g)
  assert keep_c.gather(1, co[:, None]).all()
  # frequencies: 40 000 rows of the same 16 logits
  base = torch.tensor([2.0, 1.5, 1.0, 0.5, 0.0, -0.5, -1.0, -1.5, 3.0, -3.0, 0.2, 0.1, -0.1, 2.5, -2.0, 1.2], device="cuda")
  rows = base[None].expand(40000, 16).contiguous()
  for strategy, kw in (("weighted", dict(temperature=0.7)), ("topk", dict(topk=5, temperature=1.0)), ("nucleus", dict(nucleus_p=0.8)),
                       ("composite", dict(topk=8, nucleus_p=0.9, temperature=1.5))):
    toks = U.sampling(rows, strategy, generator=g, **kw)
    lf = base.float()[None]
    if strategy in ("topk", "composite"):
      lf = U._mask_topk(lf, kw.get("topk", 0))
    if strategy in ("nucleus", "composite"):
      lf = U._mask_nucleus(lf, kw.get("nucleus_p", -1.0))
    want = torch.softmax(lf / kw.get("temperature", 1.0), -1)[0]
    got = torch.bincount(toks, minlength=16).float() / toks.numel()
    assert (got - want).abs().max() < 0.012, (strategy, got, want)
    assert (got[want == 0] == 0).all()


@pytest.mark.parametrize("name", ["llama3-8b", "mistral-7b", "gemma-2b", "gemma2-2b", "gemma3-4b", "qwen3-8b", "qwen2.5-7b", "gpt3-6b", "olmo3-7b",
                                  "llama4-17b-16e", "gpt-oss-20b"])
@pytest.mark.parametrize("head_dim", [16, 20, 128])
def test_one_kernel_for_q_k_v_and_the_cache_matches_the_separate_ones(name, head_dim, monkeypatch):
  """Padded prompts, single tokens and portions behind cached tokens through the layers' fused preparation and through the general path. Both
  round to bf16 between the same products, so each is as far from the fp32 engine as the other up to the spread of single roundings."""
  from helpers import tiny_config
  from maxtext_b200.inference.maxengine import MaxEngine
  from maxtext_b200.layers.blocks import Attention
  more = [f"head_dim={head_dim}", "max_target_length=48", "max_prefill_predict_length=40", "per_device_batch_size=3", "weight_init=normal"]
  g = torch.Generator().manual_seed(1)
  steps = [[torch.randint(1, 256, (n,), generator=g).tolist() for n in ns] for ns in ((9, 14, 3), (1, 1, 1), (1, 1, 1), (5, 2, 7), (1, 1, 1))]
  weights = None

  def logits(dtype, served):
    nonlocal weights
    used = []
    real = Attention.serves
    monkeypatch.setattr(Attention, "serves", lambda self, x, ctx: used.append(served and real(self, x, ctx)) or used[-1])
    eng = MaxEngine(tiny_config(name, extra=more + [f"dtype={dtype}", "hardware=gpu"]), device="cuda")
    eng.load_params(seed=3)
    if weights is None:
      weights = eng.model.store.master.clone()
    eng.model.store.master.copy_(weights)
    eng.model.store.sync_compute_from_master()
    state = eng.init_decode_state(3)
    out = [eng.extend(state, [0, 1, 2], toks).float() for toks in steps]
    monkeypatch.setattr(Attention, "serves", real)
    return torch.stack(out), any(used), state.caches

  want, _, _ = logits("float32", False)
  general, _, kept = logits("bfloat16", False)
  fused, ran, kept2 = logits("bfloat16", True)
  assert ran
  err = lambda a: float((a - want).norm() / want.norm())  # noqa: E731
  assert err(fused) <= 1.5 * err(general) + 2 ** -8, (err(fused), err(general))
  for a, b in zip(kept, kept2):
    for n in ("k", "v"):
      x, y = getattr(a[0], n).float(), getattr(b[0], n).float()
      assert torch.equal(x == 0, y == 0) and float((x - y).norm() / x.norm()) <= 2 ** -5


def test_decode_attention_is_the_same_bits_however_many_ctas_share_an_sm():
  """45 sequences (360 CTAs) run with two tiles per warp in shared memory, 60 (480) with three: every sequence's result depends on its own keys only."""
  from maxtext_b200.ops import backend
  E = backend.ext(required=True)
  g = torch.Generator(device="cuda").manual_seed(0)
  B, H, G, D, L = 60, 16, 8, 128, 200
  k, v = (torch.randn(B, L, G, D, device="cuda", generator=g).bfloat16() for _ in range(2))
  q = torch.randn(B, H, D, device="cuda", generator=g).bfloat16()
  ln = torch.randint(1, L - 1, (B,), device="cuda", generator=g)

  def run(n):
    part, ml = torch.empty(n, H, 1, D, device="cuda"), torch.empty(n, H, 1, 2, device="cuda")
    out = torch.empty(n, H * D, device="cuda", dtype=torch.bfloat16)
    E.cached_decode(q[:n].contiguous(), k, v, torch.arange(n, device="cuda"), ln[:n].contiguous(), 0.1, 0.0, 0, None, None, 1, part, ml, out)
    return out
  few, many = run(45), run(60)
  assert torch.equal(few, many[:45])
  b, n = 7, int(ln[7]) + 1
  s = torch.softmax(torch.einsum("gjd,ngd->gjn", q[b].view(G, 2, D).double(), k[b, :n].double()) * 0.1, -1)
  want = torch.einsum("gjn,ngd->gjd", s, v[b, :n].double()).reshape(-1)
  assert bool(((few[b].double() - want).abs() <= 2 ** -7 * want.abs().max()).all())


@pytest.mark.parametrize("D,rot", [(16, 16), (20, 16), (64, 32), (128, 128), (200, 64), (320, 320)])
@pytest.mark.parametrize("paired", [False, True])
def test_unweighted_norm_of_rotated_heads_rounds_like_the_separate_steps(D, rot, paired):
  """Rotated, rounded, normalised by the rounded row, rounded, then the factor and the temperature on the queries, each rounded. Only the sum of squares runs in
  another order, which moves a factor by an ulp of fp32: fewer than one element in 200 rounds to the other bf16 neighbour."""
  from maxtext_b200.ops import backend
  from maxtext_b200.ops import reference as ref
  E = backend.ext(required=True)
  g = torch.Generator(device="cuda").manual_seed(D)
  B, S, H, G, L = 3, 7, 4, 2, 40
  N, eps, mult, coef, every = B * S, 1e-5, 0.3, 0.1, 8.0
  q, k, v = ((torch.randn(N, n * D, device="cuda", generator=g) * 3).bfloat16() for n in (H, G, G))
  lengths = torch.tensor([5, 0, 20], device="cuda")
  pos = (lengths[:, None] + torch.arange(S, device="cuda")).reshape(-1)
  inv = ref.rope_inv_timescale(rot, 1, 10000).cuda()
  qp = torch.empty(N, H, D, device="cuda", dtype=torch.bfloat16)
  kc, vc = torch.zeros(B, L, G, D, device="cuda", dtype=torch.bfloat16), torch.zeros(B, L, G, D, device="cuda", dtype=torch.bfloat16)
  E.qkv_prep(q, k, v, D, D, pos, inv, rot, eps, qp, None, None, kc, vc, torch.arange(B, device="cuda"), lengths, None, paired=paired, temp_coef=coef,
             temp_every=every, steps=True, q_mult=mult)

  def steps(t, n):
    t = t.view(N, n, D).clone()
    E.rope_inplace(t, pos.to(torch.int32), inv, n, paired, False, rot)
    f = t.float()
    return (f * torch.rsqrt(f.pow(2).mean(-1, keepdim=True) + eps)).bfloat16()
  wk = steps(k, G)
  wq = steps(q, H) * mult
  wq = (wq.float() * (torch.log(torch.floor((pos.float() + 1) / every) + 1) * coef + 1)[:, None, None]).bfloat16()
  gk = torch.cat([kc[b, int(lengths[b]): int(lengths[b]) + S] for b in range(B)])
  for got, want in ((gk, wk), (qp, wq)):
    assert float((got != want).float().mean()) <= 1 / 200
    assert bool(((got.float() - want.float()).abs() <= 2 ** -7 * want.float().abs() + 1e-6).all())
  assert torch.equal(torch.cat([vc[b, int(lengths[b]): int(lengths[b]) + S] for b in range(B)]).reshape(N, -1), v)


@pytest.mark.parametrize("name", ["llama3-8b", "gemma2-2b", "gemma3-4b", "qwen3-8b", "qwen2.5-7b", "olmo3-7b", "llama4-17b-16e", "gpt-oss-20b"])
@pytest.mark.parametrize("head_dim", [16, 20, 128])
def test_cached_keys_of_the_first_layer_are_the_same_whichever_path_wrote_them(name, head_dim, monkeypatch):
  """Both paths read the same projections of the first layer. Where no norm follows, or one per head whose sum both take in the same order (widths in multiples
  of 8), the cached keys are the same bits; elsewhere the sum of squares (or, with biases, the product's) runs in another order, and fewer than one element
  in 200 rounds to the other neighbour. Queries show in the logits."""
  from helpers import tiny_config
  from maxtext_b200.inference.maxengine import MaxEngine
  from maxtext_b200.layers.blocks import Attention
  more = [f"head_dim={head_dim}", "max_target_length=48", "max_prefill_predict_length=40", "per_device_batch_size=3", "weight_init=normal",
          "dtype=bfloat16", "hardware=gpu"]
  g = torch.Generator().manual_seed(2)
  prompts = [torch.randint(1, 256, (n,), generator=g).tolist() for n in (30, 17, 40)]
  real, kept = Attention.serves, []
  for served in (False, True):
    used = []
    monkeypatch.setattr(Attention, "serves", lambda self, x, ctx: used.append(served and real(self, x, ctx)) or used[-1])
    eng = MaxEngine(tiny_config(name, extra=more), device="cuda")
    eng.load_params(seed=3)
    state = eng.init_decode_state(3)
    eng.extend(state, [0, 1, 2], prompts)
    assert any(used) == served
    c = state.caches[0][0]
    kept.append([torch.cat([getattr(c, n)[b, : len(p)] for b, p in enumerate(prompts)]) for n in ("k", "v")])
  (k0, v0), (k1, v1) = kept
  exact = name in ("llama3-8b", "gemma2-2b") or (name in ("gemma3-4b", "qwen3-8b") and head_dim % 8 == 0)
  for a, b in ((k0, k1), (v0, v1)):
    if exact:
      assert torch.equal(a, b)
    assert float((a != b).float().mean()) <= 1 / 200
    assert bool(((a.float() - b.float()).abs() <= 2 ** -7 * a.float().abs() + 2 ** -9 * a.float().abs().max()).all())


def test_soft_cap_behind_normalised_heads_is_exact_for_plain_layers(monkeypatch):
  """The kernel's short form of the cap holds for scores up to 0.3 of it. A plain layer's factor is part of its queries by then, so the width alone bounds nothing:
  with a factor of 4 the scores of 16 normalised lanes reach 64 under a cap of 60."""
  from helpers import tiny_config
  from maxtext_b200.inference.maxengine import MaxEngine
  from maxtext_b200.layers.blocks import Attention
  from maxtext_b200.ops import cached_attention as CA
  from maxtext_b200.ops import functional as F
  cfg = tiny_config("llama4-17b-16e", extra=["head_dim=16", "max_target_length=48", "max_prefill_predict_length=40", "per_device_batch_size=1",
                                             "weight_init=normal", "dtype=bfloat16", "hardware=gpu"])
  eng = MaxEngine(cfg, device="cuda")
  eng.load_params(seed=3)
  attns = [b.attn for layer in eng.model.runs for b in layer.blocks]
  assert any(a.l2_qk_norm for a in attns)
  for a in attns:
    a.soft_cap, a.query_scalar = 60.0, 4.0
  modes, real, serves = [], CA._flash, Attention.serves
  monkeypatch.setattr(CA, "_flash", lambda *a, **kw: modes.append(a[9]) or real(*a, **kw))
  g = torch.Generator().manual_seed(4)
  prompt = torch.randint(1, 256, (30,), generator=g).tolist()
  out = []
  for served in (False, True):
    monkeypatch.setattr(Attention, "serves", lambda self, x, ctx, s=served: s and serves(self, x, ctx))
    out.append(eng.extend(eng.init_decode_state(1), [0], [prompt]).float())
  assert modes and all(m == F.CAP_EXACT for m in modes)
  assert float((out[0] - out[1]).norm() / out[0].norm()) <= 2 ** -5


def test_served_projections_with_biases_keep_their_8_bit_scales(monkeypatch):
  """8-bit products scale a weight by its largest element. Projections with biases are products of their own, each with its scale, whichever path serves them:
  with queries' weights far larger than the keys', one scale for all of them would round the keys' differently."""
  from helpers import tiny_config
  from maxtext_b200.inference.maxengine import MaxEngine
  from maxtext_b200.layers.blocks import Attention
  from maxtext_b200.ops import quantization as Q
  cfg = tiny_config("qwen2.5-7b", extra=["base_emb_dim=128", "base_mlp_dim=256", "head_dim=64", "max_target_length=160", "max_prefill_predict_length=140",
                                         "per_device_batch_size=1", "weight_init=normal", "dtype=bfloat16", "hardware=gpu"])
  eng = MaxEngine(cfg, device="cuda")
  eng.load_params(seed=3)
  for layer in eng.model.runs:
    layer.blocks[0].attn.q.data.mul_(37.0)
  g = torch.Generator().manual_seed(4)
  prompt = torch.randint(1, 256, (128,), generator=g).tolist()
  serves, kept = Attention.serves, []
  Q.set_mode("fp8")
  try:
    for served in (False, True):
      used = []
      monkeypatch.setattr(Attention, "serves", lambda self, x, ctx: used.append(served and serves(self, x, ctx)) or used[-1])
      state = eng.init_decode_state(1)
      eng.extend(state, [0], [prompt])
      assert any(used) == served
      kept.append([getattr(state.caches[0][0], n)[0, :128].clone() for n in ("k", "v")])
  finally:
    Q.set_mode("")
  for a, b in zip(*kept):
    assert torch.equal(a, b)
