"""Each memory-bound CUDA kernel against the PyTorch definition in ops.reference."""
import pytest
import torch

from maxtext_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def _E():
  from maxtext_b200.ops import backend
  return backend.ext(required=True)


@pytest.mark.parametrize("rows,D", [(64, 4096), (37, 1024), (300, 128), (5, 8192), (129, 264)])
def test_rmsnorm_fwd_bwd(rows, D):
  E = _E()
  x = torch.randn(rows, D, device="cuda").bfloat16()
  scale = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
  y = torch.empty_like(x)
  rstd = torch.empty(rows, device="cuda")
  E.rmsnorm_fwd(x, scale, 1e-5, 0.0, y, rstd)
  yr = ref.rmsnorm(x, scale, 1e-5)
  assert (y.float() - yr.float()).abs().max() <= 2e-2
  dy = torch.randn(rows, D, device="cuda").bfloat16()
  dx = torch.empty_like(x)
  ds = torch.zeros(D, device="cuda")
  E.rmsnorm_bwd(dy, x, scale, rstd, 0.0, dx, ds)
  dxr, dsr = ref.rmsnorm_bwd(dy, x, scale, 1e-5)
  assert (dx.float() - dxr.float()).abs().max() <= 3e-2
  assert (ds - dsr).abs().max() <= 2e-2 * max(1.0, dsr.abs().max().item())


@pytest.mark.parametrize("rows,D", [(1, 8), (7, 128), (31, 512), (4800, 128), (33, 520), (700, 1032), (1300, 4096)])
def test_rmsnorm_scale_gradient_adds_every_row_once(rows, D):
  """Row counts around the blocks of the first pass and the row lanes of the second; the gradient joins what is there already. Any order of an
  fp32 sum of n products is within (n + 4) 2**-24 of the sum of their absolute values (two roundings in each product, one for rstd)."""
  E = _E()
  x, dy = (torch.randn(rows, D, device="cuda").bfloat16() for _ in range(2))
  scale = torch.ones(D, device="cuda").bfloat16()
  y, dx, rstd = torch.empty_like(x), torch.empty_like(x), torch.empty(rows, device="cuda")
  E.rmsnorm_fwd(x, scale, 1e-5, 0.0, y, rstd)
  ds = torch.full((D,), 3.0, device="cuda")
  E.rmsnorm_bwd(dy, x, scale, rstd, 0.0, dx, ds)
  terms = dy.double() * x.double() * rstd.double()[:, None]
  bound = (terms.abs().sum(0) + 3.0) * (rows + 4) * 2.0 ** -24
  assert bool(((ds.double() - 3.0 - terms.sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("rows,D,offset", [(1, 8, 0.0), (5, 512, 1.0), (3, 520, 0.0), (300, 2048, 0.0), (17, 16384, 1.0)])
def test_residual_add_and_norm_in_one_pass(rows, D, offset):
  """The pair (x + a, norm of it) is the same bits as the add and the norm on their own; its gradient is the stream's plus the norm's, rounded once:
  within one bf16 ulp (2**-8) of the sum of the two, which the separate kernels round three times."""
  from maxtext_b200.layers.blocks import Constant
  from maxtext_b200.ops import functional as F
  g = torch.Generator(device="cuda").manual_seed(rows)
  x, a, dx, dy = (torch.randn(rows, D, device="cuda", generator=g).bfloat16() for _ in range(4))

  class Scale(Constant):
    shape, main_grad, grad_written = (D,), None, False

  class Norm:
    kind, eps, scale = "rms", 1e-5, Scale((1 + 0.1 * torch.randn(D, device="cuda", generator=g)).bfloat16())
  Norm.offset = offset

  def plain(s):
    y, rstd = torch.empty_like(s), torch.empty(rows, device="cuda")
    _E().rmsnorm_fwd(s, Norm.scale.data, 1e-5, offset, y, rstd)
    return y, rstd
  for add in (a, None):
    want = x if add is None else x + a
    y, rstd = plain(want)
    with torch.no_grad():
      s, h = F.add_norm(x, add, Norm)
    assert torch.equal(s, want) and torch.equal(h, y)
    xr, ar = x.clone().requires_grad_(True), a.clone().requires_grad_(True)
    s, h = F.add_norm(xr, None if add is None else ar, Norm)
    assert torch.equal(s, want) and torch.equal(h, y)
    torch.autograd.backward([s, h], [dx, dy])
    through = torch.empty_like(x)
    _E().rmsnorm_bwd(dy, want, Norm.scale.data, rstd, offset, through, None)
    exact = through.float() + dx.float()
    assert bool(((xr.grad.float() - exact).abs() <= 2 ** -8 * (exact.abs() + through.float().abs()) + 1e-6).all())
    if add is not None:
      assert torch.equal(ar.grad, xr.grad)
    s, h = F.add_norm(xr, None if add is None else ar, Norm)       # only the stream, or only the norm, is used
    assert torch.equal(torch.autograd.grad(s, xr, dx)[0], dx)
    s, h = F.add_norm(xr, None if add is None else ar, Norm)
    assert torch.equal(torch.autograd.grad(h, xr, dy)[0], through)


@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_roundtrip_and_reference(interleaved):
  E = _E()
  B, S, H, Dh = 2, 96, 6, 128
  x = torch.randn(B, S, H, Dh, device="cuda").bfloat16()
  pos = torch.arange(S, device="cuda", dtype=torch.int32)[None].expand(B, S).contiguous()
  inv = ref.rope_inv_timescale(Dh, 1, 500000).cuda()
  want = ref.apply_rope(x[:, :, :4], pos, inv, interleaved)
  y = x.clone()
  E.rope_inplace(y.view(B * S, H, Dh), pos.reshape(-1), inv, 4, interleaved, False, Dh)
  assert (y[:, :, :4].float() - want.float()).abs().max() <= 3e-2
  assert torch.equal(y[:, :, 4:], x[:, :, 4:])
  E.rope_inplace(y.view(B * S, H, Dh), pos.reshape(-1), inv, 4, interleaved, True, Dh)
  assert (y.float() - x.float()).abs().max() <= 5e-2


@pytest.mark.parametrize("act,code", [("silu", 0), ("gelu", 1)])
def test_gated_act(act, code):
  E = _E()
  torch.manual_seed(0)
  gu = torch.randn(200, 2 * 1408, device="cuda").bfloat16()
  out = torch.empty(200, 1408, device="cuda", dtype=torch.bfloat16)
  E.gated_act_fwd(gu, out, code)
  want = ref.gated_act(gu, act).float()
  assert bool(((out.float() - want).abs() <= 1e-2 + want.abs() / 64).all())          # within two bf16 ulps of the reference
  dy = torch.randn_like(out)
  dgu = torch.empty_like(gu)
  E.gated_act_bwd(dy, gu, dgu, code)
  wantg = ref.gated_act_bwd(dy, gu, act).float()
  assert bool(((dgu.float() - wantg).abs() <= 2e-2 + wantg.abs() / 64).all())


@pytest.mark.parametrize("V", [32000, 128256, 1003 * 8])
def test_xent_fwd_bwd(V):
  E = _E()
  rows = 33
  logits = (3 * torch.randn(rows, V, device="cuda")).bfloat16()
  tg = torch.randint(0, V, (rows,), device="cuda", dtype=torch.int32)
  w = (torch.rand(rows, device="cuda") > 0.2).float()
  want, wz = ref.cross_entropy(logits, tg.long(), 1e-4)
  wd = ref.cross_entropy_dlogits(logits, tg.long(), w, 1e-4)
  loss = torch.empty(rows, device="cuda")
  z = torch.empty(rows, device="cuda")
  work = logits.clone()
  E.xent_fwd_bwd(work, tg, w, 1e-4, loss, z, True)
  assert (loss - want).abs().max() <= 2e-3 * want.abs().max()
  assert (z - wz).abs().max() <= 1e-3 * max(1.0, wz.abs().max().item())
  assert (work.float() - wd).abs().max() <= 1e-2


def test_adamw_and_sumsq():
  E = _E()
  n = 1 << 20
  p = torch.randn(n, device="cuda")
  g = torch.randn(n, device="cuda")
  m = torch.zeros(n, device="cuda")
  v = torch.zeros(n, device="cuda")
  sh = torch.empty(n, device="cuda", dtype=torch.bfloat16)
  pr, mr, vr = p.clone(), m.clone(), v.clone()
  gs = torch.tensor([0.5], device="cuda")
  for step in (1, 2, 3):
    E.adamw(p, g, m, v, sh, 1e-2, 0.9, 0.95, 1e-8, 0.0, 0.1, 1 - 0.9 ** step, 1 - 0.95 ** step, gs)
    ref.adamw_step(pr, g, mr, vr, 1e-2, 0.9, 0.95, 1e-8, 0.0, 0.1, step, 0.5)
  assert (p - pr).abs().max() <= 1e-5
  assert (sh.float() - pr).abs().max() <= 2e-2
  out = torch.zeros(1, device="cuda")
  E.sumsq(g, out)
  assert abs(out.item() - g.double().pow(2).sum().item()) <= 1e-4 * n
  out2 = torch.zeros(1, device="cuda")
  E.sumsq(g, out2)
  assert out.item() == out2.item()   # fixed reduction order


def test_embedding():
  E = _E()
  V, D, T = 1000, 256, 513
  table = torch.randn(V, D, device="cuda").bfloat16()
  tok = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
  out = torch.empty(T, D, device="cuda", dtype=torch.bfloat16)
  E.embedding_fwd(tok, table, out)
  assert torch.equal(out, table[tok.long()])
  dy = torch.randn(T, D, device="cuda").bfloat16()
  dt = torch.zeros(V, D, device="cuda")
  E.embedding_bwd(tok, dy, dt)
  want = torch.zeros(V, D, device="cuda").index_add_(0, tok.long(), dy.float())
  assert (dt - want).abs().max() <= 1e-3


@pytest.mark.gpu
def test_muon_newton_schulz_on_the_repository_gemm():
  """The GPU path runs the iteration in bf16 on this repository's GEMM; it must orthogonalise like the fp32 definition."""
  from maxtext_b200.optimizers.muon import newton_schulz
  torch.manual_seed(0)
  for shape in ((256, 512), (512, 256)):
    x = torch.randn(*shape)
    want = newton_schulz(x, steps=5)
    got = newton_schulz(x.cuda(), steps=5).float().cpu()
    assert (got - want).abs().max() < 0.05 * want.abs().max() + 0.02, (got - want).abs().max()
    sv = torch.linalg.svdvals(got)
    assert float(sv.max()) < 1.3 and float(sv.min()) > 0.4


@pytest.mark.parametrize("rows,F", [(1, 8), (2, 2048), (3, 2056), (131, 4104)])
@pytest.mark.parametrize("code", [0, 1, 2, 3])
def test_gated_act_edges(rows, F, code):
  """Odd row counts and widths around a block's 2048 columns: every element within two bf16 ulps of fp64 (one for the result, one for the exponential
  and the products in fp32 far below it)."""
  E = _E()
  g = torch.Generator(device="cuda").manual_seed(F)
  gu, dy = (torch.randn(rows, n * F, device="cuda", generator=g).bfloat16() for n in (2, 1))
  out, dgu = torch.empty_like(dy), torch.empty_like(gu)
  E.gated_act_fwd(gu, out, code)
  E.gated_act_bwd(dy, gu, dgu, code)
  x = gu.double().requires_grad_(True)
  f = {0: torch.nn.functional.silu, 1: lambda t: torch.nn.functional.gelu(t, approximate="tanh"), 2: torch.relu, 3: lambda t: t}[code]
  want = f(x[:, :F]) * x[:, F:]
  want.backward(dy.double())
  for a, b in ((out, want.detach()), (dgu, x.grad)):
    assert bool(((a.double() - b).abs() <= 2 ** -8 * b.abs() + 1e-5).all())


@pytest.mark.parametrize("heads,n_rot,dh,rot", [(1, 1, 16, 16), (5, 3, 64, 32), (40, 40, 128, 128), (33, 32, 256, 128), (3, 3, 24, 24), (4, 4, 80, 40)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_widths(heads, n_rot, dh, rot, interleaved):
  """Rotated widths that the 16-byte kernel takes and widths that it leaves to the other one; lanes and heads that are not rotated stay the same bits.
  The reference rounds its angles and products in fp32 too: one bf16 ulp of the larger lane of a pair apart at most."""
  E = _E()
  B, S = 2, 37
  x = torch.randn(B, S, heads, dh, device="cuda").bfloat16()
  pos = (torch.arange(S, device="cuda", dtype=torch.int32)[None] * 7 + 1).expand(B, S).contiguous()
  inv = ref.rope_inv_timescale(rot, 1, 10000).cuda()
  for inverse in (False, True):
    y = x.clone()
    E.rope_inplace(y.view(B * S, heads, dh), pos.reshape(-1), inv, n_rot, interleaved, inverse, rot)
    want = ref.apply_rope(x[:, :, :n_rot], pos, inv, interleaved, rot, inverse).float()
    assert bool(((y[:, :, :n_rot].float() - want).abs() <= 2 ** -7 * want.abs() + 2 ** -7).all())
    assert torch.equal(y[:, :, n_rot:], x[:, :, n_rot:]) and torch.equal(y[..., rot:], x[..., rot:])


@pytest.mark.parametrize("V", [8, 100, 8191, 8200, 32003, 151936])
def test_cross_entropy_widths(V):
  """Widths around one and two vectors per thread and with a tail, logits with -inf among them. A chain adds up to 19 vectors of 8 terms (V 151936), 32 chains
  and 32 warps meet after that: 8 + 2 * 19 + 2 * 6 roundings of positive terms and the exponential's two ulps, below 2**-18 of the sum and so of the loss
  absolutely (one vector: below 2**-19). Allowed: 2**-20 times |lse| + |loss| + 1, which is above 12 for the widest rows and above 3 for the narrowest; for
  gradients one bf16 ulp."""
  E = _E()
  g = torch.Generator(device="cuda").manual_seed(V)
  rows, ld = 5, (V + 7) // 8 * 8
  store = (torch.randn(rows, ld, device="cuda", generator=g) * 4).bfloat16()
  store[1, 3: V: 5] = float("-inf")
  tgt = torch.tensor([0, 1, V - 1, V // 2, 7], device="cuda", dtype=torch.int32)
  wt = torch.tensor([1.0, 0.5, 1.0, 0.0, 2.0], device="cuda")
  lg = store[:, :V].double()
  lse = torch.logsumexp(lg, -1)
  want = lse - lg.gather(1, tgt.long()[:, None])[:, 0]
  grad = wt.double()[:, None] * (torch.softmax(lg, -1) - torch.nn.functional.one_hot(tgt.long(), V))
  work = store.clone()
  loss, z = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
  E.xent_fwd_bwd(work[:, :V], tgt, wt, 0.0, loss, z, True)
  assert bool(((loss.double() - want).abs() <= 2 ** -20 * (lse.abs() + want.abs() + 1)).all())
  assert bool(((work[:, :V].double() - grad).abs() <= 2 ** -8 * grad.abs() + 1e-6).all())
  assert torch.equal(work[:, V:], store[:, V:])


@pytest.mark.parametrize("B,S,H,nope,rope,vd", [(1, 1, 1, 8, 16, 8), (2, 37, 16, 128, 64, 128), (3, 5, 3, 24, 32, 40), (1, 70, 2, 16, 8, 16), (2, 9, 4, 12, 16, 20)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_latent_heads(B, S, H, nope, rope, vd, interleaved):
  """The one kernel against the separate steps: the forward pass is the same bits; gradients round once or twice less, and the sum over the heads of
  the shared key part runs in another order: within two bf16 ulps of the largest addend. Widths that are no multiples of 8 take the separate steps."""
  from maxtext_b200.ops import functional as F
  g = torch.Generator(device="cuda").manual_seed(S)
  rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
  rank = 24
  q0, kva0, kv0 = rnd(B, S, H, nope + rope), rnd(B, S, rank + rope), rnd(B, S, H, nope + vd)
  pos = (torch.arange(S, device="cuda")[None] * 3 + torch.arange(B, device="cuda")[:, None])
  inv = ref.rope_inv_timescale(rope, 1, 10000).cuda()
  gr = [rnd(B, S, H, nope + rope), rnd(B, S, H, nope + rope), rnd(B, S, H, vd)]

  def run(one):
    q, kva, kv = (t.clone().requires_grad_(True) for t in (q0, kva0, kv0))
    kr = kva[..., rank:]
    if one:
      out = F.latent_heads(q, kr, kv, pos, inv, nope, 0.07, interleaved)
    else:
      k2 = F.rope(kr.reshape(B, S, 1, rope), pos, inv, interleaved)
      out = (torch.cat([q[..., :nope], F.rope(q[..., nope:], pos, inv, interleaved)], -1) * 0.07,
             torch.cat([kv[..., :nope], k2.expand(B, S, H, rope)], -1), kv[..., nope:])
    torch.autograd.backward(out, gr)
    return out, (q.grad, kva.grad, kv.grad)
  (o1, g1), (o2, g2) = run(True), run(False)
  for a, b in zip(o1, o2):
    assert torch.equal(a, b)
  with torch.no_grad():
    for a, b in zip(F.latent_heads(q0, kva0[..., rank:], kv0, pos, inv, nope, 0.07, interleaved), o2):
      assert torch.equal(a, b)
  for a, b in zip(g1, g2):
    assert bool(((a.float() - b.float()).abs() <= 2 ** -7 * b.float().abs() + 2 ** -7 * H).all())
  assert torch.equal(g1[0], g2[0]) and torch.equal(g1[2], g2[2])


def _fma(a, b, c):
  """a * b + c in fp32, rounded once (the product of two fp32 numbers is exact in fp64)."""
  return (a.double() * b.double() + c.double()).float()


@pytest.mark.parametrize("rows,D", [(1, 8), (4800, 128), (1300, 1032), (2500, 4096), (700, 16384)])
def test_stream_gradient_is_the_norms_own_plus_the_streams(rows, D):
  """The norm's gradient joins the stream's as the two would as kernels of their own: rounded, added, rounded. Blocks have several rows."""
  E = _E()
  x, dy, dres = (torch.randn(rows, D, device="cuda").bfloat16() for _ in range(3))
  scale = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()
  y, alone, joint, rstd = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x), torch.empty(rows, device="cuda")
  E.rmsnorm_fwd(x, scale, 1e-5, 0.0, y, rstd)
  E.rmsnorm_bwd(dy, x, scale, rstd, 0.0, alone, None)
  E.rmsnorm_bwd(dy, x, scale, rstd, 0.0, joint, None, dres)
  assert torch.equal(joint, alone + dres)


def test_norm_gradient_rounds_its_factors_once():
  """dx of rows of eight lanes, step by step in fp32: g = dy * scale and xhat = x * rstd rounded, their dot product a chain of fused steps,
  rstd * (g - xhat * mean) with one rounding inside. dy lies near x, so that the difference cancels and every rounding shows; blocks have many rows."""
  E = _E()
  rows, D = 400_000, 8
  x = torch.randn(rows, D, device="cuda").bfloat16()
  dy = (x.float() + 0.05 * torch.randn(rows, D, device="cuda")).bfloat16()
  scale = torch.ones(D, device="cuda").bfloat16()
  rstd = torch.rsqrt(x.float().pow(2).mean(1) + 1e-5)
  dx = torch.empty_like(x)
  E.rmsnorm_bwd(dy, x, scale, rstd, 0.25, dx, None)
  g, xh = dy.float() * 1.25, x.float() * rstd[:, None]
  dot = torch.zeros(rows, device="cuda")
  for e in range(D):
    dot = _fma(g[:, e], xh[:, e], dot)
  want = rstd[:, None] * _fma(-xh, (dot / D)[:, None].expand_as(xh), g)
  assert torch.equal(dx, want.bfloat16())


@pytest.mark.parametrize("rows,D", [(3, 8), (7, 40), (31, 512), (4736, 128), (6001, 256), (590, 1032), (1300, 1032), (1777, 4096)])
def test_norm_scale_gradient_in_its_order(rows, D):
  """The same bits as the sums in their documented order: every block (row slot) a chain of fused steps over its rows, row r of those partial sums
  to sum r % 4, the last incomplete four to sum 0, and the four in pairs."""
  E = _E()
  x, dy = (torch.randn(rows, D, device="cuda").bfloat16() for _ in range(2))
  rstd = 0.5 + torch.rand(rows, device="cuda")
  dx, ds = torch.empty_like(x), torch.full((D,), 3.0, device="cuda")
  E.rmsnorm_bwd(dy, x, torch.ones(D, device="cuda").bfloat16(), rstd, 0.0, dx, ds)
  per_block = 8 if D <= 512 else 1
  blocks = min(-(-rows // per_block), 4 * torch.cuda.get_device_properties(0).multi_processor_count)
  n = blocks * per_block
  a, xh = dy.float(), x.float() * rstd[:, None]
  part = torch.zeros(n, D, device="cuda")
  for top in range(0, rows, n):
    m = min(n, rows - top)
    part[:m] = _fma(a[top: top + m], xh[top: top + m], part[:m])
  sums = torch.zeros(4, D, device="cuda")
  whole = n // 4 * 4
  for r in range(0, whole, 4):
    sums += part[r: r + 4]
  for r in range(whole, n):
    sums[0] += part[r]
  assert torch.equal(ds, 3.0 + ((sums[0] + sums[1]) + (sums[2] + sums[3])))


@pytest.mark.parametrize("D", [64, 128])
def test_row_sums_of_the_gradient_in_their_order(D):
  """sum_d dout * out, read back through dq: with every probability 1 and no value gradient, dq = -sum * k, and one key is a unit vector. The products are
  powers of two that do not all fit into fp32 together, so another order of the sum gives other bits."""
  E = _E()
  B, S, H = 2, 128, 4
  g = torch.Generator(device="cuda").manual_seed(D)
  dout = torch.exp2(torch.randint(-3, 27, (B, S, H, D), device="cuda", generator=g).float()) * (1 - 2 * torch.randint(0, 2, (B, S, H, D), device="cuda", generator=g))
  out = torch.exp2(torch.randint(-2, 3, (B, S, H, D), device="cuda", generator=g).float())
  # the large products cancel: every pair of lanes t, t + D / 2 holds opposite ones but for a small rest
  dout[..., D // 2:] = -dout[..., : D // 2]
  out[..., D // 2:] = out[..., : D // 2]
  dout[..., ::7] += 2.0
  dout, out = dout.bfloat16(), out.bfloat16()
  q, k, v = torch.zeros(B, S, H, D, device="cuda").bfloat16(), torch.zeros(B, S, H, D, device="cuda").bfloat16(), torch.zeros(B, S, H, D, device="cuda").bfloat16()
  k[:, 0, :, 0] = 1.0
  lse = torch.zeros(B, H, S, device="cuda")
  dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
  E.flash_bwd(dout, q, k, v, out, lse, dq, dk, dv, None, None, None, None, 1.0, 0.0, True, 0, 0, 0)
  p = dout.float() * out.float()                                  # exact
  t = p[..., 0::2] + p[..., 1::2]                                 # a pair of neighbouring lanes: one rounding
  if D == 128:
    t = t[..., :32] + t[..., 32:]
  n = 32
  while n > 1:
    n //= 2
    t = t[..., :n] + t[..., n: 2 * n]
  assert torch.equal(dq[..., 0], (-t[..., 0]).bfloat16())


def _butterfly(v, op):
  """What a warp's exchanges over 16, 8, 4, 2, 1 lanes leave of v [..., 32]."""
  n = 32
  while n > 1:
    n //= 2
    v = op(v[..., :n], v[..., n: 2 * n])
  return v[..., 0]


@pytest.mark.parametrize("V", [8, 100, 8191, 32000, 32003, 102400, 151936])
def test_cross_entropy_in_its_order_and_with_full_exponentials(V):
  """Loss and gradient are the same bits as 1024 chains of eight logits each (chain c: vectors c, c + 1024, ...; the tail on chains 0 to 6), joined warp by
  warp, with fp32's own exponential. Whole vectors of -inf come before, between and behind finite ones."""
  E = _E()
  g = torch.Generator(device="cuda").manual_seed(V)
  rows, ld, nvec = 7, (V + 7) // 8 * 8, V // 8
  store = (torch.randn(rows, ld, device="cuda", generator=g) * 6).bfloat16()
  if nvec > 3:
    store[1, : (nvec // 2) * 8] = float("-inf")                  # the first vectors of every chain
    store[2, 8: 8 * (nvec - 1)] = float("-inf")
    store[3, (nvec - 1) * 8: nvec * 8] = float("-inf")
  tgt = torch.full((rows,), V - 1, device="cuda", dtype=torch.int32)
  store[:, V - 1] = 1.0
  wt = torch.rand(rows, device="cuda", generator=g) + 0.5
  x, inf = store[:, :V].float(), torch.tensor(float("-inf"), device="cuda")
  m, s = torch.full((rows, 1024), float("-inf"), device="cuda"), torch.zeros(rows, 1024, device="cuda")

  def step(f, n):
    """f [rows, n, k]: k more logits of chains 0 .. n - 1."""
    nm = torch.maximum(m[:, :n], f.amax(-1))
    base = torch.where(nm == inf, 0.0, nm)
    acc = torch.zeros_like(nm)
    for e in range(f.shape[-1]):
      acc = acc + torch.exp(f[..., e] - base)
    s[:, :n] = _fma(s[:, :n], torch.exp(m[:, :n] - base), acc)
    m[:, :n] = nm
  for top in range(0, nvec, 1024):
    n = min(1024, nvec - top)
    step(x[:, top * 8: (top + n) * 8].view(rows, n, 8), n)
  if V % 8:
    step(x[:, nvec * 8:, None], V % 8)
  join = lambda m, s: (_butterfly(m, torch.maximum), m, s)  # noqa: E731
  for _ in range(2):                                              # the 32 lanes of every warp, then the 32 warps
    m, s = m.view(rows, -1, 32), s.view(rows, -1, 32)
    top, m, s = join(m, s)
    s = _butterfly(s * torch.where(m == inf, 0.0, torch.exp(m - top[..., None])), torch.add)
    m = top
  lse = (m + torch.log(s)).view(rows)
  loss, z = torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
  work = store.clone()
  E.xent_fwd_bwd(work[:, :V], tgt, wt, 0.0, loss, z, True)
  assert bool(torch.isfinite(loss).all()) and torch.equal(loss, lse - x[:, V - 1])
  p = wt[:, None] * torch.exp(x - lse[:, None])
  assert torch.equal(work[:, : V - 1], p[:, : V - 1].bfloat16())
  last = p[:, V - 1] - wt
  assert bool(((work[:, V - 1].float() - last).abs() <= 2 ** -8 * last.abs()).all())
  assert torch.equal(work[:, V:], store[:, V:])


def test_gated_silu_over_every_gate():
  """Every bf16 gate with up and dy = 1, against fp64. __expf is within 2 + 1.173 |g| ulps (|g| < 90: 108 * 2**-23 < 2**-16), two more roundings and the one
  to bf16. Results down to bf16's smallest normal number are kept; where e^-g overflows (g < -88.73) the quotient is -0, as at -inf / inf a NaN."""
  E = _E()
  gate = torch.arange(65536, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
  gu = torch.cat([gate, torch.ones_like(gate)])[None].contiguous()
  out, dgu = torch.empty(1, 65536, device="cuda", dtype=torch.bfloat16), torch.empty_like(gu)
  E.gated_act_fwd(gu, out, 0)
  E.gated_act_bwd(torch.ones_like(out), gu, dgu, 0)
  g = gate.double()
  sig = torch.sigmoid(g)
  want, grad = g * sig, sig * (1 + g * (1 - sig))
  tiny, rel = 2.0 ** -126, 2.0 ** -8
  ok = torch.isfinite(g) & (g > -88.7)
  for got in (out[0], dgu[0, 65536:]):                            # the activation, and the gradient of `up`
    assert bool(((got.double() - want).abs() <= rel * want.abs() + tiny)[ok].all())
    assert bool((got[(g <= -88.75) & torch.isfinite(g)] == 0).all())
    assert bool(torch.isnan(got[torch.isnan(g) | (g == float("-inf"))]).all()) and bool((got[g == float("inf")] == float("inf")).all())
  # s * (1 + g * (1 - s)) cancels around its zero at g = -1.28: four fp32 roundings of terms below 2 and the exponential's error in both of its uses
  err = (dgu[0, :65536].double() - grad).abs()
  assert bool((err <= rel * grad.abs() + sig * (1 + g.abs()) * 2.0 ** -15 + tiny)[ok].all())


@pytest.mark.parametrize("at", [1, 2, 4])
def test_views_that_start_off_a_16_byte_boundary(at):
  """Contiguous slices of a flat buffer, `at` elements in: the same bits as of tensors that start on a boundary, and nothing around them is written."""
  E = _E()
  around = []

  def off(t):
    flat = torch.full((t.numel() + 16,), 7.0, device="cuda", dtype=t.dtype)
    around.append((flat, t.numel()))
    v = flat[at: at + t.numel()].view(t.shape)
    return v.copy_(t)
  rows, D, F = 37, 264, 520
  x, a, dy, dres = (torch.randn(rows, D, device="cuda").bfloat16() for _ in range(4))
  scale, rstd = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16(), torch.empty(rows, device="cuda")
  gu, dh = torch.randn(rows, 2 * F, device="cuda").bfloat16(), torch.randn(rows, F, device="cuda").bfloat16()
  logits = torch.randn(rows, 104, device="cuda").bfloat16()
  tgt, wt = torch.arange(rows, device="cuda", dtype=torch.int32), torch.rand(rows, device="cuda")
  q, k, v, do = (torch.randn(2, 65, h, 64, device="cuda").bfloat16() for h in (4, 2, 2, 4))

  def run(f):
    new = lambda t: f(torch.zeros_like(t))  # noqa: E731
    y, s, dx = new(x), new(x), new(x)
    E.rmsnorm_fwd(f(x), f(scale), 1e-5, 0.0, y, rstd, f(a), s)
    ds = torch.zeros(D, device="cuda")
    E.rmsnorm_bwd(f(dy), f(x), f(scale), rstd, 0.0, dx, ds, f(dres))
    h, dgu = new(dh), new(gu)
    E.gated_act_fwd(f(gu), h, 0)
    E.gated_act_bwd(f(dh), f(gu), dgu, 0)
    lg, loss, z = f(logits), torch.empty(rows, device="cuda"), torch.empty(rows, device="cuda")
    E.xent_fwd_bwd(lg[:, :99], tgt, wt, 0.0, loss, z, True)
    out, lse = torch.zeros_like(q), torch.empty(2, 4, 65, device="cuda")
    E.flash_fwd(q, k, v, out, lse, None, None, None, None, None, 0.1, 0.0, True, 0, 0, 0)
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    E.flash_bwd(do, q, k, v, f(out), lse, dq, dk, dv, None, None, None, None, 0.1, 0.0, True, 0, 0, 0)
    return [t.clone() for t in (y, s, dx, ds, h, dgu, lg, loss, z, dq, dk, dv)]
  want, got = run(lambda t: t.clone()), run(off)
  for i, (w, g) in enumerate(zip(want, got)):
    assert torch.equal(w, g), i
  for flat, n in around:
    assert bool((flat[:at] == 7).all()) and bool((flat[at + n:] == 7).all())
  # a gradient of latent attention's heads that comes as such a slice
  from maxtext_b200.ops import functional as Fn
  B, S, H, nope, rope, vd = 1, 5, 2, 16, 16, 8
  inv, pos = ref.rope_inv_timescale(rope, 1, 10000).cuda(), torch.arange(S, device="cuda")[None]
  src = [torch.randn(*s, device="cuda").bfloat16() for s in ((B, S, H, nope + rope), (B, S, rope), (B, S, H, nope + vd))]
  up = [torch.randn(B, S, H, n, device="cuda").bfloat16() for n in (nope + rope, nope + rope, vd)]
  grads = []
  for f in (lambda t: t, off):
    leaves = [t.clone().requires_grad_(True) for t in src]
    grads.append(torch.autograd.grad(Fn.latent_heads(*leaves, pos, inv, nope, 0.3), leaves, [f(t) for t in up]))
  for w, g in zip(*grads):
    assert torch.equal(w, g)


@pytest.mark.parametrize("rows,F", [(1, 16), (77, 96), (515, 512), (33, 768), (130, 1408), (9, 1800), (5, 2056), (3, 14336)])
def test_gated_act_block_shapes(rows, F):
  """Widths whose blocks hold one to eight pairs of rows, one or several blocks along a row, ragged last warps and odd row counts: every row the same bits
  as on its own."""
  E = _E()
  gu, dy = (torch.randn(rows, n * F, device="cuda").bfloat16() for n in (2, 1))
  out, dgu = torch.full_like(dy, 7.0), torch.full_like(gu, 7.0)
  E.gated_act_fwd(gu, out, 0)
  E.gated_act_bwd(dy, gu, dgu, 0)
  x, d = gu.double(), dy.double()
  g, u, sig = x[:, :F], x[:, F:], torch.sigmoid(x[:, :F])
  for got, want in ((out, g * sig * u), (dgu[:, F:], d * g * sig), (dgu[:, :F], d * u * sig * (1 + g * (1 - sig)))):
    assert bool(((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5).all())
  for r in {0, rows // 2, rows - 1}:
    o1, d1 = torch.empty_like(dy[:1]), torch.empty_like(gu[:1])
    E.gated_act_fwd(gu[r: r + 1].clone(), o1, 0)
    E.gated_act_bwd(dy[r: r + 1].clone(), gu[r: r + 1].clone(), d1, 0)
    assert torch.equal(o1[0], out[r]) and torch.equal(d1[0], dgu[r])


def test_add_norm_records_one_node_and_keeps_shapes():
  """Streams of any shape and stride: one autograd node between the inputs and both results (views as rows would each add one), gradients in the inputs' shapes."""
  from maxtext_b200.layers.blocks import Constant
  from maxtext_b200.ops import functional as F
  D = 264

  class Scale(Constant):
    shape, main_grad, grad_written = (D,), None, False

  class Norm:
    kind, eps, offset, scale = "rms", 1e-5, 0.0, Scale((1 + 0.1 * torch.randn(D, device="cuda")).bfloat16())
  base, a = (torch.randn(3, 5, D, device="cuda").bfloat16() for _ in range(2))
  up = [torch.randn(3, 5, D, device="cuda").bfloat16() for _ in range(2)]
  want = None
  for x0 in (base, base.transpose(0, 1).contiguous().transpose(0, 1)):        # contiguous, and rows of another order in memory
    for add in (a, None):
      xs, as_ = x0.detach().requires_grad_(True), a.clone().requires_grad_(True)
      s, h = F.add_norm(xs, as_ if add is not None else None, Norm)
      assert s.shape == h.shape == xs.shape
      assert h.grad_fn is s.grad_fn and "AddNorm" in type(h.grad_fn).__name__
      assert all(type(f).__name__ == "AccumulateGrad" for f, _ in h.grad_fn.next_functions if f is not None)
      got = torch.autograd.grad([s, h], [xs] + ([as_] if add is not None else []), up)
      assert all(t.shape == xs.shape for t in got)
      if add is None:
        continue
      want = want or (s.detach(), h.detach(), got[0])
      assert torch.equal(s, want[0]) and torch.equal(h, want[1]) and torch.equal(got[0], want[2]) and torch.equal(got[1], want[2])
      with torch.no_grad():
        s2, h2 = F.add_norm(xs, as_, Norm)
      assert torch.equal(s2, want[0]) and torch.equal(h2, want[1])


@pytest.mark.parametrize("rows,D", [(7000, 128), (7000, 512), (2500, 1032), (2500, 4096), (1500, 8192), (1000, 16384)])
@pytest.mark.parametrize("add", [False, True])
def test_rows_of_one_block_are_the_same_bits_as_on_their_own(rows, D, add):
  """More rows than blocks: a block fetches its next row before it sums the present one and takes its two sum buffers in turn. Forward and backward of
  the first and last rows of a block, of the rows between and of the last ones are the same bits as in a call of few rows, where every block has one."""
  E = _E()
  x, a, dy, dres = (torch.randn(rows, D, device="cuda").bfloat16() for _ in range(4))
  scale = (1 + 0.1 * torch.randn(D, device="cuda")).bfloat16()

  def run(x, a, dy, dres):
    y, s, dx, rstd = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x), torch.empty(x.shape[0], device="cuda")
    E.rmsnorm_fwd(x, scale, 1e-5, 0.0, y, rstd, a if add else None, s if add else None)
    E.rmsnorm_bwd(dy, x, scale, rstd, 0.0, dx, None, dres if add else None)
    return (y, rstd, dx) + ((s,) if add else ())
  whole = run(x, a, dy, dres)
  for lo in list(range(0, rows, 140)) + [rows - 3]:
    cut = slice(lo, min(rows, lo + 140))
    for w, p in zip(whole, run(*(t[cut].clone() for t in (x, a, dy, dres)))):
      assert torch.equal(w[cut], p)
  ref_y = torch.nn.functional.rms_norm((x + a if add else x).double(), (D,), scale.double(), 1e-5)
  assert bool(((whole[0].double() - ref_y).abs() <= 2 ** -7 * ref_y.abs()).all())


def test_gated_act_over_more_rows_than_one_grid_axis():
  """Narrow rows by the million: groups of row pairs beyond 65535 go on along the grid's third axis."""
  E = _E()
  rows, F = 65535 * 2 * 21 * 2 + 77, 96                        # 21 pairs of rows per block: a bit more than two times the axis
  gu = torch.randn(1, 2 * F, device="cuda").bfloat16().expand(rows, -1).contiguous()
  dy = torch.randn(1, F, device="cuda").bfloat16().expand(rows, -1).contiguous()
  out, dgu = torch.full_like(dy, 7.0), torch.full_like(gu, 7.0)
  E.gated_act_fwd(gu, out, 0)
  E.gated_act_bwd(dy, gu, dgu, 0)
  one, done = torch.empty_like(dy[:1]), torch.empty_like(gu[:1])
  E.gated_act_fwd(gu[:1], one, 0)
  E.gated_act_bwd(dy[:1], gu[:1], done, 0)
  assert bool((out == one).all()) and bool((dgu == done).all())
