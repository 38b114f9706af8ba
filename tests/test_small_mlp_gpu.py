"""Kernel MLPs of two hidden layers that run in registers: widths below and at the padded
ones, several MLPs, numbers of pairs around a warp's and a block's share, against 64 bits."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import mcconv

pytestmark = pytest.mark.gpu
DEV = "cuda"


def f64_mlp(diff, pdf, ws, bs, act):
  outs = []
  for g in range(ws[0].shape[0]):
    a = diff
    for w, b in zip(ws, bs):
      x = a @ w[g] + b[g]
      a = torch.nn.functional.elu(x) if act else torch.where(x > 0, x, 0.2 * x)
    outs.append(a)
  return torch.cat(outs, 1) / pdf[:, None]


@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("points", [False, True])
@pytest.mark.parametrize("mlps,h1,h2,m", [(1, 8, 16, 1), (1, 8, 16, 17), (1, 8, 8, 4097),
                                          (2, 6, 8, 65), (1, 5, 13, 301), (1, 1, 1, 64),
                                          (3, 8, 9, 100000), (1, 8, 16, 70001)])
def test_against_64_bits(mlps, h1, h2, m, act, points):
  g = torch.Generator(device=DEV).manual_seed(m)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  n, ns, radius = 97, 41, 0.5
  p_in, p_out = r(n, 3), r(ns, 3)
  pairs = torch.stack([torch.randint(0, n, (m,), generator=g, device=DEV),
                       torch.sort(torch.randint(0, ns, (m,), generator=g, device=DEV)).values], 1).int()
  pdf = 0.5 + torch.rand(m, generator=g, device=DEV)
  ws, bs = [r(mlps, 3, h1), r(mlps, h1, h2)], [r(mlps, 1, h1), r(mlps, 1, h2)]
  up = r(m, mlps * h2)
  got = mcconv.kernel_mlp_basis(p_in, p_out, pairs, pdf, ws, bs, radius, act, 0.2)
  grads = mcconv.kernel_mlp_grads(p_in, p_out, pairs, pdf, ws, bs, radius, up, act, 0.2,
                                  point_grads=points)
  d = lambda t: t.double().requires_grad_(True)
  i64, o64, q64, w64, b64 = d(p_in), d(p_out), d(pdf), [d(w) for w in ws], [d(b) for b in bs]
  ref = f64_mlp((i64[pairs[:, 0].long()] - o64[pairs[:, 1].long()]) / radius, q64, w64, b64, act)
  ref.backward(up.double())
  flat = lambda x: [t for y in x for t in (flat(y) if isinstance(y, (list, tuple)) else [y])]
  want = flat([w64, b64] + ([i64, o64, q64] if points else []))
  # float32 sums of up to 1e5 signed terms, some of which cancel: 1e5^0.5 * 6e-8 of the terms'
  # norm; a pre-activation within rounding of zero takes the other slope of a leaky ReLU,
  # 0.8 of one term in up to 1e5 (4 for the smallest sums here)
  assert (got.double() - ref).norm() <= 1e-6 * ref.norm()
  for a, b in zip(flat(grads), want):
    assert a.shape == b.grad.shape
    assert (a.double() - b.grad).norm() <= 1e-4 * b.grad.norm() + 1e-9


class Activation(torch.autograd.Function):
  """ELU (1) or leaky ReLU (0), slopes from the pre-activations: no number stays none."""

  @staticmethod
  def forward(ctx, x, act):
    ctx.save_for_backward(x)
    ctx.act = act
    return torch.where(x > 0, x, torch.expm1(x) if act else 0.2 * x)

  @staticmethod
  def backward(ctx, up):
    x, = ctx.saved_tensors
    return up * torch.where(x > 0, 1.0, torch.exp(x) if ctx.act else 0.2), None


# rows of the basis around the 32 values up to which the register kernel takes several MLPs
@pytest.mark.parametrize("mlps,h1,h2,m", [(2, 8, 16, 513), (4, 8, 8, 300), (3, 4, 11, 257),
                                          (32, 2, 1, 100), (5, 7, 8, 65), (33, 1, 1, 9)])
def test_several_mlps(mlps, h1, h2, m):
  test_against_64_bits(mlps, h1, h2, m, 1, False)


def kinds(t):
  return torch.stack([t.isnan(), t.isposinf(), t.isneginf()])


# what the padded units and the lanes without a pair must keep to themselves: densities of
# zero, sums that overflow, a point at infinity; in float32, as the kernels work
@pytest.mark.parametrize("act", [0, 1])
@pytest.mark.parametrize("special", ["pdf", "overflow", "point"])
@pytest.mark.parametrize("mlps,h1,h2,m", [(1, 5, 13, 3), (1, 8, 16, 65), (1, 6, 7, 33), (2, 3, 8, 17)])
def test_infinities_stay_where_they_arise(mlps, h1, h2, m, special, act):
  g = torch.Generator(device=DEV).manual_seed(m + act)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  # (back through a weight of 3e38 what is left depends on the order of the sums)
  n, points = 20, mlps == 1 and special != "overflow"
  p_in, p_out, pdf = r(n, 3), r(n, 3), 0.5 + torch.rand(m, generator=g, device=DEV)
  ws, bs = [r(mlps, 3, h1), r(mlps, h1, h2)], [r(mlps, 1, h1), r(mlps, 1, h2)]
  pairs = torch.stack([torch.randint(0, n - 1, (m,), generator=g, device=DEV),
                       torch.sort(torch.randint(0, n, (m,), generator=g, device=DEV)).values], 1).int()
  if special == "pdf":
    pdf[-1] = pdf[m // 2] = 0.0
  elif special == "overflow":
    p_in[:, 0] = 10.0 * torch.sign(r(n))          # (no pair near the limit)
    ws[0][0, 0, 0] = 3e38
  else:
    pairs[-1, 0] = n - 1
    p_in[n - 1, 1] = float("inf")
  up = r(m, mlps * h2)
  leaf = lambda t: t.clone().requires_grad_(True)
  i, o, q, w, b = leaf(p_in), leaf(p_out), leaf(pdf), [leaf(t) for t in ws], [leaf(t) for t in bs]
  diff = (i[pairs[:, 0].long()] - o[pairs[:, 1].long()]) * 2.0
  outs = []
  for k in range(mlps):
    a = diff
    for x, y in zip(w, b):      # (products one by one: no zeros of a blocked product between them)
      a = (a[:, :, None] * x[k][None]).sum(1) + y[k]
      a = Activation.apply(a, act)
    outs.append(a)
  ref = torch.cat(outs, 1) / q[:, None]
  ref.backward(up)
  got = mcconv.kernel_mlp_basis(p_in, p_out, pairs, pdf, ws, bs, 0.5, act, 0.2)
  flat = lambda x: [t for y in x for t in (flat(y) if isinstance(y, (list, tuple)) else [y])]
  grads = flat(mcconv.kernel_mlp_grads(p_in, p_out, pairs, pdf, ws, bs, 0.5, up, act, 0.2,
                                       point_grads=points))
  want = [t.grad for t in flat([w, b] + ([i, o, q] if points else []))]
  assert not ref.isfinite().all() or special != "pdf"
  for x, y in zip([got] + grads, [ref.detach()] + want):
    assert torch.equal(kinds(x), kinds(y))
