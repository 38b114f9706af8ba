"""Projection gradients without those of the basis (rigid kernel points) and with them: feature and
weight gradients against 64 bits, on every kernel that leaves them out and where none does."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import mcconv

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENGTHS = [0, 1, 7, 8, 9, 0, 0, 15, 16, 17, 24, 25, 31, 32, 33, 48, 49, 100, 0]


@pytest.mark.parametrize("lengths", [LENGTHS, [2001], []])
@pytest.mark.parametrize("c,k,k_src,offset", [
    (1, 16, 15, 0), (3, 16, 13, 0), (8, 32, 25, 1), (24, 16, 15, 0), (24, 16, 15, 1), (24, 64, 40, 0),
    (72, 16, 15, 0), (16, 16, 15, 0), (64, 16, 15, 0), (64, 16, 15, 1), (96, 16, 13, 0),
    (128, 16, 15, 0), (32, 32, 25, 0), (80, 32, 25, 0), (48, 64, 33, 0)])
def test_against_64_bits_with_and_without_the_basis(c, k, k_src, offset, lengths):
  g = torch.Generator(device=DEV).manual_seed(c + k)
  n, ns, m, cout = 211, len(lengths), sum(lengths), 24
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  # (whole numbers: dX is exact, and dfeat owes what the projection's gradients do alone)
  whole = lambda *s: torch.randint(-8, 9, s, generator=g, device=DEV).float()
  ends = torch.cumsum(torch.tensor(lengths, device=DEV), 0).int()
  nbr = torch.randint(0, n, (m,), generator=g, device=DEV)
  owner = torch.repeat_interleave(torch.arange(ns, device=DEV),
                                  torch.tensor(lengths, dtype=torch.long, device=DEV))
  pairs = torch.stack([nbr, owner], 1).int()
  basis, feat = r(m, k), r(n * c + offset)[offset:].view(n, c)
  w, up = whole(c * k_src, cout), whole(ns, cout)
  basis[:, k_src:] = 0.0
  args = (basis, feat, pairs, ends, w, up)
  op = mcconv.ProjectionGemm(k, c, cout, ns, w.device, n_in=n)
  _, df, dw = op.backward(*args, reuse_forward=False, blocks=(1, k_src, cout))
  _, df2, dw2 = op.backward(*args, reuse_forward=False, blocks=(1, k_src, cout), want_basis=False)
  b, f = basis.double()[:, :k_src], feat.double()[nbr]
  x = torch.zeros((ns, c, k_src), dtype=torch.float64, device=DEV)
  x.index_add_(0, owner, f[:, :, None] * b[:, None, :])
  dx = (up.double() @ w.double().t()).view(ns, c, k_src)
  ref_df = torch.zeros((n, c), dtype=torch.float64, device=DEV)
  ref_df.index_add_(0, nbr, torch.einsum("mck,mk->mc", dx[owner], b))
  ref_dw = x.reshape(ns, c * k_src).t() @ up.double()
  # float32 kernels: sums of random terms (see close in test_narrow_projection_gpu.py).  Else, and
  # for dw: products of values split at 2^-17, 3 * 2^-17 a term, and two of them in a row.
  single = c % 16 != 0 or offset != 0
  bound = (1 + (k * (m // n + 1)) ** 0.5) * 2.0 ** -24 if single else 3 * 2.0 ** -17
  for got in (df, df2):
    assert (got.double() - ref_df).norm() <= bound * ref_df.norm()
  for got in (dw, dw2):
    assert (got.double() - ref_dw).norm() <= 6 * 2.0 ** -17 * ref_dw.norm()
