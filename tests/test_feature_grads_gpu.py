"""Projection gradients without those of the basis (rigid kernel points): the same feature and
weight gradients as with them, on every kernel that leaves them out and where none does."""
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
def test_same_as_with_the_basis(c, k, k_src, offset, lengths):
  g = torch.Generator(device=DEV).manual_seed(c + k)
  n, ns, m, cout = 211, len(lengths), sum(lengths), 24
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  ends = torch.cumsum(torch.tensor(lengths, device=DEV), 0).int()
  pairs = torch.stack([torch.randint(0, n, (m,), generator=g, device=DEV),
                       torch.repeat_interleave(torch.arange(ns, device=DEV),
                                               torch.tensor(lengths, dtype=torch.long, device=DEV))],
                      1).int()
  basis, feat, w, up = r(m, k), r(n * c + offset)[offset:].view(n, c), r(c * k_src, cout), r(ns, cout)
  args = (basis, feat, pairs, ends, w, up)
  op = mcconv.ProjectionGemm(k, c, cout, ns, w.device, n_in=n)
  _, df, dw = op.backward(*args, reuse_forward=False, blocks=(1, k_src, cout))
  _, df2, dw2 = op.backward(*args, reuse_forward=False, blocks=(1, k_src, cout), want_basis=False)
  # two sums of the same products in another order (and, at 128 channels, of operands split at
  # another place: 3 * 2^-17 a term on either side)
  for a, b in ((df, df2), (dw, dw2)):
    assert (a - b).norm() <= 6 * 2.0 ** -17 * a.norm()
