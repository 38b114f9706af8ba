"""Warp-MMA projection and its gradients where they can go wrong: lists around eight and
sixteen pairs, samples without pairs, channels that leave a pass or a 32-channel block part
empty, one list shared by many teams."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import custom_ops as ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENGTHS = {"edges": [0, 1, 7, 8, 9, 0, 0, 15, 16, 17, 24, 25, 31, 32, 33, 48, 49, 100, 0],
           "one long list": [9001], "long and short": [3, 4000, 0, 1, 2500, 8]}


def case(c, k, lengths, seed):
  g = torch.Generator(device=DEV).manual_seed(seed)
  n, m = 211, sum(lengths)
  ends = torch.cumsum(torch.tensor(lengths, device=DEV), 0).int()
  owner = torch.repeat_interleave(torch.arange(len(lengths), device=DEV),
                                  torch.tensor(lengths, device=DEV))
  nbr = torch.randint(0, n, (m,), generator=g, device=DEV)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  return (nbr, owner, torch.stack([nbr, owner], 1).int(), ends, r(m, k), r(n, c),
          r(len(lengths), c, k))


def bound(terms):
  """A product in split bf16 is off by at most 3 * 2^-17 of its size (the middle terms'
  product and what each split leaves over).  For random signed terms the norm of a sum's error
  grows like the norm of the sum, so that this holds for sums of any length.  An MMA adds 16
  products to a float32 accumulator and cuts the sum off, 2^-24 of it on average: three
  passes over `terms` of them, one way."""
  return 3 * 2.0 ** -17 + 3 * (terms / 16 + 1) * 2.0 ** -24


def close(got, ref, terms):
  assert (got.double() - ref).norm() <= bound(terms) * ref.norm()


@pytest.mark.parametrize("lengths", sorted(LENGTHS))
@pytest.mark.parametrize("c,k", [(16, 16), (32, 16), (48, 16), (80, 16), (128, 16), (16, 32),
                                 (48, 32), (64, 32), (96, 32), (16, 64), (32, 64), (48, 64)])
def test_against_64_bits(c, k, lengths):
  nbr, owner, pairs, ends, basis, feat, up = case(c, k, LENGTHS[lengths], c + k)
  out = ops.basis_proj(basis, feat, pairs, ends)
  db, df = ops.basis_proj_grads(basis, feat, pairs, ends, up)
  f, b, u = feat.double()[nbr], basis.double(), up.double()[owner]
  ref = torch.zeros(up.shape, dtype=torch.float64, device=DEV)
  ref.index_add_(0, owner, f[:, :, None] * b[:, None, :])
  close(out, ref, max(LENGTHS[lengths]))
  close(db, torch.einsum("mck,mc->mk", u, f), c)
  ref = torch.zeros(feat.shape, dtype=torch.float64, device=DEV)
  ref.index_add_(0, nbr, torch.einsum("mck,mk->mc", u, b))
  close(df, ref, k)
