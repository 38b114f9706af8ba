"""The bound of the projection tests tells a split product from one that lost a term."""
import pytest
import torch

from test_projection_edges_gpu import bound


def split(x):
  hi = x.bfloat16().float()
  return hi.double(), (x - hi).bfloat16().double()


@pytest.mark.parametrize("terms", [1, 30, 9001])
def test_bound(terms):
  g = torch.Generator().manual_seed(terms)
  a, b = (torch.randn((terms, 24), generator=g) for _ in range(2))
  (ah, am), (bh, bm) = split(a), split(b)
  ref = a.double().T @ b.double()
  off = lambda *passes: ((sum(x.T @ y for x, y in passes) - ref).norm() / ref.norm()).item()
  assert off((ah, bh), (ah, bm), (am, bh)) < bound(terms) / 3
  for lost in ([(ah, bh)], [(ah, bh), (ah, bm)], [(ah, bh), (am, bh)], [(ah, bh), (ah, bm), (ah, bh)]):
    assert off(*lost) > 6 * bound(terms)
