"""Pooling over lists around the four rows that are loaded at a time, rows in quads of channels
and not."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import mcconv

pytestmark = pytest.mark.gpu
DEV = "cuda"


class Lists:
  def __init__(self, pairs, ends):
    self._original_neigh_ids, self._samples_neigh_ranges = pairs, ends


@pytest.mark.parametrize("c", [1, 4, 7, 64])
def test_short_lists(c):
  g = torch.Generator(device=DEV).manual_seed(c)
  lengths = torch.tensor([3, 0, 1, 2, 4, 5, 7, 8, 9, 0, 12, 13, 100], device=DEV)
  ends, m = torch.cumsum(lengths, 0).int(), int(lengths.sum())
  owner = torch.repeat_interleave(torch.arange(len(lengths), device=DEV), lengths)
  nbr = torch.randint(0, 50, (m,), generator=g, device=DEV)
  feat = torch.randn((50, c), generator=g, device=DEV)
  lists = Lists(torch.stack([nbr, owner], 1).int(), ends)
  top, mean = (mcconv.neighborhood_pool(feat, lists, mode) for mode in ("max", "avg"))
  at = 0
  for s, n in enumerate(lengths.tolist()):
    rows = feat[nbr[at:at + n]]
    at += n
    if n:
      assert torch.equal(top[s], rows.max(0).values)
      # a sum of n float32 values, one after the other
      bound = n * 2.0 ** -24 * rows.abs().double().sum(0) / n + 1e-12
      assert ((mean[s].double() - rows.double().mean(0)).abs() <= 2 * bound).all()
    else:
      assert (mean[s] == 0).all()
