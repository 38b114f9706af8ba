"""Ranges of a neighborhood whose counts are scanned in one launch (scan_direct_kernel):
at the edges of its tiles, of its four values per thread and of its range, and for more
samples than points, which take the other kernels."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import pc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n,ns", [(3, 1), (5, 5), (2100, 2047), (2100, 2048), (2100, 2049),
                                  (8195, 8193), (65536, 65536), (65537, 65537), (300, 5001)])
def test_ranges_are_the_sums_of_the_counts(n, ns):
  g = torch.Generator(device=DEV).manual_seed(n + ns)
  radius = 0.04
  pts = torch.rand((n, 2), generator=g, device=DEV)
  cloud = pc.PointCloud(pts, torch.zeros(n, dtype=torch.int32, device=DEV), 1)
  smp = pts if ns == n else torch.rand((ns, 2), generator=g, device=DEV)
  out = cloud if ns == n else pc.PointCloud(smp, torch.zeros(ns, dtype=torch.int32, device=DEV), 1)
  neigh = pc.grid_neighborhood(cloud, radius, out)
  ranges = neigh._samples_neigh_ranges.long()
  owners = neigh._neighbors[:, 1].long()
  # every pair lies in its sample's range, and nothing is missing: the lists are tested
  # against the oracle elsewhere, the counts here against all distances
  counts = torch.diff(ranges, prepend=ranges.new_zeros(1))
  assert torch.equal(torch.bincount(owners, minlength=ns), counts)
  assert int(ranges[-1]) == neigh.num_pairs == owners.shape[0]
  inv = torch.tensor(radius, device=DEV).reciprocal()
  some = torch.arange(0, ns, max(1, ns // 64), device=DEV)
  d2 = (((smp[some][:, None] - pts[None]) * inv) ** 2).sum(-1)
  near = (d2 < 1.0 - 1e-5).sum(1)       # (tests within rounding of the radius may go either way)
  far = (d2 < 1.0 + 1e-5).sum(1)
  assert bool(((counts[some] >= near) & (counts[some] <= far)).all())
