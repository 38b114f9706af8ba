"""Cell averages around the number of points from which a warp works on a cell together: the
float32 sums of a cell's points in their own order, bit for bit."""
import numpy as np
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import pc

pytestmark = pytest.mark.gpu
COUNTS = [1, 63, 64, 65, 66, 95, 96, 97, 128, 129, 2, 700, 64, 65]


@pytest.mark.parametrize("d", [2, 3, 4, 6])
def test_sums_in_order(d):
  rng = np.random.default_rng(d)
  # cell i lies at i along the first axis; the clouds' points come mixed
  cell = rng.permutation(np.repeat(np.arange(len(COUNTS)), COUNTS))
  pts = rng.uniform(0.05, 0.9, (len(cell), d)).astype(np.float32)
  pts[:, 0] += cell
  pts[np.flatnonzero(cell == 0)[0]] = 0.0      # the corner of the box
  neigh = pc.Neighborhood(pc.Grid(pc.PointCloud(torch.from_numpy(pts).cuda(),
                                                torch.zeros(len(pts), dtype=torch.int32).cuda(), 1),
                                  1.0), 1.0)
  got, _ = pc.sample(neigh, "average")
  want = []
  for i in reversed(range(len(COUNTS))):      # (cells in ascending first sorted index)
    total = np.zeros(d, np.float32)
    for p in pts[cell == i]:
      total += p
    want.append(total / np.float32(COUNTS[i]))
  np.testing.assert_array_equal(got._points.cpu().numpy(), np.stack(want))
