"""Poisson disks settled point by point (levels of up to 65 536 points) against the CPU oracle:
one to several points per eight lanes, chains through a cell, lists and cells that are too full (the
passes do those), points outside the batch, two to five dimensions."""
import numpy as np
import pytest
import torch

from oracle import pylib_ref as pr
from tensorflow_graphics_point_clouds_b200 import pc

pytestmark = pytest.mark.gpu
DEV = "cuda"


# spread 0: uniform; else points of a few clumps of that width
@pytest.mark.parametrize("n,b,d,radius,spread", [
    (1, 1, 3, 0.1, 0), (4, 1, 3, 0.5, 0), (33, 2, 3, 0.3, 0), (3000, 3, 3, 0.08, 0),
    (3000, 1, 3, 0.9, 0),            # few cells of hundreds of points
    (255, 1, 3, 2.0, 0), (257, 1, 3, 2.0, 0),     # one cell, at its limit and above
    (20000, 2, 3, 0.04, 0), (65536, 4, 3, 0.02, 0), (65537, 4, 3, 0.02, 0),
    (9000, 2, 2, 0.02, 0), (4000, 2, 4, 0.15, 0), (2000, 1, 5, 0.3, 0),
    (12000, 2, 3, 0.03, 0.02), (30000, 1, 3, 0.02, 0.1)])
def test_settled_like_the_oracle(n, b, d, radius, spread):
  rng = np.random.default_rng(n + d)
  pts = rng.uniform(0, 1, (n, d)).astype(np.float32)
  if spread:
    pts = (rng.uniform(0, 1, (5, d))[rng.integers(0, 5, n)] +
           spread * rng.standard_normal((n, d))).astype(np.float32)
  ids = np.sort(rng.integers(0, b, n)).astype(np.int32)
  grid = pr.Grid(pts, ids, b, radius)
  _, _, ref = pr.sample(pr.Neighborhood(grid, radius), 0)
  neigh = pc.Neighborhood(pc.Grid(pc.PointCloud(torch.from_numpy(pts).to(DEV),
                                                torch.from_numpy(ids).to(DEV), b), radius), radius)
  for _ in range(3):                # (blocks and lanes meet in another order every time)
    cloud, idx = pc.sample(neigh, "poisson")
    assert np.array_equal(idx.cpu().numpy(), ref)
    assert np.array_equal(cloud._points.cpu().numpy(), pts[ref])


def test_points_outside_the_batch_are_taken():
  rng = np.random.default_rng(3)
  pts = torch.from_numpy(rng.uniform(0, 1, (700, 3)).astype(np.float32)).to(DEV)
  ids = torch.zeros(700, dtype=torch.int32, device=DEV)
  ids[-20:] = 7
  ids[:10] = -1
  neigh = pc.Neighborhood(pc.Grid(pc.PointCloud(pts, ids, 1), 0.2), 0.2)
  _, idx = pc.sample(neigh, "poisson")
  inside = pc.Neighborhood(pc.Grid(pc.PointCloud(pts[10:-20], ids[10:-20], 1), 0.2), 0.2)
  _, ref = pc.sample(inside, "poisson")
  got = set(idx.tolist())
  assert set(range(10)) | set(range(680, 700)) <= got
  assert got - set(range(10)) - set(range(680, 700)) == {i + 10 for i in ref.tolist()}
