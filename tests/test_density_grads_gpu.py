"""Gradients that Neighborhood.pdf_point_grads takes: one value per pair, on the points' GPU."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import pc
from tensorflow_graphics_point_clouds_b200._lib import TfgpcError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("samples", ["own", "self", "others"])
def test_gradients_of_another_device_or_shape_are_refused(samples):
  g = torch.Generator(device="cuda").manual_seed(4)
  cloud = pc.PointCloud(torch.rand((300, 3), generator=g, device="cuda"),
                        torch.zeros(300, dtype=torch.int32, device="cuda"), 1)
  other = pc.PointCloud(cloud._points[::2].contiguous(), cloud._batch_ids[::2].contiguous(), 1)
  nb = pc.grid_neighborhood(cloud, 0.2, {"own": cloud, "self": None, "others": other}[samples])
  m = nb.num_pairs
  good = torch.rand(m, generator=g, device="cuda")
  for bad in (good.cpu(), good.cpu().numpy(), good[:, None], good[None], good[:-1], good[0]):
    with pytest.raises((TfgpcError, ValueError, RuntimeError)):
      nb.pdf_point_grads(bad)
  assert nb.pdf_point_grads(good).isfinite().all()
  assert torch.equal(nb.pdf_point_grads(good.double()).isfinite(),
                     torch.ones_like(cloud._points, dtype=torch.bool))
