"""Kernel-point weights by the inverse of sigma in two floats, and by a division where the
inverse's parts could leave the range of floats.  The coordinates are small multiples of 1/64, so
that the squared distances are exact and the linear weights have one right value in float32."""
import ctypes

import numpy as np
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import _lib

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("d,k,num", [(3, 16, 15), (3, 64, 60), (2, 8, 8), (4, 32, 25), (6, 8, 1)])
@pytest.mark.parametrize("sigma", [0.6, 1.0, 3.3333, 7e-13, 1.1e-12, 9e11, 2e12, 1e-30, 1e30])
@pytest.mark.parametrize("interpolation", [0, 1])
def test_weights(d, k, num, sigma, interpolation):
  rng = np.random.default_rng(3)
  n, m = 700, 5003
  points = rng.integers(-80, 81, (n, d)).astype(F32) / 64
  kernel = rng.integers(-64, 65, (num, d)).astype(F32) / 64
  kernel[0] = 0.0
  points[:3, 0] = np.inf, -np.inf, np.nan
  nb = np.stack([rng.integers(0, n, m), rng.integers(0, n, m)], 1).astype(np.int32)
  nb[::5, 1] = nb[::5, 0]
  nb[:4] = [[0, 9], [1, 0], [0, 0], [9, 2]]
  sigma = F32(sigma)
  t = [torch.as_tensor(a).cuda() for a in (points, nb, kernel)]
  out = torch.full((m, k), -7.0, device="cuda")
  rc = _lib.lib().tfgpc_kp_basis(
      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), d, k, num, _lib.c_i64(m),
      _lib.ptr(t[0]), _lib.ptr(t[0]), _lib.ptr(t[1]), _lib.ptr(t[2]), ctypes.c_float(1.0),
      ctypes.c_float(sigma), interpolation, _lib.ptr(out))
  assert rc == 0
  out = out.cpu().numpy()
  assert (out[:, num:] == 0).all()
  with np.errstate(invalid="ignore"):
    diff = points[nb[:, 0]] - points[nb[:, 1]]
  d2 = ((diff[:, None].astype(np.float64) - kernel[None]) ** 2).sum(2)
  dist = np.sqrt(d2.astype(F32))
  with np.errstate(over="ignore"):
    if interpolation == 0:
      assert np.array_equal(out[:, :num], np.fmax(F32(1) - dist / sigma, F32(0)))
    else:
      r = (dist / (sigma / F32(3))).astype(np.float64)
      # rounding r * r moves the exponent by 2^-24 of itself; the exponential is within 2 ulp
      want = np.exp(-np.minimum(r * r, 700.0))
      bound = want * (np.minimum(r * r, 700.0) + 4) * 2.0 ** -24 + 1e-38
      near = np.abs(out[:, :num] - want) <= bound
      assert (near | (np.isnan(want) & np.isnan(out[:, :num]))).all()


@pytest.mark.parametrize("sigma,tie", [(0.03, 0.426666617), (0.48, 0.426666617), (1.92, 0.426666617),
                                       (0.916666687, 0.401041716), (0.6, 0.1), (0.75, 0.1)])
def test_quotients_round_like_a_division(sigma, tie):
  """tie / sigma lies next to the middle of two floats, where the inverse in two floats alone
  rounds the other way.  One coordinate, so that dist is its size: the root of its rounded square."""
  rng = np.random.default_rng(7)
  m, sigma = 100000, F32(sigma)
  points = np.zeros((m, 3), F32)
  points[:, 0] = rng.uniform(0, 1.25 * sigma, m)
  points[0, 0], points[1, 0], points[2, 0] = 0.0, tie, -F32(tie)
  points[3:9, 0] = F32(tie) * F32(2) ** np.arange(-6, 0)
  nb = np.stack([np.arange(m), np.zeros(m)], 1).astype(np.int32)
  t = [torch.as_tensor(a).cuda() for a in (points, nb)]
  kernel, out = torch.zeros((1, 3)).cuda(), torch.empty((m, 8), device="cuda")
  rc = _lib.lib().tfgpc_kp_basis(
      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), 3, 8, 1, _lib.c_i64(m),
      _lib.ptr(t[0]), _lib.ptr(t[0]), _lib.ptr(t[1]), _lib.ptr(kernel), ctypes.c_float(1.0),
      ctypes.c_float(sigma), 0, _lib.ptr(out))
  assert rc == 0
  want = np.fmax(F32(1) - np.abs(points[:, 0]) / sigma, F32(0))
  assert np.array_equal(out.cpu().numpy()[:, 0], want)
