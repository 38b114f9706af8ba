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
