"""Operand splits and clears in one launch (prepare.cu), through the entries that use
them: row lengths beside the eight values a thread takes, buffers that held something
else, pairs that belong to no sample."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import custom_ops as ops
from tensorflow_graphics_point_clouds_b200 import mcconv

pytestmark = pytest.mark.gpu
DEV = "cuda"


def rel(a, b):
  return ((a.double() - b).norm() / b.norm().clamp(min=1e-30)).item()


# Rows that end inside a thread's eight values, rows that are not 16-byte aligned, a
# single row, and more values than one block of threads takes.
@pytest.mark.parametrize("n,cin,cout", [(1, 1, 1), (5, 3, 7), (257, 12, 130), (1000, 33, 64),
                                        (2049, 64, 256)])
@pytest.mark.parametrize("shift", [0, 1])
def test_linear_of_odd_rows(n, cin, cout, shift):
  g = torch.Generator(device=DEV).manual_seed(n + cin)
  # shift: inputs that start 4 bytes behind a 16-byte boundary
  x = torch.randn(n * cin + shift, generator=g, device=DEV)[shift:].view(n, cin)
  w = torch.randn(cin * cout + shift, generator=g, device=DEV)[shift:].view(cin, cout)
  b = torch.randn((1, cout), generator=g, device=DEV)
  ref = x.double() @ w.double() + b.double()
  # each product is off by at most 3 * 2^-17 of |x||w|; for random signed terms the norm of a
  # sum's error grows like the norm of the sum, so that this bounds the result's too
  assert rel(mcconv.conv1x1(x, w, b), ref) < 3 * 2.0 ** -17


@pytest.mark.parametrize("c,k", [(1, 8), (3, 16), (8, 32), (24, 8), (40, 16), (16, 16), (136, 8)])
@pytest.mark.parametrize("scratch", [False, True])
def test_pairs_of_no_sample_have_no_gradient(c, k, scratch):
  g = torch.Generator(device=DEV).manual_seed(c * k)
  n, ns, m, covered = 37, 21, 150, 131
  ends = torch.sort(torch.randint(0, covered, (ns,), generator=g, device=DEV)).values.int()
  ends[-1] = covered
  nbr = torch.randint(0, n, (m,), generator=g, device=DEV)
  owner = torch.searchsorted(ends, torch.arange(m, device=DEV, dtype=torch.int32), right=True)
  pairs = torch.stack([nbr, owner.clamp(max=ns - 1)], 1).int()
  basis = torch.randn((m, k), generator=g, device=DEV)
  feat = torch.randn((n, c), generator=g, device=DEV)
  up = torch.randn((ns, c, k), generator=g, device=DEV)
  torch.full((4 * m * k,), 7.0, device=DEV)     # (so that fresh buffers hold something)
  db, df = ops.basis_proj_grads(basis, feat, pairs, ends, up, scratch=scratch)
  assert not db[covered:].any()
  own = up.double()[owner[:covered]]
  ref_b = torch.einsum("mck,mc->mk", own, feat.double()[nbr[:covered]])
  ref_f = torch.zeros((n, c), dtype=torch.float64, device=DEV)
  ref_f.index_add_(0, nbr[:covered], torch.einsum("mck,mk->mc", own, basis.double()[:covered]))
  # sums of c, or k times the pairs of a point, products in split bf16 (3 * 2^-17 each)
  assert rel(db[:covered], ref_b) < 1e-4
  assert rel(df, ref_f) < 1e-4
