"""Projection and its gradients of narrow layers (float32 tiles of a warp) where they can go
wrong: lists around a step of pairs and around 32, samples without pairs, channels that leave a
tile part empty, pairs behind the last list, buffers off 16 bytes, several kernel MLPs."""
import pytest
import torch

from tensorflow_graphics_point_clouds_b200 import custom_ops as ops
from tensorflow_graphics_point_clouds_b200 import mcconv

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENGTHS = {"edges": [0, 1, 2, 3, 4, 5, 0, 0, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 100, 0],
           "one sample": [9001], "long and short": [3, 4000, 0, 1, 2500, 8],
           # several samples per warp, the last warp part empty
           "many": [(7 * i) % 41 for i in range(5 * 4736 + 3)]}


def case(c, k, lengths, seed, offset=0, behind=5):
  """offset: floats that features stand beside a 16-byte boundary; behind: pairs of no sample."""
  g = torch.Generator(device=DEV).manual_seed(seed)
  lengths = torch.tensor(lengths, device=DEV)
  n, m = 211, int(lengths.sum())
  owner = torch.repeat_interleave(torch.arange(len(lengths), device=DEV), lengths)
  nbr = torch.randint(0, n, (m + behind,), generator=g, device=DEV)
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  pairs = torch.stack([nbr, torch.cat([owner, owner.new_zeros(behind)])], 1).int()
  feat = r(n * c + offset)[offset:].view(n, c)
  return nbr[:m], owner, pairs, torch.cumsum(lengths, 0).int(), r(m + behind, k), feat, r(len(lengths), c, k)


def close(got, ref, terms):
  """A float32 sum of random terms: each step rounds a partial sum, whose size grows like the
  root of the terms added, by 2^-24 of it at most; summed over the steps that is sqrt(terms / 2)
  times 2^-24 of the result's size."""
  assert (got.double() - ref).norm() <= (1 + terms ** 0.5) * 2.0 ** -24 * ref.norm()


def reference(nbr, owner, basis, feat, up):
  f, b, u = feat.double()[nbr], basis.double(), up.double()[owner]
  out = torch.zeros(up.shape, dtype=torch.float64, device=DEV)
  out.index_add_(0, owner, f[:, :, None] * b[:, None, :])
  df = torch.zeros(feat.shape, dtype=torch.float64, device=DEV)
  df.index_add_(0, nbr, torch.einsum("mck,mk->mc", u, b))
  return out, torch.einsum("mck,mc->mk", u, f), df


@pytest.mark.parametrize("lengths", sorted(LENGTHS))
@pytest.mark.parametrize("k", [8, 16, 32, 64])
@pytest.mark.parametrize("c,offset", [(1, 0), (2, 0), (3, 1), (4, 0), (4, 1), (5, 0), (7, 0), (8, 0),
                                      (8, 1), (16, 0), (24, 0), (24, 1), (40, 0), (64, 0)])
def test_against_64_bits(c, offset, k, lengths):
  if lengths == "many" and c * k > 512:
    pytest.skip("the reference's [pairs, C, K] arrays")
  nbr, owner, pairs, ends, basis, feat, up = case(c, k, LENGTHS[lengths], 97 * c + k, offset)
  # (without scratch no layer goes to the tensor cores)
  out = ops.basis_proj(basis, feat, pairs, ends, scratch=False)
  db, df = ops.basis_proj_grads(basis, feat, pairs, ends, up, scratch=False)
  m, most = len(owner), max(LENGTHS[lengths])
  ref_out, ref_db, ref_df = reference(nbr, owner, basis[:m], feat, up)
  close(out, ref_out, most)
  close(db[:m], ref_db, c)
  assert not db[m:].any()
  close(df, ref_df, k * (m // 211 + 1))


@pytest.mark.parametrize("c,k,groups", [(8, 8, 2), (8, 16, 2), (8, 32, 4), (24, 8, 1), (24, 32, 4),
                                        (2, 64, 2)])
def test_columns_of_several_mlps(c, k, groups):
  """X and dX lie MLP by MLP in the layer: forward and gradients against 64 bits.  (Products of
  bf16 pairs: 3 * 2^-17 a term, see test_projection_edges_gpu.py; two of them in a row.)"""
  cout, co = 16 * groups, 16
  nbr, owner, pairs, ends, basis, feat, _ = case(c, k, LENGTHS["edges"], 5 * c + k, behind=0)
  g = torch.Generator(device=DEV).manual_seed(1)
  w = torch.randn((groups, c * k // groups, co), generator=g, device=DEV)
  up = torch.randn((len(ends), cout), generator=g, device=DEV)
  op = mcconv.ProjectionGemm(k, c, cout, len(ends), w.device)
  out = op.forward(basis, feat, pairs, ends, w, (groups, k, cout))
  db, df, dw = op.backward(basis, feat, pairs, ends, w, up, blocks=(groups, k, cout))
  ref_x, _, _ = reference(nbr, owner, basis, feat, torch.zeros((len(ends), c, k), device=DEV))
  x4 = ref_x.view(-1, c, groups, k // groups)
  w4, u3 = w.double().view(groups, c, k // groups, co), up.double().view(-1, groups, co)
  dx = torch.einsum("sgo,gcho->scgh", u3, w4).reshape(-1, c, k)
  _, ref_db, ref_df = reference(nbr, owner, basis, feat, dx)
  for got, ref in ((out, torch.einsum("scgh,gcho->sgo", x4, w4).reshape(-1, cout)),
                   (dw, torch.einsum("scgh,sgo->gcho", x4, u3).reshape(w.shape)),
                   (db, ref_db), (df, ref_df)):
    assert (got.double() - ref).norm() <= 6 * 2.0 ** -17 * ref.norm()


@pytest.mark.parametrize("c,k", [(1, 8), (1, 64), (3, 16), (8, 8), (8, 32), (7, 64), (24, 8), (40, 16)])
@pytest.mark.parametrize("ns", [3, 6, 300, 10000])
def test_ranges_that_step_back(c, k, ns):
  """A range that ends before it begins is an empty list; what lies in several samples' ranges
  belongs to each of them (and its basis gradient to any)."""
  g = torch.Generator(device=DEV).manual_seed(ns)
  steps = torch.randint(-9, 13, (ns,), generator=g, device=DEV)
  steps[0], steps[-1] = 10, 40
  ends = torch.cumsum(steps, 0).clamp(min=1)
  ends[1], ends[-1] = 4, ends.max() + 3
  begins = torch.cat([ends.new_zeros(1), ends[:-1]])
  lengths = (ends - begins).clamp(min=0)
  owner = torch.repeat_interleave(torch.arange(ns, device=DEV), lengths)
  pair = begins[owner] + torch.arange(len(owner), device=DEV) - (torch.cumsum(lengths, 0) - lengths)[owner]
  m, n = int(ends[-1]), 211
  r = lambda *s: torch.randn(s, generator=g, device=DEV)
  nbr = torch.randint(0, n, (m,), generator=g, device=DEV)
  basis, feat, up = r(m, k), r(n, c), r(ns, c, k)
  args = (basis, feat, torch.stack([nbr, nbr], 1).int(), ends.int())
  out = ops.basis_proj(*args)
  db, df = ops.basis_proj_grads(*args, up)
  ref_out, ref_db, ref_df = reference(nbr[pair], owner, basis[pair], feat, up)
  close(out, ref_out, int(lengths.max()))
  close(df, ref_df, k * (len(owner) // n + 1))
  alone = torch.bincount(pair, minlength=m)[pair] == 1
  assert alone.any()
  close(db[pair[alone]], ref_db[alone], c)
