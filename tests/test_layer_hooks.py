"""A layer's neighborhood hook and a neighborhood's get_pdf are the library's own only where
nobody replaced them: in a subclass, on the class or on the object."""
import types

import pytest

from tensorflow_graphics_point_clouds_b200 import classifier, mcconv, pc


@pytest.mark.parametrize("cls,name,own", [
    (mcconv.MCConv, "build_neighborhood", mcconv._LIBRARY_BUILD_NEIGHBORHOOD),
    (mcconv.PointConv, "_neighborhood", mcconv._LIBRARY_NEIGHBORHOOD),
    (mcconv.KPConv, "_neighborhood", mcconv._LIBRARY_NEIGHBORHOOD),
    (mcconv.KPConv, "_backward", mcconv._LIBRARY_BACKWARD),
    (mcconv.ProjectionGemm, "backward", mcconv._LIBRARY_OP_BACKWARD),
    (pc.Neighborhood, "get_pdf", mcconv._library_get_pdf())])
def test_replaced_hooks_are_seen(cls, name, own, monkeypatch):
  is_own = lambda c, obj=None: mcconv._is_own(getattr(obj or object.__new__(c), name), own)
  mine = lambda self, *args, **kw: None
  assert is_own(cls)
  assert is_own(type("Same", (cls,), {}))
  assert not is_own(type("Other", (cls,), {name: mine}))
  obj = object.__new__(cls)
  setattr(obj, name, types.MethodType(mine, obj))
  assert not is_own(cls, obj)
  setattr(obj, name, lambda *args, **kw: None)
  assert not is_own(cls, obj)
  home = next(c for c in cls.__mro__ if name in vars(c))
  monkeypatch.setattr(home, name, mine)
  assert not is_own(cls)


def test_a_neighborhood_of_the_users_own_is_not_the_librarys():
  class Mine:
    def get_pdf(self, **kw):
      return None
  assert not mcconv._is_own(Mine().get_pdf, mcconv._library_get_pdf())


@pytest.mark.parametrize("where", ["layer", "op", "class"])
def test_kernel_points_call_replaced_gradients_as_ever(where, monkeypatch):
  """A replaced _backward, an own _op and a wrapped ProjectionGemm.backward know nothing of
  gradients that leave out the basis."""
  def backward(basis, features, neighbors, ranges, weights, out_grads, reuse_forward=True,
               blocks=None):
    assert (basis, features, neighbors, ranges, weights, out_grads) == ("b", "f", "n", "r", "w", "g")
    assert blocks == (1, 15, 24)
    return "db", "df", "dw"

  neigh = types.SimpleNamespace(_original_neigh_ids="n", _samples_neigh_ranges="r")
  layer = object.__new__(mcconv.KPConv)
  layer.k, layer.cout, layer._saved = 15, 24, (neigh, "b", "f", "w")
  layer._op = object.__new__(mcconv.ProjectionGemm)
  if where == "layer":
    layer._backward = lambda out_grads: ("db", "df", "dw")
  elif where == "op":
    layer._op = types.SimpleNamespace(backward=backward)
  else:
    monkeypatch.setattr(mcconv.ProjectionGemm, "backward",
                        lambda self, *args, **kw: backward(*args, **kw))
  assert layer.backward("g") == ("df", "dw")


@pytest.mark.parametrize("replaced", [False, True])
@pytest.mark.parametrize("own_cloud", [False, True])
def test_a_replaced_fill_is_called(own_cloud, replaced, monkeypatch):
  """Every neighborhood's list comes from ops.find_neighbors_fill where somebody replaced it;
  the library's own is spared the permutation as a tensor."""
  asked = []

  class Grid:
    _cells = "cells"

    @property
    def _sorted_indices(self):
      asked.append("permutation")
      return "permutation"

  def fill(count, *rest):
    assert count is neigh._counted and rest == (() if own_cloud else ("permutation",))
    return "list" if own_cloud else ("list", "ids")

  neigh = object.__new__(pc.Neighborhood)
  neigh._nbrs = neigh._orig_ids = None
  neigh._counted, neigh._grid = types.SimpleNamespace(cells="cells"), Grid()
  neigh._equal_samples = own_cloud
  if replaced:
    monkeypatch.setattr(pc.ops, "find_neighbors_fill", fill)
  else:
    monkeypatch.setattr(pc.ops, "_cells_fill", lambda count, with_ids, inv_bw, mode:
                        ("list", "ids") if with_ids else "list")
  assert neigh._neighbors == "list"
  assert own_cloud or neigh._original_neigh_ids == "ids"
  assert bool(asked) == (replaced and not own_cloud)


def bare_classifier(monkeypatch, layers, hierarchy):
  """A classifier of these layers alone: everything around them passes its input on."""
  net = object.__new__(classifier.SmallClassifier)
  net.pool_before_head, net.bn_scale = True, 1.0
  net.radii, net.convs = [0.1 * (i + 1) for i in range(len(layers))], layers
  net.conv1x1, net.dense = [("w", "b")] * len(layers), [("w", "b")]
  net._bn_act = lambda x: x
  monkeypatch.setattr(classifier.pc, "PointCloud", lambda *args: "cloud 0")
  monkeypatch.setattr(classifier.pc, "PointHierarchy", lambda *args: hierarchy)
  for name in ("product_status", "check_product_status"):
    monkeypatch.setattr(mcconv, name, lambda *args: None)
  for name in ("conv1x1", "global_pool"):
    monkeypatch.setattr(mcconv, name, lambda x, *args, **kw: x)
  return net


@pytest.mark.parametrize("where", ["object", "class"])
@pytest.mark.parametrize("grids", [True, False])
def test_a_classifier_calls_replaced_layers_as_ever(grids, where, monkeypatch):
  """A forward of one's own need not know the parameter `neighborhood`, a hierarchy of one's own
  may have clouds alone."""
  seen = []

  def forward(features, point_cloud_in, point_cloud_out, radius, keep_for_backward=True):
    seen.append((point_cloud_in, point_cloud_out, radius, keep_for_backward))
    return features

  layers = [object.__new__(mcconv.MCConv) for _ in range(2)]
  if where == "object":
    for layer in layers:
      layer.forward = forward
  else:
    monkeypatch.setattr(mcconv.MCConv, "forward", lambda self, *args, **kw: forward(*args, **kw))
  hierarchy = types.SimpleNamespace(_point_clouds=["cloud %d" % i for i in range(3)])
  if grids:
    hierarchy._neighborhoods = [types.SimpleNamespace(_grid="grid")] * 2
  features = types.SimpleNamespace(device="cpu")
  net = bare_classifier(monkeypatch, layers, hierarchy)
  assert net.forward("points", "ids", 1, features) is features
  assert seen == [("cloud 0", "cloud 1", 0.1, False), ("cloud 1", "cloud 2", 0.2, False)]
