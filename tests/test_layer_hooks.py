"""A layer's neighborhood hook and a neighborhood's get_pdf are the library's own only where
nobody replaced them: in a subclass, on the class or on the object."""
import types

import pytest

from tensorflow_graphics_point_clouds_b200 import mcconv, pc


@pytest.mark.parametrize("cls,name,own", [
    (mcconv.MCConv, "build_neighborhood", mcconv._LIBRARY_BUILD_NEIGHBORHOOD),
    (mcconv.PointConv, "_neighborhood", mcconv._LIBRARY_NEIGHBORHOOD),
    (mcconv.KPConv, "_neighborhood", mcconv._LIBRARY_NEIGHBORHOOD),
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
