"""A layer's neighborhood hook and a neighborhood's get_pdf are the library's own only where
nobody replaced them: in a subclass, on the class or on the object."""
import types

import pytest

from tensorflow_graphics_point_clouds_b200 import mcconv, pc


@pytest.mark.parametrize("cls,name", [(mcconv.MCConv, "build_neighborhood"),
                                      (mcconv.PointConv, "_neighborhood"),
                                      (mcconv.KPConv, "_neighborhood"),
                                      (pc.Neighborhood, "get_pdf")])
def test_replaced_hooks_are_seen(cls, name, monkeypatch):
  new = lambda c: object.__new__(c)
  mine = lambda self, *args, **kw: None
  assert mcconv._is_own(new(cls), name)
  assert mcconv._is_own(new(type("Same", (cls,), {})), name)
  assert not mcconv._is_own(new(type("Other", (cls,), {name: mine})), name)
  obj = new(cls)
  setattr(obj, name, types.MethodType(mine, obj))
  assert not mcconv._is_own(obj, name)
  home = next(c for c in cls.__mro__ if name in vars(c))
  monkeypatch.setattr(home, name, mine)
  assert not mcconv._is_own(new(cls), name)


def test_a_neighborhood_of_the_users_own_is_not_the_librarys():
  class Mine:
    def get_pdf(self, **kw):
      return None
  assert not mcconv._is_own(Mine(), "get_pdf")
