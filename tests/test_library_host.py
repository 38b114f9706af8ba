"""Host-side checks that need no GPU: the C-ABI library loads, exports every
symbol that include/tfgpc.h declares, and rejects bad arguments before it
touches the device."""
import ctypes
import os
import re
import subprocess

import pytest

from tensorflow_graphics_point_clouds_b200 import _lib, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
  build.build()
  return _lib.lib()


def declared_symbols():
  text = open(os.path.join(ROOT, "include", "tfgpc.h")).read()
  text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
  return sorted(set(re.findall(r"\b(tfgpc_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(lib):
  names = declared_symbols()
  assert len(names) >= 16
  for name in names:
    assert hasattr(lib, name), name
  assert set(names) == set(_lib.SYMBOLS), "ctypes table and header disagree"


def test_version_and_empty_error(lib):
  assert lib.tfgpc_version() >= 1


def test_no_torch_types_in_header():
  text = open(os.path.join(ROOT, "include", "tfgpc.h")).read()
  assert "torch" not in text and "at::" not in text


@pytest.mark.parametrize("d", [1, 7])
def test_invalid_dimension_is_rejected(lib, d):
  rc = lib.tfgpc_compute_keys(None, d, ctypes.c_int64(4), None, None, ctypes.c_int64(1), None,
                              None, None, None)
  assert rc == 1
  assert b"dimension" in lib.tfgpc_last_error()


def test_invalid_basis_and_features_are_rejected(lib):
  i64 = ctypes.c_int64
  rc = lib.tfgpc_basis_proj(None, 12, 8, i64(1), i64(1), i64(1), None, None, None, None, None)
  assert rc == 1 and b"basis functions" in lib.tfgpc_last_error()
  rc = lib.tfgpc_basis_proj(None, 16, 9, i64(1), i64(1), i64(1), None, None, None, None, None)
  assert rc == 1 and b"input features" in lib.tfgpc_last_error()


def test_workspace_queries_grow_with_size(lib):
  i64 = ctypes.c_int64
  assert lib.tfgpc_find_neighbors_workspace_bytes(i64(10)) > 0
  assert (lib.tfgpc_sampling_workspace_bytes(i64(1 << 20))
          > lib.tfgpc_sampling_workspace_bytes(i64(1 << 10)))


def test_missing_library_fails_loudly(monkeypatch, tmp_path):
  monkeypatch.setattr(_lib, "_lib", None)
  monkeypatch.setattr(_lib, "LIB_PATH", str(tmp_path / "nope.so"))
  with pytest.raises(RuntimeError, match="no\\s+CPU or eager fallback"):
    _lib.lib()


def test_layer_entries_reject_bad_arguments(lib):
  """The entries of the KPConv / PointConv / pooling layers check their scalar
  arguments before any launch."""
  i64, f = ctypes.c_int64, ctypes.c_float
  rc = lib.tfgpc_kp_basis(None, 3, 16, 17, i64(4), None, None, None, None, f(1.0), f(1.0), 0, None)
  assert rc == 1 and b"kernel points" in lib.tfgpc_last_error()
  rc = lib.tfgpc_kp_basis(None, 3, 16, 15, i64(4), None, None, None, None, f(1.0), f(1.0), 2, None)
  assert rc == 1 and b"interpolation" in lib.tfgpc_last_error()
  rc = lib.tfgpc_kp_basis(None, 3, 12, 5, i64(4), None, None, None, None, f(1.0), f(1.0), 0, None)
  assert rc == 1 and b"basis functions" in lib.tfgpc_last_error()
  rc = lib.tfgpc_neighborhood_pool(None, 2, 8, i64(4), i64(4), i64(4), None, None, None, None)
  assert rc == 1 and b"mode" in lib.tfgpc_last_error()
  rc = lib.tfgpc_global_pool(None, 0, 8, i64(4), i64(0), None, None, None, None,
                             ctypes.c_size_t(0))
  assert rc == 1 and b"batch size" in lib.tfgpc_last_error()
  rc = lib.tfgpc_scale_bias_activation(None, i64(4), 8, None, f(1.0), None, 3, f(0.0))
  assert rc == 1 and b"activation" in lib.tfgpc_last_error()
  rc = lib.tfgpc_mcconv_workspace_bytes(16, 128, 256, i64(100), i64(100), 1)
  assert rc > 0
  assert lib.tfgpc_global_pool_workspace_bytes(i64(32)) >= 128


class CellGrid(ctypes.Structure):
  """tfgpc_cell_grid: for calls that are refused before anything is read."""
  _fields_ = [("D", ctypes.c_int), ("max_cells", ctypes.c_int), ("n", ctypes.c_int64),
              ("batch_size", ctypes.c_int64), ("arrays", ctypes.c_void_p * 13)]


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("offset", [1, 2, 6])
def test_sampling_refuses_misaligned_workspaces(lib, mode, offset):
  grid = CellGrid(3, 16, 100, 1, (ctypes.c_void_p * 13)(*[4096] * 13))
  some, i64 = ctypes.c_void_p(4096), ctypes.c_int64(0)
  need = ctypes.c_size_t(lib.tfgpc_cells_sample_workspace_bytes(ctypes.c_int64(100)))
  rc = lib.tfgpc_cells_sample(None, ctypes.byref(grid), mode, some, some, some, some,
                              ctypes.c_void_p(4096 + offset), need, ctypes.byref(i64))
  assert rc == 1 and b"aligned to 4 bytes" in lib.tfgpc_last_error()


@pytest.fixture(scope="module")
def part_end(tmp_path_factory):
  """part_end of csrc/list_parts.h, compiled for the host."""
  folder = tmp_path_factory.mktemp("list_parts")
  src, so = folder / "parts.cpp", folder / "parts.so"
  src.write_text('#include "list_parts.h"\nextern "C" int part_end(int b, int e, int p, int n, '
                 'int c) { return tfgpc::part_end(b, e, p, n, c); }\n')
  subprocess.run(["g++", "-O1", "-shared", "-fPIC", "-I", build.CSRC, str(src), "-o", str(so)],
                 check=True)
  return ctypes.CDLL(str(so)).part_end


# lists around and far beyond the length at which chunks x parts passes 2^31, up to the
# most pairs an entry accepts
@pytest.mark.parametrize("begin,pairs,parts", [
    (0, 5, 1), (7, 40, 3), (0, 7_250_000, 4736), (0, 7_300_000, 4736), (16, 9_700_000, 4736),
    (1 << 30, (1 << 30) - 1, 4736), (0, (1 << 31) - 32, 2368), (0, (1 << 31) - 1, 4736)])
def test_list_parts_cover_the_list(part_end, begin, pairs, parts):
  end, chunk = begin + pairs, 16
  ends = [begin] + [part_end(begin, end, p, parts, chunk) for p in range(1, parts + 1)]
  assert ends[-1] == end
  share = -(-pairs // chunk) // parts
  for a, b in zip(ends, ends[1:]):
    assert begin <= a <= b <= end
    assert b == end or share * chunk <= b - a <= (share + 1) * chunk


GRANTED_SRC = """
#include <chrono>
#include <thread>
#include "granted.h"
// Two threads ask for `first` and `second`, the second while the first one's request is on its
// way; then `first` is asked for again.  What the driver holds at the end.
extern "C" int held(int first, int second) {
  tfgpc::Granted granted;
  std::atomic<int> driver{0}, under_way{0}, second_done{0};
  std::thread other([&] {
    while (!under_way) std::this_thread::yield();
    granted.reach(second, [&](int size) { driver = size; return 0; });
    second_done = 1;
  });
  granted.reach(first, [&](int size) {
    driver = size;
    under_way = 1;
    for (int i = 0; i < 200 && !second_done; ++i)
      std::this_thread::sleep_for(std::chrono::milliseconds(1));
    return 0;
  });
  other.join();
  granted.reach(first, [&](int size) { driver = size; return 0; });
  return driver;
}
// A request that is refused is made again.
extern "C" int asked_after_refusal() {
  tfgpc::Granted granted;
  int asked = 0;
  granted.reach(5, [&](int) { ++asked; return 1; });
  granted.reach(5, [&](int) { ++asked; return 0; });
  granted.reach(5, [&](int) { ++asked; return 0; });
  return asked;
}
"""


def test_shared_memory_of_two_threads(tmp_path):
  """The shared memory that a kernel may take is not lowered under a thread that counts on it."""
  src, so = tmp_path / "granted.cpp", tmp_path / "granted.so"
  src.write_text(GRANTED_SRC)
  subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-shared", "-fPIC", "-I", build.CSRC,
                  str(src), "-o", str(so)], check=True)
  lib = ctypes.CDLL(str(so))
  assert lib.held(230656, 197888) == 230656
  assert lib.held(197888, 230656) == 230656
  assert lib.asked_after_refusal() == 2


def test_sums_by_neighbor_refuse_host_memory():
  """Pointers of another device never reach the kernel: raised before any launch."""
  torch = pytest.importorskip("torch")
  from tensorflow_graphics_point_clouds_b200 import _lib
  add = _lib.host().add_by_neighbor
  pairs, values = torch.zeros((3, 2), dtype=torch.int32), torch.ones(3)
  with pytest.raises(ValueError, match="GPU only"):
    add(pairs, values, 4)
  with pytest.raises(ValueError, match="GPU only"):
    add(pairs.to("meta"), values, 4)


def test_build_cell_grid_returns_a_pair(monkeypatch):
  """(grid, count); with densities there are four values, from an entry of its own."""
  pytest.importorskip("torch")
  from tensorflow_graphics_point_clouds_b200 import _lib, custom_ops
  seen = []

  class Host:
    @staticmethod
    def build_grid(*args):
      seen.append(args)
      return "grid", "count", "pdf", "packed"

  monkeypatch.setattr(_lib, "host", lambda: Host)
  grid, count = custom_ops.build_cell_grid("points", "ids", 2, [0.1] * 3, 64, max_neighs=5)
  assert (grid, count) == ("grid", "count") and seen[0][-3:] == (5, None, 0)
  both = custom_ops.build_cell_grid_with_pdf("points", "ids", 2, [0.1] * 3, 64, "inv", pdf_mode=1)
  assert both == ("grid", "count", "pdf", "packed") and seen[1][-3:] == (0, "inv", 1)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("ids", ["int32", "int64"])
def test_clouds_follow_the_default_device(dtype, ids):
  """Host arrays given to a cloud go to the default device, whatever their type is, and the
  batch ids with the points; without one they stay where they are, uncopied if they can."""
  torch = pytest.importorskip("torch")
  from tensorflow_graphics_point_clouds_b200 import pc
  points = torch.zeros((4, 3), dtype=getattr(torch, dtype))
  batch_ids = torch.zeros(4, dtype=getattr(torch, ids))
  cloud = pc.PointCloud(points, batch_ids, 1)
  assert cloud._points.device.type == cloud._batch_ids.device.type == "cpu"
  assert (cloud._points is points) == (dtype == "float32")
  assert (cloud._batch_ids is batch_ids) == (ids == "int32")
  with torch.device("meta"):
    cloud = pc.PointCloud(points, batch_ids, 1)
  assert cloud._points.device.type == cloud._batch_ids.device.type == "meta"
  assert cloud._points.dtype == torch.float32 and cloud._batch_ids.dtype == torch.int32
