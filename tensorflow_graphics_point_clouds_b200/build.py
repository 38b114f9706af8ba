"""Builds libtfgpc.so (the C-ABI CUDA library) in-tree with nvcc for sm_100a, and
_host.so (the host layer over it, C++ against torch's headers).

Usage: python -m tensorflow_graphics_point_clouds_b200.build [--force] [--verbose]
"""
import concurrent.futures
import os
import shutil
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
INCLUDE = os.path.join(os.path.dirname(HERE), "include")
LIB = os.path.join(HERE, "libtfgpc.so")
HOST_SRC = os.path.join(HERE, "host")
HOST_LIB = os.path.join(HERE, "_host.so")
OBJ_DIR = os.path.join(HERE, "build")

NVCC_FLAGS = [
    "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-lineinfo",
    "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-I", INCLUDE, "-I", CSRC,
]


def _nvcc():
  for cand in (os.environ.get("NVCC"), shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
    if cand and os.path.exists(cand):
      return cand
  raise RuntimeError("nvcc not found")


def sources():
  return sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def _newer(lib, *folders):
  """Whether lib exists and is newer than every file of the folders."""
  paths = [os.path.join(d, f) for d in folders for f in os.listdir(d)]
  return os.path.exists(lib) and os.path.getmtime(lib) >= max(os.path.getmtime(p) for p in paths)


def up_to_date():
  return _newer(LIB, CSRC, INCLUDE) and _newer(HOST_LIB, HOST_SRC, INCLUDE)


def _run(cmd, what):
  res = subprocess.run(cmd, capture_output=True, text=True)
  if res.returncode != 0:
    raise RuntimeError("%s failed:\n%s\n%s" % (what, res.stdout, res.stderr))
  return res


def build_host():
  """_host.so: links against libtfgpc.so beside it and the torch it is built with."""
  import sysconfig
  from torch.utils import cpp_extension
  flags = ["-O2", "-std=c++17", "-fPIC", "-fvisibility=hidden", "-DTORCH_EXTENSION_NAME=_host",
           "-DTORCH_API_INCLUDE_EXTENSION_H", "-I", INCLUDE, "-I", sysconfig.get_paths()["include"]]
  for d in cpp_extension.include_paths() + [os.path.join(os.path.dirname(_nvcc()), "..", "include")]:
    flags += ["-isystem", d]
  os.makedirs(OBJ_DIR, exist_ok=True)

  def compile_one(src):
    obj = os.path.join(OBJ_DIR, "host_" + src[:-4] + ".o")
    _run(["g++"] + flags + ["-c", os.path.join(HOST_SRC, src), "-o", obj], "g++ for " + src)
    return obj

  with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
    objs = list(ex.map(compile_one, sorted(f for f in os.listdir(HOST_SRC) if f.endswith(".cpp"))))
  libs = [a for d in cpp_extension.library_paths() for a in ("-L", d)]
  _run(["g++", "-shared", "-o", HOST_LIB] + objs + [LIB, "-Wl,-rpath,$ORIGIN"] + libs +
       ["-lc10", "-lc10_cuda", "-ltorch", "-ltorch_cpu", "-ltorch_python"], "linking _host.so")
  return HOST_LIB


def build(force=False, verbose=False):
  if force or not _newer(LIB, CSRC, INCLUDE):
    _build_library(verbose)
  if force or not _newer(HOST_LIB, HOST_SRC, INCLUDE):
    build_host()
  return LIB


def _build_library(verbose):
  nvcc = _nvcc()
  os.makedirs(OBJ_DIR, exist_ok=True)
  extra = ["-Xptxas", "-v"] if verbose else []

  def compile_one(src):
    obj = os.path.join(OBJ_DIR, src[:-3] + ".o")
    cmd = [nvcc] + NVCC_FLAGS + extra + ["-c", os.path.join(CSRC, src), "-o", obj]
    res = subprocess.run(cmd, capture_output=True, text=True)
    if res.returncode != 0:
      raise RuntimeError("nvcc failed for %s:\n%s\n%s" % (src, res.stdout, res.stderr))
    if verbose:
      sys.stderr.write(res.stderr)
    return obj

  with concurrent.futures.ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as ex:
    objs = list(ex.map(compile_one, sources()))
  _run([nvcc, "-shared", "-o", LIB, "-Xlinker", "-soname=libtfgpc.so"] + objs +
       ["-gencode", "arch=compute_100a,code=sm_100a"], "linking libtfgpc.so")


if __name__ == "__main__":
  print(build(force="--force" in sys.argv, verbose="--verbose" in sys.argv))
