"""The rules that chained kernels rest on (launch_chained in common.cuh), checked in the
sources: such a kernel begins before its inputs are written, and beside the one before it."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "tensorflow_graphics_point_clouds_b200", "csrc")
READ_ONLY = re.compile(r"\b__ldg\b|\bld\.global\.nc\b|const\s[^,()]*\*\s*(const\s+)?__restrict__")


def source(name):
  with open(os.path.join(CSRC, name)) as f:
    text = f.read()
  return re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", text), flags=re.S)


def with_headers(name, seen=None):
  seen = set() if seen is None else seen
  if name in seen or not os.path.exists(os.path.join(CSRC, name)):
    return ""
  seen.add(name)
  text = source(name)
  return "".join(with_headers(h, seen) for h in re.findall(r'#include "([^"]+)"', text)) + text


def functions(text):
  """{name: (is a kernel, signature, body)} of everything that runs on the GPU."""
  found = {}
  for m in re.finditer(r"__global__|__device__", text):
    brace, end = text.find("{", m.start()), text.find(";", m.start())
    if brace < 0 or 0 <= end < brace:
      continue
    signature = text[m.start():brace]
    name = re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "",
                                           signature))
    depth, at = 0, brace
    while True:
      depth += {"{": 1, "}": -1}.get(text[at], 0)
      at += 1
      if depth == 0:
        break
    if name:
      kernel, old_sig, old_body = found.get(name.group(1), (False, "", ""))
      found[name.group(1)] = (kernel or m.group(0) == "__global__", old_sig + signature,
                              old_body + text[brace:at])
  return found


def reached(name, funcs):
  todo, seen = [name], set()
  while todo:
    f = todo.pop()
    if f not in seen:
      seen.add(f)
      todo += [g for g in set(re.findall(r"\w+", funcs[f][2])) if g in funcs]
  return seen


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))


def test_a_broken_rule_is_seen():
  funcs = functions("__device__ float get(const float* p) { return __ldg(p); }\n"
                    "__global__ void a_kernel(const float* __restrict__ x) { chain_enter(); }\n"
                    "__global__ void __launch_bounds__(f(1) * 32, 1)\nb_kernel(float* x) { get(x); }")
  assert READ_ONLY.search(funcs["a_kernel"][1])
  assert reached("b_kernel", funcs) == {"b_kernel", "get"} and READ_ONLY.search(funcs["get"][2])


@pytest.mark.parametrize("name", FILES)
def test_chained_kernels(name):
  text = with_headers(name)
  funcs = functions(text)
  for kernel, (is_kernel, signature, body) in funcs.items():
    if not is_kernel:
      continue
    enter = re.search(r"chain_(enter|wait)\(", body)
    chained = enter is not None
    # a kernel with both kinds of instance: the last template argument says which
    switched = "if (CHAINED) chain_enter(" in body
    launched = False
    # launched one way or the other, by name or through a variable that holds the name
    for m in re.finditer(r"\b%s\b(?:<[^;<>()]*(?:\([^()]*\))?[^;<>()]*>)?" % kernel, text):
      line = text[text.rfind(";", 0, m.start()) + 1:m.start()]
      after = text[m.end():].lstrip()
      wanted = "true>" in m.group(0) if switched else chained
      if "__global__" in line:
        continue
      variable = re.search(r"auto\*? (\w+) =", line)
      uses = [line + after[:3]]
      if variable:
        scope = text[m.end():text.find("\n}\n", m.end())]
        until = re.search(r"auto\*? %s =" % variable.group(1), scope)
        uses = re.findall(r"[^;]*\b%s\b(?:<<<|[^;]*)" % variable.group(1),
                          scope[:until.start()] if until else scope)
        uses = [u for u in uses if "launch_chained" in u or "<<<" in u]
        assert uses, kernel
      for use in uses:
        launched = launched or "launch_chained" in use or "cudaLaunchKernelEx" in use
        by_attribute = "launch_chained" in use or "cudaLaunchKernelEx" in use
        if by_attribute or "<<<" in use:
          assert by_attribute == wanted, "%s: %s" % (kernel, use.strip()[:200])
    assert launched == chained, kernel
    if not chained:
      continue
    # inputs are written until the wait ends: no read-only loads, here or in what it calls
    # (ld_input<CHAINED> loads as the instance may)
    for f in reached(kernel, funcs) - ({"ld_input"} if switched else set()):
      assert not re.search(r"ld_input<(?!CHAINED>)", funcs[f][2]), (kernel, f)
      assert not READ_ONLY.search(funcs[f][1] + funcs[f][2]), (kernel, f)
    # and nothing is read or written before
    before = body[:enter.start()]
    assert not re.search(r"ld_global|__ldc|atomic|\bst_|mbar_wait|tma_|cp_async", before), kernel
    # tensor memory is held before the next kernel may come and ask for it
    if "tmem_alloc" in body:
      assert re.search(r"tmem_alloc.*__syncthreads\(\)", before, re.S), kernel
