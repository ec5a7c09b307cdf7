"""The per-device bookkeeping behind the kernels' shared-memory limits, on the host."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "null--space-free-6d-projection-method_b200", "csrc")

PROGRAM = r"""
#include "device_once.h"
#include <cstdio>
#include <initializer_list>
int main() {
  fame::DeviceOnce once, other;
  int runs[2] = {0, 0}, fails = 0, out = 0;
  for (int i = 0; i < 3; ++i)
    for (int d = 0; d < 2; ++d) if (once(d, [&] { ++runs[d]; return 0; }) != 0) return 1;
  if (runs[0] != 1 || runs[1] != 1) return 2;                       // once on each device
  if (other(1, [&] { ++runs[1]; return 0; }) != 0 || runs[1] != 2) return 3;  // each has its own record
  if (once(5, [&] { ++fails; return 7; }) != 7 || once(5, [&] { ++fails; return 0; }) != 0 || fails != 2) return 4;
  if (once(5, [&] { ++fails; return 7; }) != 0 || fails != 2) return 5;       // done only after a success
  for (int d : {-1, 64, -1, 64}) once(d, [&] { ++out; return 0; });
  if (out != 4) return 6;                                           // devices it cannot record
  if (once(63, [&] { return 0; }) != 0 || once(63, [&] { return 9; }) != 0) return 7;
  std::puts("ok");
  return 0;
}
"""


def test_once_per_device(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.returncode


def test_no_limit_is_set_once_per_process():
    """cudaFuncSetAttribute is called from ensure_smem, or on every launch, never from a static's
    initialiser."""
    for f in sorted(os.listdir(CSRC)):
        text = open(os.path.join(CSRC, f)).read()
        for m in re.finditer(r"cudaFuncSetAttribute", text):
            statement = text[max(text.rfind(c, 0, m.start()) for c in ";{}") :m.start()]
            assert "static" not in statement and "[]" not in statement, (f, statement)
        assert not re.search(r"static\s+(int|const\s+\w+)\s+\w+\s*=\s*(ensure_smem|cudaFuncSetAttribute|\[\]\s*\{\s*return\s+cudaFuncSet)", text), f
