"""The cut of the Taylor moments' modes, on the host: every mode once, whole stages, at most 4096."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "null--space-free-6d-projection-method_b200", "csrc")

PROGRAM = r"""
#include "moment_slices.h"
#include <cstdio>
int main() {
  for (int N = 1; N <= 7; ++N) {
    long long NF = 1;
    for (int d = 0; d < 6; ++d) NF *= 2 * N;
    for (long long slots : {1LL, 132LL, 148LL, 160LL})
      for (long long tiles = 1; tiles <= 4100; tiles += tiles < 700 ? 1 : 17) {
        int ns = 0;
        long long per = 0;
        fame::moment_slices(NF, tiles, slots, 32, 4096, &ns, &per);
        if (per > 4096 || per < 128 || per % 32 != 0 || ns < 1 || ns * per < NF || (ns - 1) * per >= NF) {
          std::printf("N=%d tiles=%lld slots=%lld: %d slices of %lld\n", N, tiles, slots, ns, per);
          return 1;
        }
      }
  }
  return 0;
}
"""


def test_slices(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "slices.cpp", tmp_path / "slices"
    src.write_text("#include <initializer_list>\n" + PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
