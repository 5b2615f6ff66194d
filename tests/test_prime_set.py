"""The set of primes whose twiddles are rows of doubles: what it cannot hold it does not
claim to, and every configuration's primes fit it."""
import ctypes
import os
import shutil
import subprocess

import pytest

from fhe_b200 import _lib

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fhe_b200", "csrc")

CHECK = r"""
#include <cstdio>
#include "modarith.cuh"
int main() {
  fhe_b200::PrimeSet s;
  int bad = 0;
  for (int i = 0; i < s.kPrimes + 70; i++) {
    const bool took = s.add(i);
    if (took != s.has(i) || took != (i < s.kPrimes)) bad++;
  }
  std::printf("%d %d\n", bad, s.kPrimes);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_the_set_holds_every_configurations_primes(tmp_path):
    source, exe = str(tmp_path / "check.cpp"), str(tmp_path / "check")
    with open(source, "w") as f:
        f.write(CHECK)
    subprocess.run(["g++", "-std=c++17", "-I", CSRC, "-o", exe, source], check=True)
    bad, capacity = map(int, subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0
    lib, most = _lib.load(), 0
    for preset, sizes in ((1, range(13, 18)), (2, (16,)), (3, (3, 4)), (4, (3, 4))):
        for log_n in sizes:
            for special in (0, 1, 2, 16):  # the fewest give the longest chains
                cfg, info = _lib.FheConfig(log_n, -1, special, -1, preset), _lib.FheEngineInfo()
                if lib.fhe_parameters_query(ctypes.byref(cfg), ctypes.byref(info), None, 0) == 0:
                    most = max(most, info.prime_count)
    assert 80 < most <= capacity
