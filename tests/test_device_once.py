"""What launches set once per device (kernel attributes) is kept for each device, from any
thread."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fhe_b200", "csrc")

CHECK = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "device_once.hpp"
int main() {
  int bad = 0;
  fhe_b200::DeviceOnce once;
  once.set_done(0);
  if (!once.done(0)) bad++;
  for (int d = 1; d < 100; d++) if (once.done(d)) bad++;
  once.set_done(70);  // beyond what it keeps: asked for again each time
  if (once.done(70) || once.done(70 - 64)) bad++;
  std::vector<std::thread> threads;
  for (int d = 0; d < 64; d++) threads.emplace_back([&once, d] { once.set_done(d); });
  for (auto &t : threads) t.join();
  for (int d = 0; d < 64; d++) if (!once.done(d)) bad++;
  std::printf("%d\n", bad);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_each_device_is_kept(tmp_path):
    source, exe = str(tmp_path / "check.cpp"), str(tmp_path / "check")
    with open(source, "w") as f:
        f.write(CHECK)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-o", exe, source], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout.strip() == "0"


def test_launchers_keep_no_flag_of_their_own():
    for name in os.listdir(CSRC):
        with open(os.path.join(CSRC, name)) as f:
            assert not re.search(r"static (bool|int) raised", f.read()), name
