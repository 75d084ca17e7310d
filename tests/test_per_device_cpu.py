"""Set-up that belongs to a device runs once for each device (contexts of one
process may be on several): the helper, compiled alone, and that no kernel's
shared-memory limit is set once per process instead."""
import glob
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "py_fof_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.cuh"
int main() {
  static pyfof::PerDeviceOnce once;
  std::atomic<int> calls[4] = {};
  std::atomic<int> wrong{0};
  std::vector<std::thread> th;
  for (int t = 0; t < 16; ++t)
    th.emplace_back([&, t] {
      for (int i = 0; i < 200; ++i) {
        const int dev = (t + i) % 4;
        // device 2 fails, the others must not notice
        const int r = once.run(dev, [&] { ++calls[dev]; return dev == 2 ? 7 : 0; });
        if (r != (dev == 2 ? 7 : 0)) ++wrong;
      }
    });
  for (auto &t : th) t.join();
  std::printf("%d %d %d %d %d %d %d\n", calls[0].load(), calls[1].load(), calls[2].load(), calls[3].load(),
              wrong.load(), (int)once.run(-1, [] { return 0; }), (int)once.run(64, [] { return 0; }));
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["1", "1", "1", "1", "0", "-1", "-1"]


def test_no_limit_is_set_once_per_process():
    for path in glob.glob(os.path.join(CSRC, "*.cu*")):
        if os.path.basename(path) == "per_device.cuh":
            continue
        assert not re.search(r"\bonce_flag\b|\bcall_once\b", open(path).read()), path
