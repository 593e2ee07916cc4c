"""The host code's memory of what a device answered, compiled and run here."""
import shutil
import subprocess

import pytest

from sonicboom_b200.csrc.build import SRC_DIR

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "device_cache.h"
int main() {
  static SbDeviceCache c;
  int asked = 0;
  auto ask = [&](int v) { return [&asked, v] { ++asked; return v; }; };
  if (c.get(0, ask(-1)) != -1 || c.get(0, ask(18)) != 18) return 1;      // a failed query is asked again
  if (c.get(0, ask(7)) != 18 || asked != 2) return 2;                    // an answer is kept
  if (c.get(1, ask(0)) != 0 || c.get(1, ask(5)) != 0) return 3;          // for its device only, also when it is none
  if (c.get(-1, ask(4)) != 4 || c.get(-1, ask(3)) != 3 || c.get(SbDeviceCache::DEVICES, ask(2)) != 2) return 4;
  std::vector<std::thread> threads;
  std::atomic<int> wrong{0};
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&] {
      for (int d = 2; d < 60; ++d) wrong += c.get(d, [d] { return 100 + d; }) != 100 + d;
    });
  for (auto& t : threads) t.join();
  return wrong ? 5 : 0;
}
"""


def test_device_cache(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(SRC_DIR), str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t"),
                    "-pthread"], check=True)
    assert subprocess.run([str(tmp_path / "t")]).returncode == 0
