"""Kernel set-up runs once on each device of a process, whichever thread comes first,
and a failure is each caller's (CPU: the class that the launchers use, with device
numbers given)."""
import subprocess

from tests.conftest import ROOT

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "once.h"
int main() {
  static B200Once once;
  std::atomic<int> runs[70] = {};
  auto setup = [&](int dev) { return once.run(dev, [&, dev] { ++runs[dev]; return dev == 3 ? 2 : 0; }); };
  std::atomic<int> wrong{0};
  std::vector<std::thread> threads;
  for (int t = 0; t < 16; ++t)
    threads.emplace_back([&, t] {
      for (int i = 0; i < 200; ++i) {
        const int dev = (t + i) % 5;
        if (setup(dev) != (dev == 3 ? 2 : 0)) ++wrong;
      }
    });
  for (auto &t : threads) t.join();
  for (int dev = 0; dev < 5; ++dev) wrong += runs[dev] != 1;
  wrong += setup(66) != 0 || setup(66) != 0 || runs[66] != 2;  // beyond the table: every time
  printf("%d\n", wrong.load());
  return wrong.load() != 0;
}
"""


def test_set_up_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{ROOT / 'mublis_b200' / 'csrc'}", str(src),
                    "-o", str(exe)], check=True)
    subprocess.run([str(exe)], check=True, timeout=60)


def test_launchers_use_it():
    """No kernel's attributes are set under a flag of the whole process."""
    for src in sorted((ROOT / "mublis_b200" / "csrc").glob("*.cu")):
        text = src.read_text()
        assert text.count("cudaFuncSetAttribute(") == 0 or "static B200Once once" in text, src.name
        assert "static std::once_flag" not in text, src.name
