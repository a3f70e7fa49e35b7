"""Kernel set-up is per device (csrc/qm_device_once.h): run once on each, by
any number of threads, again after a failure, and each device keeps its own
answer.  Compiled for the host, with a counter in the place of the CUDA calls."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "querymode_b200", "csrc")

SOURCE = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "qm_device_once.h"

int main() {
  qm_device_once once;
  std::atomic<int> runs[3] = {};
  int fail_left = 1;
  auto set = [&](int dev) {
    return once.get(dev, [&, dev] {
      runs[dev]++;
      if (dev == 2 && fail_left-- > 0) return qm_kernel_setup{1, 0};
      return qm_kernel_setup{0, 10 + dev};
    });
  };
  std::vector<std::thread> th;
  for (int t = 0; t < 8; t++)
    th.emplace_back([&, t] {
      for (int i = 0; i < 1000; i++)
        if (set(t & 1).per_sm != 10 + (t & 1)) std::printf("wrong answer\n");
    });
  for (auto &t : th) t.join();
  if (set(2).error != 1 || set(2).error != 0 || set(2).per_sm != 12) std::printf("failure kept\n");
  std::printf("%d %d %d\n", runs[0].load(), runs[1].load(), runs[2].load());
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "1 1 2\n"


def test_part_kernels_use_it():
    """No once_flag (one per process) decides a kernel's limits any more."""
    for name in os.listdir(CSRC):
        with open(os.path.join(CSRC, name)) as f:
            assert "once_flag" not in f.read(), name
