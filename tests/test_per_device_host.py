"""Occupancy tables and function attributes belong to a device, and one process may have contexts on
several: what is kept of them is kept per device (csrc/mh_per_device.h)."""
import glob
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "marinehydro.jl_gb300", "csrc")

PROGRAM = """
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "mh_per_device.h"
int main() {
  mh::PerDevice<int> table;
  std::atomic<int> made{0};
  std::vector<std::thread> threads;
  std::atomic<int> wrong{0};
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int q = 0; q < 1000; ++q) {
        const int device = (q + t) % 5;
        if (table.get(device, [&] { ++made; return 100 + device; }) != 100 + device) ++wrong;
      }
    });
  for (auto& t : threads) t.join();
  std::printf("%d %d\\n", made.load(), wrong.load());
}
"""


def test_one_value_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    assert out == ["5", "0"]  # made once for each of the five devices, never another's


def test_no_process_wide_tables():
    # a function's static initialised by a call or a lambda is made once per process
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        with open(path) as f:
            found = re.findall(r"^[ \t]+static const [^\n]*= *(?:\[|\w+\()[^\n]*", f.read(), re.M)
        assert not found, (os.path.basename(path), found)
