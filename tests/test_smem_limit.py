"""CPU: a kernel's shared-memory limit covers every launch, whatever sizes the threads of a program ask for (csrc/smem_limit.h)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# Threads launch one kernel with hundreds of sizes each, on a device of the table and on one beyond it.  `attribute` is what the
# driver holds; a launch fails if it is below the launch's own size.
PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "smem_limit.h"
int main() {
  for (int device : {0, 63, 64, 1000}) {
    tlx::SmemLimit limit;
    std::atomic<size_t> attribute{48 * 1024};
    std::atomic<int> failed{0}, calls{0};
    auto work = [&](int t) {
      for (int i = 0; i < 4000; ++i) {
        const size_t bytes = 1024 * (size_t)(1 + (i * 37 + t * 101) % 227) + 16 * (size_t)(i % 61);
        if (limit.raise(device, bytes, [&](size_t b) { ++calls; attribute = b; return 0; }) != 0) ++failed;
        std::this_thread::yield();
        if (attribute < bytes) ++failed;
      }
    };
    std::vector<std::thread> threads;
    for (int t = 0; t < 6; ++t) threads.emplace_back(work, t);
    for (auto& t : threads) t.join();
    if (failed) { std::printf("device %d: %d launches failed\n", device, failed.load()); return 1; }
    if (device < 64 && calls > 227 * 61) { std::printf("device %d: %d calls\n", device, calls.load()); return 2; }
    // an error is passed on and not remembered as a raised limit
    tlx::SmemLimit other;
    if (other.raise(device, 100000, [](size_t) { return -4; }) != -4) return 3;
    size_t got = 0;
    if (other.raise(device, 90000, [&](size_t b) { got = b; return 0; }) != 0 || got != 90000) return 4;
  }
  return 0;
}
"""


def test_limit_is_raised_and_never_lowered(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "tallax_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout
