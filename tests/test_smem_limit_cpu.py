"""The shared-memory limits of the kernels (csrc/smem_limit.h) under concurrent callers: a small host program
with a fake attribute whose setter takes its time.  Whenever raise() has returned for a size, the limit has to
be at least that size and stay there until the launch."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>
#include "smem_limit.h"
int main() {
  int bad = 0;
  for (int round = 0; round < 20; ++round) {
    cssm::SmemLimits limits;
    std::atomic<size_t> attr[2] = {{49152}, {49152}};
    std::atomic<int> short_of{0}, calls{0};
    auto work = [&](int id) {
      std::mt19937 r(round * 100 + id);
      auto nap = [&] { std::this_thread::sleep_for(std::chrono::microseconds(r() % 60)); };
      for (int i = 0; i < 40; ++i) {
        const int k = r() % 2;
        const size_t bytes = 1000 * (1 + r() % 220);
        const int e = limits.raise(&attr[k], 1, bytes, [&](size_t* n) { *n = attr[k].load(); return 0; },
                                   [&](size_t n) { nap(); attr[k].store(n); ++calls; nap(); return 0; });
        nap();                                          // the launch comes later
        if (e != 0 || attr[k].load() < bytes) ++short_of;
      }
    };
    std::vector<std::thread> t;
    for (int id = 0; id < 4; ++id) t.emplace_back(work, id);
    for (auto& x : t) x.join();
    bad += short_of.load();
    // a failing setter is reported and not remembered
    size_t now = 49152;
    auto get = [&](size_t* n) { *n = now; return 0; };
    if (limits.raise(&now, 1, 60000, get, [](size_t) { return 7; }) != 7) ++bad;
    if (limits.raise(&now, 1, 60000, get, [&](size_t n) { now = n; return 0; }) != 0 || now != 60000) ++bad;
    // a new context starts over; an unknown one (0) is asked every time
    for (unsigned long long context : {2ull, 0ull}) {
      now = 49152;
      limits.raise(&now, context, 60000, get, [&](size_t n) { now = n; return 0; });
      if (now != 60000) ++bad;
    }
    now = 49152;
    limits.raise(&now, 0, 60000, get, [&](size_t n) { now = n; return 0; });
    if (now != 60000) ++bad;
  }
  std::printf("%d\n", bad);
  return bad != 0;
}
"""


def test_limits_hold_under_concurrent_callers(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    src, exe = tmp_path / "limits.cpp", tmp_path / "limits"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "cssm_b200", "csrc"), "-o", str(exe), str(src)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, f"{r.stdout.strip()} launches found less than they had asked for"
