"""Kernels' shared memory limits: raised once per kernel and device (csrc/smem_limit.cuh, compiled
for the host with a counting stand-in for the CUDA call)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "casadi_gb300",
                    "csrc")
MAIN = r"""
#include "smem_limit.cuh"
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#define CHECK(c) if (!(c)) { std::printf("%s\n", #c); return 1; }
int main() {
  cgb::SmemLimits l;
  int a = 0, b = 0, calls = 0;
  auto ok = [&] { ++calls; return 0; };
  auto bad = [&] { ++calls; return 7; };
  CHECK(l.once(&a, 0, ok) == 0 && calls == 1);
  CHECK(l.once(&a, 0, ok) == 0 && calls == 1);  // raised already
  CHECK(l.once(&a, 1, ok) == 0 && calls == 2);  // another device has a limit of its own
  CHECK(l.once(&b, 1, ok) == 0 && calls == 3);  // and so has another kernel
  CHECK(l.once(&a, 1, ok) == 0 && calls == 3);
  CHECK(l.once(&b, 63, bad) == 7 && calls == 4);
  CHECK(l.once(&b, 63, ok) == 0 && calls == 5);  // a failure is not kept
  CHECK(l.once(&b, 63, bad) == 0 && calls == 5);
  CHECK(l.once(&b, 64, ok) == 0 && l.once(&b, 64, ok) == 0 && calls == 7);  // past the bit set
  std::atomic<int> n{0};
  std::vector<std::thread> ts;
  for (int k = 0; k < 8; ++k)
    ts.emplace_back([&] { for (int r = 0; r < 1000; ++r) l.once(&n, r % 4, [&] { ++n; return 0; }); });
  for (auto& t : ts) t.join();
  CHECK(n == 4);
  return 0;
}
"""


def test_limits_are_raised_once_per_kernel_and_device(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-x", "c++", "-I", CSRC,
                    str(tmp_path / "main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
