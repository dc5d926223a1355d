"""CPU test of the shared-memory limit that a kernel's launches raise: per device, only ever upwards, from any thread."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MAIN = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "smem_limit.h"
static std::atomic<size_t> attr[2];      // what a device's attribute stands at, and how often it was changed
static std::atomic<int> calls[2], bad;
static int ask(b200::SmemLimit& l, int dev, size_t bytes, bool refuse = false) {
  const int rc = l.raise(dev, bytes, [&](size_t n) { if (refuse) return 1; ++calls[dev]; attr[dev] = n; return 0; });
  if (rc == 0 && attr[dev] < bytes) ++bad;
  return rc;
}
int main() {
  b200::SmemLimit a;
  ask(a, 0, 100); ask(a, 0, 50); ask(a, 0, 100);             // a smaller size changes nothing
  std::printf("%zu %d ", attr[0].load(), calls[0].load());
  ask(a, 1, 60);                                             // another device has its own limit
  std::printf("%zu %d ", attr[1].load(), calls[1].load());
  std::printf("%d ", ask(a, 0, 300, true));                  // refused: not remembered as allowed
  ask(a, 0, 200);
  std::printf("%zu %d ", attr[0].load(), calls[0].load());
  b200::SmemLimit b;
  attr[0] = attr[1] = 0;
  std::vector<std::thread> t;
  for (int i = 0; i < 8; ++i)
    t.emplace_back([&b, i] { for (int j = 0; j < 20000; ++j) ask(b, (i + j) & 1, (size_t)((i * 7919 + j * 104729) % 5000) + 1); });
  for (auto& q : t) q.join();
  std::printf("%d\n", bad.load());
}
"""


def test_limit_is_per_device_and_only_raised(tmp_path):
    (tmp_path / "main.cc").write_text(MAIN)
    exe = str(tmp_path / "limit")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "relax_b200", "csrc"), str(tmp_path / "main.cc"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    assert out == ["100", "1", "60", "1", "1", "200", "2", "0"]
