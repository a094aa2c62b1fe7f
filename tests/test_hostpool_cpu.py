"""The host loops' thread pool (csrc/pd_hostpool.h), compiled on its own."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "peridem_gb300" / "csrc"

SLOTS = r"""
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <vector>
#include "pd_hostpool.h"
int main() {
  for (unsigned width : {0u, 1u, 2u, 3u, 40u})
    for (uint64_t n : {0ull, 1ull, 2ull, 1000ull}) {
      std::vector<std::atomic<int>> seen(n);
      std::atomic<unsigned> top(0);
      pdg::parallel_slots(n, width, [&](uint64_t i, unsigned slot) {
        seen[i]++;
        for (unsigned t = top; slot > t && !top.compare_exchange_weak(t, slot);) {
        }
      });
      for (auto &x : seen)
        if (x != 1) return std::printf("width %u n %llu: an index ran %d times\n", width, (unsigned long long)n, x.load()), 1;
      if (top >= (width ? width : 1)) return std::printf("width %u: slot %u\n", width, top.load()), 1;
    }
  return 0;
}
"""


def test_slots_stay_below_the_callers_width(tmp_path):
    """A loop's threads are told apart by slots below the width that its caller laid its buffers out
    for, whatever number of cores the machine has now."""
    src, exe = tmp_path / "slots.cpp", tmp_path / "slots"
    src.write_text(SLOTS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
