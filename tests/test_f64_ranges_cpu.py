"""Index arithmetic of the plain FP64 tiles (aces4_gb300/csrc/grouped.h) at the
largest k ranges that a call accepts, compiled for the host: the shares of a
tile's k steps meet end to end and stay within the range."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cstdio>
#include "grouped.h"
using namespace a4g;
int main() {
  const int top = 0x7fffffff;
  for (int K : {1, 15, 16, 17, 1000, top - 33, top - 32, top - 31, top - 17, top - 16, top - 15, top - 1, top}) {
    const int steps = ceil_div(K, kF64Step);
    if (steps < 1 || (long long)steps * kF64Step < K || (long long)(steps - 1) * kF64Step >= K) return std::printf("steps %d\n", K), 1;
    for (int ranks : {1, 2, 4, 8, 16}) {
      int at = 0;
      for (int r = 0; r < ranks; ++r) {
        const int lo = f64_step_start(int((long long)steps * r / ranks), K), hi = f64_step_start(int((long long)steps * (r + 1) / ranks), K);
        if (lo != at || hi < lo || hi > K) return std::printf("share %d of %d, K %d: %d .. %d\n", r, ranks, K, lo, hi), 1;
        at = hi;
      }
      if (at != K) return std::printf("K %d: %d\n", K, at), 1;
    }
  }
  if (ceil_div(top, 8) != 268435456) return 1;
  std::printf("ok\n");
  return 0;
}
"""


def test_shares_of_the_largest_ranges(tmp_path):
    nvcc = shutil.which("nvcc") or ("/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else None)
    if nvcc is None:
        pytest.skip("nvcc not available")
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(CHECK)
    r = subprocess.run([nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "aces4_gb300", "csrc"), "-o", str(exe), str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
