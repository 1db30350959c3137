"""The reductions' scratch slots (aces4_gb300/csrc/reduction_slots.h), compiled
for the host: launches that can be on the GPU at once never hold the same one,
however many calls lie between them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHECK = r"""
#include <cstdio>
#include <set>
#include "reduction_slots.h"
#define REQUIRE(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main() {
  a4g::SlotTable t;
  const int first = t.slot(0, 7), captured = t.slot(1, 7), other = t.slot(1, 8), second = t.slot(2, 7);
  std::set<int> all = {first, captured, other, second};
  REQUIRE(all.size() == 4);
  for (int i = 0; i < 100000; ++i) {  // calls on other streams take nothing away
    const int q = t.slot(0, 100 + i % 200);
    REQUIRE(q >= 0 && !all.count(q));
  }
  REQUIRE(t.slot(0, 7) == first && t.slot(1, 7) == captured && t.slot(1, 8) == other && t.slot(2, 7) == second);
  // a graph that is gone gives its slots back, and only its own
  REQUIRE(t.has_capture(1) && t.has_capture(2) && !t.has_capture(3));
  t.release(1);
  t.release(9);
  REQUIRE(!t.has_capture(1) && t.has_capture(2) && t.slot(2, 7) == second && t.slot(0, 7) == first);
  std::set<int> again = {t.slot(3, 1), t.slot(3, 2)};
  REQUIRE(again == (std::set<int>{captured, other}));
  // bounded: 256 streams, and graphs that come and go
  for (int i = 0; i < 1000; ++i) t.slot(0, 1000 + i);
  REQUIRE(t.slot(0, 5000) == -1 && t.slot(0, 7) == first && t.slot(4, 5000) >= 0);
  const int used = t.slots();
  for (unsigned long long c = 10; c < 50000; ++c) {
    REQUIRE(t.slot(c, 7) >= 0);
    t.release(c);
  }
  REQUIRE(t.slots() <= used + 1 && used <= a4g::SlotTable::kMaxStreams + 8);
  for (unsigned long long c = 100000; c < 100000 + a4g::SlotTable::kMaxSlots; ++c) t.slot(c, 1);
  REQUIRE(t.slots() == a4g::SlotTable::kMaxSlots && t.slot(999999, 1) == -1);
  std::printf("ok\n");
  return 0;
}
"""


def test_slots_are_never_shared(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(CHECK)
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "aces4_gb300", "csrc"), "-o", str(exe), str(src)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
