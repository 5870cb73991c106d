"""The level kernels' plan, on the CPU: every node is taken by one launch, by a unit
that can hold it, and clusters shrink to what the device has room for."""

import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "adaptive-regression-trees-art-_b200" / "csrc"

SOURCE = """
#include "level_plan.cuh"
#include <cstdio>
using namespace art;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\\n", __LINE__, #x); return 1; } } while (0)
int main() {
  const int64_t rows[] = {0, 1, 255, 256, 257, 1023, 1024, 1025, 2048, 2049, 6144, 6145, 16384, 16385, 1 << 18, int64_t(1) << 40};
  int64_t last = 0;
  for (int64_t count = 1; count <= 0x7fffffff; count += count < 20000 ? 1 : count / 7) {
    const LevelPlan a = level_small(count), b = level_large(count);
    const bool both = count > kLevelFew;
    CHECK(a.count == count && b.count == count && a.nodes >= 1 && b.nodes >= 1 && b.nodes <= kLevelThreads);
    CHECK((count + a.nodes - 1) / a.nodes <= 0x7fffffff && (count + b.nodes - 1) / b.nodes * kMaxRanks <= 0x7fffffff);
    CHECK(a.single <= kSingleRows && a.single <= a.joint && a.single != 0 && a.joint <= int64_t(32) * 8192);
    CHECK(!both || a.joint == b.joint);
    CHECK(a.joint >= last);
    last = a.joint;
    for (int64_t n : rows) {
      const int taken = (both && n <= a.single) + (both && n > a.single && n <= a.joint) + (n > b.joint);
      CHECK(taken == 1);
    }
  }
  for (int room = 1; room <= 20; ++room) {
    const int c = level_cluster([&](int size) { return size <= room; });
    CHECK(c <= room && (c == kMaxRanks || 2 * c > room) && kMaxRanks % c == 0);
  }
  return 0;
}
"""


def test_every_node_is_taken_once(tmp_path):
    (tmp_path / "plan.cpp").write_text(SOURCE)
    exe = tmp_path / "plan"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), str(tmp_path / "plan.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
