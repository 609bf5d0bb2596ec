"""The texel after a sample's origin (csrc/tex_emul.cuh, the functions the kernels call, compiled for the
host) at the ends of int, to which a coordinate beyond its range converts, with overflow checks."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_next_texel_of_a_saturated_coordinate(tmp_path):
    (tmp_path / "t.cpp").write_text(r"""
#include <algorithm>
#include <climits>
#include <cmath>
using std::max; using std::min;
static inline float __fsub_rn(float a, float b) { return a - b; }
#include "lct.h"
#include "tex_emul.cuh"
int main() {
  const int v[] = {INT_MIN, INT_MIN + 1, -2, -1, 0, 1, 6, 7, 8, INT_MAX - 1, INT_MAX};
  for (int n : {1, 2, 8})
    for (int i : v) {
      const long long want = std::min(std::max((long long)i + 1, 0LL), (long long)n - 1);
      if (std::min(std::max(lct::below_max(i) + 1, 0), n - 1) != want) return 1;
      if (std::min(std::max(lct::below_max(i), 0), n - 1) != std::min(std::max(i, 0), n - 1)) return 2;
      if ((unsigned)lct::next_texel(i) != (unsigned)((long long)i + 1)) return 3;
    }
  return 0;
}
""")
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=signed-integer-overflow",
                    "-fno-sanitize-recover=all", "-I", str(ROOT / "listctrecons_b200" / "csrc"),
                    "-I", str(ROOT / "include"), "-I", "/usr/local/cuda/include",
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    subprocess.run([str(tmp_path / "t")], check=True)
