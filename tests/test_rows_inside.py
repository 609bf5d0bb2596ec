"""The test that lets the exact backprojector read a sample's row without clamping it (csrc/footprint.cuh,
compiled for the host): wherever it holds, the row of every slice has to lie inside the quad rows
[0, nt + 2], also next to the source, where the row step K and the base M grow without bound and cancel.
Bases M around -j K at every magnitude, for one slice per thread (j from a base up to 15 slices back) and
for groups of two."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include "footprint.cuh"
// row of slice j as the kernel forms it, or false where it lies outside the quads
static bool row_ok(float j, float K, float M, float wt, int nt) {
  const float U = M + (wt + 2.0f);
  const double row = std::floor((double)std::fmaf(j, K, U));
  return row >= 0.0 && row <= nt + 2;
}
int main() {
  long inside1 = 0, inside2 = 0, bad1 = 0, bad2 = 0;
  for (int nt : {2, 8, 31, 64, 320}) {
    const float wt = 0.5f * (nt - 1);
    for (int j = 0; j < 16; ++j)
      for (int e = -10; e < 40; ++e)
        for (int m = 0; m < 64; ++m)
          for (int sg = -1; sg <= 1; sg += 2) {
            const float K = sg * std::ldexp(1.0f + m / 64.0f + (37 * m + 1) * 0x1p-23f, e);
            for (int o = -2 * nt; o <= 2 * nt; ++o) {
              const float M = -j * K + 0.5f * o;
              if (lct::rows_inside<true>(j, j, K, M, wt)) {
                ++inside1;
                bad1 += !row_ok(j, K, M, wt, nt);
              }
              if (j < 15 && lct::rows_inside<false>(j, j + 1, K, M, wt)) {
                ++inside2;
                bad2 += !row_ok(j, K, M, wt, nt) || !row_ok(j + 1, K, M, wt, nt);
              }
            }
          }
  }
  std::printf("%ld %ld %ld %ld\n", inside1, bad1, inside2, bad2);
}
"""


def test_unclamped_rows_lie_inside_the_quads(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I",
                    str(ROOT / "listctrecons_b200" / "csrc"), "-I", "/usr/local/cuda/include",
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout
    inside1, bad1, inside2, bad2 = (int(v) for v in out.split())
    assert inside1 > 10000 and inside2 > 10000
    assert bad1 == 0 and bad2 == 0
