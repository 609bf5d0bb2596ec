"""div_by and div_by2 as the kernels call them (csrc/fp32_pair.cuh compiled for the host, where fmaf is one
rounding as on the device) against the FP32 division: every 24-bit fraction of x, both signs, for the constants that
scans have; and divisors that vary from view to view, as the PI-window walk's distances do.  A divisor whose
fraction bits are all ones is the one exception of the method: there the quotient may be one ulp off."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <cuda_runtime.h>
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
static inline float2 __ffma2_rn(float2 a, float2 b, float2 c) {
  return make_float2(std::fmaf(a.x, b.x, c.x), std::fmaf(a.y, b.y, c.y));
}
#include "fp32_pair.cuh"
static float bits(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static uint32_t ubits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static long differ(float x, float d, float r) {
  const float2 p = lct::div_by2(make_float2(x, -x), d, r);
  return (lct::div_by(x, d, r) != x / d) + (lct::div_by(-x, d, r) != -x / d) + (p.x != x / d) + (p.y != -x / d);
}
int main() {
  const float consts[] = {570.0f, 595.0f, 0.6f, 1.0f, 0.5f, 0.97f, (float)(2 * M_PI / 1152), (float)(2 * M_PI / 1160),
                          (float)(2 * M_PI / 120), bits(0x3F800001), bits(0x3F800002), bits(0x3FFFFFFE),
                          1.3333334f, 1.9999995f, 30.72f, 10.4f};
  long bad = 0, bad_view = 0, ones = 0, ones_far = 0;
  for (float d : consts) {
    const float r = 1.0f / d;
    for (uint32_t f = 0; f < (1u << 23); ++f) bad += differ(bits(0x3F800000 | f), d, r);
  }
  // distances of 1 .. 2^11 mm and numerators of 2^-20 .. 2^20
  uint64_t s = 88172645463325252ull;
  auto next = [&] { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
  for (int i = 0; i < 40000000; ++i) {
    const uint64_t a = next();
    const uint32_t df = (uint32_t)a & 0x7FFFFF, de = 127 + (uint32_t)(a >> 23) % 11;
    const uint64_t b = next();
    const float d = bits(de << 23 | df), x = bits((107 + (uint32_t)(b >> 23) % 40) << 23 | ((uint32_t)b & 0x7FFFFF));
    if (df != 0x7FFFFF) bad_view += differ(x, d, 1.0f / d);
  }
  const float all = bits(0x43FFFFFF);  // just below 512
  for (uint32_t f = 0; f < (1u << 23); ++f) {
    const float x = bits(0x3F800000 | f), q = lct::div_by(x, all, 1.0f / all);
    ones += q != x / all;
    ones_far += std::labs((long)ubits(q) - (long)ubits(x / all)) > 1;
  }
  std::printf("%ld %ld %ld %ld\n", bad, bad_view, ones, ones_far);
}
"""


def test_the_kernels_division_is_the_fp32_division(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-I",
                    str(ROOT / "listctrecons_b200" / "csrc"), "-I", "/usr/local/cuda/include",
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout
    bad, bad_view, ones, ones_far = (int(v) for v in out.split())
    assert bad == 0 and bad_view == 0
    assert ones <= 2 and ones_far == 0
