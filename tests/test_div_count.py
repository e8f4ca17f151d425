"""The quotient of the serial schemes' pipeline (div_count in
fluid_gb300/csrc/k_lexsor.cu): x / n for n = 1..4 from the rounded reciprocal
and one correction step must be the correctly rounded division for every
float.  The same operations compiled for the host (fmaf) against its division:
by default both signs of every significand for n = 3 (of each 61st for the
powers of two) among the subnormals, the smallest and largest normals and in
between, infinities and NaN; with FLUID_ALL_FLOATS=1 all 2^32 floats."""
import os
import shutil
import subprocess

import pytest

SRC = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
static float of(uint32_t b) { float x; memcpy(&x, &b, 4); return x; }
static uint32_t bits(float x) { uint32_t b; memcpy(&b, &x, 4); return b; }
static float div_count(float x, float n, float r) {
  float q = x * r;
  const float e = fmaf(n, q, -x);
  if (fabsf(x) < INFINITY) q = fmaf(e, -r, q);
  return q;
}
int main(int argc, char** argv) {
  const bool all = argc > 1;
  const unsigned some[] = {0, 1, 127, 254, 255};
  unsigned long long bad = 0, seen = 0;
  for (int k = 1; k <= 4; ++k) {
    volatile float n = (float)k, one = 1.0f;
    const float r = one / n;
    for (unsigned ex = 0; ex < 256; ++ex) {
      bool in = all;
      for (unsigned s : some) in = in || s == ex;
      if (!in) continue;
      for (uint32_t sign = 0; sign < 2; ++sign)
        for (uint32_t m = 0; m < (1u << 23); m += all || k == 3 ? 1 : 61) {
          const float x = of(sign << 31 | ex << 23 | m), want = x / n, got = div_count(x, n, r);
          ++seen;
          bad += std::isnan(want) ? !std::isnan(got) : bits(want) != bits(got);
        }
    }
  }
  printf("%llu %llu\n", seen, bad);
}
"""


def test_quotient_is_the_division(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src = tmp_path / "q.cpp"
    src.write_text(SRC)
    exe = tmp_path / "q"
    # (fmaf in hardware where the machine has it, else the library's: both exact.)
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", str(src), "-o",
                    str(exe)], check=True, capture_output=True)
    everything = ["all"] if os.environ.get("FLUID_ALL_FLOATS") else []
    out = subprocess.run([str(exe)] + everything, check=True, capture_output=True, text=True,
                         timeout=3000).stdout.split()
    assert int(out[0]) >= 5 * 2 ** 24 and int(out[1]) == 0, out
