"""csrc/quotient.h against IEEE division on the CPU: equal over the range that it
states, a unit in the last place outside it."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GXX = shutil.which("g++")
pytestmark = pytest.mark.skipif(GXX is None, reason="no C++ compiler")

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "quotient.h"
static float bits(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static uint32_t word(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static long long places(float a, float b) {  // units in the last place between a and b
  auto key = [](float f) { const int32_t i = (int32_t)word(f); return i < 0 ? -(long long)(i & 0x7fffffff) : (long long)i; };
  return std::llabs(key(a) - key(b));
}
static int check(float v, float d, long long most) {
  const float inv = 1.0f / d, want = v / d, got = divided(v, d, inv);
  if (want != want ? got != got : places(want, got) <= most) return 0;
  std::printf("%a / %a: %a, not %a\n", v, d, got, want);
  return 1;
}
int main() {
  std::mt19937_64 rng(7);
  // every significand by the divisors of a few levels and lambdas
  for (int level : {0, 1, 5, 14})
    for (float lambda : {0.003f, 0.01f, 1.0f, 1234.5f, 6.7e7f}) {
      const float d = 4.0f * std::ldexp(1.0f, -2 * level) + lambda;
      for (uint32_t m = 0; m < (1u << 23); ++m)
        if (check(bits((127u << 23) | m), d, 0)) return 1;
    }
  for (long k = 0; k < 20000000; ++k) {
    const uint64_t a = rng(), b = rng();
    const float sign = a >> 63 ? -1.0f : 1.0f;
    // the stated range: d in 2^-28 .. 2^26, |v| in 2^-100 .. 2^99
    const float d = std::ldexp(1.0f + (float)(b & 0x7fffff) * 0x1p-23f, (int)((b >> 32) % 54) - 28);
    const float v = sign * std::ldexp(1.0f + (float)(a & 0x7fffff) * 0x1p-23f, (int)((a >> 32) % 200) - 100);
    if (check(v, d, 0)) return 1;
    // any finite v, subnormal ones too, by any normal d
    const float any = sign * bits((uint32_t)(a & 0x7fffffff) % 0x7f800000u), wide = bits((uint32_t)((b % 0x7f000000u) + 0x00800000u));
    if (check(any, wide, 1)) return 1;
  }
  for (float d : {0x1p-28f, 0.04f, 4.0f, 0x1.8p126f, FLT_MAX, INFINITY})
    for (float v : {0.0f, -0.0f, INFINITY, -INFINITY, NAN, 1.0f, -FLT_MAX, 0x1p-149f, 0x1p-100f})
      if (check(v, d, 1)) return 1;
  return 0;
}
"""


def test_quotient_equals_division_over_its_range(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    r = subprocess.run([GXX, "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "paintop_b200", "csrc"),
                        str(src), "-o", str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
