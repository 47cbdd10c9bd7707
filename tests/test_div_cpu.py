"""The quotients of the 2-D step (csrc/lbm_div.h) against the division, compiled for the host: the same value for
zeros, infinities, NaN and overflow and wherever the remainder is representable, within an ulp below that.  Quotients by
cs2: every float mantissa (one of them, next to a tie, an ulp off), many double ones."""
import os
import shutil
import subprocess

import pytest

PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include "lbm_div.h"
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
template <typename T> T value(int e) { return std::ldexp((T)(1.0 + (double)(rnd() >> 12) / 4503599627370496.0), e) * ((rnd() & 1) ? 1 : -1); }
template <typename T> bool same(T a, T b) { return a == b || (a != a && b != b); }
template <typename T> int run(int lo, int hi, int emin) {
  using L = std::numeric_limits<T>;
  const T inf = L::infinity(), nan = L::quiet_NaN();
  const T ds[] = {(T)(1.0 / 3.0), (T)(2.0 / 3.0), 5, 1, (T)1e-3, (T)1e-10, inf, 0, nan};
  const T xs[] = {0, -(T)0, 1, -1, inf, -inf, nan, L::max(), -L::max()};
  int bad = 0;
  for (T d : ds)
    for (T x : xs) {
      const lbm::Div<T> by{d, (T)1 / d};
      if (!same(by(x), x / d) && ++bad < 9) std::printf("x %g d %g: %g, not %g\n", (double)x, (double)d, (double)by(x), (double)(x / d));
    }
  for (int i = 0; i < 2000000; ++i) {
    const T d = i & 1 ? ds[i / 2 % 6] : value<T>((int)(rnd() % 40) - 20);
    const T x = value<T>((int)(rnd() % (hi - lo)) + lo);
    const lbm::Div<T> by{d, (T)1 / d};
    if (!(by(x) == x / d) && ++bad < 9) std::printf("x %a d %a: %a, not %a\n", (double)x, (double)d, (double)by(x), (double)(x / d));
  }
  for (int i = 0; i < 200000; ++i) {
    const T d = value<T>((int)(rnd() % 40) - 20), x = value<T>((int)(rnd() % (lo - emin)) + emin), t = x / d;
    const lbm::Div<T> by{d, (T)1 / d};
    const T ulp = std::nextafter(std::fabs(t), inf) - std::fabs(t);
    if (!(std::fabs(by(x) - t) <= ulp) && ++bad < 9) std::printf("x %a d %a: %a, not %a\n", (double)x, (double)d, (double)by(x), (double)t);
  }
  return bad;
}
template <typename T> bool cs2_special() {
  using L = std::numeric_limits<T>;
  const T inf = L::infinity(), d = lbm::ByCs2<T>::d;
  const T xs[] = {0, -(T)0, 1, -1, inf, -inf, L::quiet_NaN(), L::max(), -L::max()};
  bool ok = true;
  for (T x : xs) ok = ok && same(lbm::by_cs2<T>()(x), x / d) && same(lbm::by_two_cs2<T>()(x), x / (2 * d));
  for (int i = 0; i < 100000; ++i) {
    const T x = value<T>(L::min_exponent - (int)(rnd() % 20)), t = x / d;
    ok = ok && std::fabs(lbm::by_cs2<T>()(x) - t) <= std::nextafter(std::fabs(t), inf) - std::fabs(t);
  }
  return ok;
}
int cs2() {
  int bad = 0, off = 0;
  for (uint32_t m = 0; m < (1u << 23); ++m) {
    const uint32_t b = 0x3f800000u | m;
    float x;
    std::memcpy(&x, &b, 4);
    for (int two = 0; two < 2; ++two) {
      const float t = x / (lbm::ByCs2<float>::d * (two ? 2 : 1));
      const float e = two ? lbm::by_two_cs2<float>()(x) : lbm::by_cs2<float>()(x);
      if (e != t) (std::fabs(e - t) <= std::nextafter(t, 9.0f) - t && x == 0x1.555554p0f ? off : bad)++;
    }
  }
  for (int i = 0; i < 20000000; ++i) {
    const double x = value<double>((int)(rnd() % 200) - 100);
    if (lbm::by_cs2<double>()(x) != x / lbm::ByCs2<double>::d) ++bad;
  }
  if (bad || off != 2 || !cs2_special<float>() || !cs2_special<double>()) std::printf("cs2: bad %d off %d\n", bad, off), ++bad;
  return bad;
}
int main() {
  const int bad = cs2() + run<float>(-100, 90, -149) + run<double>(-900, 900, -1074);
  std::printf("%d\n", bad);
  return bad != 0;
}
"""


def test_quotients_match_the_division(tmp_path):
    cxx = os.environ.get("CXX", "g++")
    if not shutil.which(cxx):
        pytest.skip("no host compiler")
    from lbm._build import CSRC
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "0", r.stdout
