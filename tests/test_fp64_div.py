"""div_by (the Crank-Nicolson back substitution's quotients) against the
division, bit for bit, and rcp_newton (the direct solve's reciprocals) within
a unit in the last place from every approximation that it is made for;
csrc/fp64_div.h compiled for the host, whose double arithmetic and fma round
as the GPU's."""
import subprocess

from .conftest import ROOT

MAIN = r"""
#include "fp64_div.h"
#include <cstdint>
#include <cstdio>
using namespace anel;
static uint64_t seed = 12345;
static uint64_t next() {  // splitmix64
  uint64_t z = (seed += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}
static double of(uint64_t u) { double d; std::memcpy(&d, &u, 8); return d; }
static uint64_t bits(double d) { uint64_t u; std::memcpy(&u, &d, 8); return u; }
// mantissas: random, a few bits from the top or the bottom, all ones but a few
static uint64_t mantissa() {
  const uint64_t r = next(), m = (1ull << 52) - 1, few = next() & 7;
  switch (next() & 3) {
    case 0: return few << (next() % 50) & m;
    case 1: return ~(few << (next() % 50)) & m;
    default: return r & m;
  }
}
static double number(int lo, int hi) {
  return of((next() & 1) << 63 | (uint64_t)(lo + next() % (hi - lo + 1)) << 52 | mantissa());
}
int main() {
  long bad = 0;
  auto check = [&](double a, double b) {
    const double q = div_by(a, b, div_reciprocal(b)), w = a / b;
    if (bits(q) != bits(w) && !(q != q && w != w) && bad++ < 5) std::printf("div %a / %a: %a, not %a\n", a, b, q, w);
  };
  for (int t = 0; t < 6000000; ++t) {
    check(number(1023 - 60, 1023 + 60), number(1023 - 30, 1023 + 30));
    check(number(0, 2047), number(0, 2047));       // zeros, subnormals, infinities and NaN among them
    check(number(150, 350), number(900, 1150));    // around the ends of the ranges
    check(number(1700, 2046), number(900, 1150));
  }
  const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -5e-324, 2.2250738585072014e-308,
                            1.7976931348623157e308, 1.0, -1.0, 1e-30, 1e30};
  for (double a : special)
    for (double b : special) check(a, b);
  for (int t = 0; t < 6000000; ++t) {
    const double x = number(1023 - 900, 1023 + 900), w = 1.0 / x;
    // off by up to 2^-17, its low word zero as the hardware's
    const double y0 = of(bits(w * (1.0 + std::ldexp((double)(int64_t)next(), -63 - 17) * 0.99)) & ~0xffffffffull);
    const double y = rcp_newton(x, y0);
    const int64_t d = (int64_t)(bits(y) - bits(w));
    if ((d > 1 || d < -1) && bad++ < 10) std::printf("1 / %a from %a: %a, not %a\n", x, y0, y, w);
  }
  std::printf("%ld wrong\n", bad);
  return bad != 0;
}
"""


def test_against_the_division(tmp_path):
    src, exe = tmp_path / "main.cc", tmp_path / "main"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-Wall", "-Werror",
                    f"-I{ROOT / 'anelastic_solve_b200' / 'csrc'}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout
