"""DivBy (csrc/clb_div.h): division by the lattice spacing or its square through a stored reciprocal
gives the bits of the division, for spacings and squares over the range in use and for numerators
near every rounding boundary (quotients half-way between two doubles, and one ulp either side)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "clb_div.h"
#include <cstdint>
#include <cstdio>
#include <cstring>
static uint64_t st;
static uint64_t next() { uint64_t z = (st += 0x9e3779b97f4a7c15ull); z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull; return z ^ (z >> 31); }
static double bits(uint64_t m, int e) { uint64_t u = ((uint64_t)(1023 + e) << 52) | (m >> 12); double d; std::memcpy(&d, &u, 8); return d; }
int main()
{
  st = SEED;
  long bad = 0, n = 0;
  auto check = [&](double x, const clb::DivBy &d, double y) {
    const double a = clb::div_by(x, d), b = x / y;
    ++n;
    if (std::memcmp(&a, &b, 8) && !(a == 0 && b == 0) && bad++ < 5) std::printf("%a / %a: %a, not %a\n", x, y, a, b);
  };
  for (int k = 0; k < 400; ++k) {
    double y = k < 100 ? 6.283185307179586 / (8 + 5 * k) : bits(next(), (int)(next() % 24) - 18);
    if (k % 2) y = y * y;
    const clb::DivBy d = clb::make_div(y, (float)y);
    check(0.0, d, y);
    for (int i = 0; i < 5000; ++i) {
      const double x = bits(next(), (int)(next() % 400) - 200);
      check(i % 2 ? x : -x, d, y);
      // numerators whose quotient lies next to a half-way point between two doubles
      const double q = bits(next(), (int)(next() % 40) - 20), h = q + std::ldexp(q, -53);
      const double xh = std::fma(q, y, 0.5 * (std::nextafter(q, 1e300) - q) * y);
      check(xh, d, y);
      check(std::nextafter(xh, 1e300), d, y);
      check(std::nextafter(xh, -1e300), d, y);
      check(h * y, d, y);
    }
  }
  std::printf("%ld of %ld differ\n", bad, n);
  return bad != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host C++ compiler")
@pytest.mark.parametrize("seed", [1, 2026])
def test_div_by_gives_the_quotient_bits(tmp_path, seed):
    src = tmp_path / "t.cpp"
    src.write_text(SRC.replace("SEED", f"{seed}ull"))
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT}/cosmolattice_b200/csrc", str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
