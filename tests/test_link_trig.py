"""sincos_link (csrc/clb_trig.h) against 80-bit sines and cosines: within 0.55 of the last place where
the polynomials are taken (their truncation is below 0.03, the final rounding 0.5), on both sides of
the change to the library's functions, for FP64 and FP32."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "clb_trig.h"
#include <cstdio>
#include <random>
template <class T> static double err(T got, long double want)
{
  const T w = (T)want;
  const T up = std::nextafter(std::fabs(w), (T)10) - std::fabs(w), dn = std::fabs(w) - std::nextafter(std::fabs(w), (T)0);
  const long double ulp = std::fabs(want) < (long double)std::fabs(w) ? dn : up;
  return (double)(std::fabs((long double)got - want) / ulp);
}
template <class T> static double worst(double lo, double hi)
{
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> u(std::log(lo), std::log(hi));
  double e = 0;
  for (int i = 0; i < 300000; ++i) {
    const T x = (T)(std::exp(u(g)) * (i % 2 ? 1 : -1));
    T s, c;
    clb::sincos_link(x, &s, &c);
    e = std::fmax(e, std::fmax(err<T>(s, sinl((long double)x)), err<T>(c, cosl((long double)x))));
  }
  return e;
}
int main()
{
  const double k = clb::kSmallPhase;
  double s, c;
  clb::sincos_link(0.0, &s, &c);
  if (s != 0 || c != 1) return 1;
  std::printf("%.4f %.4f %.4f %.4f\n", worst<double>(1e-12, k), worst<float>(1e-8, k), worst<double>(k, 4.0), worst<float>(k, 4.0));
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host C++ compiler")
def test_sincos_link_is_rounded_correctly(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(SRC)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{ROOT}/cosmolattice_b200/csrc", str(src), "-o",
                    str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
    small64, small32, large64, large32 = map(float, r.stdout.split())
    assert small64 < 0.55 and small32 < 0.55, r.stdout
    assert large64 < 1.0 and large32 < 1.0, r.stdout  # the host library's own
