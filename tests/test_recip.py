"""The reciprocal of the factorisation's pivots (csrc/topx_recip.h) on the host, against long double.

The device starts from an approximation that keeps 20 bits and refines it with recip_series.  Its remainder is the
fourth power of the approximation's error, 2^-80, so what is left is the rounding of the last operation: at most 2^-53
relative, 1.0001 times that with the remainder and the long double's own rounding.  The same holds for two
Newton-Raphson steps; a series that stops at the second power leaves 1.006.
"""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "top3d_xl_b200", "csrc")

PROGRAM = r"""
#include "topx_recip.h"
#include <cstdint>
#include <cstdio>
#include <random>
int main() {
  std::mt19937_64 g(1);
  double worst = 0.0;
  for (int i = 0; i < 4000000; ++i) {
    // all mantissas, magnitudes over the pivots' range, both signs; the approximation's error up to 2^-20
    const double m = 1.0 + std::ldexp(double(g() >> 12), -52);
    const double v = std::ldexp(g() & 1 ? -m : m, int(g() % 121) - 60);
    const double t = double(int64_t(g()) >> 10) / double(int64_t(1) << 53);
    const double x = (1.0 / v) * (1.0 + t * std::ldexp(1.0, -20));
    const long double exact = 1.0L / v;
    const double e = double(std::fabs((topx::recip_series(v, x) - exact) / exact)) * std::ldexp(1.0, 53);
    if (!(e <= worst)) worst = e;
  }
  std::printf("%.9f\n", worst);
}
"""


def test_reciprocal_is_as_close_as_one_rounding(tmp_path):
    src, exe = tmp_path / "recip.cpp", tmp_path / "recip"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    worst = float(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout)
    assert 0.9 < worst <= 1.0001
