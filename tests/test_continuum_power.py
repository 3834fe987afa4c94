"""The power of the water vapour self continuum, r^((296 - T) / 36) from the
logarithm of r in two doubles (jgb_common.cuh), compiled for the host: within 2
units in the last place of the power in long double, over the ratios of the
continuum's table and 100 to 400 K."""
import os
import subprocess

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "jgb_common.cuh"
int main() {
  double worst = 0, worst_plain = 0;
  for (int i = 0; i <= 400; i++) {
    const double r = std::exp(-1.0 + 3.0 * i / 400);
    double hi, lo;
    jgb::log_parts(r, &hi, &lo);
    for (int k = 0; k <= 300; k++) {
      const double t = 100.0 + k + 0.37, x = (296 - t) / (296 - 260);
      const long double e = std::pow((long double)r, (long double)x);
      const long double ulp = std::nextafter((double)e, 1e300) - (double)e;
      const double a = (double)(std::fabs((long double)jgb::pow_of_log(hi, lo, x) - e) / ulp);
      const double b = (double)(std::fabs((long double)std::exp(std::log(r) * x) - e) / ulp);
      if (a > worst) worst = a;
      if (b > worst_plain) worst_plain = b;
    }
  }
  printf("%.4f %.4f\n", worst, worst_plain);
  return 0;
}
"""


def test_power_from_two_part_logarithm(tmp_path):
    from jurassic_gb300 import build
    src = tmp_path / "p.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "p"
    flags = [f for f in build.COMMON if f != "-lineinfo"]
    subprocess.run([build.nvcc()] + flags + [str(src), "-o", str(exe)], check=True)
    worst, plain = map(float, subprocess.run([str(exe)], check=True, capture_output=True,
                                             text=True).stdout.split())
    assert np.isfinite(worst) and worst <= 2.0
    assert plain > 2.0  # what one double of the logarithm gives
