"""The FP64 sweep's exp (csrc/exp_tang.h) where its method is worst, against
long-double exp on the host: every table node and every point half-way between
two, taken from the header's own table size, and the edges of its flush.

Relative error, at most: the table entry's rounding 2^-53, the last
multiply-add's 2^-53, and the polynomial's remainder r^5/120 at the half-way
point r = ln2/512, 3.8e-17; the rest (the reduced argument, the polynomial's own
roundings, all of them times r) is below 1e-18.  Together 2.61e-16."""
import os
import subprocess

from conftest import PKG

PROG = r"""
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include "exp_tang.h"
int main() {
  double tab[dgbgk::EXP_TAB];
  for (int j = 0; j < dgbgk::EXP_TAB; ++j) tab[j] = (double)exp2l((long double)j / dgbgk::EXP_TAB);
  const long double step = 0.693147180559945309417L / dgbgk::EXP_TAB;
  double worst[2] = {0.0, 0.0}, off[2] = {0.0, 1.0};  // nodes, half-way points; their largest and least distance from a node
  for (long k = (long)(-706.0L / step); k <= 0; ++k)
    for (int h = 0; h < 2; ++h) {
      const double x = (double)((k + 0.5L * h) * step);
      if (x > 0.0) continue;
      const long double q = x / step, d = fabsl(q - rintl(q)), ref = expl((long double)x);
      off[h] = h ? fmin(off[h], (double)d) : fmax(off[h], (double)d);
      worst[h] = fmax(worst[h], (double)fabsl(((long double)dgbgk::exp_tang(x, tab) - ref) / ref));
    }
  auto zero = [&](double x) { const double y = dgbgk::exp_tang(x, tab); return y == 0.0 && !std::signbit(y); };
  const double above = std::nextafter(-707.0, 0.0);
  const double up = std::fabs(dgbgk::exp_tang(above, tab) / (double)expl((long double)above) - 1.0);
  const double nan = std::nan("");
  int nans = 0;
  for (double x : {nan, -nan, std::copysign(nan, -1.0), std::copysign(nan, 1.0)}) nans += std::isnan(dgbgk::exp_tang(x, tab));
  printf("%.4e %.4e %.3f %.3f %.3e %d %d\n", worst[0], worst[1], off[0], off[1], up, nans,
         zero(-707.0) && zero(std::nextafter(-707.0, -708.0)) && zero(-745.0) && zero(-1e6) && zero(-1e308) &&
             zero(-INFINITY));
  return 0;
}
"""


def test_nodes_half_way_points_and_the_flush(tmp_path):
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROG)
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(PKG, "csrc"), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120).stdout.split()
    node, half, at_node, at_half, edge = map(float, out[:5])
    # the points are what they are said to be
    assert at_node < 1e-3 and at_half > 0.499
    assert node <= 2.61e-16 and half <= 2.61e-16, out
    assert edge <= 2.61e-16 and out[5:] == ["4", "1"], out
