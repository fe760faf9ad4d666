"""The widest windows that the fixed-point exponents take (csrc/gauss_fx.cuh, fx_grid_ok,
compiled for the host): pairs at the corners of the reach that the rule allows, where the sums of
products are largest, against long double."""
import os
import subprocess

import pytest

from conftest import ROOT

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "gauss_fx.cuh"
using namespace prbf;
static uint2 t1[kFxTab], t2[kFxTab];
static Grid grid(int dim, double sigma, double box, double trunc) {  // widths in sigma
  Grid g{};
  g.dim = dim;
  g.sigma = sigma;
  g.nx = g.ny = g.nz = 100;
  g.xmin = g.ymin = g.zmin = -1.0;
  g.box = box * sigma;
  g.trunc_len = trunc * sigma / 2;
  return g;
}
// WIDE: the widest truncation box that the rule takes; else the widest that is not wide
template <int DIM, bool WIDE>
static void corners(double sigma, double box) {
  double lo = 0, hi = 60;
  for (int i = 0; i < 60; i++) {
    const double mid = 0.5 * (lo + hi);
    const Grid g = grid(DIM, sigma, box, mid);
    (fx_grid_ok(g) && (WIDE || !fx_grid_wide(g)) ? lo : hi) = mid;
  }
  const double reach = 0.5 * (std::fmax(lo, box) + box) * sigma;
  const FxScale fs = fx_scale(sigma);
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(0, 1);
  double worst = 0;
  for (int i = 0; i < 400000; i++) {
    uint2 t[DIM], s[DIM];
    long double d2 = 0;
    for (int d = 0; d < DIM; d++) {
      const double a = 0.3 + 10 * sigma * U(g);
      const double b = a + (g() & 1 ? 1 : -1) * reach * (1.0 - (i % 3 ? 0.02 : 1.0) * U(g));
      t[d] = fx_coord(a, fs.hi, fs.lo);
      s[d] = fx_coord(b, fs.hi, fs.lo);
      d2 += ((long double)a - b) * ((long double)a - b);
    }
    const long double ref = expl(-d2 / (2.0L * sigma * sigma));
    const unsigned long long B = WIDE ? fx_exponent<DIM, true>(t, s) : fx_exponent<DIM>(t, s);
    const unsigned bh = (unsigned)(B >> 32);
    const unsigned long long u = fx_pow2_bits(bh, (unsigned)B, t1[(bh >> 11) & 2047], t2[bh & 2047]);
    double v;
    std::memcpy(&v, &u, 8);
    const double e = (double)(fabsl(v - ref) / ref);
    if (e > worst) worst = e;
  }
  printf("%.4g %.4g\n", reach / sigma, worst);
}
int main() {
  fx_tables(t1, t2);
  for (double box : {1.0, 3.0, 8.0}) {
    corners<2, false>(0.0125, box);
    corners<3, false>(0.026, box);
    corners<3, true>(0.026, box);
  }
  return 0;
}
"""


def test_corners_of_the_widest_windows(tmp_path):
    inc = os.path.join(CUDA, "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    src, exe = str(tmp_path / "reach.cpp"), str(tmp_path / "reach")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", inc, "-I",
                    os.path.join(ROOT, "petrbf_gb300", "csrc"), src, "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")
    rows = [[float(v) for v in ln.split()] for ln in out if ln]
    assert len(rows) == 9
    for k, (reach, worst) in enumerate(rows):
        assert reach > (18, 12, 15)[k % 3]  # sigma per axis: 2D, 3D, 3D wide
        # as for nearer pairs: the power's error, one unit of 2^-54 for the shift and for each
        # axis' squared low parts, the coordinates' half units of 2^-58 times twice the distance
        assert worst <= 3 * 2.0 ** -52 + 9 * 0.6931 * 2.0 ** -54
