"""The fixed-point exponent of the FP64 sums (csrc/gauss_fx.cuh), compiled for the host:
coordinates, pair exponents and powers of two against long double."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

SOURCE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "gauss_fx.cuh"
using namespace prbf;
static uint2 t1[kFxTab], t2[kFxTab];
static double pow2(unsigned long long B) {
  const unsigned bh = (unsigned)(B >> 32);
  const unsigned long long u = fx_pow2_bits(bh, (unsigned)B, t1[(bh >> 11) & 2047], t2[bh & 2047]);
  double d;
  std::memcpy(&d, &u, 8);
  return d;
}
template <int DIM>
static double worst_pair(std::mt19937_64& g, double sigma, double at, double reach) {
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  const FxScale fs = fx_scale(sigma);
  double worst = 0;
  for (int i = 0; i < 20000; i++) {
    uint2 t[DIM], s[DIM];
    long double d2 = 0;
    const double r = reach * sigma * std::pow(2.0, -30.0 * (i % 7) / 6.0);
    for (int d = 0; d < DIM; d++) {
      const double a = at + sigma * U(g), b = a + r * U(g);
      t[d] = fx_coord(a, fs.hi, fs.lo);
      s[d] = fx_coord(b, fs.hi, fs.lo);
      d2 += ((long double)a - b) * ((long double)a - b);
    }
    const long double ref = expl(-d2 / (2.0L * sigma * sigma));
    const double e = (double)(fabsl(pow2(fx_exponent<DIM>(t, s)) - ref) / ref);
    if (e > worst) worst = e;
  }
  return worst;
}
int main() {
  fx_tables(t1, t2);
  std::mt19937_64 g(7);
  const long double unit = 18014398509481984.0L;
  double sum = 0, sq = 0, mx = 0;
  const int N = 200000;
  for (int i = 0; i < N; i++) {
    const long long B = -(long long)(g() >> 10) - ((long long)(g() % 500) << 54);
    const long double ref = exp2l((long double)B / unit);
    const double e = (double)((pow2((unsigned long long)(kFxBias + B)) - ref) / ref);
    sum += e;
    sq += e * e;
    if (std::fabs(e) > mx) mx = std::fabs(e);
  }
  printf("%.17g %.3g %.3g %.3g\n", pow2((unsigned long long)kFxBias), sum / N, std::sqrt(sq / N), mx);
  const double sig[4] = {0.0125, 1.25e-3, 3.7, 1e-40}, at[4] = {0.3, 1e4, -1e6, 5e-39};
  for (int k = 0; k < 4; k++)
    printf("%.3g %.3g\n", worst_pair<2>(g, sig[k], at[k], 18.6), worst_pair<3>(g, sig[k], at[k], 15.1));
  return 0;
}
"""


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    inc = os.path.join(CUDA, "include")
    if not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("fx")
    src, exe = str(d / "fx.cpp"), str(d / "fx")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", inc, "-I",
                    os.path.join(ROOT, "petrbf_gb300", "csrc"), src, "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split("\n")
    return [[float(v) for v in ln.split()] for ln in out if ln]


def test_powers_of_two(report):
    one, mean, rms, worst = report[0]
    assert one == 1.0  # coincident points
    # truncations: the shifted product and the correction's high word one unit of 2^-52 each,
    # the correction's 2^-54 and its multiplier's 2^-32 of 2^-22 smaller; means compensated
    assert abs(mean) < 0.5 * 2.0 ** -54 and rms < 2.0 ** -53 and worst < 3 * 2.0 ** -52


@pytest.mark.parametrize("case", range(4))
def test_pairs_over_the_whole_reach(report, case):
    # beyond the power's error: the exponent's own truncations, at most one unit of 2^-54 for
    # the shift, one per axis for the squared low parts, and the coordinates' half units of
    # 2^-58 times twice the distance (16 units at most): 2 + 3 + 4 units of ln 2 2^-54
    bound = 3 * 2.0 ** -52 + 9 * 0.6931 * 2.0 ** -54
    assert max(report[1 + case]) < bound
