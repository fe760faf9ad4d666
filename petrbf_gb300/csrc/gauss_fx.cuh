// gauss_fx.cuh -- the FP64 Gaussian of the sums in fixed point on the integer pipe.
//
// GB300's FP64 pipe takes a warp instruction every 16 clocks per SM (measured; integer adds,
// shifts, logic and 32-bit multiply-adds 0.5, 32 x 32 -> 64-bit ones about 1.2), so the ten
// FP64 instructions a pair's exponential costs there (160 clocks) are replaced by some thirty
// integer ones and the FP64 pipe keeps only the accumulations.
//
// Coordinates: X = x sqrt(1 / (2 sigma^2 ln 2)) 2^58, rounded to an integer and kept modulo
// 2^63 as a high word h (32 bits) and a low part l (31 bits). A difference of two points'
// coordinates is exact, d = dh + dl 2^-31 with dh, dl one 32-bit subtraction each, as long as
// it stays below 2^31 in dh (16 units of the scaled coordinate: 18.8 sigma).
// Exponent: a = |d|^2 in units of 2^-54 of ln 2,
//   A = sum dh^2 + (sum dh dl >> 30)        (the dl^2 term is below one unit per axis),
// so the Gaussian is 2^(B 2^-54), B = -A: an integer part n = B >> 54 and a fraction of 11 +
// 11 + 32 bits (j1, j2, r):
//   2^(j1 / 2^11) = u 2^-31 (1 + e1 2^-54),  2^(j2 / 2^22) = t 2^-31 (1 + e2 2^-54),
//   2^(r / 2^54)  = 1 + r (c1 + c2 r) 2^-54,
// u and t integers of 32 bits whose rounding errors e1 and e2 go into the last factor: with
// V = u t (64 bits, one multiplication) and P = r (c1 + c2 r) + e1 + e2 the mantissa is
// (V + V P 2^-54) 2^-10. The shift of V and the product are centred by half a unit each, the
// smaller truncations by e2, such that the zero exponent still gives exactly 1.
// Against 64-bit-mantissa exponentials of 4x10^6 random arguments below 1, 10 and 50: mean error
// -6.6e-18, -7.6e-18, -7.8e-18; rms 7.6e-17, 7.9e-17, 7.9e-17; largest 4.1e-16. (The 1024-entry
// table and cubic on the FP64 pipe, where the rounding of its exponent factor, sigma's, grows in;
// over five widths: mean up to 5.3e-17, 5.8e-16, 2.9e-15; rms 7.8e-17 to 1.0e-16, 9.9e-17 to
// 6.7e-16, 3.2e-16 to 3.4e-15; largest 2.9e-16 to 3.6e-16, 3.8e-16 to 1.4e-15, 7.9e-16 to 6.1e-15.)
// Keeping the bits that the shift drops (one 32 x 32 -> 64-bit product and two instructions more)
// gives rms 6.1e-17 and largest 3.1e-16, and costs the 3D sum 5 %.
#pragma once
#include <cmath>

#include "common.cuh"

namespace prbf {

constexpr int kFxTab = 2048;  // entries of each table: (u, e1) and (t, e2)

// The exponent field's offset, kept in A from the start: fx_pow2 takes B = kFxBias - a, whose
// top ten bits are then the biased exponent of the mantissa's leading bit.
constexpr long long kFxBias = -(2ll << 54);

__host__ __device__ __forceinline__ unsigned fx_mulhi(unsigned a, unsigned b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (unsigned)(((unsigned long long)a * b) >> 32);
#endif
}

// 2^((B - kFxBias) 2^-54) as an FP64 number's bits, from B's words and the entries (u, e1) of
// the bits 21..11 and (t, e2) of the bits 10..0 of its high one.
__host__ __device__ __forceinline__ unsigned long long fx_pow2_bits(unsigned bh, unsigned r, uint2 p, uint2 q) {
  // c1 = ln2 2^32, c2 = ln2^2 / 2 2^10; e's product with r c1 (up to 2^32) reaches three units
  const unsigned e = p.y + q.y, c = fx_mulhi(r, 246u) + (2977044472u + (e >> 22));
  const unsigned P = fx_mulhi(r, c) + e;
  const unsigned long long V = (unsigned long long)p.x * q.x + 1024u;  // half a unit for each of
  const unsigned X = fx_mulhi((unsigned)(V >> 32), P);                 // these two truncations
  // V's leading bit (62) lands on the exponent field's lowest
  return (V >> 10) + X + ((unsigned long long)((bh >> 2) & 0x3ff00000u) << 32);
}

// B of a pair: coordinates (l, h) of target and source. WIDE (fx_grid_wide): the last axis' low
// product by itself, where the sum of all three could pass 63 bits.
template <int DIM, bool WIDE = false>
__host__ __device__ __forceinline__ unsigned long long fx_exponent(const uint2 (&t)[DIM], const uint2 (&s)[DIM]) {
  long long A = -kFxBias, C = 0;  // C carries the minus sign of B
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int d = 0; d < DIM; d++) {
    const int dh = (int)(t[d].y - s[d].y), dl = (int)(s[d].x - t[d].x);
    A += (long long)dh * dh;
    if (WIDE && d == DIM - 1)
      A -= (long long)dh * dl >> 30;
    else
      C += (long long)dh * dl;
  }
  return (unsigned long long)((C >> 30) - A);
}

// A point's scaled coordinate as (l, h): x * (shi + slo) 2^58-scaled, modulo 2^63.
__host__ __device__ __forceinline__ uint2 fx_coord(double x, double shi, double slo) {
  const double two63 = 9223372036854775808.0;
  const double p = x * shi;
  const double e = fma(x, slo, fma(x, shi, -p));  // what p rounds away, to about 2^-52 of it
  const double q = fma(-rint(p * (1.0 / two63)), two63, p);  // exact, |q| <= 2^62
  const double i = rint(q);
  const long long X = (long long)i + (long long)rint((q - i) + e);
  uint2 o;
  o.x = (unsigned)X & 0x7fffffffu;
  o.y = (unsigned)((unsigned long long)X >> 31);
  return o;
}

// sqrt(1 / (2 sigma^2 ln 2)) 2^58 as an unevaluated sum hi + lo.
struct FxScale {
  double hi, lo;
};

__host__ __device__ inline FxScale fx_scale(double sigma) {
  const double l1 = 0.6931471805599453, l2 = 2.3190468138462996e-17;  // ln 2 to 107 bits
  const double s1 = sigma * sigma, s2 = fma(sigma, sigma, -s1);
  const double v1 = 2 * (s1 * l1), v2 = 2 * (fma(s1, l1, -s1 * l1) + s1 * l2 + s2 * l1);
  const double y = 1.0 / sqrt(v1);
  const double p1 = y * y, p2 = fma(y, y, -p1);
  const double t1 = p1 * v1, t2 = fma(p1, v1, -t1);
  const double res = ((1.0 - t1) - t2) - (p1 * v2 + p2 * v1);  // 1 - y^2 v
  const double two58 = 288230376151711744.0;
  return FxScale{y * two58, 0.5 * y * res * two58};
}

// 1 / (2 pi sigma^2) rounded once (to within 2^-54 of its last place): the products and sums that
// it is multiplied with carry less than the two units that rounding each of its operations would
// put into every result alike.
inline double gauss_norm(double sigma) {
  const double plain = 1.0 / (2 * 3.141592653589793 * sigma * sigma);
  if (!(sigma > 1e-100 && sigma < 1e100)) return plain;
  const double p1 = 6.283185307179586, p2 = 2.4492935982947064e-16;  // 2 pi to 107 bits
  const double s1 = sigma * sigma, s2 = std::fma(sigma, sigma, -s1);
  const double q1 = s1 * p1, q2 = std::fma(s1, p1, -q1) + (s1 * p2 + s2 * p1);
  const double n = 1.0 / q1;
  return std::fma(n, std::fma(-n, q1, 1.0) - n * q2, n);
}

// The tables, in long double. The truncations in P drop one unit of 2^-54 on average, which e2
// gets. A zero exponent gives exactly 1: u(0) is one less than 2^31 and P = 2^23 makes up for it,
// V >> 10 = 2^52 - 2^21 + 1 and X = 2^21 - 1 (the entry of j1 = 0 is a unit low for that).
inline void fx_tables(uint2* t1, uint2* t2) {
  const long double unit = 18014398509481984.0L, one = 2147483648.0L;  // 2^54, 2^31
  for (int j = 0; j < kFxTab; j++) {
    const long double v = exp2l((long double)j / kFxTab) * one, u = j ? floorl(v) : one - 1.0L;
    t1[j].x = (unsigned)u;
    t1[j].y = j ? (unsigned)llrintl((v - u) / u * unit) : (1u << 23) - 1u;
    const long double x = expm1l((long double)j / 4194304.0L * logl(2.0L)) * one, t = floorl(x);
    t2[j].x = 2147483648u + (unsigned)t;
    t2[j].y = (unsigned)llrintl((x - t) / (one + t) * unit) + 1u;
  }
}

// The largest difference per axis, in units of the scaled coordinate, of a target and a source of
// its truncation set (or of its own cell).
inline double fx_reach(const Grid& g) {
  const double unit = std::sqrt(1.0 / (2.0 * g.sigma * g.sigma * 0.6931471805599453));
  const double half = 0.5 * g.box, reach = (g.trunc_len > half ? g.trunc_len : half) + half;
  return reach * unit;
}

// Whether the low products' sum could pass 63 bits: dh dl is below 2^58 a unit of difference, and
// the axes together reach 32 units (3D windows beyond 12.4 sigma per axis).
inline bool fx_grid_wide(const Grid& g) { return !(g.dim * fx_reach(g) < 0.99 * 32.0); }

// Whether a grid's sums can take the fixed-point form: the pairs differ by less than 16 units per
// axis and a stays below 512, the scaled coordinates stay below 2^40 units (their products keep
// 2^-8 of the last place), and sigma is far from the ends of FP64's range.
inline bool fx_grid_ok(const Grid& g) {
  if (!(g.sigma > 1e-100 && g.sigma < 1e100)) return false;
  const double unit = std::sqrt(1.0 / (2.0 * g.sigma * g.sigma * 0.6931471805599453)), d = fx_reach(g);
  if (!(d < 0.99 * 16.0 && g.dim * d * d < 0.98 * 512.0)) return false;
  const double lo[3] = {g.xmin, g.ymin, g.zmin};
  const int nc[3] = {g.nx, g.ny, g.nz};
  for (int k = 0; k < g.dim; k++) {
    const double far = std::fmax(std::fabs(lo[k]), std::fabs(lo[k] + nc[k] * g.box));
    if (!(far * unit < 1099511627776.0)) return false;
  }
  return true;
}

}  // namespace prbf
