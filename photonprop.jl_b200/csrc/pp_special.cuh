// FP64 digamma and trigamma for the device: a shift to x >= 6, then the
// asymptotic series
//   psi(x)  = ln x - 1/(2x) - sum_k B_2k / (2k x^2k)
//   psi'(x) = 1/x + 1/(2x^2) + sum_k B_2k / x^(2k+1)
// (Bernoulli numbers to B_10, B_8 for the second): within 1e-11 and 3e-10
// (absolute, at x = 6; largest seen 8.8e-12 and 1.9e-10), less above.
#pragma once

namespace ppsf {

// psi(x) and psi'(x) together, x > 0, with one reciprocal for the recurrence:
// below 6 the argument is shifted by 6, whose six terms pair up with
// q = x (x + 5), q + 4 = (x + 1)(x + 4), q + 6 = (x + 2)(x + 3):
//   sum 1/(x+k)   = (2x + 5) (1/q + 1/(q+4) + 1/(q+6))
//   sum 1/(x+k)^2 = (2q + 25)/q^2 + (2q + 17)/(q+4)^2 + (2q + 13)/(q+6)^2
// (all terms positive), then the series above.
__device__ __forceinline__ void psi_both(double x, double& psi, double& psi1) {
  const bool low = x < 6.0;
  const double q = x * (x + 5.0), q4 = q + 4.0, q6 = q + 6.0;
  const double y = low ? x + 6.0 : x, d = low ? q * q4 * q6 : 1.0;
  const double both = 1.0 / (d * y), rd = both * y, r = both * d, f = r * r;
  const double u = q4 * q6 * rd, v = q * q6 * rd, w = q * q4 * rd;
  const double s0 = low ? fma(2.0, x, 5.0) * (u + v + w) : 0.0;
  const double s1 = low ? fma(2.0, q, 25.0) * u * u + fma(2.0, q, 17.0) * v * v + fma(2.0, q, 13.0) * w * w : 0.0;
  psi = log(y) - 0.5 * r - f * (1.0 / 12 - f * (1.0 / 120 - f * (1.0 / 252 - f * (1.0 / 240 - f / 132)))) - s0;
  psi1 = s1 + r + 0.5 * f + r * f * (1.0 / 6 - f * (1.0 / 30 - f * (1.0 / 42 - f / 30)));
}

// Table-driven exponential and logarithm (P. T. P. Tang, ACM TOMS 15 (1989)
// 144 and 16 (1990) 378): the argument is reduced to 1/32 of an octave, the
// remainder's Taylor series needs few terms, and a warp's 32 lanes hold the
// table, one entry each, which a lookup takes by shuffle (all lanes take part).
// exp within 1.6 ulp (the table's entry 1, the last rounding 0.5; largest
// seen 1.09), log within 2e-16 (the table's entry) + 1.5 ulp (ln 2 times the
// exponent, two roundings; largest seen 1.3e-16 in [0.5, 2], 1.27 ulp beyond).
struct WarpTables {
  double exp2_at;         // 2^(lane / 32)
  double inv_at, log_at;  // 1 / c, rounded to FP32, and ln c, for c at the middle of [1 + lane/32, 1 + (lane + 1)/32)
  // the constants, held in registers: as literals or from constant memory
  // each costs one or two instructions per use
  double inv_ln2_32, magic, ln2_32_hi, ln2_32_lo;  // 32 / ln 2; 1.5 * 2^52; -ln 2 / 32 as 37 leading bits and the rest
  double e3, e4, e5, e6;                           // 1 / n!
  double bias, ln2;                                // 2^52 + 1023
  double l3, l4, l5, l6, l7, l8;                   // -(-1)^n / n
};
__device__ __forceinline__ double in_register(double v) {
  double r;
  asm volatile("mov.f64 %0, %1;" : "=d"(r) : "d"(v));
  return r;
}
__device__ __forceinline__ WarpTables warp_tables() {
  const double l = (double)(threadIdx.x & 31);
  WarpTables t;
  t.exp2_at = exp2(l / 32.0);
  t.inv_at = (double)(float)(1.0 / (1.0 + (l + 0.5) / 32.0));
  t.log_at = -log(t.inv_at);
  t.inv_ln2_32 = in_register(32.0 / 0.69314718055994530942);
  t.magic = in_register(6755399441055744.0);
  t.ln2_32_hi = in_register(-0x1.62e42fefap-6);
  t.ln2_32_lo = in_register(-0x1.cf79abc9e3b39p-45);
  t.e3 = in_register(1.0 / 6);
  t.e4 = in_register(1.0 / 24);
  t.e5 = in_register(1.0 / 120);
  t.e6 = in_register(1.0 / 720);
  t.bias = in_register(4503599627371519.0);
  t.ln2 = in_register(0.69314718055994530942);
  t.l3 = in_register(1.0 / 3);
  t.l4 = in_register(-1.0 / 4);
  t.l5 = in_register(1.0 / 5);
  t.l6 = in_register(-1.0 / 6);
  t.l7 = in_register(1.0 / 7);
  t.l8 = in_register(-1.0 / 8);
  return t;
}
// e^v for -708 <= v <= 708; beyond, the value at that end (an argument that is
// not a number gives one of the two).
__device__ __forceinline__ double exp_tab(double v, const WarpTables& T) {
  constexpr unsigned kLow = 0xC0862000u;  // high word of -708
  constexpr int kHigh = 0x40862000;       // high word of 708
  const int hi = min((int)min((unsigned)__double2hiint(v), kLow), kHigh);
  v = __hiloint2double(hi, __double2loint(v));
  const double t = fma(v, T.inv_ln2_32, T.magic);  // rounded to an integer, in the low word
  const int n = __double2loint(t);
  const double k = t - T.magic;
  const double r = fma(k, T.ln2_32_lo, fma(k, T.ln2_32_hi, v));
  double q = fma(r, T.e6, T.e5);
  q = fma(r, q, T.e4);
  q = fma(r, q, T.e3);
  q = fma(r, q, 0.5);
  const double p = fma(r * r, q, r);
  const double at = __shfl_sync(0xffffffffu, T.exp2_at, n);  // lane n mod 32
  const double e = fma(at, p, at);
  return __hiloint2double(__double2hiint(e) + ((n >> 5) << 20), __double2loint(e));
}
// ln y for normal y > 0 (anything else gives some number).
__device__ __forceinline__ double log_tab(double y, const WarpTables& T) {
  const int hi = __double2hiint(y);
  const double m = __hiloint2double((hi & 0x000FFFFF) | 0x3FF00000, __double2loint(y));
  const int at = hi >> 15;  // lane: the mantissa's leading five bits
  const double k = __hiloint2double(0x43300000, hi >> 20) - T.bias;  // 2^52 + biased exponent, less 2^52 + 1023
  const double r = fma(m, __shfl_sync(0xffffffffu, T.inv_at, at), -1.0);  // |r| <= 1/63: the series' ninth term is below 1e-17
  double q = fma(r, T.l8, T.l7);
  q = fma(r, q, T.l6);
  q = fma(r, q, T.l5);
  q = fma(r, q, T.l4);
  q = fma(r, q, T.l3);
  q = fma(r, q, -0.5);
  return fma(k, T.ln2, __shfl_sync(0xffffffffu, T.log_at, at)) + fma(r * r, q, r);
}

// 1 / s for 1 <= s <= 2, within 1 ulp (largest seen 0.502): the FP32 reciprocal of its leading
// bits (2^-20) and one step of Newton's iteration, third order.
__device__ __forceinline__ double reciprocal_1_2(double s) {
  const float f = __uint_as_float(__funnelshift_l(__double2loint(s), __double2hiint(s), 3) + 0x40000000u);
  float g;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(g) : "f"(f));
  const double r = __hiloint2double((int)((__float_as_uint(g) >> 3) + 0x38000000u), 0);
  const double e = fma(-s, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

}  // namespace ppsf
