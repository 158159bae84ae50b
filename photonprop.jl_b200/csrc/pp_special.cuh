// FP64 digamma and trigamma for the device: upward recurrence to x >= 6,
// then the asymptotic series
//   psi(x)  = ln x - 1/(2x) - sum_k B_2k / (2k x^2k)
//   psi'(x) = 1/x + 1/(2x^2) + sum_k B_2k / x^(2k+1)
// (Bernoulli numbers B_2..B_10); relative error below 1e-14 for x > 0.
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
  const double rd = 1.0 / (low ? q * q4 * q6 : 1.0);
  const double u = q4 * q6 * rd, v = q * q6 * rd, w = q * q4 * rd;
  const double s0 = low ? fma(2.0, x, 5.0) * (u + v + w) : 0.0;
  const double s1 = low ? fma(2.0, q, 25.0) * u * u + fma(2.0, q, 17.0) * v * v + fma(2.0, q, 13.0) * w * w : 0.0;
  const double y = low ? x + 6.0 : x;
  const double r = 1.0 / y, f = r * r;
  psi = log(y) - 0.5 * r - f * (1.0 / 12 - f * (1.0 / 120 - f * (1.0 / 252 - f * (1.0 / 240 - f / 132)))) - s0;
  psi1 = s1 + r + 0.5 * f + r * f * (1.0 / 6 - f * (1.0 / 30 - f * (1.0 / 42 - f / 30)));
}

}  // namespace ppsf
