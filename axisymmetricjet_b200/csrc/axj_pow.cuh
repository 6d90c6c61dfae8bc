// axj_pow.cuh -- mu = T**0.666 in FP64 (ModAssign.f90:20, Tvec**0.666D0) from tables,
// shared by the kernels and the host (the same operations in the same order, so the
// host evaluation reproduces the device's bits).
//
// Method (a table-driven reduction with a binomial series, after Tang's table-driven
// logarithm): T = 2^e m with m in [1, 2); j = the top 7 bits of m's fraction; c_j a 10-bit
// approximation of 1/F_j (F_j = 1 + (j + 1/2) / 128, the centre of m's interval);
// r = m c_j - 1 with one rounding (|r| < 0.006). Then
//     T^a = 2^(a e) * c_j^(-a) * (1 + r)^a,
// the first two factors from tables held as double-double (hi + lo), the third from the
// binomial series 1 + sum_{k=1..6} binom(a, k) r^k (the first term left out is below
// 3e-18). The product is formed in double-double and rounded once: within 1 ulp of
// the correctly rounded power. Exponents e outside [-16, 15] (T outside [2^-16, 2^16)),
// zero, negative, subnormal and non-finite T take exp2(a log2 T).
#pragma once

#include <cstdint>
#include <cstring>
#include <cmath>

#include "axj_common.cuh"

namespace axj {

constexpr int POW_NJ = 128;                        // mantissa intervals
constexpr int POW_E0 = -16, POW_NE = 32;           // exponents e = POW_E0 .. POW_E0 + POW_NE - 1
constexpr int POW_TAB = 4 * POW_NJ + 2 * POW_NE;   // {G_hi, G_lo, c_j, 0} per j, then {E_hi, E_lo} per e
constexpr double POW_A = 0.666;                    // the exponent 0.666D0
// binom(a, k), k = 1..6
constexpr double POW_B1 = POW_A;
constexpr double POW_B2 = POW_B1 * (POW_A - 1.0) / 2.0;
constexpr double POW_B3 = POW_B2 * (POW_A - 2.0) / 3.0;
constexpr double POW_B4 = POW_B3 * (POW_A - 3.0) / 4.0;
constexpr double POW_B5 = POW_B4 * (POW_A - 4.0) / 5.0;
constexpr double POW_B6 = POW_B5 * (POW_A - 5.0) / 6.0;

struct PowPair {
  double x, y;
};
#ifdef __CUDA_ARCH__
// (the device tables are 16-byte aligned: a pair is one load)
AXJ_HD PowPair pow_pair(const double* p) {
  const double2 v = __ldg(reinterpret_cast<const double2*>(p));
  return PowPair{v.x, v.y};
}
AXJ_HD double pow_one(const double* p) { return __ldg(p); }
AXJ_HD long long pow_bits(double x) { return __double_as_longlong(x); }
AXJ_HD double pow_from_bits(long long b) { return __longlong_as_double(b); }
AXJ_HD double pow_fallback(double T) { return exp2(POW_A * log2(T)); }
#else
inline PowPair pow_pair(const double* p) { return PowPair{p[0], p[1]}; }
inline double pow_one(const double* p) { return *p; }
inline long long pow_bits(double x) {
  long long b;
  std::memcpy(&b, &x, sizeof b);
  return b;
}
inline double pow_from_bits(long long b) {
  double x;
  std::memcpy(&x, &b, sizeof x);
  return x;
}
inline double pow_fallback(double T) { return std::exp2(POW_A * std::log2(T)); }
#endif

// Whether T lies in the tables' range (positive, exponent POW_E0 .. POW_E0 + POW_NE - 1).
AXJ_HD bool pow0666_in_range(double T) {
  const int e = ((int)(pow_bits(T) >> 32) >> 20) - 1023;  // negative T: the sign puts e out of range
  return e >= POW_E0 && e < POW_E0 + POW_NE;
}

// T**0.666 of a T in range from the tables tab[POW_TAB] (pow0666_fill); any other T gives a
// value of no meaning (without a branch, so that a thread's several powers interleave).
AXJ_HD double pow0666_table(double T, const double* __restrict__ tab) {
  const long long bits = pow_bits(T);
  const int hi = (int)(bits >> 32);
  const int e = ((hi >> 20) - 1023 - POW_E0) & (POW_NE - 1);  // in range: unchanged
  const int j = (hi >> 13) & (POW_NJ - 1);
  const double m = pow_from_bits((bits & 0x000FFFFFFFFFFFFFLL) | 0x3FF0000000000000LL);
  const PowPair g = pow_pair(tab + 4 * j), E = pow_pair(tab + 4 * POW_NJ + 2 * e);
  const double r = fma(m, pow_one(tab + 4 * j + 2), -1.0);
  double t = fma(r, POW_B6, POW_B5);
  t = fma(r, t, POW_B4);
  t = fma(r, t, POW_B3);
  t = fma(r, t, POW_B2);
  t = fma(r, t, POW_B1);
  const double q = r * t;  // (1 + r)^a - 1
  // P = 2^(a e) c_j^(-a) as ph + pl, then P (1 + q) rounded once
  const double ph = E.x * g.x;
  const double pl = fma(E.x, g.x, -ph) + fma(E.x, g.y, E.y * g.x);
  return ph + fma(ph, q, pl);
}

// T**0.666 from the tables tab[POW_TAB].
AXJ_HD double pow0666(double T, const double* __restrict__ tab) {
  return pow0666_in_range(T) ? pow0666_table(T, tab) : pow_fallback(T);
}

// The tables of pow0666, evaluated on the host in long double (64-bit significand) and
// split into double hi + lo parts.
inline void pow0666_fill(double* tab) {
  const long double a = (long double)POW_A;
  for (int j = 0; j < POW_NJ; ++j) {
    const long double F = 1.0L + ((long double)j + 0.5L) / (long double)POW_NJ;
    const double c = std::ldexp(std::nearbyint(std::ldexp((double)(1.0L / F), 9)), -9);  // 10 bits
    const long double g = powl((long double)c, -a);
    tab[4 * j] = (double)g;
    tab[4 * j + 1] = (double)(g - (long double)tab[4 * j]);
    tab[4 * j + 2] = c;
    tab[4 * j + 3] = 0.0;
  }
  for (int k = 0; k < POW_NE; ++k) {
    const long double v = exp2l(a * (long double)(POW_E0 + k));
    double* te = tab + 4 * POW_NJ + 2 * k;
    te[0] = (double)v;
    te[1] = (double)(v - (long double)te[0]);
  }
}

}  // namespace axj
