// fptab.cuh -- e^{ix} and e^x in FP64 by table lookup, for the FP64 far field, whose
// operations are what bounds it.  The scheme is Tang's (P. T. P. Tang, "Table-lookup
// algorithms for elementary functions and their error analysis", 10th IEEE Symposium on
// Computer Arithmetic, 1991): a table of exact values and of what their rounding left,
// a short polynomial in the reduced argument, one rounding at the end.  Host and device.
#pragma once
#include <cmath>
#include <cstring>
#include "bem_math.cuh"

namespace gbem {

struct SinCosTab64 {
  double c[128], s[128];   // cos, sin of j pi/64
  double cl[128], sl[128];  // what their rounding left
  double e[64], el[64];     // 2^(j/64), likewise
};
// cos(j pi/64), j = 0 .. 32, rounded, and the remainders
static const double h_cos64[33] = {
    0x1.0000000000000p+0, 0x1.ff621e3796d7ep-1, 0x1.fd88da3d12526p-1, 0x1.fa7557f08a517p-1, 0x1.f6297cff75cb0p-1,
    0x1.f0a7efb9230d7p-1, 0x1.e9f4156c62ddap-1, 0x1.e212104f686e5p-1, 0x1.d906bcf328d46p-1, 0x1.ced7af43cc773p-1,
    0x1.c38b2f180bdb1p-1, 0x1.b728345196e3ep-1, 0x1.a9b66290ea1a3p-1, 0x1.9b3e047f38741p-1, 0x1.8bc806b151741p-1,
    0x1.7b5df226aafafp-1, 0x1.6a09e667f3bcdp-1, 0x1.57d69348ceca0p-1, 0x1.44cf325091dd6p-1, 0x1.30ff7fce17035p-1,
    0x1.1c73b39ae68c8p-1, 0x1.073879922ffeep-1, 0x1.e2b5d3806f63bp-2, 0x1.b5d1009e15cc0p-2, 0x1.87de2a6aea963p-2,
    0x1.58f9a75ab1fddp-2, 0x1.294062ed59f06p-2, 0x1.f19f97b215f1bp-3, 0x1.8f8b83c69a60bp-3, 0x1.2c8106e8e613ap-3,
    0x1.917a6bc29b42cp-4, 0x1.91f65f10dd814p-5, 0.0};
static const double h_cos64_lo[33] = {
    0.0, -0x1.c57bc2e24aa15p-57, -0x1.87df6378811c7p-55, -0x1.7a0a8ca13571fp-55, 0x1.562172a361fd3p-56,
    0x1.52c7adc6b4989p-56, 0x1.760b1e2e3f81ep-55, -0x1.014c76c126527p-55, 0x1.457e610231ac2p-56,
    -0x1.e7b6bb5ab58aep-58, -0x1.6e0b1757c8d07p-56, -0x1.bc69f324e6d61p-55, 0x1.9f630e8b6dac8p-60,
    -0x1.30ee286712474p-55, -0x1.2c5e12ed1336dp-55, -0x1.0f537acdf0ad7p-56, -0x1.bdd3413b26456p-55,
    -0x1.75720992bfbb2p-55, 0x1.8076a2cfdc6b3p-57, -0x1.efcc626f74a6fp-57, 0x1.b25dd267f6600p-55,
    -0x1.a5a014347406cp-55, 0x1.e0d891d3c6841p-58, 0x1.5b362cb974183p-57, -0x1.72cedd3d5a610p-57,
    -0x1.efdc0d58cf620p-62, -0x1.5d28da2c4612dp-56, -0x1.42deef11da2c4p-57, -0x1.26d19b9ff8d82p-57,
    0x1.13000a89a11e0p-58, -0x1.e2718d26ed688p-60, -0x1.912bd0d569a90p-61, 0.0};
static void fill_sincos_tab64(SinCosTab64* t) {
  // cos((128 - j) pi/64) = cos(j pi/64) = -cos((64 - j) pi/64), sin = cos shifted by 32
  auto at = [](const double* q, int j) {
    j &= 127;
    if (j > 64) j = 128 - j;
    return j <= 32 ? q[j] : -q[64 - j];
  };
  for (int j = 0; j < 128; j++) {
    t->c[j] = at(h_cos64, j); t->cl[j] = at(h_cos64_lo, j);
    t->s[j] = at(h_cos64, j + 96); t->sl[j] = at(h_cos64_lo, j + 96);
  }
  for (int j = 0; j < 64; j++) {
    const long double v = exp2l(j / 64.0L);
    t->e[j] = (double)v;
    t->el[j] = (double)(v - (long double)t->e[j]);
  }
}

GB_HD int high_word(double x) {
#ifdef __CUDA_ARCH__
  return __double2hiint(x);
#else
  long long b;
  memcpy(&b, &x, 8);
  return (int)(b >> 32);
#endif
}
GB_HD int low_word(double x) {
#ifdef __CUDA_ARCH__
  return __double2loint(x);
#else
  long long b;
  memcpy(&b, &x, 8);
  return (int)b;
#endif
}
GB_HD double from_words(int hi, int lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double(hi, lo);
#else
  const long long b = ((long long)hi << 32) | (unsigned)lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}

constexpr double PI64_HI = 0x1.921fb54400000p-5;  // pi/64, leading 33 bits
constexpr double PI64_LO = 0x1.0b4611a626331p-39;
constexpr double EXPI_MAX = 5.0e4;                // j < 2^20: j PI64_HI is exact

// e^{ix} by table lookup: x = j pi/64 + t, |t| <= pi/128 (Cody and Waite's reduction in
// two parts), the Taylor series of sin t and cos t - 1 to t^7 and t^6 (remainders
// below 4e-18), added onto the table's values and their remainders.  Error: the last
// rounding, half a unit in the last place, and at most 2^-56 before it
GB_HD void expi64(double x, const SinCosTab64& tab, double* c, double* s) {
  if ((high_word(x) & 0x7fffffff) >= 0x40e86a00) {  // |x| >= EXPI_MAX, infinite or NaN
    sincos(x, s, c);
    return;
  }
  const double magic = 6755399441055744.0;  // 1.5 * 2^52: rounds to an integer in the low word
  const double y = fma(x, 64.0 / 3.14159265358979323846, magic);
  const int j = low_word(y) & 127;
  const double jf = y - magic;
  const double t = fma(-jf, PI64_LO, fma(-jf, PI64_HI, x));
  const double t2 = t * t;
  const double sn = fma(t * t2, fma(t2, fma(t2, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), t);
  const double cm = t2 * fma(t2, fma(t2, -1.0 / 720.0, 1.0 / 24.0), -0.5);
  const double c0 = tab.c[j], s0 = tab.s[j];
  *c = c0 + fma(c0, cm, fma(-s0, sn, tab.cl[j]));
  *s = s0 + fma(s0, cm, fma(c0, sn, tab.sl[j]));
}

// e^x by the same means: x = (64 m + j) ln2/64 + t,
// |t| <= ln2/128, the Taylor series of e^t - 1 to t^6 (remainder below 3e-20) onto
// the table's 2^(j/64) and its remainder, scaled by 2^m: at most 0.52 units in
// the last place, 12 operations of the FP64 pipe where exp takes about 17.  At imaginary k
// (two bodies, N = 3840) 11.4 -> 10.4 ms and the gradient 4.72 -> 4.36; at complex
// k, where it is one operation in thirty (9.12 -> 8.90 ms), exp stays
constexpr double LN2_64_HI = 0x1.62e42fefp-7;  // ln2/64, leading 33 bits
constexpr double LN2_64_LO = 0x1.473de6af278edp-40;
GB_HD double exp64(double x, const SinCosTab64& tab) {
  if ((high_word(x) & 0x7fffffff) >= 0x4085e000) return exp(x);  // |x| >= 700, infinite or NaN
  const double magic = 6755399441055744.0;
  const double y = fma(x, 64.0 / 0.69314718055994530942, magic);
  const int n = low_word(y), j = n & 63;
  const double jf = y - magic;
  const double t = fma(-jf, LN2_64_LO, fma(-jf, LN2_64_HI, x));
  const double q = fma(t, fma(t, fma(t, fma(t, 1.0 / 720.0, 1.0 / 120.0), 1.0 / 24.0), 1.0 / 6.0), 0.5);
  const double p = fma(t * t, q, t);
  const double v = tab.e[j], r = v + fma(v, p, tab.el[j]);
  return from_words(high_word(r) + ((n >> 6) << 20), low_word(r));
}

}  // namespace gbem
