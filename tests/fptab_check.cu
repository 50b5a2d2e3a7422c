// Host-side check of the far field's table-driven e^{ix} and e^x (fptab.cuh, the same
// code that the kernels use) against long double: prints the largest error of
// cos and sin beyond half a unit in the last place, in units of 2^-56, that of
// e^x in units in the last place, and the number of results outside the
// functions' ranges that differ from the library's.
#include <cmath>
#include <cstdio>
#include "../scuff-em_gb300/csrc/fptab.cuh"
using namespace gbem;

static double urand(unsigned long long* s) {
  *s = *s * 6364136223846793005ull + 1442695040888963407ull;
  return (double)(*s >> 11) * 0x1p-53;
}
static double ulp(double x) { return std::nextafter(std::fabs(x), INFINITY) - std::fabs(x); }
static bool same(double a, double b) { return a == b || (a != a && b != b); }

int main() {
  SinCosTab64 T;
  fill_sincos_tab64(&T);
  unsigned long long seed = 1;
  double ei = 0, ee = 0;
  auto check = [&](double x) {
    double c, s;
    expi64(x, T, &c, &s);
    const long double lc = cosl((long double)x), ls = sinl((long double)x);
    ei = fmax(ei, (double)fabsl(c - lc) - 0.5 * ulp((double)lc));
    ei = fmax(ei, (double)fabsl(s - ls) - 0.5 * ulp((double)ls));
  };
  const long double pi = 3.14159265358979323846264338327950288L, ln2 = 0.693147180559945309417232121458176568L;
  for (int i = 0; i < 400000; i++) {
    const double sg = i & 1 ? -1.0 : 1.0;
    check(sg * exp2(-30.0 + 45.6 * urand(&seed)));  // up to 5e4
    // the seams between two table entries, and the multiples of pi/64 themselves
    const long long j = (long long)(1018000 * urand(&seed));
    check(sg * (double)((j + (i & 2 ? 0.5L : 0.0L)) * pi / 64));
  }
  auto check_exp = [&](double x) {
    const long double l = expl((long double)x);
    ee = fmax(ee, (double)fabsl(exp64(x, T) - l) / ulp((double)l));
  };
  for (int i = 0; i < 400000; i++) {
    const double sg = i & 1 ? -1.0 : 1.0;
    check_exp(sg * exp2(-30.0 + 39.45 * urand(&seed)));  // up to 700
    check_exp(sg * (double)(((long long)(64600 * urand(&seed)) + (i & 2 ? 0.5L : 0.0L)) * ln2 / 64));
  }
  int bad = 0;
  for (double x : {5.0e4, -5.0e4, 1e9, (double)INFINITY, -(double)INFINITY, (double)NAN}) {
    double c, s;
    expi64(x, T, &c, &s);
    bad += !same(c, cos(x)) + !same(s, sin(x));
  }
  for (double x : {700.0, -700.0, 710.0, -746.0, (double)INFINITY, -(double)INFINITY, (double)NAN}) bad += !same(exp64(x, T), exp(x));
  printf("expi %.3f exp %.4f bad %d\n", ei * 0x1p56, ee, bad);
  return 0;
}
