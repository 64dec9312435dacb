// Host check of photic_softfp.cuh and of the two-operation constant
// divisions of photic_fastmath.cuh: the headers the kernels compile, built
// with g++, against the IEEE operations of this machine, bit for bit.  The
// reciprocal estimates are moved by up to three units of their last place,
// more than the hardware's error.
//
//   softfp_check <samples> <seed>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

namespace {
uint64_t g_state = 1;
uint64_t next() {
  g_state += 0x9e3779b97f4a7c15ULL;
  uint64_t z = g_state;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}
float moved(float x) {
  uint32_t u;
  memcpy(&u, &x, 4);
  u += (uint32_t)((int)(next() % 7) - 3);
  memcpy(&x, &u, 4);
  return x;
}
}  // namespace
#define PHOTIC_SF_PERTURB(x) moved(x)
#include "photic_softfp.cuh"

using namespace photic;

namespace {

long g_bad = 0, g_exp = 0, g_exp_rare = 0;

void same(double got, double want, const char *what, double a, double b) {
  if (memcmp(&got, &want, 8) == 0 || (got != got && want != want)) return;
  if (g_bad++ < 10) printf("%s(%a, %a): %a, want %a\n", what, a, b, got, want);
}

double from(uint64_t u) {
  double d;
  memcpy(&d, &u, 8);
  return d;
}
uint64_t of(double d) {
  uint64_t u;
  memcpy(&u, &d, 8);
  return u;
}

// A double with exponent in [lo, hi]: random, short, long runs of ones, and
// significands at either end.
double sample(int lo, int hi) {
  uint64_t m = next() & 0xfffffffffffffULL;
  switch (next() % 6) {
    case 0: m &= ~0ULL << (next() % 52); break;
    case 1: m |= (1ULL << (next() % 52)) - 1; break;
    case 2: m = 0xfffffffffffffULL - next() % 64; break;
    case 3: m = next() % 64; break;
    default: break;
  }
  const uint64_t e = (uint64_t)(1023 + lo) + next() % (uint64_t)(hi - lo + 1);
  return from(e << 52 | m);
}

}  // namespace

int main(int argc, char **argv) {
  const long n = argc > 1 ? atol(argv[1]) : 1000000;
  g_state = argc > 2 ? (uint64_t)atol(argv[2]) : 1;
  for (long i = 0; i < n; i++) {
    const int span = i & 1 ? 40 : 500;
    double a = sample(-span, span), b = sample(-span, span);
    if (next() & 1) a = -a;
    if (i % 4 == 0) {  // quotients at and beside a double
      b = sample(-40, 40);
      a = sample(0, 0) * b;
      a = from(of(a) + (uint64_t)((int64_t)(next() % 5) - 2));
    }
    same(sf::div_mid(a, b), a / b, "div", a, b);
    double s = fabs(a);
    if (i % 3 == 0) {  // roots at and beside a double
      const double q = sample(-10, 10);
      s = from(of(q * q) + (uint64_t)((int64_t)(next() % 5) - 2));
    }
    same(sf::sqrt_mid(s), ::sqrt(s), "sqrt", s, 0);
    same(fm::div_pi(a), a / 3.141592653589793, "pi", a, 0);
    same(fm::div_120(a), a / 120.0, "120", a, 0);
    same(fm::div_6(a), a / 6.0, "6", a, 0);
    {  // the exponential over the range and the scale the cost meets
      const double e = -fabs(i & 1 ? sample(-62, 8) : sample(-8, 6));
      bool ok = true;
      const double got = sf::exp_neg(e, ok);
      g_exp++;
      if (ok) same(got, fm::exp_t(e), "exp", e, 0);
      else g_exp_rare += e < -0x1p-30 && e > -350.0;
    }
    {  // small counts: as hi + lo
      const double k = (double)(1 + i % 128), hi = 1.0 / k;
      same(fm::div_const(a, k, hi, fm::recip_lo(k, hi)), a / k, "count", a, k);
      const float c = i % 3 == 0 ? 0.5f : i % 3 == 1 ? 1.0f : 2.0f;
      same(sf::add_scaled2(a, b, c), a + b * (double)c, "point", a, b);
      if ((sf::order_key(a) < sf::order_key(b)) != (a < b)) g_bad++, printf("key %a %a\n", a, b);
    }
    if (sf::lt(a, b) != (a < b) || sf::lt(b, a) != (b < a) || sf::le(a, b) != (a <= b) ||
        !sf::le(a, a) || sf::lt(a, a) || sf::lt_call(a, b) != (a < b) ||
        sf::le_call(a, b) != (a <= b))
      g_bad++, printf("comparison of %a and %a\n", a, b);
  }
  const double special[] = {0.0, -0.0, 1.0, -1.0, 2.0, INFINITY, -INFINITY, NAN, -NAN, 5e-324,
                            -5e-324, 1e-310, 2.2250738585072014e-308, 1.7976931348623157e308,
                            -1.7976931348623157e308, 1e-200, 1e200, -3.0};
  for (double a : special) {
    same(sf::sqrt(a), ::sqrt(a), "sqrt", a, 0);
    same(fm::div_pi(a), a / 3.141592653589793, "pi", a, 0);
    same(fm::div_120(a), a / 120.0, "120", a, 0);
    for (double b : special) {
      same(sf::div(a, b), a / b, "div", a, b);
      same(sf::add_scaled2(a, b, 0.5f), a + b * 0.5, "point", a, b);
      same(sf::add_scaled2(a, b, 2.0f), a + b * 2.0, "point", a, b);
      if ((sf::order_key(a) != 0 && sf::order_key(a) < sf::order_key(b)) != (a < b))
        g_bad++, printf("key %a %a\n", a, b);
      if (sf::lt(a, b) != (a < b) || sf::le(a, b) != (a <= b) || sf::lt_call(a, b) != (a < b) ||
          sf::le_call(a, b) != (a <= b))
        g_bad++, printf("comparison of %a and %a\n", a, b);
    }
  }
  for (long i = 0; i < n / 20; i++) {  // ordered sums of terms that are not negative
    double v[40];
    const int m = (int)(next() % 40), span = i % 4 == 0 ? 0 : i % 4 == 1 ? 3 : i % 4 == 2 ? 30 : 900;
    for (int j = 0; j < m; j++) v[j] = next() % 9 == 0 ? 0.0 : fabs(sample(-span, span));
    if (m && i % 97 == 0) v[next() % m] = i % 2 ? NAN : i % 3 ? INFINITY : 3e-310;
    if (m && i % 89 == 0) v[next() % m] = -1.0;
    double want = 0.0;
    for (int j = 0; j < m; j++) want = want + v[j];
    same(sf::sum_positive(v, 1, m), want, "sum", m, 0);
  }
  const double refused[] = {-0.0, 0.0, -5e-324, -354.0, -400.0, -1e300, -INFINITY, NAN};
  for (double e : refused) {
    bool ok = true;
    (void)sf::exp_neg(e, ok);
    if (ok) g_bad++, printf("exp takes %a\n", e);
  }
  printf("mismatches %ld, exponentials left to the general path %ld of %ld\n", g_bad, g_exp_rare,
         g_exp);
  return g_bad != 0;
}
