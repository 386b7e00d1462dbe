// quotient_check.cu -- the shared-divisor quotients (SharedDivisor) against
// IEEE division, and the van Leer gradient with half the divisions
// (limited_gradient_t<2>) against the reference formula, on the host: random
// operands, quotients near rounding midpoints and powers of two, divisors and
// numerators at the ends of their ranges, signed zeros, subnormals, infinities
// and NaN.  A quotient counts when SharedDivisor accepts it; the share accepted
// inside the stated ranges has to be all of them.  Exit status 0 when every
// result is bit-identical, the sign of a zero quotient aside.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include "mhc_device.cuh"
using namespace mhc;
static bool same(double a, double b) { uint64_t x, y; memcpy(&x, &a, 8); memcpy(&y, &b, 8); return x == y; }
int main() {
  long n = 0, bad = 0, refused = 0;
  auto quotient = [&](double a, double b, bool inside) {
    SharedDivisor d;
    d.set(b);
    bool ok = true;
    const double q = d.q(a, ok);
    ++n;
    if (ok ? !(same(q, a / b) || (q == 0. && a / b == 0.)) : inside) {
      if (bad++ < 10) printf("a=%a b=%a: %a, division %a, accepted %d\n", a, b, q, a / b, ok);
    }
    refused += !ok;
  };
  std::mt19937_64 rng(7);
  std::uniform_real_distribution<double> m(1., 2.), eb(-399., 398.), ea(-499., 498.), small(-20., 20.);
  auto sign = [&] { return (rng() & 1) ? 1. : -1.; };
  for (long i = 0; i < 6000000; ++i) quotient(sign() * std::ldexp(m(rng), (int)ea(rng)), sign() * std::ldexp(m(rng), (int)eb(rng)), true);
  for (long i = 0; i < 3000000; ++i) {
    // quotients at and next to a representable number or a midpoint
    const double b = sign() * std::ldexp(m(rng), (int)small(rng));
    double q = m(rng);
    if (i % 3 == 1) q = 1. + (double)(rng() % 64) * 0x1p-52;
    if (i % 3 == 2) q = 2. - (double)(rng() % 64) * 0x1p-52;
    double a = q * b;
    for (int s = 0; s < (int)(rng() % 3); ++s) a = std::nextafter(a, (rng() & 1) ? INFINITY : -INFINITY);
    quotient(a, b, true);
    const double mid = std::fma(0.5 * 0x1p-52, b, q * b);  // half an ulp of q above
    quotient(mid, b, true);
  }
  // divisors with extreme mantissas
  for (long i = 0; i < 200000; ++i) {
    const double b = (i & 1) ? 2. - 0x1p-52 * (1 + i % 7) : 1. + 0x1p-52 * (i % 7);
    quotient(m(rng), b, true);
  }
  const double sp[] = {0.0, -0.0, 1.0, -1.0, 3.0, 4.9e-324, -4.9e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
                       -1.7976931348623157e308, INFINITY, -INFINITY, NAN, 1e-160, 1e160, 1e-200, 1e200};
  for (double a : sp)
    for (double b : sp) quotient(a, b, false);
  long gn = 0, gbad = 0;
  auto gradient = [&](double gb, double gf) {
    const double r = limited_gradient_ref<2>(gb, gf), t = limited_gradient_t<2>(gb, gf);
    ++gn;
    if (!same(r, t) && !(std::isnan(r) && std::isnan(t)) && gbad++ < 10) printf("gb=%a gf=%a: %a, reference %a\n", gb, gf, t, r);
  };
  std::uniform_real_distribution<double> u(-1., 1.), e(-300., 300.);
  for (long i = 0; i < 2000000; ++i) {
    gradient(u(rng) * std::pow(10., e(rng) * 0.02), u(rng) * std::pow(10., e(rng) * 0.02));
    gradient(u(rng) * std::pow(10., e(rng)), u(rng) * std::pow(10., e(rng)));
    const double x = u(rng);
    gradient(x, x * (1. + (double)(rng() % 5) * 0x1p-52));
  }
  for (double a : sp)
    for (double b : sp) gradient(a, b);
  printf("checked %ld quotients (%ld refused), %ld gradients, mismatches %ld\n", n, refused, gn, bad + gbad);
  return bad + gbad != 0;
}
