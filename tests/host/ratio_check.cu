// ratio_check.cu -- the clamped quotients of the pente-borne fluxes
// (pb_ratio01, pb_ratio_mid, mhc_device.cuh) against the division they
// replace, on the host: random operands over the whole range, quotients a few
// ulps around 0, 1/2 and 1, signed zeros, subnormals, infinities and NaN.
// Exit status 0 when every result is bit-identical (the sign of a zero
// quotient included).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include "mhc_device.cuh"
using namespace mhc;
int main() {
  long n = 0, bad = 0;
  auto same = [](double a, double b) { uint64_t x, y; memcpy(&x, &a, 8); memcpy(&y, &b, 8); return x == y; };
  auto test = [&](double a, double b) {
    const double r = amin(amax(0., a / b), 1.), m = amin(amax(a / b - 1. / 2., -1. / 2.), 1. / 2.);
    if (!same(pb_ratio01(a, b), r) || !same(pb_ratio_mid(a, b), m)) {
      if (bad++ < 10) printf("a=%.17g b=%.17g: %.17g %.17g\n", a, b, r, m);
    }
    ++n;
  };
  std::mt19937_64 rng(99);
  std::uniform_real_distribution<double> u(-1, 1), e(-300, 300);
  for (long i = 0; i < 2000000; ++i) test(u(rng) * std::pow(10., e(rng) * 0.1), u(rng) * std::pow(10., e(rng) * 0.1));
  for (long i = 0; i < 300000; ++i) {
    const double b = u(rng) * std::pow(10., e(rng) * 0.3), k[] = {0.5, 1., -1., 2.};
    double x = b * k[i % 4];
    for (int s = 0; s < 3; ++s, x = std::nextafter(x, INFINITY)) test(x, b);
    x = b * k[i % 4];
    for (int s = 0; s < 3; ++s, x = std::nextafter(x, -INFINITY)) test(x, b);
  }
  const double sp[] = {0.0, -0.0, 1.0, -1.0, 0.5, 4.9e-324, -4.9e-324, 2.2250738585072014e-308, 1.7976931348623157e308,
                       -1.7976931348623157e308, INFINITY, -INFINITY, NAN, 1e-160, 1e160};
  for (double a : sp) for (double b : sp) test(a, b);
  printf("checked %ld quotients, mismatches %ld\n", n, bad);
  return bad != 0;
}
