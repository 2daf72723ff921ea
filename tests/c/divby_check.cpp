// Host check of div_by, less_bits and zero_bits (clblm_fpconv.cuh) against the
// machine's own division and comparisons: divisors of a few digits and any,
// dividends at multiples of the divisor, half way between and next to them.
#include <cmath>
#include <cstdio>
#include <random>

#include "clblm_fpconv.cuh"

using namespace clblm;

int main() {
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> u(0., 1.);
  long n = 0, bad = 0;
  for (int k = 0; k < 20000; ++k) {
    double d = std::pow(10., -6. + 4. * u(g));
    if (k % 3 == 0) d = (1 + (int)(5000 * u(g))) * std::pow(10., -(double)(3 + (int)(5 * u(g))));
    const double r = 1. / d;
    for (int j = 0; j < 100; ++j) {
      double x = (u(g) - 0.2) * 30.;
      if (j % 5 == 1) x = (double)(int)(4000 * u(g)) * d;
      if (j % 5 == 2) x = std::nextafter(((double)(int)(4000 * u(g)) + 0.5) * d, u(g) < 0.5 ? 0. : 100.);
      if (j % 5 == 3) x = std::floor(1e6 * u(g)) * 1e-6 * (u(g) < 0.3 ? -1 : 1);
      if (j % 5 == 4) x = std::ldexp(u(g), (int)(60 * u(g)) - 40);
      ++n;
      if (div_by(x, d, r) != x / d) bad++;
      const double b = (j & 1) ? d : u(g) - 0.5;
      if (less_bits(x, b) != (x < b) || zero_bits(x) != (x == 0.)) bad++;
    }
  }
  for (double x : {0., -1., 1., 1e-300, -1e-300, 1e300})
    for (double b : {0., 1., 2.5, -1., 1e300})
      if (less_bits(x, b) != (x < b) || zero_bits(x) != (x == 0.)) bad++;
  printf("quotients %ld mismatches %ld\n", n, bad);
  return bad != 0;
}
