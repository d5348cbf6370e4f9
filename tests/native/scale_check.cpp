// scaled() of csrc/scale_f64.cuh against the processor's multiplication: random
// significands over the whole exponent range, few-bit factors whose products tie, the ends of the
// range, zero, subnormal and infinite magnitudes, and factors that take the instruction.
#include <cmath>
#include <cstdio>
#include <limits>

#include "../../com-rs_gb300/csrc/scale_f64.cuh"

static uint64_t g_state = 0x9e3779b97f4a7c15ull;
static uint64_t next() {
  uint64_t z = (g_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

int main() {
  long bad = 0, n = 0;
  auto check = [&](double alpha, double m) {
    volatile double a = alpha, b = m;
    const double want = a * b;
    const double got = cbk::scaled(cbk::make_scale(alpha), m);
    n++;
    if (cbk::sc_bits(want) != cbk::sc_bits(got) && !(std::isnan(want) && std::isnan(got))) {
      if (bad++ < 10) std::printf("alpha %a m %a: got %a want %a\n", alpha, m, got, want);
    }
  };
  const double inf = std::numeric_limits<double>::infinity();
  const double alphas[] = {0.75, 0.8, 1.0, 0.5, 0.1, 0.9999999999999999, 1.5, 3.0, 1e-300, 1e300, 2.2250738585072014e-308,
                           5e-324, 0.0, -0.75, inf, 1.7976931348623157e308, 1.0000000000000002};
  const double mags[] = {0.0, 5e-324, 2.2250738585072014e-308, 4.4501477170144023e-308, 1.0, 1.0000000000000002,
                         0.9999999999999999, 1.3333333333333333, 1.3333333333333335, 30.0, 1e308,
                         1.7976931348623157e308, inf, 6.67, 0.1};
  for (double a : alphas) {
    for (double m : mags) check(a, m);
    for (int i = 0; i < 400000; i++) {
      const uint64_t r = next();
      // a significand of 1 to 53 random bits, exponents over the whole range or near 1
      const uint64_t mant = (r & 0xfffffffffffffull) >> (next() % 53) << (next() % 2 ? 0 : next() % 52);
      const uint64_t e = i % 2 ? 1 + next() % 2046 : 1003 + next() % 40;
      check(a, cbk::sc_from_bits((e << 52) | (mant & 0xfffffffffffffull)));
    }
  }
  for (int i = 0; i < 4000000; i++) {
    const double a = cbk::sc_from_bits(((1013 + next() % 20) << 52) | (next() & 0xfffffffffffffull));
    const double m = cbk::sc_from_bits(((1003 + next() % 40) << 52) | (next() & 0xfffffffffffffull));
    check(a, m);
  }
  std::printf("%ld products, %ld differ\n", n, bad);
  return bad != 0;
}
