// Host check of the fixed-point power (meshcfd_gb300/csrc/mcfd_pow.cuh
// compiled as plain C++) against the C library's long double powl.
//
// usage: pow_check N SEED  -> prints "cases=<n> worst=<ulp> fallback=<n>";
// the error is in units in the last place of the result.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../meshcfd_gb300/csrc/mcfd_pow.cuh"

static unsigned long long g_state;
static double uniform() {
  unsigned long long z = (g_state += 0x9e3779b97f4a7c15ull);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return (double)((z ^ (z >> 31)) >> 11) * 0x1p-53;
}

static double ulp_of(long double v) {
  int e;
  std::frexp((double)v, &e);
  return std::ldexp(1.0, e - 53);
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 100000;
  g_state = argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1;
  // exponents the solver takes, and spreads up to each stated bound
  const double fixed[] = {1.4, 1.0 / (1.4 - 1.0), 1.4 / (1.4 - 1.0), 1.5, 0.4, 5.0 / 3.0, -1.0, 2.0, 1.0, -0.5};
  double worst8 = 0.0, worst64 = 0.0;
  long bad = 0;
  for (long i = 0; i < n; ++i) {
    const int kind = (int)(i % 4);
    // near 1, over a few binades, over the whole range the exponent allows
    double y = i % 3 == 0 ? fixed[(i / 3) % 10] : (uniform() - 0.5) * (i % 3 == 1 ? 16.0 : 128.0);
    double span = kind == 0 ? 0.001 : kind == 1 ? 1.0 : kind == 2 ? 20.0 : 1000.0;
    span = std::fmin(span, 1000.0 / (std::fabs(y) + 1.0));
    const double x = std::exp2((2.0 * uniform() - 1.0) * span);
    const double r = mcfd::pow_rn(x, y);
    const long double e = powl((long double)x, (long double)y);
    const double err = (double)fabsl((long double)r - e) / ulp_of(e);
    if (!(err < 1.0)) ++bad;
    double& w = std::fabs(y) <= 8.0 ? worst8 : worst64;
    if (err > w) w = err;
  }
  // exact cases and everything the fixed-point path leaves to pow
  const double xs[] = {1.0, 2.0, 4.0, 0.25, 0.0, -0.0, -2.0, 5e-324, 1e-310, 1e308, HUGE_VAL, -HUGE_VAL, NAN};
  const double ys[] = {1.0, 2.0, -1.0, 0.5, 0.0, -0.0, 64.0, 65.0, 1000.0, 0x1p-41, HUGE_VAL, -HUGE_VAL, NAN, 3.0};
  for (double x : xs)
    for (double y : ys) {
      const double r = mcfd::pow_rn(x, y), e = std::pow(x, y);
      if (!(r == e || (std::isnan(r) && std::isnan(e)))) {
        ++bad;
        std::printf("x=%a y=%a: %a, pow %a\n", x, y, r, e);
      }
    }
  std::printf("cases=%ld bad=%ld worst8=%.4f worst64=%.4f\n", n, bad, worst8, worst64);
  return bad ? 1 : 0;
}
