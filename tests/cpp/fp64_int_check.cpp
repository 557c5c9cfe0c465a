// The integer forms of FP64 operations against the CPU's FP64 unit, bit for bit. Prints mismatches and the number of
// comparisons.
#include <cstdio>
#include <random>

#include "host_device_shim.h"

#include "../../godunov_mhd_ct_gb300/csrc/fp64_int.cuh"

using namespace gmhd;

static long bad = 0, n = 0;
static void
same(double got, double want, const char * what, double x, double y)
{
  ++n;
  const bool eq = std::isnan(want) ? std::isnan(got) : __double_as_longlong(got) == __double_as_longlong(want);
  if (!eq && ++bad <= 10)
    std::fprintf(stderr, "%s(%a, %a) = %a, not %a\n", what, x, y, got, want);
}

int
main(int argc, char ** argv)
{
  const long      reps = argc > 1 ? std::atol(argv[1]) : 400000;
  std::mt19937_64 g(2024);
  const double    edge[] = {0.0, -0.0, 1.0, -1.0, 2.0, 0.5, 3.0, 1e-300, 1e300, 2.2250738585072014e-308, 5e-324, INFINITY, -INFINITY, NAN,
                            1.7976931348623157e308, 1.0 + 2.220446049250313e-16, 2.0 - 2.220446049250313e-16, 4.0 - 4.440892098500626e-16, 1e-160, -1e160};
  auto            check = [&](double x, double y) {
    same(div64(x, y), x / y, "div", x, y);
    same(sqrt64(x), std::sqrt(x), "sqrt", x, 0);
    same(dmax(x, y), x == y ? dmax(x, y) : std::fmax(x, y), "max", x, y);
    same(dmin(x, y), x == y ? dmin(x, y) : std::fmin(x, y), "min", x, y);
    same(dpos(x), x > 0, "pos", x, 0);
    same(dgt(x, y), x > y, "gt", x, y);
    for (unsigned k = 1; k <= 3; ++k)
      same(dscale_down(x, k), std::ldexp(1.0, -(int)k) * x, "scale", x, k);
  };
  for (host_seed_units = 0; host_seed_units <= 2; ++host_seed_units)
  {
    const int units = host_seed_units;
    for (double x : edge)
      for (double y : edge)
        check(x, y);
    for (long i = 0; i < reps; ++i)
    {
      const uint64_t a = g(), b = g();
      // any bit pattern; then significands of ones, zeros and random bits with moderate exponents
      double x = __longlong_as_double((long long)a), y = __longlong_as_double((long long)b);
      host_seed_units = std::min(units, 1);
      check(x, y);
      auto pat = [&](uint64_t r) {
        uint64_t m = r & 0xfffffffffffffull;
        switch ((r >> 52) & 7)
        {
          case 0: m &= (1ull << (r >> 58)) - 1; break;
          case 1: m |= ~((1ull << ((r >> 58) % 52)) - 1) & 0xfffffffffffffull; break;
          case 2: m = 0xfffffffffffffull - (r & 3); break;
          case 3: m = r & 3; break;
          default: break;
        }
        return __longlong_as_double((long long)(((1013 + ((r >> 55) & 15)) << 52) | m));
      };
      x = pat(g());
      y = pat(g());
      check(x, y);
      same(div64(x * y, y), (x * y) / y, "div", x * y, y);
      // nearly equal significands: quotients next to a power of two
      const double z = __longlong_as_double(__double_as_longlong(x) + (long long)(g() % 9) - 4);
      same(div64(x, z), x / z, "div", x, z);
      host_seed_units = units;
      same(sqrt64(x * x), std::sqrt(x * x), "sqrt", x * x, 0);
      const double w = x * x, wn = __longlong_as_double(__double_as_longlong(w) + (long long)(g() % 5) - 2);
      same(sqrt64(wn), std::sqrt(wn), "sqrt", wn, 0);
      same(sqrt64(y), std::sqrt(y), "sqrt", y, 0);
    }
  }
  std::printf("%ld %ld\n", bad, n);
  return 0;
}
