// FP32 bounds of the CFL screen against the FP64 formula, over random states of every magnitude. Prints the number
// of violations (a value outside its bounds, or a lower bound where the formula gives NaN), of states, and of
// states with tight bounds (hi < 1.0001 lo).
#include <cstdio>
#include <random>

#include "host_device_shim.h"

#include "../../godunov_mhd_ct_gb300/csrc/cfl_screen.cuh"

int
main()
{
  std::mt19937_64                        g(12345);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  long bad = 0, n = 0, tight = 0;
  auto mag = [&](double lo, double hi) { return std::pow(10.0, lo + (hi - lo) * (0.5 + 0.5 * U(g))); };
  for (int dim = 2; dim <= 3; ++dim)
    for (int kind = 0; kind < 8; ++kind)
      for (int it = 0; it < 20000; ++it)
      {
        const double gamma0 = kind == 5 ? 1.0 + mag(-8, -1) : 1.1 + 0.9 * std::fabs(U(g));
        const double smallr = 1e-10, smallc = 1e-10, smallp = smallc * smallc / gamma0;
        double       rho = mag(-2, 2), p = mag(-3, 3), vs = mag(-3, 2), bs = mag(-3, 2);
        if (kind == 1)
          p = mag(-9, -4), bs = mag(0, 2); // low beta
        if (kind == 2)
          bs = 0.0;
        if (kind == 3)
          rho = mag(-30, 30), p = mag(-30, 30), vs = mag(-30, 30), bs = mag(-30, 30);
        double f[6], u[5];
        for (int d = 0; d < 3; ++d)
        {
          const double b = bs * U(g);
          f[2 * d] = b + (kind == 4 ? 1e3 * bs : 1e-3 * bs * U(g));
          f[2 * d + 1] = b - (kind == 4 ? 1e3 * bs : 1e-3 * bs * U(g));
        }
        if (kind == 6) // field along one axis, sound and Alfven speed nearly equal: vanishing discriminant
        {
          const int d = it % 3;
          for (int e = 0; e < 3; ++e)
            f[2 * e] = f[2 * e + 1] = e == d ? std::sqrt(gamma0 * p) * (1.0 + (it % 2) * 1e-9 * U(g)) : 0.0;
        }
        if (dim == 2)
          f[5] = f[4];
        const double v[3] = {vs * U(g), vs * U(g), vs * U(g)};
        double       b2 = 0, v2 = 0;
        for (int d = 0; d < 3; ++d)
        {
          const double c = 0.5 * (f[2 * d] + f[2 * d + 1]);
          b2 += c * c;
          v2 += v[d] * v[d];
          u[2 + d] = rho * v[d];
        }
        u[0] = rho;
        u[1] = p / (gamma0 - 1.0) + 0.5 * rho * v2 + 0.5 * b2;
        if (kind == 7 && it % 4 == 0)
          u[it % 5] = it % 8 == 0 ? NAN : -u[it % 5];
        gmhd::Sources src{};
        if (it % 3 == 1)
        {
          src.gravity = 1;
          for (double & x : src.g)
            x = mag(-4, 4) * U(g);
        }
        if (it % 5 == 1)
        {
          src.viscosity = 1;
          src.mu = mag(-6, 2);
        }
        const double dx = 1.0 / (16 << (it % 9));
        // a one-cell block with these faces
        const int    bz = dim == 3 ? 2 : 1;
        double       Bb[8] = {f[0], f[1], f[2], f[3], f[4], f[5], 0, 0};
        const double val = gmhd::cell_inv_dt_fp64(u, Bb, dim, 1, 1, 0, 0, 0, 0, 1, 2, 2, dx, gamma0, smallr, smallp, src);
        const auto   b = gmhd::cell_inv_dt_bounds(u, f, dim, (float)(1.0 / dx), (float)gamma0, (float)(gamma0 - 1.0),
                                                  (float)smallr, (float)smallp, src);
        (void)bz;
        ++n;
        if (std::isnan(val) ? !(b.lo <= 0.0f) : !(b.lo <= val && val <= b.hi))
          ++bad;
        if (b.hi < 1.0001f * b.lo)
          ++tight;
      }
  std::printf("%ld %ld %ld\n", bad, n, tight);
  return 0;
}
