// The exact path's slopes, HLLD fluxes and edge EMFs (csrc/exact_solvers.cuh) against the oracle's formulas: equal
// values (NaN for NaN, zeros of either sign). Prints mismatches, comparisons.
#include <cstdio>
#include <random>

#include "host_device_shim.h"
using std::fma;

#include "../../godunov_mhd_ct_gb300/csrc/exact_solvers.cuh"
#include "../../oracle/oracle_models.h"

static long bad = 0, n = 0;
static bool
same(double x, double y)
{
  ++n;
  const bool ok = x == y || (std::isnan(x) && std::isnan(y));
  bad += !ok;
  return ok;
}

int
main(int argc, char ** argv)
{
  const long                             reps = argc > 1 ? std::atol(argv[1]) : 30000;
  std::mt19937_64                        g(99);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  host_seed_units = 1;
  auto mag = [&](double lo, double hi) { return std::pow(10.0, lo + (hi - lo) * (0.5 + 0.5 * U(g))); };
  const double eps[] = {0.5, 1e-1, 1e-2, 1e-3, 1e-5, 1e-6, 1e-7, 1e-9, 1e-15, 0.0};
  for (int kind = 0; kind < 10; ++kind)
    for (long it = 0; it < reps; ++it)
    {
      const double e = eps[it % 10];
      double       rho = mag(-2, 2), p = mag(-2, 2), vs = mag(-2, 1), bs = mag(-2, 1);
      if (kind == 1)
        p = mag(-9, -4); // low beta
      if (kind == 2)
        vs = mag(1, 3); // supersonic: the fan on one side of the edge
      if (kind == 3)
        bs = 0.0;
      if (kind == 4)
        rho = mag(-9, 9), p = mag(-9, 9), vs = mag(-9, 9), bs = mag(-9, 9); // any scale and ratio
      double base[8] = {rho, p, vs * U(g), vs * U(g), vs * U(g), bs * U(g), bs * U(g), bs * U(g)};
      if (kind == 5)
        base[5 + it % 3] = base[5 + (it / 3) % 3] = 0.0;
      if (kind == 6) // the field along one axis, Alfven speed equal to the sound speed
      {
        base[5] = base[6] = base[7] = 0.0;
        base[5 + it % 3] = std::sqrt(5.0 / 3.0 * p);
      }
      if (kind == 7)
        base[2] = base[3] = base[4] = 0.0;
      const oracle::Settings s = oracle::make_settings(it % 2 ? 5.0 / 3.0 : 1.4, 0.5, 2.0, 1e-10, kind == 8 ? 0.3 : 1e-10, 5);
      double                 qe[4][8];
      for (auto & q : qe)
        for (int v = 0; v < 8; ++v)
        {
          q[v] = base[v] + e * (v < 2 ? base[v] * 0.9 * U(g) : (v < 5 ? vs : bs) * U(g));
          if (kind == 5 && base[v] == 0.0)
            q[v] = 0.0;
        }
      if (kind == 9 && it % 3 == 0)
        qe[it % 4][it % 8] = it % 2 ? NAN : -qe[it % 4][it % 8];
      for (int dir = 0; dir < 3; ++dir)
      {
        const int    iu = dir == 2 ? 2 : (dir == 1 ? 4 : 3), iv = dir == 2 ? 3 : (dir == 1 ? 2 : 4);
        const int    ia = dir == 2 ? 5 : (dir == 1 ? 7 : 6), ib = dir == 2 ? 6 : (dir == 1 ? 5 : 7), ic = dir == 2 ? 7 : (dir == 1 ? 6 : 5);
        const double *RT = qe[0], *LT = qe[1], *RB = qe[2], *LB = qe[3];
        const double *st[4] = {RT, RB, LT, LB};
        double       r[4], pp[4], u[4], v[4], c[4];
        for (int k = 0; k < 4; ++k)
        {
          r[k] = st[k][0];
          pp[k] = st[k][1];
          u[k] = st[k][iu];
          v[k] = st[k][iv];
          c[k] = st[k][ic];
        }
        const double got = gmhd::edge_emf_fp64(r, pp, u, v, c, 0.5 * (RT[ia] + LT[ia]), 0.5 * (RB[ia] + LB[ia]), 0.5 * (RT[ib] + RB[ib]),
                                               0.5 * (LT[ib] + LB[ib]), s.gamma0, s.smallc);
        const double want = oracle::compute_emf(qe, dir, s);
        if (!same(got, want) && bad < 30)
          std::fprintf(stderr, "emf kind %d eps %g dir %d: %a not %a\n", kind, e, dir, got, want);
      }
      double l1[8], r1[8], l2[8], r2[8], f1[8], f2[8];
      for (int v = 0; v < 8; ++v)
      {
        l1[v] = l2[v] = qe[0][v];
        r1[v] = r2[v] = qe[1][v];
      }
      l1[5] = l2[5] = r1[5] = r2[5];
      gmhd::riemann_hlld_fp64(l1, r1, f1, s.gamma0, 1.0 / (s.gamma0 - 1.0));
      oracle::riemann_hlld(l2, r2, f2, s);
      for (int v = 0; v < 8; ++v)
        if (!same(f1[v], f2[v]) && bad < 30)
          std::fprintf(stderr, "flux kind %d eps %g var %d: %a not %a\n", kind, e, v, f1[v], f2[v]);
      for (int v = 0; v < 8; ++v)
        for (double st : {1.0, 2.0, 3.0})
          same(gmhd::slope1_fp64(qe[0][v], qe[1][v], qe[2][v], st), st > 2.0 ? 0.0 : gmhd::slow_slope(qe[0][v], qe[1][v], qe[2][v], st));
    }
  std::printf("%ld %ld\n", bad, n);
  return 0;
}
