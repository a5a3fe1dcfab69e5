// Host check of the rotation of the df64 Jacobi sweeps (df_rotation,
// ttg_df64.cuh) against long double, over angles from 1 to 1e-13, norms down to
// 1e-10 of one another, equal and nearly equal columns and both signs.
//
// Bounds, u = 2^-24.  c^2 + s^2 with s = df_mul(c, tan) (5 u^2 of itself, of
// which s^2 <= 1/2 counts twice: 5 u^2) and a cosine whose residual e is formed
// from exact sums and products with four roundings of terms below u (2 u^2,
// half of it in c) and whose last sum rounds a term below u / 2 (u^2 / 2, and as
// much from the df64 it is added to): 2 (u^2 + u^2) + 5 u^2 = 9 u^2.  The
// tangent: its FP32 start is off by 4 u, which a Newton step squares (times at
// most 1/2: 8 u^2), and its quotient and slope round the correction (4 u times
// 3 u: 12 u^2): 20 u^2.
#include <cmath>
#include <cstdio>
#include <random>

#include "ttg_df64.cuh"

using namespace ttg;

static long double value(df64 a) { return static_cast<long double>(a.hi) + a.lo; }

int main()
{
  std::mt19937_64 g(1);
  std::uniform_real_distribution<double> unit(0.0, 1.0);
  std::normal_distribution<double> normal;
  const long double u2 = ldexpl(1.0L, -48);
  long double worst_t = 0.0L, worst_c = 0.0L;
  for (int it = 0; it < 2000000; ++it)
  {
    const double a = std::pow(10.0, -10.0 * unit(g));
    double b = std::pow(10.0, -10.0 * unit(g));
    if (it % 3 == 0)
      b = a * (1.0 + std::pow(10.0, -15.0 * unit(g)) * std::fabs(normal(g)));
    if (it % 7 == 0)
      b = a;
    const df64 al = df_split_pow2(a, 0), be = df_split_pow2(b, 0);
    const df64 ga = df_split_pow2(
      std::sqrt(a * b) * std::pow(10.0, -13.0 * unit(g)) * (unit(g) < 0.5 ? -1.0 : 1.0), 0);
    df64 tan, c;
    df_rotation(al, be, ga, &tan, &c);
    const df64 s = df_mul(c, tan);
    const long double z = (value(be) - value(al)) / (2.0L * value(ga));
    const long double T = (z >= 0.0L ? 1.0L : -1.0L) / (fabsl(z) + sqrtl(1.0L + z * z));
    worst_t = fmaxl(worst_t, fabsl(value(tan) / T - 1.0L));
    worst_c = fmaxl(worst_c, fabsl(value(c) * value(c) + value(s) * value(s) - 1.0L));
  }
  const bool ok = worst_c <= 9.0L * u2 && worst_t <= 20.0L * u2;
  std::printf("%s: tangent off by %.2Lf u^2, c^2 + s^2 by %.2Lf u^2\n", ok ? "OK" : "FAILED",
              worst_t / u2, worst_c / u2);
  return ok ? 0 : 1;
}
