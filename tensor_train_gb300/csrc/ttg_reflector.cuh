// FP64 pieces shared by the blocked Householder routines (ttg_wide_qr.cuh,
// ttg_wy.cuh): the scalars of a reflector, the reduction of a block's 16
// products and the columns of its T.
#pragma once

#include <cfloat>
#include <cuda_runtime.h>

namespace ttg
{
namespace
{

// The scalars of a reflector from s = x0^2 + |tail|^2 and ax = |x0|:
// n = |x|, rs = 1 / n, inv = 1 / (ax + n).  One third-order step
// (Householder's iteration: the error of the start cubed) from the hardware's
// approximations of the reciprocal root and the reciprocal, which hold at
// least 20 bits.  Before the last rounding that leaves 2^-58 of n and rs (e up
// to 2^-19, 5/16 e^3 dropped) and 2^-57 of inv (f up to 2^-19, f^3 dropped, and
// f's own rounding, 2^-54): each within 1.1 (n, rs) and 2.6 (inv) of 2^-53.
// What counts is the number of FP64 instructions (64 clocks each) that every
// other thread waits for: with the library's root and two divisions the step
// took 1.39 us per column, with these 0.6 us; the term that t's rounding leaves
// out of e is one of them (without it n and rs are off by 1.5 and 1.2; d=15
// rank-83 round 8.8 -> 9.0 ms).
__device__ __forceinline__ void reflector_scalars(double s, double ax, double* n, double* rs,
                                                  double* inv)
{
  double y, r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
  const double t = s * y;  // ~n
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(ax + t));
  const double d = fma(s, y, -t);
  // e = 1 - s y^2, with what the rounding of t left out:
  // n = s y (1 - e)^(-1/2), rs = y (1 - e)^(-1/2).
  const double e = fma(-d, y, fma(-t, y, 1.0));
  const double q = e * fma(0.375, e, 0.5);
  *n = t + fma(t, q, d);
  *rs = fma(y, q, y);
  const double f = fma(-*n, r, fma(-ax, r, 1.0));  // 1 / (ax + n) = r (1 + f + f^2 + ...)
  *inv = fma(r, fma(f, f, f), r);
}

// Sign and magnitude tests on the bit patterns: a comparison of doubles is an
// instruction of the FP64 pipe too.
__device__ __forceinline__ bool not_negative(double x)  // -0.0 counts as 0
{
  const long long b = __double_as_longlong(x);
  return b >= 0 || (b << 1) == 0;
}
// Whether a column has anything below its diagonal: tail2 > DBL_MIN for a sum
// of squares, and true for a NaN of either sign (inf - inf is 0xfff8... on a
// host), so that it reaches R and the norm.
__device__ __forceinline__ bool has_tail(double tail2)
{
  return (__double_as_longlong(tail2) & 0x7fffffffffffffffll) > __double_as_longlong(DBL_MIN);
}
__device__ __forceinline__ double copy_sign(double mag, bool positive)
{
  return __longlong_as_double(__double_as_longlong(mag) ^ (positive ? 0ll : (1ll << 63)));
}

// Sums of 16 values over the G lanes of a group by halving: lane gl ends with
// value(s) i0 .. i0 + max(16 / G, 1) in acc[0..].
template <int G>
__device__ __forceinline__ void halving_sum(double (&acc)[16], int gl)
{
  int o = G / 2;
#pragma unroll
  for (int n = 8; n >= 1; n >>= 1)
  {
    if (o == 0)
      break;
    const bool up = (gl & o) != 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i < n)
      {
        const double keep = up ? acc[i + n] : acc[i];
        const double send = up ? acc[i] : acc[i + n];
        acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    o >>= 1;
  }
  if (G == 32)
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
}

// Column i of a block's T = -tau_i T(0:i, 0:i) G(0:i, i), T(i, i) = tau_i, by
// the 32 lanes of a warp; G = V^T V above the diagonal, T upper triangular,
// both 16 x 16 and column-major in ps.
template <class Shared>
__device__ __forceinline__ void t_column(Shared& ps, int i)
{
  constexpr int kB = 16;
  static_assert(sizeof(ps.T) == kB * kB * sizeof(double), "16 reflectors per block");
  // Two lanes per row, each half of the sum.
  const int lane = threadIdx.x & 31, l = lane & (kB - 1), half = lane / kB;
  const double nt = -ps.tau[i];
  const double g = nt * ps.G[l + i * kB];  // lane q's term is -tau_i G(q, i)
  double acc = 0.0;
  for (int q0 = 0; q0 < i; q0 += 2)  // the same trips on every lane
  {
    const int q = q0 + half;
    const double gq = __shfl_sync(0xffffffffu, g, q);
    if (l <= q && q < i)
      acc = fma(ps.T[l + q * kB], gq, acc);
  }
  acc += __shfl_xor_sync(0xffffffffu, acc, kB);
  if (half == 0)
    ps.T[l + i * kB] = l < i ? acc : (l == i ? -nt : 0.0);
  __syncwarp();
}

}  // namespace
}  // namespace ttg
