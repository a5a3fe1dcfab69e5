// FP64 output tiles for products that are spread over the grid.
//
// GB300 retires 2 FP64 FMAs per clock per SM, so a tile is bound by its own
// FMAs whatever its shape (a warp's FMA holds its pipe for 64 clocks, its two
// shared-memory reads take 4); what a tile's size decides is how evenly the
// product spreads over 152 SMs.  Tiles are therefore small (16 R x 16 R, R =
// 1 or 2), and K slabs are double-buffered: the next slab's loads are in
// flight while this one is multiplied, one barrier per slab.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ttg
{
namespace
{

template <int R>
struct GridTile
{
  static constexpr int kT = 16 * R;       // tile rows and columns
  static constexpr int kK = 32 / R;       // slab depth: 512 elements per operand
  static constexpr int kLd = kT + 1;      // odd: conflict-free writes along k
  static constexpr int kDoubles = 4 * kK * kLd;  // two operands, two buffers
};

// C(i, j) = sum_{k0 <= p < k1} a(i, p) b(p, j) on the tile at (i0, j0), by
// 256 threads: thread (ty, tx) holds rows ty + 16 r and columns tx + 16 s.
// a and b are called inside the matrix only; store(i, j, value) likewise.
// a_kfast / b_kfast: consecutive threads load along p (the operand's
// contiguous direction) instead of along i / j.  The terms are added in
// ascending p.  sm: GridTile<R>::kDoubles doubles of shared memory.
template <int R, class FA, class FB, class FC>
__device__ __forceinline__ void grid_tile(int i0, int j0, int M, int N, int k0, int k1, FA a, FB b,
                                          FC store, double* sm, bool a_kfast, bool b_kfast)
{
  using G = GridTile<R>;
  constexpr int T = G::kT, KS = G::kK, LD = G::kLd;
  const int t = threadIdx.x;
  const int tx = t & 15, ty = t >> 4;
  double* As = sm;
  double* Bs = sm + 2 * KS * LD;
  // Element e of this thread's two per operand and slab.
  int ai[2], ap[2], bj[2], bp[2];
#pragma unroll
  for (int e = 0; e < 2; ++e)
  {
    const int q = t + 256 * e;
    ai[e] = a_kfast ? q / KS : q % T;
    ap[e] = a_kfast ? q % KS : q / T;
    bj[e] = b_kfast ? q / KS : q % T;
    bp[e] = b_kfast ? q % KS : q / T;
  }
  double ra[2], rb[2];
  auto load = [&](int p0) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
    {
      ra[e] = (i0 + ai[e] < M && p0 + ap[e] < k1) ? a(i0 + ai[e], p0 + ap[e]) : 0.0;
      rb[e] = (j0 + bj[e] < N && p0 + bp[e] < k1) ? b(p0 + bp[e], j0 + bj[e]) : 0.0;
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int e = 0; e < 2; ++e)
    {
      As[(buf * KS + ap[e]) * LD + ai[e]] = ra[e];
      Bs[(buf * KS + bp[e]) * LD + bj[e]] = rb[e];
    }
  };
  double acc[R][R];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int s = 0; s < R; ++s)
      acc[r][s] = 0.0;
  __syncthreads();  // the buffers may still be read by the tile before
  if (k0 < k1)
  {
    load(k0);
    put(0);
  }
  __syncthreads();
  int buf = 0;
  for (int p0 = k0; p0 < k1; p0 += KS, buf ^= 1)
  {
    const bool more = p0 + KS < k1;
    if (more)
      load(p0 + KS);
    const int kmax = k1 - p0 < KS ? k1 - p0 : KS;
    const double* A0 = As + buf * KS * LD + ty;
    const double* B0 = Bs + buf * KS * LD + tx;
#pragma unroll 8
    for (int kk = 0; kk < kmax; ++kk)
    {
      double av[R], bv[R];
#pragma unroll
      for (int r = 0; r < R; ++r)
      {
        av[r] = A0[kk * LD + 16 * r];
        bv[r] = B0[kk * LD + 16 * r];
      }
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int s = 0; s < R; ++s)
          acc[r][s] = fma(av[r], bv[s], acc[r][s]);
    }
    if (more)
    {
      put(buf ^ 1);
      __syncthreads();
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int s = 0; s < R; ++s)
    {
      const int i = i0 + ty + 16 * r, j = j0 + tx + 16 * s;
      if (i < M && j < N)
        store(i, j, acc[r][s]);
    }
}

}  // namespace
}  // namespace ttg
