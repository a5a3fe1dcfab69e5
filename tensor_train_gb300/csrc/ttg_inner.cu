// inner (algebra/tt_inner.hpp:33-47): the left-to-right environment chain of
// contract_inner_step (detail/contract.hpp:155-205) over the whole grid.
//
// Per core two dependent products, a grid barrier after each:
//   T (rb x n rap)  = E^T right_unfold(ca)
//   E' (rap x rbp)  = T_as(rb n x rap)^T left_unfold(cb)
// in 16 x 16 FP64 tiles, one per CTA and turn.  E' has few tiles and a long
// inner dimension, so it is cut into up to kInnerSlices ranges of it, one
// partial E' each; the next core's T adds the partials, in a fixed order, as
// it loads E.  What bounds it is the FP64 pipe (2 FMAs per clock per SM),
// then the 2 d barriers: d = 32, n = 4, rank 96 takes 0.36 GFLOP = 0.29 ms at
// the chip's FP64 rate; one CTA for the whole chain took 61.7 ms.
#include <cstdint>

#include <cuda_runtime.h>

#include "ttg_gemm_grid.cuh"
#include "ttg_gridbar.cuh"
#include "ttg_inner.h"
#include "ttg_kernels.h"

namespace ttg
{
namespace
{

constexpr int kInnerThreads = 256;
constexpr long long kInnerWaitCycles = 4000000000ll;  // ~2 s

__global__ void __launch_bounds__(kInnerThreads)
  inner_kernel(const double* __restrict__ ar, const CoreSlot* __restrict__ SA,
               const CoreSlot* __restrict__ SB, int d, double* scratch, int64_t env, GridBar* bar,
               double* out)
{
  __shared__ double sm[GridTile<1>::kDoubles];
  const int P = static_cast<int>(gridDim.x), me = static_cast<int>(blockIdx.x);
  double* E = scratch;
  double* En = scratch + env;
  double* T = scratch + 2 * env;
  // A chain of one CTA needs no barrier word (d = 300, rank 1: 2.56 -> 1.59 ms).
  auto wait_all = [&] {
    if (P > 1)
      return grid_barrier(bar, P, kInnerWaitCycles);
    __syncthreads();
    return true;
  };
  int slices = 0;  // partials of E, `size` doubles each; 0: the 1 x 1 start
  int64_t size = 0;
  for (int k = 0; k < d; ++k)
  {
    const int ra = SA[k].r, n = SA[k].n, rap = SA[k].rp;
    const int rb = SB[k].r, rbp = SB[k].rp;
    const double* ca = ar + SA[k].off;
    const double* cb = ar + SB[k].off;
    const int64_t w = static_cast<int64_t>(n) * rap;
    const int tn = static_cast<int>((w + 15) / 16);
    const int t1 = ((rb + 15) / 16) * tn;
    for (int t = me; t < t1; t += P)
      grid_tile<1>((t / tn) * 16, (t % tn) * 16, rb, static_cast<int>(w), 0, ra,
                   [&](int b, int a) {
                     if (slices == 0)
                       return 1.0;
                     const double* e = E + static_cast<int64_t>(a) * rb + b;
                     double v = __ldcg(e);
                     for (int s = 1; s < slices; ++s)
                       v += __ldcg(e + s * size);
                     return v;
                   },
                   [&](int a, int j) { return ca[a * w + j]; },
                   [&](int b, int j, double v) { T[b * w + j] = v; }, sm, false, false);
    if (!wait_all())
      return;
    const int K = rb * n;
    slices = inner_slices(rap, rbp, K, P);
    size = static_cast<int64_t>(rap) * rbp;
    const int per = (K + slices - 1) / slices;
    const int tm = (rap + 15) / 16, tn2 = (rbp + 15) / 16;
    for (int t = me; t < tm * tn2 * slices; t += P)
    {
      const int s = t / (tm * tn2), q = t % (tm * tn2);
      const int k0 = s * per, k1 = k0 + per < K ? k0 + per : K;
      double* Es = En + s * size;
      grid_tile<1>((q / tn2) * 16, (q % tn2) * 16, rap, rbp, k0, k1,
                   [&](int a, int p) { return __ldcg(T + static_cast<int64_t>(p) * rap + a); },
                   [&](int p, int b) { return cb[static_cast<int64_t>(p) * rbp + b]; },
                   [&](int a, int b, double v) { Es[static_cast<int64_t>(a) * rbp + b] = v; }, sm,
                   false, false);
    }
    if (!wait_all())
      return;
    double* x = E;
    E = En;
    En = x;
  }
  if (me == 0 && threadIdx.x == 0)
  {
    double v = __ldcg(E);
    for (int s = 1; s < slices; ++s)
      v += __ldcg(E + s * size);
    *out = v;
  }
}

}  // namespace

cudaError_t launch_inner(const double* ar, const CoreSlot* SA, const CoreSlot* SB, int d,
                         const InnerSizes& z, double* scratch, GridBar* bar, double* out,
                         cudaStream_t stream)
{
  cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(GridBar), stream);
  if (e != cudaSuccess)
    return e;
  int64_t env = z.env;
  void* args[] = {&ar, &SA, &SB, &d, &scratch, &env, &bar, &out};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(inner_kernel), dim3(z.grid),
                                     dim3(kInnerThreads), args, 0, stream);
}

}  // namespace ttg
