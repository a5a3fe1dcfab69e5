// Blocked (compact WY) Householder QR, Q formation and Q application of one
// CTA in FP64, for matrices whose panels fit its shared memory.  Same
// reflectors and convention as cta_householder_qr / cta_form_q / cta_apply_q.
//
// A warp's FP64 instruction holds its pipe for 64 clocks, which is also its
// latency, so a column's cost is the number of such instructions on the path
// through it.  The unblocked routines spend them on a CTA-wide norm, a root
// and two divisions on one thread, and a reduction per trailing column and
// reflector.  Here a column's norm, its products with the later columns of
// its panel and the entries of V^T V come from one pass of 8 lanes per panel
// column; the scalars are reflector_scalars; the trailing columns take kWb
// reflectors at a time with one reduction of kWb values; and Q's own columns
// of a block are one small product, -V (T V1^T), instead of kWb dependent
// updates.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ttg_device.cuh"
#include "ttg_reflector.cuh"

namespace ttg
{
namespace
{

constexpr int kWb = 16;  // reflectors per block

struct WyShared
{
  double d[kWb], row[kWb], w[kWb], inv[kWb], tau[kWb];
  double G[kWb * kWb];  // V^T V above the diagonal
  double T[kWb * kWb];  // column-major, upper triangular
};
static_assert(sizeof(WyShared) <= sizeof(CtaShared::gemm_a), "staged in the GEMM buffers");
constexpr int kWyCols = 32;  // columns per pass of an application
static_assert(2 * kWyCols * kWb * sizeof(double) <= sizeof(CtaShared::gemm_b), "");

// Doubles of shared memory for the blocks' T of c reflectors.
__device__ __forceinline__ int64_t wy_t_need(int c)
{
  return static_cast<int64_t>((c + kWb - 1) / kWb) * kWb * kWb;
}

// Householder factorisation of P (hp x nb, nb <= kWb, ld ldp) in place: R on
// and above the diagonal, the unscaled tails below (v_i = inv_i x_i).  ps:
// inv, tau and T of the block (zero past nb).  Ends with a barrier.
__device__ __noinline__ void wy_panel(double* P, int64_t ldp, int hp, int nb, WyShared& ps)
{
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (int e = t; e < kWb * kWb; e += kThreads)
    ps.T[e] = 0.0;
  __syncthreads();
  for (int i = 0; i < nb; ++i)
  {
    const double* x = P + i * ldp;
    if (t < 8 * kWb)
    {
      const int l = t >> 3, g = t & 7;
      double a = 0.0;
      if (l < nb)
      {
        const double* y = P + l * ldp;
        for (int r = i + 1 + g; r < hp; r += 8)
          a = fma(x[r], y[r], a);
      }
      a += __shfl_xor_sync(0xffffffffu, a, 4);
      a += __shfl_xor_sync(0xffffffffu, a, 2);
      a += __shfl_xor_sync(0xffffffffu, a, 1);
      if (g == 0 && l < nb)
      {
        ps.d[l] = a;
        ps.row[l] = P[l * ldp + i];
      }
    }
    else if (w == 6 && i > 0)
      t_column(ps, i - 1);
    __syncthreads();
    // tau inv = +-1 / n: warp 0 forms what the update waits for, warps 1 and
    // 2 (on other pipes, the same scalars again) the rest.
    if (w < 3)
    {
      const double tail2 = ps.d[i], x0 = ps.row[i];
      const bool up = not_negative(x0);
      double beta = x0, tau = 0.0, inv = 0.0, wi = 0.0;
      if (has_tail(tail2))
      {
        double n, rs;
        const double ax = fabs(x0);
        reflector_scalars(fma(x0, x0, tail2), ax, &n, &rs, &inv);
        inv = copy_sign(inv, up);
        wi = copy_sign(rs, up);
        beta = copy_sign(n, !up);
        tau = fma(ax, rs, 1.0);  // (n + |x0|) / n
      }
      const int l = lane < nb ? lane : 0;
      const double dot = fma(inv, ps.d[l], ps.row[l]);
      if (w == 0)
      {
        if (lane > i && lane < nb)
          ps.w[lane] = dot * wi;
      }
      else if (w == 1)
      {
        if (lane > i && lane < nb)
          P[lane * ldp + i] = fma(-tau, dot, ps.row[lane]);
        if (lane == i)
          P[i * ldp + i] = beta;
      }
      else
      {
        // G(l, i) = v_l . v_i, v_l = inv_l x_l (row i of x_l is in ps.row).
        if (lane < i)
          ps.G[lane + i * kWb] = ps.inv[lane] * dot;
        if (lane == i)
        {
          ps.inv[i] = inv;
          ps.tau[i] = tau;
        }
      }
    }
    __syncthreads();
    for (int l = i + 1 + w; l < nb; l += kWarps)
    {
      const double f = -ps.w[l];
      double* y = P + l * ldp;
      for (int r = i + 1 + lane; r < hp; r += 32)
        y[r] = fma(f, x[r], y[r]);
    }
    __syncthreads();
  }
  if (w == 6)
    t_column(ps, nb - 1);
  __syncthreads();
}

// B(0:hp, 0:ncols) <- (I - V T' V^T) B, T' = T^T (kTrans) or T; V explicit
// (hp x kWb, ld ldv, zero past nb), T in shared memory.  G lanes per column.
// Ends with a barrier.
template <int G, bool kTrans>
__device__ __forceinline__ void wy_apply_g(const double* V, int64_t ldv, int nb, int hp,
                                           const double* T, double* B, int64_t ldb, int ncols,
                                           double* Ws, double* Zs)
{
  const int t = threadIdx.x, gl = t & (G - 1), q0 = t / G;
  constexpr int kCols = kThreads / G;
  const int i0 = G == 32 ? gl >> 1 : gl * (kWb / G > 0 ? kWb / G : 1);
  constexpr int kEach = kWb / G > 0 ? kWb / G : 1;
  for (int qb = 0; qb < ncols; qb += kCols)
  {
    const int q = qb + q0;
    const int here = ncols - qb < kCols ? ncols - qb : kCols;
    double* y = B + (q < ncols ? q : qb) * ldb;
    double acc[kWb];
#pragma unroll
    for (int i = 0; i < kWb; ++i)
      acc[i] = 0.0;
    if (q < ncols)
      for (int r = gl; r < hp; r += G)
      {
        const double b = y[r];
#pragma unroll
        for (int i = 0; i < kWb; ++i)
          if (i < nb)
            acc[i] = fma(V[i * ldv + r], b, acc[i]);
      }
    halving_sum<G>(acc, gl);
    if (q < ncols)
    {
#pragma unroll
      for (int e = 0; e < kEach; ++e)
        if (G < 32 || (gl & 1) == 0)
          Ws[q0 * kWb + i0 + e] = acc[e];
    }
    __syncthreads();
    for (int e = t; e < here * kWb; e += kThreads)
    {
      const int i = e % kWb;
      const double* wq = Ws + (e - i);
      double z = 0.0;
#pragma unroll
      for (int l = 0; l < kWb; ++l)
        if (l < nb)
          z = fma(kTrans ? T[l + i * kWb] : T[i + l * kWb], wq[l], z);
      Zs[e] = z;
    }
    __syncthreads();
    if (q < ncols)
    {
      double z[kWb];
#pragma unroll
      for (int i = 0; i < kWb; ++i)
        z[i] = -Zs[q0 * kWb + i];
      for (int r = gl; r < hp; r += G)
      {
        double b = y[r];
#pragma unroll
        for (int i = 0; i < kWb; ++i)
          if (i < nb)
            b = fma(z[i], V[i * ldv + r], b);
        y[r] = b;
      }
    }
  }
  __syncthreads();
}

template <bool kTrans>
__device__ __noinline__ void wy_apply(const double* V, int64_t ldv, int nb, int hp, const double* T,
                                      double* B, int64_t ldb, int ncols, CtaShared& sh)
{
  double* Ws = &sh.gemm_b[0][0];
  double* Zs = Ws + kWyCols * kWb;
  // As few lanes per column as keep all 256 threads at work.
  if (ncols > 16)
    wy_apply_g<8, kTrans>(V, ldv, nb, hp, T, B, ldb, ncols, Ws, Zs);
  else if (ncols > 8)
    wy_apply_g<16, kTrans>(V, ldv, nb, hp, T, B, ldb, ncols, Ws, Zs);
  else
    wy_apply_g<32, kTrans>(V, ldv, nb, hp, T, B, ldb, ncols, Ws, Zs);
}

// QR of W (h x c, column-major, ld h): on return column j < k = min(h, c)
// holds the explicit v_j from its block's first row on, Ts (shared memory,
// wy_t_need(k)) the blocks' T, R (k x c, column-major, ld k) the triangle.
// stage: null when W is in shared memory, else room for h kWb doubles there.
__device__ __noinline__ void cta_qr_wy(double* W, int h, int c, double* R, double* Ts,
                                       double* stage, CtaShared& sh)
{
  const int k = h < c ? h : c;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  WyShared& ps = *reinterpret_cast<WyShared*>(&sh.gemm_a[0][0]);
  for (int j0 = 0; j0 < k; j0 += kWb)
  {
    const int nb = k - j0 < kWb ? k - j0 : kWb, hp = h - j0;
    double* P = stage ? stage : W + static_cast<int64_t>(j0) * h + j0;
    const int64_t ldp = stage ? hp : h;
    if (stage)
    {
      for (int i = w; i < nb; i += kWarps)
        for (int r = lane; r < hp; r += 32)
          P[i * ldp + r] = W[static_cast<int64_t>(j0 + i) * h + j0 + r];
      __syncthreads();
    }
    wy_panel(P, ldp, hp, nb, ps);
    // R's columns j0 .. j0 + nb, then the explicit V in their place.
    for (int i = w; i < nb; i += kWarps)
    {
      const int64_t j = j0 + i;
      for (int r = lane; r < k; r += 32)
        R[r + j * k] = r < j0 ? W[j * h + r] : (r <= j ? P[i * ldp + r - j0] : 0.0);
      __syncwarp();
      const double inv = ps.inv[i];
      for (int r = lane; r < hp; r += 32)
      {
        const double v = r < i ? 0.0 : (r == i ? 1.0 : inv * P[i * ldp + r]);
        P[i * ldp + r] = v;
        if (stage)
          W[j * h + j0 + r] = v;
      }
    }
    for (int e = t; e < kWb * kWb; e += kThreads)
      Ts[j0 * kWb + e] = ps.T[e];
    __syncthreads();
    if (j0 + nb < c)
      wy_apply<true>(P, ldp, nb, hp, Ts + j0 * kWb, W + static_cast<int64_t>(j0 + nb) * h + j0, h,
                     c - j0 - nb, sh);
  }
  // Columns past k (a wide matrix) hold R's entries in their first k rows.
  for (int64_t e = t; e < static_cast<int64_t>(k) * (c - k); e += kThreads)
    R[static_cast<int64_t>(k) * k + e] = W[(k + e / k) * static_cast<int64_t>(h) + e % k];
  __syncthreads();
}

// The block at j0 of the explicit V: in place, or copied to `stage`.
__device__ __forceinline__ const double* wy_block(const double* W, int h, int j0, int nb,
                                                  double* stage, int64_t* ldv)
{
  if (!stage)
  {
    *ldv = h;
    return W + static_cast<int64_t>(j0) * h + j0;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, hp = h - j0;
  for (int i = w; i < nb; i += kWarps)
    for (int r = lane; r < hp; r += 32)
      stage[i * hp + r] = W[static_cast<int64_t>(j0 + i) * h + j0 + r];
  __syncthreads();
  *ldv = hp;
  return stage;
}

// B (h x p, column-major, ldb) <- H_0 ... H_{k-1} B.
__device__ __noinline__ void cta_apply_q_wy(const double* W, int h, int k, const double* Ts,
                                            double* stage, double* B, int p, int64_t ldb,
                                            CtaShared& sh)
{
  for (int j0 = (k - 1) / kWb * kWb; j0 >= 0; j0 -= kWb)
  {
    const int nb = k - j0 < kWb ? k - j0 : kWb;
    int64_t ldv;
    const double* V = wy_block(W, h, j0, nb, stage, &ldv);
    wy_apply<false>(V, ldv, nb, h - j0, Ts + j0 * kWb, B + j0, ldb, p, sh);
  }
}

// Thin Q (h x k) in place from the explicit V in W.
__device__ __noinline__ void cta_form_q_wy(double* W, int h, int k, const double* Ts, double* stage,
                                           CtaShared& sh)
{
  const int t = threadIdx.x;
  double* Z = &sh.gemm_b[0][0];  // kWb x kWb, row-major
  for (int j0 = (k - 1) / kWb * kWb; j0 >= 0; j0 -= kWb)
  {
    const int nb = k - j0 < kWb ? k - j0 : kWb, hp = h - j0;
    const double* T = Ts + j0 * kWb;
    double* own = W + static_cast<int64_t>(j0) * h + j0;
    if (j0 + nb < k)
    {
      int64_t ldv;
      const double* V = wy_block(W, h, j0, nb, stage, &ldv);
      wy_apply<false>(V, ldv, nb, hp, T, W + static_cast<int64_t>(j0 + nb) * h + j0, h, k - j0 - nb,
                      sh);
    }
    // The block's own columns E - V Z, Z = T V1^T (upper triangular), V1 the
    // block's first nb rows: a row at a time by four lanes, in place.
    if (t < kWb * kWb)
    {
      const int l = t / kWb, i = t % kWb;
      double z = 0.0;
      if (l <= i && i < nb)
        for (int m = l; m <= i; ++m)
          z = fma(T[l + m * kWb], own[m * h + i], z);
      Z[t] = z;
    }
    __syncthreads();
    const int part = t & 3;
    for (int r0 = 0; r0 < hp; r0 += kThreads / 4)
    {
      const int r = r0 + (t >> 2);
      double v[kWb];
#pragma unroll
      for (int l = 0; l < kWb; ++l)
        v[l] = (l < nb && r < hp) ? -own[l * static_cast<int64_t>(h) + r] : 0.0;
      __syncwarp();
#pragma unroll
      for (int e = 0; e < kWb / 4; ++e)
      {
        const int i = 4 * e + part;
        double q = r == i ? 1.0 : 0.0;
#pragma unroll
        for (int l = 0; l < 4 * e + 4; ++l)
          q = fma(v[l], Z[l * kWb + i], q);
        if (i < nb && r < hp)
          own[i * static_cast<int64_t>(h) + r] = q;
      }
      __syncwarp();
    }
    // Rows above the block.
    for (int64_t e = t; e < static_cast<int64_t>(j0) * nb; e += kThreads)
      W[(j0 + e / j0) * static_cast<int64_t>(h) + e % j0] = 0.0;
    __syncthreads();
  }
}

}  // namespace
}  // namespace ttg
