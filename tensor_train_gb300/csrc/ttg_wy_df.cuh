// Blocked (compact WY) Householder QR, Q formation and Q application in
// df64.  Same reflectors and convention as cta_householder_qr_df /
// cta_form_q_df / cta_apply_q_df, summed in another order.
//
// A block of kWyB consecutive reflectors j0 .. j0+nb-1 acts as
//   H_j0 ... H_{j0+nb-1} = I - V T V^T      (forward, columnwise: LAPACK
//                                            dlarft; Schreiber & Van Loan,
//                                            SISC 10(1), 1989)
// with V the unit lower-trapezoidal (m - j0) x nb block of the reflector
// vectors and T upper triangular.  The one-reflector-at-a-time routines
// stream the trailing matrix three times per reflector; here the panel is
// factored in shared memory and the trailing matrix (in global or shared
// memory) is streamed three times per block (W = V^T B, W <- T' W, B -= V W),
// with V staged in shared memory as an explicit column-major block (zeros
// above its unit diagonal, zero columns past nb) so the inner loops carry no
// branches and lanes read consecutive rows.  W's sums go by halving (10
// shuffles and additions instead of 24 for 32 lanes, in the same order), and
// the formation of Q takes the T that the QR left.
//
// Which matrices take this form is fixed (Smem::form): a sum in another order
// moves singular vectors of values a relative gap g apart by 2e-14 / g, and
// 456 trains hold gaps of 1e-7.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ttg_device.cuh"
#include "ttg_device_df.cuh"
#include "ttg_job.h"

namespace ttg
{
namespace
{

// Shared staging the blocked routines need for m rows (in doubles).
__device__ __forceinline__ int64_t wy_stage_need(int m)
{
  return static_cast<int64_t>(m) * kWyB;
}

// In the CTA's GEMM staging: the blocks' T that the QR leaves for the
// formation of Q (gemm_a), the T and the Gram entries in use (gemm_b).
constexpr int kWyKept = 16 * 65 / (kWyB * kWyB);  // blocks
// The kept T of the block at j0, or null when there are more blocks than fit.
__device__ __forceinline__ df64* wy_kept_t(CtaShared& sh, int j0, int k)
{
  if ((k + kWyB - 1) / kWyB > kWyKept)
    return nullptr;
  return reinterpret_cast<df64*>(&sh.gemm_a[0][0]) + (j0 / kWyB) * kWyB * kWyB;
}
__device__ __forceinline__ df64* wy_work_t(CtaShared& sh)
{
  return reinterpret_cast<df64*>(&sh.gemm_b[0][0]);
}
__device__ __forceinline__ df64* wy_gram(CtaShared& sh)
{
  return wy_work_t(sh) + kWyB * kWyB;  // v_l . v_i above the diagonal
}

// T (kWyB x kWyB, column-major, zero outside the leading nb x nb upper
// triangle) from the Gram entries and the scales tau[0..nb), by warp 0:
// T(0:i, i) = -tau_i T(0:i, 0:i) G(0:i, i), T(i, i) = tau_i, lane l forming
// row l.  Ends with a barrier.
__device__ __forceinline__ void wy_t_from_gram(const df64* G, int nb, const df64* tau, df64* T)
{
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32)
  {
    for (int t = lane; t < kWyB * kWyB; t += 32)
      T[t] = df64{0.0f, 0.0f};
    __syncwarp();
    for (int i = 0; i < nb; ++i)
    {
      const df64 ti = tau[i], nt = df_neg(ti);
      df64 acc{0.0f, 0.0f};
      if (lane < i)
        for (int q = lane; q < i; ++q)
          acc = df_fma(T[lane + q * kWyB], df_mul(nt, G[q + i * kWyB]), acc);
      __syncwarp();
      if (lane < i)
        T[lane + i * kWyB] = acc;
      if (lane == 0)
        T[i + i * kWyB] = ti;
      __syncwarp();
    }
  }
  __syncthreads();
}

// T of the explicit block P (hp x kWyB, column-major, ld hp), from its Gram
// entries formed anew.  Ends with a barrier.
__device__ void wy_build_t_df(const df64* P, int hp, int nb, const df64* tau, df64* T, CtaShared& sh)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  df64* G = wy_gram(sh);
  for (int pr = w; pr < kWyB * kWyB; pr += kWarps)
  {
    const int l = pr % kWyB, i = pr / kWyB;
    if (l >= i || i >= nb)
      continue;
    df64 acc{0.0f, 0.0f};
    for (int r = i + lane; r < hp; r += 32)  // v_i is zero above row i
      acc = df_fma(P[r + static_cast<int64_t>(l) * hp], P[r + static_cast<int64_t>(i) * hp], acc);
    acc = df_warp_sum(acc);
    if (lane == 0)
      G[l + i * kWyB] = acc;
  }
  __syncthreads();
  wy_t_from_gram(G, nb, tau, T);
}

// B(0:hp, 0:ncols) <- (I - V T' V^T) B, T' = T^T (kTrans: the product
// H_{j0+nb-1} ... H_j0, as the factorisation applies the block) or T (the
// product H_j0 ... H_{j0+nb-1}).  B points at the block's first row,
// column stride ldb.  A group of hh_group(hp) lanes per column of B.  Ends
// with a barrier.
template <bool kTrans>
__device__ __noinline__ void wy_apply_df(const df64* P, int hp, const df64* T, df64* B, int64_t ldb,
                                         int ncols)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // G lanes per column (hh_group), 32 / G columns in flight per warp; the
  // loop bound is uniform over the warp (the group sums need every lane).
  const int G = hh_group(hp), gpw = 32 / G, gl = lane & (G - 1), gbase = lane & ~(G - 1);
  for (int cb = w * gpw; cb < ncols; cb += kWarps * gpw)
  {
    const int q = cb + lane / G;
    const bool act = q < ncols;
    df64* y = B + static_cast<int64_t>(act ? q : cb) * ldb;
    df64 acc[kWyB];
#pragma unroll
    for (int i = 0; i < kWyB; ++i)
      acc[i] = df64{0.0f, 0.0f};
    if (act)
      for (int r = gl; r < hp; r += G)
      {
        const df64 a = y[r];
#pragma unroll
        for (int i = 0; i < kWyB; ++i)
          acc[i] = df_fma(P[r + static_cast<int64_t>(i) * hp], a, acc[i]);
      }
    // The kWyB sums by halving (each step a lane keeps half of its values):
    // lane gl ends with W_li of W = V^T y; it forms (T' W)_li and the group
    // gathers all of them.
    const int o1 = G >> 1, o2 = G >> 2, o3 = G >> 3;
    df64 wi;
    {
      df64 h4[4], h2[2];
#pragma unroll
      for (int i = 0; i < 4; ++i)
      {
        const bool up = (gl & o1) != 0;
        h4[i] = df_add(up ? acc[i + 4] : acc[i], df_shfl_xor(up ? acc[i] : acc[i + 4], o1));
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
      {
        const bool up = (gl & o2) != 0;
        h2[i] = df_add(up ? h4[i + 2] : h4[i], df_shfl_xor(up ? h4[i] : h4[i + 2], o2));
      }
      const bool up = (gl & o3) != 0;
      wi = df_add(up ? h2[1] : h2[0], df_shfl_xor(up ? h2[0] : h2[1], o3));
      for (int o = o3 >> 1; o > 0; o >>= 1)
        wi = df_add(wi, df_shfl_xor(wi, o));
    }
    const int li = gl / o3;
    df64 wp{0.0f, 0.0f};
#pragma unroll
    for (int l = 0; l < kWyB; ++l)
    {
      const df64 wl{__shfl_sync(0xffffffffu, wi.hi, gbase + l * o3),
                    __shfl_sync(0xffffffffu, wi.lo, gbase + l * o3)};
      wp = df_fma(kTrans ? T[l + li * kWyB] : T[li + l * kWyB], wl, wp);
    }
#pragma unroll
    for (int i = 0; i < kWyB; ++i)
      acc[i] = df_neg(df64{__shfl_sync(0xffffffffu, wp.hi, gbase + i * o3),
                           __shfl_sync(0xffffffffu, wp.lo, gbase + i * o3)});
    if (act)
      for (int r = gl; r < hp; r += G)
      {
        df64 a = y[r];
#pragma unroll
        for (int i = 0; i < kWyB; ++i)
          a = df_fma(acc[i], P[r + static_cast<int64_t>(i) * hp], a);
        y[r] = a;
      }
  }
  __syncthreads();
}

// P (hp x kWyB, ld hp) <- the explicit V of the block of nb reflectors whose
// vectors lie below the diagonal of A(j0:, j0:j0+nb): zero above the unit
// diagonal, zero columns past nb.  Ends with a barrier.
__device__ void wy_stage_v_df(const df64* A, int64_t ld, int j0, int hp, int nb, df64* P)
{
  const int64_t total = static_cast<int64_t>(hp) * kWyB;
  for (int64_t t = threadIdx.x; t < total; t += blockDim.x)
  {
    const int r = static_cast<int>(t % hp), i = static_cast<int>(t / hp);
    df64 v{0.0f, 0.0f};
    if (i < nb)
      v = r > i ? A[(j0 + r) + static_cast<int64_t>(j0 + i) * ld] : (r == i ? df64{1.0f, 0.0f} : v);
    P[t] = v;
  }
  __syncthreads();
}

// Householder QR of A (m x c, column-major, ld) in place, as
// cta_householder_qr_df, in blocks of kWyB reflectors.  stage: shared memory
// for wy_stage_need(m) doubles.  The blocks' T stay with wy_kept_t.
__device__ __noinline__ void cta_householder_qr_df_wy(df64* A, int m, int c, int64_t ld, df64* tau,
                                                      df64* stage, CtaShared& sh)
{
  const int k = m < c ? m : c;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int j0 = 0; j0 < k; j0 += kWyB)
  {
    const int nb = k - j0 < kWyB ? k - j0 : kWyB;
    const int hp = m - j0;
    df64* P = stage;
    // The panel A(j0:m, j0:j0+nb) into shared memory, factored there.
    df64* p = P + static_cast<int64_t>(w) * hp;
    df64* own = A + j0 + static_cast<int64_t>(j0 + w) * ld;
    if (w < nb)
      for (int r = lane; r < hp; r += 32)
        p[r] = own[r];
    __syncthreads();
    cta_householder_qr_df(P, hp, nb, hp, tau + j0, sh);
    // R block and reflector vectors back to A; P becomes the explicit V.
    if (w < nb)
      for (int r = lane; r < hp; r += 32)
      {
        own[r] = p[r];
        if (r <= w)
          p[r] = df64{r == w ? 1.0f : 0.0f, 0.0f};
      }
    else
      for (int r = lane; r < hp; r += 32)
        p[r] = df64{0.0f, 0.0f};
    __syncthreads();
    if (j0 + nb >= c)
      break;
    df64* T = wy_kept_t(sh, j0, k);
    if (!T)
      T = wy_work_t(sh);
    wy_build_t_df(P, hp, nb, tau + j0, T, sh);
    wy_apply_df<true>(P, hp, T, A + j0 + static_cast<int64_t>(j0 + nb) * ld, ld, c - j0 - nb);
  }
}

// Thin Q (m x k) in place from the reflectors of cta_householder_qr_df_wy, as
// cta_form_q_df: blocks from the last, each applied to the columns already
// formed, then its own columns as one product (the GEMM staging must be as
// the QR left it).
__device__ __noinline__ void cta_form_q_df_wy(df64* A, int m, int k, int64_t ld, const df64* tau,
                                              df64* stage, CtaShared& sh)
{
  for (int j0 = ((k - 1) / kWyB) * kWyB; j0 >= 0; j0 -= kWyB)
  {
    const int nb = k - j0 < kWyB ? k - j0 : kWyB;
    const int hp = m - j0;
    df64* P = stage;
    wy_stage_v_df(A, ld, j0, hp, nb, P);
    if (j0 + nb < k)
    {
      const df64* T = wy_kept_t(sh, j0, k);
      if (!T)
      {
        wy_build_t_df(P, hp, nb, tau + j0, wy_work_t(sh), sh);
        T = wy_work_t(sh);
      }
      wy_apply_df<false>(P, hp, T, A + j0 + static_cast<int64_t>(j0 + nb) * ld, ld, k - j0 - nb);
    }
    cta_form_q_df(P, hp, nb, hp, tau + j0);
    // The block's columns: rows j0.. from P, rows above j0 zero.
    cta_each(m, nb, [&](int r, int i) {
      A[r + static_cast<int64_t>(j0 + i) * ld] =
        r >= j0 ? P[(r - j0) + static_cast<int64_t>(i) * hp] : df64{0.0f, 0.0f};
    });
    __syncthreads();
  }
}

// B (m x p, column-major df64, ldb) <- H_0 ... H_{kref-1} B, as
// cta_apply_q_df, one block pass at a time from the last block.
__device__ __noinline__ void cta_apply_q_df_wy(const df64* A, int m, int kref, int64_t lda,
                                               const df64* tau, df64* B, int p, int64_t ldb,
                                               df64* stage, CtaShared& sh)
{
  df64* T = wy_work_t(sh);
  for (int j0 = ((kref - 1) / kWyB) * kWyB; j0 >= 0; j0 -= kWyB)
  {
    const int nb = kref - j0 < kWyB ? kref - j0 : kWyB;
    const int hp = m - j0;
    df64* P = stage;
    wy_stage_v_df(A, lda, j0, hp, nb, P);
    wy_build_t_df(P, hp, nb, tau + j0, T, sh);
    wy_apply_df<false>(P, hp, T, B + j0, ldb, p);
  }
}

}  // namespace
}  // namespace ttg
