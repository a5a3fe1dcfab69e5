// Blocked Householder QR and its Q over the CTAs of a team, FP64.
//
// The unblocked form met at a grid barrier per column (~10 us each: barrier,
// norm, update of the CTA's columns one CTA-wide reduction at a time), and Q
// cost a chain of as many CTA-wide reductions: 8.2 ms per step of the d = 40,
// rank-257 sweep against a floor of 0.7 ms at the chip's FP64 rate.  Here
// kPb columns are factored by a few CTAs and applied as one block
// I - V T V^T (compact WY; LAPACK dlarft, Schreiber & Van Loan 1989):
//
//   * wide_panel: the panel's rows are cut into slabs of >= 64, one per CTA,
//     in shared memory.  Per column one exchange: each CTA publishes its
//     share of the products of the column with all kPb panel columns (its
//     norm, the next columns' dots and the entries of V^T V for T at once),
//     and every CTA adds the slabs' shares in the same order.
//   * wide_trail / wide_form_q: the trailing matrix (or Q) is cut into slabs
//     of rows times groups of columns, one CTA each, so that every SM's FP64
//     pipe has the same share; W = V^T B is exchanged between the slabs of a
//     column group only.  Q's tiles stay in shared memory over all blocks.
//
// An exchange is one 16-byte packet per value, {low word, tag, high word,
// tag}, the line of NCCL's low-latency (LL) protocol: each 8-byte half says by
// its tag that it has arrived (8-byte accesses are single), so a reader needs no fence and no flag, only a poll of the
// packet itself.  Tags never repeat within a launch, and the packets are
// zeroed before it.  Packet buffers alternate by the tag's parity: a CTA two
// exchanges ahead has all packets of the one between, whose senders have read
// the first.  Every poll is bounded like the grid barrier's.
//
// Reflector convention as cta_householder_qr (Eigen's makeHouseholder).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "ttg_device.cuh"
#include "ttg_job.h"
#include "ttg_reflector.cuh"

namespace ttg
{
namespace
{

constexpr int kPb = kWidePb;

// -- packets ------------------------------------------------------------------
__device__ __forceinline__ void packet_put(uint4* p, double v, uint32_t tag)
{
  const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v));
  asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %2};" ::"l"(p),
               "r"(static_cast<uint32_t>(u)), "r"(tag), "r"(static_cast<uint32_t>(u >> 32))
               : "memory");
}

// A packet as it is now; true when it has arrived.
__device__ __forceinline__ bool packet_try(const uint4* p, uint32_t tag, double* v)
{
  uint32_t lo, t0, hi, t1;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(lo), "=r"(t0), "=r"(hi), "=r"(t1)
               : "l"(p)
               : "memory");
  *v = __longlong_as_double(
    static_cast<long long>((static_cast<unsigned long long>(hi) << 32) | lo));
  return t0 == tag && t1 == tag;
}

// Waits for the packets p[0], p[stride], ... of which n <= N are wanted, all
// polled together (one L2 round trip per attempt for the set, not one per
// packet), and returns their sum in a fixed order; *fail = true when the wait
// gave up.
template <int N>
__device__ __forceinline__ double packets_sum(const WideJob& job, const uint4* p, int64_t stride, int n,
                                              uint32_t tag, bool* fail)
{
  double v[N];
  int polls = 0;
  long long start = 0;
  for (;;)
  {
    uint32_t lo[N], t0[N], hi[N], t1[N];
#pragma unroll
    for (int e = 0; e < N; ++e)
      asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(lo[e]), "=r"(t0[e]), "=r"(hi[e]), "=r"(t1[e])
                   : "l"(p + (e < n ? e : 0) * stride)
                   : "memory");
    bool all = true;
#pragma unroll
    for (int e = 0; e < N; ++e)
    {
      all = all && t0[e] == tag && t1[e] == tag;
      v[e] = e < n ? __longlong_as_double(static_cast<long long>(
                       (static_cast<unsigned long long>(hi[e]) << 32) | lo[e]))
                   : 0.0;
    }
    if (all)
      break;
    if ((++polls & 255) == 0)
    {
      if (start == 0)
        start = clock64();
      const bool late = clock64() - start > job.wait_cycles;
      if (late)
        atomicExch(&job.bar->err, 1);
      if (late || *reinterpret_cast<volatile int*>(&job.bar->err))
      {
        *fail = true;
        return 0.0;
      }
    }
  }
#pragma unroll
  for (int w = N / 2; w > 0; w >>= 1)
#pragma unroll
    for (int e = 0; e < N / 2; ++e)
      if (e < w && e + w < n)
        v[e] += v[e + w];
  return v[0];
}

// Slots: panel products (slab, column), the panel row's own entries, and the
// products of a block's application (slab, column, reflector), in one region
// for the sweep's own and one for a Q formed meanwhile.
__device__ __forceinline__ uint4* panel_slot(const WideJob& job, uint32_t tag, int slab, int l)
{
  return job.packets + ((tag & 1u) * (kWidePanelSlabs + 1) + slab) * kPb + l;
}
__device__ __forceinline__ uint4* trail_slot(const WideJob& job, int region, uint32_t tag, int slab,
                                             int col, int i)
{
  return job.packets + 2 * (kWidePanelSlabs + 1) * kPb +
         ((static_cast<int64_t>(2 * region + (tag & 1u)) * kWideTrailSlabs + slab) * job.c_max + col) *
           kPb +
         i;
}

// -- panel --------------------------------------------------------------------
struct PanelShared
{
  double d[kPb];       // the column's products with the panel's columns
  double row[kPb];     // the panel columns' entries in the column's row
  double w[kPb];       // what the row loses per column
  double G[kPb * kPb]; // V^T V above the diagonal
  double T[kPb * kPb]; // column-major, upper triangular
  double inv[kPb], tau[kPb];
};

// Factors columns j0 .. j0 + nb of W (h rows) on the first S CTAs of the
// team, `rows` rows from j0 on each.  On return W holds the explicit V (from
// row j0 on), R its entries, job.Tw the block's T.  Tags seq .. seq + nb.
__device__ __noinline__ bool wide_panel(const WideJob& job, int h, int k, int j0, int nb, int S,
                                        int rows, uint32_t seq, double* sm)
{
  const int me = job.rank, t = threadIdx.x;
  const int r0 = j0 + me * rows;  // this slab's first row
  const int nr = h - r0 < rows ? h - r0 : rows;
  const int ld = rows | 1;
  PanelShared& ps = *reinterpret_cast<PanelShared*>(sm);
  double* P = sm + sizeof(PanelShared) / sizeof(double);
  const int lane = t & 31, w = t >> 5;
  for (int i = w; i < nb; i += kWarps)
    for (int r = lane; r < nr; r += 32)
      P[i * ld + r] = job.W[static_cast<int64_t>(j0 + i) * h + r0 + r];
  __syncthreads();
  bool fail = false;
  for (int i = 0; i < nb; ++i)
  {
    const uint32_t tag = seq + i;
    const int j = j0 + i;           // the column, and its diagonal row
    const int lo = j + 1 > r0 ? j + 1 - r0 : 0;  // first slab row below the diagonal
    const bool owner = j >= r0 && j < r0 + nr;
    const double* x = P + i * ld;
    // Products of x below row j: 8 lanes per panel column on four warps, one
    // per FP64 pipe.  A warp's FP64 instruction holds its pipe for 64 clocks,
    // which is also its latency: what counts is their number, so one chain
    // per lane and no more lanes than this.
    if (t < 8 * kPb)
    {
      const int l = t >> 3, g = t & 7;
      double a0 = 0.0;
      if (l < nb)
      {
        const double* y = P + l * ld;
        for (int r = lo + g; r < nr; r += 8)
          a0 = fma(x[r], y[r], a0);
      }
      a0 += __shfl_xor_sync(0xffffffffu, a0, 4);
      a0 += __shfl_xor_sync(0xffffffffu, a0, 2);
      a0 += __shfl_xor_sync(0xffffffffu, a0, 1);
      if (g == 0 && l < nb)
      {
        if (S > 1)
          packet_put(panel_slot(job, tag, me, l), a0, tag);
        else
          ps.d[l] = a0;
      }
    }
    else if (owner && t < 8 * kPb + nb)
    {
      const int l = t - 8 * kPb;
      if (S > 1)
        packet_put(panel_slot(job, tag, kWidePanelSlabs, l), P[l * ld + j - r0], tag);
      else
        ps.row[l] = P[l * ld + j - r0];
    }
    // T's previous column while the packets travel (the first CTA's T is used).
    if (me == 0 && w == 6 && i > 0)
      t_column(ps, i - 1);
    if (S > 1 && t < 8 * kPb)
    {
      const int l = t >> 3, g = t & 7;
      static_assert(kWidePanelSlabs == 32, "up to four packets per lane");
      double v = 0.0;
      if (l < nb && g < S)
      {
        const int n = (S - g + 7) / 8;
        const uint4* p = panel_slot(job, tag, g, l);
        v = S <= 8 ? packets_sum<1>(job, p, 8 * kPb, n, tag, &fail)
                   : packets_sum<4>(job, p, 8 * kPb, n, tag, &fail);
      }
      __syncwarp();
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      if (g == 0)
        ps.d[l] = v;
    }
    else if (S > 1 && t < 8 * kPb + nb)
      ps.row[t - 8 * kPb] =
        packets_sum<1>(job, panel_slot(job, tag, kWidePanelSlabs, t - 8 * kPb), 0, 1, tag, &fail);
    if (__syncthreads_or(fail))
      return false;
    // The reflector, and what it takes from each later column.  tau inv =
    // +-1 / n: warp 0 forms what the update below waits for, warps 1 and 2 (on
    // other pipes, the same scalars again) the rest.
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
        if (owner && lane > i && lane < nb)
          P[lane * ld + j - r0] = fma(-tau, dot, ps.row[lane]);
        if (owner && lane == i)
          P[i * ld + j - r0] = beta;
      }
      else
      {
        // G(l, i) = v_l . v_i, v_l = inv_l x_l.
        if (lane < i)
          ps.G[lane + i * kPb] = ps.inv[lane] * dot;
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
      double* y = P + l * ld;
      for (int r = lo + lane; r < nr; r += 32)
        y[r] = fma(f, x[r], y[r]);
    }
    __syncthreads();
  }
  if (me == 0 && w == 6)
    t_column(ps, nb - 1);
  // R's entries and the explicit V.
  for (int i = w; i < nb; i += kWarps)
  {
    const int j = j0 + i;
    const double inv = ps.inv[i];
    for (int r = lane; r < nr; r += 32)
    {
      const int gr = r0 + r;
      const double x = P[i * ld + r];
      if (gr <= j)
        job.R[gr + static_cast<int64_t>(j) * k] = x;
      job.W[static_cast<int64_t>(j) * h + gr] = gr < j ? 0.0 : (gr == j ? 1.0 : inv * x);
    }
  }
  __syncthreads();
  if (me == 0)
    for (int e = t; e < kPb * kPb; e += kThreads)
      job.Tw[static_cast<int64_t>(j0 / kPb) * kPb * kPb + e] =
        (e / kPb < nb && e % kPb < nb) ? ps.T[e] : 0.0;
  __syncthreads();
  return true;
}

// -- block application ---------------------------------------------------------
// How a matrix of `hp` rows and m columns is cut for a block's application:
// St slabs of `rows` rows times Gt groups of at most nc columns.  The cost is
// the FP64 clocks of the fullest CTA: 2 kPb FMAs per element at 2 per clock,
// the slabs' sums, and an exchange's latency (~1.8 us measured).
struct TrailCut
{
  int St, Gt, rows, nc;
};

// Lane s - 1 of every warp weighs s slabs; all lanes of the CTA get the cut.
// nv: V slabs held at once (wide_q loads the next block's beside this one's).
__device__ TrailCut trail_cut(int hp, int m, int P, int64_t cap, int nv)
{
  const int s = (threadIdx.x & 31) + 1;
  const int most = P < kWideTrailSlabs ? P : kWideTrailSlabs;
  auto cut_of = [&](int slabs) {
    TrailCut k;
    k.rows = (hp + slabs - 1) / slabs;
    k.St = (hp + k.rows - 1) / k.rows;
    k.Gt = P / k.St < m ? P / k.St : m;
    k.nc = (m + k.Gt - 1) / k.Gt;
    return k;
  };
  unsigned long long best = ~0ull;
  if (s <= most)
  {
    const TrailCut k = cut_of(s);
    const int64_t need =
      static_cast<int64_t>(nv * kPb + k.nc) * (k.rows | 1) + 2 * kPb * k.nc + nv * kPb * kPb;
    // Columns and rows as the lanes of block_apply cover them, on the busiest
    // of the four FP64 pipes; wide_q starts with few of its columns and ends
    // with all, so it is weighed at four points between.
    auto clocks = [&](int nc) {
      const int w = nc <= 8 ? 4 : (nc <= 16 ? 8 : 16), G = nc <= 8 ? 32 : (nc <= 16 ? 16 : 8);
      return static_cast<unsigned long long>(kPb) * ((nc + w - 1) / w * w) *
             ((k.rows + G - 1) / G * G);
    };
    const unsigned long long work =
      nv == 1 ? clocks(k.nc)
              : (clocks((k.nc + 3) / 4) + clocks((k.nc + 1) / 2) + clocks((3 * k.nc + 3) / 4) +
                 clocks(k.nc)) /
                  4;
    if (need <= cap)
      best = (work + 8ull * k.nc * k.St + (k.St > 1 ? 3500 : 0))
               << 5 |
             static_cast<unsigned>(s - 1);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
  {
    const unsigned long long x = __shfl_xor_sync(0xffffffffu, best, o);
    best = x < best ? x : best;
  }
  if (best == ~0ull)
    return TrailCut{0, 0, 0, 0};
  return cut_of(static_cast<int>(best & 31) + 1);
}

// The tile B (nr x nc in shared memory, column-major, ldb) <- its rows of
// (I - V T' V^T) B, T' = T^T (kTrans) or T: V's rows of this slab in Vs
// (kPb columns, ldv), B's other slabs on the other CTAs of the group, whose
// shares of V^T B are exchanged under `tag` (St > 1).  col(q): the column's
// index in the exchange.  Ws, Zs: kPb nc doubles each.
template <int G, bool kTrans, class FCol>
__device__ __forceinline__ bool block_apply_g(const WideJob& job, const double* Vs, int ldv, double* Bs,
                                              int ldb, int nr, int nc, const double* Ts, double* Ws,
                                              double* Zs, int St, int slab, int region, uint32_t tag,
                                              FCol col)
{
  const int t = threadIdx.x, gl = t & (G - 1), q0 = t / G;
  constexpr int kCols = kThreads / G;
  const int i0 = G == 32 ? gl >> 1 : gl * (kPb / G > 0 ? kPb / G : 1);
  for (int qb = 0; qb < nc; qb += kCols)
  {
    const int q = qb + q0;
    double acc[kPb];
#pragma unroll
    for (int i = 0; i < kPb; ++i)
      acc[i] = 0.0;
    if (q < nc)
    {
      const double* y = Bs + q * ldb;
      for (int r = gl; r < nr; r += G)
      {
        const double b = y[r];
#pragma unroll
        for (int i = 0; i < kPb; ++i)
          acc[i] = fma(Vs[i * ldv + r], b, acc[i]);
      }
    }
    halving_sum<G>(acc, gl);
    if (q < nc)
    {
      constexpr int kEach = kPb / G > 0 ? kPb / G : 1;
#pragma unroll
      for (int e = 0; e < kEach; ++e)
        if (G < 32 || (gl & 1) == 0)
        {
          if (St > 1)
            packet_put(trail_slot(job, region, tag, slab, col(q), i0 + e), acc[e], tag);
          else
            Ws[q * kPb + i0 + e] = acc[e];
        }
    }
  }
  bool fail = false;
  if (St > 1)
    for (int e = t; e < nc * kPb; e += kThreads)
    {
      const uint4* p = trail_slot(job, region, tag, 0, col(e / kPb), e % kPb);
      const int64_t stride = job.c_max * kPb;
      double v = packets_sum<8>(job, p, stride, St < 8 ? St : 8, tag, &fail);
      if (St > 8)
        v += packets_sum<8>(job, p + 8 * stride, stride, St - 8, tag, &fail);
      Ws[e] = v;
    }
  if (__syncthreads_or(fail))
    return false;
  for (int e = t; e < nc * kPb; e += kThreads)
  {
    const int i = e % kPb;
    const double* wq = Ws + (e - i);
    double z = 0.0;
#pragma unroll
    for (int l = 0; l < kPb; ++l)
      z = fma(kTrans ? Ts[l + i * kPb] : Ts[i + l * kPb], wq[l], z);
    Zs[e] = z;
  }
  __syncthreads();
  for (int qb = 0; qb < nc; qb += kCols)
  {
    const int q = qb + q0;
    if (q >= nc)
      break;
    double z[kPb];
#pragma unroll
    for (int i = 0; i < kPb; ++i)
      z[i] = -Zs[q * kPb + i];
    double* y = Bs + q * ldb;
    int r = gl;
    for (; r + G < nr; r += 2 * G)  // two rows at a time: independent chains
    {
      double b = y[r], b2 = y[r + G];
#pragma unroll
      for (int i = 0; i < kPb; ++i)
      {
        b = fma(z[i], Vs[i * ldv + r], b);
        b2 = fma(z[i], Vs[i * ldv + r + G], b2);
      }
      y[r] = b;
      y[r + G] = b2;
    }
    if (r < nr)
    {
      double b = y[r];
#pragma unroll
      for (int i = 0; i < kPb; ++i)
        b = fma(z[i], Vs[i * ldv + r], b);
      y[r] = b;
    }
  }
  __syncthreads();
  return true;
}

template <bool kTrans, class FCol>
__device__ bool block_apply(const WideJob& job, const double* Vs, int ldv, double* Bs, int ldb, int nr,
                            int nc, const double* Ts, double* Ws, double* Zs, int St, int slab,
                            int region, uint32_t tag, FCol col)
{
  // Lanes per column: as few as keep all 256 threads at work.
  if (nc > 16)
    return block_apply_g<8, kTrans>(job, Vs, ldv, Bs, ldb, nr, nc, Ts, Ws, Zs, St, slab, region,
                                    tag, col);
  if (nc > 8)
    return block_apply_g<16, kTrans>(job, Vs, ldv, Bs, ldb, nr, nc, Ts, Ws, Zs, St, slab, region,
                                     tag, col);
  return block_apply_g<32, kTrans>(job, Vs, ldv, Bs, ldb, nr, nc, Ts, Ws, Zs, St, slab, region,
                                     tag, col);
}

// 8 bytes from global to shared memory, in flight until copies_wait; zeros
// where !in (src is not read).
__device__ __forceinline__ void copy_async(double* dst, const double* src, bool in)
{
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(in ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void copies_wait()
{
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Starts the copies of V's rows [r0, r0 + nr) of the block at j0 (zero above
// row j0 and past nb) and of the block's T into shared memory.
__device__ __forceinline__ void load_block(const double* W, const double* Tw, int h, int j0, int nb,
                                           int r0, int nr, double* Vs, int ldv, double* Ts)
{
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int i = w; i < kPb; i += kWarps)
  {
    const double* col = W + static_cast<int64_t>(i < nb ? j0 + i : j0) * h + r0;
    for (int r = lane; r < nr; r += 32)
      copy_async(Vs + i * ldv + r, col + r, i < nb && r0 + r >= j0);
  }
  for (int e = threadIdx.x; e < kPb * kPb; e += kThreads)
    copy_async(Ts + e, Tw + static_cast<int64_t>(j0 / kPb) * kPb * kPb + e, true);
}

// W's columns from j0 + nb on <- (I - V T^T V^T) W, V the block at j0.
__device__ __noinline__ bool wide_trail(const WideJob& job, int h, int c, int j0, int nb, uint32_t tag,
                                        double* sm, int64_t cap)
{
  const int c0 = j0 + nb, m = c - c0, hp = h - j0;
  const TrailCut cut = trail_cut(hp, m, job.size, cap, 1);
  const int slab = job.rank % cut.St, g = job.rank / cut.St;
  if (g >= cut.Gt)
    return true;
  const int r0 = j0 + slab * cut.rows;
  const int nr = h - r0 < cut.rows ? h - r0 : cut.rows;
  const int q0 = g * cut.nc;
  const int nc = m - q0 < cut.nc ? m - q0 : cut.nc;
  if (nc <= 0)
    return true;
  const int ld = cut.rows | 1;
  double* Vs = sm;
  double* Bs = Vs + kPb * ld;
  double* Ws = Bs + cut.nc * ld;
  double* Zs = Ws + kPb * cut.nc;
  double* Ts = Zs + kPb * cut.nc;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  load_block(job.W, job.Tw, h, j0, nb, r0, nr, Vs, ld, Ts);
  double* B = job.W + static_cast<int64_t>(c0 + q0) * h + r0;
  for (int q = w; q < nc; q += kWarps)
    for (int r = lane; r < nr; r += 32)
      copy_async(Bs + q * ld + r, B + static_cast<int64_t>(q) * h + r, true);
  copies_wait();
  __syncthreads();
  if (!block_apply<true>(job, Vs, ld, Bs, ld, nr, nc, Ts, Ws, Zs, cut.St, slab, 0, tag,
                         [&](int q) { return q0 + q; }))
    return false;
  for (int q = w; q < nc; q += kWarps)
    for (int r = lane; r < nr; r += 32)
      B[static_cast<int64_t>(q) * h + r] = Bs[q * ld + r];
  __syncthreads();
  return true;
}

// Q = H_0 ... H_{kref-1} [B; 0] (h x ncols) from the explicit blocks in W, to
// out(i, l) = out[i o_rs + l o_cs]; B column-major (nb_rows x ncols) or, with
// eye, the identity.  Formed by `size` CTAs of the team, of which this one is
// `rank` (< 0: takes no part), block by block from the last; a CTA's tile
// stays in the `cap` doubles at sm in between, so that the blocks can be
// spread over other work (no grid barrier inside).  Tags seq .. seq + blocks.
struct WideQ
{
  bool on;
  int next;  // next block; the same on every CTA of the team
  const double *W, *Tw, *B;
  double* out;
  int64_t o_rs, o_cs;
  int h, kref, nb_rows, ncols, rank, size, region;
  bool eye;
  uint32_t seq;
  double* sm;
  int64_t cap;
  // this CTA's tile
  TrailCut cut;
  int slab, g, r0, nr, nc;
  int ready, buf;  // block whose V is in (or on its way to) buffer buf; -1
};

__device__ __forceinline__ double* wide_q_tile(const WideQ& q)
{
  return q.sm + 2 * kPb * (q.cut.rows | 1);  // behind two slabs of V
}

__device__ __noinline__ void wide_q_begin(WideQ& q)
{
  q.on = true;
  q.next = (q.kref + kPb - 1) / kPb - 1;
  q.ready = -1;
  q.buf = 0;
  if (q.rank < 0)
    return;
  q.cut = trail_cut(q.h, q.ncols, q.size, q.cap, 2);
  q.slab = q.rank % q.cut.St;
  q.g = q.rank / q.cut.St;
  if (q.g >= q.cut.Gt)
  {
    q.rank = -1;
    return;
  }
  q.r0 = q.slab * q.cut.rows;
  q.nr = q.h - q.r0 < q.cut.rows ? q.h - q.r0 : q.cut.rows;
  // Columns g, g + Gt, ...: with the identity start a block touches columns
  // from its own first on, so every group gets some of each.
  q.nc = (q.ncols - q.g + q.cut.Gt - 1) / q.cut.Gt;
}

// B's tile into shared memory.
__device__ __forceinline__ void wide_q_fill(WideQ& q)
{
  const int ld = q.cut.rows | 1;
  double* Bs = wide_q_tile(q);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int c = w; c < q.nc; c += kWarps)
  {
    const int l = q.g + q.cut.Gt * c;
    for (int r = lane; r < q.nr; r += 32)
    {
      const int gr = q.r0 + r;
      Bs[c * ld + r] = q.eye ? (gr == l ? 1.0 : 0.0)
                             : (gr < q.nb_rows ? q.B[gr + static_cast<int64_t>(l) * q.nb_rows] : 0.0);
    }
  }
}

// The next block's application to this CTA's tile.
__device__ __noinline__ bool wide_q_block(const WideJob& job, WideQ& q)
{
  const int b = q.next--;
  if (q.rank < 0)
    return true;
  if (b == (q.kref + kPb - 1) / kPb - 1)
    wide_q_fill(q);  // not before: the shared memory is in use until here
  // First of this group's columns that block b touches.
  const int qa = q.eye && b * kPb > q.g ? (b * kPb - q.g + q.cut.Gt - 1) / q.cut.Gt : 0;
  if (qa >= q.nc)
    return true;
  const int ld = q.cut.rows | 1;
  double* Bs = wide_q_tile(q);
  double* Ws = Bs + q.cut.nc * ld;
  double* Zs = Ws + kPb * q.cut.nc;
  double* Ts = Zs + kPb * q.cut.nc;  // two blocks' T
  auto load = [&](int blk, int buf) {
    const int j0 = blk * kPb;
    load_block(q.W, q.Tw, q.h, j0, q.kref - j0 < kPb ? q.kref - j0 : kPb, q.r0, q.nr,
               q.sm + buf * kPb * ld, ld, Ts + buf * kPb * kPb);
  };
  if (q.ready != b)
    load(b, q.buf);
  copies_wait();
  __syncthreads();
  if (b > 0)
    load(b - 1, q.buf ^ 1);  // in flight while this block is applied
  q.ready = b - 1;
  const uint32_t tag = q.seq + static_cast<uint32_t>((q.kref + kPb - 1) / kPb - 1 - b);
  const int g = q.g, Gt = q.cut.Gt;
  const bool ok = block_apply<false>(job, q.sm + q.buf * kPb * ld, ld, Bs + qa * ld, ld, q.nr,
                                     q.nc - qa, Ts + q.buf * kPb * kPb, Ws, Zs, q.cut.St, q.slab,
                                     q.region, tag, [&](int c) { return g + Gt * (qa + c); });
  q.buf ^= 1;
  return ok;
}

// All blocks left, and the tile to its place.
__device__ __noinline__ bool wide_q_end(const WideJob& job, WideQ& q)
{
  while (q.next >= 0)
    if (!wide_q_block(job, q))
      return false;
  q.on = false;
  if (q.rank < 0)
    return true;
  copies_wait();
  __syncthreads();
  const int ld = q.cut.rows | 1;
  const double* Bs = wide_q_tile(q);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int c = w; c < q.nc; c += kWarps)
  {
    const int64_t l = q.g + q.cut.Gt * c;
    for (int r = lane; r < q.nr; r += 32)
      q.out[(q.r0 + r) * q.o_rs + l * q.o_cs] = Bs[c * ld + r];
  }
  __syncthreads();
  return true;
}

// Rows per panel slab and slabs for hp rows.
__device__ __forceinline__ int panel_rows(int hp, int P)
{
  const int most = P < kWidePanelSlabs ? P : kWidePanelSlabs;
  const int rows = (hp + most - 1) / most;
  return rows < 64 ? 64 : rows;
}

// Whether the blocked routines' tiles fit: the panel's slab, and some cut of
// the trailing matrix and of Q.
__device__ bool wide_blocked_fits(int h, int c, int P, int64_t cap)
{
  const int64_t panel = static_cast<int64_t>(kPb) * (panel_rows(h, P) | 1) +
                        static_cast<int64_t>(sizeof(PanelShared) / sizeof(double));
  return panel <= cap && trail_cut(h, c, P, cap, 2).St > 0;
}

}  // namespace
}  // namespace ttg
