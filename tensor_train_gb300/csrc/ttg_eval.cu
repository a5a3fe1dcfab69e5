// eval_at / eval_batch (algebra/tt_eval.hpp:32-112): one value per
// multi-index, the product G_0[i_0] G_1[i_1] ... G_{d-1}[i_{d-1}].
//
// 8, 16 or 32 lanes per multi-index carry a row vector through the first
// sites and a column vector back through the last ones (from eval_split on),
// and multiply the two.  Alone that is M sum r_k r_{k+1} FP64 FMAs, and GB300
// retires 2 of them per clock per SM: 2^20 indices of a d = 32, rank-64 train
// took 191 ms with the FP64 pipe 96 % busy.  The indices share their factors,
// though, so plan_eval has products formed once per combination of indices
// and looked up: tables of the row vectors after the first sites and of the
// column vectors before the last ones, which hold bit for bit what an index
// would compute by itself; and, for calls of kMatM indices or more, tables of
// the matrices of a few neighbouring sites in between (another association:
// such a call's values may differ from a smaller one's in their last bits).
// The cut is picked by counting FMAs: an index then costs one matrix per
// segment instead of one per site, and a table costs its own FMAs.
//
// A product formed ahead of its turn can leave FP64's range where the
// left-to-right products do not (four sites of 1e-100 after one of 1e250).
// So every entry formed out of order is looked at as it is stored
// (out_of_range: its exponent, and its terms where it is tiny), a table's
// entry that fails becomes a NaN, and an index that meets one, or whose value
// is not finite, is done again site by site from the left.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "ttg_eval.h"
#include "ttg_gemm_grid.cuh"

namespace ttg
{
namespace
{

constexpr int kEvalWarps = 8;  // per CTA, fewer where the vectors need the room
constexpr size_t kEvalSmemMax = 227 * 1024;

// Whether the sum y of the products x(i) p(i), i < m, formed before the
// factors to its left were known, may lack something that the left-to-right
// order keeps: it is within 2^24 of the largest double or beyond, or it is
// below 2^-900 and one of its own terms is (a larger entry has lost less than
// 2^-122 of itself; a small sum of larger terms, or of zeros, is what it is).
template <class FX, class FP>
__device__ __forceinline__ bool out_of_range(double y, int m, FX x, FP p)
{
  const int e = (__double2hiint(y) >> 20) & 0x7ff;
  if (e > 1023 + 1000)
    return true;
  if (e >= 1023 - 900)
    return false;
  for (int i = 0; i < m; ++i)
  {
    const double u = x(i), v = p(i);
    if (u != 0.0 && v != 0.0 && fabs(u * v) < 0x1p-900)
      return true;
  }
  return false;
}

// T[(i1 N2 + i2)][a][b] = sum_c A(i1, a, c) B(i2, c, b): the products of all
// pairs of two tables (or cores), one GEMM of (N1 ra) x (N2 rb) x K in
// 32 x 32 tiles.  mark: entries out of range become NaN.
__global__ void __launch_bounds__(256) merge_kernel(EvalMerge m)
{
  __shared__ double sm[GridTile<2>::kDoubles];
  const int M = m.N1 * m.ra, N = m.N2 * m.rb;
  const int tn = (N + 31) / 32;
  const int64_t tiles = static_cast<int64_t>((M + 31) / 32) * tn;
  auto A = [&](int row, int c) {
    return m.A[(row / m.ra) * m.iA + (row % m.ra) * m.aA + c * m.cA];
  };
  auto B = [&](int c, int col) { return m.B[(col / m.rb) * m.iB + c * m.aB + (col % m.rb)]; };
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x)
    grid_tile<2>(static_cast<int>(t / tn) * 32, static_cast<int>(t % tn) * 32, M, N, 0, m.K, A, B,
                 [&](int row, int col, double v) {
                   const int64_t i = static_cast<int64_t>(row / m.ra) * m.N2 + col / m.rb;
                   if (m.mark && out_of_range(v, m.K, [&](int c) { return A(row, c); },
                                              [&](int c) { return B(c, col); }))
                     v = __longlong_as_double(0x7ff8000000000000ll);
                   m.T[(i * m.ra + row % m.ra) * m.rb + col % m.rb] = v;
                 },
                 sm, m.cA == 1, m.rb == 1);
}

// y[j] = sum_i x[i] p[i * si + j * sj] for j < n, i < m, by the C lanes of a
// group (bl = lane in the group): each sum in ascending i, two j per lane at
// a time where there are that many.  kCheck: true when one of this lane's y is
// out of range.
template <int C, bool kCheck>
__device__ __forceinline__ bool group_mv(const double* p, int64_t si, int64_t sj, const double* x,
                                         int m, double* y, int n, int bl)
{
  bool lost = false;
  auto check = [&](double v, const double* q) {
    if (kCheck)
      lost = lost || out_of_range(v, m, [&](int i) { return x[i]; },
                                  [&](int i) { return q[i * si]; });
  };
  int j0 = 0;
  for (; j0 + C < n; j0 += 2 * C)
  {
    const int j = j0 + bl, j2 = j + C < n ? j + C : j;
    const double* a = p + j * sj;
    const double* b = p + j2 * sj;
    double acc = 0.0, acc2 = 0.0;
#pragma unroll 8
    for (int i = 0; i < m; ++i)
    {
      const double f = x[i];
      acc = fma(f, a[i * si], acc);
      acc2 = fma(f, b[i * si], acc2);
    }
    y[j] = acc;
    check(acc, a);
    if (j + C < n)
    {
      y[j + C] = acc2;
      check(acc2, b);
    }
  }
  if (j0 < n)
  {
    const int j = j0 + bl < n ? j0 + bl : j0;
    const double* a = p + j * sj;
    double acc = 0.0;
#pragma unroll 8
    for (int i = 0; i < m; ++i)
      acc = fma(x[i], a[i * si], acc);
    if (j0 + bl < n)
    {
      y[j0 + bl] = acc;
      check(acc, a);
    }
  }
  return lost;
}

// C lanes per multi-index.  segs[0, nl): the row vector's segments, the first
// a vector; segs[nl, nseg): the column vector's, the last a vector (none for
// a single site); segs[nseg, nseg + d): the single sites.  Shared memory: three vectors of rcap doubles per group
// and, with kStage, the segments, the modes and each group's d indices (a
// train too long for that reads them from global memory).
template <int C, bool kStage>
__global__ void __launch_bounds__(32 * kEvalWarps)
  eval_kernel(const EvalSeg* __restrict__ segs_g, int nl, int nseg, const int* __restrict__ modes_g,
              int d, const int* __restrict__ idx, int64_t M, double* __restrict__ out, int rcap,
              int* __restrict__ bad)
{
  extern __shared__ double evbuf[];
  constexpr int kPer = 32 / C;  // multi-indices per warp
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int sub = lane / C, bl = lane & (C - 1);
  const int grp = w * kPer + sub, ngrp = nw * kPer;
  double* s0 = evbuf + static_cast<int64_t>(grp) * 3 * rcap;
  EvalSeg* segs_s = reinterpret_cast<EvalSeg*>(evbuf + static_cast<int64_t>(ngrp) * 3 * rcap);
  int* modes_s = reinterpret_cast<int*>(segs_s + nseg);
  int* ix_s = modes_s + d + grp * d;
  if (kStage)
  {
    for (int t = threadIdx.x; t < nseg; t += blockDim.x)
      segs_s[t] = segs_g[t];
    for (int t = threadIdx.x; t < d; t += blockDim.x)
      modes_s[t] = modes_g[t];
    __syncthreads();
  }
  const EvalSeg* segs = kStage ? segs_s : segs_g;
  const int* modes = kStage ? modes_s : modes_g;
  const int64_t step = static_cast<int64_t>(gridDim.x) * ngrp;
  // The loop bound is the warp's; groups past the end redo the last index.
  for (int64_t first = static_cast<int64_t>(blockIdx.x) * ngrp + w * kPer; first < M; first += step)
  {
    const bool live = first + sub < M;
    const int64_t smp = live ? first + sub : M - 1;
    int mine = 0;
    for (int k = bl; k < d; k += C)
    {
      const int i = idx[smp * d + k];
      const bool in = i >= 0 && i < modes[k];
      mine |= in ? 0 : 1;
      if (kStage)
        ix_s[k] = in ? i : 0;
    }
    const unsigned wrong = __ballot_sync(0xffffffffu, mine != 0);
    const unsigned group_mask = (C == 32 ? 0xffffffffu : ((1u << C) - 1u)) << (sub * C);
    const bool ok = (wrong & group_mask) == 0u;
    __syncwarp();
    // Entry of a segment's table: the mixed-radix number of its sites' indices.
    auto entry = [&](const EvalSeg& s) {
      int64_t key = 0;
      for (int k = s.site; k < s.site + s.nsites; ++k)
      {
        int i = kStage ? ix_s[k] : idx[smp * d + k];
        if (!kStage && (i < 0 || i >= modes[k]))
          i = 0;
        key = key * modes[k] + i;
      }
      return s.p + key * s.i_stride;
    };
    double* s = s0;
    double* v = s0 + rcap;
    double* x = s0 + 2 * rcap;
    int rq = 1;
    bool lost = false;
    if (nl < nseg)
    {
      const EvalSeg& e = segs[nseg - 1];
      const double* p = entry(e);
      rq = e.r;
      for (int a = bl; a < rq; a += C)
        s[a] = p[a * e.a_stride];
      __syncwarp();
      for (int q = nseg - 2; q >= nl; --q)
      {
        const EvalSeg& g = segs[q];
        lost |= group_mv<C, true>(entry(g), 1, g.a_stride, s, g.rp, x, g.r, bl);
        rq = g.r;
        __syncwarp();
        double* t = s;
        s = x;
        x = t;
      }
    }
    {
      const EvalSeg& e = segs[0];
      const double* p = entry(e);
      for (int b = bl; b < e.rp; b += C)
        v[b] = p[b];
    }
    __syncwarp();
    for (int q = 1; q < nl; ++q)
    {
      const EvalSeg& g = segs[q];
      group_mv<C, false>(entry(g), g.a_stride, 1, v, g.r, x, g.rp, bl);
      __syncwarp();
      double* t = v;
      v = x;
      x = t;
    }
    double acc = 0.0;
    if (nl < nseg)
    {
      for (int a = bl; a < rq; a += C)
        acc = fma(v[a], s[a], acc);
#pragma unroll
      for (int o = C / 2; o > 0; o >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    else
      acc = v[0];
    const unsigned again = __ballot_sync(0xffffffffu, lost || !isfinite(acc));
    if (again)  // from the left, site by site (by the whole warp; others keep theirs)
    {
      __syncwarp();
      const EvalSeg* sites = segs_g + nseg;
      const double* p = entry(sites[0]);
      for (int b = bl; b < sites[0].rp; b += C)
        v[b] = p[b];
      __syncwarp();
      for (int k = 1; k < d; ++k)
      {
        const EvalSeg& g = sites[k];
        group_mv<C, false>(entry(g), g.a_stride, 1, v, g.r, x, g.rp, bl);
        __syncwarp();
        double* t = v;
        v = x;
        x = t;
      }
      if (again & group_mask)
        acc = v[0];
    }
    if (bl == 0 && live)
    {
      out[smp] = ok ? acc : __longlong_as_double(0x7ff8000000000000ll);
      if (!ok)
        atomicExch(bad, 1);
    }
    __syncwarp();
  }
}

// Table limits: a matrix table and all of them together stay inside the
// 129 MB L2 beside the vector tables' lines in use; a vector table is read
// once per index, from HBM at worst.
constexpr double kMatDoubles = 6.0e6, kMatTotal = 1.3e7, kVecDoubles = 1.7e7;
// FMAs that one more launch is worth: ~3 us at the chip's 0.6 TFMA/s (0 / 5e5 /
// 2e6 / 8e6, d=30 n=2 rank 16: 3000 indices 0.29 / 0.29 / 0.20 / 0.20 ms, 30 000
// 0.42 / 0.41 / 0.41 / 0.61).
constexpr double kLaunchFma = 2.0e6;
constexpr int kMostSites = 16;
// Matrix tables from this many indices on; column-vector tables of at most
// kRightN entries (and never past the middle), so that where the two vectors
// meet depends on the train alone.  Matrix tables on : off, ms: d=32 n=4 rank 64
// 8000 indices 1.45 : 1.93, 32 768 2.76 : 4.91, 2^20 28.9 : 110; rank 16 16 000
// 0.44 : 0.39, 32 768 0.50 : 0.55, 131 072 0.79 : 1.33; d=12 n=8 rank 24 32 768
// 0.33 : 0.38.  kRightN of 1 / 256 / 4096 / 65536 / 1e6, 3e5 indices: d=32 n=4 rank
// 64 12.3 / 19.6 / 18.6 / 10.9 / 12.9 ms, d=10 n=16 rank 30 1.64 / 1.55 / 1.25 / 1.14
// / 1.15; 3e4 indices 5.2 / 4.9 / 4.5 / 4.8 / 5.0 and 0.49 / 0.44 / 0.41 / 0.43 / 0.43.
constexpr int64_t kMatM = 1 << 15;
constexpr double kRightN = 65536;

// The site where the row and the column vector meet: 1 <= q < d (d for a
// single site).
int eval_split(const int* n, int d)
{
  if (d == 1)
    return 1;
  int q = d - 1;
  double N = n[d - 1];
  while (q > 1 && q > d / 2 && N * n[q - 1] <= kRightN)
    N *= n[--q];
  return q;
}

}  // namespace

EvalLayout plan_eval(const int* r, const int* n, int d, int64_t M)
{
  EvalLayout L;
  const double m = static_cast<double>(M);
  const int q = eval_split(n, d);
  // Left part [0, q): dynamic programming over the segments' ends.
  std::vector<double> best(q + 1, INFINITY);
  std::vector<int> from(q + 1, -1);
  double N = 1, cost = 0;
  for (int p = 1; p <= q; ++p)
  {
    N *= n[p - 1];
    if (p > 1)
    {
      cost += N * r[p - 1] * r[p] + kLaunchFma;
      if (p > kMostSites || N > m || N * r[p] > kVecDoubles)
        break;
    }
    best[p] = cost;
    from[p] = 0;
  }
  for (int s = 1; s < q; ++s)
  {
    double Ns = n[s], build = 0;
    for (int e = s + 1; e <= q; ++e)
    {
      if (e > s + 1)
      {
        Ns *= n[e - 1];
        build += Ns * r[s] * r[e - 1] * r[e] + kLaunchFma;
        if (M < kMatM || e - s > kMostSites || Ns > m || Ns * r[s] * r[e] > kMatDoubles)
          break;
      }
      const double c = best[s] + build + m * r[s] * r[e];
      if (c < best[e])
      {
        best[e] = c;
        from[e] = s;
      }
    }
  }
  std::vector<int> left;
  for (int e = q; e > 0; e = from[e])
    left.push_back(from[e]);
  std::reverse(left.begin(), left.end());
  left.push_back(q);
  // Matrix tables beyond the L2 budget: single sites from there on.
  double mats = 0;
  for (size_t i = 0; i + 1 < left.size(); ++i)
  {
    const int s = left[i], e = left[i + 1];
    double Ns = 1;
    for (int k = s; k < e; ++k)
      Ns *= n[k];
    const bool matrix = s > 0 && e - s > 1;
    if (matrix && mats + Ns * r[s] * r[e] > kMatTotal)
      for (int k = s; k < e; ++k)
        L.cut.push_back(k);
    else
    {
      if (matrix)
        mats += Ns * r[s] * r[e];
      L.cut.push_back(s);
    }
  }
  L.left = static_cast<int>(L.cut.size());
  // Right part [q, d): single sites, then the table [x, d).
  if (q < d)
  {
    double single = 0;
    for (int k = q; k < d - 1; ++k)
      single += m * r[k] * r[k + 1];
    double least = single;
    int x_best = d - 1;
    N = n[d - 1];
    cost = 0;
    for (int x = d - 2; x >= q; --x)
    {
      N *= n[x];
      cost += N * r[x] * r[x + 1] + kLaunchFma;
      single -= m * r[x] * r[x + 1];
      if (d - x > kMostSites || N > m || N * r[x] > kVecDoubles)
        break;
      if (single + cost < least)
      {
        least = single + cost;
        x_best = x;
      }
    }
    for (int k = q; k <= x_best; ++k)
      L.cut.push_back(k);
  }
  L.cut.push_back(d);
  // Table space: every level of every table.
  for (size_t i = 0; i + 1 < L.cut.size(); ++i)
  {
    const int s = L.cut[i], e = L.cut[i + 1];
    if (e - s < 2)
      continue;
    const bool right = static_cast<int>(i) >= L.left;
    int64_t Nt = right ? n[d - 1] : n[s];
    for (int j = 1; j < e - s; ++j)
    {
      Nt *= right ? n[d - 1 - j] : n[s + j];
      const int64_t ra = right ? r[d - 1 - j] : r[s], rb = right ? 1 : r[s + j + 1];
      L.table_doubles += (Nt * ra * rb + 31) / 32 * 32;
    }
  }
  return L;
}

// Segments, then the single sites, and the merges that fill the segments'
// tables, for cores at ar + off[k] and tables from `tab` on.
void lay_out_eval(const EvalLayout& L, const int* r, const int* n, const int64_t* off, int d,
                  const double* ar, double* tab, std::vector<EvalSeg>& segs,
                  std::vector<EvalMerge>& merges)
{
  segs.clear();
  merges.clear();
  auto take = [&](int64_t m) {
    double* p = tab;
    tab += (m + 31) / 32 * 32;
    return p;
  };
  for (size_t i = 0; i + 1 < L.cut.size(); ++i)
  {
    const int s = L.cut[i], e = L.cut[i + 1];
    const bool suffix = static_cast<int>(i) >= L.left && e - s > 1;
    EvalSeg g{};
    g.site = s;
    g.nsites = e - s;
    g.r = r[s];
    g.rp = r[e];
    // Core k as a table: index stride r', row stride n r'.
    const int k0 = suffix ? d - 1 : s;
    const double* p = ar + off[k0];
    int64_t is = r[k0 + 1], as = static_cast<int64_t>(n[k0]) * r[k0 + 1], N = n[k0];
    for (int j = 1; j < e - s; ++j)
    {
      EvalMerge m{};
      m.mark = suffix || s > 0;  // the row vectors are the left-to-right products
      const int k = suffix ? d - 1 - j : s + j;
      const int64_t ck_i = r[k + 1], ck_a = static_cast<int64_t>(n[k]) * r[k + 1];
      if (suffix)
      {
        m.A = ar + off[k];
        m.iA = ck_i;
        m.aA = ck_a;
        m.cA = 1;
        m.N1 = n[k];
        m.ra = r[k];
        m.K = r[k + 1];
        m.B = p;
        m.iB = is;
        m.aB = as;
        m.N2 = static_cast<int>(N);
        m.rb = 1;
      }
      else
      {
        m.A = p;
        m.iA = is;
        m.aA = as;
        m.cA = 1;
        m.N1 = static_cast<int>(N);
        m.ra = r[s];
        m.K = r[k];
        m.B = ar + off[k];
        m.iB = ck_i;
        m.aB = ck_a;
        m.N2 = n[k];
        m.rb = r[k + 1];
      }
      N *= n[k];
      m.T = take(N * m.ra * m.rb);
      merges.push_back(m);
      p = m.T;
      is = static_cast<int64_t>(m.ra) * m.rb;
      as = m.rb;
    }
    g.p = p;
    g.i_stride = is;
    g.a_stride = as;
    segs.push_back(g);
  }
  for (int k = 0; k < d; ++k)
    segs.push_back(EvalSeg{ar + off[k], r[k + 1], static_cast<int64_t>(n[k]) * r[k + 1], r[k], r[k + 1],
                           k, 1});
}

namespace
{

// Shape of a launch: lanes per index (the largest rank, 8 to 32), warps per
// CTA, whether the segments and indices are staged, shared memory.  8 / 16 / 32
// lanes, d=20 n=4, ms: 33 indices of rank 9 0.116 / 0.106 / 0.106, 24 0.20 / 0.18 /
// 0.13, 32 0.30 / 0.21 / 0.16 (more lanes shorten one index's chain); 3e5 of rank 8
// 0.46 / 0.54 / 0.67, 12 0.57 / 0.62 / 0.77, 32 1.27 / 1.31 / 1.37.
struct EvalShape
{
  int lanes, warps;
  bool stage;
  size_t smem;
};

EvalShape eval_shape(int nseg, int d, int rmax, int rcap)
{
  EvalShape z{rmax <= 8 ? 8 : (rmax <= 16 ? 16 : 32), kEvalWarps, true, 0};
  const size_t per = static_cast<size_t>(32 / z.lanes);  // indices per warp
  const size_t vec = sizeof(double) * 3 * static_cast<size_t>(rcap) * per;
  while (z.warps > 1 && vec * z.warps > kEvalSmemMax)
    --z.warps;
  z.smem = vec * z.warps;
  const size_t staged = z.smem + sizeof(EvalSeg) * static_cast<size_t>(nseg) +
                        sizeof(int) * static_cast<size_t>(d) * (1 + per * z.warps);
  z.stage = staged <= kEvalSmemMax;
  if (z.stage)
    z.smem = staged;
  return z;
}

using EvalKernel = void (*)(const EvalSeg*, int, int, const int*, int, const int*, int64_t, double*,
                            int, int*);

EvalKernel eval_instance(const EvalShape& z)
{
  if (z.stage)
    return z.lanes == 8 ? eval_kernel<8, true> : (z.lanes == 16 ? eval_kernel<16, true>
                                                                : eval_kernel<32, true>);
  return z.lanes == 8 ? eval_kernel<8, false> : (z.lanes == 16 ? eval_kernel<16, false>
                                                               : eval_kernel<32, false>);
}

}  // namespace

cudaError_t eval_smem_optin(int nseg, int d, int rmax, int rcap)
{
  const EvalShape z = eval_shape(nseg, d, rmax, rcap);
  return cudaFuncSetAttribute(eval_instance(z), cudaFuncAttributeMaxDynamicSharedMemorySize,
                              static_cast<int>(z.smem));
}

void launch_eval(const std::vector<EvalMerge>& merges, const EvalSeg* segs, int left, int nseg,
                 const int* modes, int d, const int* idx, int64_t M, double* out, int rmax, int rcap,
                 int* bad, int sms, cudaStream_t stream)
{
  for (const EvalMerge& m : merges)
  {
    const int64_t tiles = ((static_cast<int64_t>(m.N1) * m.ra + 31) / 32) *
                          ((static_cast<int64_t>(m.N2) * m.rb + 31) / 32);
    merge_kernel<<<static_cast<int>(std::min<int64_t>(tiles, 8LL * sms)), 256, 0, stream>>>(m);
  }
  const EvalShape z = eval_shape(nseg, d, rmax, rcap);
  const int64_t per = static_cast<int64_t>(z.warps) * (32 / z.lanes);
  const int grid =
    static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((M + per - 1) / per, 8LL * sms)));
  eval_instance(z)<<<grid, 32 * z.warps, z.smem, stream>>>(segs, left, nseg, modes, d, idx, M, out,
                                                           rcap, bad);
}

}  // namespace ttg
