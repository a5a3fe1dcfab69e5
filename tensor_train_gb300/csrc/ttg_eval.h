// Batched evaluation (ttg_eval.cu): segments of the train and the tables of
// their products.
#pragma once

#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

namespace ttg
{

// Sites [site, site + nsites) as one factor: for the mixed-radix number i of
// their indices, the r x rp matrix p[i * i_stride + a * a_stride + b].
struct EvalSeg
{
  const double* p;
  int64_t i_stride, a_stride;
  int32_t r, rp, site, nsites;
};

// T[(i1 N2 + i2)][a][b] = sum_{c < K} A(i1, a, c) B(i2, c, b); mark: NaN where
// that left FP64's range.
struct EvalMerge
{
  const double* A;
  int64_t iA, aA, cA;
  const double* B;
  int64_t iB, aB;
  double* T;
  int32_t N1, ra, K, N2, rb, mark;
};

// Cut points 0 = cut[0] < ... < d of the segments; a segment of two or more
// sites has a table.  The first `left` segments carry the row vector.
struct EvalLayout
{
  std::vector<int> cut;
  int left = 0;
  int64_t table_doubles = 0;
};

// The cheapest cut for M multi-indices of a train of ranks r[0..d] and modes
// n[0..d).
EvalLayout plan_eval(const int* r, const int* n, int d, int64_t M);
void lay_out_eval(const EvalLayout& L, const int* r, const int* n, const int64_t* off, int d,
                  const double* ar, double* tab, std::vector<EvalSeg>& segs,
                  std::vector<EvalMerge>& merges);
cudaError_t eval_smem_optin(int nseg, int d, int rmax, int rcap);
void launch_eval(const std::vector<EvalMerge>& merges, const EvalSeg* segs, int left, int nseg,
                 const int* modes, int d, const int* idx, int64_t M, double* out, int rmax, int rcap,
                 int* bad, int sms, cudaStream_t stream);

}  // namespace ttg
