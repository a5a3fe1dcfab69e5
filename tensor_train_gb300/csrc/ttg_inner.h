// Launch and buffer sizes of the inner-product chain (ttg_inner.cu).
#pragma once

#include <algorithm>
#include <cstdint>

#include "ttg_job.h"

namespace ttg
{

constexpr int kInnerSlices = 4;  // most partial environments

// Slices of the inner dimension K of an (M x N) environment: enough tiles
// for the grid, at most kInnerSlices, none shorter than a 32-deep slab.
TTG_HD inline int inner_slices(int M, int N, int K, int grid)
{
  const int64_t tiles = static_cast<int64_t>((M + 15) / 16) * ((N + 15) / 16);
  int64_t s = grid / tiles;
  s = s < (K + 31) / 32 ? s : (K + 31) / 32;
  s = s < kInnerSlices ? s : kInnerSlices;
  return s < 1 ? 1 : static_cast<int>(s);
}

// Sizes of the chain of the TTs a and b: CTAs, and the doubles of one
// environment with its partials and of T.  An environment large enough to
// fill the GPU by itself is not sliced and has no room for partials: at rank
// 20 000 they would be 9.6 GB each.
struct InnerSizes
{
  int grid = 1;
  int64_t env = 1, tmp = 1;
  // [environment | next environment | T | value and barrier word]
  int64_t scratch() const { return 2 * env + a32(tmp) + 32; }
};

inline InnerSizes inner_sizes(const CoreSlot* a, const CoreSlot* b, int d, int sms)
{
  InnerSizes z;
  auto t16 = [](int64_t n) { return (n + 15) / 16; };
  int64_t tiles = 1;  // the most 16 x 16 output tiles of any one product
  for (int k = 0; k < d; ++k)
  {
    const int64_t n = a[k].n;
    z.tmp = std::max(z.tmp, b[k].r * n * a[k].rp);
    tiles = std::max({tiles, t16(b[k].r) * t16(n * a[k].rp),
                      std::min<int64_t>(kInnerSlices, (b[k].r * n + 31) / 32) * t16(a[k].rp) *
                        t16(b[k].rp)});
  }
  z.grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(tiles, sms)));
  for (int k = 0; k < d; ++k)
    z.env = std::max(z.env, static_cast<int64_t>(a[k].rp) * b[k].rp *
                              inner_slices(a[k].rp, b[k].rp, b[k].r * a[k].n, z.grid));
  z.env = a32(z.env);
  return z;
}

}  // namespace ttg
