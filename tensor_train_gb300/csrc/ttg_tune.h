// The launch configurations that ttg_plan_autotune times (host only).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "ttg_job.h"

namespace ttg
{

// Doubles of shared memory per CTA of the sweep kernel at 1 to 4 CTAs per SM.
constexpr int kSmemOnePerSm = 25600;   // 200 KB
constexpr int kSmemTwoPerSm = 11776;   // 92 KB
constexpr int kSmemThreePerSm = 7168;  // 56 KB
constexpr int kSmemFourPerSm = 4864;   // 38 KB
constexpr int kSmemPerSm[5] = {0, kSmemOnePerSm, kSmemTwoPerSm, kSmemThreePerSm, kSmemFourPerSm};

struct TuneConfig
{
  int code;  // 1-4: per TT, CTAs per SM; 100 + b (+ 1000 with tensor cores): whole GPU; 10000 + teams
  bool wide;
  int grid, smem, jblock, tc, cps, teams = 1;
};

// What decides which configurations a plan may run in.
struct TuneInput
{
  int items = 0, sms = 0, scratch_ctas = 0;
  // df64 factorisations of matrices beyond form_doubles are blocked where the
  // panel's staging fits in as many (Smem::form); panel_doubles: the largest
  // staging that a step of the plan can ask for.  0 for FP64 plans.
  int form_doubles = 0;
  int64_t panel_doubles = 0;
  // whole-GPU and team schedules, where the plan has their work buffers
  bool can_wide = false;
  int wide_grid = 0, wide_teams_max = 1;
  bool tensor_cores = false;
  int64_t c_max = 1;  // largest rank
  // as the plan stands
  int cps = 1, jblock = 1, tc = 0, teams = 1;
  bool wide = false;
};

// Whether CTAs with `smem` doubles take the same form of every factorisation
// as any other launch of the plan: they can stage each panel that the form has
// blocked.  (The forms round differently, and a batch of hundreds of trains
// holds singular values close enough together to show it.)
inline bool keeps_form(const TuneInput& in, int smem)
{
  return std::min<int64_t>(in.form_doubles, in.panel_doubles) <= smem;
}

// The plan's own configuration first, so that tuning cannot leave it slower.
inline std::vector<TuneConfig> tune_configs(const TuneInput& in)
{
  const int grid0 = std::max(1, std::min(in.items, in.cps * in.sms));
  std::vector<TuneConfig> out;
  if (!in.wide)
    out.push_back({in.cps, false, grid0, kSmemPerSm[in.cps], in.jblock, in.tc, in.cps});
  else if (in.teams > 1)
    out.push_back({10000 + in.teams, true, in.wide_grid, kSmemOnePerSm, in.jblock, in.tc, 1, in.teams});
  else
    out.push_back({100 + in.jblock + 1000 * in.tc, true, in.wide_grid, kSmemOnePerSm, in.jblock,
                   in.tc, 1, 1});
  auto add = [&](const TuneConfig& c) {
    if (c.code != out[0].code)
      out.push_back(c);
  };
  int last = 0;
  for (int cps = 1; cps <= 4; ++cps)
  {
    const int grid = std::max(1, std::min(in.items, cps * in.sms));
    if (grid > last && (cps <= 2 || grid <= in.scratch_ctas) && keeps_form(in, kSmemPerSm[cps]))
      add({cps, false, grid, kSmemPerSm[cps], in.jblock, in.tc, cps});
    last = grid;
  }
  if (in.can_wide && in.wide_teams_max <= 1)
  {
    // The sliced-BF16 tensor-core tiles are tried only when they were
    // opted into (TTG_WIDE_TENSOR_CORES=1): they are no faster on these
    // barrier-bound sweeps and carry ~1e-12 instead of FP64 rounding per
    // product, which reached 2.6e-10 on the d=40 rank-257 round.
    for (int tc = 0; tc <= (in.tensor_cores ? 1 : 0); ++tc)
      for (int b : {2, 4, 8})
        if ((6 * in.c_max + 2) * b <= kSmemOnePerSm)
          add({100 + b + 1000 * tc, true, in.wide_grid, kSmemOnePerSm, b, tc, 1, 1});
  }
  else if (in.can_wide)
    for (int t : {4, 8, 16, 32})
      if (t <= in.wide_teams_max)
        add({10000 + t, true, in.wide_grid, kSmemOnePerSm, in.jblock, 0, 1, t});
  return out;
}

}  // namespace ttg
