// The configurations that the autotuner times (ttg_tune.h), on the host.
#include <cstdio>

#include "ttg_tune.h"

using namespace ttg;

static int g_fail = 0;
#define CHECK(cond)                                   \
  do                                                  \
    if (!(cond))                                      \
    {                                                 \
      std::printf("line %d: %s\n", __LINE__, #cond);  \
      ++g_fail;                                       \
    }                                                 \
  while (0)

int main()
{
  const int sms = 152;
  for (int items : {1, 100, 152, 153, 304, 305, 400, 455, 456, 700, 5000})
    for (int rows : {16, 608, 609, 768, 896, 897, 1280, 1472, 1473, 4000})
    {
      TuneInput in;
      in.items = items;
      in.sms = sms;
      in.scratch_ctas = items > 2 * sms ? (items < 4 * sms ? items : 4 * sms)
                                        : (items < 2 * sms ? items : 2 * sms);
      const int fp64 = static_cast<int>(tune_configs(in).size());
      CHECK(fp64 == (items <= sms ? 1 : (items <= 2 * sms ? 2 : (items <= 3 * sms ? 3 : 4))));
      in.form_doubles = items <= sms ? kSmemOnePerSm : (items >= 3 * sms ? kSmemThreePerSm : kSmemTwoPerSm);
      in.panel_doubles = static_cast<int64_t>(rows) * kWyB;
      // Every launch of a mixed plan factors each panel the same way: blocked
      // (its staging is within the form) only where its CTAs can stage it.
      const auto mixed = tune_configs(in);
      CHECK(!mixed.empty());
      for (const TuneConfig& c : mixed)
        for (int h = 8; h <= rows; ++h)
          if (static_cast<int64_t>(h) * kWyB <= in.form_doubles)
            CHECK(static_cast<int64_t>(h) * kWyB <= c.smem);
      if (rows <= 608)
        CHECK(static_cast<int>(mixed.size()) == fp64);
    }
  // Block widths of the whole-GPU Jacobi sweeps fit the shared memory.
  for (int64_t c_max : {64, 257, 533, 800, 1066, 2133})
  {
    TuneInput in;
    in.items = 1;
    in.sms = in.scratch_ctas = sms;
    in.can_wide = true;
    in.wide_grid = sms;
    in.c_max = c_max;
    for (const TuneConfig& c : tune_configs(in))
      if (c.wide)
        CHECK((6 * c_max + 2) * c.jblock <= c.smem);
  }
  // The plan's own configuration is among them, first, and each only once: the
  // teams that a few FP64 trains start in (one each, 2 to 30), a lone train over
  // part of the GPU, and any number of CTAs per SM.
  for (int items = 2; items <= 30; ++items)
  {
    TuneInput in;
    in.items = items;
    in.sms = in.scratch_ctas = sms;
    in.can_wide = in.wide = true;
    in.wide_grid = sms;
    in.c_max = 96;
    in.jblock = 4;
    in.teams = in.wide_teams_max = items;
    const auto all = tune_configs(in);
    CHECK(all[0].wide && all[0].teams == items && all[0].code == 10000 + items);
    int per_tt = 0;
    for (size_t i = 1; i < all.size(); ++i)
    {
      CHECK(all[i].code != all[0].code);
      per_tt += !all[i].wide;
    }
    CHECK(per_tt == 1);
  }
  for (int b : {1, 2, 4, 8})
  {
    TuneInput in;
    in.items = 1;
    in.sms = in.scratch_ctas = sms;
    in.can_wide = in.wide = true;
    in.wide_grid = 16;
    in.c_max = 48;
    in.jblock = b;
    const auto all = tune_configs(in);
    CHECK(all[0].wide && all[0].teams == 1 && all[0].code == 100 + b && all[0].grid == 16);
    CHECK(all.size() == (b == 1 ? 5u : 4u));
  }
  for (int cps = 1; cps <= 4; ++cps)
  {
    TuneInput in;
    in.items = 5000;
    in.sms = sms;
    in.scratch_ctas = 4 * sms;
    in.cps = cps;
    const auto all = tune_configs(in);
    CHECK(all[0].code == cps && all[0].grid == cps * sms && all.size() == 4u);
  }
  std::printf(g_fail ? "FAILED\n" : "OK\n");
  return g_fail ? 1 : 0;
}
