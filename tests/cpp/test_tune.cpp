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
  std::printf(g_fail ? "FAILED\n" : "OK\n");
  return g_fail ? 1 : 0;
}
