// Buffer sizes of the inner-product chain (ttg_inner.h), on the host: the
// partial environments fit wherever the kernel stores them, and an environment
// that fills the GPU takes no more than itself.
#include <cstdio>
#include <vector>

#include "ttg_inner.h"

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

static std::vector<CoreSlot> train(int d, int n, int r)
{
  std::vector<CoreSlot> s(d);
  for (int k = 0; k < d; ++k)
  {
    s[k].r = k ? r : 1;
    s[k].n = n;
    s[k].rp = k < d - 1 ? r : 1;
  }
  return s;
}

int main()
{
  const int sms = 152;
  for (int ra : {1, 2, 15, 16, 17, 33, 96, 97, 130, 200, 400, 2000, 23170})
    for (int rb : {1, 3, 16, 96, 113, 400, 2000, 23170})
      for (int n : {1, 2, 4})
        for (int d : {1, 2, 3, 5})
        {
          const std::vector<CoreSlot> a = train(d, n, ra), b = train(d, n, rb);
          const InnerSizes z = inner_sizes(a.data(), b.data(), d, sms);
          CHECK(z.grid >= 1 && z.grid <= sms);
          int64_t env = 1, tmp = 1;
          for (int k = 0; k < d; ++k)
          {
            const int64_t one = static_cast<int64_t>(a[k].rp) * b[k].rp;
            const int s = inner_slices(a[k].rp, b[k].rp, b[k].r * n, z.grid);
            CHECK(s >= 1 && s <= kInnerSlices);
            CHECK(s * one <= z.env);
            env = std::max(env, one);
            tmp = std::max(tmp, static_cast<int64_t>(b[k].r) * n * a[k].rp);
          }
          CHECK(tmp <= z.scratch() - 2 * z.env - 32);
          // One environment of 152 tiles or more is not sliced.
          if (env >= 256 * int64_t{sms} * 4)
            CHECK(z.scratch() <= 2 * env + tmp + 128);
        }
  if (g_fail == 0)
    std::printf("ok\n");
  return g_fail != 0;
}
