// The FP64 scalars that the QRs and the certificate form from the hardware's
// approximations, against long double, over FP64's range: reflector_scalars
// (ttg_reflector.cuh) and CertOps<double>::recip (ttg_device_df.cuh).
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "ttg_device_df.cuh"
#include "ttg_reflector.cuh"

__global__ void scalars(const double* s, const double* ax, int n, double* out)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n)
    return;
  ttg::reflector_scalars(s[i], ax[i], out + 4 * i, out + 4 * i + 1, out + 4 * i + 2);
  out[4 * i + 3] = ttg::CertOps<double>::recip(s[i]);
}

int main()
{
  const int n = 1 << 17;
  std::mt19937_64 g(3);
  std::uniform_real_distribution<double> unit(0.0, 1.0);
  std::vector<double> s(n), ax(n), out(4 * n);
  for (int i = 0; i < n; ++i)
  {
    // s from DBL_MIN to DBL_MAX (for recip also subnormal), |x0| from nothing of it to all.
    s[i] = std::ldexp(1.0 + unit(g), static_cast<int>(2046.0 * unit(g)) - 1022);
    ax[i] = i % 5 == 0 ? 0.0 : (i % 5 == 1 ? std::sqrt(s[i]) : std::sqrt(s[i]) * std::pow(10.0, -18.0 * unit(g)));
    if (i % 101 == 0)
      s[i] = std::ldexp(1.0 + unit(g), -1023 - static_cast<int>(40.0 * unit(g)));
    if (i % 103 == 0)
      s[i] = std::ldexp(1.0 + unit(g), 1018 + i % 6);
  }
  double *ds = nullptr, *da = nullptr, *d = nullptr;
  if (cudaMalloc(&ds, 8 * n) || cudaMalloc(&da, 8 * n) || cudaMalloc(&d, 32 * n))
    return 2;
  cudaMemcpy(ds, s.data(), 8 * n, cudaMemcpyHostToDevice);
  cudaMemcpy(da, ax.data(), 8 * n, cudaMemcpyHostToDevice);
  scalars<<<n / 256, 256>>>(ds, da, n, d);
  if (cudaMemcpy(out.data(), d, 32 * n, cudaMemcpyDeviceToHost))
    return 2;
  const long double u = ldexpl(1.0L, -53);
  long double wn = 0.0L, wr = 0.0L, wi = 0.0L, wc = 0.0L;
  for (int i = 0; i < n; ++i)
  {
    const double* o = &out[4 * i];
    const long double root = sqrtl(static_cast<long double>(s[i]));
    if (s[i] > 2.2250738585072014e-308)  // as has_tail has it
    {
      wn = fmaxl(wn, fabsl(o[0] / root - 1.0L));
      wr = fmaxl(wr, fabsl(o[1] * root - 1.0L));
      if (ax[i] <= root * (1.0L + 8 * u))
        wi = fmaxl(wi, fabsl(o[2] * (ax[i] + root) - 1.0L));
    }
    const long double inv = 1.0L / s[i];
    // A result below DBL_MIN rounds to a multiple of 2^-1074.
    const long double ulp = fmaxl(u * inv, ldexpl(0.5L, -1074));
    if (inv < 1.797e308L)
      wc = fmaxl(wc, fabsl(o[3] - inv) / ulp);
    else if (!std::isinf(o[3]) && !(o[3] > 1.79e308))
      wc = 1e9L;
  }
  const bool ok = wn <= 1.1L * u && wr <= 1.1L * u && wi <= 2.6L * u && wc <= 1.1L;
  std::printf("%s: in 2^-53: n %.3Lf, 1/n %.3Lf, 1/(|x0| + n) %.3Lf, 1/a %.3Lf\n", ok ? "OK" : "FAILED",
              wn / u, wr / u, wi / u, wc);
  return ok ? 0 : 1;
}
