// Backward pass of the rank model in one kernel, for widths of at most 128
// and at most 32 features (ttg_mlp.cu holds the layout and the forward pass).
//
// At the trainer's sizes (4096 rows, 10 features, width 128) the backward
// pass is 0.28 GFLOP on 4.5 MB; as separate GEMMs, masks and column sums it
// was 19 launches and 0.78 ms, most of it in kernels of one CTA (a product
// with a 4096-long inner dimension, one thread per column sum).  Here a CTA
// keeps W2 in shared memory and takes 32 rows at a time; its parameter
// gradients stay in registers over its rows and leave once, as one partial
// per CTA that mlp_reduce_kernel adds in CTA order (the result does not
// depend on scheduling).  Every product is the split-BF16 one of the
// tensor-core GEMMs (hi hi + hi lo + lo hi with x = hi + lo), as three FP32
// FMAs: an operand is kept as one word, hi above lo, and a thread's 4 x 4
// block reads 8 words per 48 FMAs.
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace ttg
{
namespace
{

constexpr int kMlpW = 128;     // padded width
constexpr int kMlpF = 32;      // most features
constexpr int kMlpRows = 32;   // rows per turn
constexpr int kMlpThreads = 256;
constexpr int kMlpLdW = kMlpW + 1;  // odd: W2 is read down its columns
constexpr int kMlpLdH = kMlpW + 4;  // 16-byte rows for the broadcast reads

struct MlpShared
{
  uint32_t W2[kMlpW * kMlpLdW];
  uint32_t H1[kMlpRows * kMlpLdH];
  uint32_t D2[kMlpRows * kMlpLdH];  // dZ2
  uint32_t D1[kMlpRows * kMlpLdH];  // dZ1
  uint32_t x[kMlpRows * kMlpF];
  uint32_t W3[kMlpW];
  float colsum[3][kMlpThreads / 32][kMlpW];
  float gb3[kMlpThreads / 32];
  double loss[kMlpThreads / 32];
};

// A float as the two BF16 values hi = bf16(x), lo = bf16(x - hi) in a word.
__device__ __forceinline__ uint32_t mlp_pack(float x)
{
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
  return (static_cast<uint32_t>(__bfloat16_as_ushort(h)) << 16) | __bfloat16_as_ushort(l);
}
__device__ __forceinline__ float mlp_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }
__device__ __forceinline__ float mlp_lo(uint32_t w) { return __uint_as_float(w << 16); }
// acc + hi hi + hi lo + lo hi.
__device__ __forceinline__ float mlp_fma(uint32_t a, uint32_t b, float acc)
{
  acc = fmaf(mlp_hi(a), mlp_hi(b), acc);
  acc = fmaf(mlp_hi(a), mlp_lo(b), acc);
  return fmaf(mlp_lo(a), mlp_hi(b), acc);
}

// acc[r][c] = sum_k A[row 4w + r][k] B(k, lane + 32 c) for k < kMlpW; A in
// shared memory with leading dimension kMlpLdH, B(k, j) = W2[j][k].
__device__ __forceinline__ void mlp_gemm(const uint32_t* A, const uint32_t* W2, int w, int lane,
                                         float acc[4][4])
{
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c)
      acc[r][c] = 0.f;
#pragma unroll 1
  for (int k = 0; k < kMlpW; k += 4)
  {
    uint4 a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
      a[r] = *reinterpret_cast<const uint4*>(A + (4 * w + r) * kMlpLdH + k);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < 4; ++c)
      {
        const int j = lane + 32 * c;
        const uint32_t b = W2[j * kMlpLdW + k + q];
#pragma unroll
        for (int r = 0; r < 4; ++r)
          acc[r][c] = mlp_fma(q == 0 ? a[r].x : (q == 1 ? a[r].y : (q == 2 ? a[r].z : a[r].w)), b,
                              acc[r][c]);
      }
  }
}

// Z1, Z2: pre-activations (N x H), y: the model's outputs.  part: nparams
// floats per CTA in parameter order; loss_part: one double per CTA.
__global__ void __launch_bounds__(kMlpThreads, 1)
  mlp_back_kernel(const float* __restrict__ W2, const float* __restrict__ W3, int F, int H,
                  const float* __restrict__ x, const float* __restrict__ t, int N,
                  const float* __restrict__ Z1, const float* __restrict__ Z2,
                  const float* __restrict__ y, float* __restrict__ part, int nparams,
                  double* __restrict__ loss_part)
{
  extern __shared__ __align__(16) unsigned char mlp_smem[];
  MlpShared& s = *reinterpret_cast<MlpShared*>(mlp_smem);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  for (int e = tid; e < kMlpW * kMlpW; e += kMlpThreads)
  {
    const int k = e / kMlpW, j = e % kMlpW;
    s.W2[k * kMlpLdW + j] = mlp_pack((k < H && j < H) ? W2[k * H + j] : 0.f);
  }
  if (tid < kMlpW)
    s.W3[tid] = mlp_pack(tid < H ? W3[tid] : 0.f);
  // Gradient accumulators of this thread over all its CTA's rows: gW2 rows
  // ty + 16 a, columns tx + 16 b; gW1 column jc, features half + 2 q; its
  // rows' share of the column sums of columns lane + 32 c.
  const int tx = tid & 15, ty = tid >> 4;
  const int jc = tid & (kMlpW - 1), half = tid / kMlpW;
  float g2[8][8], g1[kMlpF / 2], gb1[4], gb2[4], gw3[4];
  float gb3 = 0.f;
  double loss = 0.0;
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b)
      g2[a][b] = 0.f;
#pragma unroll
  for (int q = 0; q < kMlpF / 2; ++q)
    g1[q] = 0.f;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    gb1[c] = gb2[c] = gw3[c] = 0.f;
  for (int64_t r0 = static_cast<int64_t>(blockIdx.x) * kMlpRows; r0 < N;
       r0 += static_cast<int64_t>(gridDim.x) * kMlpRows)
  {
    __syncthreads();
    for (int e = tid; e < kMlpRows * F; e += kMlpThreads)
    {
      const int64_t i = r0 + e / F;
      s.x[(e / F) * kMlpF + e % F] = mlp_pack(i < N ? x[i * F + e % F] : 0.f);
    }
    float z1[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
    {
      const int64_t i = r0 + 4 * w + r;
      const bool live = i < N;
      const float e = live ? y[i] - t[i] : 0.f;
      const float dyi = 2.f * e / static_cast<float>(N);
      if (lane == 0)
      {
        gb3 += dyi;
        loss += static_cast<double>(e) * e;
      }
      // gW3 += H2^T dy; dZ2 = (dy W3^T) masked by Z2 > 0.
      const uint32_t dw = mlp_pack(dyi);
#pragma unroll
      for (int c = 0; c < 4; ++c)
      {
        const int j = lane + 32 * c;
        const bool in = live && j < H;
        z1[r][c] = in ? Z1[i * H + j] : 0.f;
        const float z2 = in ? Z2[i * H + j] : 0.f;
        s.H1[(4 * w + r) * kMlpLdH + j] = mlp_pack(fmaxf(z1[r][c], 0.f));
        gw3[c] = mlp_fma(mlp_pack(fmaxf(z2, 0.f)), dw, gw3[c]);
        const float d = z2 <= 0.f ? 0.f : mlp_fma(dw, s.W3[j], 0.f);
        gb2[c] += d;
        s.D2[(4 * w + r) * kMlpLdH + j] = mlp_pack(d);
      }
    }
    __syncwarp();  // up to the barrier below a warp reads only its own rows
    // dZ1 = (dZ2 W2^T) masked by Z1 > 0.
    float d1[4][4];
    mlp_gemm(s.D2, s.W2, w, lane, d1);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c)
      {
        const float d = z1[r][c] <= 0.f ? 0.f : d1[r][c];
        gb1[c] += d;
        s.D1[(4 * w + r) * kMlpLdH + lane + 32 * c] = mlp_pack(d);
      }
    __syncthreads();
    // gW2 += H1^T dZ2, gW1 += x^T dZ1 (rows past N hold zeros).
#pragma unroll 1
    for (int i = 0; i < kMlpRows; ++i)
    {
      uint32_t a[8], b[8];
#pragma unroll
      for (int q = 0; q < 8; ++q)
      {
        a[q] = s.H1[i * kMlpLdH + ty + 16 * q];
        b[q] = s.D2[i * kMlpLdH + tx + 16 * q];
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
#pragma unroll
        for (int v = 0; v < 8; ++v)
          g2[q][v] = mlp_fma(a[q], b[v], g2[q][v]);
      const uint32_t d = s.D1[i * kMlpLdH + jc];
#pragma unroll
      for (int q = 0; q < kMlpF / 2; ++q)
        if (half + 2 * q < F)
          g1[q] = mlp_fma(s.x[i * kMlpF + half + 2 * q], d, g1[q]);
    }
  }
  float* g = part + static_cast<int64_t>(blockIdx.x) * nparams;
  float* gW2 = g + F * H + H;
  float* gB2 = gW2 + H * H;
#pragma unroll
  for (int q = 0; q < kMlpF / 2; ++q)
    if (half + 2 * q < F && jc < H)
      g[(half + 2 * q) * H + jc] = g1[q];
#pragma unroll
  for (int a = 0; a < 8; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b)
      if (ty + 16 * a < H && tx + 16 * b < H)
        gW2[(ty + 16 * a) * H + tx + 16 * b] = g2[a][b];
#pragma unroll
  for (int c = 0; c < 4; ++c)
  {
    s.colsum[0][w][lane + 32 * c] = gb1[c];
    s.colsum[1][w][lane + 32 * c] = gb2[c];
    s.colsum[2][w][lane + 32 * c] = gw3[c];
  }
  if (lane == 0)
  {
    s.gb3[w] = gb3;
    s.loss[w] = loss;
  }
  __syncthreads();
  for (int e = tid; e < 3 * kMlpW; e += kMlpThreads)
  {
    const int which = e / kMlpW, j = e % kMlpW;
    float v = 0.f;
#pragma unroll
    for (int q = 0; q < kMlpThreads / 32; ++q)
      v += s.colsum[which][q][j];
    if (j < H)
      (which == 0 ? g + F * H : (which == 1 ? gB2 : gB2 + H))[j] = v;
  }
  if (tid == 0)
  {
    float v = 0.f;
    double l = 0.0;
    for (int q = 0; q < kMlpThreads / 32; ++q)
    {
      v += s.gb3[q];
      l += s.loss[q];
    }
    gB2[2 * H] = v;
    loss_part[blockIdx.x] = l;
  }
}

// grads[j] = sum over the CTAs' partials, in a fixed order: four ranges of
// CTAs per parameter, added in turn; *loss = mean squared error.
__global__ void __launch_bounds__(256)
  mlp_reduce_kernel(const float* __restrict__ part, const double* __restrict__ loss_part, int ctas,
                    int nparams, int N, float* __restrict__ grads, double* __restrict__ loss)
{
  __shared__ float acc[4][64];
  const int q = threadIdx.x >> 6, j = blockIdx.x * 64 + (threadIdx.x & 63);
  const int per = (ctas + 3) / 4;
  const int c1 = (q + 1) * per < ctas ? (q + 1) * per : ctas;
  float v = 0.f;
  if (j < nparams)
#pragma unroll 8
    for (int c = q * per; c < c1; ++c)
      v += part[static_cast<int64_t>(c) * nparams + j];
  acc[q][threadIdx.x & 63] = v;
  __syncthreads();
  if (q == 0 && j < nparams)
    grads[j] = (acc[0][threadIdx.x] + acc[1][threadIdx.x]) + (acc[2][threadIdx.x] + acc[3][threadIdx.x]);
  if (blockIdx.x == 0 && threadIdx.x < 32)
  {
    double l = 0.0;
    for (int c = threadIdx.x; c < ctas; c += 32)
      l += loss_part[c];
    for (int o = 16; o > 0; o >>= 1)
      l += __shfl_xor_sync(0xffffffffu, l, o);
    if (threadIdx.x == 0)
      *loss = l / N;
  }
}

}  // namespace
}  // namespace ttg
