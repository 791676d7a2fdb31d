// Learned first-bead insertion proposal: a Fourier-feature MLP trained on grid Boltzmann factors, tabulated into an
// exactly normalised, exactly samplable density.
//
// There is no counterpart in RASPA3; the proposal replaces the uniform first-bead positions of
// CBMC::growMoleculeMultipleFirstBeadSwapInsertion (src/raspakit/cbmc/multiple_first_bead.cpp:23-27) and the k-1 new
// positions of retraceMultipleFirstBeadSwapDeletion (:56-61). With trial positions drawn from a density q (per unit
// volume, relative to uniform), the Rosenbluth weight of trial i becomes exp(-beta U_i) / q(r_i); W = sum / k is then
// used in the unchanged insertion / deletion acceptance rules, which keeps detailed balance (biased-CBMC identity).
//
// Network: features phi(s) = {sin, cos}(2 pi n s_a), n = 1..16, a = x, y, z (96 inputs) of the fractional position in
// the framework unit cell; two hidden layers of 64 with SiLU; one output f(s), an unnormalised log-density. Training
// minimises (1/B) sum (f(s_i) - t_i)^2 with Adam, where t_i = max(-beta U(s_i), t_min) and U is the first bead's
// framework energy from the tricubic grids (VDW grid + q times the unit-charge Ewald grid) at uniform random s_i.
//
// Kernels (all FP32, hand-written, no tensor cores: their 32-bit accuracy is kept): a CTA takes a tile of 32 samples,
// keeps the weights and the tile's activations in shared memory and gives each thread a register tile of every layer
// product (2 samples x 4 units forward and back, 4 x 4 and 4 x 6 weights in the gradients) fed by 16-byte reads; z1, z2
// and h2 never leave the registers. Each CTA writes its gradient partial, and one more kernel sums the partials in a
// fixed order, eight threads per parameter, and
// applies Adam. Tabulation: f at the centres of G^3 cells of the unit cell; cell probabilities p_c ~ exp(f_c), mixed
// with a uniform density: q(s) = (1 - eps) G^3 p_c(s) + eps. Sampling: with probability eps a uniform position,
// else a cell by binary search of the cumulative p_c and a uniform position inside it.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "energy.cuh"

namespace
{
constexpr int kIn = 96, kH = 64;
constexpr int kParams = kH * kIn + kH + kH * kH + kH + kH + 1;  // 10433
constexpr int kOffW1 = 0, kOffB1 = kH * kIn, kOffW2 = kOffB1 + kH, kOffB2 = kOffW2 + kH * kH, kOffW3 = kOffB2 + kH,
              kOffB3 = kOffW3 + kH;
constexpr int kTile = 32;  // samples per CTA: a batch of 4,096 spreads over 128 CTAs (one per SM)
constexpr int kThreads = 256;
// Leading dimensions of the shared arrays: rows 16-byte aligned and 4 banks apart, so that the 16-byte reads of
// neighbouring rows by neighbouring lanes meet no bank conflict
constexpr int kLdIn = kIn + 4, kLdH = kH + 4;

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z)
{
  const float sg = 1.0f / (1.0f + __expf(-z));
  return sg * (1.0f + z * (1.0f - sg));
}

// FP32 numbers as integers of the same order, and back
__device__ __forceinline__ int orderedInt(float x)
{
  const int i = __float_as_int(x);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float floatOf(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

struct MlpWeights
{
  float W1[kH * kLdIn];  // [unit][input]
  float W2[kH * kLdH];   // [unit][unit of layer 1]
  float b1[kH], b2[kH], w3[kH];
  float b3, pad[3];
};
struct MlpForwardShared
{
  MlpWeights w;
  float phi[kTile * kLdIn];
  float h1[kTile * kLdH];
  float h2[kTile * kLdH];
  float f[kTile];
};
struct MlpGradShared
{
  MlpForwardShared f;
  float W2T[kH * kLdH];   // [unit of layer 1][unit]
  float dz2[kTile * kLdH];
  float dz1[kTile * kLdH];
  float df[kTile];
};

__device__ __forceinline__ float dot4(float4 a, float4 b, float acc)
{
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

__device__ void loadWeights(MlpWeights& S, const float* theta)
{
  const float4* w1 = reinterpret_cast<const float4*>(theta + kOffW1);
  for (int q = threadIdx.x; q < kH * kIn / 4; q += kThreads)
    *reinterpret_cast<float4*>(&S.W1[(q / (kIn / 4)) * kLdIn + 4 * (q % (kIn / 4))]) = w1[q];
  const float4* w2 = reinterpret_cast<const float4*>(theta + kOffW2);
  for (int q = threadIdx.x; q < kH * kH / 4; q += kThreads)
    *reinterpret_cast<float4*>(&S.W2[(q / (kH / 4)) * kLdH + 4 * (q % (kH / 4))]) = w2[q];
  if (threadIdx.x < kH)
  {
    S.b1[threadIdx.x] = theta[kOffB1 + threadIdx.x];
    S.b2[threadIdx.x] = theta[kOffB2 + threadIdx.x];
    S.w3[threadIdx.x] = theta[kOffW3 + threadIdx.x];
  }
  if (threadIdx.x == 0) S.b3 = theta[kOffB3];
}

// sin and cos of the 16 harmonics of each fractional coordinate of the tile's samples; position(i, a) is coordinate a
template <typename Position>
__device__ __forceinline__ void features(float* phi, int count, Position position)
{
  for (int q = threadIdx.x; q < kTile * 48; q += kThreads)
  {
    const int i = q / 48, r = q % 48, a = r / 16, n = r % 16 + 1;
    float sn = 0.0f, cs = 0.0f;
    if (i < count) sincospif(2.0f * static_cast<float>(n) * position(i, a), &sn, &cs);
    *reinterpret_cast<float2*>(&phi[i * kLdIn + 32 * a + 2 * (n - 1)]) = make_float2(sn, cs);
  }
}

// The 2 x 4 tile of x W^T of this thread: samples ig and ig + 16, units jq + 16 u, K inputs
template <int K, int LDX, int LDW>
__device__ __forceinline__ void tileProduct(const float* x, const float* W, int ig, int jq, float (&acc)[2][4])
{
#pragma unroll 4
  for (int k = 0; k < K; k += 4)
  {
    const float4 x0 = *reinterpret_cast<const float4*>(&x[ig * LDX + k]);
    const float4 x1 = *reinterpret_cast<const float4*>(&x[(ig + 16) * LDX + k]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
    {
      const float4 w = *reinterpret_cast<const float4*>(&W[(jq + 16 * u) * LDW + k]);
      acc[0][u] = dot4(x0, w, acc[0][u]);
      acc[1][u] = dot4(x1, w, acc[1][u]);
    }
  }
}

// Both hidden layers and the output of the tile's samples: z1 and z2 of this thread's units, h1, h2 and f in shared
// memory. Every sum runs over its inputs in order (f in one chain per sample, by the first warp): the trained weights,
// and the density tabulated from them, then do not depend on how the products are tiled.
__device__ __forceinline__ void forward(MlpForwardShared& S, int ig, int jq, float (&z1)[2][4], float (&z2)[2][4])
{
#pragma unroll
  for (int u = 0; u < 4; ++u) z1[0][u] = z1[1][u] = S.w.b1[jq + 16 * u];
  tileProduct<kIn, kLdIn, kLdIn>(S.phi, S.w.W1, ig, jq, z1);
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int u = 0; u < 4; ++u) S.h1[(ig + 16 * s) * kLdH + jq + 16 * u] = silu(z1[s][u]);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u) z2[0][u] = z2[1][u] = S.w.b2[jq + 16 * u];
  tileProduct<kH, kLdH, kLdH>(S.h1, S.w.W2, ig, jq, z2);
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int u = 0; u < 4; ++u) S.h2[(ig + 16 * s) * kLdH + jq + 16 * u] = silu(z2[s][u]);
  __syncthreads();
  if (threadIdx.x < kTile)
  {
    float acc = S.w.b3;
#pragma unroll
    for (int k = 0; k < kH; k += 4)
      acc = dot4(*reinterpret_cast<const float4*>(&S.h2[threadIdx.x * kLdH + k]),
                 *reinterpret_cast<const float4*>(&S.w.w3[k]), acc);
    S.f[threadIdx.x] = acc;
  }
}

// The bound is FP32 arithmetic on operands from shared memory: with one output per thread each FMA took two loads; in
// 2 x 4 and 4 x 4 register tiles it takes 0.4. A step on 4,096 samples: 45.6 us before, 23.6 now, and the reduction with
// the Adam step below 10.6 and 7.0 (each alone); one after the other 100 steps took 5.0 ms before, 2.6 ms so, and 2.05 ms
// with each kernel's start overlapping the end of the one before.
// One tile's loss and gradient partial; batch size B scales the loss. Samples: tile0 + i in order, or (random) drawn
// from the n_samples by splitmix64 of (seed, step, slot).
// What the kernel before writes while this one may have started (theta here, the partials in the reduction) is not declared
// __restrict__: a load through a read-only pointer may take a path that takes the data for constant while the kernel runs,
// or be moved ahead of the wait.
__global__ void __launch_bounds__(kThreads) mlpGradKernel(const float* theta, const float* __restrict__ s,
                                                          const float* __restrict__ target, int64_t n_samples,
                                                          bool random, int batch, unsigned long long seed,
                                                          long long step, float* partial, float* lossPartial)
{
  extern __shared__ __align__(16) unsigned char smraw[];
  MlpGradShared& S = *reinterpret_cast<MlpGradShared*>(smraw);
  MlpForwardShared& F = S.f;
  __shared__ int idx[kTile];
  const int tid = threadIdx.x, ig = tid / 16, jq = tid % 16;
  const int tile0 = blockIdx.x * kTile;
  const int count = min(kTile, batch - tile0);
  if (tid < kTile)
  {
    int64_t k = tid < count ? tile0 + tid : 0;
    if (random && tid < count)
    {
      unsigned long long z = seed + 0x9E3779B97F4A7C15ULL * static_cast<unsigned long long>(step * batch + tile0 + tid + 1);
      z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
      z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
      z ^= z >> 31;
      k = static_cast<int64_t>(z % static_cast<unsigned long long>(n_samples));
    }
    idx[tid] = static_cast<int>(k);
  }
  __syncthreads();
  // the samples do not depend on the step before, whose reduction this kernel's start overlaps (launchGrad)
  cudaTriggerProgrammaticLaunchCompletion();
  const float goal = tid < count ? target[idx[tid]] : 0.0f;
  features(F.phi, count, [&](int i, int a) { return s[3 * idx[i] + a]; });
  cudaGridDependencySynchronize();
  loadWeights(F.w, theta);
  __syncthreads();
  for (int q = tid; q < kH * kH; q += kThreads) S.W2T[(q % kH) * kLdH + q / kH] = F.w.W2[(q / kH) * kLdH + q % kH];
  __syncthreads();
  float z1[2][4], z2[2][4];
  forward(F, ig, jq, z1, z2);
  // dL/df = 2 (f - t) / B; dz2 = df w3 silu'(z2)
  if (tid < kTile)
  {
    float d = 0.0f, lp = 0.0f;
    if (tid < count)
    {
      const float r = F.f[tid] - goal;
      d = 2.0f * r / static_cast<float>(batch);
      lp = r * r;
    }
    S.df[tid] = d;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lp += __shfl_down_sync(0xffffffffu, lp, o);
    if (tid == 0) lossPartial[blockIdx.x] = lp;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 2; ++q)
  {
    const int i = ig + 16 * q;
    const float d = S.df[i];
#pragma unroll
    for (int u = 0; u < 4; ++u)
    {
      const int j = jq + 16 * u;
      S.dz2[i * kLdH + j] = d * F.w.w3[j] * dsilu(z2[q][u]);
    }
  }
  __syncthreads();
  float* g = partial + static_cast<long long>(blockIdx.x) * kParams;
  // dz1 = (dz2 W2) silu'(z1)
  float d1[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
  tileProduct<kH, kLdH, kLdH>(S.dz2, S.W2T, ig, jq, d1);
#pragma unroll
  for (int q = 0; q < 2; ++q)
#pragma unroll
    for (int u = 0; u < 4; ++u) S.dz1[(ig + 16 * q) * kLdH + jq + 16 * u] = d1[q][u] * dsilu(z1[q][u]);
  // W2 gradient dz2^T h1: units 4 ig + u by inputs 4 jq + v
  {
    float acc[4][4] = {};
#pragma unroll 8
    for (int i = 0; i < kTile; ++i)
    {
      const float4 a = *reinterpret_cast<const float4*>(&S.dz2[i * kLdH + 4 * ig]);
      const float4 b = *reinterpret_cast<const float4*>(&F.h1[i * kLdH + 4 * jq]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) g[kOffW2 + (4 * ig + u) * kH + 4 * jq + v] = acc[u][v];
  }
  __syncthreads();
  // W1 gradient dz1^T phi: units 4 ig + u by inputs 4 jq + v (v < 4) and 64 + 2 jq + v - 4
  {
    float acc[4][6] = {};
#pragma unroll 4
    for (int i = 0; i < kTile; ++i)
    {
      const float4 a = *reinterpret_cast<const float4*>(&S.dz1[i * kLdH + 4 * ig]);
      const float4 b = *reinterpret_cast<const float4*>(&F.phi[i * kLdIn + 4 * jq]);
      const float2 c = *reinterpret_cast<const float2*>(&F.phi[i * kLdIn + 64 + 2 * jq]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[6] = {b.x, b.y, b.z, b.w, c.x, c.y};
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 6; ++v) acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 6; ++v)
        g[kOffW1 + (4 * ig + u) * kIn + (v < 4 ? 4 * jq + v : 64 + 2 * jq + v - 4)] = acc[u][v];
  }
  // the column sums: b1, b2 and w3 by one thread each, b3 by one more
  if (tid < 2 * kH)
  {
    const float* x = tid < kH ? S.dz1 : S.dz2;
    const int j = tid % kH;
    float acc = 0.0f;
#pragma unroll 8
    for (int i = 0; i < kTile; ++i) acc += x[i * kLdH + j];
    g[(tid < kH ? kOffB1 : kOffB2) + j] = acc;
  }
  else if (tid < 3 * kH)
  {
    const int j = tid % kH;
    float acc = 0.0f;
#pragma unroll 8
    for (int i = 0; i < kTile; ++i) acc = fmaf(S.df[i], F.h2[i * kLdH + j], acc);
    g[kOffW3 + j] = acc;
  }
  else if (tid == 3 * kH)
  {
    float acc = 0.0f;
    for (int i = 0; i < kTile; ++i) acc += S.df[i];
    g[kOffB3] = acc;
  }
}

// Sum of the tile partials in tile order; with lr > 0 also an Adam step (Kingma & Ba 2015). kReduceLanes threads per
// parameter bring the partials of kReduceTiles tiles into shared memory, all their loads in flight together; one thread
// adds them in order (one thread that also loaded them waited for one load after another).
constexpr int kReduceLanes = 8, kReduceTiles = 128;
__global__ void __launch_bounds__(kThreads) reduceAdamKernel(float* theta, float* m, float* v, const float* partial,
                                                             int n_tiles, float lr, float b1, float b2, float eps,
                                                             long long t, float* grad_out, const float* lossPartial,
                                                             float* loss_out, int batch)
{
  constexpr int kItems = kThreads / kReduceLanes;
  __shared__ float tiles[kReduceTiles][kItems];
  const int item = threadIdx.x % kItems, part = threadIdx.x / kItems;
  const int p = blockIdx.x * kItems + item;  // the last one past the parameters: the loss
  const float* from = p < kParams ? partial + p : lossPartial;
  const long long stride = p < kParams ? kParams : 1;
  float c1 = 1.0f, c2 = 1.0f, gsum = 0.0f;
  if (part == 0 && lr > 0.0f)
  {
    c1 = 1.0f - powf(b1, static_cast<float>(t));
    c2 = 1.0f - powf(b2, static_cast<float>(t));
  }
  cudaTriggerProgrammaticLaunchCompletion();
  cudaGridDependencySynchronize();
  for (int base = 0; base < n_tiles; base += kReduceTiles)
  {
    const int n = min(kReduceTiles, n_tiles - base);
    if (base > 0) __syncthreads();
    if (p <= kParams)
#pragma unroll
      for (int q = 0; q < kReduceTiles / kReduceLanes; ++q)
      {
        const int b = q * kReduceLanes + part;
        if (b < n) tiles[b][item] = from[(base + b) * stride];
      }
    __syncthreads();
    if (part == 0)
    {
#pragma unroll 16
      for (int b = 0; b < n; ++b) gsum += tiles[b][item];
    }
  }
  if (part != 0 || p > kParams) return;
  if (p == kParams)
  {
    if (loss_out) *loss_out = gsum / static_cast<float>(batch);
    return;
  }
  if (grad_out) grad_out[p] = gsum;
  if (lr > 0.0f)
  {
    const float mm = b1 * m[p] + (1.0f - b1) * gsum;
    const float vv = b2 * v[p] + (1.0f - b2) * gsum * gsum;
    m[p] = mm;
    v[p] = vv;
    const float mh = mm / c1;
    const float vh = vv / c2;
    theta[p] -= lr * mh / (sqrtf(vh) + eps);
  }
}
constexpr int kReduceBlocks = (kParams + 1 + kThreads / kReduceLanes - 1) / (kThreads / kReduceLanes);

// 48^3 positions took 313 us with one output per thread and the weights loaded by every tile, now 119.
// f at n positions: s[3 * n], or (s null) the centres of cells_per_axis^3 cells. A CTA loads the weights once and takes
// every gridDim.x-th tile. If `largest` is given it receives the largest f as an ordered integer.
__global__ void __launch_bounds__(kThreads) mlpForwardKernel(const float* __restrict__ theta,
                                                             const float* __restrict__ s, int cells_per_axis, int64_t n,
                                                             float* __restrict__ out, int* __restrict__ largest)
{
  extern __shared__ __align__(16) unsigned char smraw[];
  MlpForwardShared& S = *reinterpret_cast<MlpForwardShared*>(smraw);
  const int ig = threadIdx.x / 16, jq = threadIdx.x % 16;
  loadWeights(S.w, theta);
  const long long tiles = (n + kTile - 1) / kTile;
  int best = INT_MIN;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x)
  {
    const long long tile0 = tile * kTile;
    const int count = static_cast<int>(min(static_cast<long long>(kTile), n - tile0));
    __syncthreads();
    features(S.phi, count, [&](int i, int a) -> float {
      if (s) return s[3 * (tile0 + i) + a];
      long long c = tile0 + i;
      const int G = cells_per_axis;
      if (a > 0) c /= G;
      if (a > 1) c /= G;
      return static_cast<float>((static_cast<double>(c % G) + 0.5) / G);
    });
    __syncthreads();
    float z1[2][4], z2[2][4];
    forward(S, ig, jq, z1, z2);
    if (threadIdx.x < count)
    {
      out[tile0 + threadIdx.x] = S.f[threadIdx.x];
      best = max(best, orderedInt(S.f[threadIdx.x]));
    }
  }
  if (largest)
  {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0) atomicMax(largest, best);
  }
}

// Cell probabilities of the tabulated proposal. Per block of kThreads cells: w_c = exp(f_c - max f) in FP64 into
// `density`, its running sums within the block into `cdf`, and the block's sum.
__global__ void __launch_bounds__(kThreads) cellWeightsKernel(const float* __restrict__ f, int64_t nc,
                                                              const int* __restrict__ largest,
                                                              double* __restrict__ density, double* __restrict__ cdf,
                                                              double* __restrict__ sums)
{
  __shared__ double warp_sum[kThreads / 32];
  const int64_t c = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double w = c < nc ? exp(static_cast<double>(f[c]) - static_cast<double>(floatOf(*largest))) : 0.0;
  double run = w;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    const double x = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += x;
  }
  if (lane == 31) warp_sum[warp] = run;
  __syncthreads();
  double before = 0.0;
  for (int q = 0; q < warp; ++q) before += warp_sum[q];
  run += before;
  if (c < nc)
  {
    density[c] = w;
    cdf[c] = run;
  }
  if (threadIdx.x == kThreads - 1) sums[blockIdx.x] = run;
}

// Exclusive prefix sums of the n block sums in place, by one block; sums[n] receives the total
__global__ void __launch_bounds__(1024) cellOffsetsKernel(double* sums, int n)
{
  __shared__ double warp_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double before = 0.0;
  for (int base = 0; base < n; base += 1024)
  {
    const int k = base + threadIdx.x;
    const double x = k < n ? sums[k] : 0.0;
    double run = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      const double y = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += y;
    }
    if (lane == 31) warp_sum[warp] = run;
    __syncthreads();
    double ahead = before;
    for (int q = 0; q < 32; ++q)
    {
      if (q < warp) ahead += warp_sum[q];
      before += warp_sum[q];
    }
    if (k < n) sums[k] = ahead + run - x;
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[n] = before;
}

// p_c = w_c / total: the cumulative probabilities and q_c = (1 - eps) nc p_c + eps
__global__ void __launch_bounds__(kThreads) cellTableKernel(int64_t nc, double eps, const double* __restrict__ sums,
                                                            int blocks, double* density, double* cdf)
{
  const int64_t c = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  if (c >= nc) return;
  const double total = sums[blocks];
  density[c] = (1.0 - eps) * static_cast<double>(nc) * (density[c] / total) + eps;
  cdf[c] = c == nc - 1 ? 1.0 : (sums[blockIdx.x] + cdf[c]) / total;
}

// Grid-sampled Boltzmann targets of one bead: s uniform in the unit cell, t = max(-beta U(s), t_min) with
// U = VDW grid + q * unit-charge Ewald grid (the grid branch of cbmc/interactions_framework_molecule.cpp:57-69).
__global__ void sampleTargetsKernel(rgd::Grid vdw, const double* ewald_grid, int quintic, double charge, double beta,
                                    double t_min, double c00, double c01, double c02, double c10, double c11, double c12,
                                    double c20, double c21, double c22, int64_t n, unsigned long long seed,
                                    float* s_out, float* t_out)
{
  const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double u[3];
  for (int a = 0; a < 3; ++a)
  {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ULL * static_cast<unsigned long long>(3 * i + a + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    u[a] = static_cast<double>(z >> 11) * 0x1.0p-53;
  }
  // position = cell * s (columns of the cell are the lattice vectors)
  const double x = c00 * u[0] + c10 * u[1] + c20 * u[2];
  const double y = c01 * u[0] + c11 * u[1] + c21 * u[2];
  const double z = c02 * u[0] + c12 * u[1] + c22 * u[2];
  // the scheme of the system's grids: tricubic (8 values per point) or triquintic (27)
  double e = quintic ? rgd::interpolateQuintic(vdw, x, y, z, nullptr) : rgd::interpolate(vdw, x, y, z);
  if (ewald_grid)
  {
    rgd::Grid ge = vdw;
    ge.data = ewald_grid;
    e += charge * (quintic ? rgd::interpolateQuintic(ge, x, y, z, nullptr) : rgd::interpolate(ge, x, y, z));
  }
  const double t = fmax(-beta * e, t_min);
  s_out[3 * i] = static_cast<float>(u[0]);
  s_out[3 * i + 1] = static_cast<float>(u[1]);
  s_out[3 * i + 2] = static_cast<float>(u[2]);
  t_out[i] = static_cast<float>(t);
}
}  // namespace

struct rg_mlp
{
  rg_ctx* ctx = nullptr;
  float* theta = nullptr;
  float* m = nullptr;
  float* v = nullptr;
  // the tiles' partials of the last launch, set anew by each (ensurePartial): the context's scratch, or `own`
  float* partial = nullptr;
  float* lossPartial = nullptr;
  float* own = nullptr;
  int own_tiles = 0;
  float* scalars = nullptr;  // [0] loss
  float* grad = nullptr;     // gradient of rg_mlp_loss_and_gradient
  long long t = 0;           // Adam step count
};

struct rg_proposal
{
  rg_ctx* ctx = nullptr;
  int G = 0;
  double eps = 0.0;
  rg_ctx::Slot table;         // device memory of both arrays
  double* cdf = nullptr;      // inclusive cumulative cell probabilities, G^3
  double* density = nullptr;  // q per cell relative to uniform: (1 - eps) G^3 p_c + eps
  std::vector<double> host_density;
};

namespace rgd
{
rg_status proposalExport(rg_proposal* p, const double** cdf, const double** density, int* G, double* eps)
{
  if (!p) return RG_ERR_INVALID_ARGUMENT;
  *cdf = p->cdf;
  *density = p->density;
  *G = p->G;
  *eps = p->eps;
  return RG_OK;
}
}  // namespace rgd

namespace
{
// Room for the partials of `tiles` tiles. Up to kSharedTiles (43 MB) they lie in scratch that all networks of the context
// share (their kernels are ordered by its stream): a buffer of each network's own cost its first training 0.5 ms, now and
// then 7. More than that a context would keep for good, so the network has its own.
constexpr int kSharedTiles = 1024;
rg_status ensurePartial(rg_mlp* m, int tiles)
{
  rg_ctx* ctx = m->ctx;
  const size_t bytes = sizeof(float) * (kParams + 1) * static_cast<size_t>(tiles);
  void* room = m->own;
  if (tiles <= kSharedTiles)
  {
    if (rg_status st = rg::scratch(ctx, 11, bytes, &room)) return st;
  }
  else if (m->own_tiles < tiles)
  {
    RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    cudaFree(m->own);
    m->own = nullptr;
    m->own_tiles = 0;
    RG_CUDA(ctx, cudaMalloc(reinterpret_cast<void**>(&m->own), bytes));
    m->own_tiles = tiles;
    room = m->own;
  }
  m->partial = static_cast<float*>(room);
  m->lossPartial = m->partial + static_cast<size_t>(kParams) * tiles;
  return RG_OK;
}

// Launches a training kernel; with `overlap` it may start while the kernel before it in the stream ends, and waits for
// that one's results where it says so (cudaGridDependencySynchronize). Everything it reads before has to be older: the
// first kernel of a training run is launched without, since its samples may come from the kernel before.
template <typename... Params, typename... Args>
cudaError_t launchOverlapping(void (*kernel)(Params...), int blocks, size_t shared, cudaStream_t stream, bool overlap,
                              Args... args)
{
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = shared;
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

rg_status launchGrad(rg_mlp* m, const float* s, const float* t, int64_t n, bool random, int batch,
                     unsigned long long seed, long long step, bool overlap)
{
  rg_ctx* ctx = m->ctx;
  const int tiles = (batch + kTile - 1) / kTile;
  rg_status st = ensurePartial(m, tiles);
  if (st) return st;
  constexpr int sh = static_cast<int>(sizeof(MlpGradShared));
  RG_CUDA(ctx, cudaFuncSetAttribute(mlpGradKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sh));
  RG_CUDA(ctx, launchOverlapping(mlpGradKernel, tiles, sh, ctx->stream, overlap, m->theta, s, t, n, random, batch, seed,
                                 step, m->partial, m->lossPartial));
  return RG_OK;
}
// Forward pass on n positions (s null: the centres of cells^3 cells), at most three CTAs per SM
rg_status launchForward(rg_mlp* m, const float* s, int cells, int64_t n, float* out, int* largest)
{
  rg_ctx* ctx = m->ctx;
  constexpr int sh = static_cast<int>(sizeof(MlpForwardShared));
  RG_CUDA(ctx, cudaFuncSetAttribute(mlpForwardKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sh));
  int sms = 148;
  RG_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  const int64_t tiles = (n + kTile - 1) / kTile;
  const unsigned blocks = static_cast<unsigned>(std::min<int64_t>(tiles, 3 * sms));
  mlpForwardKernel<<<blocks, kThreads, sh, ctx->stream>>>(m->theta, s, cells, n, out, largest);
  RG_CUDA(ctx, cudaGetLastError());
  return RG_OK;
}
}  // namespace

extern "C"
{
rg_status rg_mlp_create(rg_ctx* ctx, uint64_t seed, rg_mlp** out)
{
  if (!ctx || !out) return RG_ERR_INVALID_ARGUMENT;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  rg_mlp* m = new rg_mlp();
  m->ctx = ctx;
  // He-uniform initial weights (bound sqrt(6 / fan_in)), zero biases, from a seeded splitmix64 stream
  std::vector<float> h(kParams, 0.0f);
  unsigned long long state = seed;
  auto next = [&]()
  {
    state += 0x9E3779B97F4A7C15ULL;
    unsigned long long z = state;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    z ^= z >> 31;
    return static_cast<double>(z >> 11) * 0x1.0p-53;
  };
  const double a1 = std::sqrt(6.0 / kIn), a2 = std::sqrt(6.0 / kH);
  for (int i = 0; i < kH * kIn; ++i) h[kOffW1 + i] = static_cast<float>((2.0 * next() - 1.0) * a1);
  for (int i = 0; i < kH * kH; ++i) h[kOffW2 + i] = static_cast<float>((2.0 * next() - 1.0) * a2);
  for (int i = 0; i < kH; ++i) h[kOffW3 + i] = static_cast<float>((2.0 * next() - 1.0) * a2);
  cudaError_t err = cudaMalloc(reinterpret_cast<void**>(&m->theta), sizeof(float) * kParams);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&m->m), sizeof(float) * kParams);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&m->v), sizeof(float) * kParams);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&m->scalars), sizeof(float) * 4);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&m->grad), sizeof(float) * kParams);
  // every copy and fill on the context stream: the legacy default stream does not order with it
  if (!err) err = cudaMemcpyAsync(m->theta, h.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice, ctx->stream);
  if (!err) err = cudaMemsetAsync(m->m, 0, sizeof(float) * kParams, ctx->stream);
  if (!err) err = cudaMemsetAsync(m->v, 0, sizeof(float) * kParams, ctx->stream);
  if (!err) err = cudaMemsetAsync(m->scalars, 0, sizeof(float) * 4, ctx->stream);
  if (!err) err = cudaStreamSynchronize(ctx->stream);
  if (err)
  {
    rg_status st = rg::cudaFail(ctx, err, "rg_mlp_create");
    rg_mlp_destroy(m);
    return st;
  }
  *out = m;
  return RG_OK;
}

rg_status rg_mlp_destroy(rg_mlp* m)
{
  if (!m) return RG_OK;
  if (m->ctx) cudaStreamSynchronize(m->ctx->stream);
  cudaFree(m->theta);
  cudaFree(m->m);
  cudaFree(m->v);
  cudaFree(m->scalars);
  cudaFree(m->grad);
  cudaFree(m->own);
  delete m;
  return RG_OK;
}

int32_t rg_mlp_num_params(void) { return kParams; }

rg_status rg_mlp_get_params(rg_mlp* m, float* host, int32_t n)
{
  if (!m || !host || n != kParams) return RG_ERR_INVALID_ARGUMENT;
  RG_CUDA(m->ctx, cudaMemcpyAsync(host, m->theta, sizeof(float) * kParams, cudaMemcpyDeviceToHost, m->ctx->stream));
  RG_CUDA(m->ctx, cudaStreamSynchronize(m->ctx->stream));
  return RG_OK;
}

rg_status rg_mlp_set_params(rg_mlp* m, const float* host, int32_t n)
{
  if (!m || !host || n != kParams) return RG_ERR_INVALID_ARGUMENT;
  RG_CUDA(m->ctx, cudaMemcpyAsync(m->theta, host, sizeof(float) * kParams, cudaMemcpyHostToDevice, m->ctx->stream));
  RG_CUDA(m->ctx, cudaStreamSynchronize(m->ctx->stream));
  return RG_OK;
}

rg_status rg_mlp_loss_and_gradient(rg_mlp* m, const float* s_device, const float* target_device, int32_t n,
                                   float* loss, float* grad_host)
{
  if (!m || !s_device || !target_device || n < 1 || n > (1 << 24)) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = m->ctx;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  rg_status st = launchGrad(m, s_device, target_device, n, false, n, 0, 0, false);
  if (st) return st;
  const int tiles = (n + kTile - 1) / kTile;
  reduceAdamKernel<<<kReduceBlocks, kThreads, 0, ctx->stream>>>(m->theta, m->m, m->v, m->partial, tiles, 0.0f, 0.f, 0.f,
                                                               0.f, 1, m->grad, m->lossPartial, m->scalars, n);
  RG_CUDA(ctx, cudaGetLastError());
  if (grad_host)
    RG_CUDA(ctx, cudaMemcpyAsync(grad_host, m->grad, sizeof(float) * kParams, cudaMemcpyDeviceToHost, ctx->stream));
  if (loss) RG_CUDA(ctx, cudaMemcpyAsync(loss, m->scalars, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return RG_OK;
}

rg_status rg_mlp_train(rg_mlp* m, const float* s_device, const float* target_device, int64_t n_samples, int32_t steps,
                       int32_t batch, float learning_rate, uint64_t seed, float* final_loss)
{
  if (!m || !s_device || !target_device || n_samples < 1 || steps < 0 || batch < 1) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = m->ctx;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  const int tiles = (batch + kTile - 1) / kTile;
  for (int s = 0; s < steps; ++s)
  {
    rg_status st = launchGrad(m, s_device, target_device, n_samples, true, batch, seed, m->t, s > 0);
    if (st) return st;
    ++m->t;
    constexpr float b1 = 0.9f, b2 = 0.999f;
    RG_CUDA(ctx, launchOverlapping(reduceAdamKernel, kReduceBlocks, 0, ctx->stream, true, m->theta, m->m, m->v, m->partial,
                                   tiles, learning_rate, b1, b2, 1e-8f, m->t, nullptr, m->lossPartial, m->scalars, batch));
  }
  if (final_loss)
  {
    RG_CUDA(ctx, cudaMemcpyAsync(final_loss, m->scalars, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
  }
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return RG_OK;
}

rg_status rg_mlp_evaluate(rg_mlp* m, const float* s_device, int64_t n, float* out_device)
{
  if (!m || !s_device || !out_device || n < 0) return RG_ERR_INVALID_ARGUMENT;
  if (n == 0) return RG_OK;
  rg_ctx* ctx = m->ctx;
  return launchForward(m, s_device, 0, n, out_device, nullptr);
}

rg_status rg_proposal_sample_targets(rg_system* system, int pseudo_atom, double charge, double beta, double t_min,
                                     const rg_box* unit_cell, int64_t n, uint64_t seed, float* s_device,
                                     float* t_device)
{
  if (!system || !unit_cell || n < 1 || !s_device || !t_device) return RG_ERR_INVALID_ARGUMENT;
  rgd::FF ff;
  rgd::Box box;
  const double* grids[64];
  const double* ewald_grid;
  int n_types, gd[3];
  double gic[3][3];
  rg_ctx* ctx;
  rg_status st = rgd::systemExport(system, &ff, &box, grids, &ewald_grid, &n_types, gd, gic, &ctx);
  if (st) return st;
  if (pseudo_atom < 0 || pseudo_atom >= 64 || pseudo_atom >= n_types || !grids[pseudo_atom])
    return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_proposal_sample_targets: no grid for this pseudo-atom");
  rgd::Grid g{grids[pseudo_atom], gd[0], gd[1], gd[2], {}};
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b) g.ic[a][b] = gic[a][b];
  const double* c = unit_cell->cell;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  sampleTargetsKernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, ctx->stream>>>(
      g, ff.use_charge ? ewald_grid : nullptr, rgd::systemScheme(system) == RG_SCHEME_TRIQUINTIC ? 1 : 0, charge, beta,
      t_min, c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], c[8], n, seed, s_device, t_device);
  RG_CUDA(ctx, cudaGetLastError());
  return RG_OK;
}

// Bytes of a destroyed table that stay with the context at most (128^3 cells have 34 MB; 256^3, 268 MB, are freed)
constexpr size_t kKeptTable = 64 << 20;

rg_status rg_proposal_create(rg_mlp* m, int32_t cells_per_axis, double eps_uniform, rg_proposal** out)
{
  if (!m || !out || cells_per_axis < 1 || cells_per_axis > 256 || !(eps_uniform > 0.0) || eps_uniform > 1.0)
    return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = m->ctx;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  const int G = cells_per_axis;
  const int64_t nc = static_cast<int64_t>(G) * G * G;
  rg_proposal* p = new rg_proposal();
  p->ctx = ctx;
  p->G = G;
  p->eps = eps_uniform;
  // MLP outputs, block sums and the largest output in the context's scratch slot 6 (no allocation or free per table)
  const int blocks = static_cast<int>((nc + kThreads - 1) / kThreads);
  void* scr = nullptr;
  rg_status st = rg::scratch(ctx, 6, sizeof(double) * (static_cast<size_t>(blocks) + 2) + sizeof(float) * static_cast<size_t>(nc), &scr);
  if (st)
  {
    delete p;
    return st;
  }
  double* sums = static_cast<double*>(scr);
  int* largest = reinterpret_cast<int*>(sums + blocks + 1);
  float* f = reinterpret_cast<float*>(sums + blocks + 2);
  cudaError_t err = cudaSuccess;
  const size_t bytes = 2 * sizeof(double) * static_cast<size_t>(nc);
  // the kept table, unless it would be far too large for this one
  if (ctx->spare_table.bytes >= bytes && ctx->spare_table.bytes <= 8 * bytes + (1 << 20))
    std::swap(p->table, ctx->spare_table);
  else if (!(err = cudaMalloc(&p->table.ptr, bytes)))
    p->table.bytes = bytes;
  p->cdf = static_cast<double*>(p->table.ptr);
  p->density = p->cdf + nc;
  if (!err) err = cudaMemsetAsync(largest, 0x80, sizeof(int), ctx->stream);  // the integer of -3.39e38
  if (!err) st = launchForward(m, nullptr, G, nc, f, largest);
  if (!err && !st)
  {
    // p_c ~ exp(f_c - max f), cumulative in FP64
    cellWeightsKernel<<<blocks, kThreads, 0, ctx->stream>>>(f, nc, largest, p->density, p->cdf, sums);
    cellOffsetsKernel<<<1, 1024, 0, ctx->stream>>>(sums, blocks);
    cellTableKernel<<<blocks, kThreads, 0, ctx->stream>>>(nc, eps_uniform, sums, blocks, p->density, p->cdf);
    err = cudaGetLastError();
    p->host_density.resize(static_cast<size_t>(nc));
    if (!err)
      err = cudaMemcpyAsync(p->host_density.data(), p->density, sizeof(double) * nc, cudaMemcpyDeviceToHost, ctx->stream);
    if (!err) err = cudaStreamSynchronize(ctx->stream);
  }
  if (err || st)
  {
    if (!st) st = rg::cudaFail(ctx, err, "rg_proposal_create");
    rg_proposal_destroy(p);
    return st;
  }
  *out = p;
  return RG_OK;
}

rg_status rg_proposal_destroy(rg_proposal* p)
{
  if (!p) return RG_OK;
  if (p->ctx)
  {
    // a run that reads the table may be on any stream that the context had before: wait for all, as a free does
    cudaSetDevice(p->ctx->device);
    cudaDeviceSynchronize();
    // the larger of the two buffers stays with the context
    if (p->table.bytes <= kKeptTable && p->table.bytes > p->ctx->spare_table.bytes)
      std::swap(p->table, p->ctx->spare_table);
  }
  if (p->table.ptr) cudaFree(p->table.ptr);
  delete p;
  return RG_OK;
}

rg_status rg_proposal_density(rg_proposal* p, const double* s, int64_t n, double* q_out)
{
  if (!p || (n > 0 && (!s || !q_out))) return RG_ERR_INVALID_ARGUMENT;
  const int G = p->G;
  for (int64_t i = 0; i < n; ++i)
  {
    int64_t c[3];
    for (int a = 0; a < 3; ++a)
    {
      double f = s[3 * i + a] - std::floor(s[3 * i + a]);
      c[a] = std::min<int64_t>(G - 1, static_cast<int64_t>(f * G));
    }
    q_out[i] = p->host_density[c[0] + G * (c[1] + static_cast<int64_t>(G) * c[2])];
  }
  return RG_OK;
}
}
