// Test of a framework interpolation grid against the exact sums, on sm_100a.
//
// Replaces the grid test that System::createFrameworkInterpolationGrids (src/raspakit/system_interpolation_grids.cpp:
// 240-651, tricubic scheme) runs serially after each grid build: at random points of the simulation box it compares
// the interpolated energy and Cartesian gradient of a pseudo-atom's VDW grid with the analytical Lennard-Jones sum
// (the calculateTricubicFractionalAtPosition energy and gradient), each point weighted by exp(-beta E_vdw), and, where
// the analytical VDW energy is below the overlap criterion, the probe charge times the unit-charge Ewald grid against
// the analytical real-space Ewald sum. Energies are in K as in the reference.
//
// The points (Philox-generated, or given by the caller) are mapped into the unit cell and sorted into bins of about 32,
// so that a warp's 32 points lie together and it can leave out the images none of them sees. The framework's periodic
// images within rc of the unit cell (the set the grid build uses) are staged chunk by chunk in shared memory, those
// near a block's points only; each warp lists the ones near its own points and its lanes sum them in FP64 (with the
// reference's r^2 >= 0.1 clamp). The charged images are summed for the points below the overlap criterion only, which
// are sorted a second time. One thread per point then takes the device interpolant with its derivative, and the 36
// weighted sums are reduced per block and over the blocks in a fixed order. A point's own sums run over the images in
// image order whatever its place in the sorted list: deterministic.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "energy.cuh"
#include "fastmath.cuh"
#include "rng.cuh"

namespace rg
{
int buildGridImages(int grid_type, const rg_forcefield* ff, const HostBox& box, const rg_atom* atoms, int n,
                    int probe_type, std::vector<double4>& pos, std::vector<double4>& par);
}

namespace
{
constexpr int kThreads = 128;
constexpr int kPer = 2;     // images tested per thread and chunk
constexpr int kChunk = kThreads * kPer;
constexpr int kBinPoints = 32;      // points per bin aimed at
constexpr int kMaxBins = 1 << 16;
constexpr int kScanThreads = 1024;
constexpr int kMaxSlices = 64;      // parts of the image list per point
constexpr int64_t kMaxPoints = 1 << 21;  // points per round: bounds the scratch memory
constexpr int kSums = 36;   // 17 VDW sums, 17 charge sums, two counts (the layout of rg_grid_validation.sums)
constexpr int kHessSums = 48;  // triquintic scheme: 24 VDW and 24 charge Hessian sums (rg_grid_validation_hessian.sums)
template <int SCHEME>
constexpr int sumsOf() { return SCHEME == RG_SCHEME_TRIQUINTIC ? kSums + kHessSums : kSums; }

struct ValidateParams
{
  double uc[3][3], uic[3][3];  // unit cell and its inverse, c[col][row]
  double sc[3][3];             // simulation box
  rgd::Grid vdw, ewald;        // ewald.data null: no charge term
  const double4* vpos;         // VDW images: position, (4 eps, sigma^2, shift)
  const double4* vpar;
  const double4* epos;         // charged images: position, w = C q
  int n_vdw, n_ewald;
  int vdw_slices, ewald_slices;  // parts of the two image lists, each summed by blocks of its own
  double rc2, alpha, overlap, to_kelvin, charge, beta;
  long long n_points;          // of this round
  long long first_point;       // index of the round's first point in the Philox stream
  const double* points;        // fractions of the simulation box (3 per point), or null: Philox
  unsigned long long seed;
  int nbin[3];                 // bins along the cell vectors
  double4* where;              // [n_points] position in the unit cell, w = (bin, place within the bin) as bits
  double4* sorted;             // [n_points] position in the unit cell, w = index of the point as bits
  int* bins;                   // [bins + 1] counts, then (after the scan) where each bin starts; last: all
  double* vsum;                // [vdw_slices][n_points][kPart] sums of one part of the images: E, gradient (, Hessian)
  double* esum;                // [ewald_slices][n_points][kPart]
  double* partial;             // [blocks][sums]
  double* result;              // [sums] mapped pinned memory
};
template <int SCHEME>
constexpr int partOf() { return SCHEME == RG_SCHEME_TRIQUINTIC ? 10 : 4; }

__device__ __forceinline__ void accumulate(double* o, double w, double ei, double ef, const double* gi, const double* gf)
{
  o[0] += w;
  o[1] += ei * w;
  o[2] += ef * w;
  o[3] += (ef - ei) * (ef - ei) * w;
  o[4] += ef * ef * w;
#pragma unroll
  for (int a = 0; a < 3; ++a)
  {
    o[5 + a] += gi[a] * w;
    o[8 + a] += gf[a] * w;
    o[11 + a] += (gf[a] - gi[a]) * (gf[a] - gi[a]) * w;
    o[14 + a] += gf[a] * gf[a] * w;
  }
}

// Hessian sums of one term: interpolated, full, squared difference, squared full, for xx, xy, xz, yy, yz, zz
__device__ __forceinline__ void accumulateHessian(double* o, double w, const double* hi, const double* hf)
{
#pragma unroll
  for (int q = 0; q < 6; ++q)
  {
    o[q] += hi[q] * w;
    o[6 + q] += hf[q] * w;
    o[12 + q] += (hf[q] - hi[q]) * (hf[q] - hi[q]) * w;
    o[18 + q] += hf[q] * hf[q] * w;
  }
}

// H_ij += F2 dr_i dr_j + F1 delta_ij (xx, xy, xz, yy, yz, zz)
__device__ __forceinline__ void addHessian(double* h, double f1, double f2, double dx, double dy, double dz)
{
  h[0] += f2 * dx * dx + f1;
  h[1] += f2 * dx * dy;
  h[2] += f2 * dx * dz;
  h[3] += f2 * dy * dy + f1;
  h[4] += f2 * dy * dz;
  h[5] += f2 * dz * dz + f1;
}

// The point in the simulation box
__device__ __forceinline__ void pointOf(const ValidateParams& p, long long i, double r[3])
{
  double u[3];
  if (p.points)
  {
    u[0] = p.points[3 * i];
    u[1] = p.points[3 * i + 1];
    u[2] = p.points[3 * i + 2];
  }
  else
  {
    const double2 a = rgd::uniform2(p.seed, 11, p.first_point + i, 0), b = rgd::uniform2(p.seed, 11, p.first_point + i, 1);
    u[0] = a.x;
    u[1] = a.y;
    u[2] = b.x;
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) r[a] = p.sc[0][a] * u[0] + p.sc[1][a] * u[1] + p.sc[2][a] * u[2];
}

// Sum of a point's parts of channel c, in part order
template <int PART>
__device__ __forceinline__ double sumParts(const double* part, int slices, long long n, long long i, int c)
{
  double x = 0.0;
  for (int s = 0; s < slices; ++s) x += part[(static_cast<long long>(s) * n + i) * PART + c];
  return x;
}

// Every point's place in the unit cell, its bin and its place within the bin. The bins run along x, back along the next
// row and so on, so that consecutive ones touch. The second time (AGAIN) only the points that the charge term takes.
template <int PART, bool AGAIN>
__global__ void __launch_bounds__(kThreads) binPointsKernel(ValidateParams p)
{
  const long long i = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
  if (i >= p.n_points) return;
  int bin;
  double4 w;
  if constexpr (AGAIN)
  {
    w = p.where[i];
    bin = __double2hiint(w.w);
    const bool take = sumParts<PART>(p.vsum, p.vdw_slices, p.n_points, i, 0) * p.to_kelvin < p.overlap;
    if (!take)
    {
      p.where[i].w = __hiloint2double(bin, -1);
      return;
    }
  }
  else
  {
    double r[3], s[3];
    pointOf(p, i, r);
    int b[3];
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
      s[a] = rgd::fract1(p.uic[0][a] * r[0] + p.uic[1][a] * r[1] + p.uic[2][a] * r[2]);
      b[a] = max(0, min(p.nbin[a] - 1, static_cast<int>(s[a] * p.nbin[a])));
    }
    w.x = p.uc[0][0] * s[0] + p.uc[1][0] * s[1] + p.uc[2][0] * s[2];
    w.y = p.uc[0][1] * s[0] + p.uc[1][1] * s[1] + p.uc[2][1] * s[2];
    w.z = p.uc[0][2] * s[0] + p.uc[1][2] * s[1] + p.uc[2][2] * s[2];
    const int row = b[2] * p.nbin[1] + ((b[2] & 1) ? p.nbin[1] - 1 - b[1] : b[1]);
    bin = row * p.nbin[0] + ((row & 1) ? p.nbin[0] - 1 - b[0] : b[0]);
  }
  w.w = __hiloint2double(bin, atomicAdd(p.bins + bin, 1));
  p.where[i] = w;
}

// Exclusive prefix sums of the bins in one block; bins[n] receives the total
__global__ void __launch_bounds__(kScanThreads) scanBinsKernel(int* bins, int n)
{
  __shared__ int warp_sums[33];
  int before = 0;
  for (int base = 0; base < n; base += kScanThreads)
  {
    const int k = base + threadIdx.x;
    const int v = k < n ? bins[k] : 0;
    int total;
    const int off = blockExclusiveScan(v, warp_sums, &total);
    if (k < n) bins[k] = before + off;
    before += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) bins[n] = before;
}

__global__ void __launch_bounds__(kThreads) sortPointsKernel(ValidateParams p)
{
  const long long i = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
  if (i >= p.n_points) return;
  double4 w = p.where[i];
  const int place = __double2loint(w.w);
  if (place < 0) return;
  const int at = p.bins[__double2hiint(w.w)] + place;
  w.w = __longlong_as_double(i);
  p.sorted[at] = w;
}

// The analytical sums of one part (blockIdx.y) of the images at the sorted points. Lennard-Jones:
// potentialLennardJonesTricubicDerivative, U = B - A - shift, F1 = (6A - 12B)/r^2 with A = 4 eps t^3, B = A t^3; Ewald:
// potentialRealEwaldTricubicDerivative with q_A = 1; gradient = F1 (r - r_image), Hessian (HESS) F2 dr dr + F1 delta.
// The bound is the FP64 pipe: about 28 instructions per Lennard-Jones pair and 75 per charged one. 100,000 points of the
// 20.0 x 19.9 x 13.4 A cell: 105 and 250 us, where one thread per unsorted point tested every image of both lists in
// 3.63 ms.
template <int TYPE, bool HESS, bool CHECK>
__global__ void __launch_bounds__(kThreads) pairSumsKernel(ValidateParams p)
{
  constexpr bool EWALD = TYPE == RG_GRID_EWALD_REAL;
  constexpr int PART = HESS ? 10 : 4;
  __shared__ double4 cpos[kChunk];
  __shared__ double4 cpar[EWALD ? 1 : kChunk];
  __shared__ unsigned short wlists[kThreads / 32][kChunk];
  __shared__ int warp_sums[33];
  __shared__ double ext[kThreads / 32][6];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int count = p.bins[p.nbin[0] * p.nbin[1] * p.nbin[2]];
  const int first = blockIdx.x * kThreads;
  if (first >= count) return;
  const int at = first + tid;
  const bool active = at < count;
  const double4 me = p.sorted[active ? at : count - 1];
  // the box around the warp's points and around the block's, and the farthest point from each centre
  double lo[3] = {me.x, me.y, me.z}, hi[3] = {me.x, me.y, me.z};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
      lo[a] = fmin(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmax(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
  const double wc[3] = {0.5 * (lo[0] + hi[0]), 0.5 * (lo[1] + hi[1]), 0.5 * (lo[2] + hi[2])};
  if (lane == 0)
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
      ext[warp][a] = lo[a];
      ext[warp][3 + a] = hi[a];
    }
  __syncthreads();
  double bc[3], half = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
  {
    double l = ext[0][a], h = ext[0][3 + a];
#pragma unroll
    for (int w = 1; w < kThreads / 32; ++w)
    {
      l = fmin(l, ext[w][a]);
      h = fmax(h, ext[w][3 + a]);
    }
    bc[a] = 0.5 * (l + h);
    half += 0.25 * (h - l) * (h - l);
  }
  const double rc = sqrt(p.rc2);
  const double breach = rc + sqrt(half) + 1e-6, breach2 = breach * breach;
  double far2 = (me.x - wc[0]) * (me.x - wc[0]) + (me.y - wc[1]) * (me.y - wc[1]) + (me.z - wc[2]) * (me.z - wc[2]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) far2 = fmax(far2, __shfl_xor_sync(0xffffffffu, far2, o));
  const double reach = rc + sqrt(far2) + 1e-6, reach2 = reach * reach;

  const double4* __restrict__ ipos = EWALD ? p.epos : p.vpos;
  const int n_images = EWALD ? p.n_ewald : p.n_vdw, slices = EWALD ? p.ewald_slices : p.vdw_slices;
  const int per = (n_images + slices - 1) / slices;
  const int begin = blockIdx.y * per, end = min(n_images, begin + per);
  unsigned short* wl = wlists[warp];
  const double c1 = 2.0 * p.alpha * rg::kInvSqrtPi, two_a2 = 2.0 * p.alpha * p.alpha;
  double acc[PART];
#pragma unroll
  for (int c = 0; c < PART; ++c) acc[c] = 0.0;

  for (int base = begin; base < end; base += kChunk)
  {
    double4 ip[kPer];
    bool ok[kPer];
    int cnt = 0;
#pragma unroll
    for (int q = 0; q < kPer; ++q)
    {
      const int idx = base + tid * kPer + q;
      ok[q] = false;
      if (idx < end)
      {
        ip[q] = ipos[idx];
        const double dx = ip[q].x - bc[0], dy = ip[q].y - bc[1], dz = ip[q].z - bc[2];
        ok[q] = dx * dx + dy * dy + dz * dz < breach2;
        cnt += ok[q] ? 1 : 0;
      }
    }
    int total;
    int off = blockExclusiveScan(cnt, warp_sums, &total);
#pragma unroll
    for (int q = 0; q < kPer; ++q)
      if (ok[q])
      {
        cpos[off] = ip[q];
        if constexpr (!EWALD) cpar[off] = p.vpar[base + tid * kPer + q];
        ++off;
      }
    __syncthreads();
    int nw = 0;
    for (int b0 = 0; b0 < total; b0 += 32)
    {
      const int c = b0 + lane;
      bool in = false;
      if (c < total)
      {
        const double ex = cpos[c].x - wc[0], ey = cpos[c].y - wc[1], ez = cpos[c].z - wc[2];
        in = ex * ex + ey * ey + ez * ez < reach2;
      }
      const unsigned ballot = __ballot_sync(0xffffffffu, in);
      if (in) wl[nw + __popc(ballot & ((1u << lane) - 1u))] = static_cast<unsigned short>(c);
      nw += __popc(ballot);
    }
    __syncwarp();
    // branch-free: a lane whose pair lies outside has its charge, or its epsilon and shift, zeroed
#pragma unroll 2
    for (int w = 0; w < nw; ++w)
    {
      const int c = wl[w];
      const double4 a = cpos[c];
      const double dx = me.x - a.x, dy = me.y - a.y, dz = me.z - a.z;
      double rr = dx * dx + dy * dy + dz * dz;
      rr = rr > 0.1 ? rr : 0.1;
      const bool in = rr < p.rc2;
      double f0, f1, f2 = 0.0;
      if constexpr (EWALD)
      {
        double B[HESS ? 3 : 2];
        rgd::ewaldLadder<HESS ? 3 : 2, CHECK>(rr, p.alpha, c1, two_a2, B);
        const double cq = in ? a.w : 0.0;
        f0 = cq * B[0];
        f1 = -cq * B[1];
        if constexpr (HESS) f2 = cq * B[2];
      }
      else
      {
        const double4 q = cpar[c];
        const double inv = rgd::rcpHouseholder(rr);
        const double t = q.y * inv;
        const double t3 = t * t * t;
        const double A = (in ? q.x : 0.0) * t3;
        const double B = A * t3;
        f0 = B - A - (in ? q.z : 0.0);
        f1 = (6.0 * A - 12.0 * B) * inv;
        if constexpr (HESS) f2 = (168.0 * B - 48.0 * A) * inv * inv;  // potentialLennardJonesTriquinticDerivative
      }
      acc[0] += f0;
      acc[1] = fma(f1, dx, acc[1]);
      acc[2] = fma(f1, dy, acc[2]);
      acc[3] = fma(f1, dz, acc[3]);
      if constexpr (HESS) addHessian(acc + 4, f1, f2, dx, dy, dz);
    }
    __syncthreads();
  }
  if (!active) return;
  double2* out = reinterpret_cast<double2*>(
      (EWALD ? p.esum : p.vsum) +
      (static_cast<long long>(blockIdx.y) * p.n_points + __double_as_longlong(me.w)) * PART);
#pragma unroll
  for (int c = 0; c < PART / 2; ++c) out[c] = make_double2(acc[2 * c], acc[2 * c + 1]);
}

// One thread per point: the interpolated side and the weighted sums of both terms
template <int SCHEME>
__global__ void __launch_bounds__(kThreads) gridValidateKernel(ValidateParams p)
{
  constexpr bool Q = SCHEME == RG_SCHEME_TRIQUINTIC;
  constexpr int NS = sumsOf<SCHEME>();
  constexpr int PART = partOf<SCHEME>();
  __shared__ double red[kThreads / 32][NS];
  const long long i = static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x;
  const bool active = i < p.n_points;
  double r[3] = {0.0, 0.0, 0.0};
  if (active) pointOf(p, i, r);
  double full[PART];
#pragma unroll
  for (int c = 0; c < PART; ++c) full[c] = active ? sumParts<PART>(p.vsum, p.vdw_slices, p.n_points, i, c) : 0.0;
  double sums[NS];
#pragma unroll
  for (int c = 0; c < NS; ++c) sums[c] = 0.0;
  double evK = 0.0, w = 0.0;
  if (active)
  {
    double gi[3], gf[3], hi[6], hf[6];
    double ei;
    if constexpr (Q)
      ei = rgd::interpolateQuinticHessian(p.vdw, r[0], r[1], r[2], gi, hi) * p.to_kelvin;
    else
      ei = rgd::interpolateGradient(p.vdw, r[0], r[1], r[2], gi) * p.to_kelvin;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
      gi[a] *= p.to_kelvin;
      gf[a] = full[1 + a] * p.to_kelvin;
    }
    evK = full[0] * p.to_kelvin;
    w = exp(-p.beta * evK);
    accumulate(sums, w, ei, evK, gi, gf);
    sums[34] = 1.0;
    if constexpr (Q)
    {
#pragma unroll
      for (int q = 0; q < 6; ++q)
      {
        hi[q] *= p.to_kelvin;
        hf[q] = full[4 + q] * p.to_kelvin;
      }
      accumulateHessian(sums + kSums, w, hi, hf);
    }
  }
  // charge term: the unit-charge Ewald sum times the probe charge
  if (p.ewald.data && p.charge != 0.0 && active && evK < p.overlap)
  {
    const double sc = p.charge * p.to_kelvin;
    double ci[3], cf[3], chi[6], chf[6];
    double eci;
    if constexpr (Q)
      eci = rgd::interpolateQuinticHessian(p.ewald, r[0], r[1], r[2], ci, chi) * sc;
    else
      eci = rgd::interpolateGradient(p.ewald, r[0], r[1], r[2], ci) * sc;
#pragma unroll
    for (int c = 0; c < PART; ++c) full[c] = sumParts<PART>(p.esum, p.ewald_slices, p.n_points, i, c);
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
      ci[a] *= sc;
      cf[a] = full[1 + a] * sc;
    }
    accumulate(sums + 17, w, eci, full[0] * sc, ci, cf);
    sums[35] = 1.0;
    if constexpr (Q)
    {
#pragma unroll
      for (int q = 0; q < 6; ++q)
      {
        chi[q] *= sc;
        chf[q] = full[4 + q] * sc;
      }
      accumulateHessian(sums + kSums + 24, w, chi, chf);
    }
  }
  // fixed-order block reduction: warps by shuffles, then one thread per sum over the warps
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < NS; ++c)
  {
    double x = sums[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp][c] = x;
  }
  __syncthreads();
  if (threadIdx.x < NS)
  {
    double x = 0.0;
    for (int wi = 0; wi < kThreads / 32; ++wi) x += red[wi][threadIdx.x];
    p.partial[static_cast<long long>(blockIdx.x) * NS + threadIdx.x] = x;
  }
}

// One warp per sum: the blocks' partials by lane, then a fixed shuffle tree
template <int NS>
__global__ void __launch_bounds__(32) validateTotalKernel(const double* __restrict__ partial, long long blocks,
                                                          double* result)
{
  double x = 0.0;
#pragma unroll 8
  for (long long b = threadIdx.x; b < blocks; b += 32) x += partial[b * NS + blockIdx.x];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (threadIdx.x == 0) result[blockIdx.x] = x;
}

// Parts of an image list of n images for points that fill `blocks` blocks: enough blocks for about four of them on each
// place the GPU has (4 blocks of 128 threads per SM), so that the last round of blocks is a small share of the time,
// and at least one staging chunk of images each.
int slicesFor(long long blocks, int n, int sms)
{
  const long long want = (16LL * sms + blocks - 1) / blocks;
  const long long most = std::max(1, n / kChunk);
  return static_cast<int>(std::max(1LL, std::min({want, most, static_cast<long long>(kMaxSlices)})));
}

void fillGrid(rgd::Grid& g, const double* data, int nx, int ny, int nz, const rg::HostBox& unit)
{
  g.data = data;
  g.nx = nx;
  g.ny = ny;
  g.nz = nz;
  for (int c = 0; c < 3; ++c)
    for (int r = 0; r < 3; ++r) g.ic[c][r] = unit.ic[c][r];
}

// Boltzmann averages and relative errors of one block of 17 sums (system_interpolation_grids.cpp:652-700)
void derive(const double* s, double* e_table, double* e_full, double* e_rel, double* g_table, double* g_full,
            double* g_rel)
{
  const double nan = std::nan("");
  *e_table = s[0] > 0.0 ? s[1] / s[0] : nan;
  *e_full = s[0] > 0.0 ? s[2] / s[0] : nan;
  *e_rel = s[4] > 0.0 ? std::sqrt(s[3] / s[4]) : nan;
  for (int a = 0; a < 3; ++a)
  {
    g_table[a] = s[0] > 0.0 ? s[5 + a] / s[0] : nan;
    g_full[a] = s[0] > 0.0 ? s[8 + a] / s[0] : nan;
    g_rel[a] = s[14 + a] > 0.0 ? std::sqrt(s[11 + a] / s[14 + a]) : nan;
  }
}
// Checks, image staging, the launch and the block-ordered sum of the partials: sumsOf<SCHEME>() values in s
template <int SCHEME>
rg_status runValidate(rg_ctx* ctx, const char* name, const rg_forcefield* ff, const rg_box* unit_cell,
                      const rg_atom* unit_atoms, int n_unit_atoms, const rg_box* simulation_box, int probe_type, int nx,
                      int ny, int nz, const double* vdw_grid_device, const double* ewald_grid_device,
                      double probe_charge, double weight_beta, int64_t n_points, uint64_t seed, const double* points,
                      std::vector<double>& s)
{
  constexpr int NS = sumsOf<SCHEME>();
  s.assign(NS, 0.0);
  if (!ctx) return RG_ERR_INVALID_ARGUMENT;
  if (!ff || !unit_cell || !simulation_box || !vdw_grid_device || n_unit_atoms < 0 ||
      (n_unit_atoms > 0 && !unit_atoms) || n_points < 0)
    return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, std::string(name) + ": null or negative argument");
  if (nx < 2 || ny < 2 || nz < 2) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, std::string(name) + ": grid shape");
  if (probe_type < 0 || probe_type >= ff->n_types)
    return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, std::string(name) + ": probe_type out of range");
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  if (n_points == 0) return RG_OK;

  const rg::HostBox ub = rg::makeHostBox(unit_cell), sb = rg::makeHostBox(simulation_box);
  std::vector<double4> vpos, vpar, epos, epar;
  const int nv = rg::buildGridImages(RG_GRID_LENNARD_JONES, ff, ub, unit_atoms, n_unit_atoms, probe_type, vpos, vpar);
  const bool charge = ewald_grid_device != nullptr && probe_charge != 0.0;
  const int ne = charge ? rg::buildGridImages(RG_GRID_EWALD_REAL, ff, ub, unit_atoms, n_unit_atoms, 0, epos, epar) : 0;
  const int64_t round = std::min(n_points, kMaxPoints);
  const long long blocks = (round + kThreads - 1) / kThreads;

  int sms = 148;
  RG_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
  ValidateParams p{};
  p.vdw_slices = slicesFor(blocks, nv, sms);
  p.ewald_slices = charge ? slicesFor(blocks, ne, sms) : 0;
  // bins of about kBinPoints points, as near to cubes as the cell allows
  double width[3];
  rg::perpendicularWidths(ub, width);
  const double side = std::cbrt(width[0] * width[1] * width[2] * kBinPoints / static_cast<double>(round));
  for (int d = 0; d < 3; ++d) p.nbin[d] = static_cast<int>(std::min(64.0, std::max(1.0, std::round(width[d] / side))));
  while (p.nbin[0] * p.nbin[1] * p.nbin[2] > kMaxBins)
    for (int d = 0; d < 3; ++d) p.nbin[d] = std::max(1, p.nbin[d] / 2);
  const int nbins = p.nbin[0] * p.nbin[1] * p.nbin[2];

  // device scratch: images (slot 2), points (slot 3), the rest (slot 4): the places, the sorted points, the parts'
  // sums, the block partials and the bins; uploads staged through pinned slot 1, the totals in pinned slot 2
  constexpr int PART = partOf<SCHEME>();
  const size_t img_bytes = sizeof(double4) * static_cast<size_t>(2 * nv + ne + 1);
  const size_t pts_bytes = points ? sizeof(double) * 3 * static_cast<size_t>(n_points) : 0;
  const size_t n = static_cast<size_t>(round);
  const size_t work_doubles = 8 * n + PART * n * static_cast<size_t>(p.vdw_slices + p.ewald_slices) +
                              NS * static_cast<size_t>(blocks);
  void *dimg = nullptr, *dpts = nullptr, *dwork = nullptr, *stage = nullptr, *totals = nullptr, *dtotals = nullptr;
  rg_status st = rg::scratch(ctx, 2, img_bytes, &dimg);
  if (!st && points) st = rg::scratch(ctx, 3, pts_bytes, &dpts);
  if (!st) st = rg::scratch(ctx, 4, sizeof(double) * work_doubles + sizeof(int) * (static_cast<size_t>(nbins) + 1), &dwork);
  if (st) return st;
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // the pinned staging slots are free
  st = rg::pinnedScratch(ctx, 1, img_bytes + pts_bytes, &stage);
  if (!st) st = rg::pinnedScratch(ctx, 2, sizeof(double) * NS, &totals);
  if (st) return st;
  RG_CUDA(ctx, cudaHostGetDevicePointer(&dtotals, totals, 0));
  double4* h = static_cast<double4*>(stage);
  std::memcpy(h, vpos.data(), sizeof(double4) * nv);
  std::memcpy(h + nv, vpar.data(), sizeof(double4) * nv);
  if (ne) std::memcpy(h + 2 * nv, epos.data(), sizeof(double4) * ne);
  RG_CUDA(ctx, cudaMemcpyAsync(dimg, stage, img_bytes, cudaMemcpyHostToDevice, ctx->stream));
  // the points in pieces, so that one piece is on its way while the next is copied into the staging buffer
  constexpr size_t kPiece = 256 << 10;
  for (size_t o = 0; o < pts_bytes; o += kPiece)
  {
    const size_t len = std::min(kPiece, pts_bytes - o);
    char* to = reinterpret_cast<char*>(stage) + img_bytes + o;
    std::memcpy(to, reinterpret_cast<const char*>(points) + o, len);
    RG_CUDA(ctx, cudaMemcpyAsync(static_cast<char*>(dpts) + o, to, len, cudaMemcpyHostToDevice, ctx->stream));
  }

  for (int c = 0; c < 3; ++c)
    for (int r = 0; r < 3; ++r)
    {
      p.uc[c][r] = ub.c[c][r];
      p.uic[c][r] = ub.ic[c][r];
      p.sc[c][r] = sb.c[c][r];
    }
  fillGrid(p.vdw, vdw_grid_device, nx, ny, nz, ub);
  fillGrid(p.ewald, charge ? ewald_grid_device : nullptr, nx, ny, nz, ub);
  const double4* d4 = static_cast<const double4*>(dimg);
  p.vpos = d4;
  p.vpar = d4 + nv;
  p.epos = d4 + 2 * nv;
  p.n_vdw = nv;
  p.n_ewald = ne;
  p.rc2 = ff->cutoff_framework_vdw * ff->cutoff_framework_vdw;
  p.alpha = ff->ewald_alpha;
  p.overlap = ff->overlap_criteria;
  p.to_kelvin = rg::energyConversionFactor() * 6.0221419947e23 / 8.314464919;  // Units::EnergyToKelvin (units.cpp)
  p.charge = charge ? probe_charge : 0.0;
  p.beta = weight_beta;
  p.seed = seed;
  double* work = static_cast<double*>(dwork);
  p.where = reinterpret_cast<double4*>(work);
  p.sorted = p.where + n;
  p.vsum = work + 8 * n;
  p.esum = p.vsum + PART * n * static_cast<size_t>(p.vdw_slices);
  p.partial = p.esum + PART * n * static_cast<size_t>(p.ewald_slices);
  p.bins = reinterpret_cast<int*>(p.partial + NS * static_cast<size_t>(blocks));
  p.result = static_cast<double*>(dtotals);

  constexpr bool HESS = SCHEME == RG_SCHEME_TRIQUINTIC;
  const bool check = p.alpha * ff->cutoff_framework_vdw >= rgd::kErfcxMax;
  for (int64_t first = 0; first < n_points; first += round)
  {
    p.first_point = first;
    p.n_points = std::min<int64_t>(round, n_points - first);
    p.points = points ? static_cast<const double*>(dpts) + 3 * first : nullptr;
    const unsigned nb = static_cast<unsigned>((p.n_points + kThreads - 1) / kThreads);
    RG_CUDA(ctx, cudaMemsetAsync(p.bins, 0, sizeof(int) * (static_cast<size_t>(nbins) + 1), ctx->stream));
    binPointsKernel<PART, false><<<nb, kThreads, 0, ctx->stream>>>(p);
    scanBinsKernel<<<1, kScanThreads, 0, ctx->stream>>>(p.bins, nbins);
    sortPointsKernel<<<nb, kThreads, 0, ctx->stream>>>(p);
    pairSumsKernel<RG_GRID_LENNARD_JONES, HESS, false><<<dim3(nb, p.vdw_slices), kThreads, 0, ctx->stream>>>(p);
    if (charge)
    {
      RG_CUDA(ctx, cudaMemsetAsync(p.bins, 0, sizeof(int) * (static_cast<size_t>(nbins) + 1), ctx->stream));
      binPointsKernel<PART, true><<<nb, kThreads, 0, ctx->stream>>>(p);
      scanBinsKernel<<<1, kScanThreads, 0, ctx->stream>>>(p.bins, nbins);
      sortPointsKernel<<<nb, kThreads, 0, ctx->stream>>>(p);
      if (check)
        pairSumsKernel<RG_GRID_EWALD_REAL, HESS, true><<<dim3(nb, p.ewald_slices), kThreads, 0, ctx->stream>>>(p);
      else
        pairSumsKernel<RG_GRID_EWALD_REAL, HESS, false><<<dim3(nb, p.ewald_slices), kThreads, 0, ctx->stream>>>(p);
    }
    gridValidateKernel<SCHEME><<<nb, kThreads, 0, ctx->stream>>>(p);
    validateTotalKernel<NS><<<NS, 32, 0, ctx->stream>>>(p.partial, nb, p.result);
    RG_CUDA(ctx, cudaGetLastError());
    RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int c = 0; c < NS; ++c) s[c] += static_cast<const double*>(totals)[c];
  }
  return RG_OK;
}

void fillValidation(const std::vector<double>& s, rg_grid_validation* out)
{
  for (int c = 0; c < 34; ++c) out->sums[c] = s[c];
  out->n_points = static_cast<int64_t>(s[34]);
  out->n_points_charge = static_cast<int64_t>(s[35]);
  derive(s.data(), &out->energy_table, &out->energy_full, &out->energy_relative_error, out->gradient_table,
         out->gradient_full, out->gradient_relative_error);
  derive(s.data() + 17, &out->charge_energy_table, &out->charge_energy_full, &out->charge_energy_relative_error,
         out->charge_gradient_table, out->charge_gradient_full, out->charge_gradient_relative_error);
}

// Boltzmann averages and relative errors of one term's 24 Hessian sums (system_interpolation_grids.cpp:700-760)
void deriveHessian(const double* hs, double weight, double* table, double* full, double* rel)
{
  const double nan = std::nan("");
  for (int q = 0; q < 6; ++q)
  {
    table[q] = weight > 0.0 ? hs[q] / weight : nan;
    full[q] = weight > 0.0 ? hs[6 + q] / weight : nan;
    rel[q] = hs[18 + q] > 0.0 ? std::sqrt(hs[12 + q] / hs[18 + q]) : nan;
  }
}
}  // namespace

extern "C" rg_status rg_grid_validate(rg_ctx* ctx, const rg_forcefield* ff, const rg_box* unit_cell,
                                      const rg_atom* unit_atoms, int n_unit_atoms, const rg_box* simulation_box,
                                      int probe_type, int nx, int ny, int nz, const double* vdw_grid_device,
                                      const double* ewald_grid_device, double probe_charge, double weight_beta,
                                      int64_t n_points, uint64_t seed, const double* points, rg_grid_validation* out)
{
  if (ctx && !out) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_grid_validate: null or negative argument");
  std::vector<double> s;
  rg_status st = runValidate<RG_SCHEME_TRICUBIC>(ctx, "rg_grid_validate", ff, unit_cell, unit_atoms, n_unit_atoms,
                                                 simulation_box, probe_type, nx, ny, nz, vdw_grid_device,
                                                 ewald_grid_device, probe_charge, weight_beta, n_points, seed, points,
                                                 s);
  if (st) return st;
  std::memset(out, 0, sizeof(*out));
  if (n_points > 0) fillValidation(s, out);
  return RG_OK;
}

extern "C" rg_status rg_grid_validate_triquintic(rg_ctx* ctx, const rg_forcefield* ff, const rg_box* unit_cell,
                                                 const rg_atom* unit_atoms, int n_unit_atoms,
                                                 const rg_box* simulation_box, int probe_type, int nx, int ny, int nz,
                                                 const double* vdw_grid_device, const double* ewald_grid_device,
                                                 double probe_charge, double weight_beta, int64_t n_points,
                                                 uint64_t seed, const double* points, rg_grid_validation* out,
                                                 rg_grid_validation_hessian* hessian)
{
  if (ctx && (!out || !hessian))
    return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_grid_validate_triquintic: null or negative argument");
  std::vector<double> s;
  rg_status st = runValidate<RG_SCHEME_TRIQUINTIC>(ctx, "rg_grid_validate_triquintic", ff, unit_cell, unit_atoms,
                                                   n_unit_atoms, simulation_box, probe_type, nx, ny, nz,
                                                   vdw_grid_device, ewald_grid_device, probe_charge, weight_beta,
                                                   n_points, seed, points, s);
  if (st) return st;
  std::memset(out, 0, sizeof(*out));
  std::memset(hessian, 0, sizeof(*hessian));
  if (n_points == 0) return RG_OK;
  fillValidation(s, out);
  for (int c = 0; c < kHessSums; ++c) hessian->sums[c] = s[kSums + c];
  deriveHessian(s.data() + kSums, s[0], hessian->hessian_table, hessian->hessian_full,
                hessian->hessian_relative_error);
  deriveHessian(s.data() + kSums + 24, s[17], hessian->charge_hessian_table, hessian->charge_hessian_full,
                hessian->charge_hessian_relative_error);
  return RG_OK;
}
