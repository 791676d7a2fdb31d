// (c) Ewald Fourier energy of a Monte Carlo move, on device-resident structure factors.
//
// Replaces Interactions::energyDifferenceEwaldFourier (src/raspakit/interactions/ewald.cpp:1043-1244),
// Interactions::acceptEwaldMove (ewald.cpp:1565-1574), Interactions::computeEwaldFourierEnergy (ewald.cpp:352-563)
// and Interactions::precomputeEwaldFourierRigid (ewald.cpp:276-348).
//
// Layout in HBM, per system: the accepted k-vectors in the reference loop order (kx in [0,kmax], ky and kz in
// [-kmax,kmax], k != 0, integer-sphere and reciprocal-cutoff tests) as char4 (kx,ky,kz,-), the prefactor
// temp(k) = C*2pi/V*(kx==0 ? 1 : 2)*exp(-|k|^2/(4 alpha^2))/|k|^2 in FP64, and two FP64 complex structure-factor
// buffers of (1 + groups) entries per k (the total and the dU/dlambda group sums), "stored" and "trial". A move
// writes trial = stored + Delta rho; accepting swaps the two pointers instead of the reference's full vector copy.
// The Fourier energy change per k is computed as temp*(2 Re(conj(S) dRho) + |dRho|^2), algebraically the reference's
// temp*(|S + dRho|^2 - |S|^2) without the cancellation. Block partial sums are posted into mapped pinned host memory,
// where the host adds them in block order (up to kDeltaPosted blocks), or reduced in a fixed order by the last block to
// finish, which posts the totals; either is deterministic. A move of up to 16 atoms travels in the launch's parameter
// block, so one difference costs one launch and the wait for the posts. The full recompute splits the atoms into chunks
// along a second grid dimension and sums the chunks' partial structure factors in chunk order. The self, exclusion and
// net-charge terms are FP64 sums, on the host for a move or a few atoms (kHostTerms), else on the device.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "energy.cuh"

struct rg_ewald
{
  rg_ctx* ctx = nullptr;
  int n_groups = 0;
  int64_t nk = 0;
  double single_ion_sum = 0.0;  // sum_k temp(k)
  double alpha = 0.0;
  double volume = 0.0;
  rg::HostBox box{};
  rg_forcefield ff{};
  bool omit_inter = false;
  bool use_charge = true;
  // device
  char4* kvec = nullptr;
  double* temp = nullptr;
  double2* s_rigid = nullptr;  // framework structure factor, nk entries (zero if no framework)
  double2* stored = nullptr;   // nk*(1+G)
  double2* trial = nullptr;    // nk*(1+G)
  double* partial = nullptr;   // per-block partial sums
  unsigned int* counter = nullptr;
  ulonglong2* result = nullptr;  // 1 + G results and (from kTermsAt) the atoms' terms: device view of result_host
  // the k-vectors by (kx, ky) pair: the pairs, and per pair the index of the k-vector with kz = -kmax_z..kmax_z (-1:
  // not in the set)
  int n_pairs = 0;
  char2* pairs = nullptr;
  int* kmap = nullptr;
  std::vector<char2> pairs_host;
  std::vector<int> kmap_host;
  int sms = 148;
  // staging of the last staged atoms: the context's scratch, set anew by each call that stages (stageRoom)
  void* moved = nullptr;
  void* moved_host = nullptr;
  ulonglong2* result_host = nullptr;  // mapped pinned: the kernels post their sums or totals here (rg::collect)
  unsigned int calls = 0;
};

namespace
{
constexpr int kThreads = 256;
constexpr int kMaxGroups = 4;
constexpr int kMaxMoved = 512;  // old + new atoms of one move (staged in shared memory)
constexpr int kParamMoved = 16; // moves of up to this many atoms travel in the launch's parameter block

struct MovedAtom
{
  double s[3];   // fractional coordinates (inverse cell * position)
  double w;      // sign * scalingCoulomb * charge (sign -1 for old atoms)
  double wg;     // sign * charge (dU/dlambda group sums)
  int group;     // 0 = none, 1..4
  int mol_end;   // full recompute: index after the last atom of the atom's molecule (its own index if it has none)
};

// the moved atoms of a small move, passed by value in the launch parameters (no copy before the launch)
struct MovedParam
{
  MovedAtom a[kParamMoved];
};

// Sum of v over the block, complete in thread 0
template <int G>
__device__ __forceinline__ void blockSum(double (&v)[1 + G], double (*red)[1 + kMaxGroups])
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 1 + G; ++c)
  {
    double x = v[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp][c] = x;
  }
  __syncthreads();
  if (warp == 0)
  {
#pragma unroll
    for (int c = 0; c < 1 + G; ++c)
    {
      double x = lane < kThreads / 32 ? red[lane][c] : 0.0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      v[c] = x;
    }
  }
}

template <int G>
__device__ __forceinline__ void blockReduceAndFinish(double (&v)[1 + G], double* partial, unsigned int* counter,
                                                     ulonglong2* result, unsigned call, unsigned n_blocks,
                                                     unsigned block)
{
  __shared__ double red[kThreads / 32][1 + kMaxGroups];
  __shared__ bool last;
  blockSum<G>(v, red);
  if (n_blocks > 1)
  {
    if (threadIdx.x == 0)
    {
#pragma unroll
      for (int c = 0; c < 1 + G; ++c) partial[block * (1 + kMaxGroups) + c] = v[c];
      last = rg::countIn(counter) == n_blocks - 1;
    }
    __syncthreads();
    if (!last) return;
    // the last block: each thread sums the partials of blocks threadIdx.x, threadIdx.x + kThreads, ... (all its loads in
    // flight together), then the same fixed-order warp and block reduction
#pragma unroll
    for (int c = 0; c < 1 + G; ++c) v[c] = 0.0;
    for (unsigned b = threadIdx.x; b < n_blocks; b += kThreads)
    {
#pragma unroll
      for (int c = 0; c < 1 + G; ++c) v[c] += __ldcg(partial + b * (1 + kMaxGroups) + c);
    }
    blockSum<G>(v, red);
  }
  if (threadIdx.x == 0)
  {
#pragma unroll
    for (int c = 0; c < 1 + G; ++c) rg::post(result + c, v[c], call);
    *counter = 0u;  // ready for the next launch on this system
  }
}

// One thread per k-vector: the change of the structure factor caused by the moved atoms, the Fourier energy change and
// its dU/dlambda group terms, and the trial structure factor. Latency bounds it (six atoms and 1,000 k-vectors are
// 60,000 FP64 instructions), so the chain is kept short: the phase of a k-vector is the product of three entries of
// tables e^{i 2 pi m s_d}, one sincospi per thread and tile of atoms while the k-vector's own loads are in flight; a
// sincospi per atom and k-vector is a chain of as many as there are atoms. Per call with 8,124 k-vectors and 6, 30 and
// 120 atoms 18.7, 26.6 and 43.5 us before, 16.7, 23.5 and 36.4 us so, and with the results posted 12.6, 19.1 and 32.3 us.
// (One block of 1,024 threads for sets that fit it saves the second reduction, but its one SM does all the products: 17.2,
// 29.9 and 69.3 us at 1,152 k-vectors against 16.8, 23.1 and 34.6 us with blocks of 256 at 2,600.)
constexpr int kDeltaTile = 16;                 // atoms whose tables are in shared memory at a time, at most
// Up to this many blocks each block posts its own sums and the host adds them in block order: the reduction across blocks
// on the device (an atomic, a second read and sum) makes a call of 8,124 k-vectors 14.5 us long, without it 12.6
constexpr int kDeltaPosted = 64;
constexpr size_t kDeltaShared = 40 << 10;      // bytes of tables at most: fewer atoms per tile for a large kmax
template <int G>
__global__ void __launch_bounds__(kThreads) ewaldDeltaKernel(int nk, int kxm, int kym, int kzm,
                                                             const char4* __restrict__ kvec,
                                                             const double* __restrict__ temp,
                                                             const double2* __restrict__ stored,
                                                             double2* __restrict__ trial,
                                                             const MovedAtom* __restrict__ moved,
                                                             const __grid_constant__ MovedParam small, int n_moved,
                                                             int tile, double* partial, unsigned int* counter,
                                                             ulonglong2* result, unsigned call)
{
  extern __shared__ double2 tab[];  // [tile][stride]
  __shared__ MovedAtom sm[kDeltaTile];
  const int stride = kxm + kym + kzm + 3;
  const int k = blockIdx.x * kThreads + threadIdx.x;
  const bool in = k < nk;
  const int64_t row = static_cast<int64_t>(k) * (1 + G);
  const char4 kv = in ? kvec[k] : make_char4(0, 0, 0, 0);
  const double t = in ? temp[k] : 0.0;
  const double2 S = in ? stored[row] : make_double2(0.0, 0.0);
  const int atx = kv.x, aty = kxm + 1 + (kv.y < 0 ? -kv.y : kv.y), atz = kxm + kym + 2 + (kv.z < 0 ? -kv.z : kv.z);
  double2 d = make_double2(0.0, 0.0);
  double2 dg[G > 0 ? G : 1];
#pragma unroll
  for (int g = 0; g < (G > 0 ? G : 1); ++g) dg[g] = make_double2(0.0, 0.0);
  for (int base = 0; base < n_moved; base += tile)
  {
    const int n = min(tile, n_moved - base);
    if (base > 0) __syncthreads();
    constexpr int kWords = sizeof(MovedAtom) / sizeof(double);
    const double* from = reinterpret_cast<const double*>(moved ? moved + base : small.a + base);
    for (int w = threadIdx.x; w < n * kWords; w += kThreads) reinterpret_cast<double*>(sm)[w] = from[w];
    __syncthreads();
    for (int i = threadIdx.x; i < n * stride; i += kThreads)
    {
      const int a = i / stride;
      int m = i - a * stride, dim = 0;
      if (m > kxm)
      {
        m -= kxm + 1;
        dim = 1;
        if (m > kym)
        {
          m -= kym + 1;
          dim = 2;
        }
      }
      double sn, cs;
      sincospi(2.0 * (m * sm[a].s[dim]), &sn, &cs);
      tab[i] = make_double2(cs, sn);
    }
    __syncthreads();
    for (int a = 0; a < n; ++a)
    {
      const double w = sm[a].w, wg = sm[a].wg;
      const int group = sm[a].group;
      const double2* at = tab + a * stride;
      const double2 x = at[atx];
      double2 y = at[aty], z = at[atz];
      y.y = kv.y < 0 ? -y.y : y.y;
      z.y = kv.z < 0 ? -z.y : z.y;
      const double2 xy = make_double2(x.x * y.x - x.y * y.y, x.x * y.y + x.y * y.x);
      const double2 e = make_double2(xy.x * z.x - xy.y * z.y, xy.x * z.y + xy.y * z.x);
      d.x += w * e.x;
      d.y += w * e.y;
#pragma unroll
      for (int g = 0; g < G; ++g)
        if (group == g + 1)
        {
          dg[g].x += wg * e.x;
          dg[g].y += wg * e.y;
        }
    }
  }
  double v[1 + G];
#pragma unroll
  for (int c = 0; c < 1 + G; ++c) v[c] = 0.0;
  if (in)
  {
    const double2 T = make_double2(S.x + d.x, S.y + d.y);
    v[0] = t * (2.0 * (S.x * d.x + S.y * d.y) + (d.x * d.x + d.y * d.y));
    trial[row] = T;
#pragma unroll
    for (int g = 0; g < G; ++g)
    {
      const double2 SG = stored[row + 1 + g];
      const double2 TG = make_double2(SG.x + dg[g].x, SG.y + dg[g].y);
      // addFourierDUdlambda(2 temp, T, TG) - addFourierDUdlambda(2 temp, S, SG)  (ewald.cpp:166-173)
      v[1 + g] = 2.0 * t * ((T.x * TG.x + T.y * TG.y) - (S.x * SG.x + S.y * SG.y));
      trial[row + 1 + g] = TG;
    }
  }
  if (gridDim.x > kDeltaPosted)
  {
    blockReduceAndFinish<G>(v, partial, counter, result, call, gridDim.x, blockIdx.x);
    return;
  }
  __shared__ double red[kThreads / 32][1 + kMaxGroups];
  blockSum<G>(v, red);
  if (threadIdx.x == 0)
#pragma unroll
    for (int c = 0; c < 1 + G; ++c) rg::post(result + blockIdx.x * (1 + G) + c, v[c], call);
}

// Partial sums of the structure factor of one chunk of atoms, for one (kx, ky) pair per thread and MT consecutive values
// of m = |kz|. With P = w e^{2 pi i (kx s_x + ky s_y)} = (p, q) and e^{2 pi i m s_z} = (c, s) the four sums of p c, q s,
// p s and q c give both kz = m, (pc - qs, ps + qc), and kz = -m, (pc + qs, qc - ps): two FP64 FMAs per k-vector and
// atom where a complex product each takes four, and P is formed once for the pair's whole run of kz. The tables of
// e^{2 pi i m s_d} are built in shared memory per tile of atoms; x carries the atom's weight, y has both signs.
// The bound is the FP64 pipe: 4 MT + 4 instructions per atom and thread, the z phasors are broadcast reads. A recompute of
// 12,000 sites x 8,124 k-vectors took 445 us with a thread per k-vector and two complex products per atom, now 180 us.
// Output: out[chunk][m][pair] = {(sum pc, sum qs), (sum ps, sum qc)}.
constexpr int kPairWarps = 11;  // warps of a block at most
constexpr int kPairBlocks = 2;  // blocks of that size per SM
template <int MT>
__global__ void __launch_bounds__(32 * kPairWarps, kPairBlocks) ewaldPairSumsKernel(
    int n_pairs, const char2* __restrict__ pairs, const MovedAtom* __restrict__ atoms, int n_atoms, int chunk_atoms,
    int tile, int kxm, int kym, int kzm, double2* __restrict__ out)
{
  extern __shared__ double2 tab[];  // tile * ((kxm + 1) + (2 kym + 1) + mt_total)
  const int nx = kxm + 1, ny = 2 * kym + 1;
  const int m0 = blockIdx.z * MT;
  double2* tx = tab;
  double2* ty = tx + tile * nx;
  double2* tz = ty + tile * ny;
  const int pair = blockIdx.x * blockDim.x + threadIdx.x;
  const char2 pq = pairs[min(pair, n_pairs - 1)];
  const int a0 = blockIdx.y * chunk_atoms, a1 = min(n_atoms, a0 + chunk_atoms);
  double pc[MT], qs[MT], ps[MT], qc[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) pc[m] = qs[m] = ps[m] = qc[m] = 0.0;
  const int per = nx + (kym + 1) + MT;
  for (int base = a0; base < a1; base += tile)
  {
    const int na = min(tile, a1 - base);
    __syncthreads();
    for (int idx = threadIdx.x; idx < na * per; idx += blockDim.x)
    {
      const int a = idx / per, m = idx - a * per;
      const MovedAtom& at = atoms[base + a];
      const int d = m < nx ? 0 : (m < nx + kym + 1 ? 1 : 2);
      const int mm = d == 0 ? m : (d == 1 ? m - nx : m0 + m - nx - (kym + 1));
      double sn, cs;
      sincospi(2.0 * static_cast<double>(mm) * at.s[d], &sn, &cs);
      if (d == 0)
        tx[a * nx + mm] = make_double2(at.w * cs, at.w * sn);
      else if (d == 1)
      {
        ty[a * ny + kym + mm] = make_double2(cs, sn);
        ty[a * ny + kym - mm] = make_double2(cs, -sn);
      }
      else
        tz[a * MT + mm - m0] = make_double2(cs, sn);
    }
    __syncthreads();
    for (int a = 0; a < na; ++a)
    {
      const double2 x = tx[a * nx + pq.x], y = ty[a * ny + kym + pq.y];
      const double p = x.x * y.x - x.y * y.y, q = x.x * y.y + x.y * y.x;
#pragma unroll
      for (int m = 0; m < MT; ++m)
      {
        const double2 z = tz[a * MT + m];
        pc[m] = fma(p, z.x, pc[m]);
        qs[m] = fma(q, z.y, qs[m]);
        ps[m] = fma(p, z.y, ps[m]);
        qc[m] = fma(q, z.x, qc[m]);
      }
    }
  }
  if (pair >= n_pairs) return;
#pragma unroll
  for (int m = 0; m < MT; ++m)
    if (m0 + m <= kzm)
    {
      double2* o = out + 2 * ((static_cast<int64_t>(blockIdx.y) * (kzm + 1) + m0 + m) * n_pairs + pair);
      o[0] = make_double2(pc[m], qs[m]);
      o[1] = make_double2(ps[m], qc[m]);
    }
}

// Self, intramolecular exclusion and net-charge sums of the adsorbates (ewald.cpp:480-560) for the full recompute:
// thread i adds atom i's own terms and its pairs with the later atoms of its molecule. Columns: self, exclusion, net
// charge, dU/dlambda [4], charge of each group [4]; per-block sums, added in block order by the last block.
constexpr int kTerms = 11;
constexpr int kTermsAt = 8;  // where they start in the result array (the Fourier sums come first)
// results of one call at most: the recompute's, or the blocks' sums of a difference
constexpr int kResults = kDeltaPosted * (1 + kMaxGroups);
static_assert(kResults >= kTermsAt + kTerms, "room for both");
struct TermsParams
{
  const MovedAtom* atoms;
  int n_atoms, blocks;      // blocks = 0: none
  double* partial;          // [blocks][kTerms]
  unsigned int* counter;
  ulonglong2* result;
  double cell[9];           // c[col][row] by columns
  int triclinic;
  double alpha, coul, self;  // self = C alpha / sqrt(pi)
};
__device__ __forceinline__ double roundAway(double x)
{
  return static_cast<double>(static_cast<long long>(x + ((x >= 0.0) ? 0.5 : -0.5)));
}
__device__ __forceinline__ void addToGroup(double* v, int g, double x)
{
#pragma unroll
  for (int k = 0; k < kMaxGroups; ++k)
    if (g == k + 1) v[k] += x;
}
__device__ __forceinline__ void atomTerms(const TermsParams& p, int omit_inter, int block, unsigned call)
{
  const MovedAtom* __restrict__ atoms = p.atoms;
  const int n_atoms = p.n_atoms, n_blocks = p.blocks;
  __shared__ double red[kThreads / 32][kTerms];
  __shared__ bool last;
  const int i = block * kThreads + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[kTerms];
#pragma unroll
  for (int c = 0; c < kTerms; ++c) v[c] = 0.0;
  if (i < n_atoms)
  {
    const MovedAtom A = atoms[i];
    v[2] = A.w;
    addToGroup(v + 7, A.group, A.wg);
    if (!omit_inter)
    {
      v[0] = -p.self * A.w * A.w;
      addToGroup(v + 3, A.group, -2.0 * p.self * A.w * A.wg);
      const double sA = A.wg != 0.0 ? A.w / A.wg : 0.0;  // scaling; an uncharged atom has no terms
      for (int j = i + 1; j < A.mol_end; ++j)
      {
        const MovedAtom B = atoms[j];
        const double sB = B.wg != 0.0 ? B.w / B.wg : 0.0;
        double d[3], r[3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
          d[a] = A.s[a] - B.s[a];
          d[a] -= roundAway(d[a]);
        }
        double rr = 0.0;
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
          r[a] = p.triclinic ? p.cell[a] * d[0] + p.cell[3 + a] * d[1] + p.cell[6 + a] * d[2] : p.cell[4 * a] * d[a];
          rr += r[a] * r[a];
        }
        // Potentials::ewaldExclusionFactors (src/raspakit/potentials/coulomb_real_space.ixx:49-65)
        const double sc = sA * sB;
        const double x = sqrt(rr) + 0.01 * (1.0 - sc), inv = 1.0 / x;
        const double pot = erf(p.alpha * x) * inv;
        const double gauss = 2.0 * p.alpha * rg::kInvSqrtPi * exp(-p.alpha * p.alpha * x * x);
        const double dudl = pot - sc * 0.01 * ((gauss - pot) * inv);
        v[1] -= p.coul * A.w * B.w * pot;
        const double f = -p.coul * A.wg * B.wg * dudl;
        addToGroup(v + 3, A.group, sB * f);
        addToGroup(v + 3, B.group, sA * f);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < kTerms; ++c)
  {
    double x = v[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp][c] = x;
  }
  __syncthreads();
  if (threadIdx.x < kTerms)
  {
    double x = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) x += red[w][threadIdx.x];
    p.partial[block * kTerms + threadIdx.x] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0)
  {
    last = rg::countIn(p.counter) == static_cast<unsigned>(n_blocks - 1);
  }
  __syncthreads();
  if (!last) return;
  // a warp per column, the blocks by lane, then a fixed shuffle tree
  for (int c = warp; c < kTerms; c += kThreads / 32)
  {
    double x = 0.0;
    for (int b = lane; b < n_blocks; b += 32) x += __ldcg(p.partial + b * kTerms + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) rg::post(p.result + c, x, call);
  }
  if (threadIdx.x == 0) *p.counter = 0u;
}

// The chunks' sums of one (pair, m) added in a fixed order by kFinishLanes threads (a warp covers 4 neighbouring pairs),
// then both k-vectors of it: with RIGID the framework's structure factor, else the stored one and the Fourier energy
// temp (|S_fw + S_ads|^2 - |S_fw|^2) = temp (2 Re(conj(S_fw) S_ads) + |S_ads|^2) (ewald.cpp:458-468). The first
// terms.blocks blocks take the atoms' own terms meanwhile.
constexpr int kFinishLanes = 8;
template <bool RIGID>
__global__ void __launch_bounds__(kThreads) ewaldPairFinishKernel(int n_pairs, int kzm, int n_chunks,
                                                                  const double2* __restrict__ sums,
                                                                  const int* __restrict__ kmap,
                                                                  const double* __restrict__ temp, double2* s_rigid,
                                                                  double2* __restrict__ stored, int omit_inter,
                                                                  double* partial, unsigned int* counter,
                                                                  ulonglong2* result, TermsParams terms, unsigned call)
{
  if constexpr (!RIGID)
    if (static_cast<int>(blockIdx.x) < terms.blocks)
    {
      atomTerms(terms, omit_inter, blockIdx.x, call);
      return;
    }
  const unsigned block = blockIdx.x - terms.blocks;
  constexpr int kItems = kThreads / kFinishLanes;
  // the lanes of an item are kItems apart, so that a warp reads runs of neighbouring pairs
  const int item = threadIdx.x % kItems, part = threadIdx.x / kItems;
  const int64_t total = static_cast<int64_t>(n_pairs) * (kzm + 1);
  const int64_t at = static_cast<int64_t>(block) * kItems + item;
  double2 u = make_double2(0.0, 0.0), v = make_double2(0.0, 0.0);
  if (at < total)
#pragma unroll 4
    for (int c = part; c < n_chunks; c += kFinishLanes)
    {
      const double2* in = sums + 2 * (c * total + at);
      u.x += in[0].x;
      u.y += in[0].y;
      v.x += in[1].x;
      v.y += in[1].y;
    }
  __shared__ double2 su[kThreads], sv[kThreads];
  su[threadIdx.x] = u;
  sv[threadIdx.x] = v;
  __syncthreads();
  double e[1] = {0.0};
  if (part == 0 && at < total)
  {
#pragma unroll
    for (int q = 1; q < kFinishLanes; ++q)
    {
      const double2 a = su[q * kItems + item], b = sv[q * kItems + item];
      u.x += a.x;
      u.y += a.y;
      v.x += b.x;
      v.y += b.y;
    }
    const int m = static_cast<int>(at / n_pairs), pair = static_cast<int>(at - static_cast<int64_t>(m) * n_pairs);
    const int* map = kmap + static_cast<int64_t>(pair) * (2 * kzm + 1) + kzm;
#pragma unroll
    for (int sign = 0; sign < 2; ++sign)
    {
      if (sign == 1 && m == 0) break;
      const int k = sign == 0 ? map[m] : map[-m];
      if (k < 0) continue;
      const double2 A = sign == 0 ? make_double2(u.x - u.y, v.x + v.y) : make_double2(u.x + u.y, v.y - v.x);
      if constexpr (RIGID)
        s_rigid[k] = A;
      else
      {
        const double t = temp[k];
        const double2 R = s_rigid[k];
        const double own = A.x * A.x + A.y * A.y;
        e[0] += t * (2.0 * (R.x * A.x + R.y * A.y) + own);
        if (omit_inter) e[0] -= t * own;
        stored[k] = make_double2(R.x + A.x, R.y + A.y);
      }
    }
  }
  if constexpr (!RIGID)
    blockReduceAndFinish<0>(e, partial, counter, result, call, gridDim.x - terms.blocks, block);
}

// The atoms' own terms by themselves (no k-vectors, or dU/dlambda groups, whose Fourier sums take the kernels below)
__global__ void __launch_bounds__(kThreads) ewaldAtomTermsKernel(TermsParams p, int omit_inter, unsigned call)
{
  atomTerms(p, omit_inter, blockIdx.x, call);
}

// With dU/dlambda groups: per-atom phase tables e^{i 2 pi m s_d}, m = 0..kmax_d, built in shared memory for a tile of
// atoms; each thread owns one k-vector and accumulates over the tile with two complex products per atom.
constexpr int kFullTile = 32;

template <int G>
__global__ void __launch_bounds__(kThreads) ewaldFullPartialKernel(int64_t nk, const char4* __restrict__ kvec,
                                                                   const MovedAtom* __restrict__ atoms, int n_atoms,
                                                                   int chunk_atoms, int kxm, int kym, int kzm,
                                                                   double2* __restrict__ scratch)
{
  // blockIdx.y: a chunk of atoms; each thread owns one k-vector and sums the chunk's atoms with two complex products
  // per atom, from per-atom phase tables e^{i 2 pi m s_d} (m = 0..kmax_d) built in shared memory per tile
  extern __shared__ double2 tab[];  // kFullTile * (kxm+1 + kym+1 + kzm+1)
  __shared__ double wq[kFullTile], wgq[kFullTile];
  __shared__ int grp[kFullTile];
  const int stride = (kxm + 1) + (kym + 1) + (kzm + 1);
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  const int a0 = blockIdx.y * chunk_atoms, a1 = min(n_atoms, a0 + chunk_atoms);
  char4 kv = make_char4(0, 0, 0, 0);
  if (k < nk) kv = kvec[k];
  double2 acc = make_double2(0.0, 0.0);
  double2 accg[G > 0 ? G : 1];
#pragma unroll
  for (int g = 0; g < (G > 0 ? G : 1); ++g) accg[g] = make_double2(0.0, 0.0);
  for (int base = a0; base < a1; base += kFullTile)
  {
    const int na = min(kFullTile, a1 - base);
    __syncthreads();
    for (int idx = threadIdx.x; idx < na * stride; idx += blockDim.x)
    {
      int a = idx / stride, m = idx % stride;
      int d = (m <= kxm) ? 0 : ((m <= kxm + 1 + kym) ? 1 : 2);
      int mm = (d == 0) ? m : ((d == 1) ? m - (kxm + 1) : m - (kxm + 1) - (kym + 1));
      double sn, cs;
      sincospi(2.0 * static_cast<double>(mm) * atoms[base + a].s[d], &sn, &cs);
      tab[a * stride + m] = make_double2(cs, sn);
    }
    for (int a = threadIdx.x; a < na; a += blockDim.x)
    {
      wq[a] = atoms[base + a].w;
      wgq[a] = atoms[base + a].wg;
      grp[a] = atoms[base + a].group;
    }
    __syncthreads();
    if (k < nk)
    {
      const int ax = kv.x, ay = abs(kv.y), az = abs(kv.z);
      const double sy = kv.y < 0 ? -1.0 : 1.0, sz = kv.z < 0 ? -1.0 : 1.0;
      for (int a = 0; a < na; ++a)
      {
        const double2* t = tab + a * stride;
        double2 ex = t[ax], ey = t[kxm + 1 + ay], ez = t[kxm + 1 + kym + 1 + az];
        ey.y *= sy;
        ez.y *= sz;
        double2 xy = make_double2(ex.x * ey.x - ex.y * ey.y, ex.x * ey.y + ex.y * ey.x);
        double2 e = make_double2(xy.x * ez.x - xy.y * ez.y, xy.x * ez.y + xy.y * ez.x);
        acc.x += wq[a] * e.x;
        acc.y += wq[a] * e.y;
        if (G > 0)
        {
#pragma unroll
          for (int gg = 0; gg < (G > 0 ? G : 1); ++gg)
            if (grp[a] == gg + 1)
            {
              accg[gg].x += wgq[a] * e.x;
              accg[gg].y += wgq[a] * e.y;
            }
        }
      }
    }
  }
  if (k < nk)
  {
    double2* out = scratch + (static_cast<int64_t>(blockIdx.y) * nk + k) * (1 + G);
    out[0] = acc;
#pragma unroll
    for (int g = 0; g < G; ++g) out[1 + g] = accg[g];
  }
}

// The chunks' partial structure factors summed in chunk order, the framework's added, the Fourier energy and its
// dU/dlambda group terms (ewald.cpp:458-468), reduced in a fixed order by the last block.
template <int G>
__global__ void __launch_bounds__(kThreads) ewaldFullFinishKernel(int64_t nk, int n_chunks,
                                                                  const double2* __restrict__ scratch,
                                                                  const double* __restrict__ temp,
                                                                  const double2* __restrict__ s_rigid,
                                                                  double2* __restrict__ stored, int omit_inter,
                                                                  double* partial, unsigned int* counter,
                                                                  ulonglong2* result, unsigned call)
{
  const int64_t k = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  double v[1 + G];
#pragma unroll
  for (int c = 0; c < 1 + G; ++c) v[c] = 0.0;
  if (k < nk)
  {
    double2 acc = make_double2(0.0, 0.0);
    double2 accg[G > 0 ? G : 1];
#pragma unroll
    for (int g = 0; g < (G > 0 ? G : 1); ++g) accg[g] = make_double2(0.0, 0.0);
    for (int c = 0; c < n_chunks; ++c)
    {
      const double2* in = scratch + (static_cast<int64_t>(c) * nk + k) * (1 + G);
      acc.x += in[0].x;
      acc.y += in[0].y;
#pragma unroll
      for (int g = 0; g < G; ++g)
      {
        accg[g].x += in[1 + g].x;
        accg[g].y += in[1 + g].y;
      }
    }
    const double t = temp[k];
    const double2 R = s_rigid[k];
    const double2 T = make_double2(R.x + acc.x, R.y + acc.y);
    // temp*(|S_fw + S_ads|^2 - |S_fw|^2) = temp*(2 Re(conj(S_fw) S_ads) + |S_ads|^2)  (ewald.cpp:458-468)
    v[0] = t * (2.0 * (R.x * acc.x + R.y * acc.y) + (acc.x * acc.x + acc.y * acc.y));
    if (omit_inter) v[0] -= t * (acc.x * acc.x + acc.y * acc.y);
    stored[k * (1 + G)] = T;
#pragma unroll
    for (int g = 0; g < G; ++g)
    {
      // rigid group sums are zero (precomputeEwaldFourierRigid sets only the total)
      v[1 + g] = 2.0 * t * (T.x * accg[g].x + T.y * accg[g].y);
      stored[k * (1 + G) + 1 + g] = accg[g];
    }
  }
  blockReduceAndFinish<G>(v, partial, counter, result, call, gridDim.x, blockIdx.x);
}

inline int groupOf(const rg_atom& a) { return a.group_fractional & 0x0f; }

void roundHalfAwayPbc(const rg::HostBox& b, double dr[3])
{
  // SimulationBox::applyPeriodicBoundaryConditions (src/raspakit/simulationbox.ixx:131-161)
  auto rnd = [](double x) { return static_cast<double>(static_cast<long long>(x + ((x >= 0.0) ? 0.5 : -0.5))); };
  if (!b.triclinic)
  {
    dr[0] -= rnd(dr[0] * b.ic[0][0]) * b.c[0][0];
    dr[1] -= rnd(dr[1] * b.ic[1][1]) * b.c[1][1];
    dr[2] -= rnd(dr[2] * b.ic[2][2]) * b.c[2][2];
    return;
  }
  double s[3];
  rg::matvec(b.ic, dr, s);
  for (int d = 0; d < 3; ++d) s[d] -= rnd(s[d]);
  rg::matvec(b.c, s, dr);
}

// Potentials::ewaldExclusionFactors (src/raspakit/potentials/coulomb_real_space.ixx:49-65)
void exclusionFactors(double alpha, double scalingTotal, double r, double& potential, double& dudl)
{
  const double s = r + 0.01 * (1.0 - scalingTotal);
  const double inverseS = 1.0 / s;
  potential = std::erf(alpha * s) * inverseS;
  const double gaussianTerm = 2.0 * alpha * rg::kInvSqrtPi * std::exp(-alpha * alpha * s * s);
  const double firstDerivative = (gaussianTerm - potential) * inverseS;
  dudl = potential - scalingTotal * 0.01 * firstDerivative;
}

void addDud(double* arr, int gA, int gB, double sA, double sB, double factor)
{
  if (gA != 0 && gA <= kMaxGroups) arr[gA - 1] += sB * factor;
  if (gB != 0 && gB <= kMaxGroups) arr[gB - 1] += sA * factor;
}

// The columns of atomTerms on the host (ewald.cpp:480-560). Up to kHostTerms atoms this is the faster side: hidden behind
// the kernels here, while the device's chain of loads, erf and reductions made calls of 15 to 180 atoms 3 to 8 us longer.
// For 12,000 atoms the erf alone take the host 130 us, and the device's share does not show.
constexpr int kHostTerms = 256;
// Without k-vectors, or with dU/dlambda groups (whose Fourier sums have kernels of their own), the device's share is a
// launch by itself, which shows: up to this many pairs within molecules the host is the faster side. Of molecules of three
// atoms (kmax 8, one group) 270, 540, 1,200 and 2,400 take 32, 41, 62 and 114 us with the host's terms and 40, 48, 62 and 93
// with the device's; of molecules of ten 270 and 540 (1,215 and 2,430 pairs) 44 and 80, and 45 and 52.
constexpr int64_t kHostPairs = 1300;
void hostTerms(const rg_ewald* e, const rg_atom* atoms, int n_atoms, const int32_t* molecule_sizes, int n_molecules,
               double v[kTerms])
{
  const double C = rg::coulombFactor(), self = C * e->alpha / std::sqrt(rg::kPi);
  for (int i = 0; i < n_atoms; ++i)
  {
    const double q = atoms[i].charge, sc = atoms[i].scaling_coulomb;
    const int g = groupOf(atoms[i]);
    v[2] += sc * q;
    if (g != 0 && g <= kMaxGroups) v[6 + g] += q;
    if (e->omit_inter) continue;
    v[0] -= self * sc * q * sc * q;
    if (g != 0 && g <= kMaxGroups) v[2 + g] -= 2.0 * self * sc * q * q;
  }
  for (int m = 0, index = 0; m < n_molecules && !e->omit_inter; index += molecule_sizes[m++])
    for (int i = index; i < index + molecule_sizes[m]; ++i)
      for (int j = i + 1; j < index + molecule_sizes[m]; ++j)
      {
        double dr[3] = {atoms[i].x - atoms[j].x, atoms[i].y - atoms[j].y, atoms[i].z - atoms[j].z};
        roundHalfAwayPbc(e->box, dr);
        const double r = std::sqrt(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]);
        const double sA = atoms[i].scaling_coulomb, sB = atoms[j].scaling_coulomb;
        double pot, dudl;
        exclusionFactors(e->alpha, sA * sB, r, pot, dudl);
        const double prefactor = C * atoms[i].charge * atoms[j].charge;
        v[1] -= sA * sB * prefactor * pot;
        addDud(v + 3, groupOf(atoms[i]), groupOf(atoms[j]), sA, sB, -prefactor * dudl);
      }
}

// Whether the terms are the host's. The device has the atoms' fractional coordinates alone and takes the minimum image in
// those; for a cell given as rectangular whose vectors are off the axes that is another image than along its diagonal.
bool hostTermsOf(const rg_ewald* e, int n_atoms, const int32_t* molecule_sizes, int n_molecules)
{
  if (n_atoms <= kHostTerms) return true;
  if (e->nk == 0 || e->n_groups > 0)
  {
    int64_t pairs = 0;
    for (int m = 0; m < n_molecules && !e->omit_inter; ++m)
      pairs += static_cast<int64_t>(molecule_sizes[m]) * (molecule_sizes[m] - 1) / 2;
    if (pairs <= kHostPairs) return true;
  }
  bool sheared = false;
  for (int c = 0; c < 3; ++c)
    for (int r = 0; r < 3; ++r) sheared = sheared || (c != r && e->box.c[c][r] != 0.0);
  return sheared && !e->box.triclinic;
}

// fractional coordinates and signed weights of the old (sign old_sign) and new atoms of a move
void packMoved(const rg_ewald* e, const rg_atom* old_atoms, int n_old, const rg_atom* new_atoms, int n_new,
               double old_sign, MovedAtom* h)
{
  for (int i = 0; i < n_old + n_new; ++i)
  {
    const bool isOld = i < n_old;
    const rg_atom& a = isOld ? old_atoms[i] : new_atoms[i - n_old];
    const double sign = isOld ? old_sign : 1.0;
    double r[3] = {a.x, a.y, a.z};
    rg::matvec(e->box.ic, r, h[i].s);
    h[i].w = sign * a.scaling_coulomb * a.charge;
    h[i].wg = sign * a.charge;
    h[i].group = groupOf(a);
    h[i].mol_end = 0;
  }
}

// Scratch of the calls below: the context's slots, which every Ewald state on it shares (whoever stages waits for the
// stream first): the chunks' partial structure factors, the atoms' own terms, the staged atoms (device and pinned). With
// buffers of each state's own the first recompute of a state with 12,000 sites took 7.9 ms, now 0.23 ms.
constexpr int kSumsSlot = 8, kTermsSlot = 9, kMovedSlot = 10, kMovedPinnedSlot = 3;

// Staging buffers of at least n atoms, free of earlier copies
rg_status stageRoom(rg_ewald* e, int n)
{
  rg_ctx* ctx = e->ctx;
  const size_t bytes = sizeof(MovedAtom) * static_cast<size_t>(n > 0 ? n : 1);
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // the staging buffer of the previous call is free again
  if (rg_status st = rg::scratch(ctx, kMovedSlot, bytes, &e->moved)) return st;
  return rg::pinnedScratch(ctx, kMovedPinnedSlot, bytes, &e->moved_host);
}

// The atoms of a full recompute, packed and uploaded piece by piece, so that one piece is on its way while the next is
// packed; mol_end from the molecules' sizes.
rg_status stageFull(rg_ewald* e, const rg_atom* atoms, int n_atoms, const int32_t* molecule_sizes, int n_molecules)
{
  rg_ctx* ctx = e->ctx;
  if (rg_status st = stageRoom(e, n_atoms)) return st;
  MovedAtom* h = static_cast<MovedAtom*>(e->moved_host);
  constexpr int kPiece = 2048;
  int molecule = 0, end = 0;
  for (int base = 0; base < n_atoms; base += kPiece)
  {
    const int n = std::min(kPiece, n_atoms - base);
    packMoved(e, nullptr, 0, atoms + base, n, 1.0, h + base);
    // x * 0 is 0 unless x is NaN or infinite: the test of the inputs costs no pass of its own
    double zero = 0.0;
    for (int i = base; i < base + n; ++i)
    {
      const rg_atom& a = atoms[i];
      zero += ((a.x * 0.0 + a.y * 0.0) + (a.z * 0.0 + a.charge * 0.0)) + (a.scaling_vdw * 0.0 + a.scaling_coulomb * 0.0);
      while (i >= end && molecule < n_molecules) end += molecule_sizes[molecule++];
      h[i].mol_end = i < end ? end : i;
    }
    if (zero != 0.0) return rg::checkFinite(ctx, atoms, n_atoms, "rg_ewald_full");  // names the atom
    RG_CUDA(ctx, cudaMemcpyAsync(static_cast<MovedAtom*>(e->moved) + base, h + base, sizeof(MovedAtom) * n,
                                 cudaMemcpyHostToDevice, ctx->stream));
  }
  return RG_OK;
}

rg_status stageAtoms(rg_ewald* e, const rg_atom* old_atoms, int n_old, const rg_atom* new_atoms, int n_new,
                     double old_sign)
{
  rg_ctx* ctx = e->ctx;
  const int n = n_old + n_new;
  if (rg_status st = stageRoom(e, n)) return st;
  MovedAtom* h = static_cast<MovedAtom*>(e->moved_host);
  packMoved(e, old_atoms, n_old, new_atoms, n_new, old_sign, h);
  if (n > 0) RG_CUDA(ctx, cudaMemcpyAsync(e->moved, h, sizeof(MovedAtom) * n, cudaMemcpyHostToDevice, ctx->stream));
  return RG_OK;
}

template <int G>
cudaError_t launchDelta(rg_ewald* e, int n_moved, const MovedParam* small)
{
  const int kxm = e->ff.kmax_x, kym = e->ff.kmax_y, kzm = e->ff.kmax_z, nk = static_cast<int>(e->nk);
  const size_t per_atom = sizeof(double2) * (kxm + kym + kzm + 3);
  const int tile = std::max(1, std::min({kDeltaTile, n_moved, static_cast<int>(kDeltaShared / per_atom)}));
  ewaldDeltaKernel<G><<<(nk + kThreads - 1) / kThreads, kThreads, per_atom * tile, e->ctx->stream>>>(
      nk, kxm, kym, kzm, e->kvec, e->temp, e->stored, e->trial, small ? nullptr : static_cast<const MovedAtom*>(e->moved),
      small ? *small : MovedParam{}, n_moved, tile, e->partial, e->counter, e->result, ++e->calls);
  return cudaGetLastError();
}

// Pair sums and their finish over the staged atoms, for the framework (rigid) or the adsorbates. A block holds up to
// kPairWarps warps of pairs; the atoms are cut into chunks so that the blocks fill every SM once (as many narrow blocks
// per SM as make up kPairWarps warps), with at least 8 atoms each.
constexpr size_t kPairShared = 98304;  // bytes of tables at most
rg_status launchPairs(rg_ewald* e, int n_atoms, bool rigid, const TermsParams& terms, unsigned call)
{
  cudaStream_t stream = e->ctx->stream;
  const int kxm = e->ff.kmax_x, kym = e->ff.kmax_y, kzm = e->ff.kmax_z;
  // values of m per thread (their 4 MT sums leave room for two blocks per SM): the size that covers 0..kmax_z with the
  // least excess
  constexpr int sizes[3] = {7, 6, 5};
  int mt = sizes[0], covered = 1 << 30;
  for (int q : sizes)
  {
    const int c = (kzm + q) / q * q;
    if (c < covered)
    {
      covered = c;
      mt = q;
    }
  }
  const int m_tiles = covered / mt;
  const int pair_blocks = (e->n_pairs + 32 * kPairWarps - 1) / (32 * kPairWarps);
  const int warps = ((e->n_pairs + pair_blocks - 1) / pair_blocks + 31) / 32;
  const int fill = e->sms * kPairBlocks * std::max(1, kPairWarps / warps);
  const int want = std::max(1, fill / (pair_blocks * m_tiles));
  const int chunk = std::max(8, (n_atoms + want - 1) / want);
  const int n_chunks = std::max(1, (n_atoms + chunk - 1) / chunk);
  const size_t per_atom = sizeof(double2) * ((kxm + 1) + (2 * kym + 1) + mt);
  const int tile = std::max(1, std::min({32, chunk, static_cast<int>(kPairShared / per_atom)}));
  const int64_t total = static_cast<int64_t>(e->n_pairs) * (kzm + 1);
  void* scr = nullptr;
  if (rg_status st = rg::scratch(e->ctx, kSumsSlot, 2 * sizeof(double2) * static_cast<size_t>(n_chunks) * total, &scr))
    return st;
  double2* sums = static_cast<double2*>(scr);
  const MovedAtom* atoms = static_cast<const MovedAtom*>(e->moved);
  if (n_atoms > 0)
  {
    const dim3 grid(pair_blocks, n_chunks, m_tiles);
    const size_t shmem = per_atom * tile;
    // The limit of a kernel's shared memory is the device's, not the context's: always the most that any call takes, so
    // that no host thread lowers it between another's setting and launch.
    auto run = [&](auto kern)
    {
      const cudaError_t err =
          cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kPairShared));
      if (err) return err;
      kern<<<grid, 32 * warps, shmem, stream>>>(e->n_pairs, e->pairs, atoms, n_atoms, chunk, tile, kxm, kym, kzm,
                                                sums);
      return cudaGetLastError();
    };
    RG_CUDA(e->ctx, mt == 7   ? run(ewaldPairSumsKernel<7>)
                    : mt == 6 ? run(ewaldPairSumsKernel<6>)
                              : run(ewaldPairSumsKernel<5>));
  }
  else
    RG_CUDA(e->ctx, cudaMemsetAsync(sums, 0, 2 * sizeof(double2) * total, stream));
  constexpr int kItems = kThreads / kFinishLanes;
  const unsigned blocks = static_cast<unsigned>((total + kItems - 1) / kItems);
  if (rigid)
    ewaldPairFinishKernel<true><<<blocks, kThreads, 0, stream>>>(e->n_pairs, kzm, n_chunks, sums, e->kmap, e->temp,
                                                                e->s_rigid, nullptr, 0, nullptr, nullptr, nullptr, terms,
                                                                call);
  else
    ewaldPairFinishKernel<false><<<blocks + terms.blocks, kThreads, 0, stream>>>(
        e->n_pairs, kzm, n_chunks, sums, e->kmap, e->temp, e->s_rigid, e->stored, e->omit_inter ? 1 : 0,
        e->partial, e->counter, e->result, terms, call);
  RG_CUDA(e->ctx, cudaGetLastError());
  return RG_OK;
}

template <int G>
rg_status launchFull(rg_ewald* e, int n_atoms, unsigned call)
{
  // atoms split into chunks so that k-blocks x chunks fill the GPU (about four CTAs per SM), at least one tile each
  const int blocks = static_cast<int>((e->nk + kThreads - 1) / kThreads);
  const int maxChunks = std::max(1, (n_atoms + kFullTile - 1) / kFullTile);
  const int chunks = std::min(maxChunks, std::max(1, (4 * e->sms + blocks - 1) / blocks));
  const int chunkAtoms = std::max(kFullTile, (((n_atoms + chunks - 1) / chunks + kFullTile - 1) / kFullTile) * kFullTile);
  const int n_chunks = n_atoms > 0 ? (n_atoms + chunkAtoms - 1) / chunkAtoms : 1;
  const size_t need = sizeof(double2) * static_cast<size_t>(n_chunks) * e->nk * (1 + G);
  void* scr = nullptr;
  if (rg_status st = rg::scratch(e->ctx, kSumsSlot, need, &scr)) return st;
  double2* sums = static_cast<double2*>(scr);
  const int stride = (e->ff.kmax_x + 1) + (e->ff.kmax_y + 1) + (e->ff.kmax_z + 1);
  size_t shmem = sizeof(double2) * kFullTile * stride;
  auto kern = ewaldFullPartialKernel<G>;
  constexpr int most = sizeof(double2) * kFullTile * 3 * 128;  // kmax is at most 127; as in launchPairs
  RG_CUDA(e->ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  if (n_atoms > 0)
    kern<<<dim3(blocks, n_chunks), kThreads, shmem, e->ctx->stream>>>(
        e->nk, e->kvec, static_cast<const MovedAtom*>(e->moved), n_atoms, chunkAtoms, e->ff.kmax_x, e->ff.kmax_y,
        e->ff.kmax_z, sums);
  else
    cudaMemsetAsync(sums, 0, need, e->ctx->stream);
  ewaldFullFinishKernel<G><<<blocks, kThreads, 0, e->ctx->stream>>>(e->nk, n_chunks, sums, e->temp, e->s_rigid,
                                                                    e->stored, e->omit_inter ? 1 : 0, e->partial,
                                                                    e->counter, e->result, call);
  RG_CUDA(e->ctx, cudaGetLastError());
  return RG_OK;
}

}  // namespace

extern "C"
{
rg_status rg_ewald_create(rg_ctx* ctx, const rg_forcefield* ff, const rg_box* box, int n_groups, rg_ewald** out)
{
  if (!ctx || !ff || !box || !out) return RG_ERR_INVALID_ARGUMENT;
  if (n_groups < 0 || n_groups > kMaxGroups) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_ewald_create: groups");
  if (ff->kmax_x < 0 || ff->kmax_y < 0 || ff->kmax_z < 0 || ff->kmax_x > 127 || ff->kmax_y > 127 || ff->kmax_z > 127)
    return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_ewald_create: kmax must be in [0, 127]");
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  rg_ewald* e = new rg_ewald();
  e->ctx = ctx;
  e->n_groups = n_groups;
  e->box = rg::makeHostBox(box);
  e->ff = *ff;
  e->ff.epsilon = e->ff.sigma = e->ff.shift = nullptr;
  e->ff.lj = nullptr;
  e->alpha = ff->ewald_alpha;
  e->volume = e->box.volume;
  e->omit_inter = ff->omit_inter != 0;
  e->use_charge = ff->use_charge != 0;
  // k-vector set and prefactors in the reference order (ewald.cpp:1098-1146)
  std::vector<char4> kv;
  std::vector<double> tp;
  const double ax[3] = {e->box.ic[0][0], e->box.ic[1][0], e->box.ic[2][0]};
  const double ay[3] = {e->box.ic[0][1], e->box.ic[1][1], e->box.ic[2][1]};
  const double az[3] = {e->box.ic[0][2], e->box.ic[1][2], e->box.ic[2][2]};
  const double prefactor = rg::coulombFactor() * (2.0 * rg::kPi / e->volume);
  const double alpha_squared = ff->ewald_alpha * ff->ewald_alpha;
  double sum = 0.0;
  for (int kx = 0; kx <= ff->kmax_x; ++kx)
  {
    const double factor = (kx == 0) ? (1.0 * prefactor) : (2.0 * prefactor);
    for (int ky = -ff->kmax_y; ky <= ff->kmax_y; ++ky)
      for (int kz = -ff->kmax_z; kz <= ff->kmax_z; ++kz)
      {
        double kvv[3];
        for (int d = 0; d < 3; ++d)
          kvv[d] = 2.0 * rg::kPi * kx * ax[d] + 2.0 * rg::kPi * ky * ay[d] + 2.0 * rg::kPi * kz * az[d];
        double rksq = kvv[0] * kvv[0] + kvv[1] * kvv[1] + kvv[2] * kvv[2];
        uint64_t ksq = static_cast<uint64_t>(kx * kx + ky * ky + kz * kz);
        if ((ksq != 0) && (ksq <= ff->recip_int_cutoff_sq) && (rksq < ff->recip_cutoff_sq))
        {
          double t = factor * std::exp((-0.25 / alpha_squared) * rksq) / rksq;
          kv.push_back(make_char4(static_cast<signed char>(kx), static_cast<signed char>(ky),
                                  static_cast<signed char>(kz), 0));
          tp.push_back(t);
          sum += t;
        }
      }
  }
  e->nk = static_cast<int64_t>(kv.size());
  e->single_ion_sum = sum;
  const int64_t nk = e->nk > 0 ? e->nk : 1;
  // the (kx, ky) pairs in list order and where each pair's kz are in the list
  const int nz = 2 * ff->kmax_z + 1;
  for (int64_t k = 0; k < e->nk; ++k)
  {
    if (k == 0 || kv[k].x != kv[k - 1].x || kv[k].y != kv[k - 1].y)
    {
      e->pairs_host.push_back(make_char2(kv[k].x, kv[k].y));
      e->kmap_host.resize(e->kmap_host.size() + nz, -1);
    }
    e->kmap_host[e->kmap_host.size() - nz + ff->kmax_z + kv[k].z] = static_cast<int>(k);
  }
  e->n_pairs = static_cast<int>(e->pairs_host.size());
  // blocks that reduce through `partial`: one thread per k-vector, or kFinishLanes per (pair, |kz|)
  const int64_t finish = (static_cast<int64_t>(e->n_pairs) * (ff->kmax_z + 1) * kFinishLanes + kThreads - 1) / kThreads;
  const int64_t blocks = std::max((nk + kThreads - 1) / kThreads, finish);
  auto alloc = [&](void** p, size_t b) { return cudaMalloc(p, b); };
  cudaError_t err = cudaSuccess;
  if (!err) err = alloc(reinterpret_cast<void**>(&e->kvec), sizeof(char4) * nk);
  if (!err) err = alloc(reinterpret_cast<void**>(&e->temp), sizeof(double) * nk);
  if (!err) err = alloc(reinterpret_cast<void**>(&e->s_rigid), sizeof(double2) * nk);
  if (!err) err = alloc(reinterpret_cast<void**>(&e->stored), sizeof(double2) * nk * (1 + n_groups));
  if (!err) err = alloc(reinterpret_cast<void**>(&e->trial), sizeof(double2) * nk * (1 + n_groups));
  if (!err) err = alloc(reinterpret_cast<void**>(&e->partial), sizeof(double) * blocks * (1 + kMaxGroups));
  if (!err) err = alloc(reinterpret_cast<void**>(&e->counter), sizeof(unsigned int) * 4);
  if (!err && e->n_pairs > 0) err = alloc(reinterpret_cast<void**>(&e->pairs), sizeof(char2) * e->n_pairs);
  if (!err && e->n_pairs > 0) err = alloc(reinterpret_cast<void**>(&e->kmap), sizeof(int) * e->kmap_host.size());
  if (!err && e->n_pairs > 0)
    err = cudaMemcpyAsync(e->pairs, e->pairs_host.data(), sizeof(char2) * e->n_pairs, cudaMemcpyHostToDevice, ctx->stream);
  if (!err && e->n_pairs > 0)
    err = cudaMemcpyAsync(e->kmap, e->kmap_host.data(), sizeof(int) * e->kmap_host.size(), cudaMemcpyHostToDevice,
                          ctx->stream);
  if (!err)
    err = cudaHostAlloc(reinterpret_cast<void**>(&e->result_host), sizeof(ulonglong2) * kResults, cudaHostAllocMapped);
  if (!err) err = cudaHostGetDevicePointer(reinterpret_cast<void**>(&e->result), e->result_host, 0);
  if (!err) std::memset(e->result_host, 0, sizeof(ulonglong2) * kResults);
  if (!err) err = cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, ctx->device);
  if (!err && e->nk > 0)
    err = cudaMemcpyAsync(e->kvec, kv.data(), sizeof(char4) * e->nk, cudaMemcpyHostToDevice, ctx->stream);
  if (!err && e->nk > 0)
    err = cudaMemcpyAsync(e->temp, tp.data(), sizeof(double) * e->nk, cudaMemcpyHostToDevice, ctx->stream);
  if (!err) err = cudaMemsetAsync(e->s_rigid, 0, sizeof(double2) * nk, ctx->stream);
  if (!err) err = cudaMemsetAsync(e->stored, 0, sizeof(double2) * nk * (1 + n_groups), ctx->stream);
  if (!err) err = cudaMemsetAsync(e->counter, 0, sizeof(unsigned int) * 4, ctx->stream);
  if (!err) err = cudaStreamSynchronize(ctx->stream);
  if (err)
  {
    rg_status st = rg::cudaFail(ctx, err, "rg_ewald_create");
    rg_ewald_destroy(e);
    return st;
  }
  *out = e;
  return RG_OK;
}

rg_status rg_ewald_destroy(rg_ewald* e)
{
  if (!e) return RG_OK;
  if (e->ctx) cudaStreamSynchronize(e->ctx->stream);
  cudaFree(e->kvec);
  cudaFree(e->temp);
  cudaFree(e->s_rigid);
  cudaFree(e->stored);
  cudaFree(e->trial);
  cudaFree(e->partial);
  cudaFree(e->counter);
  cudaFree(e->pairs);
  cudaFree(e->kmap);
  if (e->result_host) cudaFreeHost(e->result_host);
  delete e;
  return RG_OK;
}

rg_status rg_ewald_info(rg_ewald* e, int64_t* n_kvectors, double* single_ion_sum)
{
  if (!e) return RG_ERR_INVALID_ARGUMENT;
  if (n_kvectors) *n_kvectors = e->nk;
  if (single_ion_sum) *single_ion_sum = e->single_ion_sum;
  return RG_OK;
}

rg_status rg_ewald_set_framework(rg_ewald* e, const rg_atom* fw, int n_fw)
{
  if (!e || (n_fw > 0 && !fw) || n_fw < 0) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = e->ctx;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  if (n_fw == 0 || e->nk == 0)
  {
    RG_CUDA(ctx, cudaMemsetAsync(e->s_rigid, 0, sizeof(double2) * (e->nk > 0 ? e->nk : 1), ctx->stream));
    return RG_OK;
  }
  rg_status st = stageAtoms(e, fw, n_fw, nullptr, 0, 1.0);
  if (st) return st;
  st = launchPairs(e, n_fw, true, TermsParams{}, 0u);
  if (st) return st;
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return RG_OK;
}

rg_status rg_ewald_full(rg_ewald* e, const rg_atom* atoms, int n_atoms, const int32_t* molecule_sizes, int n_molecules,
                        double net_charge_framework, rg_ewald_energy* out)
{
  if (!e || !out || (n_atoms > 0 && !atoms) || n_atoms < 0 || (n_molecules > 0 && !molecule_sizes))
    return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = e->ctx;
  std::memset(out, 0, sizeof(rg_ewald_energy));
  if (!e->use_charge) return rg::checkFinite(ctx, atoms, n_atoms, "rg_ewald_full");
  if (!e->omit_inter)
  {
    int64_t total = 0;
    bool bad = false;
    for (int m = 0; m < n_molecules; ++m)
    {
      bad = bad || molecule_sizes[m] < 0;
      total += molecule_sizes[m];
    }
    if (bad || total > n_atoms)
    {
      if (rg_status fs = rg::checkFinite(ctx, atoms, n_atoms, "rg_ewald_full")) return fs;
      return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_ewald_full: molecule sizes");
    }
  }
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  const int G = e->n_groups;
  const bool host_terms = hostTermsOf(e, n_atoms, molecule_sizes, n_molecules);
  if (e->nk == 0 && host_terms)
  {
    if (rg_status st = rg::checkFinite(ctx, atoms, n_atoms, "rg_ewald_full")) return st;
  }
  else if (rg_status st = stageFull(e, atoms, n_atoms, molecule_sizes, e->omit_inter ? 0 : n_molecules))
    return st;
  const double C = rg::coulombFactor();
  const double alpha = e->alpha;
  // self, exclusion and net-charge sums: on the device beside the Fourier sums, or, for a few atoms, on the host while
  // the kernels are in flight
  TermsParams tp{};
  tp.atoms = static_cast<const MovedAtom*>(e->moved);
  tp.n_atoms = n_atoms;
  tp.blocks = host_terms ? 0 : (n_atoms + kThreads - 1) / kThreads;
  void* scr = nullptr;
  if (rg_status st = rg::scratch(ctx, kTermsSlot, sizeof(double) * kTerms * static_cast<size_t>(std::max(1, tp.blocks)), &scr))
    return st;
  tp.partial = static_cast<double*>(scr);
  tp.counter = e->counter + 1;
  tp.result = e->result + kTermsAt;
  for (int c = 0; c < 3; ++c)
    for (int r = 0; r < 3; ++r) tp.cell[3 * c + r] = e->box.c[c][r];
  tp.triclinic = e->box.triclinic ? 1 : 0;
  tp.alpha = alpha;
  tp.coul = C;
  tp.self = C * alpha / std::sqrt(rg::kPi);
  const unsigned call = ++e->calls;
  if (e->nk > 0)
  {
    rg_status st;
    switch (G)
    {
      case 0: st = launchPairs(e, n_atoms, false, tp, call); break;
      case 1: st = launchFull<1>(e, n_atoms, call); break;
      case 2: st = launchFull<2>(e, n_atoms, call); break;
      case 3: st = launchFull<3>(e, n_atoms, call); break;
      default: st = launchFull<4>(e, n_atoms, call); break;
    }
    if (st) return st;
  }
  if (tp.blocks > 0 && (e->nk == 0 || G > 0))
  {
    ewaldAtomTermsKernel<<<tp.blocks, kThreads, 0, ctx->stream>>>(tp, e->omit_inter ? 1 : 0, call);
    RG_CUDA(ctx, cudaGetLastError());
  }
  if (e->nk > 0 || tp.blocks > 0)
    if (rg_status st = rg::leave(ctx)) return st;
  double own[kTerms] = {};
  if (host_terms) hostTerms(e, atoms, n_atoms, molecule_sizes, n_molecules, own);
  double all[kTermsAt + kTerms] = {};
  if (e->nk > 0)
    if (rg_status st = rg::collect(ctx, e->result_host, 1 + G, call, all, "rg_ewald_full")) return st;
  if (tp.blocks > 0)
    if (rg_status st = rg::collect(ctx, e->result_host + kTermsAt, kTerms, call, all + kTermsAt, "rg_ewald_full")) return st;
  const double* res = all;
  const double* terms = host_terms ? own : all + kTermsAt;
  out->ewald_self = terms[0];
  out->ewald_exclusion = terms[1];
  for (int g = 0; g < 4; ++g) out->dudlambda_ewald[g] = terms[3 + g];
  const double netChargeAdsorbates = terms[2];
  const double* netChargeDerivative = terms + 7;
  const double uIon = -(e->single_ion_sum - C * alpha / std::sqrt(rg::kPi));
  double netFourier = 0.0, netDudl[4] = {0, 0, 0, 0};
  if (e->omit_inter)
  {
    netFourier = 2.0 * uIon * net_charge_framework * netChargeAdsorbates;
    for (int g = 0; g < 4; ++g) netDudl[g] = 2.0 * uIon * net_charge_framework * netChargeDerivative[g];
  }
  else
  {
    netFourier = uIon * (2.0 * net_charge_framework + netChargeAdsorbates) * netChargeAdsorbates;
    for (int g = 0; g < 4; ++g)
      netDudl[g] = 2.0 * uIon * (net_charge_framework + netChargeAdsorbates) * netChargeDerivative[g];
  }
  out->ewald_fourier = (e->nk > 0 ? res[0] : 0.0) + netFourier;
  for (int g = 0; g < G && e->nk > 0; ++g) out->dudlambda_ewald[g] += res[1 + g];
  for (int g = 0; g < 4; ++g) out->dudlambda_ewald[g] += netDudl[g];
  return RG_OK;
}

rg_status rg_ewald_delta(rg_ewald* e, const rg_atom* new_atoms, int n_new, const rg_atom* old_atoms, int n_old,
                         double net_charge, const double* net_charge_derivative_ext, rg_ewald_energy* out)
{
  if (!e || !out || n_new < 0 || n_old < 0 || (n_new > 0 && !new_atoms) || (n_old > 0 && !old_atoms))
    return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = e->ctx;
  std::memset(out, 0, sizeof(rg_ewald_energy));
  if (rg_status fs = rg::checkFinite(ctx, new_atoms, n_new, "rg_ewald_delta")) return fs;
  if (rg_status fs = rg::checkFinite(ctx, old_atoms, n_old, "rg_ewald_delta")) return fs;
  if (!e->use_charge) return RG_OK;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  const int G = e->n_groups;
  const int n = n_old + n_new;
  if (n > kMaxMoved) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_ewald_delta: at most 512 old + new atoms");
  double res[1 + kMaxGroups] = {0, 0, 0, 0, 0};
  if (e->nk > 0)
  {
    MovedParam small{};
    const bool inParams = n <= kParamMoved;
    if (inParams)
      packMoved(e, old_atoms, n_old, new_atoms, n_new, -1.0, small.a);
    else
    {
      rg_status st = stageAtoms(e, old_atoms, n_old, new_atoms, n_new, -1.0);
      if (st) return st;
    }
    const MovedParam* sp = inParams ? &small : nullptr;
    cudaError_t err;
    switch (G)
    {
      case 0: err = launchDelta<0>(e, n, sp); break;
      case 1: err = launchDelta<1>(e, n, sp); break;
      case 2: err = launchDelta<2>(e, n, sp); break;
      case 3: err = launchDelta<3>(e, n, sp); break;
      default: err = launchDelta<4>(e, n, sp); break;
    }
    if (err) return rg::cudaFail(ctx, err, "ewaldDeltaKernel");
    if (rg_status st = rg::leave(ctx)) return st;
  }
  // the moved atoms' own terms, while the kernel is in flight
  const double C = rg::coulombFactor();
  const double alpha = e->alpha;
  // intramolecular exclusion (ewald.cpp:1164-1219): old +, new -; pairs matched on moleculeId
  auto exclusion = [&](const rg_atom* atoms, int count, double sign)
  {
    for (int i = 0; i < count; ++i)
      for (int j = i + 1; j < count; ++j)
      {
        if (atoms[i].molecule_id != atoms[j].molecule_id) continue;
        double dr[3] = {atoms[i].x - atoms[j].x, atoms[i].y - atoms[j].y, atoms[i].z - atoms[j].z};
        roundHalfAwayPbc(e->box, dr);
        const double r = std::sqrt(dr[0] * dr[0] + dr[1] * dr[1] + dr[2] * dr[2]);
        const double sA = atoms[i].scaling_coulomb, sB = atoms[j].scaling_coulomb;
        double pot, dudl;
        exclusionFactors(alpha, sA * sB, r, pot, dudl);
        const double prefactor = C * atoms[i].charge * atoms[j].charge;
        out->ewald_exclusion += sign * sA * sB * prefactor * pot;
        addDud(out->dudlambda_ewald, groupOf(atoms[i]), groupOf(atoms[j]), sA, sB, sign * prefactor * dudl);
      }
  };
  exclusion(old_atoms, n_old, 1.0);
  exclusion(new_atoms, n_new, -1.0);
  // self energy (ewald.cpp:1221-1238)
  const double prefactor_self = C * alpha / std::sqrt(rg::kPi);
  for (int i = 0; i < n_old; ++i)
  {
    const double q = old_atoms[i].charge, sc = old_atoms[i].scaling_coulomb;
    const int g = groupOf(old_atoms[i]);
    out->ewald_self += prefactor_self * sc * q * sc * q;
    if (g != 0) out->dudlambda_ewald[g - 1] += 2.0 * prefactor_self * sc * q * q;
  }
  for (int i = 0; i < n_new; ++i)
  {
    const double q = new_atoms[i].charge, sc = new_atoms[i].scaling_coulomb;
    const int g = groupOf(new_atoms[i]);
    out->ewald_self -= prefactor_self * sc * q * sc * q;
    if (g != 0) out->dudlambda_ewald[g - 1] -= 2.0 * prefactor_self * sc * q * q;
  }
  // net-charge correction difference (ewald.cpp:181-208)
  double deltaCharge = 0.0, dNew[4], dOld[4];
  for (int g = 0; g < 4; ++g) dNew[g] = dOld[g] = net_charge_derivative_ext ? net_charge_derivative_ext[g] : 0.0;
  for (int i = 0; i < n_old; ++i)
  {
    deltaCharge -= old_atoms[i].scaling_coulomb * old_atoms[i].charge;
    const int g = groupOf(old_atoms[i]);
    if (g != 0) dOld[g - 1] += old_atoms[i].charge;
  }
  for (int i = 0; i < n_new; ++i)
  {
    deltaCharge += new_atoms[i].scaling_coulomb * new_atoms[i].charge;
    const int g = groupOf(new_atoms[i]);
    if (g != 0) dNew[g - 1] += new_atoms[i].charge;
  }
  const double uIon = -(e->single_ion_sum - C * alpha / std::sqrt(rg::kPi));
  const double netChargeNew = net_charge + deltaCharge;
  out->ewald_fourier = uIon * (netChargeNew * netChargeNew - net_charge * net_charge);
  for (int g = 0; g < 4; ++g) out->dudlambda_ewald[g] += 2.0 * uIon * (netChargeNew * dNew[g] - net_charge * dOld[g]);
  if (e->nk > 0)
  {
    const int blocks = static_cast<int>((e->nk + kThreads - 1) / kThreads), posts = blocks <= kDeltaPosted ? blocks : 1;
    double sums[kDeltaPosted * (1 + kMaxGroups)];
    rg_status st = rg::collect(ctx, e->result_host, posts * (1 + G), e->calls, sums, "rg_ewald_delta");
    if (st) return st;
    for (int b = 0; b < posts; ++b)
      for (int c = 0; c < 1 + G; ++c) res[c] += sums[b * (1 + G) + c];
  }
  out->ewald_fourier += res[0];
  for (int g = 0; g < G; ++g) out->dudlambda_ewald[g] += res[1 + g];
  return RG_OK;
}

rg_status rg_ewald_accept(rg_ewald* e)
{
  if (!e) return RG_ERR_INVALID_ARGUMENT;
  if (!e->use_charge) return RG_OK;
  // acceptEwaldMove (ewald.cpp:1565-1574): storedEik = trialEik, done as a pointer swap
  double2* t = e->stored;
  e->stored = e->trial;
  e->trial = t;
  return RG_OK;
}

rg_status rg_ewald_get_structure_factors(rg_ewald* e, int which, double* host, int64_t n_doubles)
{
  if (!e || !host) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = e->ctx;
  const int64_t need = 2 * e->nk * (1 + e->n_groups);
  if (n_doubles < need) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_ewald_get_structure_factors: buffer too small");
  const double2* src = which == 0 ? e->stored : (which == 1 ? e->trial : e->s_rigid);
  const int64_t cnt = which == 2 ? 2 * e->nk : need;
  RG_CUDA(ctx, cudaMemcpyAsync(host, src, sizeof(double) * cnt, cudaMemcpyDeviceToHost, ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return RG_OK;
}

rg_status rg_ewald_set_structure_factors(rg_ewald* e, const double* host, int64_t n_doubles)
{
  if (!e || !host) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = e->ctx;
  const int64_t need = 2 * e->nk * (1 + e->n_groups);
  if (n_doubles != need) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_ewald_set_structure_factors: size");
  RG_CUDA(ctx, cudaMemcpyAsync(e->stored, host, sizeof(double) * need, cudaMemcpyHostToDevice, ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return RG_OK;
}
}

namespace rgd
{
rg_status ewaldExport(rg_ewald* e, const char4** kvec, const double** temp, const double2** s_rigid, int64_t* nk,
                      int kmax[3], double* alpha, double* single_ion_sum)
{
  if (!e) return RG_ERR_INVALID_ARGUMENT;
  *kvec = e->kvec;
  *temp = e->temp;
  *s_rigid = e->s_rigid;
  *nk = e->nk;
  kmax[0] = e->ff.kmax_x;
  kmax[1] = e->ff.kmax_y;
  kmax[2] = e->ff.kmax_z;
  *alpha = e->alpha;
  *single_ion_sum = e->single_ion_sum;
  return RG_OK;
}

cudaError_t ewaldRunPrefactors(const rg_ewald* e, const std::vector<int4>& runs, std::vector<double>& out)
{
  std::vector<double> temp(static_cast<size_t>(e->nk));
  out.assign(2 * static_cast<size_t>(e->ff.kmax_z + 1) * runs.size(), 0.0);
  if (e->nk == 0) return cudaSuccess;
  cudaError_t err =
      cudaMemcpyAsync(temp.data(), e->temp, sizeof(double) * temp.size(), cudaMemcpyDeviceToHost, e->ctx->stream);
  if (!err) err = cudaStreamSynchronize(e->ctx->stream);
  for (size_t r = 0; r < runs.size() && !err; ++r)
  {
    const int lo = static_cast<short>(runs[r].w & 0xffff), hi = runs[r].w >> 16;
    for (int kz = lo; kz <= hi; ++kz)
      out[(2 * static_cast<size_t>(std::abs(kz)) + (kz < 0 ? 1 : 0)) * runs.size() + r] =
          temp[static_cast<size_t>(runs[r].z + kz - lo)];
  }
  return err;
}

std::vector<int4> ewaldRuns(const rg_ewald* e)
{
  std::vector<int4> runs;
  const int nz = 2 * e->ff.kmax_z + 1;
  for (int pr = 0; pr < e->n_pairs; ++pr)
  {
    const int* map = e->kmap_host.data() + static_cast<size_t>(pr) * nz;
    for (int z0 = 0; z0 < nz;)
    {
      if (map[z0] < 0)
      {
        ++z0;
        continue;
      }
      int z1 = z0;
      while (z1 + 1 < nz && map[z1 + 1] == map[z1] + 1) ++z1;
      const int lo = z0 - e->ff.kmax_z, hi = z1 - e->ff.kmax_z;
      runs.push_back(make_int4(e->pairs_host[pr].x, e->pairs_host[pr].y, map[z0],
                               static_cast<int>((static_cast<unsigned>(hi) << 16) | (static_cast<unsigned>(lo) & 0xffffu))));
      z0 = z1 + 1;
    }
  }
  auto reach = [](const int4& r) { return std::max(-static_cast<int>(static_cast<short>(r.w & 0xffff)), r.w >> 16); };
  std::stable_sort(runs.begin(), runs.end(), [&](const int4& x, const int4& y) { return reach(x) > reach(y); });
  return runs;
}
}  // namespace rgd

// ---------------------------------------------------------------------------------------------------------------------
// The structure-factor update of many systems in one launch (the Fourier part of energyDifferenceEwaldFourier,
// ewald.cpp:1098-1162, for one move in each of n systems that share the box, the force field and the k-vectors).
//
// Each system keeps two structure-factor buffers, stored and trial, and a flag says which is which; an accepted move
// flips its system's flag (acceptEwaldMove, ewald.cpp:1565-1574, without a copy). The launch is (k-range, system). The
// traffic per system and move is 32 bytes per k-vector (read S, write the trial S); k-vectors and prefactors are shared
// by all systems and stay in L2.
// ---------------------------------------------------------------------------------------------------------------------
struct rg_ewald_batch
{
  rg_ewald* ewald = nullptr;
  rg_ctx* ctx = nullptr;  // of the Ewald state, which may be gone when the batch is destroyed
  int n = 0;
  // [2][n][slots]: S(k) by rows of (|kz|, sign), a row holding the k-vectors of that kz of all runs side by side, so that
  // neighbouring threads, which take neighbouring runs, read and write neighbouring numbers
  double2* sk = nullptr;
  int64_t slots = 0;
  int* slot_of = nullptr;          // [nk]: where each k-vector is
  int* row_start = nullptr;        // [2 (kmax_z + 1)]
  std::vector<unsigned char> cur;  // [n]: which buffer holds the stored S(k) of system s
  // the moved atoms (fractional coordinates and signed charge), their counts and the buffer flags of one call: one
  // block of memory on the device and one pinned on the host, so that a call uploads it in one copy
  unsigned char* upload = nullptr;
  unsigned char* upload_host = nullptr;
  double* partial = nullptr;       // [n][blocks]
  double* result = nullptr;        // device view of result_host
  double* result_host = nullptr;   // [n] mapped pinned
  int blocks = 0;                  // blocks per system
  int n_runs = 0;
  double* run_temp = nullptr;      // prefactor of kz = +m, -m of run r at [(2 m + (sign < 0)) n_runs + r]
  int4* runs = nullptr;            // runs of consecutive kz of one (kx, ky), longest first (rgd::ewaldRuns)
  // device time of the last rg_ewald_batch_delta: events before the atom upload, before and after the kernel
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  float upload_ms = 0.0f, kernel_ms = 0.0f;
};

namespace
{
constexpr int kBatchAtoms = 16;   // old + new atoms of one system's move
constexpr int kBatchM = 2;        // consecutive |kz| of one thread (five spill at three blocks per SM)

// The upload of one call: n * stride atoms, n counts, n flags
inline size_t batchUploadBytes(int n, int stride)
{
  return sizeof(double4) * static_cast<size_t>(n) * stride + (sizeof(int) + 1) * static_cast<size_t>(n);
}

// Shared memory of a block: the phasors exp(2 pi i m s_d) of its system's moved atoms (x: m = 0..kmax_x with the atom's
// weight, y: m = -kmax_y..kmax_y, z: m = 0..kmax_z).
__host__ __device__ inline size_t batchSharedBytes(int stride, int kxm, int kym, int kzm)
{
  return sizeof(double2) * static_cast<size_t>(stride) * ((kxm + 1) + (2 * kym + 1) + (kzm + 1));
}

// Blocks (part, system). An item is one run of kz of a (kx, ky) and kBatchM values of m = |kz|; block `part` of a system
// takes every gridDim.x-th group of kThreads items. With P = w e^{2 pi i (kx s_x + ky s_y)} = (p, q) and
// (c, s) = e^{2 pi i m s_z} the sums over the atoms of p c, q s, p s and q c give Delta rho at both kz = m and kz = -m,
// four FMAs for two k-vectors, and every z phasor is read by a whole warp at once. S(k) goes straight from HBM to the
// thread that adds to it and back (rows by kz, see rg_ewald_batch): the bound is HBM, 32 bytes per k-vector. Before, a
// thread took one k-vector at a time in list order and read two phasors per atom and k-vector from shared memory, whose
// bandwidth bound it: 114 us for 1,184 systems of 8,124 k-vectors. With four |kz| per thread, whose sums came before the
// loads of S, three blocks fitted on an SM: 88 us. With two, S loaded first, four blocks fit: 73 us, and 79 with the
// kernel behind it that adds the blocks' energies (47 us at the measured copy rate, were all of S read and all of the trial
// S written through HBM).
__global__ void __launch_bounds__(kThreads, 4) ewaldBatchDeltaKernel(
    const int4* __restrict__ runs, int n_runs, const int* __restrict__ row_start, int64_t slots, int n_systems,
    const double* __restrict__ run_temp, double2* sk, const unsigned char* __restrict__ upload, int atom_stride, int kxm,
    int kym, int kzm, double* partial)
{
  extern __shared__ double2 tab[];
  __shared__ double red[kThreads / 32];
  const int sys = blockIdx.y;
  const double4* atoms = reinterpret_cast<const double4*>(upload) + static_cast<int64_t>(sys) * atom_stride;
  const int* counts = reinterpret_cast<const int*>(reinterpret_cast<const double4*>(upload) +
                                                   static_cast<int64_t>(n_systems) * atom_stride);
  const int cur = reinterpret_cast<const unsigned char*>(counts + n_systems)[sys];
  const int na = counts[sys];
  const double2* S = sk + (static_cast<int64_t>(cur) * n_systems + sys) * slots;
  double2* T = sk + (static_cast<int64_t>(1 - cur) * n_systems + sys) * slots;
  const int nx = kxm + 1, ny = 2 * kym + 1, nz = kzm + 1;
  double2* ex = tab;
  double2* ey = ex + atom_stride * nx;
  double2* ez = ey + atom_stride * ny;
  const int per = nx + (kym + 1) + nz;
  for (int idx = threadIdx.x; idx < na * per; idx += kThreads)
  {
    const int a = idx / per, m = idx - a * per;
    const double4 at = atoms[a];
    const int dim = m < nx ? 0 : (m < nx + kym + 1 ? 1 : 2);
    const int mm = dim == 0 ? m : (dim == 1 ? m - nx : m - nx - (kym + 1));
    double sn, cs;
    sincospi(2.0 * static_cast<double>(mm) * (dim == 0 ? at.x : (dim == 1 ? at.y : at.z)), &sn, &cs);
    if (dim == 0)
      ex[a * nx + mm] = make_double2(at.w * cs, at.w * sn);
    else if (dim == 1)
    {
      ey[a * ny + kym + mm] = make_double2(cs, sn);
      ey[a * ny + kym - mm] = make_double2(cs, -sn);
    }
    else
      ez[a * nz + mm] = make_double2(cs, sn);
  }
  __syncthreads();
  const int groups = (nz + kBatchM - 1) / kBatchM;
  double e = 0.0;
  for (int item = blockIdx.x * kThreads + threadIdx.x; item < n_runs * groups; item += gridDim.x * kThreads)
  {
    const int g = item / n_runs, r = item - g * n_runs, m0 = g * kBatchM;
    const int4 run = runs[r];
    const int lo = static_cast<short>(run.w & 0xffff), hi = run.w >> 16;
    if (m0 > max(-lo, hi)) continue;
    // S(k) first: its loads are in flight while the sums are formed
    double2 sk[2][kBatchM];
    int at[2][kBatchM];
#pragma unroll
    for (int sign = 0; sign < 2; ++sign)
#pragma unroll
      for (int m = 0; m < kBatchM; ++m)
      {
        const int kz = sign == 0 ? m0 + m : -(m0 + m);
        const bool in = kz >= lo && kz <= hi && (sign == 0 || kz != 0);
        at[sign][m] = in ? row_start[2 * (m0 + m) + sign] + r : -1;
        sk[sign][m] = in ? __ldcs(S + at[sign][m]) : make_double2(0.0, 0.0);
      }
    double pc[kBatchM], qs[kBatchM], ps[kBatchM], qc[kBatchM];
#pragma unroll
    for (int m = 0; m < kBatchM; ++m) pc[m] = qs[m] = ps[m] = qc[m] = 0.0;
#pragma unroll 1
    for (int a = 0; a < na; ++a)
    {
      const double2 x = ex[a * nx + run.x], y = ey[a * ny + kym + run.y];
      const double p = x.x * y.x - x.y * y.y, q = x.x * y.y + x.y * y.x;
#pragma unroll
      for (int m = 0; m < kBatchM; ++m)
      {
        const double2 z = ez[a * nz + min(m0 + m, kzm)];
        pc[m] = fma(p, z.x, pc[m]);
        qs[m] = fma(q, z.y, qs[m]);
        ps[m] = fma(p, z.y, ps[m]);
        qc[m] = fma(q, z.x, qc[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < kBatchM; ++m)
    {
      // Delta rho at kz = +m in (u, v), at kz = -m in (w, z)
      const double u = pc[m] - qs[m], v = ps[m] + qc[m], w = pc[m] + qs[m], z = qc[m] - ps[m];
      pc[m] = u;
      ps[m] = v;
      qs[m] = w;
      qc[m] = z;
    }
#pragma unroll
    for (int sign = 0; sign < 2; ++sign)
    {
#pragma unroll
      for (int m = 0; m < kBatchM; ++m)
        if (at[sign][m] >= 0)
        {
          const double dx = sign == 0 ? pc[m] : qs[m], dy = sign == 0 ? ps[m] : qc[m];
          e += run_temp[(2 * (m0 + m) + sign) * n_runs + r] * (2.0 * (sk[sign][m].x * dx + sk[sign][m].y * dy) + (dx * dx + dy * dy));
          __stcs(T + at[sign][m], make_double2(sk[sign][m].x + dx, sk[sign][m].y + dy));
        }
    }
  }
  // fixed-order reduction: warps, then the block; ewaldBatchTotalKernel adds the blocks. (A last block per system, found
  // with a counter, kept every block until its fence and its atomic had returned.)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if (lane == 0) red[warp] = e;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    double x = 0.0;
    for (int q = 0; q < kThreads / 32; ++q) x += red[q];
    partial[static_cast<long long>(sys) * gridDim.x + blockIdx.x] = x;
  }
}

// S(k) of one system between list order (k * stride) and its slots
__global__ void __launch_bounds__(kThreads) ewaldBatchPermuteKernel(int64_t nk, const int* __restrict__ slot_of,
                                                                    double2* list, int64_t stride, double2* slots,
                                                                    int to_slots)
{
  const int64_t k = static_cast<int64_t>(blockIdx.x) * kThreads + threadIdx.x;
  if (k >= nk) return;
  if (to_slots)
    slots[slot_of[k]] = list[k * stride];
  else
    list[k * stride] = slots[slot_of[k]];
}

// The blocks' energies of each system added in block order, into mapped host memory
__global__ void __launch_bounds__(kThreads) ewaldBatchTotalKernel(int n, int blocks, const double* __restrict__ partial,
                                                                  double* result)
{
  const int sys = blockIdx.x * kThreads + threadIdx.x;
  if (sys >= n) return;
  double x = 0.0;
  for (int b = 0; b < blocks; ++b) x += partial[static_cast<long long>(sys) * blocks + b];
  result[sys] = x;
}
}  // namespace

extern "C"
{
rg_status rg_ewald_batch_create(rg_ewald* e, int n_systems, rg_ewald_batch** out)
{
  if (!e || !out || n_systems < 1 || n_systems > 65535) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = e->ctx;
  if (e->n_groups != 0)
    return rg::fail(ctx, RG_ERR_UNSUPPORTED, "rg_ewald_batch_create: the batch carries no dU/dlambda groups");
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  rg_ewald_batch* b = new rg_ewald_batch();
  b->ewald = e;
  b->ctx = e->ctx;
  b->n = n_systems;
  const int64_t nk = std::max<int64_t>(1, e->nk);
  // the runs come longest first, so that the rows of large |kz| hold the first runs only
  std::vector<int4> runs = rgd::ewaldRuns(e);
  const int rows = 2 * (e->ff.kmax_z + 1);
  std::vector<int> row_start(rows, 0), row_len(rows, 0), slot_of(static_cast<size_t>(nk), 0);
  for (int pass = 0; pass < 2; ++pass)
  {
    for (size_t r = 0; r < runs.size(); ++r)
    {
      const int lo = static_cast<short>(runs[r].w & 0xffff), hi = runs[r].w >> 16;
      for (int kz = lo; kz <= hi; ++kz)
      {
        const int row = 2 * std::abs(kz) + (kz < 0 ? 1 : 0);
        if (pass == 0)
          row_len[row] = static_cast<int>(r) + 1;
        else
          slot_of[static_cast<size_t>(runs[r].z + kz - lo)] = row_start[row] + static_cast<int>(r);
      }
    }
    if (pass == 0)
    {
      for (int row = 1; row < rows; ++row) row_start[row] = row_start[row - 1] + row_len[row - 1];
      b->slots = std::max(1, row_start[rows - 1] + row_len[rows - 1]);
    }
  }
  if (runs.empty()) runs.push_back(make_int4(0, 0, 0, 0));
  b->n_runs = static_cast<int>(runs.size());
  std::vector<double> run_temp;
  cudaError_t err = rgd::ewaldRunPrefactors(e, runs, run_temp);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&b->run_temp), sizeof(double) * run_temp.size());
  if (!err)
    err = cudaMemcpyAsync(b->run_temp, run_temp.data(), sizeof(double) * run_temp.size(), cudaMemcpyHostToDevice, ctx->stream);
  // Blocks per system: as many as there are groups of kThreads items when the systems are few; for many systems fewer, so
  // that a block's phasor tables serve more k-vectors (four blocks per place on the GPU remain: 1,184 systems of 3,609 and
  // of 8,124 k-vectors take 40.4 and 72.8 us, with six 44.5 and 73.2; 700 systems 31.8 and 50.3, with two 34.1 and 60.6)
  const int64_t items = static_cast<int64_t>(b->n_runs) * ((e->ff.kmax_z + kBatchM) / kBatchM);
  const int64_t most = std::max<int64_t>(1, (items + kThreads - 1) / kThreads);
  b->blocks = static_cast<int>(std::min<int64_t>(most, std::max<int64_t>(1, 16LL * e->sms / n_systems)));
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&b->slot_of), sizeof(int) * slot_of.size());
  if (!err) err = cudaMemcpyAsync(b->slot_of, slot_of.data(), sizeof(int) * slot_of.size(), cudaMemcpyHostToDevice, ctx->stream);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&b->row_start), sizeof(int) * rows);
  if (!err) err = cudaMemcpyAsync(b->row_start, row_start.data(), sizeof(int) * rows, cudaMemcpyHostToDevice, ctx->stream);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&b->runs), sizeof(int4) * runs.size());
  if (!err) err = cudaMemcpyAsync(b->runs, runs.data(), sizeof(int4) * runs.size(), cudaMemcpyHostToDevice, ctx->stream);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&b->sk), sizeof(double2) * 2 * n_systems * b->slots);
  if (!err) err = cudaMemsetAsync(b->sk, 0, sizeof(double2) * 2 * n_systems * b->slots, ctx->stream);
  const size_t upload = batchUploadBytes(n_systems, kBatchAtoms);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&b->upload), upload);
  if (!err) err = cudaMallocHost(reinterpret_cast<void**>(&b->upload_host), upload);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&b->partial), sizeof(double) * n_systems * b->blocks);
  if (!err) err = cudaHostAlloc(reinterpret_cast<void**>(&b->result_host), sizeof(double) * n_systems, cudaHostAllocMapped);
  if (!err) err = cudaHostGetDevicePointer(reinterpret_cast<void**>(&b->result), b->result_host, 0);
  for (int i = 0; i < 3 && !err; ++i) err = cudaEventCreate(&b->ev[i]);
  if (!err) err = cudaStreamSynchronize(ctx->stream);
  if (err)
  {
    rg_status st = rg::cudaFail(ctx, err, "rg_ewald_batch_create");
    rg_ewald_batch_destroy(b);
    return st;
  }
  b->cur.assign(n_systems, 0);
  *out = b;
  return RG_OK;
}

rg_status rg_ewald_batch_destroy(rg_ewald_batch* b)
{
  if (!b) return RG_OK;
  if (b->ctx) cudaStreamSynchronize(b->ctx->stream);
  cudaFree(b->sk);
  cudaFree(b->upload);
  cudaFree(b->partial);
  cudaFree(b->slot_of);
  cudaFree(b->row_start);
  cudaFree(b->runs);
  cudaFree(b->run_temp);
  if (b->upload_host) cudaFreeHost(b->upload_host);
  if (b->result_host) cudaFreeHost(b->result_host);
  for (cudaEvent_t ev : b->ev)
    if (ev) cudaEventDestroy(ev);
  delete b;
  return RG_OK;
}

rg_status rg_ewald_batch_set(rg_ewald_batch* b, int system, const double* sk)
{
  if (!b || system < 0 || system >= b->n) return RG_ERR_INVALID_ARGUMENT;
  rg_ewald* e = b->ewald;
  rg_ctx* ctx = e->ctx;
  if (e->nk == 0) return RG_OK;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  double2* dst = b->sk + (static_cast<long long>(b->cur[system]) * b->n + system) * b->slots;
  double2* list = e->stored;  // entry 0 of each k
  if (sk)
  {
    for (int64_t i = 0; i < 2 * e->nk; ++i)
      if (!std::isfinite(sk[i])) return rg::fail(ctx, RG_ERR_NONFINITE, "rg_ewald_batch_set: NaN or infinite S(k)");
    void* scr = nullptr;
    if (rg_status st = rg::scratch(ctx, kSumsSlot, sizeof(double2) * e->nk, &scr)) return st;
    list = static_cast<double2*>(scr);
    RG_CUDA(ctx, cudaMemcpyAsync(list, sk, sizeof(double2) * e->nk, cudaMemcpyHostToDevice, ctx->stream));
  }
  ewaldBatchPermuteKernel<<<static_cast<unsigned>((e->nk + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(
      e->nk, b->slot_of, list, sk ? 1 : 1 + e->n_groups, dst, 1);
  RG_CUDA(ctx, cudaGetLastError());
  if (!sk) return rg::leave(ctx);
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));  // the caller's buffer may be pinned
  return RG_OK;
}

rg_status rg_ewald_batch_get(rg_ewald_batch* b, int system, int which, double* sk)
{
  if (!b || !sk || system < 0 || system >= b->n || (which != 0 && which != 1)) return RG_ERR_INVALID_ARGUMENT;
  rg_ewald* e = b->ewald;
  rg_ctx* ctx = e->ctx;
  if (e->nk == 0) return RG_OK;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  const int buf = which == 0 ? b->cur[system] : 1 - b->cur[system];
  void* scr = nullptr;
  if (rg_status st = rg::scratch(ctx, kSumsSlot, sizeof(double2) * e->nk, &scr)) return st;
  double2* list = static_cast<double2*>(scr);
  ewaldBatchPermuteKernel<<<static_cast<unsigned>((e->nk + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(
      e->nk, b->slot_of, list, 1, b->sk + (static_cast<long long>(buf) * b->n + system) * b->slots, 0);
  RG_CUDA(ctx, cudaGetLastError());
  RG_CUDA(ctx, cudaMemcpyAsync(sk, list, sizeof(double2) * e->nk, cudaMemcpyDeviceToHost, ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return RG_OK;
}

rg_status rg_ewald_batch_delta(rg_ewald_batch* b, const rg_atom* atoms, int max_atoms, const int32_t* n_new,
                               const int32_t* n_old, double* delta_fourier)
{
  if (!b || !atoms || !n_new || !n_old || !delta_fourier || max_atoms < 1) return RG_ERR_INVALID_ARGUMENT;
  rg_ewald* e = b->ewald;
  rg_ctx* ctx = e->ctx;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  // the staging buffers are free: every call ends by synchronising the stream; system s's atoms are packed at
  // s * stride (stride = max_atoms, at most kBatchAtoms)
  const int stride = std::min(max_atoms, kBatchAtoms);
  double4* packed = reinterpret_cast<double4*>(b->upload_host);
  int* counts = reinterpret_cast<int*>(packed + static_cast<size_t>(b->n) * stride);
  for (int s = 0; s < b->n; ++s)
  {
    if (n_new[s] < 0 || n_old[s] < 0 || n_new[s] + n_old[s] > std::min(max_atoms, kBatchAtoms))
      return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_ewald_batch_delta: at most 16 old + new atoms per system");
    const rg_atom* a = atoms + static_cast<long long>(s) * max_atoms;
    if (rg_status fs = rg::checkFinite(ctx, a, n_new[s] + n_old[s], "rg_ewald_batch_delta")) return fs;
    // new atoms with +q, old atoms with -q
    double4* to = packed + static_cast<size_t>(s) * stride;
    for (int i = 0; i < n_new[s] + n_old[s]; ++i)
    {
      const double r[3] = {a[i].x, a[i].y, a[i].z};
      double f[3];
      rg::matvec(e->box.ic, r, f);
      to[i] = make_double4(f[0], f[1], f[2], (i < n_new[s] ? 1.0 : -1.0) * a[i].scaling_coulomb * a[i].charge);
    }
    counts[s] = e->use_charge ? n_new[s] + n_old[s] : 0;
  }
  std::memcpy(counts + b->n, b->cur.data(), b->n);
  if (e->nk == 0 || !e->use_charge)
  {
    for (int s = 0; s < b->n; ++s) delta_fourier[s] = 0.0;
    return RG_OK;
  }
  RG_CUDA(ctx, cudaEventRecord(b->ev[0], ctx->stream));
  RG_CUDA(ctx, cudaMemcpyAsync(b->upload, b->upload_host, batchUploadBytes(b->n, stride), cudaMemcpyHostToDevice,
                               ctx->stream));
  const int kxm = e->ff.kmax_x, kym = e->ff.kmax_y, kzm = e->ff.kmax_z;
  const size_t shmem = batchSharedBytes(stride, kxm, kym, kzm);
  constexpr int most = 200 * 1024;  // the limit set as in launchPairs
  if (shmem > most)
    return rg::fail(ctx, RG_ERR_UNSUPPORTED, "rg_ewald_batch_delta: kmax too large for the shared-memory tables");
  RG_CUDA(ctx, cudaFuncSetAttribute(ewaldBatchDeltaKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  dim3 grid(b->blocks, b->n);
  RG_CUDA(ctx, cudaEventRecord(b->ev[1], ctx->stream));
  ewaldBatchDeltaKernel<<<grid, kThreads, shmem, ctx->stream>>>(b->runs, b->n_runs, b->row_start, b->slots, b->n,
                                                               b->run_temp, b->sk, b->upload, stride, kxm, kym, kzm,
                                                               b->partial);
  ewaldBatchTotalKernel<<<(b->n + kThreads - 1) / kThreads, kThreads, 0, ctx->stream>>>(b->n, b->blocks, b->partial,
                                                                                      b->result);
  RG_CUDA(ctx, cudaGetLastError());
  RG_CUDA(ctx, cudaEventRecord(b->ev[2], ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  RG_CUDA(ctx, cudaEventElapsedTime(&b->upload_ms, b->ev[0], b->ev[1]));
  RG_CUDA(ctx, cudaEventElapsedTime(&b->kernel_ms, b->ev[1], b->ev[2]));
  std::memcpy(delta_fourier, b->result_host, sizeof(double) * b->n);
  return RG_OK;
}

rg_status rg_ewald_batch_timing(rg_ewald_batch* b, float* upload_ms, float* kernel_ms)
{
  if (!b) return RG_ERR_INVALID_ARGUMENT;
  if (upload_ms) *upload_ms = b->upload_ms;
  if (kernel_ms) *kernel_ms = b->kernel_ms;
  return RG_OK;
}

rg_status rg_ewald_batch_accept(rg_ewald_batch* b, const uint8_t* accept)
{
  if (!b || !accept) return RG_ERR_INVALID_ARGUMENT;
  // the flags travel with the next call's atoms
  for (int s = 0; s < b->n; ++s)
    if (accept[s]) b->cur[s] ^= 1;
  return RG_OK;
}
}  // extern "C"
