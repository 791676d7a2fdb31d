// Device-resident grand-canonical Monte Carlo of rigid molecules: many independent chains, one CTA per chain.
//
// Each CTA runs a chain for a number of moves per launch, entirely on the device: the moves, energies, Rosenbluth
// weights and acceptance tests of the reference's
//   translation    src/raspakit/mc_moves/component/translation.cpp:30-200
//   rotation       src/raspakit/mc_moves/component/rotation.cpp:30-190
//   CBMC insertion src/raspakit/mc_moves/component/insertion_cbmc.cpp:34-207 (first beads: cbmc/multiple_first_bead.cpp
//                  :20-49; rigid orientations: cbmc/operators.cpp:951-970; selection: cbmc/util.cpp:14-47)
//   CBMC deletion  src/raspakit/mc_moves/component/deletion_cbmc.cpp:34-195 (retrace: cbmc/multiple_first_bead.cpp:51-76)
// with the framework-molecule energy from the tricubic grids, the molecule-molecule Lennard-Jones and real-space Ewald
// pair sums, and the Ewald Fourier energy change on the chain's own structure factors (which include the framework).
//
// Work split inside a CTA of 128 threads. A move is a chain of short dependent steps, so each step is spread over the
// CTA: a set's framework energy takes one lane per corner of each (atom, grid) interpolation; its molecule-molecule
// pairs take a warp per set, which tests all distances and lists the pairs within a cutoff, and evaluates the listed
// pairs of all its sets together; the exponentials of a selection take one lane per trial; the orientations of an
// insertion are drawn by another warp than its first beads; the Ewald change takes one thread per run of kz of a
// (kx, ky) and three values of |kz|, both signs from the same four sums, from phasor tables in shared memory. The chain's
// structure factors (and their change), its molecule count, energy and statistics stay in shared memory for the whole
// launch where they fit. All sums are in a fixed order (deterministic); arithmetic is FP64. Random numbers come from a
// counter-based generator (Philox-4x32-10, Salmon et al., SC'11) keyed by seed and chain and counted by (move, slot),
// so any thread can draw any move's numbers without shared state.
//
// What bounds it: the latency of a move's chain of steps, with four CTAs per SM to fill the gaps (44 % of the issue slots
// used), and before that the code's own size: at 211 KB for four chains at different places of it, waiting for the next
// instruction was two fifths of all stalls; the kernel is kept at 77 KB. 200 moves of 1,184 chains at a loading of about
// eight CO2 (kmax 8): 21.5 ms with all of S in global memory and a thread per k-vector, pair and trial, now 6.1 ms.
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "energy.cuh"
#include "fastmath.cuh"
#include "rng.cuh"

namespace
{
constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxAtoms = 8;     // atoms per molecule
constexpr int kMaxTrials = 16;   // first-bead positions / orientations per step
constexpr int kMaxK = 16;        // kmax per axis + 1 supported by the phase tables
constexpr int kEwaldM = 3;       // values of |kz| of one thread's share of a run
constexpr size_t kSharedPerCta = 50 * 1024;  // dynamic shared memory with which four CTAs fit on an SM
constexpr int kPairRoom = 64;    // listed pairs of a warp (evaluated 32 at a time)
constexpr int kSetsPerWarp = kMaxTrials / kWarps;

struct Component
{
  int n_atoms;
  int starting_bead;
  int types[kMaxAtoms];
  double charges[kMaxAtoms];
  double masses[kMaxAtoms];
  double offsets[kMaxAtoms][3];
  double self_excl;  // Ewald self + exclusion energy one inserted molecule adds (ewald.cpp:1164-1238, new-atom terms)
};

struct Params
{
  rgd::FF ff;
  rgd::Box box;
  rgd::Grid grid;            // data unused; shape and inverse cell
  const double* vdw_grid[kMaxAtoms];  // grid of each component atom's type (NULL = no framework term)
  const double* ewald_grid;
  int quintic;  // the grids hold the 27 triquintic values per point (RG_SCHEME_TRIQUINTIC) instead of 8
  double rcv_fw2, rcv_mol2, rcc2;
  Component comp;
  double beta, fugacity, volume;
  double max_translation, max_rotation;
  double p_translation, p_rotation, p_swap;
  int k1, k2;
  int capacity;
  int use_ewald;
  int64_t nk;
  int kmax[3];
  // runs of consecutive kz of one (kx, ky): {kx, ky, first k, (first kz, last kz) as shorts}, and the prefactor of the
  // k-vector with kz = +m, -m of run r at [(2 m + (sign < 0)) n_runs + r] (0: not in the run)
  int n_runs;
  const int4* runs;
  const double* run_temp;
  unsigned long long seed;
  // learned first-bead proposal (null: uniform): inclusive cumulative cell probabilities and the density relative to
  // uniform, over G^3 cells of the unit cell; the simulation box is rep[0] x rep[1] x rep[2] unit cells
  const double* prop_cdf;
  const double* prop_q;
  int prop_G;
  double prop_eps;
  double uc[3][3];   // unit cell c[col][row]
  double uic[3][3];  // its inverse
  int rep[3];
  // per-chain state
  double4* pos;              // [chain][capacity * n_atoms]
  double2* sk;               // [chain][nk] structure factors (framework included)
  double2* dsk;              // [chain][nk] scratch: structure-factor change of the current move (null: in shared memory)
  int* n;                    // [chain]
  double* energy;            // [chain]
  double* stats;             // [chain][kStats]
};

constexpr int kStats = 24;  // attempted[4], accepted[4], sum_n, sum_n2, sum_energy, samples, block_n[5] (sums), block_cnt

// The kernel's code has to stay small: four chains of an SM are at different places of it, and fetching instructions was
// what held the kernel (211 KB of code: 6.3 of 16.4 cycles per instruction waiting for the next one). So each phase
// stands once in the move's loop, and what several places call stays a function.
__device__ __noinline__ double2 uniform2(unsigned long long seed, int stream, long long move, uint32_t slot)
{
  uint32_t c[4] = {slot, static_cast<uint32_t>(move), static_cast<uint32_t>(move >> 32), static_cast<uint32_t>(stream)};
  uint32_t k0 = static_cast<uint32_t>(seed), k1 = static_cast<uint32_t>(seed >> 32);
#pragma unroll 2
  for (int r = 0; r < 10; ++r) rgd::philoxRound(c, k0, k1);
  return rgd::uniformsOf(c);
}
__device__ __noinline__ double expCall(double x) { return exp(x); }
__device__ __noinline__ double erfcCall(double x) { return erfc(x); }
__device__ __noinline__ void sincospiCall(double x, double* sn, double* cs) { sincospi(x, sn, cs); }

// random slots of one move
enum Slot
{
  kSlotMove = 0,       // (move kind, insertion-or-deletion)
  kSlotPick = 1,       // (molecule, direction)
  kSlotChange = 2,     // (displacement or angle, acceptance)
  kSlotSelect = 3,     // (first-bead selection, orientation selection)
  kSlotFirst = 16,     // + 4 t: first-bead position t (up to 8 numbers)
  kSlotOrient = 128    // + 2 t: orientation t (3 numbers)
};

__device__ __forceinline__ void rotationFromUniforms(double u1, double u2, double u3, double R[3][3])
{
  // uniform unit quaternion (Shoemake) -> rotation matrix
  double s2, c2, s3, c3;
  sincospiCall(2 * u2, &s2, &c2);
  sincospiCall(2 * u3, &s3, &c3);
  const double a = sqrt(1 - u1), b = sqrt(u1);
  const double x = a * s2, y = a * c2, z = b * s3, w = b * c3;
  R[0][0] = 1 - 2 * (y * y + z * z);
  R[0][1] = 2 * (x * y - z * w);
  R[0][2] = 2 * (x * z + y * w);
  R[1][0] = 2 * (x * y + z * w);
  R[1][1] = 1 - 2 * (x * x + z * z);
  R[1][2] = 2 * (y * z - x * w);
  R[2][0] = 2 * (x * z - y * w);
  R[2][1] = 2 * (y * z + x * w);
  R[2][2] = 1 - 2 * (x * x + y * y);
}

// One pair of component atoms at full scaling: 4 eps, 1 / sigma^2, shift (0 without a Lennard-Jones term), C q_A q_B
struct PairTerm
{
  double eps4, inv_sig2, shift, qq;
};

struct Shared
{
  double pairE[kMaxTrials];  // per set (or half set) of evaluateSets: the molecule-molecule energy, and an overlap
  int pairOv[kMaxTrials];
  double logq[kMaxTrials];
  double red[kWarps];
  double pair_rr[kWarps][kPairRoom];
  int pair_code[kWarps][kPairRoom];  // set of the warp << 8 | component atom << 4 | partner atom
  int list[kMaxAtoms];               // component atoms of the sets
  int n;
  int sel;
  double W, E;
  double energy;
  double stats[24];
};

// Dynamic shared memory: per trial and component atom the position and (orientations) the offset from the first bead,
// the framework energies of a set's atoms, the pair table, the phasor tables of the moved atoms, and (SMEM) the chain's
// structure factors and their change.
struct Dyn
{
  double* trial;    // [kMaxTrials][na][3]
  double* rel;      // [kMaxTrials][na][3]
  double* gridE;    // [kMaxTrials][na][2]
  PairTerm* pair;   // [na][na]
  int* gridOv;      // [kMaxTrials][na]
  double2* ex;      // [2 na][kx + 1], weighted by the signed charge
  double2* ey;      // [2 na][2 ky + 1]
  double2* ez;      // [2 na][kz + 1]
  double2* S;       // [nk]
  double2* D;       // [nk]
};
__host__ __device__ constexpr size_t dynFixedBytes(int na, const int* kmax, bool ewald)
{
  size_t b = sizeof(double) * kMaxTrials * na * 8 + sizeof(PairTerm) * na * na + ((sizeof(int) * kMaxTrials * na + 15) & ~size_t(15));
  if (ewald) b += sizeof(double2) * 2 * na * ((kmax[0] + 1) + (2 * kmax[1] + 1) + (kmax[2] + 1));
  return b;
}
constexpr int kTopK[3] = {kMaxK - 1, kMaxK - 1, kMaxK - 1};
static_assert(dynFixedBytes(kMaxAtoms, kTopK, true) <= kSharedPerCta, "no launch takes more than kSharedPerCta");
__device__ __forceinline__ Dyn dynOf(const Params& p)
{
  extern __shared__ __align__(16) unsigned char dynSmem[];
  const int na = p.comp.n_atoms;
  Dyn d;
  d.trial = reinterpret_cast<double*>(dynSmem);
  d.rel = d.trial + kMaxTrials * na * 3;
  d.gridE = d.rel + kMaxTrials * na * 3;
  d.pair = reinterpret_cast<PairTerm*>(d.gridE + kMaxTrials * na * 2);
  d.gridOv = reinterpret_cast<int*>(d.pair + na * na);
  d.ex = reinterpret_cast<double2*>(reinterpret_cast<unsigned char*>(d.gridOv) + ((sizeof(int) * kMaxTrials * na + 15) & ~size_t(15)));
  d.ey = d.ex + 2 * na * (p.kmax[0] + 1);
  d.ez = d.ey + 2 * na * (2 * p.kmax[1] + 1);
  d.S = d.ez + 2 * na * (p.kmax[2] + 1);
  d.D = d.S + p.nk;
  return d;
}

// Energy of one pair at full scaling: Lennard-Jones (potentials/pair_vdw.ixx:85-101) within its cutoff, whose overlap is
// tested, and real-space Ewald (pair_coulomb.ixx:51-77) within its own
__device__ __forceinline__ double pairEnergy(const Params& p, const PairTerm& t, double rr, int* ov)
{
  double e = 0.0;
  if (rr < p.rcv_mol2)
  {
    const double x = rr * t.inv_sig2;
    const double i3 = rgd::rcpHouseholder(x * x * x);
    e = t.eps4 * (i3 * (i3 - 1.0)) - t.shift;
    if (!(e <= p.ff.overlap)) *ov = 1;  // NaN too: the reciprocal's refinement makes it of 0 and of subnormal numbers
  }
  if (p.ff.use_charge && rr < p.rcc2)
  {
    const double invr = rgd::rsqrtHouseholder(rr), ar = p.ff.alpha * (rr * invr);
    const double ec = ar < rgd::kErfcxMax ? rgd::erfcFromExp64<false>(ar, expCall(-ar * ar)) : erfcCall(ar);
    e += t.qq * ec * invr;
  }
  return e;
}

// Round to nearest for |x| < 2^51, on the FP64 pipe (a tie goes to the even number; either gives the same distance)
__device__ __forceinline__ double nearest(double x) { return (x + 6755399441055744.0) - 6755399441055744.0; }

// a / n for 0 <= a < 2^21 and small n, from the FP32 reciprocal of n (off by a 2^-22.5 of the quotient, below 1 / (2 n))
constexpr int kDivideSmall = 1 << 21;
__device__ __forceinline__ int divideSmall(int a, float inv) { return static_cast<int>((static_cast<float>(a) + 0.5f) * inv); }

// External energies (framework grids + other molecules) of `ns` sets of the `cnt` component atoms sh.list, at
// d.trial[set][atom], without molecule `skip`: left in sh.pairE, d.gridE and their overlap flags for setEnergy. Two sets
// (old and new positions) are halved between the warps. Block-wide; ends with a barrier.
__device__ __forceinline__ int halvesOf(int ns) { return 2 * ns <= kWarps ? 2 : 1; }
template <bool QUINTIC>  // the system's grids: triquintic (27 values per point) or tricubic (8)
__device__ __forceinline__ void evaluateSets(const Params& p, Shared& sh, const Dyn& d, const double4* cpos, int n, int ns,
                                             int cnt, int skip)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int na = p.comp.n_atoms;
  // framework: lanes of a group of 8 take the corners of one (set, atom, grid); triquintic grids one lane each
  constexpr int kCorners = QUINTIC ? 1 : 8;
  const int tasks = ns * cnt * 2 * kCorners;
  const float inv_cnt = 1.0f / static_cast<float>(cnt), inv_na = 1.0f / static_cast<float>(na);
#pragma unroll 1
  for (int base = 32 * warp; base < tasks; base += kThreads)
  {
    const int idx = base + lane;
    const int item = idx / kCorners, g = item & 1, sj = item >> 1;
    double v = 0.0;
    int ai = 0;
    if (idx < tasks)
    {
      const int s = divideSmall(sj, inv_cnt);
      ai = sh.list[sj - s * cnt];
      rgd::Grid gg = p.grid;
      gg.data = p.vdw_grid[ai];
      if (g == 1 && gg.data) gg.data = p.ff.use_charge ? p.ewald_grid : nullptr;
      if (gg.data)
      {
        const double* r = d.trial + 3 * (s * na + ai);
        if constexpr (QUINTIC)
          v = rgd::interpolateQuintic(gg, r[0], r[1], r[2], nullptr);
        else
          v = rgd::interpolateLaneCorner(gg, r[0], r[1], r[2], idx & 7);
      }
    }
    if constexpr (!QUINTIC)
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (idx < tasks && (QUINTIC || (idx & 7) == 0))
    {
      if (g == 0) d.gridOv[sj] = v > p.ff.overlap ? 1 : 0;
      d.gridE[item] = g == 0 ? v : p.comp.charges[ai] * v;
    }
  }
  // molecule-molecule pairs: warp w takes (half) sets w, w + kWarps, ...
  const double reach2 = p.ff.use_charge ? fmax(p.rcv_mol2, p.rcc2) : p.rcv_mol2;
  double e[kSetsPerWarp];
  int ov = 0;  // bit q: an overlap in the warp's q-th set
#pragma unroll
  for (int q = 0; q < kSetsPerWarp; ++q) e[q] = 0.0;
  double* rrs = sh.pair_rr[warp];
  int* codes = sh.pair_code[warp];
  int listed = 0;
  // one loop over the distance tests of all the warp's sets, whose last turn only evaluates what is still listed
  const int halves = halvesOf(ns), nv = ns * halves;
  const int total = n * na * cnt, length = (total + halves - 1) / halves;
  const int rounds = (length + 31) / 32;  // of one (half) set
  const int turns = warp < nv ? (nv - warp + kWarps - 1) / kWarps * rounds : 0;
  int q = 0, round = 0;
#pragma unroll 1
  for (int turn = 0; turn <= turns; ++turn)
  {
    const bool testing = turn < turns;
    if (testing)
    {
      const int v = warp + q * kWarps, half = halves == 2 ? v & 1 : 0, s = halves == 2 ? v >> 1 : v;
      const int t = half * length + 32 * round + lane;
      bool in = false;
      double rr = 0.0;
      int code = 0;
      if (32 * round + lane < length && t < total)
      {
        // t runs over partner atoms, and over the set's atoms within a partner
        const int b = total < kDivideSmall ? divideSmall(t, inv_cnt) : t / cnt, j = t - b * cnt;
        const int m = total < kDivideSmall ? divideSmall(b, inv_na) : b / na;
        if (m != skip)
        {
          const int ai = sh.list[j];
          const double4 B = cpos[b];
          const double* r = d.trial + 3 * (s * na + ai);
          double dx = B.x - r[0], dy = B.y - r[1], dz = B.z - r[2];
          if (!p.box.triclinic)
          {
            dx -= nearest(dx * p.box.ic[0][0]) * p.box.c[0][0];
            dy -= nearest(dy * p.box.ic[1][1]) * p.box.c[1][1];
            dz -= nearest(dz * p.box.ic[2][2]) * p.box.c[2][2];
          }
          else
            rgd::pbc(p.box, dx, dy, dz);
          rr = dx * dx + dy * dy + dz * dz;
          in = rr < reach2;
          code = q << 8 | ai << 4 | (b - m * na);
        }
      }
      const unsigned ballot = __ballot_sync(0xffffffffu, in);
      if (in)
      {
        const int at = listed + __popc(ballot & ((1u << lane) - 1u));
        rrs[at] = rr;
        codes[at] = code;
      }
      listed += __popc(ballot);
      if (++round == rounds)
      {
        round = 0;
        ++q;
      }
    }
    const int count = listed >= 32 ? 32 : (testing ? 0 : listed);
    if (count == 0) continue;
    listed -= count;  // the last ones listed; the others stay
    __syncwarp();
    if (lane < count)
    {
      const int code = codes[listed + lane];
      int o = 0;
      const double x = pairEnergy(p, d.pair[((code >> 4) & 15) * na + (code & 15)], rrs[listed + lane], &o);
      ov |= o << (code >> 8);
#pragma unroll
      for (int u = 0; u < kSetsPerWarp; ++u)
        if (code >> 8 == u) e[u] += x;
    }
    __syncwarp();
  }
  ov = __reduce_or_sync(0xffffffffu, ov);
#pragma unroll
  for (int u = 0; u < kSetsPerWarp; ++u)
  {
    const int v = warp + u * kWarps;
    if (v >= nv) break;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e[u] += __shfl_down_sync(0xffffffffu, e[u], o);
    if (lane == 0)
    {
      sh.pairE[v] = e[u];
      sh.pairOv[v] = (ov >> u) & 1;
    }
  }
  __syncthreads();
}

// The energy of set s of the last evaluateSets, and whether it overlaps
__device__ __forceinline__ double setEnergy(const Shared& sh, const Dyn& d, int ns, int cnt, int s, int* ov)
{
  const int halves = halvesOf(ns);
  double e = sh.pairE[s * halves];
  int o = sh.pairOv[s * halves];
  if (halves == 2)
  {
    e += sh.pairE[2 * s + 1];
    o |= sh.pairOv[2 * s + 1];
  }
#pragma unroll 1
  for (int j = 0; j < cnt; ++j)
  {
    const double2 g = reinterpret_cast<const double2*>(d.gridE)[s * cnt + j];
    e += g.x + g.y;
    o |= d.gridOv[s * cnt + j];
  }
  *ov = o;
  return e;
}

// Ewald Fourier energy change of the moved atoms: `nNew` atoms of set newSet with their charges, `nOld` of set oldSet
// with the opposite ones; leaves the change of the structure factors in D. Block-wide; returns the energy on every
// thread. P = w e^{2 pi i (kx s_x + ky s_y)} = (p, q) and (c, s) = e^{2 pi i m s_z} give kz = m as (pc - qs, ps + qc)
// and kz = -m as (pc + qs, qc - ps): four FMAs per atom for two k-vectors.
__device__ __forceinline__ double blockEwaldDelta(const Params& p, Shared& sh, const Dyn& d, const double2* S, double2* D, int newSet,
                                  int nNew, int oldSet, int nOld)
{
  const Component& c = p.comp;
  const int na = c.n_atoms, nAt = nNew + nOld;
  const int nx = p.kmax[0] + 1, ny = 2 * p.kmax[1] + 1, nz = p.kmax[2] + 1;
  const int per = nx + (p.kmax[1] + 1) + nz;
#pragma unroll 1
  for (int idx = threadIdx.x; idx < nAt * per; idx += kThreads)
  {
    const int a = idx / per, m = idx - a * per;
    const int ai = a < nNew ? a : a - nNew;
    const double* r = d.trial + 3 * ((a < nNew ? newSet : oldSet) * na + ai);
    const int dim = m < nx ? 0 : (m < nx + p.kmax[1] + 1 ? 1 : 2);
    const int mm = dim == 0 ? m : (dim == 1 ? m - nx : m - nx - (p.kmax[1] + 1));
    const double s = p.box.ic[0][dim] * r[0] + p.box.ic[1][dim] * r[1] + p.box.ic[2][dim] * r[2];
    double sn, cs;
    sincospiCall(2.0 * static_cast<double>(mm) * s, &sn, &cs);
    if (dim == 0)
    {
      const double w = a < nNew ? c.charges[ai] : -c.charges[ai];
      d.ex[a * nx + mm] = make_double2(w * cs, w * sn);
    }
    else if (dim == 1)
    {
      d.ey[a * ny + p.kmax[1] + mm] = make_double2(cs, sn);
      d.ey[a * ny + p.kmax[1] - mm] = make_double2(cs, -sn);
    }
    else
      d.ez[a * nz + mm] = make_double2(cs, sn);
  }
  __syncthreads();
  const int groups = (nz + kEwaldM - 1) / kEwaldM;
  double e = 0.0;
#pragma unroll 1
  for (int item = threadIdx.x; item < p.n_runs * groups; item += kThreads)
  {
    const int g = item / p.n_runs, run_at = item - g * p.n_runs, m0 = g * kEwaldM;
    const int4 run = p.runs[run_at];
    const int lo = static_cast<short>(run.w & 0xffff), hi = run.w >> 16;
    if (m0 > max(-lo, hi)) continue;
    double pc[kEwaldM], qs[kEwaldM], ps[kEwaldM], qc[kEwaldM];
#pragma unroll
    for (int m = 0; m < kEwaldM; ++m) pc[m] = qs[m] = ps[m] = qc[m] = 0.0;
#pragma unroll 1
    for (int a = 0; a < nAt; ++a)
    {
      const double2 x = d.ex[a * nx + run.x], y = d.ey[a * ny + p.kmax[1] + run.y];
      const double pp = x.x * y.x - x.y * y.y, qq = x.x * y.y + x.y * y.x;
#pragma unroll
      for (int m = 0; m < kEwaldM; ++m)
      {
        const double2 z = d.ez[a * nz + min(m0 + m, nz - 1)];
        pc[m] = fma(pp, z.x, pc[m]);
        qs[m] = fma(qq, z.y, qs[m]);
        ps[m] = fma(pp, z.y, ps[m]);
        qc[m] = fma(qq, z.x, qc[m]);
      }
    }
    const int first = run.z - lo;  // index of kz = 0, were it in the run
#pragma unroll
    for (int m = 0; m < kEwaldM; ++m)
#pragma unroll
      for (int sign = 0; sign < 2; ++sign)
      {
        const int kz = sign == 0 ? m0 + m : -(m0 + m);
        if (kz < lo || kz > hi || (sign == 1 && kz == 0)) continue;
        const double2 dr = sign == 0 ? make_double2(pc[m] - qs[m], ps[m] + qc[m])
                                     : make_double2(pc[m] + qs[m], qc[m] - ps[m]);
        const double2 s = S[first + kz];
        e += p.run_temp[(2 * (m0 + m) + sign) * p.n_runs + run_at] *
             (2.0 * (s.x * dr.x + s.y * dr.y) + (dr.x * dr.x + dr.y * dr.y));
        D[first + kz] = dr;
      }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) sh.red[threadIdx.x >> 5] = e;
  __syncthreads();
  double tot = 0.0;
  for (int w = 0; w < kWarps; ++w) tot += sh.red[w];
  return tot;
}

__device__ __forceinline__ void blockAcceptEwald(const Params& p, double2* S, const double2* D)
{
#pragma unroll 2
  for (int k = threadIdx.x; k < p.nk; k += kThreads)
  {
    const double2 d = D[k], s = S[k];
    S[k] = make_double2(s.x + d.x, s.y + d.y);
  }
}

// CBMC::selectTrialPosition (cbmc/util.cpp:14-47) over the non-overlapping trials, by one warp with a lane per trial:
// the chosen trial (the first whose running sum of weights reaches u times their total, else the last) and the
// Rosenbluth weight sum_i exp(-beta U_i) / k, or -1 if every trial overlaps (`in`: the lane holds one that does not). The
// log weight of trial t is -beta U_t - log q_t (logq 0: uniform, q = 1).
__device__ __forceinline__ int selectTrial(double E, bool in, double logq, int k, double beta, double u, double* W)
{
  const int lane = threadIdx.x & 31;
  const unsigned mask = __ballot_sync(0xffffffffu, in);
  if (mask == 0u)
  {
    *W = 0.0;
    return -1;
  }
  const double lw = in ? -beta * E - logq : -1e300;
  double largest = lw;
#pragma unroll
  for (int o = kMaxTrials / 2; o > 0; o >>= 1) largest = fmax(largest, __shfl_xor_sync(0xffffffffu, largest, o));
  largest = __shfl_sync(0xffffffffu, largest, 0);
  double run = in ? expCall(lw - largest) : 0.0, w = in ? expCall(lw) : 0.0;
#pragma unroll
  for (int o = 1; o < kMaxTrials; o <<= 1)
  {
    const double x = __shfl_up_sync(0xffffffffu, run, o);
    if (lane >= o) run += x;
    w += __shfl_xor_sync(0xffffffffu, w, o);
  }
  *W = __shfl_sync(0xffffffffu, w, 0) / static_cast<double>(k);
  const double ws = u * __shfl_sync(0xffffffffu, run, kMaxTrials - 1);
  const unsigned reach = __ballot_sync(0xffffffffu, in && !(run < ws));
  return reach ? __ffs(reach) - 1 : 31 - __clz(mask);
}

// Proposal density (relative to uniform) of a position: the cell of its unit-cell fractional coordinates.
__device__ __forceinline__ double proposalDensity(const Params& p, const double r[3])
{
  int c[3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
  {
    const double s = rgd::fract1(p.uic[0][a] * r[0] + p.uic[1][a] * r[1] + p.uic[2][a] * r[2]);
    c[a] = min(p.prop_G - 1, static_cast<int>(s * p.prop_G));
  }
  return p.prop_q[c[0] + p.prop_G * (c[1] + p.prop_G * c[2])];
}

template <bool QUINTIC, bool SMEM>
__global__ void __launch_bounds__(kThreads, 4) gcmcKernel(Params p, long long move0, int nmoves, int record,
                                                          long long block_len)
{
  const int chain = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ Shared sh;
  const Dyn d = dynOf(p);
  const Component& c = p.comp;
  const int na = c.n_atoms, sb = c.starting_bead;
  double4* cpos = p.pos + static_cast<long long>(chain) * p.capacity * na;
  double* st = p.stats + static_cast<long long>(chain) * kStats;
  double2* gS = p.sk + static_cast<long long>(chain) * p.nk;
  double2* S = SMEM ? d.S : gS;
  double2* D = SMEM ? d.D : p.dsk + static_cast<long long>(chain) * p.nk;
  const double ptot = p.p_translation + p.p_rotation + p.p_swap;

  // the chain's state of this launch
  for (int i = threadIdx.x; i < na * na; i += kThreads)
  {
    const int idx = c.types[i % na] * p.ff.n + c.types[i / na];
    const bool lj = p.ff.lj[idx] != 0;
    d.pair[i] = {lj ? p.ff.eps4[idx] : 0.0, lj ? 1.0 / p.ff.sig2[idx] : 1.0, lj ? p.ff.shift[idx] : 0.0,
                 p.ff.coul * c.charges[i % na] * c.charges[i / na]};
  }
  if (SMEM && p.use_ewald)
    for (int k = threadIdx.x; k < p.nk; k += kThreads) S[k] = gS[k];
  if (threadIdx.x < kStats) sh.stats[threadIdx.x] = st[threadIdx.x];
  if (threadIdx.x == 0)
  {
    sh.n = p.n[chain];
    sh.energy = p.energy[chain];
  }
  __syncthreads();

  for (int it = 0; it < nmoves; ++it)
  {
    const long long mv = move0 + it;
    const int n = sh.n;
    // the move's own numbers: four lanes of each warp draw one block each
    static_assert(kSlotMove == 0 && kSlotPick == 1 && kSlotChange == 2 && kSlotSelect == 3, "slots of lanes 0..3");
    const double2 uLane = uniform2(p.seed, chain, mv, lane & 3);
    auto fromLane = [&](int l)
    { return make_double2(__shfl_sync(0xffffffffu, uLane.x, l), __shfl_sync(0xffffffffu, uLane.y, l)); };
    const double2 uMove = fromLane(kSlotMove), uPick = fromLane(kSlotPick), uChange = fromLane(kSlotChange),
                  uSel = fromLane(kSlotSelect);
    const double x = uMove.x * ptot;
    const int kind = x < p.p_translation ? 0 : (x < p.p_translation + p.p_rotation ? 1 : (uMove.y < 0.5 ? 2 : 3));
    const bool swap = kind >= 2, insert = kind == 2, retrace = kind == 3;
    // the molecule moved, deleted or (the next place) inserted
    const int m = insert ? n : min(n - 1, static_cast<int>(uPick.x * n));
    bool alive = insert ? n < p.capacity : n > 0;  // the move goes on
    const int skip = insert ? -1 : m;
    double W1 = 1.0, e1 = 0.0;  // first bead: Rosenbluth weight and energy
    int chosen = 0;

    // Translation and rotation: one evaluation, of set 0 (new positions) and set 1 (old). Swap: two, the first-bead
    // positions and then the orientations about the chosen one.
    if (alive)
    {
      if (!swap)
      {
        const int dir = min(2, static_cast<int>(3.0 * uPick.y));
        if (threadIdx.x < na)
        {
          const int i = threadIdx.x;
          const double4 o = cpos[m * na + i];
          const double old[3] = {o.x, o.y, o.z};
          double now[3];
          if (kind == 0)
          {
            const double disp = p.max_translation * 2.0 * (uChange.x - 0.5);
#pragma unroll
            for (int r = 0; r < 3; ++r) now[r] = old[r] + (r == dir ? disp : 0.0);
          }
          else
          {
            const double angle = p.max_rotation * 2.0 * (uChange.x - 0.5);
            double sn, cs;
            sincospiCall(angle * (1.0 / rg::kPi), &sn, &cs);
            double com[3] = {0, 0, 0}, wsum = 0.0;
#pragma unroll 1
            for (int j = 0; j < na; ++j)
            {
              const double4 q = cpos[m * na + j];
              com[0] += c.masses[j] * q.x;
              com[1] += c.masses[j] * q.y;
              com[2] += c.masses[j] * q.z;
              wsum += c.masses[j];
            }
            const double inv = 1.0 / wsum;
            double r[3], q[3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
              com[k] *= inv;
              r[k] = old[k] - com[k];
            }
            // about axis dir: (a, b) are the two others in cyclic order
            q[0] = dir == 0 ? r[0] : (dir == 1 ? sn * r[2] + cs * r[0] : cs * r[0] - sn * r[1]);
            q[1] = dir == 0 ? cs * r[1] - sn * r[2] : (dir == 1 ? r[1] : sn * r[0] + cs * r[1]);
            q[2] = dir == 0 ? sn * r[1] + cs * r[2] : (dir == 1 ? cs * r[2] - sn * r[0] : r[2]);
#pragma unroll
            for (int k = 0; k < 3; ++k) now[k] = com[k] + q[k];
          }
#pragma unroll
          for (int r = 0; r < 3; ++r)
          {
            d.trial[3 * i + r] = now[r];
            d.trial[3 * (na + i) + r] = old[r];
          }
          sh.list[i] = i;
        }
      }
      else
      {
        // first-bead trial positions on warp 0 (retrace: trial 0 is the existing first bead); each lane's four draws
        if (warp == 0 && lane < p.k1)
        {
          const int t = lane;
          double* r = d.trial + 3 * (t * na + sb);
          if (retrace && t == 0)
          {
            const double4 o = cpos[m * na + sb];
            r[0] = o.x;
            r[1] = o.y;
            r[2] = o.z;
          }
          else
          {
            const double2 a = uniform2(p.seed, chain, mv, kSlotFirst + 4 * t);
            const double2 b = uniform2(p.seed, chain, mv, kSlotFirst + 4 * t + 1);
            double sf[3] = {a.x, a.y, b.x};
            bool tabulated = false;
            if (p.prop_cdf)
            {
              const double2 u = uniform2(p.seed, chain, mv, kSlotFirst + 4 * t + 2);
              tabulated = !(u.x < p.prop_eps);
              if (tabulated)
              {
                // a cell of the tabulated proposal (binary search of the cumulative probabilities), a uniform point in
                // it, and a uniformly chosen unit-cell replica of the simulation box
                const double2 v = uniform2(p.seed, chain, mv, kSlotFirst + 4 * t + 3);
                const int G = p.prop_G;
                int lo = 0, hi = G * G * G - 1;
                while (lo < hi)
                {
                  const int mid = (lo + hi) >> 1;
                  if (p.prop_cdf[mid] < u.y)
                    lo = mid + 1;
                  else
                    hi = mid;
                }
                const int ci = lo % G, cj = (lo / G) % G, ck = lo / (G * G);
                const double at[3] = {ci + a.x, cj + a.y, ck + b.x}, pick[3] = {b.y, v.x, v.y};
#pragma unroll
                for (int q = 0; q < 3; ++q)
                  sf[q] = at[q] / G + static_cast<double>(min(p.rep[q] - 1, static_cast<int>(pick[q] * p.rep[q])));
              }
            }
            // SimulationBox::randomPosition (simulationbox.cpp:132-135), or the cell's point in unit cells
#pragma unroll
            for (int q = 0; q < 3; ++q)
              r[q] = tabulated ? p.uc[0][q] * sf[0] + p.uc[1][q] * sf[1] + p.uc[2][q] * sf[2]
                               : p.box.c[0][q] * sf[0] + p.box.c[1][q] * sf[1] + p.box.c[2][q] * sf[2];
          }
          sh.logq[t] = p.prop_cdf ? log(proposalDensity(p, r)) : 0.0;
        }
        // the orientations' offsets from the first bead, meanwhile, on warp 1
        if (warp == 1 && lane < p.k2 && !(retrace && lane == 0))
        {
          const double2 a = uniform2(p.seed, chain, mv, kSlotOrient + 2 * lane);
          const double2 b = uniform2(p.seed, chain, mv, kSlotOrient + 2 * lane + 1);
          double R[3][3];
          rotationFromUniforms(a.x, a.y, b.x, R);
          double* rel = d.rel + 3 * lane * na;
#pragma unroll 1
          for (int i = 0; i < na; ++i)
#pragma unroll
            for (int r = 0; r < 3; ++r)
              rel[3 * i + r] = R[r][0] * (c.offsets[i][0] - c.offsets[sb][0]) +
                               R[r][1] * (c.offsets[i][1] - c.offsets[sb][1]) +
                               R[r][2] * (c.offsets[i][2] - c.offsets[sb][2]);
        }
        if (threadIdx.x == 0) sh.list[0] = sb;
      }
      __syncthreads();
#pragma unroll 1
      for (int phase = 0; phase < (swap ? 2 : 1); ++phase)
      {
        const int ns = swap ? (phase == 0 ? p.k1 : p.k2) : 2, cnt = swap ? (phase == 0 ? 1 : na - 1) : na;
        evaluateSets<QUINTIC>(p, sh, d, cpos, n, ns, cnt, skip);
        if (!swap) break;
        if (warp == 0)
        {
          double W, E = 0.0;
          int ov = 1;
          if (lane < ns) E = setEnergy(sh, d, ns, cnt, lane, &ov);
          int sel = selectTrial(E, !ov, phase == 0 && lane < ns ? sh.logq[lane] : 0.0, ns, p.beta,
                                phase == 0 ? uSel.x : uSel.y, &W);
          if (retrace) sel = __shfl_sync(0xffffffffu, ov, 0) ? -1 : 0;
          E = __shfl_sync(0xffffffffu, E, max(sel, 0));
          if (lane == 0)
          {
            sh.sel = sel;
            sh.W = W;
            sh.E = E;
          }
        }
        __syncthreads();
        chosen = sh.sel;
        W1 *= sh.W;
        e1 += sh.E;
        if (chosen < 0)
        {
          alive = false;
          break;
        }
        if (phase == 1) break;
        const double fb[3] = {d.trial[3 * (chosen * na + sb)], d.trial[3 * (chosen * na + sb) + 1],
                              d.trial[3 * (chosen * na + sb) + 2]};
        __syncthreads();
        // orientation trials about the first bead (retrace: trial 0 is the existing orientation)
#pragma unroll 1
        for (int q = threadIdx.x; q < p.k2 * na; q += kThreads)
        {
          double* r = d.trial + 3 * q;
          if (retrace && q < na)
          {
            const double4 o = cpos[m * na + q];
            r[0] = o.x;
            r[1] = o.y;
            r[2] = o.z;
          }
          else
#pragma unroll
            for (int k = 0; k < 3; ++k) r[k] = fb[k] + d.rel[3 * q + k];
        }
        if (threadIdx.x < na && static_cast<int>(threadIdx.x) != sb)
          sh.list[threadIdx.x - (static_cast<int>(threadIdx.x) > sb ? 1 : 0)] = threadIdx.x;
        __syncthreads();
      }
    }
    int accepted = 0;
    double dE = 0.0;
    if (alive)
    {
      double dEw = 0.0;
      if (p.use_ewald)
      {
        dEw = blockEwaldDelta(p, sh, d, S, D, chosen, retrace ? 0 : na, swap ? chosen : 1, insert ? 0 : na);
        if (swap) dEw += insert ? c.self_excl : -c.self_excl;
      }
      double pacc;
      if (!swap)
      {
        int ov, old_ov;
        dE = setEnergy(sh, d, 2, na, 0, &ov) - setEnergy(sh, d, 2, na, 1, &old_ov) + dEw;
        pacc = expCall(-p.beta * dE);
        accepted = !ov && uChange.y < pacc;
      }
      else
      {
        dE = insert ? e1 + dEw : dEw - e1;
        pacc = expCall(-p.beta * dEw);
        if (insert)
          pacc = W1 < 1e-150 ? 0.0 : pacc * p.beta * p.fugacity * p.volume / static_cast<double>(n + 1) * W1;
        else
          pacc = pacc * static_cast<double>(n) / (p.beta * p.fugacity * p.volume) / W1;
        accepted = uChange.y < pacc;
      }
      if (accepted)
      {
        if (threadIdx.x < na)
        {
          const double* r = d.trial + 3 * (chosen * na + threadIdx.x);
          if (!retrace)
            cpos[m * na + threadIdx.x] = make_double4(r[0], r[1], r[2], 0.0);
          else if (m != n - 1)
            cpos[m * na + threadIdx.x] = cpos[(n - 1) * na + threadIdx.x];
        }
        if (p.use_ewald) blockAcceptEwald(p, S, D);
      }
    }
    if (threadIdx.x == 0)
    {
      if (accepted)
      {
        sh.energy += dE;
        if (swap) sh.n = insert ? n + 1 : n - 1;
      }
      if (record)
      {
        const int nn = sh.n;
        double* q = sh.stats;
        q[kind] += 1.0;
        q[4 + kind] += accepted ? 1.0 : 0.0;
        q[8] += nn;
        q[9] += static_cast<double>(nn) * nn;
        q[10] += sh.energy;
        q[11] += 1.0;
        const long long b = block_len > 0 ? static_cast<long long>(q[11] - 1.0) / block_len : 0;
        if (b < 5) q[12 + b] += nn;
      }
    }
    __syncthreads();
  }
  if (SMEM && p.use_ewald)
    for (int k = threadIdx.x; k < p.nk; k += kThreads) gS[k] = S[k];
  if (threadIdx.x < kStats) st[threadIdx.x] = sh.stats[threadIdx.x];
  if (threadIdx.x == 0)
  {
    p.n[chain] = sh.n;
    p.energy[chain] = sh.energy;
  }
}
}  // namespace

struct rg_gcmc
{
  rg_ctx* ctx = nullptr;
  Params p{};
  int n_chains = 0;
  long long moves_done = 0;
  long long recorded = 0;
  long long block_len = 0;
  size_t shmem = 0;
  bool smem = true;  // the structure factors fit in shared memory
  int4* runs = nullptr;
  double* run_temp = nullptr;
  int max_moves_per_launch = 2048;
};

extern "C"
{
rg_status rg_gcmc_create(rg_system* system, rg_ewald* ewald, const rg_gcmc_component* comp,
                         const rg_gcmc_params* params, int n_chains, rg_gcmc** out)
{
  if (!system || !comp || !params || !out || n_chains < 1) return RG_ERR_INVALID_ARGUMENT;
  if (comp->n_atoms < 1 || comp->n_atoms > kMaxAtoms || comp->starting_bead < 0 || comp->starting_bead >= comp->n_atoms)
    return RG_ERR_INVALID_ARGUMENT;
  if (params->n_first_bead_trials < 1 || params->n_first_bead_trials > kMaxTrials ||
      params->n_orientation_trials < 1 || params->n_orientation_trials > kMaxTrials || params->max_molecules < 1)
    return RG_ERR_INVALID_ARGUMENT;
  rgd::FF ff;
  rgd::Box box;
  const double* grids[64];
  const double* ewald_grid = nullptr;
  int n_types, gdims[3];
  double gic[3][3];
  rg_ctx* ctx;
  rg_status st = rgd::systemExport(system, &ff, &box, grids, &ewald_grid, &n_types, gdims, gic, &ctx);
  if (st) return st;
  for (int i = 0; i < comp->n_atoms; ++i)
    if (comp->types[i] < 0 || comp->types[i] >= n_types) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_gcmc: type");
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  rg_gcmc* g = new rg_gcmc();
  g->ctx = ctx;
  g->n_chains = n_chains;
  Params& p = g->p;
  p.ff = ff;
  p.box = box;
  p.grid.nx = gdims[0];
  p.grid.ny = gdims[1];
  p.grid.nz = gdims[2];
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b) p.grid.ic[a][b] = gic[a][b];
  p.comp.n_atoms = comp->n_atoms;
  p.comp.starting_bead = comp->starting_bead;
  for (int i = 0; i < comp->n_atoms; ++i)
  {
    p.comp.types[i] = comp->types[i];
    p.comp.charges[i] = comp->charges[i];
    p.comp.masses[i] = comp->masses[i];
    for (int d = 0; d < 3; ++d) p.comp.offsets[i][d] = comp->offsets[3 * i + d];
    p.vdw_grid[i] = comp->types[i] < 64 ? grids[comp->types[i]] : nullptr;
  }
  p.ewald_grid = ewald_grid;
  p.quintic = rgd::systemScheme(system) == RG_SCHEME_TRIQUINTIC ? 1 : 0;
  p.rcv_fw2 = params->cutoff_framework_vdw * params->cutoff_framework_vdw;
  p.rcv_mol2 = params->cutoff_molecule_vdw * params->cutoff_molecule_vdw;
  p.rcc2 = params->cutoff_coulomb * params->cutoff_coulomb;
  p.beta = params->beta;
  p.fugacity = params->fugacity;
  p.volume = box.volume;
  p.max_translation = params->max_translation;
  p.max_rotation = params->max_rotation;
  p.p_translation = params->p_translation;
  p.p_rotation = params->p_rotation;
  p.p_swap = params->p_swap;
  p.k1 = params->n_first_bead_trials;
  p.k2 = params->n_orientation_trials;
  p.capacity = params->max_molecules;
  p.seed = params->seed;
  p.use_ewald = (ewald != nullptr && ff.use_charge) ? 1 : 0;
  int64_t nk = 0;
  const double2* s_rigid = nullptr;
  if (p.use_ewald)
  {
    double alpha, single_ion;
    const char4* kvec;
    const double* temp;
    st = rgd::ewaldExport(ewald, &kvec, &temp, &s_rigid, &nk, p.kmax, &alpha, &single_ion);
    if (st)
    {
      delete g;
      return st;
    }
    if (p.kmax[0] + 1 > kMaxK || p.kmax[1] + 1 > kMaxK || p.kmax[2] + 1 > kMaxK)
    {
      delete g;
      return rg::fail(ctx, RG_ERR_UNSUPPORTED, "rg_gcmc: kmax per axis at most 15");
    }
    // self + exclusion energy added by one inserted molecule (ewald.cpp:1164-1238, new-atom terms, scaling 1)
    const double C = rg::coulombFactor();
    double se = 0.0;
    const double pself = C * alpha / std::sqrt(rg::kPi);
    for (int i = 0; i < comp->n_atoms; ++i) se -= pself * comp->charges[i] * comp->charges[i];
    for (int i = 0; i < comp->n_atoms; ++i)
      for (int j = i + 1; j < comp->n_atoms; ++j)
      {
        double d2 = 0.0;
        for (int d = 0; d < 3; ++d)
        {
          const double dd = comp->offsets[3 * i + d] - comp->offsets[3 * j + d];
          d2 += dd * dd;
        }
        const double r = std::sqrt(d2);
        se -= C * comp->charges[i] * comp->charges[j] * std::erf(alpha * r) / r;
      }
    p.comp.self_excl = se;
    p.nk = nk;
  }
  // The structure factors and their change stay in shared memory where four CTAs still fit on an SM (the registers'
  // limit): at kmax 8 the 1,152 k-vectors of the sphere take 37 KB. Larger sets stay in global memory. 200 moves of 1,184
  // chains in a box of CO2 with the former kernel, all in global memory, and with this one: 13.5 and 5.5 ms at 1,182
  // k-vectors (shared now), 20.5 and 13.8 at 3,609 (global), 39.6 and 30.8 at 6,062; of 148 chains at 3,609 7.4 and 4.4.
  const size_t fixed = dynFixedBytes(comp->n_atoms, p.kmax, p.use_ewald != 0);
  const size_t sk_bytes = 2 * sizeof(double2) * static_cast<size_t>(nk);
  g->smem = fixed + sk_bytes <= kSharedPerCta;
  g->shmem = fixed + (g->smem ? sk_bytes : 0);
  if (p.use_ewald)
  {
    // the k-vectors as runs of kz, and their prefactors by (|kz|, sign, run)
    const std::vector<int4> runs = rgd::ewaldRuns(ewald);  // longest first: the threads of large |kz| are neighbours
    p.n_runs = static_cast<int>(runs.size());
    std::vector<double> rt;
    cudaError_t err = rgd::ewaldRunPrefactors(ewald, runs, rt);
    if (!err && !runs.empty()) err = cudaMalloc(reinterpret_cast<void**>(&g->runs), sizeof(int4) * runs.size());
    if (!err && !runs.empty()) err = cudaMalloc(reinterpret_cast<void**>(&g->run_temp), sizeof(double) * rt.size());
    if (!err && !runs.empty())
      err = cudaMemcpyAsync(g->runs, runs.data(), sizeof(int4) * runs.size(), cudaMemcpyHostToDevice, ctx->stream);
    if (!err && !runs.empty())
      err = cudaMemcpyAsync(g->run_temp, rt.data(), sizeof(double) * rt.size(), cudaMemcpyHostToDevice, ctx->stream);
    if (!err) err = cudaStreamSynchronize(ctx->stream);
    p.runs = g->runs;
    p.run_temp = g->run_temp;
    // all chains start from the framework structure factor
    const size_t skb = sizeof(double2) * static_cast<size_t>(nk) * n_chains;
    if (!err) err = cudaMalloc(reinterpret_cast<void**>(&p.sk), skb);
    if (!err && !g->smem) err = cudaMalloc(reinterpret_cast<void**>(&p.dsk), skb);
    for (int c = 0; c < n_chains && !err; ++c)
      err = cudaMemcpyAsync(p.sk + static_cast<size_t>(c) * nk, s_rigid, sizeof(double2) * nk,
                            cudaMemcpyDeviceToDevice, ctx->stream);
    if (err)
    {
      rg_gcmc_destroy(g);
      return rg::cudaFail(ctx, err, "rg_gcmc_create (structure factors)");
    }
  }
  const size_t posb = sizeof(double4) * static_cast<size_t>(n_chains) * p.capacity * comp->n_atoms;
  cudaError_t err = cudaMalloc(reinterpret_cast<void**>(&p.pos), posb);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&p.n), sizeof(int) * n_chains);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&p.energy), sizeof(double) * n_chains);
  if (!err) err = cudaMalloc(reinterpret_cast<void**>(&p.stats), sizeof(double) * kStats * n_chains);
  if (!err) err = cudaMemsetAsync(p.pos, 0, posb, ctx->stream);
  if (!err) err = cudaMemsetAsync(p.n, 0, sizeof(int) * n_chains, ctx->stream);
  if (!err) err = cudaMemsetAsync(p.energy, 0, sizeof(double) * n_chains, ctx->stream);
  if (!err) err = cudaMemsetAsync(p.stats, 0, sizeof(double) * kStats * n_chains, ctx->stream);
  if (!err) err = cudaStreamSynchronize(ctx->stream);
  if (err)
  {
    rg_gcmc_destroy(g);
    return rg::cudaFail(ctx, err, "rg_gcmc_create");
  }
  // The limit belongs to the kernel on the device, which the objects of all contexts share: the most that any of them
  // takes, so that no host thread lowers it between another's setting and launch.
  auto kern = p.quintic ? (g->smem ? gcmcKernel<true, true> : gcmcKernel<true, false>)
                        : (g->smem ? gcmcKernel<false, true> : gcmcKernel<false, false>);
  err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSharedPerCta));
  if (err)
  {
    rg_gcmc_destroy(g);
    return rg::cudaFail(ctx, err, "rg_gcmc_create");
  }
  *out = g;
  return RG_OK;
}

rg_status rg_gcmc_destroy(rg_gcmc* g)
{
  if (!g) return RG_OK;
  if (g->ctx) cudaStreamSynchronize(g->ctx->stream);
  cudaFree(g->p.pos);
  cudaFree(g->p.sk);
  cudaFree(g->p.dsk);
  cudaFree(g->p.n);
  cudaFree(g->p.energy);
  cudaFree(g->p.stats);
  cudaFree(g->runs);
  cudaFree(g->run_temp);
  delete g;
  return RG_OK;
}

rg_status rg_gcmc_run(rg_gcmc* g, int64_t moves, int record)
{
  if (!g || moves < 0) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = g->ctx;
  RG_CUDA(ctx, cudaSetDevice(ctx->device));
  if (record && g->block_len == 0) g->block_len = moves / 5 > 0 ? moves / 5 : 1;
  int64_t left = moves;
  while (left > 0)
  {
    const int chunk = static_cast<int>(left < g->max_moves_per_launch ? left : g->max_moves_per_launch);
    auto launch = [&](auto kern)
    {
      kern<<<g->n_chains, kThreads, g->shmem, ctx->stream>>>(g->p, g->moves_done, chunk, record, g->block_len);
      return cudaGetLastError();
    };
    RG_CUDA(ctx, g->p.quintic ? (g->smem ? launch(gcmcKernel<true, true>) : launch(gcmcKernel<true, false>))
                              : (g->smem ? launch(gcmcKernel<false, true>) : launch(gcmcKernel<false, false>)));
    g->moves_done += chunk;
    left -= chunk;
  }
  return RG_OK;
}

rg_status rg_gcmc_results(rg_gcmc* g, rg_gcmc_chain_result* out)
{
  if (!g || !out) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = g->ctx;
  std::vector<int> n(g->n_chains);
  std::vector<double> e(g->n_chains), s(static_cast<size_t>(kStats) * g->n_chains);
  RG_CUDA(ctx, cudaMemcpyAsync(n.data(), g->p.n, sizeof(int) * g->n_chains, cudaMemcpyDeviceToHost, ctx->stream));
  RG_CUDA(ctx, cudaMemcpyAsync(e.data(), g->p.energy, sizeof(double) * g->n_chains, cudaMemcpyDeviceToHost,
                               ctx->stream));
  RG_CUDA(ctx, cudaMemcpyAsync(s.data(), g->p.stats, sizeof(double) * s.size(), cudaMemcpyDeviceToHost, ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (int c = 0; c < g->n_chains; ++c)
  {
    rg_gcmc_chain_result& r = out[c];
    std::memset(&r, 0, sizeof(r));
    const double* q = &s[static_cast<size_t>(c) * kStats];
    r.n_molecules = n[c];
    r.energy = e[c];
    for (int k = 0; k < 4; ++k)
    {
      r.attempted[k] = static_cast<int64_t>(q[k]);
      r.accepted[k] = static_cast<int64_t>(q[4 + k]);
    }
    r.sum_n = q[8];
    r.sum_n2 = q[9];
    r.sum_energy = q[10];
    r.samples = static_cast<int64_t>(q[11]);
    for (int b = 0; b < 5; ++b) r.block_n[b] = g->block_len > 0 ? q[12 + b] / static_cast<double>(g->block_len) : 0.0;
  }
  return RG_OK;
}

rg_status rg_gcmc_get_positions(rg_gcmc* g, int chain, double* xyz, int capacity_atoms, int* n_molecules)
{
  if (!g || !xyz || !n_molecules || chain < 0 || chain >= g->n_chains) return RG_ERR_INVALID_ARGUMENT;
  rg_ctx* ctx = g->ctx;
  int n = 0;
  RG_CUDA(ctx, cudaMemcpyAsync(&n, g->p.n + chain, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  const int na = g->p.comp.n_atoms;
  if (n * na > capacity_atoms) return rg::fail(ctx, RG_ERR_INVALID_ARGUMENT, "rg_gcmc_get_positions: buffer too small");
  std::vector<double4> pos(static_cast<size_t>(n) * na);
  if (n > 0)
    RG_CUDA(ctx, cudaMemcpyAsync(pos.data(), g->p.pos + static_cast<size_t>(chain) * g->p.capacity * na,
                                 sizeof(double4) * n * na, cudaMemcpyDeviceToHost, ctx->stream));
  RG_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (int i = 0; i < n * na; ++i)
  {
    xyz[3 * i] = pos[i].x;
    xyz[3 * i + 1] = pos[i].y;
    xyz[3 * i + 2] = pos[i].z;
  }
  *n_molecules = n;
  return RG_OK;
}
}

extern "C" rg_status rg_gcmc_set_proposal(rg_gcmc* g, rg_proposal* proposal, const rg_box* unit_cell)
{
  if (!g) return RG_ERR_INVALID_ARGUMENT;
  Params& p = g->p;
  if (!proposal)
  {
    p.prop_cdf = nullptr;
    p.prop_q = nullptr;
    return RG_OK;
  }
  if (!unit_cell) return RG_ERR_INVALID_ARGUMENT;
  rg_status st = rgd::proposalExport(proposal, &p.prop_cdf, &p.prop_q, &p.prop_G, &p.prop_eps);
  if (st) return st;
  const rg::HostBox ub = rg::makeHostBox(unit_cell);
  for (int a = 0; a < 3; ++a)
    for (int b = 0; b < 3; ++b)
    {
      p.uc[a][b] = ub.c[a][b];
      p.uic[a][b] = ub.ic[a][b];
    }
  // the simulation box must be an integer replication of the unit cell along each lattice vector
  for (int d = 0; d < 3; ++d)
  {
    double ratio = 0.0, n2 = 0.0;
    for (int r = 0; r < 3; ++r)
    {
      ratio += p.box.c[d][r] * ub.c[d][r];
      n2 += ub.c[d][r] * ub.c[d][r];
    }
    ratio /= n2;
    const int rep = static_cast<int>(std::lround(ratio));
    double err = 0.0;
    for (int r = 0; r < 3; ++r) err += std::fabs(p.box.c[d][r] - rep * ub.c[d][r]);
    if (rep < 1 || err > 1e-6)
    {
      p.prop_cdf = nullptr;
      p.prop_q = nullptr;
      return rg::fail(g->ctx, RG_ERR_INVALID_ARGUMENT, "rg_gcmc_set_proposal: box is not a replication of the unit cell");
    }
    p.rep[d] = rep;
  }
  return RG_OK;
}
