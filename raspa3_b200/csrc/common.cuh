// Shared host/device helpers of libraspagpu: the context, error plumbing, device scratch and small math.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "../../include/raspa_gpu.h"

struct rg_ctx
{
  int device = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  std::string last_error;
  // Grow-only device scratch slots, reused across calls on this context.
  struct Slot
  {
    void* ptr = nullptr;
    size_t bytes = 0;
  };
  std::vector<Slot> scratch;
  // Pinned host staging slots.
  std::vector<Slot> pinned;
  // Second stream for device-to-host copies that overlap the work of `stream`, and events to order the two (created
  // on first use).
  cudaStream_t copy_stream = nullptr;
  std::vector<cudaEvent_t> events;
  // The device memory of a tabulated proposal that was destroyed, for the next one (one buffer of up to 64 MB, freed with
  // the context): freeing and mapping it anew took 1 to 5 ms when nothing else held its pages.
  Slot spare_table;
  // Recorded behind the last kernel of a call that returned before the stream was done with it (rg::leave), until the
  // stream is changed: the next stream's work comes after it.
  cudaEvent_t left = nullptr;
  bool left_pending = false;
};

namespace rg
{
constexpr double kPi = 3.141592653589793238462643383279502884;
constexpr double kInvSqrtPi = 0.564189583547756286948079451560772586;

// Unit constants with the reference's expressions (src/raspakit/units.cpp:14-98).
inline double energyConversionFactor() { return 1.6605402e-27 * 1e-10 * 1e-10 / (1e-12 * 1e-12); }
inline double coulombFactor()
{
  return 1.60217733e-19 * 1.60217733e-19 / (4.0 * kPi * 8.8541878176e-12 * 1e-10 * energyConversionFactor());
}

rg_status fail(rg_ctx* ctx, rg_status code, const std::string& msg);
rg_status cudaFail(rg_ctx* ctx, cudaError_t err, const char* what);
// Device scratch slot `slot` of at least `bytes` (grows; contents undefined).
rg_status scratch(rg_ctx* ctx, int slot, size_t bytes, void** out);
// Pinned host slot `slot` of at least `bytes`.
rg_status pinnedScratch(rg_ctx* ctx, int slot, size_t bytes, void** out);
// The context's copy stream and its event `i` (created on first use).
rg_status copyStream(rg_ctx* ctx, cudaStream_t* out);
rg_status event(rg_ctx* ctx, int i, cudaEvent_t* out);
// Makes the context stream wait for everything queued on the copy stream so far.
rg_status joinCopies(rg_ctx* ctx);

// Marks the end of the work that a call leaves on the stream when it returns: results that are posted (rg::post) say
// nothing of the kernel's other stores, nor of the counters that it resets behind them. On the same stream the next kernel
// comes after them all; rg_ctx_set_stream waits for the mark. A stream that is being captured is refused.
rg_status leave(rg_ctx* ctx);

// Takes n results that the kernels of call number `call` post (rg::post) into mapped host memory `from`, as soon as each
// is there. A launch that failed, or a stream that cannot be waited for (one being captured), ends the wait with its
// error.
rg_status collect(rg_ctx* ctx, const ulonglong2* from, int n, unsigned int call, double* out, const char* what);

// RG_ERR_NONFINITE (with a message naming `what`) if any position, charge or scaling factor of the atoms is NaN or
// infinite, RG_OK otherwise. Host inputs are checked before anything is launched.
rg_status checkFinite(rg_ctx* ctx, const rg_atom* atoms, long long n, const char* what);
rg_status checkFiniteBox(rg_ctx* ctx, const rg_box* box, const char* what);

struct HostBox
{
  double c[3][3];   // c[col][row]
  double ic[3][3];  // inverse, same convention
  bool triclinic;
  double volume;
};
HostBox makeHostBox(const rg_box* b);
void perpendicularWidths(const HostBox& b, double w[3]);
// The supercell that `cutoff` sizes in the reference's grid builds (ceil(2 cutoff / width) unit cells per axis,
// SimulationBox::smallestNumberOfUnitCellsForMinimumImagesConvention, simulationbox.cpp:150-156): half its lengths
// (h, rectangular) and its inverse as ic[d][k] (fraction d from Cartesian k). Returns whether its minimum image can
// drop pairs within the pair cutoff `rc`, i.e. whether it is narrower than 2 rc along some axis.
bool supercellClip(const HostBox& b, double rc, double cutoff, double h[3], double ic[3][3]);
inline void matvec(const double m[3][3], const double v[3], double out[3])
{
  for (int r = 0; r < 3; ++r) out[r] = m[0][r] * v[0] + m[1][r] * v[1] + m[2][r] * v[2];
}
}  // namespace rg

#define RG_CUDA(ctx, call)                                   \
  do                                                         \
  {                                                          \
    cudaError_t _e = (call);                                 \
    if (_e != cudaSuccess) return rg::cudaFail(ctx, _e, #call); \
  } while (0)

namespace rg
{
// Counts a block in at the end of its part, by one thread behind a barrier of the block, and returns how many were in
// before: what the block has written is visible to whoever counts in later. (__threadfence before a relaxed atomic is a
// sequentially consistent fence: with 290 blocks ending together it took 2,000 to 9,000 cycles.)
__device__ __forceinline__ unsigned int countIn(unsigned int* counter)
{
  unsigned int before;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(counter) : "memory");
  return before;
}

// A result for the host (rg::collect): two 64-bit words, each half of the value beside the call's number, so that the
// host knows by itself when a value has arrived. A flag written after the values needs a system-wide fence before it,
// which waits for the bus: the trial energies of 10 positions against 12,000 sites spent 8 of 15 us of their kernel in two
// of them.
__device__ __forceinline__ void post(ulonglong2* to, double x, unsigned int call)
{
  const unsigned long long v = static_cast<unsigned long long>(__double_as_longlong(x));
  const unsigned long long t = static_cast<unsigned long long>(call) << 32;
  asm volatile("st.relaxed.sys.global.v2.u64 [%0], {%1, %2};" ::"l"(to), "l"(t | (v & 0xffffffffull)), "l"(t | (v >> 32))
               : "memory");
}
}  // namespace rg

// Block-wide exclusive scan of one int per thread (blockDim.x a multiple of 32, <= 1024). `warp_sums` is shared
// scratch of 33 ints; callers separate two scans with a __syncthreads. Returns the exclusive prefix; *total receives the block sum. Contains two __syncthreads.
__device__ __forceinline__ int blockExclusiveScan(int v, int* warp_sums, int* total)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
  {
    int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0)
  {
    int w = (lane < nwarps) ? warp_sums[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
      int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    if (lane < nwarps) warp_sums[lane] = wi - w;  // exclusive warp offsets
    if (lane == nwarps - 1) warp_sums[32] = wi;   // block total
  }
  __syncthreads();
  int res = warp_sums[warp] + incl - v;
  *total = warp_sums[32];
  return res;
}
