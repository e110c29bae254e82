// Shared device helpers for the SpecAnn kernels (sm_100a).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/specann_b200.h"

namespace sa {

constexpr int kThreads = 512;             // threads per CTA of the persistent kernels
constexpr int kWarps = kThreads / 32;
constexpr int kShortMax = 64;             // rows with at most this many entries are "short"
constexpr int kChunk = 256;               // entries per chunk of a long row
constexpr int kSegMax = 256;              // entries per short segment at most (= one warp tile)
constexpr int kSegRows = 64;              // rows per short segment at most
constexpr int kTileIt = kSegMax / 32;     // entries per lane of a tile
constexpr int kNcvMax = 64;               // largest Lanczos basis
// Polls after which a barrier wait gives up. A poll is a round trip to L2 and, in grid_barrier_n, a sleep of
// about 64 ns as well: some tens of seconds, well above what one CTA can make the others wait.
constexpr unsigned long long kSpinLimit = 1ull << 25;
constexpr int kMaxSplits = 8;             // column splits of an operator larger than L2 (split.cu)

// One tile of the SpMV work list: at most kSegMax stored entries starting at e0.
//   row >= 0: a short segment of rows [row, row + nrows);
//   row < 0:  a chunk of the long row -(row + 1).
//   meta bits 0-8: entries in the tile; segment: bits 9-15 nrows; chunk: bits 9-31 hold
//   (multi-chunk row id + 1), 0 when the row fits in one chunk.
struct WorkItem {
  long long e0;
  int row;
  int meta;
};
__host__ __device__ __forceinline__ int item_len(int meta) { return meta & 511; }
__host__ __device__ __forceinline__ int item_nrows(int meta) { return (meta >> 9) & 127; }
__host__ __device__ __forceinline__ int item_mc(int meta) { return (int)((unsigned)meta >> 9) - 1; }

// Device-resident synchronisation block of a persistent kernel (zeroed before launch).
struct GridSync {
  unsigned int count;
  unsigned int gen;
  int error;
  unsigned int arrivals;   // CTAs that have arrived at grid_arrive_wait since the block was zeroed
};

__device__ __forceinline__ unsigned int ld_volatile_u32(const unsigned int* p) {
  return *((volatile const unsigned int*)p);
}
__device__ __forceinline__ int ld_volatile_i32(const int* p) {
  return *((volatile const int*)p);
}

// Barrier of `expected` co-resident CTAs (a cooperative grid, or a team of CTAs inside one),
// with an epilogue run by the last CTA to arrive (the whole CTA runs it, after every other CTA's
// writes are visible) before the others are released. Waits are bounded: after spin_limit polls
// the barrier records SA_ERR_BARRIER_TIMEOUT in gs->error and returns false, and a waiting CTA
// also stops as soon as another CTA has recorded an error; the caller must then return. The
// decision is taken by thread 0 and shared through shared memory, so the whole CTA returns the
// same value.
template <class Epilogue>
__device__ __forceinline__ bool grid_barrier_n(GridSync* gs, unsigned int expected, Epilogue&& epi,
                                               unsigned long long spin_limit = kSpinLimit) {
  __shared__ unsigned int s_last, s_gen;
  __shared__ int s_err;
  __syncthreads();
  if (threadIdx.x == 0) {
    s_gen = ld_volatile_u32(&gs->gen);
    __threadfence();
    unsigned int arrived = atomicAdd(&gs->count, 1u);
    s_last = (arrived == expected - 1) ? 1u : 0u;
    s_err = 0;
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    epi();
    __syncthreads();
    if (threadIdx.x == 0) {
      gs->count = 0;
      __threadfence();
      atomicAdd(&gs->gen, 1u);
      if (ld_volatile_i32(&gs->error)) s_err = 1;
    }
  } else if (threadIdx.x == 0) {
    unsigned long long spins = 0;
    while (ld_volatile_u32(&gs->gen) == s_gen) {
      __nanosleep(64);
      if (ld_volatile_i32(&gs->error)) break;
      if (++spins > spin_limit) {
        atomicExch(&gs->error, SA_ERR_BARRIER_TIMEOUT);
        break;
      }
    }
    __threadfence();
    if (ld_volatile_i32(&gs->error)) s_err = 1;
  }
  __syncthreads();
  return s_err == 0;
}

template <class Epilogue>
__device__ __forceinline__ bool grid_barrier(GridSync* gs, Epilogue&& epi) {
  return grid_barrier_n(gs, gridDim.x, epi);
}

__device__ __forceinline__ bool grid_barrier(GridSync* gs) {
  return grid_barrier_n(gs, gridDim.x, [] {});
}

// Barrier of `expected` co-resident CTAs without an epilogue: every CTA adds one to a counter that is
// never reset and waits until it reaches epoch * expected (epoch: this CTA's number of barriers, the
// same in every thread). A CTA leaves as soon as the last one has arrived, one L2 round trip earlier
// than from grid_barrier_n, whose last CTA works alone first and then releases the others. Waits are
// bounded in the same way (after spin_limit polls the barrier records SA_ERR_BARRIER_TIMEOUT and
// returns false, as it does when another CTA has recorded an error).
__device__ __forceinline__ bool grid_arrive_wait(GridSync* gs, unsigned int expected, unsigned int& epoch,
                                                 unsigned long long spin_limit = kSpinLimit) {
  __shared__ int s_fail;
  __syncthreads();
  ++epoch;
  if (threadIdx.x == 0) {
    int fail = 0;
    __threadfence();
    atomicAdd(&gs->arrivals, 1u);
    const unsigned int target = epoch * expected;
    unsigned long long polls = 0;
    while ((int)(ld_volatile_u32(&gs->arrivals) - target) < 0) {
      if ((++polls & 63) != 0) continue;
      if (ld_volatile_i32(&gs->error)) { fail = 1; break; }
      if (polls > 4096) __nanosleep(64);
      if (polls > spin_limit) {
        atomicExch(&gs->error, SA_ERR_BARRIER_TIMEOUT);
        fail = 1;
        break;
      }
    }
    __threadfence();
    s_fail = fail;
  }
  __syncthreads();
  return s_fail == 0;
}

// Barrier of all CTAs of this CTA's cluster (hardware; about 0.25 us), with the ordering of global
// memory among them that a grid barrier gives.
__device__ __forceinline__ void cluster_arrive_wait() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// threadIdx.x, read again where it is called: what a phase of a persistent kernel derives from it is
// computed in the phase, instead of being hoisted out of the kernel's loop and held in registers (or
// spilled) across all the other phases.
__device__ __forceinline__ int tid_here() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}

// Device clock in ns (phase timers of the persistent kernels).
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ---------------------------------------------------------------------------------------------
// Counter-based random streams (identical to oracle/selection.py and the host code).
// ---------------------------------------------------------------------------------------------
constexpr unsigned long long kSelSalt = 0x5E1EC7ED5EED0001ull;
constexpr long long kFinalStreamBase = 1ll << 20;

__host__ __device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  unsigned long long z = x;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

struct SelKeys {
  unsigned long long k[4];
  unsigned long long mask;
  unsigned int shift;
};

__host__ __device__ inline int domain_bits(long long n) {
  int b = 0;
  unsigned long long v = (unsigned long long)(n - 1);
  while (v) { ++b; v >>= 1; }
  return b < 1 ? 1 : b;
}

__host__ __device__ inline SelKeys make_sel_keys(unsigned long long seed, long long stream, long long n) {
  SelKeys s;
  unsigned long long base = splitmix64(seed ^ kSelSalt);
  for (int r = 0; r < 4; ++r) s.k[r] = splitmix64(base + 4ull * (unsigned long long)stream + (unsigned long long)r);
  int b = domain_bits(n);
  s.mask = (b >= 64) ? ~0ull : ((1ull << b) - 1ull);
  s.shift = (unsigned int)((b + 1) / 2);
  return s;
}

__host__ __device__ __forceinline__ unsigned long long sel_perm(unsigned long long x, const SelKeys& s) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const unsigned long long add = s.k[r] & s.mask;
    const unsigned long long mul = ((s.k[r] >> 32) | 1ull) & 0xFFFFFFFFull;
    x = (x + add) & s.mask;
    x = (x * mul) & s.mask;
    x = x ^ (x >> s.shift);
  }
  return x;
}

// rank(i): a bijection of [0, n) (cycle walking; terminates because i's cycle contains i < n).
__host__ __device__ __forceinline__ long long sel_rank(long long i, const SelKeys& s, long long n) {
  unsigned long long y = sel_perm((unsigned long long)i, s);
  while (y >= (unsigned long long)n) y = sel_perm(y, s);
  return (long long)y;
}

// Standard normal from a counter (Box-Muller on two 53-bit uniforms in (0, 1]).
__device__ __forceinline__ double normal_from_counter(unsigned long long key, long long i) {
  const unsigned long long h1 = splitmix64(key ^ (2ull * (unsigned long long)i));
  const unsigned long long h2 = splitmix64(key ^ (2ull * (unsigned long long)i + 1ull));
  const double u1 = ((double)(h1 >> 11) + 1.0) * (1.0 / 9007199254740992.0);
  const double u2 = (double)(h2 >> 11) * (1.0 / 9007199254740992.0);
  return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

// ---------------------------------------------------------------------------------------------
// Reductions (fixed order: results do not depend on timing).
// ---------------------------------------------------------------------------------------------
template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <int G, typename T>
__device__ __forceinline__ T group_sum(T v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum of one double (all threads get the result). Uses a kWarps scratch array.
__device__ __forceinline__ double block_sum(double v, double* scratch) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (wid == 0) {
    t = (lane < (int)(blockDim.x >> 5)) ? scratch[lane] : 0.0;
    t = warp_sum(t);
    if (lane == 0) scratch[0] = t;
  }
  __syncthreads();
  t = scratch[0];
  __syncthreads();
  return t;
}

__device__ __forceinline__ long long rp_load(const int* rp, long long i) { return (long long)__ldg(rp + i); }
__device__ __forceinline__ long long rp_load(const long long* rp, long long i) { return __ldg(rp + i); }

// ---- a kernel launched behind the one that prepares its input ----------------------------------
// The standalone operator is two kernels, the scaling of x and the SpMV. The SpMV's launch (its CTAs with
// their shared memory) runs while the scaling still works; its threads wait here before they read
// anything that the scaling writes. Without the launch attribute both calls do nothing. Operator at
// n = 2^20 125.2 -> 119.9 us, at n = 150,001 with values in +-1..100 28.7 -> 26.7 us (panels, one CTA per SM:
// launched as the scaling starts). The work list's CTAs, two per SM, are launched as it ends: earlier they
// find room only beside the scaling's and are spread unevenly (BA(100000, 10) 20.9 us one after the
// other, 22.2 launched early, 18.5 launched late; in FP64 26.7, 28.4 and 24.6).
__device__ __forceinline__ void allow_dependent() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline cudaError_t launch_behind(void (*kernel)(KArgs...), int grid, int threads, int smem, cudaStream_t stream,
                                 Args... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

}  // namespace sa
