// Execution policies shared by the persistent kernels: which threads work on one problem and how
// its phases are separated.
#pragma once
#include "common.cuh"

namespace sa {

// sync runs an epilogue on the last CTA to arrive before the others leave; meet only waits for all of
// them (epoch: the caller's count of them, from first_epoch).
//
// GridPolicy: one problem on the whole grid. A cooperative grid separates phases on the control block's
// GridSync; a grid that is one cluster (cluster = 1, only meet is used) by the cluster's barrier.
struct GridPolicy {
  static constexpr bool kShareRitz = false;      // every CTA runs the Ritz test itself
  static constexpr bool kManyPositions = false;  // positions of the vector phases are shared by lanes, or streamed
  int cluster = 0;
  __device__ __forceinline__ long long tid() const { return (long long)blockIdx.x * blockDim.x + tid_here(); }
  __device__ __forceinline__ long long nthr() const { return (long long)gridDim.x * blockDim.x; }
  __device__ __forceinline__ int block() const { return blockIdx.x; }
  __device__ __forceinline__ int nblocks() const { return gridDim.x; }
  template <class E>
  __device__ __forceinline__ bool sync(GridSync* gs, E&& e) const { return grid_barrier(gs, e); }
  __device__ __forceinline__ bool sync(GridSync* gs) const { return grid_barrier(gs); }
  __device__ __forceinline__ unsigned int first_epoch(GridSync*) const { return 0; }   // zeroed before the launch
  __device__ __forceinline__ bool meet(GridSync* gs, unsigned int& epoch) const {
    if (cluster) {
      cluster_arrive_wait();
      return true;
    }
    return grid_arrive_wait(gs, gridDim.x, epoch);
  }
};

// TeamPolicy: one problem on the CTAs [b0, b0 + nb) of a cooperative grid (batched solves: every
// team works through its own list of problems). Phases are separated by a barrier of the nb CTAs
// on the team's own GridSync (the control block's is not used); a team of one CTA uses
// __syncthreads, with the epilogue run by the whole CTA.
struct TeamPolicy {
  // The team's first CTA runs the Ritz test for all: four CTAs share an SM's FP64 units here, and the
  // redundant tests cost more than the barrier that hands the result over (a sweep of
  // twelve problems, n to 16,346: 104 ms with a test in every CTA, 100 ms with one a team).
  static constexpr bool kShareRitz = true;
  static constexpr bool kManyPositions = true;   // a team of few CTAs has many positions a thread
  int b0, nb;
  GridSync* gs;
  __device__ __forceinline__ long long tid() const { return (long long)(blockIdx.x - b0) * blockDim.x + tid_here(); }
  __device__ __forceinline__ long long nthr() const { return (long long)nb * blockDim.x; }
  __device__ __forceinline__ int block() const { return (int)blockIdx.x - b0; }
  __device__ __forceinline__ int nblocks() const { return nb; }
  template <class E>
  __device__ __forceinline__ bool sync(GridSync*, E&& e) const {
    if (nb == 1) {
      __syncthreads();
      e();
      __syncthreads();
      return true;
    }
    return grid_barrier_n(gs, (unsigned int)nb, [&] {
      // (every CTA of the team has left its last meet)
      if (threadIdx.x == 0) *((volatile unsigned int*)&gs->arrivals) = 0u;
      e();
    });
  }
  __device__ __forceinline__ bool sync(GridSync* g) const { return sync(g, [] {}); }
  // A solve and a search are followed by sync, which sets the counter back (left to run on, it would pass
  // 2^32 in a long run, and the number of barriers could not be had from it any more).
  __device__ __forceinline__ unsigned int first_epoch(GridSync*) const { return 0; }
  __device__ __forceinline__ bool meet(GridSync*, unsigned int& epoch,
                                       unsigned long long spin_limit = kSpinLimit) const {
    if (nb == 1) {
      __syncthreads();
      return true;
    }
    return grid_arrive_wait(gs, (unsigned int)nb, epoch, spin_limit);
  }
};

}  // namespace sa
