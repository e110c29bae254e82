// Diagnostics of parts of the persistent kernels by themselves: the barrier between their phases
// (sa_meet_selftest), and the streamed vector phases (sa_stream_selftest), one CTA each over its range
// of rows, without the rest of a Lanczos step.
#include <algorithm>

#include "alpha_body.cuh"

namespace sa {

namespace {

// A team's solves of `meets` barriers each. tick counts the CTAs that came to a barrier, words[b] says
// whether CTA b passed them all (bit 0) and whether it left one before every CTA had come (bit 1).
__global__ void meet_selftest_kernel(GridSync* gs, unsigned int* tick, int nb, int solves, int meets,
                                     unsigned int first_epoch, unsigned long long spin_limit, int* words) {
  const TeamPolicy pol{0, nb, gs};
  bool ok = true, early = false;
  unsigned int before = 0;   // CTAs that have to come before this barrier ends
  for (int s = 0; s < solves && ok; ++s) {
    if (s > 0) ok = pol.sync(gs);
    unsigned int epoch = s > 0 ? pol.first_epoch(gs) : first_epoch;
    for (int m = 0; m < meets && ok; ++m) {
      if (threadIdx.x == 0) atomicAdd(tick, 1u);
      before += (unsigned int)gridDim.x;
      ok = pol.meet(gs, epoch, spin_limit);
      if (ok && ld_volatile_u32(tick) < before) early = true;
    }
    __syncthreads();
  }
  const int any = __syncthreads_or(early);
  if (threadIdx.x == 0) words[blockIdx.x] = (ok ? 1 : 0) | (any ? 2 : 0);
}

template <typename T, int kBufs>
__global__ void __launch_bounds__(kThreads, 1) stream_selftest_kernel(const __grid_constant__ sa_stream_test P,
                                                                     unsigned long long spin_limit, int* words) {
  extern __shared__ __align__(128) char stream_smem[];
  __shared__ unsigned long long bars[kBufs];
  __shared__ double dots[kWarps * kPartCols];
  __shared__ double h[kNcvMax];
  constexpr int VW = 16 / sizeof(T);
  const T* V = (const T*)P.V;
  const int j = P.j;
  if (threadIdx.x == 0) {
    // (a second arrival that nothing makes: the copies land, but no wait for them ends)
    for (int q = 0; q < kBufs; ++q) mbar_init(&bars[q], P.withhold ? 2 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int k = threadIdx.x; k <= j; k += blockDim.x) h[k] = P.h[k];
  __syncthreads();
  unsigned par = 0;
  VecStream<T, kBufs> S(stream_smem, bars, par, words, (P.n + VW - 1) / VW * VW, blockIdx.x, gridDim.x);
  S.spin_limit = spin_limit;
  bool ok = stream_dots(S, V, P.ldv, (const T*)P.w, (T*)P.u, j, 0, P.a3, P.b3, dots);
  if (ok) {
    __syncthreads();
    for (int c = threadIdx.x; c <= j + 1; c += blockDim.x) {
      double acc = 0.0;
      for (int w = 0; w < kWarps; ++w) acc += dots[w * kPartCols + c];
      P.dots[(long long)blockIdx.x * (j + 2) + c] = acc;
    }
    __threadfence();   // w' in u, read back by the copies of the update
    __syncthreads();
    double ww = 0.0;
    ok = stream_update(S, V, P.ldv, (const T*)P.u, (const T*)P.sigma, (T*)P.w, (T*)P.u, j, h, ww);
  }
  if (threadIdx.x == 0) {
    words[1 + blockIdx.x] = ok ? 1 : 0;
    if (P.withhold && S.tiles) {
      // the withheld arrivals, then the copies still in flight
      const int groups = (j + 2 + kStreamVecs - 1) / kStreamVecs * S.tiles;
      for (int q = 0; q < kBufs && q < groups; ++q) {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&bars[q])) : "memory");
        for (unsigned long long spins = 0; !mbar_try_wait(&bars[q], 0);)
          if (++spins > kPanelSpinLimit) break;
      }
    }
  }
}

template <typename T, int kBufs>
int run_stream_selftest(const sa_stream_test& P, unsigned long long spin_limit, int blocks, int* words, cudaStream_t st) {
  auto k = stream_selftest_kernel<T, kBufs>;
  const int smem = kBufs * kStreamVecs * kStreamTile;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return SA_ERR_CUDA;
  k<<<blocks, kThreads, smem, st>>>(P, spin_limit, words);
  count_launches(1);
  return cudaGetLastError() == cudaSuccess ? SA_OK : SA_ERR_CUDA;
}

}  // namespace

}  // namespace sa

using namespace sa;

extern "C" int sa_meet_selftest(int32_t blocks, int32_t expected, int32_t solves, int32_t meets, uint32_t first_epoch,
                                uint64_t spin_limit, void* scratch, size_t scratch_bytes, int32_t* status,
                                int32_t* passed_blocks, int32_t* early_blocks, void* stream) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return SA_ERR_CUDA;
  const size_t head = sizeof(GridSync) + 16;
  if (blocks < 1 || blocks > sms || expected < blocks || solves < 1 || solves > 1000 || meets < 1 || meets > 1000 ||
      spin_limit < 1 || spin_limit > kSpinLimit || !scratch || ((uintptr_t)scratch & 15) ||
      scratch_bytes < head + 4 * (size_t)blocks || !status || !passed_blocks || !early_blocks)
    return SA_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  GridSync gs = {};
  gs.arrivals = first_epoch * (uint32_t)expected;
  int* words = (int*)((char*)scratch + head);
  int32_t host[1024];
  if (cudaMemsetAsync(scratch, 0, head + 4 * (size_t)blocks, st) != cudaSuccess ||
      cudaMemcpyAsync(scratch, &gs, sizeof(gs), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return SA_ERR_CUDA;
  meet_selftest_kernel<<<blocks, 128, 0, st>>>((GridSync*)scratch, (unsigned int*)((char*)scratch + sizeof(GridSync)),
                                               expected, solves, meets, first_epoch, spin_limit, words);
  count_launches(1);
  if (cudaGetLastError() != cudaSuccess ||
      cudaMemcpyAsync(&gs, scratch, sizeof(gs), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaMemcpyAsync(host, words, 4 * (size_t)blocks, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return SA_ERR_CUDA;
  *status = gs.error;
  *passed_blocks = *early_blocks = 0;
  for (int b = 0; b < blocks; ++b) {
    *passed_blocks += host[b] & 1;
    *early_blocks += (host[b] >> 1) & 1;
  }
  return SA_OK;
}

extern "C" int sa_stream_selftest(const sa_stream_test* p, int32_t* words, int32_t* status, int32_t* passed_blocks,
                                  void* stream) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return SA_ERR_CUDA;
  if (!p || !words || !status || !passed_blocks || (p->precision != 32 && p->precision != 64) || p->buffers < 1 ||
      p->buffers > 3 || p->blocks < 1 || p->blocks > sms || p->j < 0 || p->j >= kNcvMax || p->n < 1 || p->ldv < p->n ||
      (p->ldv * (p->precision / 8)) % 16 != 0 || !p->V || !p->w || !p->u || !p->sigma || !p->h || !p->dots ||
      (((uintptr_t)p->V | (uintptr_t)p->w | (uintptr_t)p->u | (uintptr_t)p->sigma) & 15) || p->spin_limit < 1 ||
      p->spin_limit > kPanelSpinLimit)
    return SA_ERR_INVALID_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(words, 0, 4 * (size_t)(1 + p->blocks), st) != cudaSuccess) return SA_ERR_CUDA;
  int rc;
  if (p->precision == 32) {
    rc = p->buffers == 1   ? run_stream_selftest<float, 1>(*p, p->spin_limit, p->blocks, words, st)
         : p->buffers == 2 ? run_stream_selftest<float, 2>(*p, p->spin_limit, p->blocks, words, st)
                           : run_stream_selftest<float, 3>(*p, p->spin_limit, p->blocks, words, st);
  } else {
    rc = p->buffers == 1   ? run_stream_selftest<double, 1>(*p, p->spin_limit, p->blocks, words, st)
         : p->buffers == 2 ? run_stream_selftest<double, 2>(*p, p->spin_limit, p->blocks, words, st)
                           : run_stream_selftest<double, 3>(*p, p->spin_limit, p->blocks, words, st);
  }
  if (rc != SA_OK) return rc;
  int32_t host[1 + 1024];
  if (cudaMemcpyAsync(host, words, 4 * (size_t)(1 + p->blocks), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return SA_ERR_CUDA;
  *status = host[0];
  *passed_blocks = 0;
  for (int b = 0; b < p->blocks; ++b) *passed_blocks += host[1 + b];
  return SA_OK;
}
