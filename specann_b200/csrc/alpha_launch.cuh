// The alpha-solve kernel and its launch (device code in alpha_body.cuh), instantiated per precision in
// alpha_f32.cu and alpha_f64.cu.
#pragma once
#include <algorithm>

#include "alpha_body.cuh"

namespace sa {

PanelArgs panel_args(const sa_handle* h);
template <typename T, typename RP>
SpmvArgs<T, RP> split_args(const sa_handle* h, int s);

template <typename T, typename RP, int kMode>
__global__ void __launch_bounds__(kThreads, 1) alpha_kernel(const __grid_constant__ AlphaArgs<T, RP> A) {
  alpha_body<T, RP, GridPolicy, kWarps, kMode>(A, GridPolicy{A.cluster});
}

// ---- host side ------------------------------------------------------------------------------

template <typename T, typename RP>
const void* alpha_kernel_of(int mode) {
  if (mode == ALPHA_PANEL) return (const void*)alpha_kernel<T, RP, ALPHA_PANEL>;
  if (mode == ALPHA_PANEL_SMALL) return (const void*)alpha_kernel<T, RP, ALPHA_PANEL_SMALL>;
  if (mode == ALPHA_LARGE) return (const void*)alpha_kernel<T, RP, ALPHA_LARGE>;
  return (const void*)alpha_kernel<T, RP, ALPHA_SMALL>;
}

// Vector phases streamed through shared memory when a thread has more than half a 16-byte position of
// the vectors, held in registers below. One step's dots and update at n = 2^16 in FP64 (43 % of a
// position): 16.9 us in registers, 24 us streamed; at n = 2^20 in FP32 (346 %): 71 us in registers
// (85 us where they spill), 52.5 us streamed; with panels at n = 2^16 in FP32 (22 %): 18.4 against 26.3 us.
inline int alpha_mode(const sa_handle* h) {
  const long long positions = h->n * (h->prec == 32 ? 4 : 8) / 16;
  const bool large = 2 * positions > (long long)h->blocks * kThreads;
  if (h->panel_on) return large ? ALPHA_PANEL : ALPHA_PANEL_SMALL;
  return h->split_on || large ? ALPHA_LARGE : ALPHA_SMALL;
}

// CTAs of the one cluster that a problem runs on, 0 for the whole (cooperative) grid. A cluster's hardware
// barrier takes 0.25 us where the grid's takes over 1 us, but only 8 or 16 SMs work: it pays while
// every warp has at most one tile of the work list. One alpha, grid against cluster: ER(1024) 1.37
// against 1.18 ms, ER(2500) 1.53 against 1.35 ms, ER(4000), at 1.5 tiles a warp, 1.75 against 1.71 ms,
// in FP64 1.76 against 1.79 ms.
inline int alpha_cluster(const sa_handle* h) {
  if (h->n_items <= 8 * kWarps) return 8;
  return h->n_items <= 16 * kWarps ? 16 : 0;
}

template <typename T, typename RP>
int launch_alpha(sa_handle* h, const sa_alpha_params* p) {
  AlphaArgs<T, RP> A;
  A.S.rowptr = (const RP*)h->rowptr;
  A.S.col = h->col;
  A.S.val = (const T*)h->val;
  A.S.items = h->items;
  A.S.n_items = h->n_items;
  A.S.mc_base = h->mc_base;
  A.S.mc_count = h->mc_count;
  A.S.long_part = (T*)h->long_part;
  A.S.scol = h->packed ? h->scol : nullptr;
  A.S.wmag = (T)h->wmag;
  A.n = h->n;
  A.ldv = h->ldv;
  A.sigma = (T*)h->sigma;
  A.ld = h->ld;
  A.aoff = h->aoff;
  A.V = (T*)h->V;
  A.w = (T*)h->w;
  A.u = (T*)h->u;
  A.ylast = (const T*)h->yv[h->iy_last];
  A.yprev = (const T*)h->yv[h->iy_prev];
  A.yout = (T*)h->yv[h->iy_out];
  A.v0 = (const T*)p->v0;
  A.part = h->blk_part;
  A.ctrl = h->actrl;
  A.bits = h->scratch;
  A.W = h->W;
  A.p = *p;
  A.has_last = h->has_last ? 1 : 0;
  A.has_prev = h->has_prev ? 1 : 0;
  A.half_log2_c = 0.5 * std::log2(h->c);
  A.sqrt_c = std::sqrt(h->c);
  A.group = h->group;
  A.dense = h->dense;
  // Algorithmic bytes of one operator application, whatever the layout: the CSR (column + value per
  // entry, row pointers) and the vectors x, sigma, y. The panel and split layouts stream their own
  // (smaller or larger) encodings; the roofline is stated against this figure.
  A.spmv_bytes = (double)h->nnz * (4.0 + sizeof(T)) + (double)(h->n + 1) * sizeof(RP) + 3.0 * (double)h->n * sizeof(T);
  const int mode = alpha_mode(h);
  const void* kernel = alpha_kernel_of<T, RP>(mode);
  A.panel = alpha_panels(mode) ? panel_args(h) : PanelArgs{};
  const int dyn = std::max(alpha_panels(mode) ? panel_smem_bytes((int)sizeof(T)) : 0,
                           alpha_streams(mode) ? stream_smem_bytes((int)sizeof(T), alpha_panels(mode)) : 0);
  if (dyn > 0) {
    // set on every launch: the attribute belongs to the current device
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dyn) !=
        cudaSuccess)
      return SA_ERR_CUDA;
  }
  A.long_rows = mode == ALPHA_LARGE || h->n_mc > 0;   // (the splits have row chunks of their own)
  A.n_splits = 0;
  A.split_part = nullptr;
  if (mode == ALPHA_LARGE && h->split_on) {
    A.n_splits = h->n_splits;
    for (int q = 0; q < h->n_splits; ++q) A.split[q] = split_args<T, RP>(h, q);
    A.split_part = (T*)h->split_part;
  }
  void* args[] = {&A};
  const int ctas = mode == ALPHA_SMALL ? alpha_cluster(h) : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)dyn;
  cfg.stream = h->stream;
  cudaLaunchAttribute at[1];
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaError_t e = cudaErrorUnknown;
  if (ctas > 0) {
    A.cluster = 1;
    cfg.gridDim = dim3(ctas);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    e = ctas > 8 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : cudaSuccess;
    if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, kernel, args);
    if (e != cudaSuccess) cudaGetLastError();   // no such cluster on this device: the whole grid
  }
  if (e != cudaSuccess) {
    A.cluster = 0;
    cfg.gridDim = dim3(h->blocks);
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    e = cudaLaunchKernelExC(&cfg, kernel, args);
  }
  count_launches(1);
  return e == cudaSuccess ? SA_OK : SA_ERR_CUDA;
}

}  // namespace sa
