// Batched single-flip local search over all distinct candidates as one persistent cooperative
// kernel, with a cache of the local fields h_ic = sum_j J_ij s_cj and snapshot passes.
//
// Pass semantics (both decided from the pass-start state; bit-exact with oracle/specann_oracle.py):
//   priority (default): a wanting node flips unless a wanting neighbour has a lower rank in the
//     pass's permutation, so the flips form an independent set and every flip lowers the energy
//     by its gain (phases D1: wanting masks and ranks, D2: blocking check, U);
//   snapshot: every wanting node flips (phases D1, U).
// Layout (node-major, so one read of a CSR row serves every candidate):
//   sb[i * kw + t]     bit c of word t: spin of candidate 32 t + c at node i is +1
//   h[i * kp + c]      local field of node i in candidate c (int32 for integer couplings, which
//                      makes every gain and energy exact; double otherwise)
//   flipm[i * kw + t]  candidates flipping at node i in the current pass
// A pass: (D1) every selected node decides for every candidate from the pass-start state; wanting nodes
// go to a queue (snapshot: flip). In priority passes only nodes of which a field or a spin has changed
// since their wanting mask was computed (U marks them in prio) read their fields; for the others the
// mask still holds. (D2) one warp per queued node (one CTA for a long row) finds the flips that no
// neighbour blocks, flips the node's spin bits and appends (node, chunk) entries to a work list; (U) one
// warp per entry scatters the field changes 2 J_ij s_i(new) to the neighbours of the chunk for the
// flipped candidates (integer atomics: exact and order-independent). Arrays that other CTAs change
// during the kernel (h, sb, flipm, the lists) are read with ld.global.cg: the per-SM L1 is not coherent
// with their writes. After a pass every CTA reads the flip counts and applies the stopping rules of
// flip_refinement / gpu_final_sweep (models/spectral_annealing.py:983-1112) itself.
//
// What bounds it: chains of dependent loads (queue -> row -> neighbours -> their masks) over a few
// thousand nodes, so the phases keep many loads in flight: batches of 8 field loads in D1, two row
// entries per lane in D2, the entries of a chunk over the lanes in U, and two CTAs per SM. Search of 128
// candidates on BA(2^16, m = 20): 16.4 -> 7.5 ms, and 5.9 ms with the masks of unchanged nodes kept; of 40
// on BA(200003, m = 15), integer weights: 15.5 -> 7.1 -> 5.2 ms.
#pragma once
#include <cmath>
#include <cstring>
#include <type_traits>

#include "common.cuh"
#include "handle.cuh"
#include "spmv.cuh"
#include "policy.cuh"

namespace sa {

void count_launches(int k);

template <typename GT>
struct EAccOf { using type = typename std::conditional<std::is_same<GT, int>::value, long long, double>::type; };

template <typename VT, typename RP, typename GT>
struct LsArgs {
  using EAccPtr = typename EAccOf<GT>::type*;
  const RP* rowptr;
  const int* col;
  const VT* val;
  const WorkItem* items;
  long long n_items;
  long long n;
  int k, kp, kw, cp;
  uint32_t* sb;
  GT* h;
  uint32_t* flipm;
  long long* wl;
  long long wl_cap;
  uint32_t* wm;          // wanting masks of the pass (priority passes), n x kw
  int* prio;             // rank of the node in the pass's permutation (INT_MAX if not selected)
  int* wq;               // wanting nodes of the pass
  int priority;          // 1: priority passes, 0: snapshot passes
  LsCtrl* ctrl;
  EAccPtr ebefore;      // kp sums of s_i h_i (energy = -sum / 2): int64 or double
  EAccPtr eafter;
  const uint32_t* cand;
  uint32_t* refined;
  long long W;
  sa_ls_params p;
  long long m_main, m_final;
};

template <typename GT>
__device__ __forceinline__ GT coupling_as(float v);
template <>
__device__ __forceinline__ int coupling_as<int>(float v) { return __float2int_rn(v); }
template <>
__device__ __forceinline__ double coupling_as<double>(float v) { return (double)v; }
template <typename GT>
__device__ __forceinline__ GT coupling_as(double v);
template <>
__device__ __forceinline__ int coupling_as<int>(double v) { return __double2int_rn(v); }
template <>
__device__ __forceinline__ double coupling_as<double>(double v) { return v; }

template <typename GT>
__device__ __forceinline__ GT xor_sum_above(GT v, int cp) {
  for (int o = cp; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Local fields of the candidate word t for entries [e0, e1) of a row (lanes: element slot
// lane / cp, candidate lane % cp). Returns the sum for candidate 32 t + lane % cp in every lane.
template <typename VT, typename RP, typename GT>
__device__ __forceinline__ GT row_field(const LsArgs<VT, RP, GT>& A, long long e0, long long e1, int t) {
  const int lane = threadIdx.x & 31;
  const int ne = 32 / A.cp, es = lane / A.cp, c = lane % A.cp;
  GT acc = GT(0);
  for (long long e = e0 + es; e < e1; e += ne) {
    const int j = __ldg(A.col + e);
    const GT v = coupling_as<GT>(__ldg(A.val + e));
    const uint32_t word = A.sb[(long long)j * A.kw + t];
    acc += ((word >> c) & 1u) ? v : -v;
  }
  return xor_sum_above(acc, A.cp);
}

// Per-candidate sums of s_i h_i over all nodes into out[kp] (64-bit integer sums for int32 fields:
// exact and order-independent; FP64 sums otherwise).
template <typename GT>
using EAcc = typename std::conditional<std::is_same<GT, int>::value, long long, double>::type;

__device__ __forceinline__ void acc_add(long long* p, long long v) {
  atomicAdd((unsigned long long*)p, (unsigned long long)v);
}
__device__ __forceinline__ void acc_add(double* p, double v) { atomicAdd(p, v); }

template <typename VT, typename RP, typename GT>
__device__ void energy_phase(const LsArgs<VT, RP, GT>& A, EAcc<GT>* out, EAcc<GT>* sacc, long long gwarp,
                             long long nwarps) {
  using E = EAcc<GT>;
  const int lane = threadIdx.x & 31;
  const int ne = 32 / A.cp, slot = lane / A.cp, c = lane % A.cp;
  for (int q = threadIdx.x; q < A.kp; q += blockDim.x) sacc[q] = E(0);
  __syncthreads();
  for (int t = 0; t < A.kw; ++t) {
    E acc = E(0);
    for (long long base = gwarp * ne; base < A.n; base += nwarps * ne) {
      const long long i = base + slot;
      if (i < A.n) {
        const uint32_t word = __ldcg(A.sb + i * A.kw + t);
        const GT hv = __ldcg(A.h + i * A.kp + 32 * t + c);
        acc += ((word >> c) & 1u) ? (E)hv : -(E)hv;
      }
    }
    for (int o = A.cp; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (slot == 0 && 32 * t + c < A.kp) acc_add(&sacc[32 * t + c], acc);
  }
  __syncthreads();
  for (int q = threadIdx.x; q < A.kp; q += blockDim.x) acc_add(&out[q], sacc[q]);
  __syncthreads();
}

// The kw words of a node's mask (p: its first one), zeros above.
__device__ __forceinline__ void ld_words(const uint32_t* p, int kw, uint32_t (&w)[4]) {
  w[0] = w[1] = w[2] = w[3] = 0u;
  if (kw == 4) {
    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p));
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else if (kw == 2) {
    const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
    w[0] = v.x; w[1] = v.y;
  } else {
    w[0] = __ldcg(p);
    if (kw == 3) { w[1] = __ldcg(p + 1); w[2] = __ldcg(p + 2); }
  }
}

// Local fields of all candidates (cp = 32: lane c has candidate 32 t + c) for entries [e0, e1) of a row,
// in entry order: the warp reads 32 entries at a time, then each entry's spin words, eight entries in
// flight, or four of several words each. Eight instead of four: energies of 20
// candidates on BA(3000, 10) 0.126 -> 0.111 ms, with real couplings 0.136 -> 0.123 ms.
template <typename VT, typename RP, typename GT>
__device__ __forceinline__ void row_fields(const LsArgs<VT, RP, GT>& A, long long e0, long long e1, GT (&acc)[4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int t = 0; t < 4; ++t) acc[t] = GT(0);
  for (long long e = e0; e < e1; e += 32) {
    const int cnt = (int)((e1 - e < 32) ? e1 - e : 32);
    int j = 0;
    GT v = GT(0);
    if (lane < cnt) {
      j = __ldg(A.col + e + lane);
      v = coupling_as<GT>(__ldg(A.val + e + lane));
    }
    if (A.kw == 1) {
      for (int g = 0; g < cnt; g += 8) {
        uint32_t w[8];
        GT vv[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int src = (g + q < cnt) ? g + q : 0;
          const int jj = __shfl_sync(0xffffffffu, j, src);
          vv[q] = __shfl_sync(0xffffffffu, v, src);
          if (g + q < cnt) w[q] = __ldcg(A.sb + jj);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (g + q < cnt) acc[0] += ((w[q] >> lane) & 1u) ? vv[q] : -vv[q];
      }
      continue;
    }
    for (int g = 0; g < cnt; g += 4) {
      uint32_t w[4][4];
      GT vv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int src = (g + q < cnt) ? g + q : 0;
        const int jj = __shfl_sync(0xffffffffu, j, src);
        vv[q] = __shfl_sync(0xffffffffu, v, src);
        if (g + q < cnt) ld_words(A.sb + (long long)jj * A.kw, A.kw, w[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (g + q < cnt) {
#pragma unroll
          for (int t = 0; t < 4; ++t) acc[t] += ((w[q][t] >> lane) & 1u) ? vv[q] : -vv[q];
        }
      }
    }
  }
}

constexpr int kLsLongRow = 512;   // entries above which a wanting node's row is checked by a whole CTA
// Values of prio beside the ranks: a selected node's rank is below both "not selected" values.
constexpr int kLsChanged = -1;            // set by U: a field or a spin of the node changed in the last pass
constexpr int kLsSkipped = 0x7fffffff;    // not selected; its wanting mask is the current one
constexpr int kLsSkippedOld = 0x7ffffffe; // not selected, and changed since its mask was computed
constexpr int kLsSpread = 8;      // flips of a node up to which U spreads its entries over the lanes

template <typename VT, typename RP, typename GT, class Pol>
__device__ __forceinline__ void ls_body(const LsArgs<VT, RP, GT>& A, const Pol& pol) {
  __shared__ EAcc<GT> s_acc[128];           // per-CTA energy sums
  __shared__ int s_cnt[128];                // this CTA's flips of the pass
  __shared__ unsigned int s_active[4];      // candidates that have not yet had a pass without a flip
  __shared__ unsigned int s_block[4];       // blocking masks of a long row
  __shared__ unsigned long long s_total;
  LsCtrl* C = A.ctrl;
  const int lane = threadIdx.x & 31;
  const long long gtid = pol.tid();
  const long long nthreads = pol.nthr();
  const long long gwarp = gtid >> 5, nwarps = nthreads >> 5;
  const long long n = A.n;
  const int cp = A.cp, ne = 32 / cp, slot = lane / cp, c = lane % cp, kw = A.kw;
  unsigned int epoch = pol.first_epoch(&C->gs);
  auto meet = [&]() -> bool { return pol.meet(&C->gs, epoch); };
  // phase timer: the first CTA's thread 0 charges the time since its previous mark to a phase
  const bool timer = pol.block() == 0 && threadIdx.x == 0;
  unsigned long long t_mark = timer ? global_ns() : 0ull;
  auto mark = [&](int ph) {
    if (timer) {
      const unsigned long long t = global_ns();
      C->tph[ph] += t - t_mark;
      t_mark = t;
    }
  };

  // ---- L0: candidate-major packed spins -> node-major bits; zero the fields -----------------
  if (pol.block() == 0) {
    if (threadIdx.x == 0)
      for (int q = 0; q < 4; ++q) C->tph[q] = 0ull;
    for (int q = threadIdx.x; q < 3 * (int)(sizeof(LsPass) / 4); q += blockDim.x) ((unsigned int*)C->pass)[q] = 0u;
  }
  if (threadIdx.x < 4) {
    const int b = A.k - 32 * (int)threadIdx.x;
    s_active[threadIdx.x] = b >= 32 ? 0xffffffffu : (b > 0 ? (1u << b) - 1u : 0u);
  }
  if (threadIdx.x == 0) s_total = 0ull;
  for (long long i = gtid; i < n; i += nthreads) {
    for (int t = 0; t < A.kw; ++t) {
      uint32_t word = 0u;
      const int c1 = min(A.k, 32 * t + 32);
      for (int q = 32 * t; q < c1; ++q) {
        const uint32_t cw = __ldg(A.cand + (long long)q * A.W + (i >> 5));
        word |= ((cw >> (i & 31)) & 1u) << (q - 32 * t);
      }
      A.sb[i * A.kw + t] = word;
    }
    if (A.priority) A.prio[i] = kLsChanged;
  }
  for (long long q = gtid; q < n * A.kp; q += nthreads) A.h[q] = GT(0);
  for (long long q = gtid; q < A.kp; q += nthreads) { A.ebefore[q] = 0; A.eafter[q] = 0; }
  if (!meet()) return;

  // ---- L1: local fields h = J s for all candidates (work-list balanced) ---------------------
  for (long long itm = gwarp; itm < A.n_items; itm += nwarps) {
    const long long e0 = __ldg(&A.items[itm].e0);
    const int irow = __ldg(&A.items[itm].row);
    const int meta = __ldg(&A.items[itm].meta);
    const long long row0 = irow >= 0 ? irow : -((long long)irow + 1);
    const long long row1 = irow >= 0 ? irow + item_nrows(meta) : row0 + 1;
    for (long long r = row0; r < row1; ++r) {
      const long long rs = irow >= 0 ? rp_load(A.rowptr, r) : e0;
      const long long re = irow >= 0 ? rp_load(A.rowptr, r + 1) : e0 + item_len(meta);
      GT f[4];
      if (cp == 32) row_fields(A, rs, re, f);
      else f[0] = row_field(A, rs, re, 0);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (t >= kw || slot != 0 || 32 * t + c >= A.kp) continue;
        if (irow >= 0) A.h[r * A.kp + 32 * t + c] = f[t];
        else atomicAdd(&A.h[r * A.kp + 32 * t + c], f[t]);
      }
    }
  }
  if (!meet()) return;
  energy_phase(A, A.ebefore, s_acc, gwarp, nwarps);
  if (!meet()) return;
  mark(0);

  // ---- passes ------------------------------------------------------------------------------
  const bool has_final = A.p.num_rounds > 0 && A.p.final_sweep_iters > 0;
  int phase = A.p.max_iterations > 0 ? 0 : (has_final ? 1 : 2);   // 0 main loop, 1 final sweep, 2 done
  int it = 0, round = 0, sub = 0, final_passes = 0, set = 0;
  // D1 tiles: TN nodes, whose `steps` (node group, candidate word) loads a warp takes 8 at a time
  const int TN = cp < 32 || kw == 1 ? 32 : (kw == 2 ? 16 : 8);
  const int steps = (TN / ne) * kw, inv_kw = (65536 + kw - 1) / kw;
  const unsigned int cmask = cp == 32 ? 0xffffffffu : (1u << cp) - 1u;
  while (phase != 2) {
    LsPass* const cur = &C->pass[set];
    const long long m = phase == 0 ? A.m_main : A.m_final;
    const bool all_sel = m >= n;
    const SelKeys keys = make_sel_keys(A.p.seed, phase == 0 ? (long long)it : kFinalStreamBase + round, n);
    for (int q = threadIdx.x; q < 128; q += blockDim.x) s_cnt[q] = 0;
    __syncthreads();
    auto push_chunks = [&](long long i, long long deg) {
      const long long nch = deg > kChunk ? (deg + kChunk - 1) / kChunk : 1;
      const long long pos = (long long)atomicAdd(&cur->wl, (unsigned long long)nch);
      for (long long q = 0; q < nch && pos + q < A.wl_cap; ++q) A.wl[pos + q] = (i << 22) | q;
    };
    // D1: every selected node decides for every candidate from the pass-start state. Snapshot
    // passes flip the wanting pairs here; priority passes record the wanting masks and ranks.
    for (long long tile = gwarp * TN; tile < n; tile += nwarps * TN) {
      bool selb = false, old = false;   // old: the node's wanting mask has to be computed again
      if (lane < TN && tile + lane < n) {
        int rk = 0;
        if (A.priority) {
          const int was = __ldcg(A.prio + tile + lane);
          old = was == kLsChanged || was == kLsSkippedOld;
        }
        if (all_sel && !A.priority) {
          selb = true;
        } else {
          const long long r = sel_rank(tile + lane, keys, n);
          selb = r < m;
          rk = (int)r;
        }
        if (A.priority) A.prio[tile + lane] = selb ? rk : (old ? kLsSkippedOld : kLsSkipped);
      }
      const uint32_t selmask = __ballot_sync(0xffffffffu, selb && (old || !A.priority));
      uint32_t want = 0u;   // nodes of the tile that want some candidate
      if (A.priority) {
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        if (selb && !old) ld_words(A.wm + (tile + lane) * kw, kw, w);
        want = __ballot_sync(0xffffffffu, (w[0] | w[1] | w[2] | w[3]) != 0u);
      }
      for (int f0 = 0; f0 < steps; f0 += 8) {
        const int s0 = (f0 * inv_kw) >> 16, s1 = ((min(f0 + 8, steps) - 1) * inv_kw) >> 16;
        if (!(selmask & ((2u << (s1 * ne + ne - 1)) - 1u) & ~((1u << (s0 * ne)) - 1u))) continue;
        uint32_t word[8];
        GT hv[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int s = ((f0 + q) * inv_kw) >> 16, t = f0 + q - s * kw, node = s * ne + slot;
          const long long i = tile + node;
          word[q] = 0u;
          hv[q] = GT(0);
          if (f0 + q < steps && ((selmask >> node) & 1u)) {
            word[q] = __ldcg(A.sb + i * kw + t);
            hv[q] = __ldcg(A.h + i * A.kp + 32 * t + c);
          }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (f0 + q >= steps) break;
          const int s = ((f0 + q) * inv_kw) >> 16, t = f0 + q - s * kw, node = s * ne + slot;
          const long long i = tile + node;
          // (a node that is not read has a zero field here)
          const bool f = (32 * t + c < A.k) && (((word[q] >> c) & 1u) ? (hv[q] < GT(0)) : (hv[q] > GT(0)));
          const uint32_t bal = __ballot_sync(0xffffffffu, f);
          const uint32_t bits = cp == 32 ? bal : ((bal >> (slot * cp)) & cmask);
          if (c == 0 && ((selmask >> node) & 1u)) {
            (A.priority ? A.wm : A.flipm)[i * kw + t] = bits;
            if (!A.priority && bits) A.sb[i * kw + t] = word[q] ^ bits;
          }
          if (!A.priority && f) atomicAdd(&s_cnt[32 * t + c], 1);
          if (bal) {
            if (cp == 32) want |= 1u << s;
            else
              for (int sl = 0; sl < ne; ++sl)
                if ((bal >> (sl * cp)) & cmask) want |= 1u << (s * ne + sl);
          }
        }
      }
      if (want) {
        const bool mine = (want >> lane) & 1u;
        const long long i = tile + lane;
        const long long deg = mine ? rp_load(A.rowptr, i + 1) - rp_load(A.rowptr, i) : 0;
        if (!A.priority) {
          if (mine) push_chunks(i, deg);
        } else {
          // one reservation per tile and queue
          const uint32_t big = __ballot_sync(0xffffffffu, deg > kLsLongRow), small = want & ~big;
          unsigned int at = 0u, at_big = 0u;
          if (lane == 0) {
            if (small) at = atomicAdd(&cur->wq, (unsigned int)__popc(small));
            if (big) at_big = atomicAdd(&cur->lq, (unsigned int)__popc(big));
          }
          at = __shfl_sync(0xffffffffu, at, 0);
          at_big = __shfl_sync(0xffffffffu, at_big, 0);
          const uint32_t below = (1u << lane) - 1u;
          if ((small >> lane) & 1u) A.wq[at + __popc(small & below)] = (int)i;
          if ((big >> lane) & 1u) A.wq[n - 1 - (long long)(at_big + __popc(big & below))] = (int)i;
        }
      }
    }
    if (A.priority) {
      if (!meet()) return;
      // every CTA is past the reading of the last pass's counters: the set of the pass after next
      if (pol.block() == 0)
        for (int q = threadIdx.x; q < (int)(sizeof(LsPass) / 4); q += blockDim.x)
          ((unsigned int*)&C->pass[set == 0 ? 2 : set - 1])[q] = 0u;
      // D2: a wanting node flips the candidates for which no wanting neighbour has a lower rank (the
      // blocking masks are OR-reduced over the row). Long rows: one CTA each.
      auto commit = [&](long long i, const uint32_t (&W)[4], long long deg) {
        for (int t = 0; t < kw; ++t) {
          A.flipm[i * kw + t] = W[t];
          if (W[t]) A.sb[i * kw + t] = __ldcg(A.sb + i * kw + t) ^ W[t];
        }
        push_chunks(i, deg);
      };
      const long long nlq = (long long)ld_volatile_u32(&cur->lq), nwq = (long long)ld_volatile_u32(&cur->wq);
      for (long long e = pol.block(); e < nlq; e += pol.nblocks()) {
        const long long i = (long long)__ldcg(A.wq + n - 1 - e);
        const int pi = __ldcg(A.prio + i);
        const long long rs = rp_load(A.rowptr, i), re = rp_load(A.rowptr, i + 1);
        uint32_t B[4] = {0u, 0u, 0u, 0u}, W[4];
        if (threadIdx.x < 4) s_block[threadIdx.x] = 0u;
        __syncthreads();
        for (long long p = rs + threadIdx.x; p < re; p += blockDim.x) {
          const int j = __ldg(A.col + p);
          if (__ldcg(A.prio + j) < pi) {
            uint32_t w[4];
            ld_words(A.wm + (long long)j * kw, kw, w);
#pragma unroll
            for (int t = 0; t < 4; ++t) B[t] |= w[t];
          }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint32_t b = __reduce_or_sync(0xffffffffu, B[t]);
          if (lane == 0 && b) atomicOr(&s_block[t], b);
        }
        __syncthreads();
        ld_words(A.wm + i * kw, kw, W);
        uint32_t any = 0u;
#pragma unroll
        for (int t = 0; t < 4; ++t) any |= (W[t] &= ~s_block[t]);
        if (threadIdx.x < 32) {
#pragma unroll
          for (int t = 0; t < 4; ++t)
            if ((W[t] >> lane) & 1u) atomicAdd(&s_cnt[32 * t + lane], 1);
          if (lane == 0 && any) commit(i, W, re - rs);
        }
        __syncthreads();
      }
      int cnt[4] = {0, 0, 0, 0};
      long long i = gwarp < nwq ? (long long)__ldcg(A.wq + gwarp) : 0;
      for (long long e = gwarp; e < nwq; e += nwarps) {
        const long long next = e + nwarps < nwq ? (long long)__ldcg(A.wq + e + nwarps) : 0;
        const int pi = __ldcg(A.prio + i);
        const long long rs = rp_load(A.rowptr, i), re = rp_load(A.rowptr, i + 1);
        uint32_t W[4], B[4] = {0u, 0u, 0u, 0u};
        ld_words(A.wm + i * kw, kw, W);
        for (long long p = rs + lane; p < re; p += 64) {
          const bool two = p + 32 < re;
          const int j0 = __ldg(A.col + p), j1 = two ? __ldg(A.col + p + 32) : 0;
          const int p0 = __ldcg(A.prio + j0), p1 = two ? __ldcg(A.prio + j1) : kLsSkipped;
          uint32_t w0[4] = {0u, 0u, 0u, 0u}, w1[4] = {0u, 0u, 0u, 0u};
          if (p0 < pi) ld_words(A.wm + (long long)j0 * kw, kw, w0);
          if (p1 < pi) ld_words(A.wm + (long long)j1 * kw, kw, w1);
#pragma unroll
          for (int t = 0; t < 4; ++t) B[t] |= w0[t] | w1[t];
        }
        uint32_t any = 0u;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (t < kw) W[t] &= ~__reduce_or_sync(0xffffffffu, B[t]);
          any |= W[t];
          cnt[t] += (W[t] >> lane) & 1u;
        }
        if (lane == 0 && any) commit(i, W, re - rs);
        i = next;
      }
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (cnt[t]) atomicAdd(&s_cnt[32 * t + lane], cnt[t]);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < A.k; q += blockDim.x)
      if (s_cnt[q]) atomicAdd(&cur->counts[q], s_cnt[q]);
    if (!meet()) return;
    mark(1);

    // U: scatter field changes of the flipped (node, candidate) pairs. Few flips: the chunk's entries
    // over the lanes, flip after flip; many: candidates over the lanes, entry after entry, where the
    // updates of an entry share sectors (from about 8 of the 128-byte line's 32 on).
    const long long nwl = min((long long)*((volatile unsigned long long*)&cur->wl), A.wl_cap);
    for (long long e = gwarp; e < nwl; e += nwarps) {
      const long long ent = __ldcg(A.wl + e);
      const long long i = ent >> 22;
      const long long q = ent & ((1ll << 22) - 1);
      const long long rs = rp_load(A.rowptr, i), re = rp_load(A.rowptr, i + 1);
      uint32_t F[4], S[4];
      ld_words(A.flipm + i * kw, kw, F);
      ld_words(A.sb + i * kw, kw, S);
      const long long cb = rs + q * kChunk;
      const long long ce = (cb + kChunk < re) ? cb + kChunk : re;
      if (A.priority && q == 0 && lane == 0) A.prio[i] = kLsChanged;
      if (__popc(F[0]) + __popc(F[1]) + __popc(F[2]) + __popc(F[3]) <= kLsSpread) {
        for (long long p = cb + lane; p < ce; p += 32) {
          const int j = __ldg(A.col + p);
          GT* hj = A.h + (long long)j * A.kp;
          if (A.priority) A.prio[j] = kLsChanged;
          const GT v2 = GT(2) * coupling_as<GT>(__ldg(A.val + p));
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            for (uint32_t b = F[t]; b; b &= b - 1u) {
              const int cc = __ffs(b) - 1;
              atomicAdd(hj + 32 * t + cc, ((S[t] >> cc) & 1u) ? v2 : -v2);
            }
          }
        }
        continue;
      }
      if (A.priority)
        for (long long p = cb + lane; p < ce; p += 32) A.prio[__ldg(A.col + p)] = kLsChanged;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (!((F[t] >> c) & 1u)) continue;
        const bool up = (S[t] >> c) & 1u;
#pragma unroll 4
        for (long long p = cb + slot; p < ce; p += ne) {
          const int j = __ldg(A.col + p);
          const GT v = coupling_as<GT>(__ldg(A.val + p));
          atomicAdd(&A.h[(long long)j * A.kp + 32 * t + c], up ? GT(2) * v : GT(-2) * v);
        }
      }
    }
    if (!meet()) return;
    // the stopping rules, in every CTA
    const int cq = (int)threadIdx.x < A.k ? __ldcg(&cur->counts[threadIdx.x]) : 0;
    if (threadIdx.x < 128) {
      const unsigned int flipped = __ballot_sync(0xffffffffu, cq > 0);
      if (lane == 0 && phase == 0) s_active[threadIdx.x >> 5] &= flipped;
      if (pol.block() == 0) {
        // (32 candidates can flip more than 2^31 spins in a pass)
        const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)cq & 0xffffu);
        const unsigned hi = __reduce_add_sync(0xffffffffu, (unsigned)cq >> 16);
        if (lane == 0) atomicAdd(&s_total, ((unsigned long long)hi << 16) + lo);
      }
    }
    const bool any = __syncthreads_or(cq > 0);
    if (!A.priority && pol.block() == 0)   // (a snapshot pass has no barrier between D1 and here)
      for (int q = threadIdx.x; q < (int)(sizeof(LsPass) / 4); q += blockDim.x)
        ((unsigned int*)&C->pass[set == 0 ? 2 : set - 1])[q] = 0u;
    set = set == 2 ? 0 : set + 1;
    if (phase == 0) {
      it += 1;
      if (!(s_active[0] | s_active[1] | s_active[2] | s_active[3]) || it >= A.p.max_iterations) {
        phase = has_final ? 1 : 2;
        round = 0;
        sub = 0;
      }
    } else {
      sub += 1;
      final_passes += 1;
      if (!any || sub >= A.p.final_sweep_iters) {
        round += 1;
        sub = 0;
        if (round >= A.p.num_rounds) phase = 2;
      }
    }
    mark(2);
  }
  if (timer) {
    C->it = it;
    C->final_passes = final_passes;
    C->total_flips = (long long)s_total;
  }

  // ---- energies after, refined candidates back to candidate-major ---------------------------
  energy_phase(A, A.eafter, s_acc, gwarp, nwarps);
  const long long pairs = (long long)A.k * A.W;
  for (long long pr = gwarp; pr < pairs; pr += nwarps) {
    const long long cq = pr / A.W, wd = pr % A.W;
    const long long i = wd * 32 + lane;
    bool bit = false;
    if (i < n) bit = (__ldcg(A.sb + i * A.kw + (cq >> 5)) >> (cq & 31)) & 1u;
    const uint32_t word = __ballot_sync(0xffffffffu, bit);
    if (lane == 0) A.refined[cq * A.W + wd] = word;
  }
  mark(3);
}

}  // namespace sa
