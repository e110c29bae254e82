// One alpha of the SpecAnn sweep as one persistent cooperative kernel: start vector / predictor,
// warm-started thick-restart Lanczos for the smallest eigenpair of S_rho = rho I - N_alpha with
// FP64 inner products and an FP64 tridiagonal Ritz solve, the Ritz-matrix guard, sign alignment,
// the true residual, and rounding to packed spins with an order-independent signature.
//
// CTAs rewrite V, w, u and y between phases and the per-SM L1 is not coherent with writes from
// other SMs, so every read of those arrays inside this kernel uses ld.global.cg (L2).
//
// Vectors (basis V, w, u, y) are in T (float or double); every inner product and norm is
// accumulated in double; the projected tridiagonal T_j lives in double in the control block.
// Between phases the CTAs meet at a barrier; then every CTA reduces the per-CTA partial sums itself, in
// CTA order, and takes the Lanczos decisions in its own copy of the control block. All copies are the
// same, so every CTA follows the same control path, results do not depend on timing, and no CTA waits
// for another one's decision.
#pragma once
#include <cmath>
#include <cstdio>
#include <type_traits>

#include "common.cuh"
#include "handle.cuh"
#include "spmv.cuh"
#include "panel.cuh"
#include "policy.cuh"

namespace sa {

void count_launches(int k);

constexpr int kPartCols = kNcvMax + 8;   // columns of partial sums that a phase reduces at most

enum Action : int { ACT_NEXT = 0, ACT_REPASS = 1, ACT_RESTART = 2, ACT_REJECT = 3, ACT_DONE = 4, ACT_ERROR = 5,
                    ACT_P0_AGAIN = 6 };

constexpr double kLog2Clamp = -39.86313713864835;   // log2(1e-12)
constexpr int kRestartDefault = 8;   // Ritz vectors kept by an implicit restart (at most ncv / 2)
constexpr int kRestartMax = 16;
constexpr double kTinyNorm = 1e-12;

template <typename T, typename RP>
struct AlphaArgs {
  SpmvArgs<T, RP> S;
  long long n, ldv;
  T* sigma;
  const double* ld;
  const double* aoff;    // per-vertex exponent offsets (a_i = alpha + aoff[i]) or null
  T* V;
  T* w;
  T* u;
  const T* ylast;
  const T* yprev;
  T* yout;
  const T* v0;
  double* part;          // per-CTA partial sums: two buffers of kPartCols columns x CTAs
  AlphaCtrl* ctrl;
  uint32_t* bits;        // scratch candidate (W words)
  long long W;
  sa_alpha_params p;
  int has_last, has_prev;
  double half_log2_c;
  double sqrt_c;
  int group;
  double spmv_bytes;     // algorithmic bytes of one fused SpMV
  double* dense;         // implicit-restart scratch (dense T, then dense Q)
  PanelArgs panel;       // column-panel layout of the operator (ALPHA_PANEL; panel_smem_bytes(sizeof(T)) and
                         // at least stream_smem_bytes(sizeof(T)) of dynamic shared memory)
  SpmvArgs<T, RP> split[kMaxSplits];   // L2 column splits of the operator (n_splits > 0): one
  int n_splits;                        // work-list pass per split, partial row sums in split_part
  T* split_part;
  int long_rows;         // rows of several chunks in the work list (RowStep::fixed is in use)
  int cluster;           // the grid is one cluster (GridPolicy)
};

// ---- small dense helpers for the projected tridiagonal (double, one CTA) --------------------

// A tridiagonal as its recurrences read it, in shared memory: row i is {a_i, b_{i-1}^2} (b_{-1} = 0),
// padded to a multiple of kTriBlock rows with {2^60, 0}: such a row multiplies both minors by a
// positive number and takes no part in a sign count.
constexpr int kTriBlock = 8;
constexpr int kTriPad = kNcvMax + 2 * kTriBlock;
__host__ __device__ constexpr int tri_blocks(int m) { return (m + kTriBlock - 1) / kTriBlock; }

// Stages the tridiagonal (a, b; size m) in `tri` (all threads; the caller synchronises).
__device__ __forceinline__ void tri_stage(const double* a, const double* b, int m, double2* tri) {
  for (int i = threadIdx.x; i < tri_blocks(m) * kTriBlock; i += blockDim.x) {
    const double bb = (i > 0 && i < m) ? b[i - 1] : 0.0;
    tri[i] = make_double2(i < m ? a[i] : 0x1p60, bb * bb);
  }
}

// Power of two that brings the larger of two doubles to [1, 2) (their biased exponent on the integer
// pipe; two zeros or subnormals are scaled by 2^1022).
__device__ __forceinline__ double pow2_normaliser(double p, double q) {
  const int e = max(max((__double2hiint(p) >> 20) & 0x7FF, (__double2hiint(q) >> 20) & 0x7FF), 1);
  return __hiloint2double((2046 - e) << 20, 0);
}

// Number of eigenvalues of the tridiagonal below x: sign changes of the leading principal minors
// det(T_k - x I), computed with the three-term recurrence. What bounds it is one dependent DFMA a row
// (8.7 cycles), so nothing else may stand on that chain: a block of kTriBlock rows is read while the one
// before it is worked on, signs are counted on the integer pipe, and the pair of minors is scaled
// once per block by a power of two taken from the middle of the block, without a branch (entries
// below 2^60 cannot leave the double range in between). A zero minor counts as positive: the minor
// after it has the opposite sign of the one before.
__device__ __forceinline__ int sturm_count(const double2* tri, int blocks, double x) {
  double pp = 0.0, pc = 1.0, f = 1.0;
  int cnt = 0;
  double2 r[kTriBlock];
#pragma unroll
  for (int q = 0; q < kTriBlock; ++q) r[q] = tri[q];
#pragma unroll 1
  for (int k = 1; k <= blocks; ++k) {
    double2 nx[kTriBlock];
    const double2* next = tri + (k < blocks ? k : 0) * kTriBlock;
#pragma unroll
    for (int q = 0; q < kTriBlock; ++q) nx[q] = next[q];
#pragma unroll
    for (int q = 0; q < kTriBlock; ++q) {
      const double pn = fma(r[q].x - x, pc, -__dmul_rn(r[q].y, pp));   // (the product is off the chain)
      cnt += (int)((unsigned)(__double2hiint(pn) ^ __double2hiint(pc)) >> 31);
      pp = pc;
      pc = pn;
      if (q == kTriBlock / 2 - 1) f = pow2_normaliser(pc, pp);
    }
    pc *= f;
    pp *= f;
#pragma unroll
    for (int q = 0; q < kTriBlock; ++q) r[q] = nx[q];
  }
  return cnt;
}

// The minors det(T_{m-1} - x), det(T_m - x) and the derivative of the latter by x, up to one common
// power of two, by the same recurrence (pad rows are left out: they are no factor of a derivative).
struct Minors {
  double pm1, p, dp;
};

__device__ __forceinline__ void minor_step(const double2& r, double x, double& pp, double& pc, double& dp, double& dc) {
  const double d = r.x - x;
  const double pn = fma(d, pc, -__dmul_rn(r.y, pp));
  const double dn = fma(d, dc, -fma(r.y, dp, pc));
  pp = pc; pc = pn; dp = dc; dc = dn;
}

__device__ __forceinline__ Minors last_minors(const double2* tri, int m, double x) {
  double pp = 0.0, pc = 1.0, dp = 0.0, dc = 0.0, f = 1.0;
  int k = 0;
  double2 r[kTriBlock];
#pragma unroll
  for (int q = 0; q < kTriBlock; ++q) r[q] = tri[q];
#pragma unroll 1
  for (; k + kTriBlock <= m; k += kTriBlock) {
    double2 nx[kTriBlock];   // (the staging is padded, so a block past the last one can be read)
#pragma unroll
    for (int q = 0; q < kTriBlock; ++q) nx[q] = tri[k + kTriBlock + q];
#pragma unroll
    for (int q = 0; q < kTriBlock; ++q) {
      minor_step(r[q], x, pp, pc, dp, dc);
      if (q == kTriBlock / 2 - 1) f = fmin(pow2_normaliser(pc, pp), pow2_normaliser(dc, dp));
    }
    pc *= f; pp *= f; dc *= f; dp *= f;
#pragma unroll
    for (int q = 0; q < kTriBlock; ++q) r[q] = nx[q];
  }
#pragma unroll
  for (int q = 0; q < kTriBlock - 1; ++q)
    if (k + q < m) minor_step(r[q], x, pp, pc, dp, dc);
  return Minors{pp, pc, dc};
}

// Gershgorin interval of the staged tridiagonal, widened by its rounding (one full warp).
__device__ __forceinline__ void tri_interval(const double2* tri, int m, double* lo_out, double* hi_out) {
  const int lane = threadIdx.x & 31;
  double lo = 1e300, hi = -1e300;
#pragma unroll 1
  for (int i = lane; i < m; i += 32) {
    const double r = sqrt(tri[i].y) + (i + 1 < m ? sqrt(tri[i + 1].y) : 0.0);
    lo = fmin(lo, tri[i].x - r);
    hi = fmax(hi, tri[i].x + r);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
  }
  const double pad = 1e-12 * fmax(1.0, fmax(fabs(lo), fabs(hi)));
  *lo_out = lo - pad;
  *hi_out = hi + pad;
}

// Threads of the multisection below, their barrier, and how many of them hold `p`. Four warps, one per
// scheduler, keep a row of the Sturm recurrence at its DFMA latency (about 13 cycles); with sixteen
// warps the FP64 pipe bounds it (about 38 cycles a row) for only two more bits a round.
constexpr int kRitzThreads = 128;
__device__ __forceinline__ int ritz_sync_count(bool p) {
  int c;
  asm volatile(
      "{\n .reg .pred q;\n setp.ne.s32 q, %1, 0;\n barrier.cta.red.popc.aligned.u32 %0, 1, %2, q;\n}"
      : "=r"(c)
      : "r"((int)p), "n"(kRitzThreads)
      : "memory");
  return c;
}

// Smallest eigenvalue of the tridiagonal (a, b; size m), and the squared last component of its unit
// eigenvector, -det(T_{m-1} - x) / det'(T_m - x), in *s2 (every thread of the CTA gets both).
//   1. A bracket, from Sturm counts at kRitzThreads points at a time: the threads whose point lies below
//      the eigenvalue form a prefix, so their number, from one barrier, is the bracket in every thread's
//      registers. hint_lo < hint_hi is a bracket to try first (from the previous step: by interlacing
//      the smallest eigenvalue of T_m is at most the previous smallest Ritz value, and the previous
//      residual bounds how far below it can be unless a new, lower eigenvalue appears). Its points
//      halve the distance to hint_hi every second point, since near convergence the Ritz value moves
//      by about the residual squared; the round itself shows whether the bracket holds the eigenvalue,
//      else the Gershgorin interval is cut twice into kRitzThreads + 1 parts.
//   2. Newton's iteration on det(T_m - x) from the bracket's lower end, by one warp: to the left of the
//      smallest root of a polynomial with only real roots it increases to that root, quadratically
//      (two to four evaluations here). It ends when the step no longer changes x, and the last
//      evaluation gives *s2 too.
//   3. If Newton leaves the bracket or takes too long (clustered roots), multisection to the end.
// One test costs about DFMA latency x rows x evaluations. Each recurrence has one call site: the code
// of a Lanczos step is read again at every step, and what does not stay in the instruction cache costs
// as much as the arithmetic.
__device__ __forceinline__ double smallest_eig_block(const double* ag, const double* bg, int m, double* s2,
                                                  double hint_lo = 0.0, double hint_hi = -1.0) {
  __shared__ double s_r, s_s2;
  __shared__ double2 tri[kTriPad];
  const int t = tid_here();
  tri_stage(ag, bg, m, tri);
  __syncthreads();
  if (t < kRitzThreads) {
    constexpr int P = kRitzThreads;
    const int blocks = tri_blocks(m);
    double lo = 0.0, hi = 0.0, x = 0.0, c2 = 1.0;
    bool hint = hint_lo < hint_hi, newton = true;
    if (!hint) tri_interval(tri, m, &lo, &hi);
    // rounds to go before Newton's iteration; on its failure, rounds to the end
    int rounds = hint ? 1 : 2;
    while (true) {
      for (; rounds > 0 && (newton || hi - lo > 1e-15 * fmax(1.0, fabs(hi))); --rounds) {
        // hint: point k is hint_hi - w 2^(-k / 2), the last one hint_hi; else P cuts of [lo, hi]
        const double w = hint ? hint_hi - hint_lo : (hi - lo) * (1.0 / (P + 1));
        auto point = [&](int k) {
          if (!hint) return lo + w * (double)(k + 1);
          if (k == P - 1) return hint_hi;
          return hint_hi - w * ((k & 1) ? 0.70710678118654752 : 1.0) * __hiloint2double((1023 - (k >> 1)) << 20, 0);
        };
        const int f = ritz_sync_count(sturm_count(tri, blocks, point(t)) == 0);
        if (hint && (f == 0 || f == P)) {
          hint = false;
          tri_interval(tri, m, &lo, &hi);
          rounds = 3;
          continue;
        }
        const double nlo = f > 0 ? point(f - 1) : lo;
        if (f < P) hi = point(f);
        lo = nlo;
        hint = false;
      }
      // every warp iterates alike (no exchange); without Newton one evaluation, for c2
      x = newton ? lo : 0.5 * (lo + hi);
      const double tiny = 1e-16 * fmax(1.0, fabs(hi));
      bool done = false;
      for (int it = 0; it < (newton ? 16 : 1) && !done; ++it) {
        const Minors q = last_minors(tri, m, x);
        const double inv = -1.0 / q.dp;
        const double step = q.p * inv;
        c2 = q.pm1 * inv;
        done = !newton || !(step > tiny);
        if (!done) x += step;
      }
      if (!newton || (done && x <= hi + tiny && isfinite(c2))) break;
      newton = false;
      rounds = 9;
    }
    if (t == 0) {
      s_r = x;
      s_s2 = isnan(c2) ? 1.0 : fmin(fmax(c2, 0.0), 1.0);
    }
  }
  __syncthreads();
  const double r = s_r;
  *s2 = s_s2;
  __syncthreads();
  return r;
}

// The same as a call, for the rare invariant subspace at a restart.
static __device__ __noinline__ double smallest_eig_call(const double* a, const double* b, int m) {
  double s2;
  return smallest_eig_block(a, b, m, &s2);
}

// Unit eigenvector of the tridiagonal (a, b; size m) for its smallest eigenvalue theta into s (the first
// warp). With T - theta I factored from the top (pivots u_k) and from the bottom (pivots l_k), the
// vector is 1 at the row r where the two meet with the smallest gamma_r = u_r + l_r - (a_r - theta) and
// follows from the pivots' ratios on both sides; gamma_r / |z| is its residual. T - theta I is
// semidefinite, so neither factorisation needs pivoting. The two chains of divisions run in two
// lanes at once: 33 rows take about 6 k cycles where inverse iteration in one thread took 52 k.
// scratch: 4 kNcvMax doubles of shared memory.
static __device__ __noinline__ void tridiag_eigvec(const double* a, const double* b, int m, double theta, double* s,
                                                   double* scratch) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  double* u = scratch;
  double* l = scratch + kNcvMax;
  double* fu = scratch + 2 * kNcvMax;   // s_k / s_{k+1} above the meeting row
  double* fl = scratch + 3 * kNcvMax;   // s_k / s_{k-1} below it
  double big = 0.0;
  for (int i = lane; i < m; i += 32) big = fmax(big, fmax(fabs(a[i]), i + 1 < m ? fabs(b[i]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  const double tiny = fmax(big, 1e-300) * 1e-20;
  if (lane < 2) {
    double p = 0.0;
    for (int i = 0; i < m; ++i) {
      const int k = lane == 0 ? i : m - 1 - i;
      const double bb = i == 0 ? 0.0 : b[lane == 0 ? k - 1 : k];
      const double f = i == 0 ? 0.0 : bb / p;
      p = (a[k] - theta) - bb * f;
      if (fabs(p) < tiny) p = tiny;
      (lane == 0 ? u : l)[k] = p;
      if (i > 0) (lane == 0 ? fu : fl)[lane == 0 ? k - 1 : k + 1] = -f;
    }
  }
  __syncwarp();
  // the meeting row
  double g = 1e300;
  int r = 0;
  for (int i = lane; i < m; i += 32) {
    const double gi = fabs(u[i] + l[i] - (a[i] - theta));
    if (gi < g) {
      g = gi;
      r = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double og = __shfl_xor_sync(0xffffffffu, g, o);
    const int orow = __shfl_xor_sync(0xffffffffu, r, o);
    if (og < g || (og == g && orow < r)) {
      g = og;
      r = orow;
    }
  }
  if (lane == 0) {
    s[r] = 1.0;
    double z = 1.0;
    for (int k = r - 1; k >= 0; --k) s[k] = z = z * fu[k];
  } else if (lane == 1) {
    double z = 1.0;
    for (int k = r + 1; k < m; ++k) s[k] = z = z * fl[k];
  }
  __syncwarp();
  double nrm = 0.0;
  for (int i = lane; i < m; i += 32) nrm += s[i] * s[i];
  nrm = sqrt(warp_sum(nrm));
  for (int i = lane; i < m; i += 32) s[i] /= nrm;
  __syncwarp();
}

// All eigenvalues of the staged tridiagonal in ascending order into out[m] (the CTA): four lanes per
// eigenvalue, three of them probing the quarters of its bracket in each of 27 rounds.
__device__ inline void all_eigs_block(const double2* tri, int m, double* out) {
  const int sub = threadIdx.x & 3, blocks = tri_blocks(m);
  double lo0, hi0;
  tri_interval(tri, m, &lo0, &hi0);
  for (int base = 0; base < m; base += blockDim.x >> 2) {
    const int q = min(base + (int)(threadIdx.x >> 2), m - 1);
    if (base + (int)((threadIdx.x & ~31) >> 2) >= m) break;   // a warp without an eigenvalue of its own
    double lo = lo0, hi = hi0;
    for (int it = 0; it < 27; ++it) {
      const double w = 0.25 * (hi - lo);
      // points whose count leaves eigenvalue q above them form a prefix of the three
      const bool above = sub < 3 && sturm_count(tri, blocks, lo + w * (double)(sub + 1)) <= q;
      const unsigned g = (__ballot_sync(0xffffffffu, above) >> (threadIdx.x & 28)) & 7u;
      const int k = __popc(g);
      if (k < 3) hi = lo + w * (double)(k + 1);
      lo += w * (double)k;
    }
    if (sub == 0) out[q] = 0.5 * (lo + hi);
  }
}

// Implicit restart with exact shifts (the CTA): the m - kk largest Ritz values of the tridiagonal
// (a, b; size m) are the shifts of implicit QR steps. Each step is a bulge chase on the tridiagonal
// itself (diagonal d, off-diagonal e and the one bulge entry): rotation r acts on rows and columns
// r, r + 1 as T <- G T G^T with G = [[c, s], [-s, c]], and on the rows of Q (Qg, m x m row-major,
// Q <- Q G^T). Rotation r of a shift touches d[r], d[r + 1] and e[r - 1 .. r + 1] (the entries that
// the next rotation changes again stay in registers), so the next shift follows three rotations
// behind: thread s chases shift s and all chases advance together, m - 1 + 3
// (m - kk - 1) steps instead of (m - kk)(m - 1), each of them a square root's latency; the other
// threads apply the rotations of the step before to Q meanwhile. The values are those of one chase after
// the other. Afterwards Q^T T Q has a leading kk x kk tridiagonal, written back to a and b, and the
// residual of the kept basis is V Q[:, kk] T+[kk][kk-1] + w Q[m-1][kk-1] (w: the pending unnormalised
// Lanczos vector). scratch: scratch_len >= 2 kTriPad + 7 kNcvMax doubles of shared memory, 16-byte
// aligned.
static __device__ __noinline__ void implicit_restart(AlphaCtrl* C, double* Qg, int m, int kk, double* scratch,
                                                     int scratch_len) {
  // Q is built in the rest of the scratch when it fits there
  constexpr int kFixed = 2 * kTriPad + 7 * kNcvMax;
  const bool inside = kFixed + m * m <= scratch_len;
  double* Qd = inside ? scratch + kFixed : Qg;
  double2* tri = (double2*)scratch;
  double* d = scratch + 2 * kTriPad;
  double* e = d + kNcvMax;
  double* ritz = e + kNcvMax;
  double2* rot = (double2*)(ritz + kNcvMax);   // two steps' rotations, one per shift
  const int t = threadIdx.x;
  tri_stage(C->a, C->b, m, tri);
  for (int i = t; i < m; i += blockDim.x) {
    d[i] = C->a[i];
    e[i] = (i + 1 < m) ? C->b[i] : 0.0;
  }
  for (int idx = t; idx < m * m; idx += blockDim.x) Qd[idx] = (idx / m == idx % m) ? 1.0 : 0.0;
  __syncthreads();
  all_eigs_block(tri, m, ritz);
  __syncthreads();
  const int ns = m - kk, steps = (m - 1) + 3 * (ns - 1);
  const int nw = blockDim.x >> 5, wid = t >> 5;
  const int cw = (ns + 31) >> 5;               // warps that chase; the others work on Q (all, if too few)
  const int qw = nw > cw ? nw - cw : nw, q0 = nw > cw ? wid - cw : wid;
  // what this chase carries from rotation to rotation: T[r+1][r-1] (the bulge), T[r][r-1], T[r][r] and
  // T[r+1][r] as the rotation before left them
  double g = 0.0, xe = 0.0, dr = 0.0, er = 0.0;
  for (int step = 0; step <= steps; ++step) {
    // rotation r = step - 3 s of shift s (the largest Ritz value first)
    const int r = step - 3 * t;
    if (t < ns && r >= 0 && r < m - 1) {
      if (r == 0) {
        dr = d[0];
        er = e[0];
        xe = dr - ritz[m - 1 - t];
        g = er;
      }
      const double dn = d[r + 1], en = (r + 2 < m) ? e[r + 1] : 0.0;
      const double h = fma(xe, xe, g * g);
      const double inv = (h == 0.0) ? 0.0 : rsqrt(h);
      const double c = (h == 0.0) ? 1.0 : xe * inv;
      const double sn = g * inv;
      rot[(step & 1) * kNcvMax + t] = make_double2(c, sn);
      if (r > 0) e[r - 1] = h * inv;
      const double cc = c * c, ss = sn * sn, cs = c * sn, t2 = 2.0 * cs * er;
      d[r] = cc * dr + t2 + ss * dn;
      xe = fma(cs, dn - dr, (cc - ss) * er);
      dr = ss * dr - t2 + cc * dn;
      g = sn * en;
      er = c * en;
      if (r == m - 2) {
        d[m - 1] = dr;
        e[m - 2] = xe;
      }
    }
    // the rotations of the step before, on every row of Q (disjoint pairs of columns): a warp per row,
    // a lane per shift
    const int prev = step - 1;
    if (prev >= 0 && q0 >= 0) {
      const int s_lo = max(0, (prev - (m - 2) + 2) / 3), s_hi = min(ns - 1, prev / 3);
      for (int s = s_lo + (t & 31); s <= s_hi; s += 32) {
        const double2 cs = rot[(prev & 1) * kNcvMax + s];
        double* col = Qd + prev - 3 * s;
#pragma unroll 4
        for (int q = q0; q < m; q += qw) {
          const double pv = col[q * m], qv = col[q * m + 1];
          col[q * m] = cs.x * pv + cs.y * qv;
          col[q * m + 1] = -cs.y * pv + cs.x * qv;
        }
      }
    }
    __syncthreads();
  }
  if (t < kk) {
    C->a[t] = d[t];
    if (t + 1 < kk) C->b[t] = e[t];
  }
  if (t == 0) {
    C->irl_beta = e[kk - 1];
    C->irl_sigma = Qd[(m - 1) * m + (kk - 1)];
    C->irl_k = kk;
  }
  if (inside)
    for (int idx = t; idx < m * m; idx += blockDim.x) Qg[idx] = Qd[idx];
  __syncthreads();
}

// sum_{k <= jmax} coef[k] V[k][i] in double, with the basis loads issued 8 at a time (independent
// loads keep the memory pipeline full; a plain loop over k would wait for each load in turn).
template <typename T>
__device__ __forceinline__ double basis_combine(const T* V, long long ldv, long long i, int jmax, const double* coef) {
  double acc = 0.0;
#pragma unroll 1
  for (int kb = 0; kb <= jmax; kb += 8) {
    T vv[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) vv[q] = (kb + q <= jmax) ? __ldcg(V + (long long)(kb + q) * ldv + i) : T(0);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (kb + q <= jmax) acc += coef[kb + q] * (double)vv[q];
  }
  return acc;
}

// 16-byte vector access to VW = 16 / sizeof(T) consecutive rows (rows of V, w, u, sigma are
// 256-byte aligned). Vector phases handle VW rows per thread per iteration, so every load
// instruction moves 16 bytes and a thread keeps several of them in flight.
template <typename T> struct Vec16;
template <> struct Vec16<float> { using type = float4; };
template <> struct Vec16<double> { using type = double2; };

template <typename T>
__device__ __forceinline__ void ld16(const T* p, T* out) {
  const typename Vec16<T>::type v = __ldcg(reinterpret_cast<const typename Vec16<T>::type*>(p));
  const T* c = reinterpret_cast<const T*>(&v);
#pragma unroll
  for (int r = 0; r < (int)(16 / sizeof(T)); ++r) out[r] = c[r];
}

template <typename T>
__device__ __forceinline__ void st16(T* p, const T* in) {
  typename Vec16<T>::type v;
  T* c = reinterpret_cast<T*>(&v);
#pragma unroll
  for (int r = 0; r < (int)(16 / sizeof(T)); ++r) c[r] = in[r];
  *reinterpret_cast<typename Vec16<T>::type*>(p) = v;
}

// ---- reductions of per-CTA partials --------------------------------------------------------

// Sum part[col * nblocks + blk] over blocks for cols [0, ncols) into out[col] (fixed order; not inlined:
// one copy serves every phase).
static __device__ __noinline__ void reduce_partials(const double* part, int nblocks, int ncols, double* out) {
  // a warp takes up to kCols columns (nw apart) and puts the loads of all of them in flight at once
  constexpr int kCols = 3;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int c0 = wid; c0 < ncols; c0 += nw * kCols) {
    double acc[kCols];
#pragma unroll
    for (int cc = 0; cc < kCols; ++cc) acc[cc] = 0.0;
    for (int b0 = lane; b0 < nblocks; b0 += 32 * 5) {
      double pv[kCols][5];
#pragma unroll
      for (int cc = 0; cc < kCols; ++cc) {
        const int c = c0 + cc * nw;
#pragma unroll
        for (int q = 0; q < 5; ++q) {
          pv[cc][q] = 0.0;
          if (c < ncols && b0 + 32 * q < nblocks) pv[cc][q] = __ldcg(part + (long long)c * nblocks + b0 + 32 * q);
        }
      }
#pragma unroll
      for (int cc = 0; cc < kCols; ++cc) {
#pragma unroll
        for (int q = 0; q < 5; ++q) acc[cc] += pv[cc][q];
      }
    }
#pragma unroll 1
    for (int cc = 0; cc < kCols && c0 + cc * nw < ncols; ++cc) {
      const double v = warp_sum(cc == 0 ? acc[0] : (cc == 1 ? acc[1] : acc[2]));
      if (lane == 0) out[c0 + cc * nw] = v;
    }
  }
  __syncthreads();
}

// This CTA's sums of up to three values per thread into out[0..nv) of thread 0..nv-1's return value (one
// copy, as above). sm: 3 doubles per warp.
static __device__ __noinline__ double cta_sums(double v0, double v1, double v2, int nv, double* sm) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll 1
  for (int q = 0; q < nv; ++q) {
    const double r = warp_sum(q == 0 ? v0 : (q == 1 ? v1 : v2));
    if (lane == 0) sm[wid * 3 + q] = r;
  }
  __syncthreads();
  double acc = 0.0;
  if ((int)threadIdx.x < nv)
    for (int w = 0; w < nw; ++w) acc += sm[w * 3 + threadIdx.x];
  return acc;
}

// A phase's sums over all CTAs of a solve. put stores this CTA's sum of a column, block_put reduces NV
// values per thread first, all_sum waits for every CTA and leaves the totals of `cols` columns in
// tot[] of every CTA. The partial sums (part: 2 x COLS x CTAs doubles) alternate between two buffers,
// since a CTA may store those of the next phase while another one still reads these; a single CTA's
// sums are the totals. sm: 3 doubles per warp of shared memory, tot: COLS.
template <class Pol, int COLS>
struct PhaseSums {
  const Pol& pol;
  GridSync* gs;
  double* part;
  double* sm;
  double* tot;
  unsigned int epoch;
  int buf = 0;
  __device__ __forceinline__ PhaseSums(const Pol& p, GridSync* g, double* pt, double* s, double* t)
      : pol(p), gs(g), part(pt), sm(s), tot(t), epoch(p.first_epoch(g)) {}
  __device__ __forceinline__ bool meet() { return pol.meet(gs, epoch); }
  __device__ __forceinline__ void put(int col, double v) {
    const int nblk = pol.nblocks();
    if (nblk == 1) tot[col] = v;
    else __stcg(part + ((long long)buf * COLS + col) * nblk + pol.block(), v);
  }
  template <int NV>
  __device__ __forceinline__ void block_put(const double (&v)[NV], int cols = NV) {
    static_assert(NV <= 3, "staging of block_put");
    const double acc = cta_sums(v[0], NV > 1 ? v[NV > 1] : 0.0, NV > 2 ? v[NV > 2 ? 2 : 0] : 0.0, cols, sm);
    if ((int)threadIdx.x < cols) put(threadIdx.x, acc);
  }
  __device__ __forceinline__ bool all_sum(int cols) {
    if (!meet()) return false;
    if (pol.nblocks() > 1) reduce_partials(part + (long long)buf * COLS * pol.nblocks(), pol.nblocks(), cols, tot);
    buf ^= 1;
    return true;
  }
};

// Sums of N (a power of two) values per lane over the warp: lane l returns the sum of value
// l / (32 / N). Halving the values at each of the first exchanges takes N - 1 + log2(32 / N) exchanges
// instead of 5 N.
template <int N>
__device__ __forceinline__ double warp_sum_batch(double (&v)[N]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = N / 2, o = 16; h >= 1; h >>= 1, o >>= 1) {
#pragma unroll
    for (int q = 0; q < h; ++q) {
      const double keep = (lane & o) ? v[q + h] : v[q], give = (lane & o) ? v[q] : v[q + h];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (int o = 16 / N; o >= 1; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// ---- the vector phases of a Lanczos step -----------------------------------------------------
// (Inlined: a call would save and restore tens of registers of 512 threads through local memory, which
// cost 4 to 15 us a phase at n = 2^20.)

// P2: the three-term step w' = w - a3 V[j] - b3 V[j-1] (first pass only), then this warp's parts of the
// reorthogonalisation coefficients h_k = V_k . w' (k <= j) and of w' . w' in red[warp][0 .. j + 1].
// Removing the dominant components explicitly first keeps the single Gram-Schmidt pass stable. w' goes to
// u (whose gathers are over), so that w can be read by several groups of threads.
template <typename T, bool kReadBack>
__device__ __forceinline__ void lanczos_dots(const T* V, long long ldv, const T* w, T* u, long long nvt, int j, int pass2,
                                          double a3, double b3, double* red_all, int gtid, int nthreads) {
  constexpr int VW = 16 / sizeof(T);
  const int lane = tid_here() & 31;
  double* red = red_all + (tid_here() >> 5) * kPartCols;
  const T* Vj = V + (long long)j * ldv;
  const T* Vm = V + (long long)(j > 0 ? j - 1 : 0) * ldv;
  for (int c = lane; c <= j + 1; c += 32) red[c] = 0.0;
  __syncwarp();
  // threads to spare: group g of them takes the batches g, g + groups, ... of basis vectors (each forms
  // w' itself), so that a small problem waits for one batch of loads instead of all of them in turn; with
  // one group a thread can read the w' back that it has stored (kReadBack)
  constexpr int KB = 4;
  const int batches = (j + KB) / KB;
  const int nvw = ((int)nvt + 31) & ~31;
  const int groups = max(1, min(batches, nthreads / nvw));
  const int span = (nthreads / groups) & ~31;
  const int grp = gtid / span, pos = gtid - grp * span;
  if (grp >= groups) return;
  for (int kb = grp * KB; kb <= j; kb += groups * KB) {
    const T* Vk = V + (long long)kb * ldv;
    double acc[KB], ww = 0.0;
#pragma unroll
    for (int q = 0; q < KB; ++q) acc[q] = 0.0;
    for (int iv = pos; iv < (int)nvt; iv += span) {
      const long long i0 = (long long)iv * VW;
      // every load of the position before the first use or store, so that all are in flight
      T wv[VW], vj[VW], vm[VW], vk[KB][VW];
      const bool form = !pass2 && (!kReadBack || kb == 0 || groups > 1);
      ld16(form || pass2 ? w + i0 : u + i0, wv);
      if (form) {
        ld16(Vj + i0, vj);
        ld16(Vm + i0, vm);
      }
#pragma unroll
      for (int q = 0; q < KB; ++q)
        if (kb + q <= j) ld16(Vk + q * ldv + i0, vk[q]);
      if (form) {
#pragma unroll
        for (int r = 0; r < VW; ++r) {
          double x = (double)wv[r] - a3 * (double)vj[r];
          if (j > 0) x -= b3 * (double)vm[r];
          wv[r] = (T)x;
        }
        if (kb == 0) st16(u + i0, wv);
      }
#pragma unroll
      for (int r = 0; r < VW; ++r) {
        const double wd = (double)wv[r];
        if (kb == 0) ww += wd * wd;
#pragma unroll
        for (int q = 0; q < KB; ++q)
          if (kb + q <= j) acc[q] += (double)vk[q][r] * wd;
      }
    }
    const double d = warp_sum_batch(acc);
    if ((lane & 7) == 0 && kb + (lane >> 3) <= j) red[kb + (lane >> 3)] = d;
    if (kb == 0) {
      ww = warp_sum(ww);
      if (lane == 0) red[j + 1] = ww;
    }
  }
}

// P3 for a batch team, whose threads have many positions: one thread a position. The lanes' split of
// lanczos_update, which then is one lane wide, left the update of 256 problems (n to 2^17, 145 teams) at 172 s
// of team time; this takes 73 s and the sweep 7.0 instead of 8.2 s (with 8 vectors in flight 97 s and 7.3).
template <typename T>
__device__ __forceinline__ double lanczos_update_all(const T* V, long long ldv, const T* src, const T* sigma, T* w, T* u,
                                                     long long nvt, int j, const double* h, int gtid, int nthreads) {
  constexpr int VW = 16 / sizeof(T), KB = 4;
  double ww = 0.0;
  for (int iv = gtid; iv < (int)nvt; iv += nthreads) {
    const long long i0 = (long long)iv * VW;
    T wv[VW], sg[VW];
    double corr[VW];
    ld16(src + i0, wv);
    ld16(sigma + i0, sg);
#pragma unroll
    for (int r = 0; r < VW; ++r) corr[r] = 0.0;
    const T* Vk = V + i0;
    for (int kb = 0; kb <= j; kb += KB, Vk += KB * ldv) {
      T vk[KB][VW];
#pragma unroll
      for (int q = 0; q < KB; ++q)
        if (kb + q <= j) ld16(Vk + q * ldv, vk[q]);
#pragma unroll
      for (int q = 0; q < KB; ++q) {
        if (kb + q <= j) {
          const double hk = h[kb + q];
#pragma unroll
          for (int r = 0; r < VW; ++r) corr[r] += hk * (double)vk[q][r];
        }
      }
    }
    T uv[VW];
#pragma unroll
    for (int r = 0; r < VW; ++r) {
      wv[r] = (T)((double)wv[r] - corr[r]);
      uv[r] = sg[r] * wv[r];
      ww += (double)wv[r] * (double)wv[r];
    }
    st16(w + i0, wv);
    st16(u + i0, uv);
  }
  return ww;
}

// P3: w = src - sum_k h_k V_k and u = sigma w; returns this thread's part of w . w. With threads to
// spare, up to 8 lanes of a warp share a position and split its basis vectors between them.
template <typename T>
__device__ __forceinline__ double lanczos_update(const T* V, long long ldv, const T* src, const T* sigma, T* w, T* u,
                                                 long long nvt, int j, const double* h, int gtid, int nthreads) {
  constexpr int VW = 16 / sizeof(T), KB = 4;
  double ww = 0.0;
  int sl = 0;
  while (sl < 3 && (nvt << (sl + 1)) <= nthreads) ++sl;
  const int lane = tid_here() & 31, per = 32 >> sl, sub = lane >> (5 - sl), lanes = 1 << sl;
  for (long long iv0 = (long long)(gtid >> 5) * per; iv0 < nvt; iv0 += nthreads >> sl) {
    const long long iv = iv0 + (lane & (per - 1)), i0 = iv * VW;
    const bool mine = iv < nvt;
    T wv[VW];
    double corr[VW];
#pragma unroll
    for (int r = 0; r < VW; ++r) corr[r] = 0.0;
    if (mine) {
      ld16(src + i0, wv);
      for (int kb = sub; kb <= j; kb += KB * lanes) {
        T vk[KB][VW];
#pragma unroll
        for (int q = 0; q < KB; ++q)
          if (kb + q * lanes <= j) ld16(V + (long long)(kb + q * lanes) * ldv + i0, vk[q]);
#pragma unroll
        for (int q = 0; q < KB; ++q) {
          if (kb + q * lanes <= j) {
            const double hk = h[kb + q * lanes];
#pragma unroll
            for (int r = 0; r < VW; ++r) corr[r] += hk * (double)vk[q][r];
          }
        }
      }
    }
#pragma unroll 1
    for (int o = per; o < 32; o <<= 1) {
#pragma unroll
      for (int r = 0; r < VW; ++r) corr[r] += __shfl_xor_sync(0xffffffffu, corr[r], o);
    }
    if (mine && sub == 0) {
      T sg[VW], uv[VW];
      ld16(sigma + i0, sg);
#pragma unroll
      for (int r = 0; r < VW; ++r) {
        wv[r] = (T)((double)wv[r] - corr[r]);
        uv[r] = sg[r] * wv[r];
        ww += (double)wv[r] * (double)wv[r];
      }
      st16(w + i0, wv);
      st16(u + i0, uv);
    }
  }
  return ww;
}

// The same two phases for problems that fill the GPU: every CTA owns a contiguous range of rows and
// streams the vectors' tiles of it (kStreamTile bytes a vector, kStreamVecs vectors a group) into
// shared memory with bulk asynchronous copies, kStreamBufs groups in flight. What bounds them is the
// reading of the basis (from L2 and HBM); loads held in registers either keep too few bytes in flight
// or take so many registers that the persistent kernel spills them through an L1 that the panels leave
// 30 KB. At n = 2^20 (20 vectors) the dots move 3.3 TB/s and the update 3.8 TB/s with the FP32 to FP64
// conversions (16 a cycle and SM) next in line; one step's dots and update went from 73 to 52.5 us,
// Ritz test and barriers included.
// Buffers: three where the panels take as much shared memory anyway (FP32). Without panels two, since the
// gathers of the work list and of the splits live on what is left to L1: with three (28 KB of L1) a step's
// SpMV on BA(2^22, 10) took 900 us, with two (92 KB) 617 us, the vector phases 132 and 135 us; on BA(2^20, 4)
// 105 and 70 us, and 48 and 46 us. Tiles of 8 KB with two buffers (156 KB of L1): SpMV 567 and 68 us, vector
// phases 167 and 56 us.
constexpr int kStreamTile = 16 * 1024;
constexpr int kStreamVecs = 4;
__host__ __device__ constexpr int stream_bufs(int elem, bool panels) { return panels && elem == 4 ? 3 : 2; }
__host__ __device__ constexpr int stream_smem_bytes(int elem, bool panels) {
  return stream_bufs(elem, panels) * kStreamVecs * kStreamTile;
}

template <typename T, int kBufs>
struct VecStream {
  static constexpr int VW = 16 / sizeof(T);
  static constexpr int kTileRows = kStreamTile / sizeof(T);
  static constexpr int kChunks = kStreamTile / (16 * kThreads);   // 16-byte chunks of a tile per thread
  char* smem;
  unsigned long long* bars;   // kBufs mbarriers of one arrival
  unsigned& par;              // their phase bits
  int* err;
  unsigned long long spin_limit = kPanelSpinLimit;
  long long r0;               // first row, rows of the range and of a tile, number of tiles
  int rows, sub, tiles;

  // the CTA's range of n_pad rows (a multiple of VW)
  __device__ __forceinline__ VecStream(char* sm, unsigned long long* b, unsigned& p, int* e, long long n_pad, int blk,
                                       int nblk)
      : smem(sm), bars(b), par(p), err(e) {
    const long long per = ((n_pad + nblk - 1) / nblk + VW - 1) / VW * VW;
    r0 = min(n_pad, per * blk);
    rows = (int)(min(n_pad, r0 + per) - r0);
    tiles = (rows + kTileRows - 1) / kTileRows;
    sub = tiles ? ((rows + tiles - 1) / tiles + VW - 1) / VW * VW : 0;
  }
  __device__ __forceinline__ int tile_rows(int t) const { return min(sub, rows - t * sub); }
  __device__ __forceinline__ long long tile_row0(int t) const { return r0 + (long long)t * sub; }

  // Runs nv vectors (vec(v): the v-th one's base) over all tiles. begin(t) and end(t) bracket a tile;
  // group(t, g, m, base) works on vectors 4 g .. 4 g + m - 1 of tile t, whose tiles lie kStreamTile
  // apart from base. False, with SA_ERR_BARRIER_TIMEOUT in *err, if a copy does not complete in time.
  template <class Vec, class Begin, class Group, class End>
  __device__ __forceinline__ bool run(int nv, Vec&& vec, Begin&& begin, Group&& group, End&& end) {
    const int ng = (nv + kStreamVecs - 1) / kStreamVecs, total = ng * tiles;
    // copies of group k, by the first lanes of one warp (one vector each: in a single thread their issue
    // would hold up its warp, and with it the group)
    auto issue = [&](int k) {
      const int q = threadIdx.x & 31;
      const int t = k / ng, g = k - t * ng, b = k % kBufs;
      const int m = min(kStreamVecs, nv - g * kStreamVecs);
      const unsigned bytes = (unsigned)(tile_rows(t) * sizeof(T));
      if (q == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bars[b])), "r"(bytes * m)
                     : "memory");
      __syncwarp();
      if (q < m) {
        if (k < kBufs) fence_proxy_async();   // (before the first copies; a refill only follows reads)
        bulk_load(smem + (b * kStreamVecs + q) * kStreamTile, vec(g * kStreamVecs + q) + tile_row0(t), bytes, &bars[b]);
      }
    };
    const int wid = threadIdx.x >> 5;
    if (wid < kBufs && wid < total) issue(wid);
    int k = 0;
    for (int t = 0; t < tiles; ++t) {
      begin(t);
      for (int g = 0; g < ng; ++g, ++k) {
        const int b = k % kBufs;
        const unsigned par0 = par;
        bool late = false;
        for (unsigned long long spins = 0; !mbar_try_wait(&bars[b], (par0 >> b) & 1u);)
          if (++spins > spin_limit) {
            late = true;
            break;
          }
        late = __any_sync(0xffffffffu, late);
        par ^= 1u << b;
        if (!late) group(t, g, min(kStreamVecs, nv - g * kStreamVecs), smem + b * kStreamVecs * kStreamTile);
        if (__syncthreads_or(late)) {
          // as in the panel SpMV: record, wait (bounded) for the copies in flight, return together
          if (threadIdx.x == 0) {
            atomicExch(err, SA_ERR_BARRIER_TIMEOUT);
            for (int q = k; q < k + kBufs && q < total; ++q) {
              const int qb = q % kBufs;
              for (unsigned long long spins = 0; !mbar_try_wait(&bars[qb], (par0 >> qb) & 1u);)
                if (++spins > spin_limit) break;
            }
          }
          __syncthreads();
          return false;
        }
        if (wid == k % kWarps && k + kBufs < total) issue(k + kBufs);
      }
      end(t);
    }
    return true;
  }
};

// P2 streamed. The vectors in order: w, V[j], V[j-1], V[0], V[1], ..., V[j-2]; the first three give w',
// which stays in registers for the tile.
template <typename T, int kBufs>
__device__ __forceinline__ bool stream_dots(VecStream<T, kBufs>& S, const T* V, long long ldv, const T* w, T* u, int j, int pass2,
                                            double a3, double b3, double* red_all) {
  constexpr int VW = VecStream<T, kBufs>::VW, NC = VecStream<T, kBufs>::kChunks;
  const int tid = tid_here(), lane = tid & 31;
  double* red = red_all + (tid >> 5) * kPartCols;
  for (int c = lane; c <= j + 1; c += 32) red[c] = 0.0;
  __syncwarp();
  auto index = [&](int v) { return v == 1 ? j : (v == 2 ? j - 1 : v - 3); };
  double wd[NC][VW], ww = 0.0;
  const bool ok = S.run(
      j + 2, [&](int v) { return v == 0 ? w : V + (long long)index(v) * ldv; }, [](int) {},
      [&](int t, int g, int m, const char* base) {
        const T* x = (const T*)base;
        const int cnt = S.tile_rows(t);
        if (g == 0) {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int at = (c * kThreads + tid) * VW;
            T wv[VW];
#pragma unroll
            for (int r = 0; r < VW; ++r) wv[r] = T(0);
            if (at < cnt) {
              ld_filled16(x + at, wv);
              if (!pass2) {
                T vj[VW], vm[VW];
                ld_filled16(x + kStreamTile / sizeof(T) + at, vj);
                if (j > 0) ld_filled16(x + 2 * (kStreamTile / sizeof(T)) + at, vm);
#pragma unroll
                for (int r = 0; r < VW; ++r) {
                  double y = (double)wv[r] - a3 * (double)vj[r];
                  if (j > 0) y -= b3 * (double)vm[r];
                  wv[r] = (T)y;
                }
                st16(u + S.tile_row0(t) + at, wv);
              }
            }
#pragma unroll
            for (int r = 0; r < VW; ++r) {
              wd[c][r] = (double)wv[r];
              ww += wd[c][r] * wd[c][r];
            }
          }
        }
        double acc[kStreamVecs];
#pragma unroll
        for (int q = 0; q < kStreamVecs; ++q) {
          acc[q] = 0.0;
          if (q < m && (g > 0 || q > 0)) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              const int at = (c * kThreads + tid) * VW;
              if (at < cnt) {
                T vk[VW];
                ld_filled16(x + q * (kStreamTile / sizeof(T)) + at, vk);
#pragma unroll
                for (int r = 0; r < VW; ++r) acc[q] += (double)vk[r] * wd[c][r];
              }
            }
          }
        }
        const double d = warp_sum_batch(acc);
        const int q = lane >> 3, v = g * kStreamVecs + q;
        if ((lane & 7) == 0 && q < m && v > 0) red[index(v)] += d;
      },
      [](int) {});
  ww = warp_sum(ww);
  if (lane == 0) red[j + 1] = ww;
  return ok;
}

// P3 streamed: the vectors in order src, sigma, V[0], ..., V[j]. Adds this thread's part of w . w to ww.
template <typename T, int kBufs>
__device__ __forceinline__ bool stream_update(VecStream<T, kBufs>& S, const T* V, long long ldv, const T* src, const T* sigma,
                                              T* w, T* u, int j, const double* h, double& ww) {
  constexpr int VW = VecStream<T, kBufs>::VW, NC = VecStream<T, kBufs>::kChunks;
  const int tid = tid_here();
  T wv[NC][VW], sg[NC][VW];
  double corr[NC][VW];
  return S.run(
      j + 3, [&](int v) { return v == 0 ? src : (v == 1 ? sigma : V + (long long)(v - 2) * ldv); },
      [&](int) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
          for (int r = 0; r < VW; ++r) corr[c][r] = 0.0;
      },
      [&](int t, int g, int m, const char* base) {
        const T* x = (const T*)base;
        const int cnt = S.tile_rows(t);
#pragma unroll
        for (int q = 0; q < kStreamVecs; ++q) {
          if (q >= m) break;
          const double hk = (g > 0 || q > 1) ? h[g * kStreamVecs + q - 2] : 0.0;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int at = (c * kThreads + tid) * VW;
            if (at < cnt) {
              T vk[VW];
              ld_filled16(x + q * (kStreamTile / sizeof(T)) + at, vk);
              if (g == 0 && q < 2) {
#pragma unroll
                for (int r = 0; r < VW; ++r) (q == 0 ? wv : sg)[c][r] = vk[r];
              } else {
#pragma unroll
                for (int r = 0; r < VW; ++r) corr[c][r] += hk * (double)vk[r];
              }
            }
          }
        }
      },
      [&](int t) {
        const int cnt = S.tile_rows(t);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int at = (c * kThreads + tid) * VW;
          if (at < cnt) {
            T uv[VW];
#pragma unroll
            for (int r = 0; r < VW; ++r) {
              wv[c][r] = (T)((double)wv[c][r] - corr[c][r]);
              uv[r] = sg[c][r] * wv[c][r];
              ww += (double)wv[c][r] * (double)wv[c][r];
            }
            st16(w + S.tile_row0(t) + at, wv[c]);
            st16(u + S.tile_row0(t) + at, uv);
          }
        }
      });
}

// Restart: kept basis V[0..kk) <- V Q[:, 0..kk) and the new residual f = V Q[:, kk] beta + w sig (in w,
// with u = sigma f), row by row in place (all m inputs of a row are read before its kk outputs are
// written); returns this thread's part of f . f. q: m x (kk + 1) in shared memory. KK: kk when it is
// known at compile time (the default), else 0.
template <typename T, int KK>
__device__ __forceinline__ double restart_basis(T* V, long long ldv, T* w, T* u, const T* sigma, long long n, int m, int kk_,
                                             const double* q, double beta, double sig, long long gtid,
                                             long long nthreads) {
  constexpr int KM = KK > 0 ? KK : kRestartMax;
  const int kk = KK > 0 ? KK : kk_;
  double ff = 0.0;
#pragma unroll 1
  for (long long i = gtid; i < n; i += nthreads) {
    double y[KM + 1];
#pragma unroll
    for (int c = 0; c <= KM; ++c) y[c] = 0.0;
    const double wi = (double)__ldcg(w + i);
#pragma unroll 1
    for (int r0 = 0; r0 < m; r0 += 8) {
      T vr[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) vr[r] = (r0 + r < m) ? __ldcg(V + (long long)(r0 + r) * ldv + i) : T(0);
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r0 + r < m) {
          const double* qr = q + (r0 + r) * (kk + 1);
#pragma unroll
          for (int c = 0; c <= KM; ++c)
            if (KK > 0 || c <= kk) y[c] += (double)vr[r] * qr[c];
        }
      }
    }
#pragma unroll
    for (int c = 0; c < KM; ++c)
      if (KK > 0 || c < kk) V[(long long)c * ldv + i] = (T)y[c];
    double yk = y[KM];
    if (KK == 0) {
#pragma unroll
      for (int c = 0; c <= KM; ++c)
        if (c == kk) yk = y[c];
    }
    const T f = (T)(yk * beta + wi * sig);
    w[i] = f;
    u[i] = sigma[i] * f;
    ff += (double)f * (double)f;
  }
  return ff;
}

template <typename T>
__device__ __forceinline__ T vload(const T* p) { return *((volatile const T*)p); }

__device__ __forceinline__ unsigned long long word_mix(long long widx, unsigned int word) {
  return splitmix64(((unsigned long long)widx << 32) ^ (unsigned long long)word ^ 0xA5A5000000000000ull);
}

// ---- the alpha-solve kernel ----------------------------------------------------------------

// Shared work space of a CTA: the SpMV's staging, the warps' dots, or the tridiagonal solvers' and the
// restart's scratch (never two of them at a time).
template <typename T, int NW>
union AlphaWork {
  SpmvSmem<T, NW> spmv;
  double dots[NW * kPartCols];
  double restart[kNcvMax * (kRestartMax + 1)];
};

template <typename T, int NW>
__device__ __forceinline__ AlphaWork<T, NW>& alpha_work() {
  __shared__ __align__(16) AlphaWork<T, NW> w;
  return w;
}

// What a row does with its sum s = sum_j val_ij u_j: in a Lanczos step (P1) V[j] = w * inv_b and
// w <- S V[j], adding V[j] . w to acc; in the final pass (last) |S y - theta y|^2 is added to it.
template <typename T>
struct RowStep {
  const T* xin;   // w, or y in the final pass
  const T* sigma;
  T* vj;
  T* w;
  T rho, inv_b;
  double theta;
  bool last;
  double acc;
  // Parts of V[j] . w from rows that any warp may finish, as multiples of 1 / scale: their sum is exact, so
  // a_j, and with it every later step, does not depend on which warp it was.
  double scale;
  long long fixed;
  __device__ __forceinline__ RowInputs<T> pre(long long r) const { return RowInputs<T>{__ldcg(xin + r), __ldcg(sigma + r)}; }
  template <bool kAny = false>
  __device__ __forceinline__ void fin(long long r, T s, const RowInputs<T>& in) {
    const T wr = in.x;
    const T sw = rho * wr - in.s * s;
    if (last) {
      const double rr = (double)sw - theta * (double)wr;
      acc += rr * rr;
    } else {
      const T vr = wr * inv_b;
      const T wn = sw * inv_b;
      vj[r] = vr;
      w[r] = wn;
      const double part = (double)vr * (double)wn;
      if (kAny) fixed += __double2ll_rn(part * scale);
      else acc += part;
    }
  }
};

// The operator layouts.
template <typename T>
__device__ __forceinline__ bool panel_pass(const PanelArgs& P, const T* u, int blk, int nblk, unsigned long long* bars,
                                        unsigned& par, int* err, RowStep<T>& out) {
  extern __shared__ __align__(128) char panel_smem[];
  RowStep<T> f = out;
  unsigned pr = par;
  const bool ok = panel_spmv<T>(P, u, blk, nblk, panel_smem, bars, pr, err, [&](long long r) { return f.pre(r); },
                                [&](long long r, T s, const RowInputs<T>& in) { f.fin(r, s, in); });
  par = pr;
  out.acc = f.acc;
  return ok;
}

// mode: bit 0 the first of the passes that make up a row's sum, bit 1 the last one (sums between the
// passes in `part`).
template <typename T, typename RP, int NW>
__device__ __forceinline__ void items_pass(const SpmvArgs<T, RP>& S, const T* u, int gwarp, int nwarps, RowStep<T>& out,
                                        T* part, int mode) {
  RowStep<T> f = out;
  const SpmvArgs<T, RP> L = S;
  auto row = [&](auto any, long long r, T s) {
    const T sum = (mode & 1) ? s : __ldcg(part + r) + s;
    if (mode & 2) f.template fin<decltype(any)::value>(r, sum, f.pre(r));
    else __stcg(part + r, sum);
  };
  spmv_items<T, RP, false, NW>(L, u, gwarp, nwarps, alpha_work<T, NW>().spmv,
                               [&](long long r, T s) { row(std::false_type{}, r, s); },
                               [&](long long r, T s) { row(std::true_type{}, r, s); });
  out.fixed = f.fixed;
  out.acc = f.acc;
}

// What a kernel is compiled for: the work list with register-held vector phases (small problems and the batch
// kernel); the column panels with streamed vector phases; the work list or the L2 column splits with
// streamed vector phases; the column panels with register-held ones. All in one spilled up to 916 bytes a
// thread through the little L1 that the panels leave; each by itself spills 284 to 484 bytes of stores in
// FP32 and 204 to 604 in FP64, outside the phases' inner loops.
enum AlphaMode : int { ALPHA_SMALL = 0, ALPHA_PANEL = 1, ALPHA_LARGE = 2, ALPHA_PANEL_SMALL = 3 };
__host__ __device__ constexpr bool alpha_panels(int mode) { return mode == ALPHA_PANEL || mode == ALPHA_PANEL_SMALL; }
__host__ __device__ constexpr bool alpha_streams(int mode) { return mode == ALPHA_PANEL || mode == ALPHA_LARGE; }

// NW: warps per CTA at most (sizes the shared staging).
template <typename T, typename RP, class Pol, int NW, int kMode>
__device__ __forceinline__ void alpha_body(const AlphaArgs<T, RP>& A, const Pol& pol) {
  static_assert(2 * kTriPad + 7 * kNcvMax <= kNcvMax * (kRestartMax + 1), "restart scratch too small");
  AlphaWork<T, NW>& work = alpha_work<T, NW>();
  __shared__ double sm[3 * NW];
  __shared__ double tot[kPartCols];   // totals of the last phase's partial sums
  __shared__ AlphaCtrl ctl;
  __shared__ unsigned long long pbars[kPanelBufs], vbars[stream_bufs(sizeof(T), alpha_panels(kMode))];
  double* const sq = work.restart;
  AlphaCtrl* const C = &ctl;     // this CTA's copy of the control block
  AlphaCtrl* const G = A.ctrl;   // barrier, flags and signature of the whole grid; the copy that is published
  const long long n = A.n;
  const long long gtid = pol.tid();
  const long long nthreads = pol.nthr();
  const int nblk = pol.nblocks(), blk = pol.block();
  const sa_alpha_params& P = A.p;
  const double rho = P.rho;
  const double bound = 10.0 * (P.rho + P.gershgorin);
  // |a_j| is at most 2 rho < bound: 2^61 / bound or more keeps the sums of RowStep::fixed below 2^62
  const double fix_scale = scalbn(1.0, 60 - ilogb(fmax(bound, 1.0)));
  const int ncv = P.ncv;
  constexpr int VW = 16 / sizeof(T);
  const long long nvt = (n + VW - 1) / VW;   // positions of the vector phases
  unsigned ppar = 0;   // phase bits of the panel barriers
  if (alpha_panels(kMode)) panel_init(pbars, kPanelBufs);
  unsigned vpar = 0;   // and of the vector streams'
  if (alpha_streams(kMode)) panel_init(vbars, stream_bufs(sizeof(T), alpha_panels(kMode)));
  PhaseSums<Pol, kPartCols> sums(pol, &G->gs, A.part, sm, tot);
  // one operator application (this thread's sum goes to f.acc); false on a timed-out wait
  auto apply = [&](RowStep<T>& f) -> bool {
    if constexpr (alpha_panels(kMode)) {
      return panel_pass<T>(A.panel, A.u, blk, nblk, pbars, ppar, &G->gs.error, f);
    } else {
      // pass q adds the row sums of split q (the work list is one pass); a barrier makes them visible to
      // the next pass
      const int passes = kMode == ALPHA_LARGE && A.n_splits > 0 ? A.n_splits : 1;
#pragma unroll 1
      for (int q = 0; q < passes; ++q) {
        const bool last = q + 1 == passes;
        const SpmvArgs<T, RP>& S = kMode == ALPHA_LARGE && A.n_splits > 0 ? A.split[q] : A.S;
        items_pass<T, RP, NW>(S, A.u, (int)(pol.tid() >> 5), (int)(nthreads >> 5), f, A.split_part,
                              (q == 0 ? 1 : 0) | (last ? 2 : 0));
        if (!last && !sums.meet()) return false;
      }
      return true;
    }
  };

  // phase timer: CTA 0 thread 0 charges the time since the previous barrier exit to a phase
  unsigned long long t_mark = (blk == 0 && threadIdx.x == 0) ? global_ns() : 0ull;
  auto mark = [&](int ph) {
    if (blk == 0 && threadIdx.x == 0) {
      const unsigned long long t = global_ns();
      C->tph[ph] += t - t_mark;
      t_mark = t;
    }
  };
  // the control block as the host and the batched sweep read it (all but the barrier, the flag and the
  // signature, which the grid shares)
  auto publish = [&] {
    if (blk != 0) return;
    __syncthreads();
    for (int i = threadIdx.x; i < kNcvMax; i += blockDim.x) {
      G->a[i] = C->a[i];
      G->b[i] = C->b[i];
      G->h[i] = C->h[i];
      G->s[i] = C->s[i];
    }
    if (threadIdx.x == 0) {
      G->theta = C->theta;
      G->inv_b = C->inv_b;
      G->ww = C->ww;
      G->scale = C->scale;
      G->nrm_y = C->nrm_y;
      G->rr = C->rr;
      G->j = C->j;
      G->action = C->action;
      G->iters = C->iters;
      G->restarts = C->restarts;
      G->mode = C->mode;
      G->pred_residual = C->pred_residual;
      G->pred_accepted = C->pred_accepted;
      G->status = C->status;
      G->degree_scale = C->degree_scale;
      G->align_dot = C->align_dot;
      G->res_est = C->res_est;
      G->bytes = C->bytes;
      G->spmvs = C->spmvs;
      for (int q = 0; q < 6; ++q) G->tph[q] = C->tph[q];
    }
  };

  // ---------------- P0: sigma, degree scale, start vector --------------------------------------
  int mode = P.start_mode;
  if (threadIdx.x == 0) {
    if (blk == 0) {
      G->nonfinite = 0;
      G->sig = 0ull;
    }
    C->mode = mode;
    C->test_pred = (mode == SA_START_DIAGONAL || mode == SA_START_SECANT || mode == SA_START_TANGENT) ? 1 : 0;
    C->pred_accepted = -1;
    C->pred_residual = nan("");
    C->iters = 0;
    C->restarts = 0;
    C->status = SA_OK;
    C->secant_sign = 1;
    C->bytes = 0.0;
    C->spmvs = 0;
    C->theta = C->res_est = C->nrm_y = C->rr = C->scale = C->align_dot = C->ww = 0.0;
    C->j = 0;
    C->pass2 = 0;
    for (int q = 0; q < 6; ++q) C->tph[q] = 0ull;
  }
  // the vector phases move whole 16-byte positions: the rows of the last one past n are zeros in
  // every vector (they are inside each array's allocation) and stay zeros
  {
    const int past = (int)(nvt * VW - n);
    for (long long i = gtid; i < (long long)past * (ncv + 3); i += nthreads) {
      const int k = (int)(i / past);
      T* const x = k < ncv ? A.V + (long long)k * A.ldv : (k == ncv ? A.w : (k == ncv + 1 ? A.u : A.sigma));
      x[n + i % past] = T(0);
    }
  }
  {
    double ds = 0.0;
#pragma unroll 1
    for (long long i = gtid; i < n; i += nthreads) {
      const double ldi = (double)A.ld[i];
      const double ai = A.aoff ? P.alpha + A.aoff[i] : P.alpha;
      const double logD = (ai == 0.0) ? 0.0 : ai * ldi;
      const double logDc = fmax(logD, kLog2Clamp);
      A.sigma[i] = (T)exp2(-0.5 * logDc - A.half_log2_c);
      ds += exp2(logD);
    }
    double v[1] = {ds};
    sums.block_put(v);
  }
  if (!sums.all_sum(1)) return;
  if (threadIdx.x == 0) {
    C->degree_scale = tot[0];
    C->bytes += (double)n * (8.0 + sizeof(T));
  }
  mark(0);

  if (mode == SA_START_SECANT && A.has_prev) {
    double v[1] = {0.0};
#pragma unroll 1
    for (long long i = gtid; i < n; i += nthreads) v[0] += (double)A.ylast[i] * (double)A.yprev[i];
    sums.block_put(v);
    if (!sums.all_sum(1)) return;
    if (threadIdx.x == 0) {
      C->secant_sign = (tot[0] < 0.0) ? -1 : 1;
      C->bytes += 2.0 * (double)n * sizeof(T);
    }
    mark(0);
  }

  while (true) {   // P0 loop (repeats for a predictor fallback or rejection)
    __syncthreads();
    mode = C->mode;
    const int sgn = C->secant_sign;
    const unsigned long long key = splitmix64(P.seed ^ 0x57A27000ull) ^ splitmix64((unsigned long long)P.stream_id + 0x1234567ull);
    double v[3] = {0.0, 0.0, 0.0};   // ||v0||^2, ||s||^2 (secant), ||y||^2 (secant)
#pragma unroll 1
    for (long long i = gtid; i < n; i += nthreads) {
      double x;
      if (mode == SA_START_RANDOM) {
        x = (double)(T)normal_from_counter(key, i);
      } else if (mode == SA_START_PREV) {
        x = (double)A.ylast[i];
      } else if (mode == SA_START_GIVEN) {
        x = (double)A.v0[i];
      } else if (mode == SA_START_TANGENT) {
        // first-order step along the eigenvector tangent dy/dalpha at alpha_prev (given in v0)
        x = (double)(T)(A.ylast[i] + (T)(P.alpha - P.alpha_prev) * A.v0[i]);
      } else if (mode == SA_START_DIAGONAL) {
        const double ldi = fmax((double)A.ld[i], kLog2Clamp);
        const T wgt = (T)exp2(0.5 * (P.alpha - P.alpha_prev) * ldi);
        x = (double)(T)(wgt * A.ylast[i]);
      } else {   // SECANT
        const T yl = A.ylast[i];
        const T yp = A.has_prev ? (T)(sgn * A.yprev[i]) : yl;
        const T sdiff = (T)(yl - yp);
        x = (double)(T)(yl + (T)P.secant_gamma * sdiff);
        v[1] += (double)sdiff * (double)sdiff;
      }
      const T xt = (T)x;
      A.w[i] = xt;
      A.u[i] = A.sigma[i] * xt;
      v[0] += (double)xt * (double)xt;
    }
    v[2] = v[0];
    sums.block_put(v);
    if (!sums.all_sum(3)) return;
    if (threadIdx.x == 0) {
      const int md = C->mode;
      const double nrm = sqrt(tot[0]);
      const double nin = (md == SA_START_RANDOM) ? 0.0 : ((md == SA_START_SECANT || md == SA_START_TANGENT) ? 2.0 : 1.0);
      C->bytes += (double)n * sizeof(T) * (2.0 + nin) + (md == SA_START_DIAGONAL ? 8.0 * n : 0.0);
      C->action = ACT_NEXT;
      if (md == SA_START_DIAGONAL && nrm < kTinyNorm) {
        C->mode = SA_START_RANDOM;           // utils/predictors.py:22-25
        C->action = ACT_P0_AGAIN;
      } else if (md == SA_START_SECANT &&
                 (!A.has_prev || sqrt(tot[1]) < kTinyNorm || nrm < kTinyNorm)) {
        C->mode = SA_START_PREV;             // utils/predictors.py:44-55
        C->action = ACT_P0_AGAIN;
      } else if (md == SA_START_TANGENT && (!A.has_last || !(nrm >= kTinyNorm) || !isfinite(nrm))) {
        C->mode = SA_START_PREV;             // as the secant fallback
        C->action = ACT_P0_AGAIN;
      } else if (!(nrm > 0.0) || !isfinite(nrm)) {
        C->status = SA_ERR_NONFINITE;
        C->action = ACT_ERROR;
      } else {
        C->inv_b = 1.0 / nrm;
        C->j = 0;
        C->pass2 = 0;
      }
      C->ritz_ok = 0;
    }
    mark(0);
    __syncthreads();
    const int act = C->action;
    if (act == ACT_P0_AGAIN) continue;
    if (act == ACT_ERROR) {
      publish();
      return;
    }

    // ---------------- Lanczos steps ----------------------------------------------------------
    bool restart_p0 = false;
    while (true) {
      const int j = C->j;
      const int pass2 = C->pass2;
      const bool last = C->action == ACT_DONE;   // the final pass: the true residual of y (F2)
      if (!pass2 && (!last || P.residual_check)) {
        // P1: V[j] = w * inv_b; w <- S V[j]; partial sums of a_j = V[j] . w. (The final pass shares the
        // operator's code: F2 |S y - theta y|^2.)
        RowStep<T> f{last ? A.yout : A.w, A.sigma, A.V + (long long)j * A.ldv, A.w, (T)rho, (T)C->inv_b, C->theta, last, 0.0, fix_scale, 0ll};
        if (!apply(f)) return;
        // the fixed-point part in two columns, whose sums are exact integers in any order
        const int cols = !last && !alpha_panels(kMode) && A.long_rows ? 3 : 1;
        const double pa[3] = {f.acc, (double)(f.fixed >> 32), (double)(f.fixed & 0xffffffffll)};
        sums.block_put(pa, cols);
        if (last) break;
        if (!sums.all_sum(cols)) return;
        if (threadIdx.x == 0) {
          C->a[j] = cols == 1 ? tot[0] : tot[0] + (tot[1] * 0x1p32 + tot[2]) / fix_scale;
          C->bytes += A.spmv_bytes + (double)n * sizeof(T);
          C->spmvs += 1;
        }
        mark(1);
        __syncthreads();
      }
      if (last) break;
      // P2: three-term step and reorthogonalisation coefficients
      {
        const double a3 = pass2 ? 0.0 : C->a[j], b3 = (pass2 || j == 0) ? 0.0 : C->b[j - 1];
        if constexpr (alpha_streams(kMode)) {
          extern __shared__ __align__(128) char stream_smem[];
          VecStream<T, stream_bufs(sizeof(T), alpha_panels(kMode))> S(stream_smem, vbars, vpar, &G->gs.error, nvt * VW, blk, nblk);
          if (!stream_dots(S, A.V, A.ldv, A.w, A.u, j, pass2, a3, b3, work.dots)) return;
        } else {
          lanczos_dots<T, Pol::kManyPositions>(A.V, A.ldv, A.w, A.u, nvt, j, pass2, a3, b3, work.dots, (int)pol.tid(), (int)nthreads);
        }
        __syncthreads();
        if (threadIdx.x <= j + 1) {
          double acc = 0.0;
#pragma unroll 4
          for (int w = 0; w < (int)(blockDim.x >> 5); ++w) acc += work.dots[w * kPartCols + threadIdx.x];
          sums.put(threadIdx.x, acc);
        }
        if (!sums.all_sum(j + 2)) return;
        if (threadIdx.x <= j) C->h[threadIdx.x] = tot[threadIdx.x];
        if (threadIdx.x == 0) {
          C->ww = tot[j + 1];
          C->a[j] += tot[j];
          C->bytes += (double)n * sizeof(T) * (double)(j + 2 + (pass2 ? 0 : 3));
        }
        mark(2);
        __syncthreads();
      }
      // P3: w = w' - sum_k h_k V_k ; u = sigma w ; ww2
      {
        const T* src = pass2 ? A.w : A.u;
        double v[1] = {0.0};
        if constexpr (alpha_streams(kMode)) {
          extern __shared__ __align__(128) char stream_smem[];
          VecStream<T, stream_bufs(sizeof(T), alpha_panels(kMode))> S(stream_smem, vbars, vpar, &G->gs.error, nvt * VW, blk, nblk);
          if (!stream_update(S, A.V, A.ldv, src, A.sigma, A.w, A.u, j, C->h, v[0])) return;
        } else {
          if (Pol::kManyPositions && 2 * nvt > nthreads)
            v[0] = lanczos_update_all<T>(A.V, A.ldv, src, A.sigma, A.w, A.u, nvt, j, C->h, (int)pol.tid(), (int)nthreads);
          else
            v[0] = lanczos_update<T>(A.V, A.ldv, src, A.sigma, A.w, A.u, nvt, j, C->h, (int)pol.tid(), (int)nthreads);
        }
        sums.block_put(v);
      }
      if (!sums.all_sum(1)) return;
      const double ww2 = tot[0];
      const double bj = sqrt(ww2);
      if (threadIdx.x == 0) {
        const double aj = C->a[j];
        C->action = ACT_NEXT;
        C->bytes += (double)n * sizeof(T) * (double)(j + 5);
        if (!C->pass2) C->iters += 1;
        if (!isfinite(aj) || !isfinite(bj) || fabs(aj) > bound || bj > bound) {
          C->status = SA_ERR_BREAKDOWN;   // models/spectral_annealing.py:85-120
          C->action = ACT_ERROR;
        } else if (C->test_pred && j == 0) {
          C->test_pred = 0;
          C->pred_residual = bj;
          C->pred_accepted = (bj > P.pred_tol) ? 0 : 1;
          if (bj > P.pred_tol) {           // models/spectral_annealing.py:610-612
            C->mode = SA_START_PREV;
            C->iters = 0;
            C->action = ACT_REJECT;
          }
        }
        if (C->action == ACT_NEXT && !C->pass2 && ww2 < 1e-4 * C->ww && bj > 1e-14 * bound) {
          C->pass2 = 1;                    // second Gram-Schmidt pass
          C->action = ACT_REPASS;
        }
        C->pass2 = (C->action == ACT_REPASS) ? 1 : 0;
      }
      __syncthreads();
      if (C->action == ACT_NEXT) {
        const int m = j + 1;
        double s2;
        // previous step's Ritz value and residual estimate as the bracket to try first
        double hlo = 0.0, hhi = -1.0;
        if (m >= 2 && C->ritz_ok) {
          const double th0 = C->theta, r0 = C->res_est;
          const double pad = 1e-12 * fmax(1.0, fabs(th0));
          hlo = th0 - 2.0 * r0 - pad;
          hhi = th0 + pad;
        }
        double th = 0.0;
        const bool shared_test = Pol::kShareRitz && nblk > 1;
        if (!shared_test || blk == 0) th = smallest_eig_block(C->a, C->b, m, &s2, hlo, hhi);
        if (shared_test) {
          if (blk == 0 && threadIdx.x == 0) {
            G->theta = th;
            G->scale = s2;
          }
          if (!sums.meet()) return;
          if (blk != 0) {
            th = vload(&G->theta);
            s2 = vload(&G->scale);
          }
        }
        if (threadIdx.x == 0) {
          const double res = bj * sqrt(s2);
          const bool invariant = bj <= 1e-14 * bound;
          C->theta = th;
          C->res_est = invariant ? 0.0 : res;
          C->ritz_ok = 1;
          const bool conv = invariant || res <= P.tol;
          if (conv || C->iters >= P.maxiter) {
            C->status = conv ? SA_OK : SA_ERR_NOT_CONVERGED;
            C->b[j] = bj;
            C->action = ACT_DONE;
          } else if (m >= ncv) {
            C->restarts += 1;
            C->action = ACT_RESTART;
          } else {
            C->b[j] = bj;
            C->inv_b = 1.0 / bj;
            C->j = j + 1;
          }
        }
        __syncthreads();
        if (C->action == ACT_DONE) {
          tridiag_eigvec(C->a, C->b, m, th, C->s, sq);
          __syncthreads();
        }
      }
      const int act = C->action;
      if (act == ACT_RESTART) {
        // the first CTA runs the implicit restart; Q and the new tridiagonal reach the others in
        // global memory
        if (blk == 0) {
          const int keep = P.restart_keep > 0 ? P.restart_keep : kRestartDefault;
          const int kk = max(1, min(min(keep, kRestartMax), ncv / 2));
          implicit_restart(C, A.dense + kNcvMax * kNcvMax, j + 1, kk, sq, (int)(sizeof(work) / sizeof(double)));
          if (threadIdx.x < kk) {
            G->a[threadIdx.x] = C->a[threadIdx.x];
            G->b[threadIdx.x] = C->b[threadIdx.x];
          }
          if (threadIdx.x == 0) {
            G->irl_beta = C->irl_beta;
            G->irl_sigma = C->irl_sigma;
            G->irl_k = C->irl_k;
          }
        }
        if (!sums.meet()) return;
        if (blk != 0) {
          const int kk = vload(&G->irl_k);
          if (threadIdx.x < kk) {
            C->a[threadIdx.x] = vload(&G->a[threadIdx.x]);
            C->b[threadIdx.x] = vload(&G->b[threadIdx.x]);
          }
          if (threadIdx.x == 0) {
            C->irl_beta = vload(&G->irl_beta);
            C->irl_sigma = vload(&G->irl_sigma);
            C->irl_k = kk;
          }
          __syncthreads();
        }
      }
      mark(3);
      if (act == ACT_NEXT) continue;
      if (act == ACT_REPASS) continue;
      if (act == ACT_ERROR) {
        publish();
        return;
      }
      if (act == ACT_REJECT) { restart_p0 = true; break; }
      if (act == ACT_RESTART) {
        // kept basis V[0..kk) <- V Q[:, 0..kk) and the new residual
        // f = V Q[:, kk] T+[kk][kk-1] + w Q[m-1][kk-1], row by row in place (all m inputs of a row
        // are read before its kk outputs are written)
        const int m = j + 1;
        const int kk = C->irl_k;
        const double beta_hat = C->irl_beta, sig_q = C->irl_sigma;
        const double* Qd = A.dense + kNcvMax * kNcvMax;
#pragma unroll 1
        for (int idx = threadIdx.x; idx < m * (kk + 1); idx += blockDim.x) {
          const int r = idx / (kk + 1), c = idx % (kk + 1);
          sq[idx] = vload(Qd + r * m + c);
        }
        __syncthreads();
        const double v[1] = {kk == kRestartDefault
                                 ? restart_basis<T, kRestartDefault>(A.V, A.ldv, A.w, A.u, A.sigma, n, m, kk, sq, beta_hat, sig_q, pol.tid(), nthreads)
                                 : restart_basis<T, 0>(A.V, A.ldv, A.w, A.u, A.sigma, n, m, kk, sq, beta_hat, sig_q, pol.tid(), nthreads)};
        sums.block_put(v);
        if (!sums.all_sum(1)) return;
        const double nf = sqrt(tot[0]);
        const bool invariant = !(nf > 1e-14 * bound) || !isfinite(nf);
        double th = 0.0;
        if (invariant) th = smallest_eig_call(C->a, C->b, kk);
        if (threadIdx.x == 0) {
          C->pass2 = 0;
          C->bytes += (double)n * sizeof(T) * (double)(m + kk + 3);
          if (invariant) {
            // the kept basis spans an invariant subspace: finish with its Ritz vector
            C->theta = th;
            C->j = kk - 1;
            C->res_est = 0.0;
            C->status = SA_OK;
            C->action = ACT_DONE;
          } else {
            C->b[kk - 1] = nf;
            C->inv_b = 1.0 / nf;
            C->j = kk;
            C->action = ACT_NEXT;
          }
        }
        mark(4);
        __syncthreads();
        if (C->action == ACT_DONE) {
          tridiag_eigvec(C->a, C->b, kk, th, C->s, sq);
          __syncthreads();
        } else {
          continue;
        }
      }
      // ---------------- F1: Ritz vector y = V s, norm, alignment dot ------------------------------
      const int jf = C->j;
      const bool align = P.align && A.has_last;
      {
        double v[2] = {0.0, 0.0};
        int bad = 0;
#pragma unroll 1
        for (long long i = pol.tid(); i < n; i += nthreads) {
          const double y = basis_combine(A.V, A.ldv, i, jf, C->s);
          const T yt = (T)y;
          if (!isfinite((double)yt)) bad = 1;
          A.yout[i] = yt;
          A.u[i] = A.sigma[i] * yt;
          v[0] += (double)yt * (double)yt;
          if (align) v[1] += (double)yt * (double)A.ylast[i];
        }
        if (bad) atomicOr(&G->nonfinite, 1);
        sums.block_put(v);
      }
      if (!sums.all_sum(2)) return;
      if (threadIdx.x == 0) {
        const double nrm = sqrt(tot[0]);
        C->nrm_y = nrm;
        C->align_dot = align ? tot[1] : 0.0;
        C->bytes += (double)n * sizeof(T) * (double)(jf + 3 + (align ? 1 : 0));
        const double sg = (align && tot[1] < 0.0) ? -1.0 : 1.0;
        C->scale = (nrm > 0.0) ? sg / nrm : sg;
      }
      mark(5);
      __syncthreads();
    }
    if (restart_p0) continue;
    break;
  }

  // ---------------- F2: rounding (the residual's sum was stored by the final operator pass) --------
  const double scale = C->scale;
  {
    if (P.round) {
      const long long nr = (n + 31) & ~31ll;
      const T ts = (T)scale;
      unsigned long long hs = 0ull;
#pragma unroll 1
      for (long long i = pol.tid(); i < nr; i += nthreads) {
        bool bit = false;
        if (i < n) {
          const T x = (T)(A.yout[i] * ts) * (T)((double)A.sigma[i] * A.sqrt_c);
          bit = x >= T(0);
        }
        const unsigned int word = __ballot_sync(0xffffffffu, bit);
        if ((threadIdx.x & 31) == 0) {
          A.bits[i >> 5] = word;
          hs += word_mix(i >> 5, word);
        }
      }
      if ((threadIdx.x & 31) == 0 && hs) atomicAdd(&G->sig, hs);
    }
  }
  if (!sums.all_sum(P.residual_check ? 1 : 0)) return;
  if (threadIdx.x == 0) {
    C->rr = P.residual_check ? tot[0] : 0.0;
    if (P.residual_check) { C->bytes += A.spmv_bytes; C->spmvs += 1; }
    if (P.round) C->bytes += (double)n * sizeof(T) + (double)n / 8.0;
    C->bytes += 2.0 * (double)n * sizeof(T);   // F3
  }
  mark(5);
  // F3: y <- scale * y (aligned, unit norm)
  {
    const T ts = (T)scale;
#pragma unroll 1
    for (long long i = pol.tid(); i < n; i += nthreads) A.yout[i] = A.yout[i] * ts;
  }
  mark(5);
  publish();
}

}  // namespace sa
