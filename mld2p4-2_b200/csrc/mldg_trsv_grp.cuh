// mldg_trsv_grp.cuh -- grouped unit-triangular solve.
//
// A sparse triangular solve is bound by its chain of dependency levels: each
// level costs one hand-off through L2 (about 1 us) however few rows it has.
// Here consecutive levels are joined into groups whose diagonal blocks L_gg
// are inverted explicitly when the plan is built (mldg_trigrp.h), so that
//   x_g = (W b)_g - (V x)_g,  W = diag_g(L_gg^{-1}),  V = diag_g(L_gg^{-1}) L_g<
// with one hand-off per group.  The price is fill: V and W hold more entries
// than L, streamed once each.  Measured against the level-by-level solve it
// replaced (us a solve, FP64): 4,096 rows, 46 levels in about 5 groups, 39 -> 18;
// 1,030,301 rows, 301 levels in 87 groups (11 entries a row instead of 3),
// 356 -> 155; a Gauss-Seidel factor of 15,850 wide rows, 207 -> 100.  A group
// costs 1.5-3 us, round trips of polls and gathers, where its bytes would
// stream in under 0.5: a grid barrier a group instead (one cooperative kernel a
// pair) took 2.4 us at the least, W b as a pass of its own 20-35 us a solve.
//
// The rows are cut into warp tasks of 32/(KC*tpr) rows of one group, KC columns
// and tpr lanes per (row, column), tpr a power of two so that a lane holds at
// most eight entries of the row (one pass of loads); wider blocks of columns
// are further tasks, KC being the columns of one 32-byte sector.  Entry m of a
// row belongs to lane m % tpr, and each lane's entries are stored four to a
// 16-byte index load, the warp's loads contiguous: first W's, which need no
// wait, then V's by ascending position, so that the newest dependencies come
// last.
//
// Warps claim tasks in group order from a ticket counter (two ahead: the next
// task's descriptor is loaded, the one after it claimed), so the
// lowest unfinished task always runs and every wait ends, whichever blocks are
// resident; rows of a task belong to one group and never wait on one another.
// A value of x is its own flag: it holds the sentinel until it is written.
// Each solve puts the sentinel (and a zero ticket counter) back into buffers
// that an earlier solve is finished with, so no separate pass does.
#pragma once

#include <climits>

#include "mldg_multi.cuh"

namespace mldg {

template <typename T>
struct GrpMat {
  int ntask;         // row tasks
  const int4 *desc;  // first slot group, slot groups per lane (W | V << 16), first position, rows << 8 | log2(tpr)
  const int4 *idx;   // four entries of a lane: column indices, -1 = none
  const T *val;      // and their values
};

template <typename T>
struct GrpArgs {
  GrpMat<T> m;
  int K, ncb;     // columns, column blocks of KC
  const T *rhs;   // b, indexed as W's columns were stored
  T *x;           // the solution in position order, sentinel on entry
  T *reset;       // put back to the sentinel
  const int *orig;
  T *out;         // out[orig] = alpha*x + beta*out[orig], or null
  T alpha, beta;
  int *ctr, *ctr_reset;
  int *err;
  int share, least;  // blocks that the solves running at once share (0: keep the whole grid), and a solve's fewest
};

// Grouped solves running on the device (those with a share).  A solve alone
// has the device to itself, two (FP64) or three (FP32) blocks an SM, most of them
// waiting; where handles are used by threads of their own, one solve's waiting
// blocks would keep the others' off the SMs, so that the warps of blocks beyond
// an equal share leave after one task, and the next kernel is not let in early.
// (Handles of idim 24..96, a thread each, ms until each has made an application:
// 24 of them in FP32 18.2 with whole grids; 6.8, 7.9, 9.9 with 1.5, 2, 2.25 blocks
// an SM shared; 7.2 with level-by-level solves; 16 of them 11.7; 5.3, 5.9, 6.9;
// 6.4; 8 of them 7.4; 4.1, 4.1, 4.4; 6.1; 2 of them 1.6, 1.4 with 2, 2.3.  FP64: 24
// of them 24.8; 8.0, 9.1, 12.7 with 1, 1.33, 1.5 blocks; 7.8; 16 of them 15.8;
// 5.9, 6.9, 9.2; 6.7; 8 of them 9.0; 4.5, 4.6, 5.3; 6.4.  Leaving before any task
// cost a solve alone 1 %: the count's round trip.)  One column only: the wider
// blocks' kernels with the same lines compiled slower (a solve of 32 right-hand
// sides at idim=64 45.9 -> 48.0 ms), so that they keep their whole grids.
static __device__ int g_grp_running;
template <int KC>
constexpr bool kGrpShares = KC == 1;

__device__ __forceinline__ void grp_vals(const double *p, double *v) {
  const double2 a = __ldg(reinterpret_cast<const double2 *>(p)), b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void grp_vals(const float *p, float *v) {
  const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
// entries of two consecutive slot groups q, q + R (the second only if two)
template <typename T, int R>
__device__ __forceinline__ void grp_pass(const GrpMat<T> &m, size_t q, bool two, int (&j)[8], T (&v)[8]) {
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const bool has = u == 0 || two;
    const int4 jj = has ? __ldg(m.idx + q + u * R) : make_int4(-1, -1, -1, -1);
    j[4 * u] = jj.x;
    j[4 * u + 1] = jj.y;
    j[4 * u + 2] = jj.z;
    j[4 * u + 3] = jj.w;
    if (has) {
      grp_vals(m.val + 4 * (q + u * R), v + 4 * u);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) v[4 * u + e] = T(0);
    }
  }
}

// Lane 0 polls p until it is written (a bounded wait); the warp goes on together.
template <typename T>
__device__ __forceinline__ void grp_gate(const T *p, int lane, int lim, int *err) {
  typedef typename Bits<T>::U U;
  for (int it = 0;; ++it) {
    int go = 1;
    if (lane == 0) {
      go = Bits<T>::load(p) != (U)Sentinel<T>::bits;
      if (!go && it >= lim) {
        atomicExch(err, kErrTimeout);
        go = 1;
      }
      if (!go && (it % kSpinCheck) == kSpinCheck - 1) go = ld_relaxed_u32(err) != 0u;
    }
    if (__shfl_sync(0xffffffffu, go, 0)) return;
  }
}

template <typename T, int KC>
__global__ void __launch_bounds__(256) k_trsv_grp(GrpArgs<T> a) {
  if (kGrpShares<KC> && a.share)
    pdl_wait();  // the solve before it on the same handle no longer counts
  else
    pdl_enter();
  constexpr int R = 32 / KC;
  typedef typename Bits<T>::U U;
  const U sent = (U)Sentinel<T>::bits;
  const int lane = threadIdx.x & 31, c = lane % KC, rs = lane / KC;
  const int K = a.K, ncb = a.ncb, ntask = a.m.ntask * ncb;
  const int lim = spin_limit();
  if (blockIdx.x == 0 && threadIdx.x == 0) *a.ctr_reset = 0;
  int pend = 0;
  if (lane == 0) pend = atomicAdd(a.ctr, 1);
  bool leaves = false;
  int running = 0;
  if (kGrpShares<KC> && a.share && lane == 0)
    running = blockIdx.x == 0 && threadIdx.x == 0 ? atomicAdd(&g_grp_running, 1) + 1
                                                  : (int)ld_relaxed_u32(&g_grp_running);
  int k = __shfl_sync(0xffffffffu, pend, 0);
  int4 d = k < ntask ? __ldg(a.m.desc + k / ncb) : make_int4(0, 0, 0, 0);
  if (kGrpShares<KC> && a.share) {
    running = __shfl_sync(0xffffffffu, running, 0);
    if (running <= 1)
      pdl_launch();
    else  // (block 0 never leaves: all tasks are claimed)
      leaves = (int)blockIdx.x >= max(a.least, a.share / running);
  }
  if (lane == 0) pend = leaves ? INT_MAX : atomicAdd(a.ctr, 1);
  while (k < ntask) {
    const int kn = __shfl_sync(0xffffffffu, pend, 0);
    if (lane == 0) pend = leaves ? INT_MAX : atomicAdd(a.ctr, 1);
    const int4 dn = kn < ntask ? __ldg(a.m.desc + kn / ncb) : make_int4(0, 0, 0, 0);
    const int col = (k % ncb) * KC + c;
    const int lt = d.w & 255, row = rs >> lt, nsw = d.y & 0xffff, nsv = d.y >> 16;
    const size_t q0 = (size_t)d.x + rs, qv = q0 + (size_t)nsw * R;
    int j[8];
    T v[8];
    if (nsv) grp_pass<T, R>(a.m, qv, nsv > 1, j, v);  // V's first pass, in flight while W's is summed
    T acc = T(0);
    for (int s = 0; s < nsw; s += 2) {
      int jw[8];
      T vw[8], b[8];
      grp_pass<T, R>(a.m, q0 + (size_t)s * R, s + 1 < nsw, jw, vw);
#pragma unroll
      for (int e = 0; e < 8; ++e) b[e] = jw[e] >= 0 ? __ldg(a.rhs + (size_t)jw[e] * K + col) : T(0);
#pragma unroll
      for (int e = 0; e < 8; ++e) acc = fma(vw[e], b[e], acc);
    }
    for (int s = 0; s < nsv; s += 2) {
      if (s) grp_pass<T, R>(a.m, qv + (size_t)s * R, s + 1 < nsv, j, v);
      // One lane polls the warp's newest dependency; then every lane reads its
      // values, and reads again those that are still missing.  (Polling all of
      // them from the start fills the SMs' load pipes with uncoalesced polls:
      // 1.04 ms instead of 0.72 for the four solves of 1,030,301 rows.)
      int jg = -1;
#pragma unroll
      for (int e = 0; e < 8; ++e) jg = max(jg, j[e]);
      jg = __reduce_max_sync(0xffffffffu, jg);
      if (jg >= 0) grp_gate(a.x + (size_t)jg * K + (col - c), lane, lim, a.err);
      U raw[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) raw[e] = j[e] >= 0 ? Bits<T>::load(a.x + (size_t)j[e] * K + col) : (U)0;
      for (int it = 0;; ++it) {
        bool missing = false;
#pragma unroll
        for (int e = 0; e < 8; ++e) missing |= (raw[e] == sent);
        if (!missing) break;
        if (it >= lim) {
          atomicExch(a.err, kErrTimeout);
          break;
        }
        if ((it % kSpinCheck) == kSpinCheck - 1) {
          if (ld_relaxed_u32(a.err) != 0u) break;
          __nanosleep(32);
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
          if (raw[e] == sent) raw[e] = Bits<T>::load(a.x + (size_t)j[e] * K + col);
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) acc = fma(-v[e], Bits<T>::from(raw[e] == sent ? (U)0 : raw[e]), acc);
    }
    for (int o = 0; o < lt; ++o) acc += __shfl_xor_sync(0xffffffffu, acc, KC << o);
    if ((rs & ((1 << lt) - 1)) == 0 && row < (d.w >> 8)) {
      const size_t p = (size_t)(d.z + row) * K + col;
      const T xv = Bits<T>::canon(acc);
      Bits<T>::store(a.x + p, xv);
      a.reset[p] = Sentinel<T>::value();
      if (a.out) {
        const size_t o = (size_t)a.orig[d.z + row] * K + col;
        T w = a.alpha * xv;
        if (a.beta != T(0)) w = fma(a.beta, a.out[o], w);
        a.out[o] = w;
      }
    }
    k = kn;
    d = dn;
  }
  if (kGrpShares<KC> && a.share && blockIdx.x == 0 && threadIdx.x == 0) atomicSub(&g_grp_running, 1);
}

}  // namespace mldg
