// Gauss-Jordan elimination steps on matrix rows held in registers, shared by
// the block inverses (zinv.cu) and the grouped solve (rgf_grouped.cu).
//
// TPR threads hold one row, CPT columns each (column c of the step order in
// thread c % TPR), rows stay where they are (implicit partial pivoting by the
// LAPACK izamax rule: the first row of maximal |Re| + |Im|).  Step k: every
// warp names its best unused row, the row p of the best of them is published,
// and every row takes x_r <- x_r - (x_rk / p_k) p, the pivot row itself
// 0 + p / p_k.  The published row carries 1 in column k and each row clears
// its own entry there, so one formula covers all columns (-x_rk / p_k in column
// k, 1 / p_k in the pivot row).
//
// A chain of dependent steps: what a step costs is its latency.  Measured on
// B200 in cycles: 323 for the five-level butterfly over (value, index) pairs
// that a pivot search by shuffles takes, 28 for redux.sync and about 15 for a
// ballot; 237 for the reciprocal; 23 for a dependent DFMA; 25-40 for a barrier;
// 2 per DFMA of a warp on its scheduler; 4 per 16-byte shared store
// instruction on the SM, however few lanes store.  Hence
//   * the search compares |Re| + |Im| by its bit pattern (a non-negative double
//     orders as an integer): one redux.sync over the high words and a ballot,
//     a second pair only when the high words tie;
//   * two barriers per step: with one, every warp has to store its candidate
//     row before it (1056 of 2700 cycles per step at 256 rows of 32 columns);
//   * the register row is rotated by one column every TPR steps as it is
//     updated (x[j] <- f(x[j + 1])), so the step's column is always register 0
//     and no step selects over the row.
#pragma once

#include "common.cuh"

// Shared state of one elimination: the best row of every warp, and the pivot
// row of the step (TPR segments of CPT columns, padded so that the threads of a
// row read different banks).
template <int TPR, int CPT, int NWARPS>
struct GjRegs {
  static constexpr int SEG = TPR > 1 ? CPT + 1 : CPT;
  cplx prow[TPR * SEG];
  cplx piv[NWARPS];
  unsigned long long key[NWARPS];
  int row[NWARPS];
};

// Lanes whose key is the largest of the warp (all 32 lanes take part).
__device__ __forceinline__ unsigned gj_argmax(unsigned long long key) {
  const unsigned hi = (unsigned)(key >> 32);
  const unsigned m = __reduce_max_sync(0xffffffffu, hi);
  unsigned b = __ballot_sync(0xffffffffu, hi == m);
  if (b & (b - 1)) {
    const unsigned lo = hi == m ? (unsigned)key : 0u;
    const unsigned ml = __reduce_max_sync(0xffffffffu, lo);
    b = __ballot_sync(0xffffffffu, hi == m && lo == ml);
  }
  return b;
}

// `steps` steps (at most TPR * CPT) starting from column 0 of the register
// rows.  used: the row is no candidate (already a pivot, or past the matrix:
// such a row must be zero).  pivs[k] (shared) receives the pivot row of step k;
// returns 0, or 1 + the first step whose pivot is exactly zero.  Afterwards
// x[j] holds column ((j + steps / TPR) % CPT) * TPR + c_own, and the caller
// needs a barrier before it reads pivs.
template <int TPR, int CPT, int NWARPS>
__device__ __forceinline__ int gj_eliminate(cplx (&x)[CPT], int steps, int r_own, int c_own, bool used,
                                            GjRegs<TPR, CPT, NWARPS>& sm, int* pivs) {
  constexpr int SEG = GjRegs<TPR, CPT, NWARPS>::SEG;
  const int lane = threadIdx.x & 31, warp = NWARPS > 1 ? threadIdx.x >> 5 : 0;
  int zero_at = 0;
#pragma unroll 1
  for (int k = 0; k < steps; ++k) {
    const int own = k & (TPR - 1);  // the thread of each row that holds the step's column, in x[0]
    cplx f = x[0];  // the row's entry in the step's column
    if (TPR > 1) {
      const int src = (lane & ~(TPR - 1)) | own;
      f.x = __shfl_sync(0xffffffffu, f.x, src);
      f.y = __shfl_sync(0xffffffffu, f.y, src);
    }
    if (c_own == own) x[0] = cmk(0, 0);
    // 0: not a candidate; else the bits of |Re| + |Im| with the sign bit set.  A
    // NaN may carry either sign, so that bit must not decide: every candidate's
    // key is in [2^63, 2^64), in the order of the values, and a row that was a
    // pivot already is never named again (a NaN entry has the largest key and
    // becomes the pivot).
    unsigned long long key =
        used ? 0ull : (unsigned long long)__double_as_longlong(cabs1(f)) | 0x8000000000000000ull;
    const int best = __ffs(gj_argmax(key)) - 1;  // first lane of the first best row
    int pw = 0;
    if (lane == best) {
      sm.piv[warp] = f;
      sm.key[warp] = key;
      sm.row[warp] = r_own;
    }
    if (NWARPS > 1) {
      __syncthreads();
      key = lane < NWARPS ? sm.key[lane] : 0ull;
      pw = __ffs(gj_argmax(key)) - 1;  // rows ascend with the warps
    } else {
      __syncwarp();
    }
    const int p = sm.row[pw];
    const cplx piv = sm.piv[pw];
    if (r_own == p) {  // the pivot row; the other warps take the reciprocal meanwhile
      cplx* mine = sm.prow + c_own * SEG;
#pragma unroll
      for (int j = 0; j < CPT; ++j) mine[j] = x[j];
      if (c_own == own) mine[0] = cmk(1, 0);
    }
    if (piv.x == 0.0 && piv.y == 0.0 && !zero_at) zero_at = k + 1;
    if (threadIdx.x == 0) pivs[k] = p;
    const cplx d = crecip_pivot(piv);
    if (NWARPS > 1) __syncthreads();
    else __syncwarp();
    const cplx* prow = sm.prow + c_own * SEG;
    const bool is_p = r_own == p;
    const cplx fd = is_p ? cmk(-d.x, -d.y) : cmul(f, d);
    if (is_p) {
      used = true;
#pragma unroll
      for (int j = 0; j < CPT; ++j) x[j] = cmk(0, 0);
    }
    if (own == TPR - 1) {
      const cplx first = cfms(fd, prow[0], x[0]);
#pragma unroll
      for (int j = 0; j + 1 < CPT; ++j) x[j] = cfms(fd, prow[j + 1], x[j + 1]);
      x[CPT - 1] = first;
    } else {
#pragma unroll
      for (int j = 0; j < CPT; ++j) x[j] = cfms(fd, prow[j], x[j]);
    }
  }
  return zero_at;
}
