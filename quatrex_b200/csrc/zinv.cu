// Batched complex FP64 inverse: in-place Gauss-Jordan elimination with partial
// pivoting.  Replaces qttools.kernels.linalg.inv
// (src/qttools/kernels/linalg/inv.py:6-40, LAPACK getrf/getri, or getrf/getrs on
// the GPU).  Pivot choice follows the LAPACK izamax rule: the first row (in the
// current row order) of maximal |Re| + |Im|.
//
// Three forms, chosen in launch_zinv:
//   n <= 64            zinv_regs_kernel: the whole matrix in the registers of one
//                      CTA
//   n <= 512           zinv_panel_kernel + zinv_update_kernel per panel of
//                      columns, zinv_split_unscramble_kernel at the end
//   no scratch memory  zinv_gj_kernel: one launch, one CTA per matrix
//
// Algorithm of the blocked forms for an n x n matrix X (a copy of A), panel
// width w:
//   for each panel of columns [k0, k0 + w):
//     1. eliminate the n x w panel in registers column by column without moving
//        rows: pick the pivot row among the rows not yet used, eliminate the
//        column from all other rows, scale the pivot row;
//     2. turn the pivot sequence into the row permutation sigma that the
//        classic row-swapping Gauss-Jordan would apply (position k0 + j takes
//        pivot row p_j, the displaced row goes to p_j's position), and record
//        each swap for the final column unscrambling;
//     3. apply the panel's row operations to every other column at once, a
//        rank-w update on DMMA (mma.sync m16n8k4 f64) tiles:
//          X[i, c] <- [i not in panel] X[sigma(i), c]
//                     + sum_j P[sigma(i), j] X[p_j, c]
//        in column slabs, the pivot rows staged in shared memory;
//   finally undo the row interchanges as column interchanges in reverse order.
// The matrix itself stays in global memory; shared memory holds the panel
// (n x Wp, XOR-swizzled so that both row-per-thread access and DMMA fragment
// loads are conflict-free), slabs of pivot rows and the permutation arrays.
#include <algorithm>
#include <cstdlib>

#include "gj_regs.cuh"
#include "kernels.h"

namespace {

constexpr int THREADS = 256;
constexpr int NWARPS = THREADS / 32;

// Shape of the one-launch form (n > 64).
struct InvShape {
  int w;   // panel width, a multiple of 8
  int cw;  // columns per update slab (multiple of 32)
};

__host__ __device__ inline InvShape inv_shape(int n) {
  InvShape s;
  s.w = n > 96 && n <= 256 ? 32 : 16;
  const int row_tiles = (n + 31) / 32;
  s.cw = 32 * (row_tiles >= NWARPS ? 1 : NWARPS / row_tiles);
  return s;
}

// complex elements of the update slabs: pivot rows and panel rows, double buffered
__host__ __device__ inline int slab_elems(const InvShape& s) { return 4 * s.w * (s.cw + 2); }

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  int bytes = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

inline size_t inv_smem_bytes(int n) {
  const InvShape s = inv_shape(n);
  const size_t panel = (size_t)n * s.w * sizeof(cplx);
  const size_t slabs = (size_t)slab_elems(s) * sizeof(cplx);
  const size_t ints = (size_t)(3 * n + 32 + 4) * sizeof(int);
  // pivot candidates of two column parities (several rows a thread)
  const size_t cand = 2 * NWARPS * (sizeof(double) + sizeof(int) + (1 + s.w) * sizeof(cplx));
  return panel + slabs + ints + (n > THREADS ? cand : 0) + 256;
}

// swizzled panel index: row r, column c (c < wp, wp multiple of 8)
__device__ __forceinline__ int pidx(int r, int c, int wp) {
  int sw = ((r & 1) << 2) | ((r >> 1) & 3);
  return r * wp + (c ^ sw);
}

// Two adjacent complex elements in one 32-byte access.  The caller guarantees
// 32-byte alignment: pair_access_ok() for the matrix and an even column.
__device__ __forceinline__ void ld_pair(const cplx* p, cplx& a, cplx& b) {
  asm volatile("ld.global.v4.f64 {%0,%1,%2,%3}, [%4];\n"
               : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y)
               : "l"(p));
}
__device__ __forceinline__ void st_pair(cplx* p, cplx a, cplx b) {
  asm volatile("st.global.v4.f64 [%0], {%1,%2,%3,%4};\n" ::"l"(p), "d"(a.x), "d"(a.y), "d"(b.x), "d"(b.y)
               : "memory");
}
// Element (i, c) of X with c even starts on a 32-byte boundary, and the pair
// (c, c + 1) lies on one side of every even column boundary (n, panel edges
// k0 and k0 + w, which are even when n is).
__device__ __forceinline__ bool pair_access_ok(const cplx* X, int64_t ldx, int n) {
  return (reinterpret_cast<uintptr_t>(X) & 31) == 0 && (ldx & 1) == 0 && (n & 1) == 0;
}

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ void argmax_combine(double& v, int& i, double v2, int i2) {
  if (v2 > v || (v2 == v && i2 < i)) {
    v = v2;
    i = i2;
  }
}

// Shared-memory arrays of one matrix's elimination (see zinv_gj_kernel); those
// from red_v on with several rows a thread only.
struct GjSmem {
  cplx* P;
  int* pos2row;
  int* row2pos;
  int* perm;
  int* pivs;
  double* red_v;
  cplx* red_piv;
  int* red_i;
  cplx* cand;
};

__device__ inline GjSmem gj_smem_layout(unsigned char* base, int n, int w, int slab) {
  GjSmem s;
  s.P = reinterpret_cast<cplx*>(base);
  cplx* Rs = s.P + (size_t)n * w;
  s.pos2row = reinterpret_cast<int*>(Rs + slab);
  s.row2pos = s.pos2row + n;
  s.perm = s.row2pos + n;  // swap partner of each column (final unscramble)
  // doubles after the int arrays: round the offset up to 16 bytes (3n ints is
  // not a multiple of 8 bytes for odd n)
  s.pivs = s.perm + n;  // pivot row of each column of the current panel
  s.red_v = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(s.pivs + 32) + 15) & ~uintptr_t(15));
  s.red_piv = reinterpret_cast<cplx*>(s.red_v + 2 * NWARPS);  // column-kk entry of each warp's candidate
  s.red_i = reinterpret_cast<int*>(s.red_piv + 2 * NWARPS);
  // per warp and column parity: the panel row of the warp's pivot candidate
  s.cand = reinterpret_cast<cplx*>(s.red_i + 2 * NWARPS + 2);
  s.cand = reinterpret_cast<cplx*>((reinterpret_cast<uintptr_t>(s.cand) + 15) & ~uintptr_t(15));
  return s;
}

// Eliminates a panel of at most CPT columns and of up to RPT * THREADS rows
// that the threads of the CTA hold RPT rows each (row r0 + q * THREADS in
// reg[q]): the steps of gj_eliminate for more rows than threads.  Column kk of the
// register rows is picked by selects.  24 matrices of n = 512 take 11.1 ms; 12.0
// with all columns unrolled and static, 12.8 with one update formula for the
// pivot row and the others on top, as in gj_eliminate (registers).
template <int RPT, int CPT>
__device__ __forceinline__ void gj_eliminate_rows(cplx (&reg)[RPT][CPT], int n, int k0, int w, const GjSmem& sm,
                                                  int& zero_pivot) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bool used[RPT];
#pragma unroll
  for (int q = 0; q < RPT; ++q) used[q] = tid + q * THREADS < k0;  // the pivots of earlier panels
  // One barrier per column: every warp publishes the panel row of its own
  // best candidate before the barrier, so afterwards the winner's row is read
  // directly.
#pragma unroll 32
  for (int kk = 0; kk < w; ++kk) {
    // each row reads and clears its column-kk entry: the staged pivot row
    // carries 1 there, so the update below is one x - fd p for every entry
    // (-fd at column kk) and p d for the pivot row (d at kk)
    cplx colv[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      cplx v = cmk(0, 0);
#pragma unroll
      for (int j = 0; j < CPT; ++j)
        if (j == kk) {
          v = reg[q][j];
          reg[q][j] = cmk(0, 0);
        }
      colv[q] = v;
    }
    // A NaN entry counts as infinite: every candidate is then above the -1 of
    // the rows that are none, and the same row is found by all lanes.
    double bv = -1.0;
    int bi = n;
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int r = tid + q * THREADS;
      if (r < n && !used[q]) argmax_combine(bv, bi, fmin(cabs1(colv[q]), (double)INFINITY), r);
    }
    // butterfly: every lane ends with the warp's best candidate
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const double v2 = __shfl_xor_sync(0xffffffffu, bv, off);
      const int i2 = __shfl_xor_sync(0xffffffffu, bi, off);
      argmax_combine(bv, bi, v2, i2);
    }
    const int slot = (kk & 1) * NWARPS;
    cplx* my_cand = sm.cand + (slot + warp) * CPT;
#pragma unroll
    for (int q = 0; q < RPT; ++q)
      if (tid + q * THREADS == bi) {
#pragma unroll
        for (int j = 0; j < CPT; ++j)
          if (j < w) my_cand[j] = reg[q][j];
        my_cand[kk] = cmk(1, 0);
        sm.red_piv[slot + warp] = colv[q];
      }
    if (lane == 0) {
      sm.red_v[slot + warp] = bv;
      sm.red_i[slot + warp] = bi;
    }
    __syncthreads();  // candidates of every warp visible
    // best over the warps: every group of NWARPS lanes holds all candidates
    double v = sm.red_v[slot + lane % NWARPS];
    int p = sm.red_i[slot + lane % NWARPS];
#pragma unroll
    for (int off = NWARPS / 2; off > 0; off >>= 1) {
      const double v2 = __shfl_xor_sync(0xffffffffu, v, off);
      const int i2 = __shfl_xor_sync(0xffffffffu, p, off);
      argmax_combine(v, p, v2, i2);
    }
    const int pw = (p % THREADS) >> 5;  // the warp that holds row p published it
    const cplx* prow = sm.cand + (slot + pw) * CPT;
    const cplx piv = sm.red_piv[slot + pw];
    if (piv.x == 0.0 && piv.y == 0.0 && !zero_pivot) zero_pivot = k0 + kk + 1;
    const cplx d = crecip_pivot(piv);
    if (tid == 0) sm.pivs[kk] = p;
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int r = tid + q * THREADS;
      if (r >= n) continue;
      if (r == p) {
        used[q] = true;
#pragma unroll
        for (int j = 0; j < CPT; ++j)
          if (j < w) reg[q][j] = cmul(prow[j], d);
      } else {
        const cplx fd = cmul(colv[q], d);
#pragma unroll
        for (int j = 0; j < CPT; ++j)
          if (j < w) reg[q][j] = cfms(fd, prow[j], reg[q][j]);
      }
    }
  }
}

// Steps 1 and 2 for the panel [k0, k0 + w) of X (rows in the current order):
// eliminate it in registers, turn its pivots into the row permutation sigma
// (pos2row / row2pos, relative to the current order) and the swaps
// perm[k0 .. k0 + w), and leave the eliminated panel in P (rows in the current
// order).  TPR threads a row of CPT columns each, or (TPR = 1) RPT rows a
// thread.  Ends with a CTA barrier.
template <int TPR, int RPT, int CPT>
__device__ __forceinline__ void gj_panel(int n, int k0, int w, const cplx* X, int64_t ldx, const GjSmem& sm,
                                         int& zero_pivot) {
  constexpr int W = TPR * CPT;
  static_assert(TPR == 1 || RPT == 1, "several rows a thread: whole rows");
  cplx* P = sm.P;
  int* pos2row = sm.pos2row;
  int* row2pos = sm.row2pos;
  int* perm = sm.perm;
  int* pivs = sm.pivs;
  const int tid = threadIdx.x;
    // ---- 1. stage the panel (rows in the current order of X), every
    // element in flight at once (asynchronous copies)
    for (int idx = tid; idx < n * w; idx += THREADS) {
      int r = idx / w, c = idx % w;
      cp_async16(&P[pidx(r, c, W)], &X[(int64_t)r * ldx + k0 + c], true);
    }
    cp_async_commit();
    for (int r = tid; r < n; r += THREADS) {
      pos2row[r] = r;
      row2pos[r] = r;
    }
    cp_async_wait<0>();
    __syncthreads();

    // The thread's panel entries live in registers during the elimination:
    // reg[q][j] = P[r_own + q * rstride][c_own + j * TPR].
    const int rstride = THREADS / TPR, r_own = tid / TPR, c_own = tid % TPR;
    cplx reg[RPT][CPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q)
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const int r = r_own + q * rstride, c = c_own + j * TPR;
        reg[q][j] = (r < n && c < w) ? P[pidx(r, c, W)] : cmk(0, 0);
      }
    // rows before k0 are the pivots of earlier panels (rows are in the new order now)
    int turned = 0;
    if constexpr (RPT == 1) {
      __shared__ GjRegs<TPR, CPT, NWARPS> regs;
      const int zero = gj_eliminate<TPR, CPT, NWARPS>(reg[0], w, r_own, c_own, r_own < k0 || r_own >= n, regs, pivs);
      if (zero && !zero_pivot) zero_pivot = k0 + zero;
      turned = w / TPR;
    } else {
      gj_eliminate_rows<RPT, CPT>(reg, n, k0, w, sm, zero_pivot);
    }
    // classic row-swap semantics of the panel's pivots: position k0 + kk
    // receives row pivs[kk], the displaced row goes to the pivot's position
    if (tid == 0) {
      for (int kk = 0; kk < w; ++kk) {
        const int k = k0 + kk, p = pivs[kk];
        const int qpos = row2pos[p];
        const int rk = pos2row[k];
        pos2row[k] = p;
        row2pos[p] = k;
        pos2row[qpos] = rk;
        row2pos[rk] = qpos;
        perm[k] = qpos;
      }
    }
    // panel back to shared memory for the update
#pragma unroll
    for (int q = 0; q < RPT; ++q)
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const int r = r_own + q * rstride, c = ((j + turned) % CPT) * TPR + c_own;
        if (r < n && c < w) P[pidx(r, c, W)] = reg[q][j];
      }
    __syncthreads();
}

template <int TPR, int RPT, int CPT>
__global__ void __launch_bounds__(THREADS, 1)
    zinv_gj_kernel(int n, int64_t batch, const cplx* a_base, int64_t lda, int64_t sa,
                   cplx* x_base, int64_t ldx, int64_t sx, int* info, const int* active) {
  qtx_grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const InvShape shp = inv_shape(n);
  constexpr int W = TPR * CPT;  // = shp.w
  const int CW = shp.cw;
  const int LDR = CW + 2;
  const GjSmem sm = gj_smem_layout(smem_raw, n, W, slab_elems(shp));
  cplx* P = sm.P;
  cplx* Rs = P + (size_t)n * W;  // two slabs of W x LDR (pivot rows, panel rows)
  int* pos2row = sm.pos2row;
  int* perm = sm.perm;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;

  for (int64_t e = blockIdx.x; e < batch; e += gridDim.x) {
    if (active && !active[e]) continue;
    const cplx* A = a_base + e * sa;
    cplx* X = x_base + e * sx;
    int zero_pivot = 0;

    if (A != X || lda != ldx) {
      for (int idx = tid; idx < n * n; idx += THREADS) {
        int r = idx / n, c = idx % n;
        X[(int64_t)r * ldx + c] = A[(int64_t)r * lda + c];
      }
    }
    __syncthreads();

    for (int k0 = 0; k0 < n; k0 += W) {
      const int w = min(W, n - k0);
      gj_panel<TPR, RPT, CPT>(n, k0, w, X, ldx, sm, zero_pivot);

      // ---- 3. rank-w update of the other columns, slabs of CW columns.
      // Output position i reads X[sigma(i)], and sigma(i) is either i itself or
      // a row of [k0, k0 + w) (a row displaced by a pivot swap); the pivot rows
      // X[p_j] and the rows of [k0, k0 + w) of the slab are staged in shared
      // memory first, so afterwards every thread reads and writes only its own
      // positions of X and one barrier per slab suffices.
      const int row_tiles = (n + 31) / 32;
      const int col_tiles = CW / 32;
      const int nslab = (n + CW - 1) / CW;
      // slabs with at least one column outside the panel, staged double buffered
      auto next_slab = [&](int from) {
        int sl = from;
        while (sl < nslab && (sl * CW >= k0 && min(sl * CW + CW, n) <= k0 + w)) ++sl;
        return sl;
      };
      auto stage = [&](int sl, int buf) {
        cplx* Rb = Rs + (size_t)buf * 2 * W * LDR;
        cplx* Db = Rb + (size_t)W * LDR;
        const int cs = sl * CW;
        for (int idx = tid; idx < w * CW; idx += THREADS) {
          int j = idx / CW, cc = idx % CW;
          int c = cs + cc;
          bool ok = c < n;
          cp_async16(&Rb[j * LDR + cc], ok ? &X[(int64_t)pos2row[k0 + j] * ldx + c] : X, ok);
          cp_async16(&Db[j * LDR + cc], ok ? &X[(int64_t)(k0 + j) * ldx + c] : X, ok);
        }
        cp_async_commit();
      };
      const int ntiles = row_tiles * col_tiles;
      // Accumulator start values of a tile: output position i starts from
      // X[sigma(i)].  Rows with sigma(i) == i load straight from X under one
      // predicate each (no branch between global and shared memory), so the
      // 32 loads of a thread are in flight together; the few rows displaced
      // by a pivot swap are then patched from the staged rows D.
      auto load_own = [&](int tile, int c0, double (&are)[2][4][4], double (&aim)[2][4][4]) {
        const int row0 = (tile / col_tiles) * 32, col0 = (tile % col_tiles) * 32;
        bool own[2][2];
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int i = row0 + mi * 16 + g + 8 * h;
            own[mi][h] = i < n && !(i >= k0 && i < k0 + w) && pos2row[i] == i;
          }
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int i = row0 + mi * 16 + g + ((q >> 1) << 3);
              const int c = c0 + col0 + ni * 8 + 2 * t + (q & 1);
              are[mi][ni][q] = 0.0;
              aim[mi][ni][q] = 0.0;
              if (own[mi][q >> 1] && c < n) {
                const cplx y = X[(int64_t)i * ldx + c];
                are[mi][ni][q] = y.x;
                aim[mi][ni][q] = y.y;
              }
            }
      };
      auto patch_displaced = [&](int tile, int c0, const cplx* D, double (&are)[2][4][4],
                                 double (&aim)[2][4][4]) {
        const int row0 = (tile / col_tiles) * 32, col0 = (tile % col_tiles) * 32;
#pragma unroll
        for (int mi = 0; mi < 2; ++mi)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int i = row0 + mi * 16 + g + 8 * h;
            if (i < n && !(i >= k0 && i < k0 + w)) {
              const int src = pos2row[i];
              if (src != i) {
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                  for (int q2 = 0; q2 < 2; ++q2) {
                    const int cc = col0 + ni * 8 + 2 * t + q2;
                    if (c0 + cc < n) {
                      const cplx y = D[(src - k0) * LDR + cc];
                      are[mi][ni][2 * h + q2] = y.x;
                      aim[mi][ni][2 * h + q2] = y.y;
                    }
                  }
              }
            }
          }
      };
      int slab = next_slab(0);
      int buf = 0;
      if (slab < nslab) stage(slab, 0);
      while (slab < nslab) {
        const int c0 = slab * CW;
        const int nxt = next_slab(slab + 1);
        // the other buffer was last read before the barrier that ended the
        // previous slab, so it can be refilled now
        if (nxt < nslab) stage(nxt, buf ^ 1);
        else cp_async_commit();
        cp_async_wait<1>();
        __syncthreads();
        cplx* R = Rs + (size_t)buf * 2 * W * LDR;  // pivot rows p_j      (w x CW)
        cplx* D = R + (size_t)W * LDR;             // rows k0 + j         (w x CW)
        for (int tile = warp; tile < ntiles; tile += NWARPS) {
          const int rt = tile / col_tiles, ct = tile % col_tiles;
          const int row0 = rt * 32, col0 = ct * 32;
          double acc_re[2][4][4], acc_im[2][4][4];
          load_own(tile, c0, acc_re, acc_im);
          patch_displaced(tile, c0, D, acc_re, acc_im);
          int prow_idx[2][2];
#pragma unroll
          for (int mi = 0; mi < 2; ++mi) {
            int i0 = row0 + mi * 16 + g, i1 = i0 + 8;
            prow_idx[mi][0] = i0 < n ? pos2row[i0] : -1;
            prow_idx[mi][1] = i1 < n ? pos2row[i1] : -1;
          }
          for (int kk = 0; kk < w; kk += 4) {
            const int kc = kk + t;
            cplx af[2][2], bf[4];
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                int pr = prow_idx[mi][h];
                af[mi][h] = (pr >= 0 && kc < w) ? P[pidx(pr, kc, W)] : cmk(0, 0);
              }
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) bf[ni] = (kc < w) ? R[kc * LDR + col0 + ni * 8 + g] : cmk(0, 0);
            // real parts first, then imaginary: 16 independent accumulators
            // separate the two products that feed the same accumulator
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
              for (int ni = 0; ni < 4; ++ni) {
                dmma(acc_re[mi][ni], af[mi][0].x, af[mi][1].x, bf[ni].x);
                dmma(acc_im[mi][ni], af[mi][0].x, af[mi][1].x, bf[ni].y);
              }
#pragma unroll
            for (int mi = 0; mi < 2; ++mi)
#pragma unroll
              for (int ni = 0; ni < 4; ++ni) {
                dmma(acc_re[mi][ni], -af[mi][0].y, -af[mi][1].y, bf[ni].y);
                dmma(acc_im[mi][ni], af[mi][0].y, af[mi][1].y, bf[ni].x);
              }
          }
#pragma unroll
          for (int mi = 0; mi < 2; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                int i = row0 + mi * 16 + g + ((q >> 1) << 3);
                int c = c0 + col0 + ni * 8 + 2 * t + (q & 1);
                if (i < n && c < n && !(c >= k0 && c < k0 + w))
                  X[(int64_t)i * ldx + c] = cmk(acc_re[mi][ni][q], acc_im[mi][ni][q]);
              }
        }
        __syncthreads();
        slab = nxt;
        buf ^= 1;
      }
      cp_async_wait<0>();
      // ---- panel columns: final panel values in the new row order
      for (int idx = tid; idx < n * w; idx += THREADS) {
        int i = idx / w, c = idx % w;
        X[(int64_t)i * ldx + k0 + c] = P[pidx(pos2row[i], c, W)];
      }
      // rows are now in the new order: the pivot rows so far sit at positions < k0 + w
      __syncthreads();
    }

    // ---- undo the row interchanges as column interchanges, in reverse order
    int* colsrc = pos2row;  // reuse: column permutation
    for (int c = tid; c < n; c += THREADS) colsrc[c] = c;
    __syncthreads();
    if (tid == 0) {
      for (int k = n - 1; k >= 0; --k) {
        int q = perm[k];
        int tmp = colsrc[k];
        colsrc[k] = colsrc[q];
        colsrc[q] = tmp;
      }
    }
    __syncthreads();
    {
      constexpr int rows_per_slab = W;
      for (int r0 = 0; r0 < n; r0 += rows_per_slab) {
        int nr = min(rows_per_slab, n - r0);
        for (int idx = tid; idx < nr * n; idx += THREADS) {
          int r = idx / n, c = idx % n;
          P[idx] = X[(int64_t)(r0 + r) * ldx + c];
        }
        __syncthreads();
        for (int idx = tid; idx < nr * n; idx += THREADS) {
          int r = idx / n, c = idx % n;
          X[(int64_t)(r0 + r) * ldx + c] = P[r * n + colsrc[c]];
        }
        __syncthreads();
      }
    }
    // sticky: callers zero info once and read it after several launches
    if (info && tid == 0 && zero_pivot) info[e] = zero_pivot;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Blocks of up to 64: the whole matrix in registers (gj_regs.cuh), one CTA per
// matrix, four threads per row (four warps up to 32 rows, eight up to 64).  The
// row and column permutations are applied on the store: the row-swapping
// elimination would hold row p_k at position k, so with pos(r) the step at which
// row r was the pivot, X[pos(r)][p_c] = M[r][c].
// Bound by the chain of n dependent steps: about 1100 cycles each at 32 rows,
// 1700 at 64.  Measured on B200, us per call with its status read: b = 32, 8
// matrices 44 (66 with the blocked kernel), b = 64, 32 matrices 89 (147).
template <int TPR, int CPT, int NW>
__global__ void __launch_bounds__(32 * NW, 16 / NW)
    zinv_regs_kernel(int n, int64_t batch, const cplx* a_base, int64_t lda, int64_t sa, cplx* x_base, int64_t ldx,
                     int64_t sx, int* info, const int* active) {
  qtx_grid_dependency();
  __shared__ GjRegs<TPR, CPT, NW> sm;
  __shared__ int pivs[TPR * CPT], pos[TPR * CPT];
  const int r = threadIdx.x / TPR, cl = threadIdx.x % TPR;
  for (int64_t e = blockIdx.x; e < batch; e += gridDim.x) {
    if (active && !active[e]) continue;
    const cplx* A = a_base + e * sa;
    cplx* X = x_base + e * sx;
    cplx x[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const int c = cl + j * TPR;
      x[j] = r < n && c < n ? A[(int64_t)r * lda + c] : cmk(0, 0);
    }
    const int zero = gj_eliminate<TPR, CPT, NW>(x, n, r, cl, r >= n, sm, pivs);
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += 32 * NW) pos[pivs[k]] = k;
    __syncthreads();
    if (r < n) {
      cplx* row = X + (int64_t)pos[r] * ldx;
      const int turned = n / TPR;
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const int c = ((j + turned) % CPT) * TPR + cl;
        if (c < n) row[pivs[c]] = x[j];
      }
    }
    // sticky: callers zero info once and read it after several launches
    if (info && threadIdx.x == 0 && zero) info[e] = zero;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Larger blocks: every panel of 32 columns (16 above 256 rows) is two
// launches.  zinv_panel_kernel, one CTA per matrix and a row per thread,
// eliminates the panel in registers (gj_regs.cuh) and leaves in global scratch
// the eliminated panel P (n x W, rows in the order before the panel's
// permutation), sigma (pos2row) and the column swaps; zinv_update_kernel
// applies its rank-w update to the other columns, a CTA per (matrix, 32-column
// slab) with all n rows, so a CTA stages the pivot rows R = X[sigma(k0 + j)]
// and the panel-position rows D = X[k0 + j] of its slab itself before it
// writes any of them.  The column chain of the elimination runs on as many SMs
// as there are matrices, the updates on all.
//
// Bounds: the panel by its chain of dependent steps (about 2000 cycles each at
// 256 rows), the update by the latency of its loads and DMMAs (DMMA pipe 61 %
// active and 2.2 TB/s of DRAM traffic at b = 256, 148 matrices; 56 % and 3.3
// TB/s at b = 512, 40 matrices).  Measured on B200, ms per call, against three
// launches per panel (the pivot rows copied by one of their own) below 80-124
// matrices and the one-launch kernel of that time above:
//     b = 100,  24 matrices 0.18 (0.28)     b = 128, 100 matrices 0.27 (0.41)
//     b = 256,  16 matrices 0.54 (0.82)     b = 256,  64 matrices 0.84 (1.26)
//     b = 256, 148 matrices 1.31 (1.65)     b = 300,  20 matrices 0.84 (1.43)
//     b = 512,  24 matrices 2.62 (4.26)     b = 512, 148 matrices 9.4 (13.0)

struct SplitScratch {
  cplx* p;     // batch x n x W
  int* sigma;  // batch x n
  int* perm;   // batch x n
};

inline int panel_width(int n) { return n <= 256 ? 32 : 16; }

inline size_t panel_smem(int n, int W) {
  return (size_t)n * W * sizeof(cplx) + (size_t)(2 * n + 2 * W) * sizeof(int);
}

// The panel [k0, k0 + w) of every matrix; W = TPR * CPT columns, TPR threads a
// row, 32 NW / TPR >= n rows.
template <int TPR, int CPT, int NW>
__global__ void __launch_bounds__(32 * NW)
    zinv_panel_kernel(int n, int64_t batch, const cplx* a_base, int64_t lda, int64_t sa, cplx* x_base, int64_t ldx,
                      int64_t sx, int k0, SplitScratch sc, int* info, const int* active) {
  qtx_grid_dependency();
  constexpr int W = TPR * CPT, NT = 32 * NW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ GjRegs<TPR, CPT, NW> sm;
  cplx* P = reinterpret_cast<cplx*>(smem_raw);  // n x W, swizzled
  int* pos2row = reinterpret_cast<int*>(P + (size_t)n * W);
  int* row2pos = pos2row + n;
  int* pivs = row2pos + n;
  int* swaps = pivs + W;
  const int tid = threadIdx.x, row = tid / TPR, cl = tid % TPR;
  const int w = min(W, n - k0);
  for (int64_t e = blockIdx.x; e < batch; e += gridDim.x) {
    if (active && !active[e]) continue;
    cplx* X = x_base + e * sx;
    const cplx* src = X + k0;
    int64_t lds = ldx;
    if (k0 == 0) {
      src = a_base + e * sa;
      lds = lda;
    }
    // the panel through shared memory: coalesced copies, then a row per thread
    for (int idx = tid; idx < n * w; idx += NT) {
      const int r = idx / w, c = idx % w;
      cp_async16(&P[pidx(r, c, W)], &src[(int64_t)r * lds + c], true);
    }
    cp_async_commit();
    for (int r = tid; r < n; r += NT) {
      pos2row[r] = r;
      row2pos[r] = r;
    }
    cp_async_wait<0>();
    __syncthreads();
    cplx x[CPT];
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const int c = cl + j * TPR;
      x[j] = row < n && c < w ? P[pidx(row, c, W)] : cmk(0, 0);
    }
    // rows before k0 are the pivots of earlier panels (rows are in the new order now)
    const int zero = gj_eliminate<TPR, CPT, NW>(x, w, row, cl, row < k0 || row >= n, sm, pivs);
    if (row < n) {
      const int turned = w / TPR;
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const int c = ((j + turned) % CPT) * TPR + cl;
        if (c < w) P[pidx(row, c, W)] = x[j];
      }
    }
    __syncthreads();
    // row-swap semantics of the panel's pivots: position k0 + kk receives row
    // pivs[kk], the displaced row goes to the pivot's position
    if (tid == 0) {
      for (int kk = 0; kk < w; ++kk) {
        const int k = k0 + kk, p = pivs[kk];
        const int qpos = row2pos[p], rk = pos2row[k];
        pos2row[k] = p;
        row2pos[p] = k;
        pos2row[qpos] = rk;
        row2pos[rk] = qpos;
        swaps[kk] = qpos;
      }
    }
    cplx* pe = sc.p + e * (int64_t)n * W;
    for (int idx = tid; idx < n * w; idx += NT) {
      const int r = idx / w, c = idx % w;
      pe[(int64_t)r * W + c] = P[pidx(r, c, W)];
    }
    __syncthreads();
    for (int r = tid; r < n; r += NT) sc.sigma[e * n + r] = pos2row[r];
    for (int kk = tid; kk < w; kk += NT) sc.perm[e * n + k0 + kk] = swaps[kk];
    // the panel columns of X: final values in the new row order.  (Where X is
    // still A, k0 = 0 and out of place, the update brings the other columns.)
    for (int idx = tid; idx < n * w; idx += NT) {
      const int i = idx / w, c = idx % w;
      X[(int64_t)i * ldx + k0 + c] = P[pidx(pos2row[i], c, W)];
    }
    // the first exact zero pivot of the matrix (earlier panels win)
    if (info && tid == 0 && zero && info[e] == 0) info[e] = k0 + zero;
    __syncthreads();
  }
}

// Eight warps, 16 rows of the slab each at a time, two CTAs per SM: what
// bounds a CTA is the latency of its loads (the start values, then the staged
// rows), so twice the warps of a 32-row tile count for more than its reuse of R.
constexpr int UPD_THREADS = 256;
constexpr int UPD_ROWS = UPD_THREADS / 2;  // rows of one pass
constexpr int UPD_CW = 32;        // columns per CTA
constexpr int UPD_LDR = UPD_CW + 2;

inline size_t update_smem(int n, int W) {
  return (size_t)UPD_ROWS * W * sizeof(cplx) + (size_t)2 * W * UPD_LDR * sizeof(cplx) + (size_t)n * sizeof(int);
}

// Position i of the slab: [i not in panel] S[sigma(i)] + sum_j P[sigma(i), j] R[j],
// S = X, or A for the first panel of an out-of-place call (S and X are then
// different matrices and every element of X outside the panel is written here).
__global__ void __launch_bounds__(UPD_THREADS, 2)
    zinv_update_kernel(int n, int64_t batch, const cplx* s_base, int64_t lds, int64_t ss, cplx* x_base, int64_t ldx,
                       int64_t sx, int k0, int w, int W, SplitScratch sc, const int* active) {
  qtx_grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cplx* P = reinterpret_cast<cplx*>(smem_raw);  // per warp 16 rows P[sigma(i)], swizzled
  cplx* R = P + UPD_ROWS * W;                   // w x UPD_LDR
  cplx* D = R + W * UPD_LDR;                    // w x UPD_LDR
  int* sig = reinterpret_cast<int*>(D + W * UPD_LDR);
  const int g = lane >> 2, t = lane & 3;
  cplx* Pw = P + warp * 16 * W;
  const int c0 = blockIdx.x * UPD_CW;
  // a slab inside the panel has nothing to update
  if (c0 >= k0 && min(c0 + UPD_CW, n) <= k0 + w) return;
  for (int64_t e = blockIdx.y; e < batch; e += gridDim.y) {
    if (active && !active[e]) continue;
    const cplx* S = s_base + e * ss;
    cplx* X = x_base + e * sx;
    const bool pairs = pair_access_ok(X, ldx, n) && pair_access_ok(S, lds, n);
    const cplx* pe = sc.p + e * (int64_t)n * W;
    for (int i = tid; i < n; i += UPD_THREADS) sig[i] = sc.sigma[e * n + i];
    __syncthreads();
    for (int idx = tid; idx < w * UPD_CW; idx += UPD_THREADS) {
      const int j = idx / UPD_CW, cc = idx % UPD_CW;
      const bool ok = c0 + cc < n;
      cp_async16(&R[j * UPD_LDR + cc], ok ? &S[(int64_t)sig[k0 + j] * lds + c0 + cc] : S, ok);
      cp_async16(&D[j * UPD_LDR + cc], ok ? &S[(int64_t)(k0 + j) * lds + c0 + cc] : S, ok);
    }
    bool staged = false;
    for (int row0 = warp * 16; row0 < n || !staged; row0 += UPD_ROWS) {
      // the warp's own P rows (no other warp reads them)
      for (int idx = lane; idx < 16 * W; idx += 32) {
        const int i = row0 + idx / W, c = idx % W;
        const bool ok = i < n && c < w;
        cp_async16(&Pw[pidx(idx / W, c, W)], ok ? &pe[(int64_t)sig[i] * W + c] : pe, ok);
      }
      cp_async_commit();
      // Rows that start from themselves load while the staged copies are in
      // flight (only this warp writes these positions); rows displaced by a
      // pivot swap (sigma(i) is then a row of [k0, k0 + w)) are patched from D
      // after the barrier, positions inside the panel start from zero.
      double acc_re[4][4], acc_im[4][4];
      int src_of[2];  // sigma(i), -1 past the matrix
      bool in_panel[2];
#pragma unroll
      for (int hq = 0; hq < 2; ++hq) {
        const int i = row0 + g + hq * 8;
        in_panel[hq] = i >= k0 && i < k0 + w;
        const int src = i < n ? sig[i] : -1;
        src_of[hq] = src;
        const bool own = i < n && src == i && !in_panel[hq];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          const int c = c0 + ni * 8 + 2 * t;  // even
          cplx y0 = cmk(0, 0), y1 = cmk(0, 0);
          if (own) {
            const cplx* p = S + (int64_t)i * lds + c;
            if (pairs) {
              if (c < n) ld_pair(p, y0, y1);
            } else {
              if (c < n) y0 = p[0];
              if (c + 1 < n) y1 = p[1];
            }
          }
          acc_re[ni][hq * 2] = y0.x;
          acc_im[ni][hq * 2] = y0.y;
          acc_re[ni][hq * 2 + 1] = y1.x;
          acc_im[ni][hq * 2 + 1] = y1.y;
        }
      }
      cp_async_wait<0>();
      if (!staged) {
        __syncthreads();
        staged = true;
      } else {
        __syncwarp();
      }
      if (row0 >= n) break;
#pragma unroll
      for (int hq = 0; hq < 2; ++hq) {
        const int i = row0 + g + hq * 8;
        const int src = src_of[hq];
        if (src >= 0 && src != i && !in_panel[hq]) {
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int ql = 0; ql < 2; ++ql) {
              const int cc = ni * 8 + 2 * t + ql;
              const cplx y = D[(src - k0) * UPD_LDR + cc];
              acc_re[ni][hq * 2 + ql] = y.x;
              acc_im[ni][hq * 2 + ql] = y.y;
            }
        }
      }
      for (int kk = 0; kk < w; kk += 4) {
        const int kc = kk + t;
        cplx af[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) af[h] = kc < w ? Pw[pidx(g + h * 8, kc, W)] : cmk(0, 0);
        cplx bf[4];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) bf[ni] = kc < w ? R[kc * UPD_LDR + ni * 8 + g] : cmk(0, 0);
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          dmma(acc_re[ni], af[0].x, af[1].x, bf[ni].x);
          dmma(acc_im[ni], af[0].x, af[1].x, bf[ni].y);
        }
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          dmma(acc_re[ni], -af[0].y, -af[1].y, bf[ni].y);
          dmma(acc_im[ni], af[0].y, af[1].y, bf[ni].x);
        }
      }
#pragma unroll
      for (int hq = 0; hq < 2; ++hq) {
        const int i = row0 + g + hq * 8;
        if (i >= n) continue;
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          const int c = c0 + ni * 8 + 2 * t;  // even
          const cplx v0 = cmk(acc_re[ni][hq * 2], acc_im[ni][hq * 2]);
          const cplx v1 = cmk(acc_re[ni][hq * 2 + 1], acc_im[ni][hq * 2 + 1]);
          cplx* p = X + (int64_t)i * ldx + c;
          if (pairs) {
            if (c < n && !(c >= k0 && c < k0 + w)) st_pair(p, v0, v1);
          } else {
            if (c < n && !(c >= k0 && c < k0 + w)) p[0] = v0;
            if (c + 1 < n && !(c + 1 >= k0 && c + 1 < k0 + w)) p[1] = v1;
          }
        }
      }
      __syncwarp();  // every lane is done with the warp's P rows
    }
    __syncthreads();
  }
}

// Undo the row interchanges as column interchanges (reverse order),
// UNS_ROWS rows per CTA.
constexpr int UNS_ROWS = 8;

inline size_t split_unscramble_smem(int n) {
  return 2 * ((n * sizeof(int) + 15) & ~size_t(15)) + (size_t)UNS_ROWS * n * sizeof(cplx);
}

__global__ void __launch_bounds__(THREADS)
    zinv_split_unscramble_kernel(int n, int64_t batch, cplx* x_base, int64_t ldx, int64_t sx, SplitScratch sc,
                                 const int* active) {
  qtx_grid_dependency();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const size_t iw = (n * sizeof(int) + 15) & ~size_t(15);
  int* colsrc = reinterpret_cast<int*>(smem_raw);
  int* perm = reinterpret_cast<int*>(smem_raw + iw);
  cplx* rows = reinterpret_cast<cplx*>(smem_raw + 2 * iw);
  const int tid = threadIdx.x;
  const int r0 = blockIdx.x * UNS_ROWS, nr = min(UNS_ROWS, n - r0);
  for (int64_t e = blockIdx.y; e < batch; e += gridDim.y) {
    if (active && !active[e]) continue;
    cplx* X = x_base + e * sx;
    for (int c = tid; c < n; c += THREADS) perm[c] = sc.perm[e * n + c];
    __syncthreads();
    // undoing the swaps from the last to the first leaves column c with what
    // the swaps, applied to its index from the first to the last, arrive at
    for (int c = tid; c < n; c += THREADS) {
      int y = c;
      for (int k = 0; k < n; ++k) {
        const int q = perm[k];
        y = y == k ? q : (y == q ? k : y);
      }
      colsrc[c] = y;
    }
    for (int idx = tid; idx < nr * n; idx += THREADS) {
      const int r = idx / n, c = idx % n;
      rows[idx] = X[(int64_t)(r0 + r) * ldx + c];
    }
    __syncthreads();
    for (int idx = tid; idx < nr * n; idx += THREADS) {
      const int r = idx / n, c = idx % n;
      X[(int64_t)(r0 + r) * ldx + c] = rows[r * n + colsrc[c]];
    }
    __syncthreads();
  }
}

}  // namespace

namespace {

template <int TPR, int RPT, int CPT>
void launch_inv_r(int n, int64_t batch, MatView a, MutView x, int* info, const int* active, cudaStream_t stream) {
  const size_t smem = inv_smem_bytes(n);
  qtx_opt_in_smem((const void*)zinv_gj_kernel<TPR, RPT, CPT>, smem);
  int grid = (int)(batch < 65535 ? batch : 65535);
  qtx_launch(zinv_gj_kernel<TPR, RPT, CPT>, grid, THREADS, smem, stream, n, batch, a.ptr, a.ld, a.stride, x.ptr,
             x.ld, x.stride, info, active);
}

template <int TPR, int CPT, int NW>
void launch_regs(int n, int64_t batch, MatView a, MutView x, int* info, const int* active, cudaStream_t stream) {
  const unsigned grid = (unsigned)(batch < (int64_t)1 << 30 ? batch : (int64_t)1 << 30);
  qtx_launch(zinv_regs_kernel<TPR, CPT, NW>, grid, 32 * NW, 0, stream, n, batch, a.ptr, a.ld, a.stride, x.ptr, x.ld,
             x.stride, info, active);
}

// QTX_INV_SPLIT_BELOW sends batches of that many matrices or more of n > 64 to
// the one-launch kernel (0: all of them), which takes no scratch.  The two-launch
// panels are the faster form at every batch measured (b = 256: 1.31 against 1.50
// ms for 148 matrices, 0.54 against 1.26 for 16), so by default all batches take
// them.
int64_t split_below() {
  static const int64_t v = [] {
    const char* e = getenv("QTX_INV_SPLIT_BELOW");
    return e ? (int64_t)atoll(e) : INT64_MAX;
  }();
  return v;
}

size_t split_bytes(int n, int64_t batch) {
  return sizeof(cplx) * (size_t)batch * n * panel_width(n) + sizeof(int) * (size_t)batch * 2 * n + 256;
}

template <int TPR, int CPT, int NW>
void launch_split(int n, int64_t batch, MatView a, MutView x, void* scratch, int* info, const int* active,
                  cudaStream_t stream) {
  constexpr int W = TPR * CPT;
  const unsigned gb = (unsigned)(batch < 65535 ? batch : 65535);
  const unsigned nslab = (n + UPD_CW - 1) / UPD_CW;
  const size_t psmem = panel_smem(n, W), usmem = update_smem(n, W), xsmem = split_unscramble_smem(n);
  qtx_opt_in_smem((const void*)zinv_panel_kernel<TPR, CPT, NW>, psmem);
  qtx_opt_in_smem((const void*)zinv_update_kernel, usmem);
  qtx_opt_in_smem((const void*)zinv_split_unscramble_kernel, xsmem);
  SplitScratch sc;
  sc.p = reinterpret_cast<cplx*>(scratch);
  sc.sigma = reinterpret_cast<int*>(sc.p + (size_t)batch * n * W);
  sc.perm = sc.sigma + (size_t)batch * n;

  for (int k0 = 0; k0 < n; k0 += W) {
    const int w = std::min(W, n - k0);
    qtx_launch(zinv_panel_kernel<TPR, CPT, NW>, gb, 32 * NW, psmem, stream, n, batch, a.ptr, a.ld, a.stride, x.ptr,
               x.ld, x.stride, k0, sc, info, active);
    qtx_check_launch("zinv_panel_kernel");
    // the first update reads A itself, so an out-of-place call needs no copy
    const MatView from = k0 == 0 ? a : MatView(x);
    qtx_launch(zinv_update_kernel, dim3(nslab, gb), UPD_THREADS, usmem, stream, n, batch, from.ptr, from.ld,
               from.stride, x.ptr, x.ld, x.stride, k0, w, W, sc, active);
    qtx_check_launch("zinv_update_kernel");
  }
  qtx_launch(zinv_split_unscramble_kernel, dim3((n + UNS_ROWS - 1) / UNS_ROWS, gb), THREADS, xsmem, stream, n, batch,
             x.ptr, x.ld, x.stride, sc, active);
  qtx_check_launch("zinv_split_unscramble_kernel");
}

}  // namespace

size_t zinv_workspace_bytes(int n, int64_t batch) {
  return n <= 64 || n > 512 || batch >= split_below() ? 0 : split_bytes(n, batch);
}

void launch_zinv(int n, int64_t batch, MatView a, MutView x, int* info, const int* active, cudaStream_t stream,
                 bool may_allocate) {
  if (n <= 0 || batch <= 0) return;
  if (n > 512) throw QtxError(QTX_E_UNSUPPORTED, "qtx inverse: block size above 512");
  if (n <= 32) {
    launch_regs<4, 8, 4>(n, batch, a, x, info, active, stream);
    qtx_check_launch("zinv_regs_kernel");
    return;
  }
  if (n <= 64) {
    launch_regs<4, 16, 8>(n, batch, a, x, info, active, stream);
    qtx_check_launch("zinv_regs_kernel");
    return;
  }
  // without scratch (not allowed, or none left) the one-launch kernel runs
  void* scratch =
      may_allocate && batch < split_below() ? qtx_malloc_async(split_bytes(n, batch), stream) : nullptr;
  if (scratch) {
    if (n <= 128) launch_split<2, 16, 8>(n, batch, a, x, scratch, info, active, stream);
    else if (n <= 256) launch_split<1, 32, 8>(n, batch, a, x, scratch, info, active, stream);
    else if (n <= 384) launch_split<1, 16, 12>(n, batch, a, x, scratch, info, active, stream);
    else launch_split<1, 16, 16>(n, batch, a, x, scratch, info, active, stream);
    cudaFreeAsync(scratch, stream);
    return;
  }
  // the instances of inv_shape's panel widths: W = TPR * CPT
  if (n <= 96) launch_inv_r<2, 1, 8>(n, batch, a, x, info, active, stream);
  else if (n <= 128) launch_inv_r<2, 1, 16>(n, batch, a, x, info, active, stream);
  else if (n <= 256) launch_inv_r<1, 1, 32>(n, batch, a, x, info, active, stream);
  else launch_inv_r<1, 2, 16>(n, batch, a, x, info, active, stream);
  qtx_check_launch("zinv_gj_kernel");
}
