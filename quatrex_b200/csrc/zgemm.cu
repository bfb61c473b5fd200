// Batched complex FP64 GEMM on the sm_100a FP64 tensor path (DMMA,
// mma.sync m16n8k4 f64), the work-horse of every RGF block product.
//
// D = alpha op(A) op(B) + beta C + gamma C2 over a strided batch, op in
// {none, conjugate transpose}.  Complex products use the 4M real
// decomposition on split fragments: Re += Ar Br - Ai Bi, Im += Ar Bi + Ai Br,
// four DMMAs per 16x8 complex tile step.
//
// K step 16, double-buffered cp.async pipeline, 4 warps, and two CTA tiles:
//   64x64, warp tile 32x32, two CTAs per SM (80 KB each)
//   32x32, warp tile 16x16, four CTAs per SM (40 KB each)
// Bound by the DMMA pipe where the tiles fill whole waves (89 % active with
// 64x64 tiles at b = 256, 148 matrices; 83 % with 32x32 ones at b = 96, 592
// matrices; 67 % at b = 100, where a third of the tiles' area is padding), so
// the choice is the one with the shorter last wave: see wide_tile().  Per output element both run the same DMMA sequence, so the
// result does not depend on the tile.
//
// Tried and not kept: three real products instead of four (Gauss's identity,
// in either variant): 9 % faster at b = 256 (0.565 against 0.623 ms for 148
// matrices; the fragment sums hold the shared FP64 pipe), but the surface
// Green's functions of the decimation then end 1.3 times (1.16 times with the
// chains cut in two) further from an extended-precision result.
// Tiles stay complex-interleaved in shared memory so one 16-byte load yields
// both parts of an element; the padded row strides (20 and 66 / 34 complex) make
// every 8-lane fragment load hit 8 distinct 16-byte bank groups.
#include <algorithm>

#include "kernels.h"

namespace {

constexpr int BK = 16, STAGES = 2, THREADS = 128;
constexpr int LD_KMAJOR = BK + 4;  // tile stored [row][k]: 20 complex = 320 B rows

template <int TILE>
struct Cfg {
  static constexpr int W = TILE / 2, MI = W / 16, NI = W / 8;  // warp tile W x W: MI x NI DMMA tiles
  static constexpr int LD_MMAJOR = TILE + 2;                   // tile stored [k][row]: 66 / 34 complex
  static constexpr int ELEMS = TILE * LD_KMAJOR > BK * LD_MMAJOR ? TILE * LD_KMAJOR : BK * LD_MMAJOR;
  static constexpr int SMEM_BYTES = STAGES * 2 * ELEMS * (int)sizeof(cplx);
  static constexpr int CTAS_PER_SM = TILE == 64 ? 2 : 4;
};

__device__ __forceinline__ void dmma(double (&c)[4], double a0, double a1, double b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a0), "d"(a1), "d"(b0));
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int bytes = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

struct Params {
  int m, n, k;
  int64_t batch;
  const cplx* a; int64_t lda, sa;
  const cplx* b; int64_t ldb, sb;
  const cplx* c; int64_t ldc, sc; cplx beta;
  const cplx* c2; int64_t ldc2, sc2; cplx gamma;
  cplx* d; int64_t ldd, sd; cplx alpha;
  const int* active;
  const cplx* diag_shift;
  int op_a, op_b;
};

// Products of one launch (grid.y picks one).
struct Group {
  Params p[ZGEMM_GROUP_MAX];
};

// Load one K-slice of op(A) (TILE x BK) into shared memory.
template <int TILE, int OPA>
__device__ __forceinline__ void load_a(cplx* sm, const Params& p, const cplx* a, int m0, int k0, int tid) {
#pragma unroll
  for (int r = 0; r < (TILE * BK) / THREADS; ++r) {
    int idx = tid + r * THREADS;
    if (OPA == OP_N) {
      int row = idx / BK, col = idx % BK;  // A stored m x k
      int gm = m0 + row, gk = k0 + col;
      bool ok = gm < p.m && gk < p.k;
      const cplx* src = ok ? a + (int64_t)gm * p.lda + gk : a;
      cp_async16(sm + row * LD_KMAJOR + col, src, ok);
    } else {
      int krow = idx / TILE, mcol = idx % TILE;  // A stored k x m
      int gk = k0 + krow, gm = m0 + mcol;
      bool ok = gm < p.m && gk < p.k;
      const cplx* src = ok ? a + (int64_t)gk * p.lda + gm : a;
      cp_async16(sm + krow * Cfg<TILE>::LD_MMAJOR + mcol, src, ok);
    }
  }
}

// Load one K-slice of op(B) (BK x TILE) into shared memory.
template <int TILE, int OPB>
__device__ __forceinline__ void load_b(cplx* sm, const Params& p, const cplx* b, int n0, int k0, int tid) {
#pragma unroll
  for (int r = 0; r < (TILE * BK) / THREADS; ++r) {
    int idx = tid + r * THREADS;
    if (OPB == OP_N) {
      int krow = idx / TILE, ncol = idx % TILE;  // B stored k x n
      int gk = k0 + krow, gn = n0 + ncol;
      bool ok = gn < p.n && gk < p.k;
      const cplx* src = ok ? b + (int64_t)gk * p.ldb + gn : b;
      cp_async16(sm + krow * Cfg<TILE>::LD_MMAJOR + ncol, src, ok);
    } else {
      int nrow = idx / BK, kcol = idx % BK;  // B stored n x k
      int gn = n0 + nrow, gk = k0 + kcol;
      bool ok = gn < p.n && gk < p.k;
      const cplx* src = ok ? b + (int64_t)gn * p.ldb + gk : b;
      cp_async16(sm + nrow * LD_KMAJOR + kcol, src, ok);
    }
  }
}

template <int TILE, int OPA>
__device__ __forceinline__ cplx frag_a(const cplx* sm, int m, int k) {
  if (OPA == OP_N) return sm[m * LD_KMAJOR + k];
  cplx v = sm[k * Cfg<TILE>::LD_MMAJOR + m];
  return make_double2(v.x, -v.y);
}
template <int TILE, int OPB>
__device__ __forceinline__ cplx frag_b(const cplx* sm, int k, int n) {
  if (OPB == OP_N) return sm[k * Cfg<TILE>::LD_MMAJOR + n];
  cplx v = sm[n * LD_KMAJOR + k];
  return make_double2(v.x, -v.y);
}

// One K step of 4: fragments of lane (g, t) at rows / columns m + 16 mi (+ 8),
// n + 8 ni and depth k, four DMMAs per complex tile.
template <int TILE, int OPA, int OPB>
__device__ __forceinline__ void mma_step(const cplx* sa, const cplx* sb, int m, int n, int k,
                                         double (&acc_re)[Cfg<TILE>::MI][Cfg<TILE>::NI][4],
                                         double (&acc_im)[Cfg<TILE>::MI][Cfg<TILE>::NI][4]) {
  using C = Cfg<TILE>;
  cplx af[C::MI][2], bf[C::NI];
#pragma unroll
  for (int mi = 0; mi < C::MI; ++mi) {
    af[mi][0] = frag_a<TILE, OPA>(sa, m + mi * 16, k);
    af[mi][1] = frag_a<TILE, OPA>(sa, m + mi * 16 + 8, k);
  }
#pragma unroll
  for (int ni = 0; ni < C::NI; ++ni) bf[ni] = frag_b<TILE, OPB>(sb, k, n + ni * 8);
  // first product of every accumulator, then the second (the order
  // within each accumulator is unchanged: Ar Br, -Ai Bi / Ar Bi, Ai Br)
#pragma unroll
  for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
    for (int ni = 0; ni < C::NI; ++ni) {
      dmma(acc_re[mi][ni], af[mi][0].x, af[mi][1].x, bf[ni].x);
      dmma(acc_im[mi][ni], af[mi][0].x, af[mi][1].x, bf[ni].y);
    }
#pragma unroll
  for (int mi = 0; mi < C::MI; ++mi)
#pragma unroll
    for (int ni = 0; ni < C::NI; ++ni) {
      dmma(acc_re[mi][ni], -af[mi][0].y, -af[mi][1].y, bf[ni].y);
      dmma(acc_im[mi][ni], af[mi][0].y, af[mi][1].y, bf[ni].x);
    }
}

template <int TILE, int OPA, int OPB>
__device__ __forceinline__ void gemm_tile(const Params& p, int m0, int n0) {
  using C = Cfg<TILE>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx* smem = reinterpret_cast<cplx*>(smem_raw);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wm0 = (warp >> 1) * C::W, wn0 = (warp & 1) * C::W;
  const int ktiles = (p.k + BK - 1) / BK;
  // a warp tile outside the matrix only copies (small tile: the wide one is
  // taken where the tiles are full)
  const bool has_tile = m0 + wm0 < p.m && n0 + wn0 < p.n;

  for (int64_t e = blockIdx.z; e < p.batch; e += gridDim.z) {
    if (p.active && !p.active[e]) continue;
    const cplx* a = p.a + e * p.sa;
    const cplx* b = p.b + e * p.sb;

    double acc_re[C::MI][C::NI][4], acc_im[C::MI][C::NI][4];
#pragma unroll
    for (int i = 0; i < C::MI; ++i)
#pragma unroll
      for (int j = 0; j < C::NI; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc_re[i][j][q] = acc_im[i][j][q] = 0.0;

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
      if (s < ktiles) {
        cplx* sa = smem + s * 2 * C::ELEMS;
        load_a<TILE, OPA>(sa, p, a, m0, s * BK, tid);
        load_b<TILE, OPB>(sa + C::ELEMS, p, b, n0, s * BK, tid);
      }
      cp_async_commit();
    }

    for (int kt = 0; kt < ktiles; ++kt) {
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      {
        int nk = kt + STAGES - 1;
        if (nk < ktiles) {
          cplx* sa = smem + (nk % STAGES) * 2 * C::ELEMS;
          load_a<TILE, OPA>(sa, p, a, m0, nk * BK, tid);
          load_b<TILE, OPB>(sa + C::ELEMS, p, b, n0, nk * BK, tid);
        }
        cp_async_commit();
      }
      if (TILE == 32 && !has_tile) continue;
      const cplx* sa = smem + (kt % STAGES) * 2 * C::ELEMS;
      const cplx* sb = sa + C::ELEMS;
      if (TILE == 32 && (kt + 1) * BK > p.k) {
        // steps past k hold zeros and are left out
#pragma unroll 1
        for (int kk = 0; kk < p.k - kt * BK; kk += 4)
          mma_step<TILE, OPA, OPB>(sa, sb, wm0 + g, wn0 + g, kk + t, acc_re, acc_im);
        continue;
      }
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4)
        mma_step<TILE, OPA, OPB>(sa, sb, wm0 + g, wn0 + g, kk + t, acc_re, acc_im);
    }
    cp_async_wait<0>();
    __syncthreads();

    // Epilogue: D = alpha acc + beta C + gamma C2
    cplx* d = p.d + e * p.sd;
    const cplx* c = p.c ? p.c + e * p.sc : nullptr;
    const cplx* c2 = p.c2 ? p.c2 + e * p.sc2 : nullptr;
#pragma unroll
    for (int mi = 0; mi < C::MI; ++mi) {
#pragma unroll
      for (int ni = 0; ni < C::NI; ++ni) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          int row = m0 + wm0 + mi * 16 + g + ((q >> 1) << 3);
          int col = n0 + wn0 + ni * 8 + 2 * t + (q & 1);
          if (row < p.m && col < p.n) {
            cplx v = cmul(p.alpha, cmk(acc_re[mi][ni][q], acc_im[mi][ni][q]));
            if (c) v = cfma(p.beta, c[(int64_t)row * p.ldc + col], v);
            if (c2) v = cfma(p.gamma, c2[(int64_t)row * p.ldc2 + col], v);
            if (p.diag_shift && row == col) v = cadd(v, p.diag_shift[e]);
            d[(int64_t)row * p.ldd + col] = v;
          }
        }
      }
    }
  }
}

template <int TILE, int OPA, int OPB>
__global__ void __launch_bounds__(THREADS, Cfg<TILE>::CTAS_PER_SM) zgemm_dmma_kernel(Params p) {
  qtx_grid_dependency();
  gemm_tile<TILE, OPA, OPB>(p, blockIdx.y * TILE, blockIdx.x * TILE);
}

// Several products, grid.y picks one (32x32 tiles in row order along grid.x).
__global__ void __launch_bounds__(THREADS, Cfg<32>::CTAS_PER_SM) zgemm_group_kernel(const __grid_constant__ Group g) {
  qtx_grid_dependency();
  const Params& p = g.p[blockIdx.y];
  const int ntiles_n = (p.n + 31) / 32;
  const int m0 = (int)(blockIdx.x / ntiles_n) * 32, n0 = (int)(blockIdx.x % ntiles_n) * 32;
  if (m0 >= p.m) return;  // fewer tiles than the largest product
  if (p.op_a == OP_N) {
    if (p.op_b == OP_N) gemm_tile<32, OP_N, OP_N>(p, m0, n0);
    else gemm_tile<32, OP_N, OP_C>(p, m0, n0);
  } else {
    if (p.op_b == OP_N) gemm_tile<32, OP_C, OP_N>(p, m0, n0);
    else gemm_tile<32, OP_C, OP_C>(p, m0, n0);
  }
}

template <int TILE, int OPA, int OPB>
void launch_t(const Params& p, cudaStream_t stream) {
  constexpr int smem = Cfg<TILE>::SMEM_BYTES;
  // opt-in to the large shared-memory carve-out (per device)
  qtx_opt_in_smem((const void*)zgemm_dmma_kernel<TILE, OPA, OPB>, smem);
  const dim3 grid(ceil_div_u(p.n, TILE), ceil_div_u(p.m, TILE), (unsigned)(p.batch < 65535 ? p.batch : 65535));
  qtx_launch(zgemm_dmma_kernel<TILE, OPA, OPB>, grid, THREADS, smem, stream, p);
}

int sm_count() {
  int dev = 0, sms = 0;
  QTX_CUDA_TRY(cudaGetDevice(&dev));
  QTX_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return sms;
}

// Waves of the resident CTAs that `tiles` take.
template <int TILE>
int64_t waves(int64_t tiles, int sms) {
  const int64_t resident = (int64_t)Cfg<TILE>::CTAS_PER_SM * sms;
  return (tiles + resident - 1) / resident;
}
template <int TILE>
int64_t tiles_of(const Params& p) {
  return (int64_t)((p.m + TILE - 1) / TILE) * ((p.n + TILE - 1) / TILE) * p.batch;
}

// The tile whose waves finish first.  A full wave of 64x64 tiles covers twice
// the outputs of a full wave of 32x32 ones in twice the time, less about
// 1.5 % (b = 256, 148 matrices, 8.0 waves: 0.614 ms against 0.623 ms).  A
// nearly empty last wave costs more than that: 32x32 / 64x64 tiles take
// 9.0 / 17.4 us for 32 matrices of b = 64, 17.9 / 24.0 us for 24 of b = 100,
// 66 / 86 us for 100 of b = 128, 0.796 / 0.878 ms for 24 of b = 512; 84 / 81
// us for 16 of b = 256 (two waves against one).
bool wide_tile(const Params& p, int sms) {
  if (p.m > 32 * 65535) return true;  // grid.y
  return 0.985 * 2.0 * (double)waves<64>(tiles_of<64>(p), sms) <= (double)waves<32>(tiles_of<32>(p), sms);
}

template <int OPA, int OPB>
void launch_op(const Params& p, int sms, cudaStream_t stream) {
  if (wide_tile(p, sms)) launch_t<64, OPA, OPB>(p, stream);
  else launch_t<32, OPA, OPB>(p, stream);
}

void launch_one(const Params& p, int sms, cudaStream_t stream) {
  if (p.op_a == OP_N && p.op_b == OP_N) launch_op<OP_N, OP_N>(p, sms, stream);
  else if (p.op_a == OP_N && p.op_b == OP_C) launch_op<OP_N, OP_C>(p, sms, stream);
  else if (p.op_a == OP_C && p.op_b == OP_N) launch_op<OP_C, OP_N>(p, sms, stream);
  else launch_op<OP_C, OP_C>(p, sms, stream);
  qtx_check_launch("zgemm_dmma_kernel");
}

void launch_several(const Group& g, int count, cudaStream_t stream) {
  constexpr int smem = Cfg<32>::SMEM_BYTES;
  qtx_opt_in_smem((const void*)zgemm_group_kernel, smem);
  int64_t tiles = 0, batch = 0;
  for (int q = 0; q < count; ++q) {
    tiles = std::max(tiles, tiles_of<32>(g.p[q]) / g.p[q].batch);
    batch = std::max(batch, g.p[q].batch);
  }
  qtx_launch(zgemm_group_kernel, dim3((unsigned)tiles, count, (unsigned)std::min<int64_t>(batch, 65535)), THREADS,
             smem, stream, g);
  qtx_check_launch("zgemm_group_kernel");
}

Params params_of(const GemmCall& g) {
  Params p;
  p.m = g.m; p.n = g.n; p.k = g.k; p.batch = g.batch;
  p.a = g.a.ptr; p.lda = g.a.ld; p.sa = g.a.stride;
  p.b = g.b.ptr; p.ldb = g.b.ld; p.sb = g.b.stride;
  p.c = g.c.ptr; p.ldc = g.c.ld; p.sc = g.c.stride; p.beta = g.beta;
  p.c2 = g.c2.ptr; p.ldc2 = g.c2.ld; p.sc2 = g.c2.stride; p.gamma = g.gamma;
  p.d = g.d.ptr; p.ldd = g.d.ld; p.sd = g.d.stride; p.alpha = g.alpha;
  p.active = g.active;
  p.diag_shift = g.diag_shift;
  p.op_a = g.op_a;
  p.op_b = g.op_b;
  return p;
}

}  // namespace

// Products of up to GROUP_WAVES waves of 32x32 tiles share a launch.  A product
// of less than one wave costs its latency whatever runs beside it; the group
// kernel itself is about 2 us slower than the one-product kernel (it looks its
// operands up in the parameter array), so products that fill the GPU for many
// waves keep their own launches.
constexpr int GROUP_WAVES = 4;

void launch_zgemm_group(const GemmCall* calls, int count, cudaStream_t stream) {
  Group g;
  int n = 0;
  const int sms = sm_count();
  auto flush = [&]() {
    if (n == 1) launch_one(g.p[0], sms, stream);
    else if (n > 1) launch_several(g, n, stream);
    n = 0;
  };
  for (int q = 0; q < count; ++q) {
    if (calls[q].m <= 0 || calls[q].n <= 0 || calls[q].batch <= 0) continue;
    const Params p = params_of(calls[q]);
    if (waves<32>(tiles_of<32>(p), sms) > GROUP_WAVES) {
      launch_one(p, sms, stream);
      continue;
    }
    g.p[n++] = p;
    if (n == ZGEMM_GROUP_MAX) flush();
  }
  flush();
}

void launch_zgemm(const GemmCall& g, cudaStream_t stream) {
  if (g.m <= 0 || g.n <= 0 || g.batch <= 0) return;
  launch_one(params_of(g), sm_count(), stream);
}
