// dgemm.cu — FP64 GEMM with BOLA's rounding (src/gemm.rs:88-377), on DFMA.
//
// GB300's FP64 rate is ~1.25 TFLOP/s through DFMA (DMMA m8n8k4 measures 12%
// lower and shares the pipe: both at once retire no more), so this kernel is
// compute-bound at every shape BOLA's path produces: even a rank-32 update
// reads 16 B per 64 flop.  A 64x64 tile of depth 32 keeps an SM busy for 32 us,
// so what is left to gain is balance: every launch mixes tile sizes, large
// tiles for the full rounds and ever smaller ones for what remains (plan_tiles
// below); outputs too small for the GPU split K, over the CTAs of a cluster or
// over partial sums in memory; and the unfused edge elements run beside the
// tiles.
//
// Accumulation order, per element of C in BOLA's full 8x4 micro-tiles:
//   c = beta-scaled C;  for each K chunk of kc (64 in gemm, 32 in syrk):
//     acc = 0; for k in chunk: acc = fma(op(A)[i,k], op(B)[k,j], acc);
//     c = fma(alpha, acc, c)
// and in BOLA's partial edge tiles (rows >= m rounded down to 8, or columns
// >= n rounded down to 4): c = c + (alpha * op(B)[k,j]) * op(A)[i,k], unfused.
#include <cooperative_groups.h>

#include "common.cuh"
#include "sm100.cuh"

namespace bola {
namespace {

namespace cg = cooperative_groups;

constexpr int KT = 8;    // K depth of one shared-memory stage (divides every kc)
constexpr int STG = 4;   // stages: three in flight while one is used
constexpr int EDGE_T = 64;  // edge elements per CTA, of one row or one column (a thread each)
// Threads per tile side, each with a TM x TN block of C in registers.  A
// multiply-add takes two operands from shared memory, and GB300 feeds its FP64
// pipe at 98% of the measured peak with 4x4 per thread, 92% with 2x2, and 83%
// with 2x2 and a single CTA on an SM (4864 x 32..96, K = 4096); so 4x4 for 64x64
// tiles, 4x2 for 32x32 (128 threads), 2x2 for 16x16 (64 threads).  8x8 (64
// threads, an element each) is for outputs so small that a warp's own chain of
// multiply-adds, 65 cycles each, is what takes the time.
template <int B>
struct Tile {
  static constexpr int TM = B == 8 ? 1 : B == 16 ? 2 : 4, TN = B == 64 ? 4 : B == 8 ? 1 : 2;
  static constexpr int TX = B / TM, TY = B / TN, NT = TX * TY;
};

struct GemmArgs {
  int64_t m, n, m8, n4, K;
  double alpha, beta;
  const double *A, *B;
  double *C;
  int64_t lda, ldb, ldc;
  int kc;
  const int32_t *info;
  int tri;
  int first;       // this launch is the product's first
  int edge;        // CTAs that take the edge elements
  int big;         // CTAs with a 64x64 cell, a 32x32 block, a 16x16 block
  int n32, n16;
  int fm, fn;      // cells across: full ones
  int gm, gn;      // and all
  int cps;         // split K: chunks per CTA (and pass over the cluster)
  double *P;       // split K over memory: chunk ch of (i, j) at P[i + j m8 + ch m8 n4]
};

__device__ __forceinline__ bool tri_keep(int tri, int64_t i, int64_t j) {
  if (tri == 0) return true;
  const int64_t bi = i >> 5, bj = j >> 5;
  return tri == 1 ? (bi < bj) : (bi > bj);
}

template <bool T>
__device__ __forceinline__ double op_a(const double *A, int64_t lda, int64_t i, int64_t k) {
  return T ? A[k + i * lda] : A[i + k * lda];
}
template <bool T>
__device__ __forceinline__ double op_b(const double *B, int64_t ldb, int64_t k, int64_t j) {
  return T ? B[j + k * ldb] : B[k + j * ldb];
}

template <int BM, int BN>
__host__ __device__ constexpr size_t stage_bytes() {
  return sizeof(double) * STG * KT * (BM + 1 + BN + 1);
}

// Asynchronous copy of one double into shared memory; zero if !valid.
__device__ __forceinline__ void copy_async8(double *dst, const double *src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(sm100::smem_u32(dst)), "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}

// The chunk accumulators of the tile at (i0, j0) over K chunks [ch0, ch1):
// chunk_done(ch, acc) gets each of them.  The operands come through a ring of
// STG stages filled by asynchronous copies, three stages (>= 6000 cycles of
// products) ahead: loads staged through registers, one 16-deep stage ahead,
// left a CTA that was alone on its SM waiting for memory a quarter of its time.
// Run by the CTA's NT threads, or (TEAM) by one of its teams of NT threads, each
// with a ring of its own.
template <int BM, int BN, int TM, int TN, int NT, bool TA, bool TB, bool TEAM = false, typename F>
__device__ __forceinline__ void tile_chunks(const GemmArgs &g, int64_t i0, int64_t j0, int64_t ch0, int64_t ch1,
                                            unsigned char *smem, F &&chunk_done) {
  constexpr int TX = BM / TM, TY = BN / TN;
  constexpr int AE = (BM * KT + NT - 1) / NT, BE = (BN * KT + NT - 1) / NT;  // (a 16-wide stage is less than 256 threads)
  static_assert(TX * TY == NT, "threads");
  double(*As)[KT][BM + 1] = reinterpret_cast<double(*)[KT][BM + 1]>(smem);
  double(*Bs)[KT][BN + 1] = reinterpret_cast<double(*)[KT][BN + 1]>(smem + sizeof(double) * STG * KT * (BM + 1));
  const int tid = TEAM ? threadIdx.x % NT : threadIdx.x, tx = tid % TX, ty = tid / TX;
  auto sync = [] {
    if constexpr (TEAM) {
      __syncwarp();
      asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / NT), "n"(NT) : "memory");
    } else {
      __syncthreads();
    }
  };
  const int64_t kbeg = ch0 * g.kc, kend = imin(ch1 * g.kc, g.K);
  const int nst = (int)((kend - kbeg + KT - 1) / KT);
  // this thread's elements of a stage: where they are now, and whether their row or column exists
  const double *pa[AE], *pb[BE];
  bool va[AE], vb[BE];
#pragma unroll
  for (int t = 0; t < AE; ++t) {
    const int e = tid + NT * t, ii = TA ? e / KT : e % BM, kk = TA ? e % KT : e / BM;
    va[t] = i0 + ii < g.m8;
    pa[t] = va[t] ? g.A + (TA ? (kbeg + kk) + (i0 + ii) * g.lda : (i0 + ii) + (kbeg + kk) * g.lda) : g.A;
  }
#pragma unroll
  for (int t = 0; t < BE; ++t) {
    const int e = tid + NT * t, jj = TB ? e % BN : e / KT, kk = TB ? e / BN : e % KT;
    vb[t] = j0 + jj < g.n4;
    pb[t] = vb[t] ? g.B + (TB ? (j0 + jj) + (kbeg + kk) * g.ldb : (kbeg + kk) + (j0 + jj) * g.ldb) : g.B;
  }
  const int64_t da = TA ? KT : KT * g.lda, db = TB ? KT * g.ldb : KT;
  auto fetch = [&](int s) {  // stage s, in order
    if (s < nst) {
      const int left = (int)imin(KT, kend - kbeg - (int64_t)s * KT), buf = s % STG;
#pragma unroll
      for (int t = 0; t < AE; ++t) {
        const int e = tid + NT * t, ii = TA ? e / KT : e % BM, kk = TA ? e % KT : e / BM;
        const bool v = va[t] && kk < left;
        if (BM * KT % NT == 0 || e < BM * KT) copy_async8(&As[buf][kk][ii], v ? pa[t] : g.A, v);
        pa[t] += da;
      }
#pragma unroll
      for (int t = 0; t < BE; ++t) {
        const int e = tid + NT * t, jj = TB ? e % BN : e / KT, kk = TB ? e / BN : e % KT;
        const bool v = vb[t] && kk < left;
        if (BN * KT % NT == 0 || e < BN * KT) copy_async8(&Bs[buf][kk][jj], v ? pb[t] : g.B, v);
        pb[t] += db;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  double acc[TM][TN];
#pragma unroll
  for (int s = 0; s < STG - 1; ++s) fetch(s);
  const int kc = g.kc;
  int kin = 0;  // depth within the current chunk
  int64_t ch = ch0;
  for (int s = 0; s < nst; ++s) {
    if (kin == 0) {
#pragma unroll
      for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int q = 0; q < TN; ++q) acc[r][q] = 0.0;
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(STG - 2) : "memory");
    sync();  // stage s is there for every thread, and stage s - 1 is used up
    fetch(s + STG - 1);
    const int buf = s % STG;
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      double a[TM], b[TN];
#pragma unroll
      for (int r = 0; r < TM; ++r) a[r] = As[buf][kk][tx + TX * r];
#pragma unroll
      for (int q = 0; q < TN; ++q) b[q] = Bs[buf][kk][ty + TY * q];
#pragma unroll
      for (int r = 0; r < TM; ++r)
#pragma unroll
        for (int q = 0; q < TN; ++q) acc[r][q] = fused(a[r], b[q], acc[r][q]);
    }
    kin += KT;
    if (kin == kc || s + 1 == nst) {
      chunk_done(ch++, acc);
      kin = 0;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  sync();  // the ring may be filled again
}

// One B x B tile of C over all of K, on NT threads.
template <int B, int NT, bool TA, bool TB>
__device__ __forceinline__ void tile_direct(const GemmArgs &g, int64_t i0, int64_t j0, unsigned char *smem) {
  constexpr int TM = NT == Tile<B>::NT ? Tile<B>::TM : B / 16, TN = NT == Tile<B>::NT ? Tile<B>::TN : B / 16;
  constexpr int TX = B / TM, TY = B / TN;
  if (i0 >= g.m8 || j0 >= g.n4) return;
  if (g.tri == 1 && (i0 >> 5) >= ((j0 + B - 1) >> 5)) return;
  if (g.tri == 2 && ((i0 + B - 1) >> 5) <= (j0 >> 5)) return;
  const int64_t ci = i0 + threadIdx.x % TX, cj = j0 + threadIdx.x / TX;
  // C as loaded: nothing waits for it (nor scales it) before the first chunk is done
  double c[TM][TN];
#pragma unroll
  for (int r = 0; r < TM; ++r)
#pragma unroll
    for (int q = 0; q < TN; ++q) {
      const int64_t gi = ci + TX * r, gj = cj + TY * q;
      c[r][q] = gi < g.m8 && gj < g.n4 && g.beta != 0.0 ? g.C[gi + gj * g.ldc] : 0.0;
    }
  bool scale = g.beta != 0.0 && g.beta != 1.0;
  auto apply_beta = [&] {
    if (!scale) return;
    scale = false;
#pragma unroll
    for (int r = 0; r < TM; ++r)
#pragma unroll
      for (int q = 0; q < TN; ++q) c[r][q] = __dmul_rn(c[r][q], g.beta);
  };
  tile_chunks<B, B, TM, TN, NT, TA, TB>(g, i0, j0, 0, (g.K + g.kc - 1) / g.kc, smem,
                                        [&](int64_t, double(&acc)[TM][TN]) {
                                          apply_beta();
#pragma unroll
                                          for (int r = 0; r < TM; ++r)
#pragma unroll
                                            for (int q = 0; q < TN; ++q)
                                              c[r][q] = fused(g.alpha, acc[r][q], c[r][q]);
                                        });
  apply_beta();
#pragma unroll
  for (int r = 0; r < TM; ++r)
#pragma unroll
    for (int q = 0; q < TN; ++q) {
      const int64_t gi = ci + TX * r, gj = cj + TY * q;
      if (gi < g.m8 && gj < g.n4 && tri_keep(g.tri, gi, gj)) g.C[gi + gj * g.ldc] = c[r][q];
    }
}

// BOLA's edge tiles (add_scalar_kernel, src/gemm.rs:357-377): unfused
// c += (alpha * b) * a over all k in order.  A CTA takes 64 elements of one
// row below m8 or of one column right of n4, a thread each.  An element's chain
// is two FP64 operations per k, 128 cycles for a warp alone on its
// sub-partition; everything else a warp issues adds to that, so the operands
// come through the same ring of asynchronous copies as the tiles' (loads and
// address arithmetic per element: 420 cycles per k).
__host__ __device__ constexpr size_t edge_bytes() {
  return sizeof(double) * STG * KT * (EDGE_T + 2);
}
__host__ __device__ inline int64_t edge_ctas(int64_t m, int64_t n, int64_t m8, int64_t n4) {
  return (m - m8) * cdiv(n, EDGE_T) + (n - n4) * cdiv(m8, EDGE_T);
}
template <bool TA, bool TB>
__device__ __forceinline__ void edge_elements(const GemmArgs &g, int64_t block, unsigned char *smem) {
  double(*V)[KT][EDGE_T + 1] = reinterpret_cast<double(*)[KT][EDGE_T + 1]>(smem);
  double(*S)[KT] = reinterpret_cast<double(*)[KT]>(smem + sizeof(double) * STG * KT * (EDGE_T + 1));
  const int tid = threadIdx.x;
  // the 64 elements run over columns of C (row i) or over rows (column j); V
  // holds the operand that runs with them, S the other one
  const int64_t across = cdiv(g.n, EDGE_T), rows = (g.m - g.m8) * across;
  const bool row = block < rows;
  int64_t i, j, v0, vn;
  if (row) {
    i = g.m8 + block / across;
    v0 = block % across * EDGE_T;
    vn = g.n;
    j = v0 + tid;
  } else {
    const int64_t down = cdiv(g.m8, EDGE_T), f = block - rows;
    j = g.n4 + f / down;
    v0 = f % down * EDGE_T;
    vn = g.m8;
    i = v0 + tid;
  }
  // strides of V along its elements and along k, and of S along k
  const int64_t ve = row ? (TB ? 1 : g.ldb) : (TA ? g.lda : 1), vk = row ? (TB ? g.ldb : 1) : (TA ? 1 : g.lda);
  const int64_t sk = row ? (TA ? 1 : g.lda) : (TB ? g.ldb : 1);
  const double *vp = (row ? g.B : g.A) + v0 * ve;
  const double *sp = row ? g.A + (TA ? i * g.lda : i) : g.B + (TB ? j : j * g.ldb);
  const bool ek = vk == 1;  // k runs fastest in memory: consecutive threads along k
  const bool mine = v0 + tid < vn && tri_keep(g.tri, i, j);
  double c = 0.0;
  if (mine && g.beta != 0.0) {
    c = g.C[i + j * g.ldc];
    if (g.beta != 1.0) c = __dmul_rn(c, g.beta);
  }
  const int nst = (int)((g.K + KT - 1) / KT);
  const double *src[KT];  // this thread's KT elements of a stage: where they are now
#pragma unroll
  for (int t = 0; t < KT; ++t) {
    const int e = tid + EDGE_T * t, el = ek ? e / KT : e % EDGE_T, kk = ek ? e % KT : e / EDGE_T;
    src[t] = v0 + el < vn ? vp + el * ve + kk * vk : nullptr;
  }
  auto fetch = [&](int s) {
    if (s < nst) {
      const int left = (int)imin(KT, g.K - (int64_t)s * KT), buf = s % STG;
#pragma unroll
      for (int t = 0; t < KT; ++t) {
        const int e = tid + EDGE_T * t, el = ek ? e / KT : e % EDGE_T, kk = ek ? e % KT : e / EDGE_T;
        const bool v = src[t] != nullptr && kk < left;
        copy_async8(&V[buf][kk][el], v ? src[t] : vp, v);
        if (src[t] != nullptr) src[t] += KT * vk;
      }
      if (tid < KT) copy_async8(&S[buf][tid], tid < left ? sp + (s * (int64_t)KT + tid) * sk : sp, tid < left);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const bool unit = g.alpha == 1.0 || g.alpha == -1.0;  // scales exactly: a sign instead of a product
  const long long flip = g.alpha == -1.0 ? (long long)0x8000000000000000ull : 0;
#pragma unroll
  for (int s = 0; s < STG - 1; ++s) fetch(s);
  for (int s = 0; s < nst; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STG - 2) : "memory");
    __syncthreads();
    fetch(s + STG - 1);
    const int buf = s % STG, left = (int)imin(KT, g.K - (int64_t)s * KT);
    double t[KT], x[KT];
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) {
      const double v = V[buf][kk][tid], w = S[buf][kk];
      const double bv = row ? v : w;
      x[kk] = row ? w : v;
      t[kk] = unit ? __longlong_as_double(__double_as_longlong(bv) ^ flip) : __dmul_rn(g.alpha, bv);
    }
    if (left == KT) {
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) c = add_prod(c, t[kk], x[kk]);
    } else {
#pragma unroll
      for (int kk = 0; kk < KT; ++kk)
        if (kk < left) c = add_prod(c, t[kk], x[kk]);
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (mine) g.C[i + j * g.ldc] = c;
}

// t-th cell (ci > cj) below the diagonal, row by row.
__device__ __forceinline__ void strictly_lower(int t, int &ci, int &cj) {
  int r = (int)((1.f + sqrtf(1.f + 8.f * (float)t)) * 0.5f);
  while ((int64_t)r * (r - 1) / 2 > t) --r;
  while ((int64_t)(r + 1) * r / 2 <= t) ++r;
  ci = r;
  cj = t - (int)((int64_t)r * (r - 1) / 2);
}

// Cell t in launch order.  Whole C: the full cells column by column, then the
// ragged bottom row and right column.  A triangle: the cells off the diagonal
// row by row, then (DIAG) the cells on it.
template <bool DIAG>
__device__ __forceinline__ void cell_at(const GemmArgs &g, int t, int &ci, int &cj) {
  if (g.tri == 0) {
    const int full = g.fm * g.fn;
    if (t < full) {
      ci = t % g.fm;
      cj = t / g.fm;
    } else if (t - full < (g.gm - g.fm) * g.gn) {
      ci = g.fm;
      cj = t - full;
    } else {
      ci = t - full - (g.gm - g.fm) * g.gn;
      cj = g.fn;
    }
    return;
  }
  const int gs = max(g.gm, g.gn), off = (int)((int64_t)gs * (gs - 1) / 2);
  if (DIAG && t >= off) {
    ci = cj = t - off;
  } else {
    strictly_lower(t, ci, cj);
  }
  if (g.tri == 1) {
    const int x = ci;
    ci = cj;
    cj = x;
  }
}

// A product takes up to three launches, one after the other on the stream but
// side by side on the GPU: each is a programmatic dependent of the one before,
// touches other elements of C, lets the next one start as soon as its CTAs are
// placed, and waits for the one before at its end only, so that what follows on
// the stream finds all of them done.
// The first one waits for whatever precedes the product before it lets the
// others start.
struct InParallel {
  __device__ explicit InParallel(const GemmArgs &g) {
    if (g.first) sm100::grid_dependency_wait();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  }
  __device__ ~InParallel() { sm100::grid_dependency_wait(); }
};

template <bool TA, bool TB>
__global__ void __launch_bounds__(EDGE_T) gemm_edges(const __grid_constant__ GemmArgs g) {
  __shared__ __align__(16) unsigned char smem[edge_bytes()];
  InParallel ip(g);
  if (!stop_flag(g.info)) edge_elements<TA, TB>(g, blockIdx.x, smem);
}

// All of K in one CTA per tile: the first `big` cells of 64x64 as one tile
// each, the others as 32x32 and, the last of them, 16x16 blocks.  104 registers
// a thread: two CTAs then leave an SM room for one of the small kernels of a
// factorisation's critical stream (a 32-row solve, a swap), which otherwise
// waits for a tile to end.
template <bool TA, bool TB>
__global__ void __maxnreg__(104) gemm_grid64(const __grid_constant__ GemmArgs g) {
  __shared__ __align__(16) unsigned char smem[stage_bytes<64, 64>()];
  InParallel ip(g);
  if (stop_flag(g.info)) return;
  int b = (int)blockIdx.x, ci, cj;
  if (b < g.big) {
    cell_at<true>(g, b, ci, cj);
    tile_direct<64, Tile<64>::NT, TA, TB>(g, 64 * (int64_t)ci, 64 * (int64_t)cj, smem);
    return;
  }
  b -= g.big;
  const int q = b < g.n32 ? b : g.n32 + (b - g.n32) / 4;  // the 32x32 block
  cell_at<true>(g, g.big + q / 4, ci, cj);
  const int64_t i0 = 64 * (int64_t)ci + 32 * (q & 1), j0 = 64 * (int64_t)cj + 32 * ((q >> 1) & 1);
  if (b < g.n32) {
    tile_direct<32, Tile<64>::NT, TA, TB>(g, i0, j0, smem);
  } else {
    const int h = (b - g.n32) & 3;
    tile_direct<16, Tile<64>::NT, TA, TB>(g, i0 + 16 * (h & 1), j0 + 16 * (h >> 1), smem);
  }
}

// The same with cells of 32x32, in up to two launches: BT = 32 takes the first
// n32 cells, BT = 16 the others as 16x16 blocks (BT = 8: cells of 8x8, all of
// them).
template <int BT, bool TA, bool TB>
__global__ void __launch_bounds__(Tile<BT>::NT, BT == 32 ? 5 : BT == 16 ? 10 : 12)
gemm_grid32(const __grid_constant__ GemmArgs g) {
  __shared__ __align__(16) unsigned char smem[stage_bytes<BT, BT>()];
  InParallel ip(g);
  if (stop_flag(g.info)) return;
  const int b = (int)blockIdx.x;
  int ci, cj;
  if (BT != 16) {
    cell_at<false>(g, b, ci, cj);
    tile_direct<BT, Tile<BT>::NT, TA, TB>(g, BT * (int64_t)ci, BT * (int64_t)cj, smem);
  } else {
    cell_at<false>(g, g.n32 + b / 4, ci, cj);
    tile_direct<BT, Tile<BT>::NT, TA, TB>(g, 32 * (int64_t)ci + 16 * (b & 1), 32 * (int64_t)cj + 16 * ((b >> 1) & 1), smem);
  }
}

// K split over memory: a CTA leaves the accumulators of its chunks of a 32x32
// tile in P, and gemm_fold adds them to C in chunk order.
template <bool TA, bool TB>
__global__ void __launch_bounds__(Tile<32>::NT, 5) gemm_partial(const __grid_constant__ GemmArgs g) {
  using T = Tile<32>;
  __shared__ __align__(16) unsigned char smem[stage_bytes<32, 32>()];
  InParallel ip(g);
  if (stop_flag(g.info)) return;
  const int64_t nchunks = (g.K + g.kc - 1) / g.kc, nsplit = (nchunks + g.cps - 1) / g.cps;
  const int64_t t = blockIdx.x / nsplit, sp = blockIdx.x % nsplit;
  int ci, cj;
  cell_at<false>(g, (int)t, ci, cj);
  const int64_t i0 = 32 * (int64_t)ci, j0 = 32 * (int64_t)cj;
  tile_chunks<32, 32, T::TM, T::TN, T::NT, TA, TB>(
      g, i0, j0, sp * g.cps, imin(nchunks, (sp + 1) * g.cps), smem, [&](int64_t ch, double(&acc)[T::TM][T::TN]) {
        double *p = g.P + ch * (g.m8 * g.n4);
#pragma unroll
        for (int r = 0; r < T::TM; ++r)
#pragma unroll
          for (int q = 0; q < T::TN; ++q) {
            const int64_t gi = i0 + threadIdx.x % T::TX + T::TX * r, gj = j0 + threadIdx.x / T::TX + T::TY * q;
            if (gi < g.m8 && gj < g.n4) p[gi + gj * g.m8] = acc[r][q];
          }
      });
}

// The fold is a chain of one multiply-add (~65 cycles) per chunk and element; the
// next FOLD_U chunks' sums are on their way meanwhile (one at a time, a load each:
// 700 cycles a chunk; 64 x 64 x 100,000: 535 us of 1210).
constexpr int FOLD_T = 128, FOLD_U = 16;
__global__ void __launch_bounds__(FOLD_T) gemm_fold(const __grid_constant__ GemmArgs g) {
  if (stop_flag(g.info)) return;
  const int64_t e = (int64_t)blockIdx.x * FOLD_T + threadIdx.x, plane = g.m8 * g.n4;
  if (e >= plane) return;
  const int64_t i = e % g.m8, j = e / g.m8;
  if (!tri_keep(g.tri, i, j)) return;
  double c = 0.0;
  if (g.beta != 0.0) {
    c = g.C[i + j * g.ldc];
    if (g.beta != 1.0) c = __dmul_rn(c, g.beta);
  }
  const int64_t nchunks = (g.K + g.kc - 1) / g.kc;
  const double *p = g.P + e;
  double next[FOLD_U];
  auto fetch = [&](int64_t ch0) {
#pragma unroll
    for (int u = 0; u < FOLD_U; ++u) next[u] = ch0 + u < nchunks ? p[(ch0 + u) * plane] : 0.0;
  };
  fetch(0);
  for (int64_t ch0 = 0; ch0 < nchunks; ch0 += FOLD_U) {
    double v[FOLD_U];
#pragma unroll
    for (int u = 0; u < FOLD_U; ++u) v[u] = next[u];
    fetch(ch0 + FOLD_U);
#pragma unroll
    for (int u = 0; u < FOLD_U; ++u)
      if (ch0 + u < nchunks) c = fused(g.alpha, v[u], c);
  }
  g.C[i + j * g.ldc] = c;
}

// K split over the CTAs of a cluster: each leaves its chunks' accumulators in
// its shared memory, and every CTA then folds its share of the tile's elements
// over all chunks in order, reading the others' through distributed shared
// memory.  A CTA has TEAMS teams of a tile's threads, each with chunks of its own
// (g.cps at a time): four for 8x8 tiles where K has more chunks than the cluster
// CTAs, since a team by itself leaves the FP64 pipe waiting for its own chain
// (without memory, 16 x 16 x 32,768: 112 us with teams, 242 without; 64 x 64 x
// 16,384: 153 and 226).  Teams of 16x16 tiles want clusters of eight for as many
// CTAs, and those share SMs: 280 us for the latter.  No CTA may leave the cluster's
// barriers early, so *info is looked at when C is written.
constexpr int SPLIT_TEAMS = 4;
template <int BT, int TEAMS, bool TA, bool TB>
__global__ void __launch_bounds__(Tile<BT>::NT *TEAMS) gemm_split(const __grid_constant__ GemmArgs g) {
  constexpr int TM = Tile<BT>::TM, TN = Tile<BT>::TN, TX = Tile<BT>::TX, TY = Tile<BT>::TY, NT = Tile<BT>::NT;
  constexpr int TILE = BT * BT, RING = (int)stage_bytes<BT, BT>(), T = NT * TEAMS;
  static_assert(RING % 16 == 0, "the teams' rings");
  __shared__ __align__(16) unsigned char smem[RING * TEAMS];
  extern __shared__ __align__(16) unsigned char part_raw[];
  double *part = reinterpret_cast<double *>(part_raw);  // [TEAMS][cps][TILE], element (i, j) at i + BT j
  const int team = threadIdx.x / NT, tid = threadIdx.x % NT;
  cg::cluster_group cluster = cg::this_cluster();
  const int ns = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  InParallel ip(g);
  int ci, cj;
  cell_at<false>(g, (int)blockIdx.x / ns, ci, cj);
  const int64_t i0 = BT * (int64_t)ci, j0 = BT * (int64_t)cj;
  const int64_t nchunks = (g.K + g.kc - 1) / g.kc;
  // this thread's elements of the fold
  constexpr int EP = TILE / 2 > T ? TILE / 2 / T : 1;  // clusters of 2 and more
  const int share = (TILE + ns - 1) / ns;
  double c[EP];
  int el[EP];
  double *cp[EP];
#pragma unroll
  for (int h = 0; h < EP; ++h) {
    const int f = (int)threadIdx.x + T * h;
    el[h] = rank * share + f;
    const int64_t gi = i0 + el[h] % BT, gj = j0 + el[h] / BT;
    cp[h] = f < share && el[h] < TILE && gi < g.m8 && gj < g.n4 && tri_keep(g.tri, gi, gj) ? g.C + gi + gj * g.ldc : nullptr;
    c[h] = 0.0;
    if (cp[h] != nullptr && g.beta != 0.0) {
      c[h] = *cp[h];
      if (g.beta != 1.0) c[h] = __dmul_rn(c[h], g.beta);
    }
  }
  const int per = TEAMS * g.cps;  // chunks of a CTA at a time
  for (int64_t base = 0; base < nchunks; base += (int64_t)ns * per) {
    const int64_t first = base + (int64_t)rank * per;
    const int64_t ch0 = imin(nchunks, first + (int64_t)team * g.cps), ch1 = imin(nchunks, ch0 + g.cps);
    tile_chunks<BT, BT, TM, TN, NT, TA, TB, (TEAMS > 1)>(
        g, i0, j0, ch0, ch1, smem + RING * team, [&](int64_t ch, double(&acc)[TM][TN]) {
          double *p = part + (ch - first) * TILE + tid % TX + BT * (tid / TX);
#pragma unroll
          for (int r = 0; r < TM; ++r)
#pragma unroll
            for (int q = 0; q < TN; ++q) p[TX * r + BT * TY * q] = acc[r][q];
        });
    cluster.sync();
    const int64_t end = imin(nchunks, base + (int64_t)ns * per);
#pragma unroll
    for (int h = 0; h < EP; ++h) {
      if (cp[h] == nullptr) continue;
      int64_t ch = base;
      for (int r = 0; r < ns && ch < end; ++r) {
        const double *p = cluster.map_shared_rank(part, r) + el[h];
        const int cnt = (int)imin(per, end - ch);
        for (int s0 = 0; s0 < cnt; s0 += 8) {
          double v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = s0 + u < cnt ? p[(s0 + u) * TILE] : 0.0;
#pragma unroll
          for (int u = 0; u < 8; ++u)
            if (s0 + u < cnt) c[h] = fused(g.alpha, v[u], c[h]);
        }
        ch += cnt;
      }
    }
    cluster.sync();
  }
  if (stop_flag(g.info)) return;
#pragma unroll
  for (int h = 0; h < EP; ++h)
    if (cp[h] != nullptr) *cp[h] = c[h];
}

// ---- planning ------------------------------------------------------------------

// The launches of one product.  An SM's time for a CTA is its tile area x depth
// / 2 cycles (two FP64 multiply-adds per clock), whatever the tile, so the
// plan fills the GPU with the largest tiles in full rounds over all SMs and
// cuts what remains into smaller ones, so that the last round is short:
//  - GRID64: 64x64 cells, two CTAs per SM (registers), in full rounds of
//    2 x SMs; the remaining and the ragged cells as 32x32 blocks, and those
//    that would again start a round of their own as 16x16 blocks (worth a
//    CTA's ~2 us of launch and first loads from a depth of 128 on);
//  - GRID32, below 2 x SMs cells: 32x32 blocks in full rounds, the rest 16x16;
//  - GRID8: 8x8 blocks;
//  - CLUSTER: K over clusters of 2, 4 or 8 CTAs (6 with teams), where that
//    shortens the most loaded SM's time (a fold costs ~70 cycles a chunk and two
//    barriers), by one team of threads or four in each;
//  - MEMORY: K in pieces of `cps` chunks over memory, where many chunks allow
//    a finer balance than 8 CTAs (two more passes over the partial sums, a
//    launch and the fold's chain), up to SPLIT_BYTES of them; beyond what the
//    pool keeps, mapping them again takes 1.6 us per MiB (512 x 512 x 8192, 256
//    MiB: 3.62 ms, 4.02 when each call is waited for; 3.93 over clusters).
// The last four are compared by the cycles they are estimated to take.
enum Path { GRID64, GRID32, GRID8, CLUSTER, MEMORY };
struct TilePlan {
  GemmArgs g;
  Path path = GRID32;
  int split = 1, tile = 32, teams = 1;  // CLUSTER: CTAs, tile, teams in a CTA
  int rounds = 0;            // GRID32: 32x32 blocks side by side on an SM
  int64_t cells = 0;
};
constexpr int64_t SPLIT_BYTES = (int64_t)1 << 30;
constexpr int64_t KEPT_BYTES = (int64_t)64 << 20;  // what the scratch pool keeps between calls
constexpr int64_t SM_SMEM = 224 * 1024;  // shared memory of an SM that CTAs can take

// Cells of `t` x `t` that C's main region has: full ones, all, and all that a triangle keeps.
struct Cells {
  int fm, fn, gm, gn;
  int64_t full, all;
};
Cells count_cells(int64_t m8, int64_t n4, int t, int tri, bool diag) {
  Cells c;
  c.fm = (int)(m8 / t);
  c.fn = (int)(n4 / t);
  c.gm = (int)cdiv(m8, t);
  c.gn = (int)cdiv(n4, t);
  if (tri == 0) {
    c.full = (int64_t)c.fm * c.fn;
    c.all = (int64_t)c.gm * c.gn;
  } else {
    const int64_t f = imin(c.fm, c.fn), gs = imax(c.gm, c.gn);
    c.full = f * (f - 1) / 2;
    c.all = gs * (gs - 1) / 2 + (diag ? gs : 0);
  }
  return c;
}

TilePlan plan_tiles(const GemmArgs &args, int sms, bool may_alloc) {
  TilePlan p;
  p.g = args;
  GemmArgs &g = p.g;
  g.edge = (int)edge_ctas(g.m, g.n, g.m8, g.n4);
  if (g.m8 == 0 || g.n4 == 0) return p;
  const int64_t slots = 2 * (int64_t)sms, nch = (g.K + g.kc - 1) / g.kc;
  Cells c = count_cells(g.m8, g.n4, 64, g.tri, true);
  if (c.full >= slots) {
    p.path = GRID64;
    g.big = (int)(c.full / slots * slots);
    const int64_t rest = 4 * (c.all - g.big), small = g.K >= 128 ? rest % slots : 0;
    g.n32 = (int)(rest - small);
    g.n16 = (int)(4 * small);
  } else {
    c = count_cells(g.m8, g.n4, 32, g.tri, false);
    // 32x32 blocks in rounds of o CTAs on every SM (at most five: registers;
    // fewer than three leave the FP64 pipe waiting), the rest as 16x16
    const int64_t per_sm = c.all / sms;
    double least = 1e300;
    for (int o = 1; o <= 5; ++o) {
      if (o < 3 && o < per_sm) continue;
      const int64_t n32 = per_sm / o * o * sms, n16 = 4 * (c.all - n32);
      const double t = 4.0 * (double)(n32 / sms) + 1.05 * (double)cdiv(n16, sms);
      if (t < least) {
        least = t;
        p.rounds = o;
        g.n32 = (int)n32;
        g.n16 = (int)n16;
      }
    }
    // Cycles per step of k on the most loaded SM, `ctas` CTAs of t x t tiles:
    // the FP64 pipe's (at the efficiency measured for the tile's registers
    // with several CTAs on an SM), but at least one warp's own.
    auto per_k = [](int t, int64_t ctas) {
      const double pipe = t == 32 ? 528.0 : t == 16 ? 138.0 : 48.0, own = t == 32 ? 660.0 : t == 16 ? 320.0 : 100.0;
      return ctas == 0 ? 0.0 : imax(1, ctas) * pipe > own ? (double)ctas * pipe : own;
    };
    double best = (double)g.K * (per_k(32, cdiv(g.n32, sms)) + (g.n32 > 0 ? 138.0 * (double)cdiv(g.n16, sms)
                                                                          : per_k(16, cdiv(g.n16, sms))));
    for (int t = 8; t <= 32; t *= 2) {
      if (t < 32 && g.tri != 0) continue;  // (a triangle's cells are 32x32 blocks)
      const int64_t T = count_cells(g.m8, g.n4, t, g.tri, false).all;
      for (int s = t == 8 ? 1 : 2; s <= 8 && (s == 1 || s <= nch); s *= 2) {
        const double cost = per_k(t, cdiv(T * s, sms)) * (double)imin(g.K, cdiv(nch, s) * g.kc) +
                            (s > 1 ? 3000.0 + 70.0 * (double)nch : 0.0);
        if (cost < 0.95 * best) {
          best = cost;
          p.path = s == 1 ? GRID8 : CLUSTER;
          p.split = s;
          p.tile = t;
          p.teams = 1;
        }
      }
      // The same by teams: 37 to 44 cycles per step of k and team; clusters of s
      // leave about 4 s SMs over, until there are enough for several rounds.
      double by_teams = 1e300;
      int s_teams = 0;
      for (int s = 2; s <= 8 && t == 8 && nch > 8; s += 2) {
        const int64_t fit = imax(1, sms - 4 * s);
        const int64_t ctas = cdiv(T * s, T * s <= 2 * fit ? fit : sms);
        const double cost = SPLIT_TEAMS * (double)ctas * (ctas == 1 ? 44.0 : 37.0) *
                                (double)imin(g.K, cdiv(nch, s * SPLIT_TEAMS) * g.kc) +
                            3000.0 + 70.0 * (double)nch;
        if (cost < by_teams) {
          by_teams = cost;
          s_teams = s;
        }
      }
      if (by_teams < 0.95 * best) {
        best = by_teams;
        p.path = CLUSTER;
        p.split = s_teams;
        p.tile = t;
        p.teams = SPLIT_TEAMS;
      }
    }
    const int64_t bytes = 8 * nch * g.m8 * g.n4;
    if (may_alloc && nch >= 16 && bytes <= SPLIT_BYTES)
      for (int cps = 1; cps <= 4; ++cps) {
        const double cost = per_k(32, cdiv(c.all * cdiv(nch, cps), sms)) * (double)(cps * g.kc) + 10000.0 +
                            (double)bytes / (bytes > KEPT_BYTES ? 255.0 : 1500.0) + 70.0 * (double)nch;
        if (cost < best) {
          best = cost;
          p.path = MEMORY;
          g.cps = cps;
        }
      }
  }
  if (p.path == CLUSTER || p.path == GRID8) {
    c = count_cells(g.m8, g.n4, p.tile, g.tri, false);
    // at most 64 KB of partial sums a CTA, 32 of one with teams (which takes up to four an SM)
    g.cps = (int)imin(cdiv(nch, p.split * p.teams), (p.teams > 1 ? 4096 : 8192) / (p.tile * p.tile * p.teams));
  }
  p.cells = c.all;
  g.fm = c.fm;
  g.fn = c.fn;
  g.gm = c.gm;
  g.gn = c.gn;
  return p;
}

// partial: the memory of a MEMORY plan.
template <bool TA, bool TB>
int launch_plan(cudaStream_t s, TilePlan &p, double *partial) {
  GemmArgs &g = p.g;
  bool beside = false;  // a launch of this product precedes
  auto launch = [&](void (*kern)(const GemmArgs), int64_t ctas, int threads, int cluster = 0, size_t smem = 0) -> int {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    g.first = beside ? 0 : 1;
    attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    if (cluster > 0) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
      attr[cfg.numAttrs].val.clusterDim.x = (unsigned)cluster;
      attr[cfg.numAttrs].val.clusterDim.y = 1;
      attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
    BOLA_TRY(roomy(kern));
    BOLA_TRY_CUDA(cudaLaunchKernelEx(&cfg, kern, g));
    beside = true;
    return 0;
  };
  if (g.edge > 0) {
    ProfScope prof(s, "dgemm_edge", 2.0 * (double)((g.m - g.m8) * g.n + g.m8 * (g.n - g.n4)) * (double)g.K);
    BOLA_TRY(launch(gemm_edges<TA, TB>, g.edge, EDGE_T));
    if (profiling_on()) beside = false;  // timed apart
  }
  if (p.cells == 0) return 0;
  const bool two = p.path == MEMORY || (p.path == GRID32 && g.n32 > 0 && g.n16 > 0);
  ProfScope prof(s, "dgemm", 2.0 * (double)g.m8 * (double)g.n4 * (double)g.K,
                 8.0 * ((double)g.m8 * g.K + (double)g.K * g.n4 + 2.0 * (double)g.m8 * g.n4), two ? 2 : 1);
  if (p.path == GRID64) return launch(gemm_grid64<TA, TB>, g.big + g.n32 + g.n16, Tile<64>::NT);
  if (p.path == GRID8) return launch(gemm_grid32<8, TA, TB>, p.cells, Tile<8>::NT);
  if (p.path == GRID32) {
    // An SM takes as many CTAs as fit as soon as others end, so the 16x16
    // blocks would pile up on the SMs that finish first (1024^3: 2529 us).  A
    // CTA that asks for its even share of what shared memory the 32x32 blocks
    // leave spreads them (1812 us).
    size_t pad = 0;
    if (g.n32 > 0 && g.n16 > 0) {
      const int64_t per_sm = cdiv(g.n16, num_sms()), left = SM_SMEM - p.rounds * (int64_t)(stage_bytes<32, 32>() + 1024);
      const int64_t share = left / per_sm - 1024 - (int64_t)stage_bytes<16, 16>();
      if (share > 0) pad = (size_t)share;
      if (pad + stage_bytes<16, 16>() > 48 * 1024)
        BOLA_TRY_CUDA(cudaFuncSetAttribute(gemm_grid32<16, TA, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)SM_SMEM - 16 * 1024));
    }
    if (g.n32 > 0) BOLA_TRY(launch(gemm_grid32<32, TA, TB>, g.n32, Tile<32>::NT));
    return g.n16 > 0 ? launch(gemm_grid32<16, TA, TB>, g.n16, Tile<16>::NT, 0, pad) : 0;
  }
  if (p.path == CLUSTER) {
    void (*kern)(const GemmArgs) = p.tile == 32   ? gemm_split<32, 1, TA, TB>
                                   : p.tile == 16 ? gemm_split<16, 1, TA, TB>
                                   : p.teams == 1 ? gemm_split<8, 1, TA, TB>
                                                  : gemm_split<8, SPLIT_TEAMS, TA, TB>;
    const size_t smem = (size_t)g.cps * p.teams * p.tile * p.tile * sizeof(double);
    if (smem + stage_bytes<32, 32>() > 48 * 1024)
      BOLA_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024));
    return launch(kern, p.cells * p.split,
                  p.teams * (p.tile == 32 ? Tile<32>::NT : p.tile == 16 ? Tile<16>::NT : Tile<8>::NT), p.split, smem);
  }
  const int64_t nch = (g.K + g.kc - 1) / g.kc;
  g.P = partial;
  BOLA_TRY(launch(gemm_partial<TA, TB>, p.cells * cdiv(nch, g.cps), Tile<32>::NT));
  gemm_fold<<<(unsigned)cdiv(g.m8 * g.n4, FOLD_T), FOLD_T, 0, s>>>(g);
  BOLA_CHECK_LAUNCH();
  return 0;
}

// may_alloc: the partial sums of a split K may be parked in device memory.
int dgemm_body(cudaStream_t s, char ta, char tb, int64_t m, int64_t n, int64_t k, double alpha, const double *A,
               int64_t lda, const double *B, int64_t ldb, double beta, double *C, int64_t ldc, int kc,
               const int32_t *info, int tri, bool may_alloc) {
  if (m <= 0 || n <= 0) return 0;
  const bool TA = upc(ta) != 'N', TB = upc(tb) != 'N';
  GemmArgs g = {};
  g.m = m;
  g.n = n;
  g.m8 = (m / 8) * 8;
  g.n4 = (n / 4) * 4;
  g.K = (alpha == 0.0 || k < 0) ? 0 : k;  // alpha == 0: only the beta pass
  g.alpha = alpha;
  g.beta = beta;
  g.A = A;
  g.B = B;
  g.C = C;
  g.lda = lda;
  g.ldb = ldb;
  g.ldc = ldc;
  g.kc = kc;
  g.info = info;
  g.tri = tri;
  TilePlan p = plan_tiles(g, num_sms(), may_alloc);
  Scratch part;
  if (p.path == MEMORY && part.alloc((size_t)(8 * cdiv(g.K, kc) * g.m8 * g.n4), s) != 0) {
    cudaGetLastError();  // (there is a plan that needs no memory)
    p = plan_tiles(g, num_sms(), false);
  }
  double *const P = part.as<double>();
  if (!TA && !TB) return launch_plan<false, false>(s, p, P);
  if (!TA && TB) return launch_plan<false, true>(s, p, P);
  if (TA && !TB) return launch_plan<true, false>(s, p, P);
  return launch_plan<true, true>(s, p, P);
}

}  // namespace

int dgemm_exact(cudaStream_t s, char ta, char tb, int64_t m, int64_t n, int64_t k, double alpha,
                const double *A, int64_t lda, const double *B, int64_t ldb, double beta, double *C,
                int64_t ldc, int kc, const int32_t *info, int tri) {
  return dgemm_body(s, ta, tb, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, kc, info, tri, true);
}

}  // namespace bola

namespace {

int check_gemm(char transa, char transb, int64_t m, int64_t n, int64_t k, double alpha, int64_t lda, int64_t ldb,
               int64_t ldc) {
  // BOLA validates nothing beyond the empty-matrix exit (src/gemm.rs:106-108);
  // negative sizes and leading dimensions that cannot address the operands are
  // rejected here because a GPU out-of-bounds access would not stay local.
  if (m < 0) return -3;
  if (n < 0) return -4;
  if (k < 0) return -5;
  if (m == 0 || n == 0) return 0;
  const bool ta = bola::upc(transa) != 'N', tb = bola::upc(transb) != 'N';
  if (k > 0 && alpha != 0.0 && lda < bola::imax(1, ta ? k : m)) return -8;
  if (k > 0 && alpha != 0.0 && ldb < bola::imax(1, tb ? n : k)) return -10;
  if (ldc < bola::imax(1, m)) return -13;
  return 0;
}

}  // namespace

extern "C" int bola_dgemm(char transa, char transb, int64_t m, int64_t n, int64_t k, double alpha,
                          const double *a, int64_t lda, const double *b, int64_t ldb, double beta,
                          double *c, int64_t ldc, bola_stream_t stream) {
  BOLA_TRY(check_gemm(transa, transb, m, n, k, alpha, lda, ldb, ldc));
  return bola::dgemm_exact((cudaStream_t)stream, transa, transb, m, n, k, alpha, a, lda, b, ldb, beta,
                           c, ldc, 64, nullptr, 0);
}

// The allocation-free DGEMM (include/bola_gb300.h): partial sums of a split K
// stay on chip.  It keeps its documented limit, as callers test for it: outputs
// of fewer tiles than SMs (64x64, or the smaller ones with the least area on the
// most loaded SM) whose partial sums, a 64-deep chunk each, would take between
// 64 MiB and 1 GiB of memory.  (The tiles of the limit are not the plan's.)
extern "C" int bola_dgemm_noalloc(char transa, char transb, int64_t m, int64_t n, int64_t k, double alpha,
                                  const double *a, int64_t lda, const double *b, int64_t ldb, double beta,
                                  double *c, int64_t ldc, bola_stream_t stream) {
  using namespace bola;
  BOLA_TRY(check_gemm(transa, transb, m, n, k, alpha, lda, ldb, ldc));
  const int64_t m8 = (m / 8) * 8, n4 = (n / 4) * 4, nchunks = alpha == 0.0 ? 0 : cdiv(k, 64);
  if (m8 > 0 && n4 > 0 && nchunks >= 2) {
    const int sms = num_sms();
    const int tiles_of[5][2] = {{64, 64}, {64, 32}, {32, 64}, {32, 32}, {64, 16}};
    int64_t tiles = 0;
    double best = 1e300;
    for (const auto &t : tiles_of) {
      const int64_t T = cdiv(m8, t[0]) * cdiv(n4, t[1]);
      const double cost = (double)cdiv(T, sms) * t[0] * t[1];
      if (cost < best * 0.999) {
        best = cost;
        tiles = T;
      }
    }
    const double bytes = 8.0 * (double)nchunks * (double)m8 * (double)n4;
    if (tiles < sms && bytes <= (double)(1u << 30) && bytes > (double)BOLA_NOALLOC_SCRATCH_BYTES)
      return fail(BOLA_ERR_UNSUPPORTED,
                  "bola_dgemm_noalloc: the partial sums of a split K would take %.0f bytes of scratch memory (%lld "
                  "chunks x %lld x %lld doubles), and this call does not take shapes beyond %llu; use bola_dgemm",
                  bytes, (long long)nchunks, (long long)m8, (long long)n4,
                  (unsigned long long)BOLA_NOALLOC_SCRATCH_BYTES);
  }
  return dgemm_body((cudaStream_t)stream, transa, transb, m, n, k, alpha, a, lda, b, ldb, beta, c, ldc, 64, nullptr, 0,
                    false);
}
