// trsm.cu — triangular solves with BOLA's recursion and rounding
// (src/trsm.rs:33-376).
//
// The host walks BOLA's recursion (halving down to 64) and issues the exact
// DGEMM for every off-diagonal block, so >97% of the flops run in the GEMM
// kernel.  The <=64 base cases run on the GPU with BOLA's per-element order:
//   left, no transpose  — column forward/back substitution with BOLA's daxpy
//                         (left_n_base: a warp per right-hand side, rows
//                         across lanes);
//   left, transpose, and right — a system is a right-hand side or a row of B:
//                         a warp per system (tri_warp) while there are few;
//                         some hundreds to thousands of ascending ones of
//                         order <= 32 eight lanes per system (tri_asc32); a
//                         thread per system beyond (left_t_base, right_base).
#include "common.cuh"
#include "sm100.cuh"

namespace bola {
namespace {

constexpr int STOP = 64;  // TRSM_RECURSION_STOP (src/trsm.rs:8)

__global__ void scale_matrix(int64_t m, int64_t n, double alpha, double *B, int64_t ldb,
                             const int32_t *info) {
  sm100::grid_dependency_wait();
  if (stop_flag(info)) return;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m * n) return;
  const int64_t i = e % m, j = e / m;
  B[i + j * ldb] = __dmul_rn(B[i + j * ldb], alpha);
}

// store(e, load(e)) for e < count, a thread's loads eight at a time in flight
// while it has that many (the compiler keeps a load behind the store to shared
// memory before it).
template <typename L, typename S>
__device__ __forceinline__ void copy_in(int count, L &&load, S &&store) {
  constexpr int U = 8;
  const int step = blockDim.x;
  int e = threadIdx.x;
  for (; e + (U - 1) * step < count; e += U * step) {
    double v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = load(e + u * step);
#pragma unroll
    for (int u = 0; u < U; ++u) store(e + u * step, v[u]);
  }
  for (; e < count; e += step) store(e, load(e));
}

// Loads the m x m triangle block (column-major, ld = STOP) into shared memory.
__device__ __forceinline__ void load_tri(double *sA, const double *A, int64_t lda, int m) {
  copy_in(
      m * m, [&](int e) { return A[e % m + (int64_t)(e / m) * lda]; },
      [&](int e, double v) { sA[e % m + (e / m) * STOP] = v; });
}

// Left side, op(A) = A: trsm_lnl / trsm_lnu base cases (src/trsm.rs:96-123, 136-163).
// A warp per right-hand side, two rows per lane, one warp per sub-partition
// (the chain of a step, broadcast, division, multiply-add, is what it waits
// for; eight warps per CTA queued two on a sub-partition's FP64 pipe).
constexpr int LN_WARPS = 4;
template <bool LOWER>
__global__ void __launch_bounds__(32 * LN_WARPS)
left_n_base(int m, int64_t n, bool unit, const double *A, int64_t lda, double *B,
            int64_t ldb, int lanes, const int32_t *info) {
  sm100::grid_dependency_wait();
  __shared__ double sA[STOP * STOP];
  __shared__ Divisor dv[STOP];
  if (stop_flag(info)) return;
  load_tri(sA, A, lda, m);
  __syncthreads();
  if (!unit) {
    if (threadIdx.x < m) dv[threadIdx.x] = divisor(sA[threadIdx.x * (STOP + 1)]);
    __syncthreads();
  }
  const int lane = threadIdx.x & 31;
  const int64_t col = (int64_t)blockIdx.x * LN_WARPS + (threadIdx.x >> 5);
  if (col >= n) return;
  double *bc = B + col * ldb;
  double b[2] = {lane < m ? bc[lane] : 0.0, lane + 32 < m ? bc[lane + 32] : 0.0};
  // column k of the triangle, a step ahead
  auto column = [&](int k, double(&a)[2]) {
    a[0] = sA[lane + k * STOP];
    a[1] = sA[(lane + 32) + k * STOP];
  };
  double an[2];
  column(LOWER ? 0 : m - 1, an);
#pragma unroll 2
  for (int step = 0; step < m; ++step) {
    const int k = LOWER ? step : m - 1 - step;
    const double a[2] = {an[0], an[1]};
    if (step + 1 < m) column(LOWER ? k + 1 : k - 1, an);
    const double bk = __shfl_sync(0xffffffffu, k < 32 ? b[0] : b[1], k & 31);
    if (!nonzero64(bk)) continue;  // BOLA skips zero entries (src/trsm.rs:101,141)
    double u = bk;
    if (!unit) {
      u = div_rn(bk, dv[k]);
      if (k == lane) b[0] = u;
      if (k == lane + 32) b[1] = u;
      if (!nonzero64(u)) continue;  // daxpy returns early for a zero scale (src/utilities.rs:108)
    }
    // daxpy over rows k+1..m-1 (lower) or 0..k-1 (upper) with alpha = -u: the
    // last len % lanes rows are its unfused tail
    const int len = LOWER ? m - k - 1 : k, end = LOWER ? m : k, cut = end - (len & (lanes - 1));
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (LOWER ? (k >= 31 + 32 * h || m <= 32 * h) : k <= 32 * h) continue;  // no row of this half
      const int i = lane + 32 * h;
      const bool in = LOWER ? (i > k && i < m) : i < k;
      const double f = __fma_rn(-u, a[h], b[h]);
      if (cut < end && end > 32 * h && cut < 32 * h + 32) {  // (uniform) the tail lies in this half
        const double t = add_prod(b[h], -u, a[h]);
        if (in) b[h] = i < cut ? f : t;
      } else if (in) {
        b[h] = f;
      }
    }
  }
  if (lane < m) bc[lane] = b[0];
  if (lane + 32 < m) bc[lane + 32] = b[1];
}

// The base cases whose updates are BOLA's unfused t - a x, a warp per system
// (a right-hand side on the left, a row of B on the right), of order n <= 64.
// T[k][j] is the coefficient of x_k in equation j.
//  - Ascending (ltu, rnu, rtl: x_0 first, equation j takes k < j in ascending
//    order): once x_k is final every later equation subtracts it, two
//    equations per lane.
//  - Descending with ascending sums (ltl, rnl, rtu: x_{n-1} first, equation j
//    takes k > j in ascending order, the newest solution first): equation j is
//    one chain of n - 1 - j subtractions.  Its products are formed a lane per
//    k, all but the newest one a step ahead; the chain itself, ~65 cycles per
//    subtraction, is the bound (n = 48: 35 us; a thread per system, product
//    after product: 81 us).
// Left: t / a_jj; right: t * (1 / a_jj), and a zero coefficient is skipped.
constexpr int TW_WARPS = 4;
constexpr int TW_PITCH = STOP + 1;
template <bool ASC, bool RIGHT>
__global__ void __launch_bounds__(32 * TW_WARPS)
tri_warp(int n, int64_t systems, bool unit, bool transposed, const double *A, int64_t lda, double *B,
         int64_t elem, int64_t sys, const int32_t *info) {
  sm100::grid_dependency_wait();
  __shared__ double T[STOP * TW_PITCH];
  __shared__ Divisor dv[STOP];
  __shared__ __align__(16) double pbuf[TW_WARPS][2][STOP];
  if (stop_flag(info)) return;
  copy_in(
      n * n, [&](int e) { return A[e % n + (int64_t)(e / n) * lda]; },
      [&](int e, double v) {
        const int r = e % n, c = e / n;  // a(r, c): (k, j), or (j, k) when transposed
        T[transposed ? c * TW_PITCH + r : r * TW_PITCH + c] = v;
      });
  __syncthreads();
  if (!unit) {
    if (threadIdx.x < n) dv[threadIdx.x] = divisor(T[threadIdx.x * (TW_PITCH + 1)]);
    __syncthreads();
  }
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t s = (int64_t)blockIdx.x * TW_WARPS + warp;
  if (s >= systems) return;
  double *b = B + s * sys;
  double x[2] = {lane < n ? b[lane * elem] : 0.0, lane + 32 < n ? b[(lane + 32) * elem] : 0.0};
  auto finish = [&](double t, int j) { return unit ? t : RIGHT ? __dmul_rn(t, dv[j].y) : div_rn(t, dv[j]); };
  if (ASC) {
    double tn[2] = {T[lane], T[lane + 32]};
    for (int k = 0; k < n; ++k) {
      const double a[2] = {tn[0], tn[1]};
      if (k + 1 < n) {
        tn[0] = T[(k + 1) * TW_PITCH + lane];
        tn[1] = T[(k + 1) * TW_PITCH + lane + 32];
      }
      const double xk = finish(__shfl_sync(FULL, k < 32 ? x[0] : x[1], k & 31), k);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int j = lane + 32 * h;
        if (j == k) x[h] = xk;
        if (k >= 31 + 32 * h || n <= 32 * h) continue;
        const double u = sub_prod(x[h], a[h], xk);
        if (j > k && (!RIGHT || nonzero64(a[h]))) x[h] = u;
      }
    }
  } else {
    // products of equation j with the solutions k >= j + 2, into pbuf[.][j & 1];
    // which coefficients are zero (right) in zero[j & 1]
    uint64_t zero[2] = {0, 0};
    auto products = [&](int j, uint64_t &z) {
      z = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int k = lane + 32 * h;
        const bool in = k > j + 1 && k < n;
        const double a = in ? T[k * TW_PITCH + j] : 1.0;
        if (j + 1 < 31 + 32 * h && n > 32 * h) {  // (uniform) some k of this half
          const double p = __dmul_rn(a, x[h]);
          if (in) pbuf[warp][j & 1][k] = p;
        }
        if (RIGHT) z |= (uint64_t)__ballot_sync(FULL, in && !nonzero64(a)) << (32 * h);
      }
    };
    double newest = 0.0;
    for (int j = n - 1; j >= 0; --j) {
      if (j >= 1) products(j - 1, zero[(j - 1) & 1]);  // equation j - 1, with the solutions from j + 1 on
      double t = __shfl_sync(FULL, j < 32 ? x[0] : x[1], j & 31);
      const double *p = pbuf[warp][j & 1];
      const uint64_t z = zero[j & 1];
      if (j + 1 < n) {
        const double a = T[(j + 1) * TW_PITCH + j];
        if (!RIGHT || nonzero64(a)) t = sub_prod(t, a, newest);
      }
      int k = j + 2;
      if (z == 0) {
        if ((k & 1) && k < n) t = __dsub_rn(t, p[k++]);
#pragma unroll 4
        for (; k + 1 < n; k += 2) {
          const double2 v = *reinterpret_cast<const double2 *>(&p[k]);
          t = __dsub_rn(t, v.x);
          t = __dsub_rn(t, v.y);
        }
        if (k < n) t = __dsub_rn(t, p[k]);
      } else {
        for (; k < n; ++k)
          if (!((z >> k) & 1u)) t = __dsub_rn(t, p[k]);
      }
      newest = finish(t, j);
      if (lane == (j & 31)) x[j >> 5] = newest;
      __syncwarp();
    }
  }
  if (lane < n) b[lane * elem] = x[0];
  if (lane + 32 < n) b[(lane + 32) * elem] = x[1];
}

// Left side, op(A) = A^T: trsm_ltl / trsm_ltu base cases (src/trsm.rs:176-188, 215-227).
constexpr int TCOLS = 32;  // right-hand sides per block in the transposed base case

template <bool LOWER>
__global__ void __launch_bounds__(TCOLS)
left_t_base(int m, int64_t n, bool unit, const double *A, int64_t lda, double *B,
            int64_t ldb, const int32_t *info) {
  sm100::grid_dependency_wait();
  __shared__ double sA[STOP * STOP];
  __shared__ double sB[STOP * TCOLS];
  if (stop_flag(info)) return;
  load_tri(sA, A, lda, m);
  const int64_t c0 = (int64_t)blockIdx.x * TCOLS;
  const int nc = (int)imin(TCOLS, n - c0);
  for (int e = threadIdx.x; e < m * TCOLS; e += blockDim.x) {
    const int i = e % m, c = e / m;
    sB[c + i * TCOLS] = c < nc ? B[i + (c0 + c) * ldb] : 0.0;
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (c < nc) {
    for (int step = 0; step < m; ++step) {
      const int i = LOWER ? m - 1 - step : step;
      double t = sB[c + i * TCOLS];
      if (LOWER) {
        for (int k = i + 1; k < m; ++k) t = sub_prod(t, sA[k + i * STOP], sB[c + k * TCOLS]);
      } else {
        for (int k = 0; k < i; ++k) t = sub_prod(t, sA[k + i * STOP], sB[c + k * TCOLS]);
      }
      if (!unit) t = t / sA[i + i * STOP];
      sB[c + i * TCOLS] = t;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < m * TCOLS; e += blockDim.x) {
    const int i = e % m, cc = e / m;
    if (cc < nc) B[i + (c0 + cc) * ldb] = sB[cc + i * TCOLS];
  }
}

// Right side base cases (src/trsm.rs:253-273, 285-305, 317-337, 349-369).
// V: 0 = rnl, 1 = rnu, 2 = rtl, 3 = rtu.  A thread per row of B: the CTA's
// rows of B and the triangle are staged in shared memory (the row chains then
// never wait on global loads), and the reciprocals of the diagonal, which
// every row multiplies by, are formed once per CTA.
constexpr int RB_ROWS = 128;

inline size_t right_base_smem(int n) { return ((size_t)n * n + n + (size_t)RB_ROWS * n) * sizeof(double); }

template <int V>
__global__ void __launch_bounds__(RB_ROWS)
right_base(int64_t m, int n, bool unit, const double *A, int64_t lda, double *B,
           int64_t ldb, const int32_t *info) {
  sm100::grid_dependency_wait();
  extern __shared__ double rb_smem[];
  double *sA = rb_smem;      // n x n, ld n
  double *rd = sA + n * n;   // 1 / a(j, j)
  double *sB = rd + n;       // column k of the CTA's rows at sB[k * RB_ROWS]
  if (stop_flag(info)) return;
  const int64_t i0 = (int64_t)blockIdx.x * RB_ROWS;
  const int rows = (int)imin(RB_ROWS, m - i0);
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) sA[e] = A[(e % n) + (int64_t)(e / n) * lda];
  for (int e = threadIdx.x; e < RB_ROWS * n; e += blockDim.x) {
    const int r = e % RB_ROWS, k = e / RB_ROWS;
    sB[e] = r < rows ? B[(i0 + r) + (int64_t)k * ldb] : 0.0;
  }
  __syncthreads();
  if (!unit && threadIdx.x < n) rd[threadIdx.x] = 1.0 / sA[threadIdx.x * (n + 1)];
  __syncthreads();
  constexpr bool descending = (V == 0 || V == 3);
  if (threadIdx.x < rows) {
    double *b = sB + threadIdx.x;
    for (int step = 0; step < n; ++step) {
      const int j = descending ? n - 1 - step : step;
      double bj = b[j * RB_ROWS];
      const int k0 = descending ? j + 1 : 0;
      const int k1 = descending ? n : j;
      for (int k = k0; k < k1; ++k) {
        // rnl/rnu read a(k, j); rtl/rtu read a(j, k)
        const double akj = (V <= 1) ? sA[k + j * n] : sA[j + k * n];
        if (nonzero64(akj)) bj = sub_prod(bj, akj, b[k * RB_ROWS]);
      }
      if (!unit) bj = __dmul_rn(bj, rd[j]);
      b[j * RB_ROWS] = bj;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < RB_ROWS * n; e += blockDim.x) {
    const int r = e % RB_ROWS, k = e / RB_ROWS;
    if (r < rows) B[(i0 + r) + (int64_t)k * ldb] = sB[e];
  }
}

// The ascending base cases (ltu, rnu, rtl) for n <= 32 and many systems: as in
// tri_warp, but eight lanes per system, lane q holding unknowns q, q + 8, ...
// in registers, so that four systems share a warp's instructions.  (Four lanes
// per system issue a quarter less in all, but 550 FP64 instructions on a
// warp's path instead of 170; beside a GEMM, whose sixteen warps an SM queue on
// the same pipe, that made 126 us of one block column's solve at n = 4096.)
constexpr int AL = 8;  // lanes per system
constexpr int AS_THREADS = 64;
constexpr int AS_SYS = AS_THREADS / AL;

template <bool RIGHT>
__global__ void __launch_bounds__(AS_THREADS)
tri_asc32(int n, int64_t systems, bool unit, bool transposed, const double *A, int64_t lda, double *B,
          int64_t elem, int64_t sys, const int32_t *info) {
  sm100::grid_dependency_wait();
  __shared__ double T[32 * 33];  // coefficient of x_k in equation j at T[k * 33 + j]
  __shared__ Divisor dv[32];
  if (stop_flag(info)) return;
  for (int e = threadIdx.x; e < n * n; e += AS_THREADS) {
    const int r = e % n, c = e / n;
    T[transposed ? c * 33 + r : r * 33 + c] = A[r + (int64_t)c * lda];
  }
  __syncthreads();
  if (!unit && threadIdx.x < n) dv[threadIdx.x] = divisor(T[threadIdx.x * 34]);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  // lanes of a system: consecutive along the elements where those are
  // contiguous (left), else along the systems (right: the rows of B)
  const int q = RIGHT ? lane / (32 / AL) : lane & (AL - 1), w = RIGHT ? lane & (32 / AL - 1) : lane / AL;
  const int64_t s = (int64_t)blockIdx.x * AS_SYS + (threadIdx.x >> 5) * (32 / AL) + w;
  const bool on = s < systems;  // lanes of a missing system still take part in the shuffles
  double *b = B + s * sys;
  double x[32 / AL];
#pragma unroll
  for (int c = 0; c < 32 / AL; ++c) x[c] = on && q + AL * c < n ? b[(q + AL * c) * elem] : 0.0;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    if (k < n) {
      if (!unit && q == (k & (AL - 1))) x[k / AL] = RIGHT ? __dmul_rn(x[k / AL], dv[k].y) : div_rn(x[k / AL], dv[k]);
      const int src = RIGHT ? (k & (AL - 1)) * (32 / AL) + w : w * AL + (k & (AL - 1));
      const double xk = __shfl_sync(0xffffffffu, x[k / AL], src);
#pragma unroll
      for (int c = k / AL; c < 32 / AL; ++c) {  // (earlier unknowns are done)
        const int j = q + AL * c;
        const double a = T[k * 33 + j];
        const double u = sub_prod(x[c], a, xk);
        if (j > k && j < n && (!RIGHT || nonzero64(a))) x[c] = u;  // right: BOLA skips a zero a
      }
    }
  }
  if (!on) return;
#pragma unroll
  for (int c = 0; c < 32 / AL; ++c)
    if (q + AL * c < n) b[(q + AL * c) * elem] = x[c];
}

// Which kernel takes a base case of order n, by what each costs.  A thread per
// system takes its own chain's time (n = 64: ~280k cycles) for any number up to
// the threads that fit and the fewest instructions per system; a warp per system
// the shortest chain and the most; tri_asc32 lies between.  Measured crossings
// (us for n = 8, 16, 32, 64 and a number of systems; 'L' 'U' 'T' 'N' unless said):
//  - descending: a warp to 1064 systems (64 x 1000: 200 against 214), 608 for
//    n <= 8 (8 x 1000: 10.7 against 9.8);
//  - ascending, n > 32: a warp to 100 n systems where each unknown takes a
//    quotient, 155 n where it takes a product or nothing (64 x 4000: 140 against
//    207, 64 x 8000: 263 against 207; 'R' 144 to 193 against 250);
//  - ascending, n <= 32: a warp to 912 systems; a thread beyond for n <= 8 (8 x
//    100,000: 47 against 147); else tri_asc32, whose time grows with the systems
//    (32 x 8000: 41 to 43, 32 x 32,000: 143 to 147), or a thread each, whose time
//    grows by whole rounds of 128 on every SM (62 to 69, 120 to 126), by the
//    estimates below in us, which follow the measured ones within a tenth.
enum class Base { WARP, ASC32, THREAD };
Base descending_base(int64_t n, int64_t systems) {
  return systems <= (n <= 8 ? 608 : 1064) ? Base::WARP : Base::THREAD;
}
Base ascending_base(int64_t n, int64_t systems, bool right, bool unit) {
  if (n > 32) return systems <= (right || unit ? 155 : 100) * n ? Base::WARP : Base::THREAD;
  if (systems <= 912) return Base::WARP;
  if (n <= 8) return Base::THREAD;
  const double rounds = (double)cdiv(systems, 128 * (int64_t)num_sms()), size = (double)n;
  const bool less = unit && !right;  // neither a quotient nor a product per unknown, no zero tests
  const double thread = 5.0 + rounds * (less ? 0.047 : 0.056) * size * size;
  const double asc32 = 6.0 + 0.001 * (double)systems * (less ? 1.05 + 0.044 * size : 1.25 + 0.095 * size);
  return asc32 < thread ? Base::ASC32 : Base::THREAD;
}

struct Ctx {
  cudaStream_t s;
  bool unit;
  int lanes;
  const int32_t *info;
};

int base_left_n(const Ctx &c, bool lower, int64_t m, int64_t n, const double *A, int64_t lda, double *B,
                int64_t ldb) {
  ProfScope prof(c.s, "trsm_base", (double)m * m * n);
  const unsigned g = (unsigned)cdiv(n, LN_WARPS);
  BOLA_TRY(roomy(lower ? left_n_base<true> : left_n_base<false>));
  if (lower)
    BOLA_TRY_CUDA(launch_after(left_n_base<true>, dim3(g), 32 * LN_WARPS, 0, c.s, (int)m, n, c.unit, A, lda, B, ldb,
                               c.lanes, c.info));
  else
    BOLA_TRY_CUDA(launch_after(left_n_base<false>, dim3(g), 32 * LN_WARPS, 0, c.s, (int)m, n, c.unit, A, lda, B, ldb,
                               c.lanes, c.info));
  BOLA_CHECK_LAUNCH();
  return 0;
}

int base_left_t(const Ctx &c, bool lower, int64_t m, int64_t n, const double *A, int64_t lda, double *B,
                int64_t ldb) {
  ProfScope prof(c.s, "trsm_base", (double)m * m * n);
  const Base base = lower ? descending_base(m, n) : ascending_base(m, n, false, c.unit);
  if (base == Base::ASC32) {
    BOLA_TRY(roomy(tri_asc32<false>));
    BOLA_TRY_CUDA(launch_after(tri_asc32<false>, dim3((unsigned)cdiv(n, AS_SYS)), AS_THREADS, 0, c.s, (int)m, n,
                               c.unit, false, A, lda, B, 1, ldb, c.info));
    BOLA_CHECK_LAUNCH();
    return 0;
  }
  if (base == Base::WARP) {
    const unsigned gw = (unsigned)cdiv(n, TW_WARPS);
    BOLA_TRY(roomy(lower ? tri_warp<false, false> : tri_warp<true, false>));
    if (lower)
      BOLA_TRY_CUDA(launch_after(tri_warp<false, false>, dim3(gw), 32 * TW_WARPS, 0, c.s, (int)m, n, c.unit, false, A,
                                 lda, B, 1, ldb, c.info));
    else
      BOLA_TRY_CUDA(launch_after(tri_warp<true, false>, dim3(gw), 32 * TW_WARPS, 0, c.s, (int)m, n, c.unit, false, A,
                                 lda, B, 1, ldb, c.info));
    BOLA_CHECK_LAUNCH();
    return 0;
  }
  const unsigned g = (unsigned)cdiv(n, TCOLS);
  if (lower)
    BOLA_TRY_CUDA(launch_after(left_t_base<true>, dim3(g), TCOLS, 0, c.s, (int)m, n, c.unit, A, lda, B, ldb, c.info));
  else
    BOLA_TRY_CUDA(launch_after(left_t_base<false>, dim3(g), TCOLS, 0, c.s, (int)m, n, c.unit, A, lda, B, ldb, c.info));
  BOLA_CHECK_LAUNCH();
  return 0;
}

template <int V>
int launch_right_base(const Ctx &c, int64_t m, int64_t n, const double *A, int64_t lda, double *B, int64_t ldb) {
  constexpr bool asc = V == 1 || V == 2;
  const Base base = asc ? ascending_base(n, m, true, c.unit) : descending_base(n, m);
  if (base == Base::WARP) {
    BOLA_TRY(roomy(tri_warp<asc, true>));
    BOLA_TRY_CUDA(launch_after(tri_warp<asc, true>, dim3((unsigned)cdiv(m, TW_WARPS)), 32 * TW_WARPS, 0, c.s, (int)n,
                               m, c.unit, V >= 2, A, lda, B, ldb, 1, c.info));
    BOLA_CHECK_LAUNCH();
    return 0;
  }
  if constexpr (asc) {
    if (base == Base::ASC32) {
      BOLA_TRY(roomy(tri_asc32<true>));
      BOLA_TRY_CUDA(launch_after(tri_asc32<true>, dim3((unsigned)cdiv(m, AS_SYS)), AS_THREADS, 0, c.s, (int)n, m,
                                 c.unit, V >= 2, A, lda, B, ldb, 1, c.info));
      BOLA_CHECK_LAUNCH();
      return 0;
    }
  }
  const size_t smem = right_base_smem((int)n);
  // (always the largest order's, so that no thread lowers what another is about to launch with)
  if (smem > 48 * 1024)
    BOLA_TRY_CUDA(cudaFuncSetAttribute(right_base<V>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)right_base_smem(STOP)));
  BOLA_TRY(roomy(right_base<V>));
  BOLA_TRY_CUDA(launch_after(right_base<V>, dim3((unsigned)cdiv(m, RB_ROWS)), RB_ROWS, smem, c.s, m, (int)n, c.unit,
                             A, lda, B, ldb, c.info));
  BOLA_CHECK_LAUNCH();
  return 0;
}

int base_right(const Ctx &c, int v, int64_t m, int64_t n, const double *A, int64_t lda, double *B,
               int64_t ldb) {
  ProfScope prof(c.s, "trsm_base", (double)m * n * n);
  switch (v) {
    case 0: return launch_right_base<0>(c, m, n, A, lda, B, ldb);
    case 1: return launch_right_base<1>(c, m, n, A, lda, B, ldb);
    case 2: return launch_right_base<2>(c, m, n, A, lda, B, ldb);
    default: return launch_right_base<3>(c, m, n, A, lda, B, ldb);
  }
}

int gemm_upd(const Ctx &c, char ta, char tb, int64_t m, int64_t n, int64_t k, const double *A, int64_t lda,
             const double *B, int64_t ldb, double *C, int64_t ldc) {
  return dgemm_exact(c.s, ta, tb, m, n, k, -1.0, A, lda, B, ldb, 1.0, C, ldc, 64, c.info, 0);
}

// src/trsm.rs:95-131
int lnl(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (m <= STOP) return base_left_n(c, true, m, n, a, lda, b, ldb);
  const int64_t m1 = m / 2, m2 = m - m1;
  BOLA_TRY(lnl(c, m1, n, a, lda, b, ldb));
  BOLA_TRY(gemm_upd(c, 'N', 'N', m2, n, m1, a + m1, lda, b, ldb, b + m1, ldb));
  return lnl(c, m2, n, a + m1 + m1 * lda, lda, b + m1, ldb);
}
// src/trsm.rs:135-170
int lnu(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (m <= STOP) return base_left_n(c, false, m, n, a, lda, b, ldb);
  const int64_t m1 = m / 2, m2 = m - m1;
  BOLA_TRY(lnu(c, m2, n, a + m1 + m1 * lda, lda, b + m1, ldb));
  BOLA_TRY(gemm_upd(c, 'N', 'N', m1, n, m2, a + m1 * lda, lda, b + m1, ldb, b, ldb));
  return lnu(c, m1, n, a, lda, b, ldb);
}
// src/trsm.rs:174-209
int ltl(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (m <= STOP) return base_left_t(c, true, m, n, a, lda, b, ldb);
  const int64_t m1 = m / 2, m2 = m - m1;
  BOLA_TRY(ltl(c, m2, n, a + m1 + m1 * lda, lda, b + m1, ldb));
  BOLA_TRY(gemm_upd(c, 'T', 'N', m1, n, m2, a + m1, lda, b + m1, ldb, b, ldb));
  return ltl(c, m1, n, a, lda, b, ldb);
}
// src/trsm.rs:213-248
int ltu(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (m <= STOP) return base_left_t(c, false, m, n, a, lda, b, ldb);
  const int64_t m1 = m / 2, m2 = m - m1;
  BOLA_TRY(ltu(c, m1, n, a, lda, b, ldb));
  BOLA_TRY(gemm_upd(c, 'T', 'N', m2, n, m1, a + m1 * lda, lda, b, ldb, b + m1, ldb));
  return ltu(c, m2, n, a + m1 + m1 * lda, lda, b + m1, ldb);
}
// src/trsm.rs:252-280
int rnl(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (n <= STOP) return base_right(c, 0, m, n, a, lda, b, ldb);
  const int64_t n1 = n / 2, n2 = n - n1;
  BOLA_TRY(rnl(c, m, n2, a + n1 + n1 * lda, lda, b + n1 * ldb, ldb));
  BOLA_TRY(gemm_upd(c, 'N', 'N', m, n1, n2, b + n1 * ldb, ldb, a + n1, lda, b, ldb));
  return rnl(c, m, n1, a, lda, b, ldb);
}
// src/trsm.rs:284-312
int rnu(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (n <= STOP) return base_right(c, 1, m, n, a, lda, b, ldb);
  const int64_t n1 = n / 2, n2 = n - n1;
  BOLA_TRY(rnu(c, m, n1, a, lda, b, ldb));
  BOLA_TRY(gemm_upd(c, 'N', 'N', m, n2, n1, b, ldb, a + n1 * lda, lda, b + n1 * ldb, ldb));
  return rnu(c, m, n2, a + n1 + n1 * lda, lda, b + n1 * ldb, ldb);
}
// src/trsm.rs:316-344
int rtl(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (n <= STOP) return base_right(c, 2, m, n, a, lda, b, ldb);
  const int64_t n1 = n / 2, n2 = n - n1;
  BOLA_TRY(rtl(c, m, n1, a, lda, b, ldb));
  BOLA_TRY(gemm_upd(c, 'N', 'T', m, n2, n1, b, ldb, a + n1, lda, b + n1 * ldb, ldb));
  return rtl(c, m, n2, a + n1 + n1 * lda, lda, b + n1 * ldb, ldb);
}
// src/trsm.rs:348-376
int rtu(const Ctx &c, int64_t m, int64_t n, const double *a, int64_t lda, double *b, int64_t ldb) {
  if (n <= STOP) return base_right(c, 3, m, n, a, lda, b, ldb);
  const int64_t n1 = n / 2, n2 = n - n1;
  BOLA_TRY(rtu(c, m, n2, a + n1 + n1 * lda, lda, b + n1 * ldb, ldb));
  BOLA_TRY(gemm_upd(c, 'N', 'T', m, n1, n2, b + n1 * ldb, ldb, a + n1 * lda, lda, b, ldb));
  return rtu(c, m, n1, a, lda, b, ldb);
}

}  // namespace

// src/trsm.rs:33-91: alpha pre-scale, then dispatch (case-insensitive).
int trsm_exact(cudaStream_t s, char side, char uplo, char transa, char diag, int64_t m, int64_t n,
               double alpha, const double *A, int64_t lda, double *B, int64_t ldb, const int32_t *info) {
  if (m <= 0 || n <= 0) return 0;
  if (alpha != 1.0) {
    ProfScope prof(s, "scale", (double)m * n);
    BOLA_TRY_CUDA(launch_after(scale_matrix, dim3((unsigned)cdiv(m * n, 256)), 256, 0, s, m, n, alpha, B, ldb, info));
    BOLA_CHECK_LAUNCH();
  }
  Ctx c{s, upc(diag) == 'U', lanes(), info};
  const bool left = upc(side) == 'L', upper = upc(uplo) == 'U', notrans = upc(transa) == 'N';
  if (left) {
    if (notrans) return upper ? lnu(c, m, n, A, lda, B, ldb) : lnl(c, m, n, A, lda, B, ldb);
    return upper ? ltu(c, m, n, A, lda, B, ldb) : ltl(c, m, n, A, lda, B, ldb);
  }
  if (notrans) return upper ? rnu(c, m, n, A, lda, B, ldb) : rnl(c, m, n, A, lda, B, ldb);
  return upper ? rtu(c, m, n, A, lda, B, ldb) : rtl(c, m, n, A, lda, B, ldb);
}

}  // namespace bola

extern "C" int bola_dtrsm(char side, char uplo, char transa, char diag, int64_t m, int64_t n,
                          double alpha, const double *a, int64_t lda, double *b, int64_t ldb,
                          bola_stream_t stream) {
  if (m < 0) return -5;
  if (n < 0) return -6;
  if (m == 0 || n == 0) return 0;
  const int64_t k = bola::upc(side) == 'L' ? m : n;
  if (lda < bola::imax(1, k)) return -9;
  if (ldb < bola::imax(1, m)) return -11;
  return bola::trsm_exact((cudaStream_t)stream, side, uplo, transa, diag, m, n, alpha, a, lda, b, ldb,
                          nullptr);
}
