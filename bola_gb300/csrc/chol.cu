// chol.cu — the low-precision Cholesky of the mixed-precision SPD solver (no
// BOLA counterpart; the FP64 answer it must reach is BOLA's potrf('L') +
// trsm solve, src/potrf.rs:101-181, src/potrf2.rs:25-80, src/trsm.rs:95-209).
//
// W = fl(D A D) (D: powers of two making the diagonal O(1)) is factored in
// place, W = L L^T, right-looking with 64-column panels, lower triangle only:
//   chol_dblock   the 64 x 64 diagonal block, in one CTA's shared memory;
//   chol_l21      L21 = W21 L11^-T, one thread per row (no pivoting, so no
//                 exchange between CTAs: the panel is a parallel solve), and
//                 the K-major operand of the update (bf16, tf32 hi/lo, or the
//                 exact bf16 slices of the FP64-accurate factor);
//   the update    W22 -= L21 L21^T on tcgen05 (tc_update / oz_update), only
//                 tiles reaching the diagonal or below it: A and B operands
//                 are the same L21 rows.
// Look-ahead as in the LU (slu.cu): the next panel's 64 columns are updated
// on the high-priority stream, the rest on the low-priority stream overlaps
// the next panel.  Afterwards chol_to_lu rewrites the factor in the LU form
// the refinement's triangular solves use: unit-lower L D^-1 below the
// diagonal, U = D L^T on and above it (D = diag(L)).
#include <cmath>

#include "common.cuh"
#include "mixed.cuh"
#include "sm100.cuh"

namespace bola {
namespace {

constexpr int CNB = 64;  // panel width = update depth

__device__ __forceinline__ float sqrtT(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrtT(double x) { return sqrt_rn(x); }
__device__ __forceinline__ float recipT(float x) { return 1.f / x; }
__device__ __forceinline__ double recipT(double x) { return recip_rn(x); }
__device__ __forceinline__ bool positive(float x) { return x > 0.f && x <= 3.4e38f; }
__device__ __forceinline__ bool positive(double x) { return x > 0.0 && x <= 1.7e308; }

__device__ __forceinline__ bool factor_stopped(const int32_t *info, const uint64_t *track) {
  return *(volatile const int32_t *)info != 0 || (track != nullptr && *(volatile const int32_t *)(track + 2) != 0);
}

// The diagonal block W[0:jb, 0:jb] (lower) = L11 L11^T, one CTA.  A pivot
// that is not positive (or not finite) stops the factorisation: *info = its
// global 1-based column, and every later kernel of the factorisation returns
// at once.  Tracks max/min of L_kk^2 (the U diagonal of the LU form) and
// gives up as the LU panel does.
//
// Bound by the chain of a column (square root, reciprocal, scale, the next
// column's update): one warp walks it, two rows per lane, while eight warps
// apply each finished column to the columns after the next one.  Measured on
// one GB300 with L21 of 1400 rows after it: @@D us a panel in FP32 (82 with
// three CTA barriers a column and a division per updated element's index).
constexpr int CH_UPD = 8;
constexpr int CH_T = 32 * (1 + CH_UPD);
constexpr int CHP = CNB + 1;  // pitch: column j of row i at a[j * CHP + i]
enum { CH_UPDATED = 1, CH_SCALED = 2 };
__device__ __forceinline__ void ch_sync(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(CH_T) : "memory");
}
__device__ __forceinline__ void ch_arrive(int id) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(CH_T) : "memory");
}
template <typename T>
__global__ void __launch_bounds__(CH_T)
chol_dblock(T *W, int64_t ldw, int jb, int32_t col0, int64_t n, int32_t *info, uint64_t *track, double give_up) {
  __shared__ T a[CNB * CHP];
  __shared__ int stop;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) stop = factor_stopped(info, track) ? 1 : 0;
  __syncthreads();
  if (stop) return;
  for (int e = tid; e < CNB * CNB; e += CH_T) {
    const int i = e % CNB, j = e / CNB;
    a[j * CHP + i] = (i < jb && j < jb && i >= j) ? W[i + j * ldw] : T(0);
  }
  __syncthreads();
  T umax = T(0), umin = T(INFINITY);
  if (warp == 0) {
    T c[2] = {a[lane], a[lane + 32]};
    for (int l = 0; l < jb; ++l) {
      const T d = __shfl_sync(0xffffffffu, l < 32 ? c[0] : c[1], l & 31);
      if (!positive(d)) {
        if (lane == 0) {
          stop = 1;
          atomicCAS(info, 0, col0 + l + 1);
        }
        ch_arrive(CH_SCALED);
        break;
      }
      const T r = sqrtT(d), inv = recipT(r);
      T x[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = lane + 32 * h;
        x[h] = i == l ? r : c[h] * inv;
        if (i >= l) a[l * CHP + i] = x[h];
      }
      umax = d > umax ? d : umax;
      umin = d < umin ? d : umin;
      ch_sync(CH_UPDATED);  // column l - 1 is applied everywhere
      const int nx = l + 1 < jb ? l + 1 : l;
      c[0] = a[nx * CHP + lane];
      c[1] = a[nx * CHP + lane + 32];
      ch_arrive(CH_SCALED);
      const T xj = __shfl_sync(0xffffffffu, nx < 32 ? x[0] : x[1], nx & 31);
      c[0] = fmaT(-x[0], xj, c[0]);
      c[1] = fmaT(-x[1], xj, c[1]);
    }
  } else {
    for (int l = 0; l < jb; ++l) {
      ch_arrive(CH_UPDATED);
      ch_sync(CH_SCALED);
      if (stop) break;
      const T *xl = a + l * CHP;
      const T x0 = xl[lane], x1 = xl[lane + 32];
      for (int j0 = l + 1 + warp; j0 < jb; j0 += 4 * CH_UPD) {
        T v[4], w[4], xj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * CH_UPD < jb ? j0 + u * CH_UPD : jb - 1;
          v[u] = a[j * CHP + lane];
          w[u] = a[j * CHP + lane + 32];
          xj[u] = xl[j];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * CH_UPD;
          if (j >= jb) break;
          if (j < 32) {
            const T t = fmaT(-x0, xj[u], v[u]);
            if (lane >= j) a[j * CHP + lane] = t;
          }
          const T t = fmaT(-x1, xj[u], w[u]);
          if (lane + 32 >= j) a[j * CHP + lane + 32] = t;
        }
      }
    }
  }
  __syncthreads();
  for (int e = tid; e < jb * jb; e += CH_T) {
    const int i = e % jb, j = e / jb;
    if (i >= j) W[i + j * ldw] = a[j * CHP + i];
  }
  if (tid == 0 && track != nullptr && !stop) {
    // the U diagonal of the LU form is L_kk^2 = the pivots: their running extent and the give-up test
    const uint64_t mx = (uint64_t)__double_as_longlong((double)umax), mn = (uint64_t)__double_as_longlong((double)umin);
    if (mx > track[0]) track[0] = mx;
    if (mn < track[1]) track[1] = mn;
    const double gmx = __longlong_as_double((long long)track[0]), gmn = __longlong_as_double((long long)track[1]);
    const double spread = gmn > 0.0 ? gmx / gmn : INFINITY;
    if (give_up_now(spread, give_up, col0 + jb, n)) *(volatile int32_t *)(track + 2) = 1;
  }
}

// L21 = W21 L11^-T for the rows jb..mp-1 of the panel (one thread per row),
// written back to W and as row (row - jb) of the update's K-major operand.
// Eight columns at a time: their eight sums, in registers, take the earlier
// columns in order from shared memory (one value of the row's and eight of
// L11's per step), then each other; so eight chains are in flight and the loop
// stays in the instruction cache, where 64 columns unrolled into one chain each
// did neither.
template <typename T>
struct alignas(16) Vec8 {
  T v[8];
};
constexpr int L21_T = 64;
template <typename T>
constexpr size_t l21_smem() {
  return sizeof(T) * (CNB * CNB + CNB + CNB * L21_T);
}
template <typename T>
__global__ void __launch_bounds__(L21_T)
chol_l21(T *W, int64_t ldw, int64_t mp, int jb, int kind, void *aop, float *aop_lo, int32_t *aexp, int64_t cap,
         const int32_t *info, const uint64_t *track) {
  extern __shared__ __align__(16) unsigned char l21_raw[];
  T *Lt = reinterpret_cast<T *>(l21_raw);  // L(k, q) at Lt[q * CNB + k]
  T *rd = Lt + CNB * CNB;
  T *vs = rd + CNB + threadIdx.x;  // this thread's value k at vs[k * L21_T]
  __shared__ int stop;
  if (threadIdx.x == 0) stop = factor_stopped(info, track) ? 1 : 0;
  __syncthreads();
  if (stop) return;
  for (int e = threadIdx.x; e < CNB * CNB; e += L21_T) {
    const int i = e % CNB, j = e / CNB;
    Lt[e] = (i < jb && j < jb && i >= j) ? W[i + j * ldw] : T(0);
  }
  const int64_t row = jb + (int64_t)blockIdx.x * L21_T + threadIdx.x;
#pragma unroll 16
  for (int k = 0; k < CNB; ++k) vs[k * L21_T] = k < jb && row < mp ? W[row + k * ldw] : T(0);
  __syncthreads();
  for (int k = threadIdx.x; k < CNB; k += L21_T) rd[k] = k < jb ? recipT(Lt[k * (CNB + 1)]) : T(0);
  __syncthreads();
  if (row >= mp) return;
#pragma unroll 1
  for (int kb = 0; kb < CNB; kb += 8) {
    T x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = vs[(kb + r) * L21_T];
#pragma unroll 4
    for (int q = 0; q < kb; ++q) {
      const T vq = vs[q * L21_T];
      const Vec8<T> l = *reinterpret_cast<const Vec8<T> *>(Lt + q * CNB + kb);
#pragma unroll
      for (int r = 0; r < 8; ++r) x[r] = fmaT(-vq, l.v[r], x[r]);
    }
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const Vec8<T> l = *reinterpret_cast<const Vec8<T> *>(Lt + (kb + p) * CNB + kb);
      x[p] *= rd[kb + p];  // zero beyond jb (rd = 0 there)
#pragma unroll
      for (int r = p + 1; r < 8; ++r) x[r] = fmaT(-x[p], l.v[r], x[r]);
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) vs[(kb + r) * L21_T] = x[r];
  }
  T v[CNB];
#pragma unroll
  for (int k = 0; k < CNB; ++k) {
    v[k] = vs[k * L21_T];
    if (k < jb) W[row + k * ldw] = v[k];
  }
  if (aop == nullptr) return;
  if constexpr (sizeof(T) == 4) {
    write_operand_row(kind, aop, aop_lo, row - jb, v);
  } else {
    write_slices_row(v, row - jb, cap, static_cast<__nv_bfloat16 *>(aop), aexp);
  }
}

// The diagonal of L, before chol_to_lu overwrites it.
template <typename T>
__global__ void chol_diag(int64_t n, const T *W, int64_t ldw, T *dg) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dg[i] = W[i + i * ldw];
}

// LU form of a Cholesky factor: W[i,j] = L_ij / L_jj (i > j), W[i,j] = L_ii L_ji
// (i <= j).  One CTA per 32 x 32 tile (I, J) with I >= J: it reads its lower
// tile and writes the lower tile and the transposed upper tile (J, I), which
// no other CTA touches.
template <typename T>
__global__ void __launch_bounds__(256) chol_to_lu(int64_t n, T *W, int64_t ldw, const T *dg) {
  __shared__ T t[32][33];
  const int64_t I = blockIdx.x, J = blockIdx.y;
  if (J > I) return;
  const int64_t i0 = I * 32, j0 = J * 32;
  for (int e = threadIdx.x; e < 32 * 32; e += 256) {
    const int r = e & 31, c = e >> 5;
    const int64_t i = i0 + r, j = j0 + c;
    t[r][c] = (i < n && j < n && i >= j) ? W[i + j * ldw] : T(0);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 32 * 32; e += 256) {
    const int r = e & 31, c = e >> 5;
    const int64_t i = i0 + r, j = j0 + c;
    if (i >= n || j >= n || i < j) continue;
    if (i > j) W[i + j * ldw] = t[r][c] / dg[j];
  }
  for (int e = threadIdx.x; e < 32 * 32; e += 256) {
    const int c = e & 31, r = e >> 5;  // upper element (j0 + c, i0 + r) = L_jj L_ij, walking rows fastest
    const int64_t i = i0 + r, j = j0 + c;
    if (i >= n || j >= n || i < j) continue;
    W[j + i * ldw] = dg[j] * t[r][c];
  }
}

__global__ void zero_info(int32_t *p) { *p = 0; }
__global__ void track_reset(uint64_t *t) {
  t[0] = 0;
  t[1] = 0x7ff0000000000000ull;
  t[2] = 0;
}

template <typename T>
int chol_lookahead(MixedLU &lu, cudaStream_t s, T *W, int64_t ldw, int32_t *info, double give_up) {
  constexpr bool fp64 = sizeof(T) == 8;
  const int64_t n = lu.n;
  BOLA_TRY_CUDA(cudaEventRecord(lu.ev_in, s));
  BOLA_TRY_CUDA(cudaStreamWaitEvent(lu.sp, lu.ev_in, 0));
  zero_info<<<1, 1, 0, lu.sp>>>(info);
  track_reset<<<1, 1, 0, lu.sp>>>(lu.track);
  BOLA_CHECK_LAUNCH();
  BOLA_TRY_CUDA(cudaEventRecord(lu.ev_in, lu.sp));
  BOLA_TRY_CUDA(cudaStreamWaitEvent(lu.su, lu.ev_in, 0));
  uint64_t *track = std::isinf(give_up) ? nullptr : lu.track;
  const int32_t *abort = track ? reinterpret_cast<const int32_t *>(track + 2) : nullptr;
  bool wide_pending = false;
  for (int64_t j = 0, k = 0; j < n; j += CNB, ++k) {
    const int jb = (int)imin(CNB, n - j);
    const int64_t mp = n - j;
    const bool upd = j + jb < n;
    const int buf = (int)(k & 1);
    T *Wp = W + j + j * ldw;
    {
      ProfScope prof(lu.sp, fp64 ? "chol_panel64" : "chol_panel", (double)mp * jb * jb / 2.0,
                     2.0 * sizeof(T) * (double)mp * jb, 2);
      chol_dblock<T><<<1, CH_T, 0, lu.sp>>>(Wp, ldw, jb, (int32_t)j, n, info, track, give_up);
      if (mp > jb) {
        if (l21_smem<T>() > 48 * 1024)
          BOLA_TRY_CUDA(cudaFuncSetAttribute(chol_l21<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)l21_smem<T>()));
        chol_l21<T><<<(unsigned)cdiv(mp - jb, L21_T), L21_T, l21_smem<T>(), lu.sp>>>(
            Wp, ldw, mp, jb, lu.kind, upd ? lu.aop[buf] : nullptr, fp64 ? nullptr : lu.aop_lo[buf],
            fp64 ? lu.ea[buf] : nullptr, lu.cap_n, info, track);
      }
      BOLA_CHECK_LAUNCH();
    }
    if (!upd) continue;
    // the update of step k writes columns the previous wide update also writes
    if (wide_pending) BOLA_TRY_CUDA(cudaStreamWaitEvent(lu.sp, lu.ev_wide, 0));
    wide_pending = false;
    const int64_t m2 = mp - jb, n2 = n - j - jb;
    const int64_t nb_next = imin(CNB, n2);
    T *W22 = W + (j + jb) + (j + jb) * ldw;
    auto update = [&](cudaStream_t st, int64_t cols, int64_t boff) -> int {
      if constexpr (fp64)
        return oz_update(st, m2, cols, lu.mapA[buf], lu.mapA64[buf], lu.cap_n, lu.cap_n, lu.ea[buf], lu.ea[buf],
                         W22 + boff * ldw, ldw, lu.err, boff, abort, true);
      else
        return tc_update(st, lu.kind, m2, cols, lu.mapA[buf], lu.mapA64[buf], lu.mapAlo[buf], lu.mapAlo64[buf],
                         W22 + boff * ldw, ldw, lu.err, boff, abort, true);
    };
    BOLA_TRY(update(lu.sp, nb_next, 0));  // the next panel's columns
    if (n2 > nb_next) {
      BOLA_TRY_CUDA(cudaEventRecord(lu.ev_sw, lu.sp));
      BOLA_TRY_CUDA(cudaStreamWaitEvent(lu.su, lu.ev_sw, 0));
      BOLA_TRY(update(lu.su, n2 - nb_next, nb_next));
      BOLA_TRY_CUDA(cudaEventRecord(lu.ev_wide, lu.su));
      wide_pending = true;
    }
  }
  if (wide_pending) BOLA_TRY_CUDA(cudaStreamWaitEvent(lu.sp, lu.ev_wide, 0));
  BOLA_TRY_CUDA(cudaEventRecord(lu.ev_done, lu.sp));
  BOLA_TRY_CUDA(cudaStreamWaitEvent(s, lu.ev_done, 0));
  return 0;
}

}  // namespace

int MixedLU::factor_chol(cudaStream_t s, float *W, int64_t ldw, int32_t *info, double give_up) {
  return chol_lookahead<float>(*this, s, W, ldw, info, give_up);
}

int MixedLU::factor_chol64(cudaStream_t s, double *W, int64_t ldw, int32_t *info, double give_up) {
  return chol_lookahead<double>(*this, s, W, ldw, info, give_up);
}

// The LU form of a finished Cholesky factor (see chol_to_lu); dg: n scratch elements.
template <typename T>
int chol_lu_form(cudaStream_t s, int64_t n, T *W, int64_t ldw, T *dg) {
  ProfScope prof(s, "chol_to_lu", 0.0, 3.0 * sizeof(T) * (double)n * n / 2.0, 2);
  chol_diag<T><<<(unsigned)cdiv(n, 256), 256, 0, s>>>(n, W, ldw, dg);
  const unsigned nt = (unsigned)cdiv(n, 32);
  chol_to_lu<T><<<dim3(nt, nt), 256, 0, s>>>(n, W, ldw, dg);
  BOLA_CHECK_LAUNCH();
  return 0;
}
template int chol_lu_form<float>(cudaStream_t, int64_t, float *, int64_t, float *);
template int chol_lu_form<double>(cudaStream_t, int64_t, double *, int64_t, double *);

}  // namespace bola

// The low-precision Cholesky alone, for tests and profiling: the lower
// triangle of W (n x n FP32, SPD) is replaced by L (W = L L^T); *info
// (device) = the first column whose pivot is not positive, or 0.  Synchronous.
extern "C" int bola_spotrf_mixed(int kind, int64_t n, float *w, int64_t ldw, int32_t *info, bola_stream_t stream) {
  using namespace bola;
  if (kind < 0 || kind > 2) return -1;
  if (n < 0 || n > 8192) return -2;
  if (ldw < imax(1, n)) return -4;
  if (n == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  MixedLU lu;
  int st = lu.reserve(n, kind, s);
  if (st == 0) st = lu.factor_chol(s, w, ldw, info);
  int32_t err = 0;
  if (st == 0 && lu.err) st = cudaMemcpyAsync(&err, lu.err, sizeof err, cudaMemcpyDeviceToHost, s) == cudaSuccess ? 0 : BOLA_ERR_CUDA;
  if (cudaStreamSynchronize(s) != cudaSuccess && st == 0) st = cuda_fail(cudaGetLastError(), "bola_spotrf_mixed");
  lu.destroy();
  if (st == 0 && err != 0) st = fail(BOLA_ERR_CUDA, "mixed Cholesky: a bounded wait expired (code %d)", err);
  return st;
}
