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

// The U diagonal of the LU form is L_kk^2 = the pivots: their running extent and the give-up test.
__device__ __forceinline__ void track_pivots(uint64_t *track, double umax, double umin, double give_up, int64_t done,
                                             int64_t n) {
  const uint64_t mx = (uint64_t)__double_as_longlong(umax), mn = (uint64_t)__double_as_longlong(umin);
  if (mx > track[0]) track[0] = mx;
  if (mn < track[1]) track[1] = mn;
  const double gmx = __longlong_as_double((long long)track[0]), gmn = __longlong_as_double((long long)track[1]);
  const double spread = gmn > 0.0 ? gmx / gmn : INFINITY;
  if (give_up_now(spread, give_up, done, n)) *(volatile int32_t *)(track + 2) = 1;
}

// The diagonal block W[0:jb, 0:jb] (lower) = L11 L11^T, one CTA.  A pivot
// that is not positive (or not finite) stops the factorisation: *info = its
// global 1-based column, and every later kernel of the factorisation returns
// at once.  Tracks max/min of L_kk^2 (the U diagonal of the LU form) and
// gives up as the LU panel does.
//
//
// FP32: a thread per row and group of eight columns, its eight values in
// registers throughout.  A group's two warps take its 8 x 8 block through
// shared memory, every thread factors it for itself (no exchange on the
// chain of square roots) while solving its own row against it, and the groups
// right of it then take the eight columns at once.  Bound by the chain of the
// 64 square roots and reciprocals.  Measured on one GB300, launches
// serialised: 18.5 us; 36 with one warp on the chain, a column at a time.
constexpr int CD_T = CNB * CNB / 8;
constexpr int XP = 12;  // pitch of a row of eight values: float4 reads by row meet no bank twice
__global__ void __launch_bounds__(CD_T)
chol_dblock32(float *W, int64_t ldw, int jb, int32_t col0, int64_t n, int32_t *info, uint64_t *track,
              double give_up) {
  __shared__ __align__(16) float D[8][8], X[2][CNB][XP];
  __shared__ float piv[CNB];
  __shared__ int stop;
  sm100::grid_dependency_wait();
  const int tid = threadIdx.x, i = tid & (CNB - 1), grp = tid / CNB;
  if (tid == 0) stop = factor_stopped(info, track) ? 1 : 0;
  float v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = i < jb && 8 * grp + c <= i ? W[i + (8 * grp + c) * ldw] : 0.f;
  __syncthreads();
  if (stop) return;
  const int ngroups = (jb + 7) / 8;
#pragma unroll 1
  for (int g = 0; g < ngroups; ++g) {
    const int kb = 8 * g, w = jb - kb < 8 ? jb - kb : 8;
    if (grp == g) {
      if (i / 8 == g) {
        *reinterpret_cast<float4 *>(&D[i & 7][0]) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(&D[i & 7][4]) = make_float4(v[4], v[5], v[6], v[7]);
      }
      __syncwarp();  // (the barrier counts a warp at its first arrival)
      asm volatile("bar.sync 1, %0;" ::"n"(CNB) : "memory");
      float d[8][8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c <= r; c += 4) {
          const float4 q = *reinterpret_cast<const float4 *>(&D[r][c]);
          d[r][c] = q.x;
          d[r][c + 1] = q.y;
          d[r][c + 2] = q.z;
          d[r][c + 3] = q.w;
        }
      bool ok = true;
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        if (p >= w || !ok) continue;  // (the same in every thread)
        const float dp = d[p][p];
        if (!positive(dp)) {
          ok = false;
          if (i == kb) {
            stop = 1;
            atomicCAS(info, 0, col0 + kb + p + 1);
          }
          continue;
        }
        if (i == kb) piv[kb + p] = dp;
        const float r = sqrtT(dp), inv = recipT(r);
        v[p] = i == kb + p ? r : v[p] * inv;
#pragma unroll
        for (int q = p + 1; q < 8; ++q) {
          d[q][p] *= inv;
          v[q] = fmaT(-v[p], d[q][p], v[q]);
        }
#pragma unroll
        for (int q = p + 1; q < 8; ++q)
#pragma unroll
          for (int t = p + 1; t <= q; ++t) d[q][t] = fmaT(-d[q][p], d[t][p], d[q][t]);
        if (i >= kb + p && i < jb) W[i + (kb + p) * ldw] = v[p];
      }
      float *x = X[g & 1][i];
      *reinterpret_cast<float4 *>(x) = make_float4(v[0], v[1], v[2], v[3]);
      *reinterpret_cast<float4 *>(x + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
    __syncthreads();
    if (stop) return;
    if (grp > g && (i | 31) >= 8 * grp) {  // (warps wholly above the diagonal have no part)
      const float4 xa = *reinterpret_cast<const float4 *>(X[g & 1][i]);
      const float4 xb = *reinterpret_cast<const float4 *>(X[g & 1][i] + 4);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4 ya = *reinterpret_cast<const float4 *>(X[g & 1][8 * grp + c]);
        const float4 yb = *reinterpret_cast<const float4 *>(X[g & 1][8 * grp + c] + 4);
        v[c] = fmaT(-xa.x, ya.x, v[c]);
        v[c] = fmaT(-xa.y, ya.y, v[c]);
        v[c] = fmaT(-xa.z, ya.z, v[c]);
        v[c] = fmaT(-xa.w, ya.w, v[c]);
        v[c] = fmaT(-xb.x, yb.x, v[c]);
        v[c] = fmaT(-xb.y, yb.y, v[c]);
        v[c] = fmaT(-xb.z, yb.z, v[c]);
        v[c] = fmaT(-xb.w, yb.w, v[c]);
      }
    }
  }
  if (tid < 32 && track != nullptr) {
    float mx = 0.f, mn = INFINITY;
    for (int k = tid; k < jb; k += 32) {
      mx = fmaxf(mx, piv[k]);
      mn = fminf(mn, piv[k]);
    }
    for (int off = 16; off > 0; off >>= 1) {
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, off));
    }
    if (tid == 0) track_pivots(track, mx, mn, give_up, col0 + jb, n);
  }
}

// FP64: bound by the chain of a column (square root, reciprocal, scale, the next
// column's update): one warp walks it, two rows per lane, while eight warps
// apply each finished column to the columns after the next one.
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
__global__ void __launch_bounds__(CH_T)
chol_dblock64(double *W, int64_t ldw, int jb, int32_t col0, int64_t n, int32_t *info, uint64_t *track, double give_up) {
  using T = double;
  __shared__ T a[CNB * CHP];
  __shared__ int stop;
  sm100::grid_dependency_wait();
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
        ch_sync(CH_UPDATED);  // (every update warp has read stop for column l - 1)
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
  if (tid == 0 && track != nullptr && !stop) track_pivots(track, umax, umin, give_up, col0 + jb, n);
}

// L21 = W21 L11^-T for the rows jb..mp-1 of the panel, written back to W and
// as row (row - jb) of the update's K-major operand.  A lane per row (32 rows
// per CTA), a warp per group of eight columns, its values in registers: the
// groups solve in turn against L11's diagonal 8 x 8 blocks and the ones right
// of them take the eight columns at once (a warp reads L11 by broadcast), so
// the chain is 64 multiplications and eight barriers.  Measured on one GB300
// with 1400 rows, launches serialised: FP32 7 us (21 with a thread per row),
// FP64 38 (95).
template <typename T>
struct alignas(16) Vec8 {
  T v[8];
};
constexpr int L21_R = 32;
constexpr int L21_T = 8 * L21_R;
template <typename T>
__host__ __device__ constexpr int l21_pitch() {  // of a row of eight values: 16-byte reads by row meet no bank twice
  return sizeof(T) == 4 ? 12 : 10;
}
template <typename T>
constexpr size_t l21_smem() {
  return sizeof(T) * (CNB * CNB + CNB + 2 * L21_R * l21_pitch<T>());
}
template <typename T>
__global__ void __launch_bounds__(L21_T)
chol_l21(T *W, int64_t ldw, int64_t mp, int jb, int kind, void *aop, float *aop_lo, int32_t *aexp, int64_t cap,
         const int32_t *info, const uint64_t *track) {
  extern __shared__ __align__(16) unsigned char l21_raw[];
  T *Lt = reinterpret_cast<T *>(l21_raw);  // L(k, q) at Lt[q * CNB + k]
  T *rd = Lt + CNB * CNB;
  T *X = rd + CNB;  // the group's columns of row r at X[(g & 1) L21_R * XPT + r * XPT]
  constexpr int XPT = l21_pitch<T>();
  __shared__ uint64_t mag[8][L21_R];
  __shared__ int stop;
  sm100::grid_dependency_wait();
  const int tid = threadIdx.x, r = tid & 31, grp = tid >> 5;
  if (tid == 0) stop = factor_stopped(info, track) ? 1 : 0;
  const int64_t row = jb + (int64_t)blockIdx.x * L21_R + r;
  T v[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) v[c] = 8 * grp + c < jb && row < mp ? W[row + (8 * grp + c) * ldw] : T(0);
#pragma unroll 8
  for (int e = tid; e < CNB * CNB; e += L21_T) {
    const int i = e % CNB, j = e / CNB;
    Lt[e] = (i < jb && j < jb && i >= j) ? W[i + j * ldw] : T(0);
  }
  __syncthreads();
  if (stop) return;
  if (tid < CNB) rd[tid] = tid < jb ? recipT(Lt[tid * (CNB + 1)]) : T(0);
  __syncthreads();
#pragma unroll 1
  for (int g = 0; g < 8; ++g) {
    T *x = X + ((g & 1) * L21_R + r) * XPT;
    if (grp == g) {
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const Vec8<T> l = *reinterpret_cast<const Vec8<T> *>(Lt + (8 * g + p) * CNB + 8 * g);
        v[p] *= rd[8 * g + p];  // zero beyond jb (rd = 0 there)
#pragma unroll
        for (int q = p + 1; q < 8; ++q) v[q] = fmaT(-v[p], l.v[q], v[q]);
      }
      Vec8<T> o;
#pragma unroll
      for (int p = 0; p < 8; ++p) o.v[p] = v[p];
      *reinterpret_cast<Vec8<T> *>(x) = o;
    }
    __syncthreads();
    if (grp > g) {
      const Vec8<T> xr = *reinterpret_cast<const Vec8<T> *>(x);
#pragma unroll
      for (int p = 0; p < 8; ++p) {
        const Vec8<T> l = *reinterpret_cast<const Vec8<T> *>(Lt + (8 * g + p) * CNB + 8 * grp);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = fmaT(-xr.v[p], l.v[q], v[q]);
      }
    }
  }
  if (row < mp)
#pragma unroll
    for (int c = 0; c < 8; ++c)
      if (8 * grp + c < jb) W[row + (8 * grp + c) * ldw] = v[c];
  if (aop == nullptr) return;
  if constexpr (sizeof(T) == 4) {
    if (row < mp) write_operand_part(kind, aop, aop_lo, row - jb, 8 * grp, v);
  } else {
    uint64_t m = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const uint64_t mc = oz_mag(v[c]);
      m = mc > m ? mc : m;
    }
    mag[grp][r] = m;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) m = mag[q][r] > m ? mag[q][r] : m;
    if (row < mp) {
      const int e = oz_exponent(m);
      if (grp == 0) aexp[row - jb] = e;
      write_slices_part(v, e, row - jb, 8 * grp, cap, static_cast<__nv_bfloat16 *>(aop));
    }
  }
}

// The diagonal of L, before chol_to_lu overwrites it.
template <typename T>
__global__ void chol_diag(int64_t n, const T *W, int64_t ldw, T *dg) {
  sm100::grid_dependency_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) dg[i] = W[i + i * ldw];
}

// LU form of a Cholesky factor: W[i,j] = L_ij / L_jj (i > j), W[i,j] = L_ii L_ji
// (i <= j).  One CTA per 32 x 32 tile (I, J) with I >= J: it reads its lower
// tile and writes the lower tile and the transposed upper tile (J, I), which
// no other CTA touches.
template <typename T>
__global__ void __launch_bounds__(256) chol_to_lu(int64_t n, T *W, int64_t ldw, const T *dg) {
  sm100::grid_dependency_wait();
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
      StepLaunch D(dim3(1), dim3(fp64 ? CH_T : CD_T), 0, lu.sp, true);
      if constexpr (fp64)
        BOLA_TRY_CUDA(cudaLaunchKernelEx(&D.cfg, chol_dblock64, Wp, ldw, jb, (int32_t)j, n, info, track, give_up));
      else
        BOLA_TRY_CUDA(cudaLaunchKernelEx(&D.cfg, chol_dblock32, Wp, ldw, jb, (int32_t)j, n, info, track, give_up));
      if (mp > jb) {
        StepLaunch L(dim3((unsigned)cdiv(mp - jb, L21_R)), dim3(L21_T), l21_smem<T>(), lu.sp, true);
        BOLA_TRY_CUDA(cudaLaunchKernelEx(&L.cfg, chol_l21<T>, Wp, ldw, mp, jb, lu.kind, upd ? lu.aop[buf] : nullptr,
                                         fp64 ? (float *)nullptr : lu.aop_lo[buf],
                                         fp64 ? lu.ea[buf] : (int32_t *)nullptr, lu.cap_n, (const int32_t *)info,
                                         (const uint64_t *)track));
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
                         W22 + boff * ldw, ldw, lu.err, boff, abort, true, st == lu.sp);
      else
        return tc_update(st, lu.kind, m2, cols, lu.mapA[buf], lu.mapA64[buf], lu.mapAlo[buf], lu.mapAlo64[buf],
                         W22 + boff * ldw, ldw, lu.err, boff, abort, true, st == lu.sp);
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
  BOLA_TRY_CUDA(launch_after(chol_diag<T>, dim3((unsigned)cdiv(n, 256)), 256, 0, s, n, W, ldw, dg));
  const unsigned nt = (unsigned)cdiv(n, 32);
  BOLA_TRY_CUDA(launch_after(chol_to_lu<T>, dim3(nt, nt), 256, 0, s, n, W, ldw, dg));
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
