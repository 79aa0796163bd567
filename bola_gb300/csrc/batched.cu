// batched.cu — many small independent solves of uneven size in one persistent
// launch (no BOLA counterpart; each system's answer must match BOLA's FP64
// getrf/potrf + trsm solve within rounding).
//
// Plan (host, once per batch shape): systems are bucketed by order n; each
// bucket has a group size G (threads per system: 32, 64, 128 or 256, from the
// autotuned table) and work items of 256/G systems of that bucket, ordered by
// decreasing cost (largest first, for load balance).  Solve (device): a grid
// of persistent 256-thread CTAs pulls items from an atomic counter; the CTA
// splits into 256/G groups, each factoring one system in place in global
// memory (L2-resident: at most 512 KB per system) with partial pivoting (LU)
// or Cholesky in panels of 8 columns (a panel in registers, a row per thread;
// register-tiled trailing updates), and then solving its right-hand sides, 8
// rows at a time.  A group synchronises with its own named barrier, so a
// system's arithmetic never depends on which systems share its CTA: every
// result is the same alone and in any mix.
// FP64 throughout; all waits are barriers (no spin loops).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"

namespace bola {
namespace {

constexpr int BT = 256;         // threads per CTA
constexpr int MAXG = BT / 32;   // groups per CTA at most
constexpr int ITEM = 3 + MAXG;  // ints per work item: G, count, panel width, system ids
constexpr int NBUCKET = 8;
// upper n of each bucket (inclusive)
constexpr int BUCKET_N[NBUCKET] = {16, 32, 48, 64, 96, 128, 192, 1 << 30};

struct SystemDesc {
  int32_t n, nrhs, kind, lda, ldb, pad;
  double *a, *b;
};
static_assert(sizeof(SystemDesc) == sizeof(bola_system), "bola_system layout");

__device__ __forceinline__ void group_sync(int G, int g) {
  if (G == 32) {
    __syncwarp();
  } else if (G == BT) {
    __syncthreads();
  } else {
    __syncwarp();  // (the barrier counts a warp at its first arrival)
    asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(G) : "memory");
  }
}

// What the groups of a CTA share.  A group never has fewer threads than its
// system has rows, so a thread holds a row of the panel in registers, and the
// arrays are indexed by the CTA's warp or thread.
constexpr int PBMAX = 16;
struct Shared {
  double cand[2][MAXG][PBMAX + 1];  // a warp's pivot candidate: its row of the panel, 1 / its value
  double row[2][MAXG][PBMAX + 1];   // a group's row k, as above (Cholesky: column k's panel rows)
  uint4 key[2][MAXG];               // a warp's largest |value| (high word + 1, low word), its row
  int piv[MAXG][PBMAX];             // the panel's interchanges
  Divisor dv[BT];                   // a system's diagonal, to divide by
};

// ---- blocked factorisation pieces -------------------------------------------
// The factorisations below run in panels of PB columns: pivots inside the
// panel update only the panel's columns; the rest of the matrix then gets the
// whole panel at once (U12 by a small forward substitution, A22 by register
// tiles of TR x TC elements per thread), so each trailing element is loaded
// and stored once per panel instead of once per pivot.  Every element still
// receives fma(-l_ik, u_kj, a_ij) for k in increasing order, with the values
// the unblocked order gives it (row interchanges move whole rows, deferred
// updates included), so results are those of the unblocked algorithm, bit for
// bit.
// The panel width PB (8, 12 or 16 columns) is chosen per size bucket and
// travels with each work item; the register tile TR x TC (TC = 4, TR = 4 or
// 2) is chosen per plan, since it sets the kernel's register count.  Neither
// changes any element's sequence of operations.
constexpr int TC = 4;

// A[c0:n, c0:n] -= A[c0:n, k0:k0+kb] * A[k0:k0+kb, c0:n] (lower = false), or
// its lower triangle -= A[c0:n, k0:k0+kb] * A[c0:n, k0:k0+kb]^T (lower = true),
// with c0 = k0 + kb.
template <int TR>
__device__ void group_trailing(double *A, int lda, int n, int k0, int kb, bool lower, int t, int G) {
  const int c0 = k0 + kb, m2 = n - c0;
  if (m2 <= 0) return;
  const int tr = (m2 + TR - 1) / TR, tc = (m2 + TC - 1) / TC;
  // tile (ti, tj): the full tr x tc grid, or its lower triangle (ti >= tj) packed by columns
  int ti = t, tj = 0, dq = 0, dr = 0;
  if (lower) {
    while (ti >= tr && tj < tr) {
      ti -= tr - tj - 1;
      ++tj;
    }
  } else {
    dq = G / tr;
    dr = G % tr;
    ti = t % tr;
    tj = t / tr;
  }
  const int ntiles = lower ? tr * (tr + 1) / 2 : tr * tc;
  for (int e = t; e < ntiles; e += G) {
    const int i0 = c0 + ti * TR, j0 = c0 + tj * TC;
    const int nr = n - i0, nc = n - j0;  // rows and columns left: the tile's own where they reach TR and TC
    double *pc = A + i0 + (int64_t)j0 * lda;
    double acc[TR][TC];
#pragma unroll
    for (int c = 0; c < TC; ++c)
#pragma unroll
      for (int r = 0; r < TR; ++r) acc[r][c] = (r < nr && c < nc) ? pc[r + (int64_t)c * lda] : 0.0;
    const double *pl = A + i0 + (int64_t)k0 * lda;
    const double *pu = lower ? A + j0 + (int64_t)k0 * lda : A + k0 + (int64_t)j0 * lda;
    const int64_t su = lower ? 1 : lda, step = lower ? lda : 1;
#pragma unroll 1
    for (int q = 0; q < kb; ++q) {
      double l[TR], u[TC];
#pragma unroll
      for (int r = 0; r < TR; ++r) l[r] = r < nr ? pl[r] : 0.0;
#pragma unroll
      for (int c = 0; c < TC; ++c) u[c] = c < nc ? pu[c * su] : 0.0;
      pl += lda;
      pu += step;
#pragma unroll
      for (int r = 0; r < TR; ++r)
#pragma unroll
        for (int c = 0; c < TC; ++c) acc[r][c] = fma(-l[r], u[c], acc[r][c]);
    }
#pragma unroll
    for (int c = 0; c < TC; ++c)
#pragma unroll
      for (int r = 0; r < TR; ++r)
        if (r < nr && c < nc && (!lower || i0 + r >= j0 + c)) pc[r + (int64_t)c * lda] = acc[r][c];
    if (lower) {
      ti += G;
      while (ti >= tr && tj < tr) {
        ti -= tr - tj - 1;
        ++tj;
      }
    } else {
      ti += dr;
      tj += dq;
      if (ti >= tr) {
        ti -= tr;
        ++tj;
      }
    }
  }
}

// At the top of a loop that rarely runs twice: its invariant loads are not kept
// in registers across the iterations (whole blocks of L would be).
__device__ __forceinline__ void reload() { asm volatile("" ::: "memory"); }

// The first `done` interchanges of the panel of kb columns on all columns and
// on the right-hand sides, a column per thread.  A column of the panel came out
// of the registers with those up to its own (all of them from column `done` on,
// where the panel stopped) and takes the ones after it.
__device__ __forceinline__ void group_swaps(const SystemDesc &S, int k0, int kb, int done, const int *piv, int t,
                                            int G) {
  for (int j = t; j < S.n + S.nrhs; j += G) {
    double *col = j < S.n ? S.a + (int64_t)j * S.lda : S.b + (int64_t)(j - S.n) * S.ldb;
#pragma unroll 1
    for (int r = j >= k0 && j < k0 + kb ? j - k0 + 1 : 0; r < done; ++r) {
      const int p = piv[r];
      if (p == k0 + r) continue;
      const double x = col[p];
      col[p] = col[k0 + r];
      col[k0 + r] = x;
    }
  }
}

// U12 = L11^-1 A12 for the panel rows k0..k0+kb-1 (unit lower L11), a column
// per thread: row r takes fma(-l_rq, u_q, u_r) for q < r in increasing q.
template <int PB>
__device__ __forceinline__ void group_u12(double *A, int lda, int n, int k0, int kb, int t, int G) {
  for (int j = k0 + kb + t; j < n; j += G) {
    reload();
    double u[PB];
#pragma unroll
    for (int r = 0; r < PB; ++r) u[r] = r < kb ? A[(k0 + r) + (int64_t)j * lda] : 0.0;
#pragma unroll
    for (int q = 0; q < PB - 1; ++q)
#pragma unroll
      for (int r = q + 1; r < PB; ++r)
        if (r < kb) u[r] = fma(-A[(k0 + r) + (int64_t)(k0 + q) * lda], u[q], u[r]);
#pragma unroll
    for (int r = 1; r < PB; ++r)
      if (r < kb) A[(k0 + r) + (int64_t)j * lda] = u[r];
  }
}

// Triangular solve of the right-hand sides in blocks of SB rows: a block's own
// triangle by a thread per right-hand side, then the rows still open take its
// SB values at once, an element per thread.  Every element receives its
// fma(-a_ik, x_k, b_i) in the order of the unblocked solve.  UP: from the last
// row; DIV: by the diagonal (dv); TRANS: element (i, k) of the triangle is A[k, i].
constexpr int SB = 8;
template <bool UP, bool DIV, bool TRANS>
__device__ __forceinline__ void group_trsv(const SystemDesc &S, const Divisor *dv, int t, int G, int g) {
  const int n = S.n, nr = S.nrhs;
  const int64_t lda = S.lda, ldb = S.ldb, sr = TRANS ? lda : 1, sc = TRANS ? 1 : lda;
  const double *A = S.a;
  double *B = S.b;
  const int nblk = (n + SB - 1) / SB;
  for (int s = 0; s < nblk; ++s) {
    const int k0 = SB * (UP ? nblk - 1 - s : s), kb = n - k0 < SB ? n - k0 : SB;
    for (int c = t; c < nr; c += G) {
      reload();
      double *x = B + k0 + c * ldb;
      double b[SB];  // the rows in the order of the solve, the current one in slot 0
      const int q0 = UP ? kb - 1 : 0, dir = UP ? -1 : 1;
#pragma unroll
      for (int z = 0; z < SB; ++z) b[z] = z < kb ? x[q0 + dir * z] : 0.0;
#pragma unroll 1
      for (int z = 0; z < kb; ++z) {
        const int q = k0 + q0 + dir * z;
        const double y = DIV ? div_rn(b[0], dv[q]) : b[0];
        x[q - k0] = y;
#pragma unroll
        for (int r = 1; r < SB; ++r) {
          if (z + r >= kb) break;
          b[r - 1] = fma(-A[(q + dir * r) * sr + q * sc], y, b[r]);
        }
      }
    }
    group_sync(G, g);
    const int i0 = UP ? 0 : k0 + kb, m = UP ? k0 : n - i0;
    if (m > 0) {
      const int dq = G / m, dr = G % m;
      int i = t % m, c = t / m;
      for (int e = t; e < m * nr; e += G) {
        reload();
        const double *x = B + k0 + c * ldb, *a = A + (i0 + i) * sr + k0 * sc;
        double acc = B[(i0 + i) + c * ldb];
#pragma unroll
        for (int z = 0; z < SB; ++z) {
          const int q = UP ? SB - 1 - z : z;
          if (q < kb) acc = fma(-a[q * sc], x[q], acc);
        }
        B[(i0 + i) + c * ldb] = acc;
        i += dr;
        c += dq;
        if (i >= m) {
          i -= m;
          ++c;
        }
      }
    }
    group_sync(G, g);
  }
}

// LU with partial pivoting of one system by a group, then L y = P b and U x = y.
// A panel stays in registers, a row per thread: per column one barrier, before
// which every warp leaves its candidate's row (largest |value|, ties to the
// lowest row, NaN never; compared on the integer pipe) and row k is left for
// the candidate's place.
template <int PB, int TR>
__device__ int group_lu_solve(const SystemDesc &S, int t, int G, int g, Shared &sh) {
  const unsigned FULL = 0xffffffffu;
  const int n = S.n, lda = S.lda, nw = G >> 5, w0 = g * nw, warp = w0 + (t >> 5);
  double *A = S.a;
  int info = 0;
  for (int k0 = 0; k0 < n && info == 0; k0 += PB) {
    const int kb = n - k0 < PB ? n - k0 : PB;
    const bool in = t >= k0 && t < n;
    double v[PB];  // this row's columns, the current one in slot 0
#pragma unroll
    for (int c = 0; c < PB; ++c) v[c] = c < kb && in ? A[t + (int64_t)(k0 + c) * lda] : 0.0;
    int done = kb;
#pragma unroll 1
    for (int c = 0; c < kb; ++c) {
      const int k = k0 + c, par = c & 1;
      const uint32_t hi = (uint32_t)__double2hiint(v[0]) & 0x7fffffffu, lo = (uint32_t)__double2loint(v[0]);
      const bool valid = t >= k && t < n && (hi < 0x7ff00000u || (hi == 0x7ff00000u && lo == 0));
      const uint32_t kh = valid ? hi + 1u : 0u;
      const double inv_own = recip_rn(valid ? v[0] : 1.5);  // (beside the search; 1.5: no special case)
      const uint32_t mh = __reduce_max_sync(FULL, kh);
      const uint32_t ml = __reduce_max_sync(FULL, kh == mh ? lo : 0u);
      const unsigned b = __ballot_sync(FULL, kh == mh && lo == ml);
      const bool first = (t & 31) == __ffs(b) - 1;
      if (first) sh.key[par][warp] = make_uint4(mh, ml, (uint32_t)t, 0u);
      if (first || t == k) {
#pragma unroll 1
        for (int two = 0; two < 2; ++two) {
          if (two ? t != k : !first) continue;
          double *o = two ? sh.row[par][g] : sh.cand[par][warp];
#pragma unroll
          for (int q = 0; q < PB; ++q) o[q] = v[q];
          o[PBMAX] = inv_own;
        }
      }
      group_sync(G, g);
      uint4 best = sh.key[par][w0];
      int bw = w0;
      for (int q = 1; q < nw; ++q) {
        const uint4 o = sh.key[par][w0 + q];
        if (o.x > best.x || (o.x == best.x && o.y > best.y)) {
          best = o;
          bw = w0 + q;
        }
      }
      const double *kr = sh.row[par][g], *pr = best.x != 0u ? sh.cand[par][bw] : kr;
      const int p = best.x != 0u ? (int)best.z : k;
      if (!nonzero64(pr[0])) {
        info = k + 1;
        done = c;
        // this column and the panel's others as they stand
#pragma unroll
        for (int q = 0; q < PB; ++q)
          if (c + q < kb && in) A[t + (int64_t)(k + q) * lda] = v[q];
        break;
      }
      if (t == 0) sh.piv[g][c] = p;
      if (p != k && (t == p || t == k)) {
        const double *o = t == p ? kr : pr;
#pragma unroll
        for (int q = 0; q < PB; ++q) v[q] = o[q];
      }
      const double l = t > k ? v[0] * pr[PBMAX] : v[0];
      if (in) A[t + (int64_t)k * lda] = l;
#pragma unroll
      for (int q = 1; q < PB; ++q) {
        if (c + q >= kb) break;
        v[q - 1] = t > k ? fma(-l, pr[q], v[q]) : v[q];
      }
    }
    group_sync(G, g);
    // (a zero pivot ends the factorisation with the interchanges found so far)
    group_swaps(S, k0, kb, done, sh.piv[g], t, G);
    group_sync(G, g);
    if (info == 0 && k0 + kb < n) {
      group_u12<PB>(A, lda, n, k0, kb, t, G);
      group_sync(G, g);
      group_trailing<TR>(A, lda, n, k0, kb, false, t, G);
      group_sync(G, g);
    }
  }
  if (info) return info;
  Divisor *dv = sh.dv + g * G;
  if (t < n) dv[t] = divisor(A[t + (int64_t)t * lda]);
  group_sync(G, g);
  group_trsv<false, false, false>(S, dv, t, G, g);  // unit lower
  group_trsv<true, true, false>(S, dv, t, G, g);    // upper
  return 0;
}

// Cholesky A = L L^T (lower) of one system by a group, then L y = b, L^T x = y.
// The panel as above; per column one barrier for the pivot's reciprocal root,
// one for the panel's rows of the scaled column.
template <int PB, int TR>
__device__ int group_chol_solve(const SystemDesc &S, int t, int G, int g, Shared &sh) {
  const int n = S.n, lda = S.lda;
  double *A = S.a;
  int info = 0;
  for (int k0 = 0; k0 < n && info == 0; k0 += PB) {
    const int kb = n - k0 < PB ? n - k0 : PB;
    double v[PB];  // this row's columns, the current one in slot 0
#pragma unroll
    for (int c = 0; c < PB; ++c) v[c] = c < kb && t >= k0 + c && t < n ? A[t + (int64_t)(k0 + c) * lda] : 0.0;
#pragma unroll 1
    for (int c = 0; c < kb; ++c) {
      const int k = k0 + c;
      double *x = sh.row[c & 1][g];
      if (t == k) {
        // d > 0 (NaN excluded) on the bits
        const long long db = __double_as_longlong(v[0]);
        const bool pos = db > 0 && db <= 0x7ff0000000000000ll;
        if (pos) {
          v[0] = sqrt_rn(v[0]);
          A[k + (int64_t)k * lda] = v[0];
          x[PBMAX] = recip_rn(v[0]);
        }
        sh.piv[g][c] = pos;
      }
      group_sync(G, g);
      if (!sh.piv[g][c]) {
        info = k + 1;
        // this column and the panel's others as they stand
#pragma unroll
        for (int q = 0; q < PB; ++q)
          if (c + q < kb && t >= k + q && t < n) A[t + (int64_t)(k + q) * lda] = v[q];
        break;
      }
      const bool below = t > k && t < n;
      if (below) {
        v[0] *= x[PBMAX];
        A[t + (int64_t)k * lda] = v[0];
        if (t < k0 + kb) x[t - k0] = v[0];
      }
      group_sync(G, g);
      if (below) {
        const double l = v[0];
#pragma unroll
        for (int q = 1; q < PB; ++q) {
          if (c + q >= kb) break;
          v[q - 1] = fma(-l, x[c + q], v[q]);
        }
      }
    }
    group_sync(G, g);
    if (info == 0 && k0 + kb < n) {
      group_trailing<TR>(A, lda, n, k0, kb, true, t, G);
      group_sync(G, g);
    }
  }
  if (info) return info;
  Divisor *dv = sh.dv + g * G;
  if (t < n) dv[t] = divisor(A[t + (int64_t)t * lda]);
  group_sync(G, g);
  group_trsv<false, true, false>(S, dv, t, G, g);  // L y = b
  group_trsv<true, true, true>(S, dv, t, G, g);    // L^T x = y
  return 0;
}

template <int PB, int TR>
__device__ int group_solve(const SystemDesc &S, int t, int G, int g, Shared &sh) {
  return S.kind == 1 ? group_chol_solve<PB, TR>(S, t, G, g, sh) : group_lu_solve<PB, TR>(S, t, G, g, sh);
}

// Bound by FP64 issue (88% of it, 4000 systems of order 8 to 256) once enough groups share
// an SM: CTAS CTAs (batch_ctas), rather than the two that the registers of the
// trailing update's tile would leave, a few values spilled.  Measured on one
// GB300, half LU and half Cholesky: 20,000 systems of order 8 to 256 48.4 ms
// (64.1 with two CTAs and the panel's columns one after the other through global
// memory, 48.8 with its groups tuned); 4000 of order 8 to 64 0.50 ms (0.62).
template <int TR, int CTAS>
__global__ void __launch_bounds__(BT, CTAS)
batched_solve_kernel(const SystemDesc *__restrict__ sys, const int32_t *__restrict__ items, int32_t nitems,
                     int32_t *counter, int32_t *info) {
  __shared__ int32_t cur[ITEM];
  __shared__ __align__(16) Shared sh;
  const int tid = threadIdx.x;
  for (;;) {
    if (tid == 0) {
      const int it = atomicAdd(counter, 1);
      cur[0] = it < nitems ? items[(int64_t)it * ITEM] : 0;
      for (int q = 1; q < ITEM; ++q) cur[q] = it < nitems ? items[(int64_t)it * ITEM + q] : 0;
    }
    __syncthreads();
    const int G = cur[0];
    if (G == 0) break;
    const int g = tid / G, t = tid % G;
    if (g < cur[1]) {
      const int id = cur[3 + g];
      const SystemDesc S = sys[id];
      const int pb = cur[2];
      const int r = pb == 16   ? group_solve<16, TR>(S, t, G, g, sh)
                    : pb == 12 ? group_solve<12, TR>(S, t, G, g, sh)
                               : group_solve<8, TR>(S, t, G, g, sh);
      if (t == 0) info[id] = r;
    }
    __syncthreads();
  }
}

struct Plan {
  int32_t count = 0, nitems = 0;
  int32_t *items = nullptr;    // device
  int32_t *counter = nullptr;  // device
  int grid = 0;
  double flops = 0.0;
  int group[NBUCKET];
  int tile = 4;  // register tile rows of the kernel (4 or 2)
  int ctas = 3;  // per SM (batch_ctas)
  cudaGraphExec_t exec = nullptr;
  const void *g_sys = nullptr;
  const void *g_info = nullptr;
};

int bucket_of(int n) {
  int b = 0;
  while (n > BUCKET_N[b]) ++b;
  return b;
}

}  // namespace

// Work items of a batch: per size bucket, systems by decreasing n, BT/G
// systems per item; items by decreasing cost.  flat holds ITEM int32 per item.
int batch_items(int32_t count, const int32_t *n, const int32_t *kind, const int32_t *group_size,
                std::vector<int32_t> &flat, int32_t *nitems, int *group, double *flops, const int32_t *panel_width) {
  static const int kDefault[NBUCKET] = {32, 32, 64, 64, 128, 128, 256, 256};
  int pbw[NBUCKET];
  for (int b = 0; b < NBUCKET; ++b) {
    int gsz = group_size ? group_size[b] : kDefault[b];
    if (gsz != 32 && gsz != 64 && gsz != 128 && gsz != 256) gsz = kDefault[b];
    gsz = std::max(gsz, kDefault[b]);  // a thread per row at least
    group[b] = gsz;
    const int pw = panel_width ? panel_width[b] : 8;
    pbw[b] = (pw == 12 || pw == 16) ? pw : 8;
  }
  double fl = 0.0;
  std::vector<std::vector<int>> byb(NBUCKET);
  for (int i = 0; i < count; ++i) {
    if (n[i] < 1 || n[i] > 256)
      return fail(-2, "bola_batch_plan_create: system %d has n = %d (supported 1..256)", i, n[i]);
    byb[bucket_of(n[i])].push_back(i);
    const double nn = n[i];
    fl += (kind && kind[i] == 1) ? nn * nn * nn / 3.0 : 2.0 * nn * nn * nn / 3.0;
  }
  struct It {
    double cost;
    std::vector<int32_t> v;
  };
  std::vector<It> its;
  for (int b = 0; b < NBUCKET; ++b) {
    auto &ids = byb[b];
    std::sort(ids.begin(), ids.end(), [&](int x, int y) { return n[x] > n[y] || (n[x] == n[y] && x < y); });
    const int G = group[b], per = BT / G;
    for (size_t s = 0; s < ids.size(); s += per) {
      It it;
      it.v.assign(ITEM, 0);
      it.v[0] = G;
      it.v[2] = pbw[b];
      int c = 0;
      double cost = 0.0;
      for (size_t q = s; q < ids.size() && c < per; ++q, ++c) {
        it.v[3 + c] = ids[q];
        cost = std::max(cost, (double)n[ids[q]] * n[ids[q]] * n[ids[q]] / G);
      }
      it.v[1] = c;
      it.cost = cost;
      its.push_back(std::move(it));
    }
  }
  std::stable_sort(its.begin(), its.end(), [](const It &x, const It &y) { return x.cost > y.cost; });
  flat.assign(its.size() * ITEM, 0);
  for (size_t i = 0; i < its.size(); ++i) std::memcpy(&flat[i * ITEM], its[i].v.data(), sizeof(int32_t) * ITEM);
  if (flops) *flops = fl;
  if (nitems) *nitems = (int32_t)its.size();
  return 0;
}

// CTAs per SM: four where most of the flops are in systems of order above 128
// (their barriers and chains need the company), three below, where the values
// that a fourth CTA spills cost more (3 | 4: 20,000 of order 8 to 256 50.1 |
// 48.4 ms, 2000 of order 129 to 256 9.4 | 9.1, 4000 of order 8 to 128 1.87 |
// 2.01, of order 8 to 64 0.50 | 0.65).
int batch_ctas(int32_t count, const int32_t *n, const int32_t *kind) {
  double all = 0.0, large = 0.0;
  for (int i = 0; i < count; ++i) {
    const double f = (double)n[i] * n[i] * n[i] * (kind && kind[i] == 1 ? 1.0 : 2.0);
    all += f;
    if (n[i] > 128) large += f;
  }
  return 2.0 * large > all ? 4 : 3;
}

using BatchKernel = void (*)(const SystemDesc *, const int32_t *, int32_t, int32_t *, int32_t *);
BatchKernel batch_kernel(int tile, int ctas) {
  if (tile == 2) return ctas == 4 ? batched_solve_kernel<2, 4> : batched_solve_kernel<2, 3>;
  return ctas == 4 ? batched_solve_kernel<4, 4> : batched_solve_kernel<4, 3>;
}

int batch_grid(int32_t nitems, int tile, int ctas) {
  int occ = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, batch_kernel(tile, ctas), BT, 0);
  return std::max(1, std::min((int)nitems, num_sms() * std::max(occ, 1)));
}

void launch_kernel(cudaStream_t s, int tile, int ctas, int grid, const bola_system *systems, const int32_t *items,
                   int32_t nitems, int32_t *counter, int32_t *info) {
  batch_kernel(tile, ctas)<<<grid, BT, 0, s>>>(reinterpret_cast<const SystemDesc *>(systems), items, nitems, counter,
                                               info);
}

// One persistent launch over nitems work items (device array); *counter is
// the work queue's head and is reset here.
int batch_launch(cudaStream_t s, const bola_system *systems, const int32_t *items, int32_t nitems, int32_t *counter,
                 int32_t *info, int tile, int ctas) {
  if (nitems == 0) return 0;
  BOLA_TRY_CUDA(cudaMemsetAsync(counter, 0, sizeof(int32_t), s));
  launch_kernel(s, tile, ctas, batch_grid(nitems, tile, ctas), systems, items, nitems, counter, info);
  BOLA_CHECK_LAUNCH();
  return 0;
}

}  // namespace bola

using namespace bola;

extern "C" {

int bola_batch_plan_create_tuned(int32_t count, const int32_t *n, const int32_t *kind,
                                 const bola_batch_tuning *tuning, bola_batch_plan *plan_out) {
  if (count < 0) return -1;
  if (!plan_out) return -5;
  if (tuning && tuning->tile_rows != 0 && tuning->tile_rows != 2 && tuning->tile_rows != 4) return -4;
  Plan *P = new Plan();
  P->count = count;
  P->tile = (tuning && tuning->tile_rows == 2) ? 2 : 4;
  std::vector<int32_t> flat;
  const int st = batch_items(count, n, kind, tuning ? tuning->group_size : nullptr, flat, &P->nitems, P->group,
                             &P->flops, tuning ? tuning->panel_width : nullptr);
  if (st != 0) {
    delete P;
    return st;
  }
  if (cudaMalloc(&P->items, sizeof(int32_t) * std::max<size_t>(flat.size(), 1)) != cudaSuccess ||
      cudaMalloc(&P->counter, sizeof(int32_t)) != cudaSuccess) {
    delete P;
    return fail(BOLA_ERR_CUDA, "bola_batch_plan_create: device allocation failed");
  }
  if (!flat.empty()) cudaMemcpy(P->items, flat.data(), sizeof(int32_t) * flat.size(), cudaMemcpyHostToDevice);
  P->ctas = batch_ctas(count, n, kind);
  P->grid = batch_grid(P->nitems, P->tile, P->ctas);
  *plan_out = reinterpret_cast<bola_batch_plan>(P);
  return 0;
}

int bola_batch_plan_create(int32_t count, const int32_t *n, const int32_t *kind, const int32_t *group_size,
                           bola_batch_plan *plan_out) {
  bola_batch_tuning t;
  std::memset(&t, 0, sizeof t);
  if (group_size) std::memcpy(t.group_size, group_size, sizeof t.group_size);
  return bola_batch_plan_create_tuned(count, n, kind, &t, plan_out);
}

int bola_batch_solve(bola_batch_plan plan, const bola_system *systems, int32_t *info, bola_stream_t stream) {
  Plan *P = reinterpret_cast<Plan *>(plan);
  if (!P) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  if (P->nitems == 0) return 0;
  ProfScope prof(s, "batched_solve", P->flops, 0.0, 2);
  BOLA_TRY_CUDA(cudaMemsetAsync(P->counter, 0, sizeof(int32_t), s));
  launch_kernel(s, P->tile, P->ctas, P->grid, systems, P->items, P->nitems, P->counter, info);
  BOLA_CHECK_LAUNCH();
  return 0;
}

int bola_batch_solve_graph(bola_batch_plan plan, const bola_system *systems, int32_t *info, bola_stream_t stream) {
  Plan *P = reinterpret_cast<Plan *>(plan);
  if (!P) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  if (P->nitems == 0) return 0;
  if (P->exec && (P->g_sys != systems || P->g_info != info)) {
    cudaGraphExecDestroy(P->exec);
    P->exec = nullptr;
  }
  if (!P->exec) {
    cudaStream_t cap;
    BOLA_TRY_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    cudaGraph_t g;
    BOLA_TRY_CUDA(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(P->counter, 0, sizeof(int32_t), cap);
    launch_kernel(cap, P->tile, P->ctas, P->grid, systems, P->items, P->nitems, P->counter, info);
    BOLA_TRY_CUDA(cudaStreamEndCapture(cap, &g));
    BOLA_TRY_CUDA(cudaGraphInstantiate(&P->exec, g, 0));
    cudaGraphDestroy(g);
    cudaStreamDestroy(cap);
    P->g_sys = systems;
    P->g_info = info;
  }
  ProfScope prof(s, "batched_solve", P->flops, 0.0, 2);
  BOLA_TRY_CUDA(cudaGraphLaunch(P->exec, s));
  return 0;
}

int bola_batch_plan_info(bola_batch_plan plan, int32_t *nitems, int32_t *grid, double *flops) {
  Plan *P = reinterpret_cast<Plan *>(plan);
  if (!P) return -1;
  if (nitems) *nitems = P->nitems;
  if (grid) *grid = P->grid;
  if (flops) *flops = P->flops;
  return 0;
}

int bola_batch_plan_destroy(bola_batch_plan plan) {
  Plan *P = reinterpret_cast<Plan *>(plan);
  if (!P) return 0;
  if (P->exec) cudaGraphExecDestroy(P->exec);
  if (P->items) cudaFree(P->items);
  if (P->counter) cudaFree(P->counter);
  delete P;
  return 0;
}

}  // extern "C"

// ---- the tuning table on disk --------------------------------------------------
namespace {

// The integers of the JSON array that follows "key": in text (at most cap).
int json_ints(const std::string &text, const char *key, int32_t *out, int cap) {
  const std::string k = std::string("\"") + key + "\"";
  size_t p = text.find(k);
  if (p == std::string::npos) return -1;
  p = text.find_first_not_of(" \t\r\n:", p + k.size());
  if (p == std::string::npos) return -1;
  if (text[p] != '[') {  // a scalar
    char *end = nullptr;
    const long v = std::strtol(text.c_str() + p, &end, 10);
    if (end == text.c_str() + p) return -1;
    out[0] = (int32_t)v;
    return 1;
  }
  int cnt = 0;
  ++p;
  while (cnt < cap) {
    p = text.find_first_not_of(" \t\r\n,", p);
    if (p == std::string::npos) return -1;
    if (text[p] == ']') break;
    char *end = nullptr;
    const long v = std::strtol(text.c_str() + p, &end, 10);
    if (end == text.c_str() + p) return -1;
    out[cnt++] = (int32_t)v;
    p = (size_t)(end - text.c_str());
  }
  return cnt;
}

}  // namespace

extern "C" int bola_batch_tuning_save(const char *path, const bola_batch_tuning *t) {
  if (!path || !t) return -1;
  FILE *f = std::fopen(path, "w");
  if (!f) return fail(-2, "bola_batch_tuning_save: cannot write %s", path);
  int dev = 0;
  cudaDeviceProp prop;
  std::memset(&prop, 0, sizeof prop);
  if (cudaGetDevice(&dev) == cudaSuccess) cudaGetDeviceProperties(&prop, dev);
  std::fprintf(f, "{\n  \"format\": \"bola_gb300 batched tuning 1\",\n  \"device\": \"%s\",\n  \"sms\": %d,\n",
               prop.name, prop.multiProcessorCount);
  const int32_t *arrs[2] = {t->group_size, t->panel_width};
  const char *names[2] = {"group_size", "panel_width"};
  for (int a = 0; a < 2; ++a) {
    std::fprintf(f, "  \"%s\": [", names[a]);
    for (int b = 0; b < NBUCKET; ++b) std::fprintf(f, "%d%s", arrs[a][b], b + 1 < NBUCKET ? ", " : "");
    std::fprintf(f, "],\n");
  }
  std::fprintf(f, "  \"tile_rows\": %d\n}\n", t->tile_rows);
  std::fclose(f);
  return 0;
}

extern "C" int bola_batch_tuning_load(const char *path, bola_batch_tuning *t, int32_t *sms_recorded) {
  if (!path || !t) return -1;
  FILE *f = std::fopen(path, "r");
  if (!f) return fail(-2, "bola_batch_tuning_load: cannot read %s", path);
  std::string text;
  char buf[4096];
  size_t got;
  while ((got = std::fread(buf, 1, sizeof buf, f)) > 0) text.append(buf, got);
  std::fclose(f);
  bola_batch_tuning r;
  std::memset(&r, 0, sizeof r);
  int32_t sms = 0;
  if (json_ints(text, "group_size", r.group_size, NBUCKET) != NBUCKET ||
      json_ints(text, "panel_width", r.panel_width, NBUCKET) != NBUCKET ||
      json_ints(text, "tile_rows", &r.tile_rows, 1) != 1)
    return fail(-2, "bola_batch_tuning_load: %s is not a tuning table", path);
  json_ints(text, "sms", &sms, 1);
  for (int b = 0; b < NBUCKET; ++b) {
    const int g = r.group_size[b], w = r.panel_width[b];
    if ((g != 0 && g != 32 && g != 64 && g != 128 && g != 256) || (w != 0 && w != 8 && w != 12 && w != 16))
      return fail(-3, "bola_batch_tuning_load: bucket %d has group %d / panel width %d", b, g, w);
  }
  if (r.tile_rows != 0 && r.tile_rows != 2 && r.tile_rows != 4)
    return fail(-3, "bola_batch_tuning_load: tile_rows %d", r.tile_rows);
  *t = r;
  if (sms_recorded) *sms_recorded = sms;
  return 0;
}
