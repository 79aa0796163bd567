// getrf.cu — LU with partial pivoting, BOLA's blocking and rounding
// (src/getrf.rs:37-101, src/getrf2.rs:39-185).
//
// Blocked right-looking LU with BOLA's NB = 32.  Per block column:
//   1. panel_lu_cluster: one thread-block CLUSTER (up to 16 CTAs, the panel's
//      rows spread over them and held in shared memory) factors the
//      (m-j) x 32 panel column by column: idamax under BOLA's lane order,
//      candidates and the pivot row exchanged through distributed shared
//      memory, reciprocal scale and BOLA's pairwise rank-1 update by warps of
//      their own (panel_lu, rows in global memory, for taller panels).
//   2. step_swap_trsm: the 32 row interchanges applied to every other column
//      (BOLA's two laswp calls) fused with BOLA's 32-row unit-lower trsm on
//      the right block row.
//   3. the exact DGEMM for the rank-32 trailing update (from n = 512 on split:
//      the next panel's columns on a high-priority stream, the rest overlapping
//      the next panel on a low-priority one).
// Every element sees the same operation sequence as in BOLA, so A and ipiv
// come out bit-identical (for the SIMD width selected).
#include <cooperative_groups.h>

#include <atomic>
#include <cstddef>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "sm100.cuh"

namespace cg = cooperative_groups;

namespace bola {
namespace {

constexpr int PNB = 32;   // panel width: BOLA's NB (src/getrf.rs:11) / recursion stop (src/getrf2.rs:11)
constexpr int PT = 256;   // threads per CTA in the panel kernel
constexpr int MAXC = 16;  // largest cluster (non-portable size on sm_103)
constexpr size_t SMEM_DATA_LIMIT = 200 * 1024;
constexpr int64_t LOOK_AHEAD_MIN = 512;

struct PanelPub {  // what a CTA publishes to the rest of the cluster each column
  int64_t v;
  int64_t key;
  int64_t g;  // panel row of this CTA's best candidate, -1 if none
  double best_row[PNB];
  double row_j[PNB];  // the current pivot-position row, from the CTA that owns it
};

constexpr size_t panel_base_bytes() {
  return 2 * sizeof(PanelPub) + (PT / 32) * sizeof(Cand) + PNB * sizeof(double) + 4 * sizeof(int64_t) +
         2 * sizeof(double);
}

// Unblocked LU of an mp x nb panel (nb <= 32), iterative_getrf2 of
// src/getrf2.rs:131-185, for panels too tall for the cluster's shared memory:
// the rows stay in global memory (L2), one full cluster barrier per column.
// Panels whose rows fit in shared memory take panel_lu_cluster below.
__global__ void __launch_bounds__(PT)
panel_lu(double *A, int64_t lda, int64_t mp, int nb, int32_t *ipiv, int32_t *info, int32_t add_on_success,
         int32_t col0, int lanes, int64_t R) {
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks();
  const int cr = (int)cluster.block_rank();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PanelPub *pub = reinterpret_cast<PanelPub *>(smem_raw);
  Cand *red = reinterpret_cast<Cand *>(pub + 2);
  double *prow = reinterpret_cast<double *>(red + PT / 32);
  int64_t *bc = reinterpret_cast<int64_t *>(prow + PNB);
  double *pinv = reinterpret_cast<double *>(bc + 4);  // 1 / pivot of the current column

  // Uniform across the cluster: the only writer of *info in this kernel acts
  // after a cluster barrier that every CTA reaches after this read.
  if (stop_flag(info)) return;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r0 = (int64_t)cr * R;
  const int64_t r1 = imin(mp, r0 + R);
  const int64_t nr = r1 > r0 ? r1 - r0 : 0;
  auto el = [&](int64_t il, int c) -> double & { return A[(r0 + il) + (int64_t)c * lda]; };
  __syncthreads();

  const int steps = (int)imin(mp, nb);
  bool failed = false;
  for (int j = 0; j < steps; ++j) {
    PanelPub *my = &pub[j & 1];
    const int64_t nlen = mp - j;
    // -- idamax over this CTA's rows >= j
    Cand best = cand_none();
    for (int64_t il = tid; il < nr; il += PT) {
      const int64_t g = r0 + il;
      if (g < j) continue;
      const Cand c = make_cand(el(il, j), g - j, nlen, lanes);
      if (cand_better(c, best)) best = c;
    }
    best = warp_best(best);
    if (lane == 0) red[warp] = best;
    __syncthreads();
    if (tid == 0) {
      Cand b = red[0];
      for (int w = 1; w < PT / 32; ++w)
        if (cand_better(red[w], b)) b = red[w];
      my->v = b.v;
      my->key = b.key;
      my->g = (b.v > -2) ? j + b.idx : -1;
      bc[0] = my->g;
    }
    __syncthreads();
    const int64_t myg = bc[0];
    if (tid < nb) {
      if (myg >= 0) my->best_row[tid] = el(myg - r0, tid);
      if (j >= r0 && j < r1) my->row_j[tid] = el(j - r0, tid);
    }
    cluster.sync();
    // -- cluster-wide winner (same total order in every CTA)
    if (warp == 0) {
      Cand c = cand_none();
      if (lane < C) {
        const PanelPub *rp = cluster.map_shared_rank(my, lane);
        c.v = rp->v;
        c.key = rp->key;
        c.idx = rp->g;
      }
      c = warp_best(c);
      if (lane == 0) bc[1] = (c.v < 0) ? (int64_t)j : c.idx;  // idamax -> 0 when nothing qualifies
    }
    __syncthreads();
    const int64_t jp = bc[1];
    const int owner_j = (int)(j / R), owner_p = (int)(jp / R);
    if (tid < nb) {
      const PanelPub *src = cluster.map_shared_rank(my, jp == j ? owner_j : owner_p);
      const double v = (jp == j) ? src->row_j[tid] : src->best_row[tid];
      prow[tid] = v;
      if (tid == j) pinv[0] = 1.0 / v;  // once per CTA, not once per thread
    }
    __syncthreads();
    const double pv = prow[j];
    if (cr == 0 && tid == 0) ipiv[j] = (int32_t)(jp + 1);
    if (!nonzero64(pv)) {  // exact zero pivot: BOLA's "Matrix is singular" (src/getrf2.rs:166-168)
      if (cr == 0 && tid == 0) *info = col0 + j + 1;
      failed = true;
      break;
    }
    // -- row interchange across the whole panel width (src/getrf2.rs:144-150)
    if (jp != j) {
      if (cr == owner_j && tid < nb) el(j - r0, tid) = prow[tid];
      if (cr == owner_p && tid < nb) {
        const PanelPub *sj = cluster.map_shared_rank(my, owner_j);
        el(jp - r0, tid) = sj->row_j[tid];
      }
    }
    __syncthreads();
    // -- reciprocal scale (src/getrf2.rs:152-164) and rank-1 update (ger, src/ger.rs:28-61)
    if (j < mp - 1) {
      const double inv = pinv[0];
      const int64_t mr = mp - j - 1;
      const int64_t rows_vec = (mr / lanes) * lanes;
      const int ncols = nb - j - 1;
      const int n_unrolled = ncols - (ncols % 2);
      const bool do_ger = j < steps - 1;
      for (int64_t il = tid; il < nr; il += PT) {
        const int64_t g = r0 + il;
        if (g <= j) continue;
        const double x = __dmul_rn(el(il, j), inv);
        el(il, j) = x;
        if (!do_ger) continue;
        const bool vec = (g - j - 1) < rows_vec;
        for (int t = 0; t < n_unrolled; t += 2) {
          const int c0 = j + 1 + t;
          const double t0 = -prow[c0], t1 = -prow[c0 + 1];
          if (!nonzero64(t0) && !nonzero64(t1)) continue;
          double &a0 = el(il, c0);
          double &a1 = el(il, c0 + 1);
          a0 = fused_or_unfused(vec, x, t0, a0);
          a1 = fused_or_unfused(vec, x, t1, a1);
        }
        if (ncols % 2) {
          const int c = nb - 1;
          const double t = -prow[c];
          if (nonzero64(t)) el(il, c) = add_prod(el(il, c), t, x);
        }
      }
    }
    __syncthreads();
  }
  if (!failed && cr == 0 && add_on_success != 0)
    for (int t = tid; t < steps; t += PT) ipiv[t] += add_on_success;
  cluster.sync();  // no CTA may leave while another can still read its shared memory
}

// What a panel leaves for the kernels that follow: its interchanges composed
// (position q < 32 takes old panel row SRC[q]; old row q < 32 goes to position
// TO[q], or stays among the first 32 if -1) and the value of *info after it,
// which those kernels stop on: the next panel, whose zero pivot must not stop
// them, runs beside them.
enum { PLAN_SRC = 0, PLAN_TO = PNB, PLAN_STOP = 2 * PNB, PLAN_INTS = 2 * PNB + 16 };

// BOLA's rank-1 step by pivot p (src/getrf2.rs:152-164 with src/ger.rs:28-61):
// ger walks columns p+1.. in pairs, skipping
// a pair whose two pivot-row entries are both zero, with the fused vector
// body for rows below mr rounded down to the SIMD width and the unfused tail
// after; an odd last column is always unfused (and skipped when zero).
struct GerStep {
  int p, nun;       // pivot column, columns of the paired part (ncols rounded down to even)
  int64_t vec_end;  // rows g with g - p - 1 < vec_end take the fused body
};
__device__ __forceinline__ GerStep ger_step(int p, int nb, int64_t mp, int lanes) {
  GerStep s;
  s.p = p;
  s.nun = (nb - p - 1) & ~1;
  s.vec_end = (mp - p - 1) & ~(int64_t)(lanes - 1);
  return s;
}
// A warp's pivot candidate for one column, as every CTA of the cluster gets it.
struct alignas(16) PivHdr {
  uint32_t lo, hi;  // the candidate's value (bits)
  uint32_t row;     // (row in its CTA's shared memory) << 16 | position in the panel; PIV_NONE: no candidate
  uint32_t pad;
};
constexpr uint32_t PIV_NONE = 0xffffffffu;

// BOLA's idamax order (make_cand) for one search, in pieces that one warp
// reduction mostly decides: a larger major wins, then a larger low word of
// |x|, then a smaller key.  Major 0: no candidate; 1: an element that idamax
// never selects (NaN, and zero except in short searches).
struct PivOrder {
  int base, nch, sl;  // first searched position, chunks of BOLA's vector body, log2(lanes)
  bool small;         // BOLA's scalar search
};
__device__ __forceinline__ PivOrder piv_order(int j, int mp, int lanes) {
  PivOrder o;
  o.base = j;
  o.sl = lanes == 4 ? 2 : 1;
  o.nch = (mp - j) >> (o.sl + 2);
  o.small = o.nch == 0;
  return o;
}
__device__ __forceinline__ uint32_t piv_major(const PivOrder &o, uint32_t hi, uint32_t lo) {
  hi &= 0x7fffffffu;
  const bool nan = hi > 0x7ff00000u || (hi == 0x7ff00000u && lo != 0);
  return nan || ((hi | lo) == 0 && !o.small) ? 1u : hi + 2;
}
__device__ __forceinline__ uint32_t piv_key(const PivOrder &o, int pos) {
  const int idx = pos - o.base, sc = o.sl + 2;
  if (idx >= (o.nch << sc)) return (uint32_t)idx;
  const int r = idx & ((1 << sc) - 1);
  return (uint32_t)(((r & ((1 << o.sl) - 1)) * 4 + (r >> o.sl)) * o.nch + (idx >> sc));
}
__device__ __forceinline__ bool piv_better(const PivOrder &o, uint32_t ma, uint32_t la, int pa, uint32_t mb, uint32_t lb,
                                           int pb) {
  if (ma != mb) return ma > mb;
  if (ma > 1 && la != lb) return la > lb;
  return piv_key(o, pa) < piv_key(o, pb);
}
// The lane that holds the warp's best candidate.
__device__ __forceinline__ int piv_best_lane(const PivOrder &o, uint32_t major, uint32_t lo, int pos) {
  const unsigned FULL = 0xffffffffu;
  const uint32_t mj = __reduce_max_sync(FULL, major);
  unsigned m = __ballot_sync(FULL, major == mj);
  if ((m & (m - 1)) && mj > 0) {
    bool in = major == mj;
    if (mj > 1) {
      const uint32_t ml = __reduce_max_sync(FULL, in ? lo : 0u);
      in = in && lo == ml;
    }
    const uint32_t key = in ? piv_key(o, pos) : PIV_NONE;
    const uint32_t mk = __reduce_min_sync(FULL, key);
    m = __ballot_sync(FULL, in && key == mk);
  }
  return __ffs(m) - 1;
}

constexpr int PIV_WARPS = 4;  // one per sub-partition
constexpr int UPD_WARPS = 8;
constexpr int PIV_T = 32 * PIV_WARPS;
constexpr int PAN_T = 32 * (PIV_WARPS + UPD_WARPS);
constexpr int PAN_ROWS = 32;  // rows per CTA aimed at
enum { BAR_UPDATED = 1, BAR_SCALED = 2 };
// Named barriers between the pivot warps and the update warps; a warp that
// has diverged must be whole again before it takes part.
__device__ __forceinline__ void bar_sync(int id) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(PAN_T) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(PAN_T) : "memory");
}
__host__ __device__ constexpr int panel_pitch(int R) { return R | 1; }  // odd: a row's columns lie in different banks
inline size_t panel_smem(int64_t R) {
  return sizeof(double) * PNB * (size_t)panel_pitch((int)R) + sizeof(int32_t) * (size_t)R;
}

// Unblocked LU of an mp x nb panel (BOLA's iterative_getrf2), the rows spread
// over a cluster and held in shared memory.  What bounds it is the chain of
// one column after the other: find the pivot, agree on it, divide by it, bring
// the next column up to date.  So the chain has warps of its own and carries
// nothing else:
//  - rows never move; a row's position (where BOLA's interchanges would have
//    put it) is kept beside it and decides its place in BOLA's idamax order
//    and in the fused or unfused part of ger;
//  - four pivot warps hold the current column in registers: they scale it,
//    bring the next one up to date and search it, and each sends its candidate
//    (16 bytes: value, row, position) to every CTA by st.async onto the
//    receiver's mbarrier; every warp then knows the pivot and forms its
//    reciprocal while the pivot's CTA sends the pivot row after it;
//  - eight update warps apply pivot j to the columns right of j + 1 meanwhile;
//    they are done before the next pivot's row is read.
// Each exchange is double-buffered by the column's parity: a CTA sends its
// candidates for column j + 2 only once it has everyone's for column j + 1,
// and those are sent after column j's were read.  Waits are bounded: one that
// runs out stops the panel with *info = BOLA_INFO_WAIT_EXPIRED.
// Every element sees BOLA's operations in BOLA's order.  RPT: rows per pivot
// thread (R <= 128 RPT).
// Measured on one GB300, alone on the GPU: 1024 x 32 in 52 us (203 with the same
// warps on the search and the update, four CTA barriers a column), about 2600
// cycles a column; 4096 x 32 in 96 us.  Beside a wide DGEMM, whose older warps
// the FP64 pipe serves first, a 4096-row panel takes 147 us on average.
template <int RPT>
__global__ void __launch_bounds__(PAN_T, 1)
panel_lu_cluster(double *A, int64_t lda, int64_t mp64, int nb, int32_t *ipiv, int32_t *info, int32_t add_on_success,
                 int32_t col0, int lanes, int64_t R64, int32_t *plan, bool fresh) {
  sm100::grid_dependency_wait();
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks();
  const int cr = (int)cluster.block_rank();
  __shared__ PivHdr hdr[2][MAXC * PIV_WARPS];
  __shared__ __align__(16) double prow[2][PNB];  // the pivot row (columns right of the pivot are used)
  __shared__ uint64_t hbar[2], rbar[2];  // every candidate / the pivot row has landed
  __shared__ int hfail[2], rfail[2], sstop;  // a wait for candidates / for a row ran out (by parity); the panel ends
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int mp = (int)mp64, R = (int)R64, RP = panel_pitch(R);
  double *data = reinterpret_cast<double *>(smem_raw);  // column c of local row il: data[c * RP + il]
  int32_t *spos = reinterpret_cast<int32_t *>(data + PNB * RP);

  // Uniform across the cluster: the only writer of *info here acts after
  // the cluster barrier that every CTA passes after this read.  (fresh: the
  // first panel, which resets *info instead.)
  if (!fresh && stop_flag(info)) {
    if (plan != nullptr && cr == 0 && threadIdx.x == 0) plan[PLAN_STOP] = *info;
    return;
  }

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (fresh && cr == 0 && tid == 0) *info = 0;
  const int r0 = cr * R, nr = max(0, min(mp, r0 + R) - r0);
  for (int il0 = 0; il0 < nr; il0 += 64) {
    double t[3][2];
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = warp + q * (PAN_T / 32), il = il0 + 32 * h + lane;
        t[q][h] = c < nb && il < nr ? A[(r0 + il) + (int64_t)c * lda] : 0.0;
      }
#pragma unroll
    for (int q = 0; q < 3; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = warp + q * (PAN_T / 32), il = il0 + 32 * h + lane;
        if (c < nb && il < nr) data[c * RP + il] = t[q][h];
      }
  }
  for (int il = tid; il < nr; il += PAN_T) spos[il] = r0 + il;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      sm100::mbar_init(&hbar[i], 1);
      sm100::mbar_init(&rbar[i], 1);
    }
    sm100::fence_mbar_init();
    hfail[0] = hfail[1] = rfail[0] = rfail[1] = sstop = 0;
  }
  __syncthreads();
  cluster.sync();  // every CTA runs, its mbarriers initialised and its rows loaded, before the first push

  const int steps = min(mp, nb);
  // log2 of the pivot warps per CTA that can hold rows
  const int lsend = R <= 32 ? 0 : R <= 64 ? 1 : 2;
  if (warp < PIV_WARPS) {
    const bool sends = warp < (1 << lsend) && lane < C;
    const uint32_t hdr_at = sm100::cluster_addr(&hdr[0][(cr << lsend) + (warp & ((1 << lsend) - 1))], min(lane, C - 1));
    const uint32_t hbar_at = sm100::cluster_addr(&hbar[0], min(lane, C - 1));
    const int S = C << lsend;
    double a[RPT];  // column j of this thread's rows, up to date
    int g[RPT];     // their positions; -1: no row
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int il = tid + PIV_T * r;
      g[r] = il < nr ? r0 + il : -1;
      a[r] = il < nr ? data[il] : 0.0;
    }
    for (int j = 0; j < steps; ++j) {
      const int par = j & 1;
      const uint32_t phase = (uint32_t)(j >> 1) & 1u;
      const bool next = j < steps - 1;  // then j + 1 < nb as well
      const PivOrder o = piv_order(j, mp, lanes);
      // -- this warp's candidate, to every CTA
      if (warp < (1 << lsend)) {
        uint32_t mj = 0, lo = 0, hi = 0, row = PIV_NONE;
        int pos = -1;
#pragma unroll
        for (int r = 0; r < RPT; ++r) {
          const uint32_t h = (uint32_t)__double2hiint(a[r]), l = (uint32_t)__double2loint(a[r]);
          const uint32_t m = g[r] >= j ? piv_major(o, h, l) : 0u;
          if (RPT == 1 || (m > 0 && piv_better(o, m, l, g[r], mj, lo, pos))) {
            mj = m;
            hi = h;
            lo = l;
            pos = g[r];
            row = m > 0 ? (uint32_t)(tid + PIV_T * r) << 16 | (uint32_t)pos : PIV_NONE;
          }
        }
        const int bl = piv_best_lane(o, mj, lo, pos);
        hi = __shfl_sync(0xffffffffu, hi, bl);
        lo = __shfl_sync(0xffffffffu, lo, bl);
        row = __shfl_sync(0xffffffffu, row, bl);
        if (sends)
          sm100::st_async4(hdr_at + par * (uint32_t)sizeof(hdr[0]), lo, hi, row, 0u, hbar_at + par * 8u);
      }
      if (tid == PIV_T - 1) {  // (a warp that mostly sends nothing)
        sm100::mbar_arrive_expect_tx(&hbar[par], (uint32_t)(S * sizeof(PivHdr)));
        if (next) sm100::mbar_arrive_expect_tx(&rbar[par], (uint32_t)(PNB * sizeof(double)));
      }
      // -- the cluster's pivot, the same in every CTA
      if (!sm100::bounded_wait(&hbar[par], phase)) hfail[par] = 1;
      double pv;
      uint32_t prw;
      int wc;  // its CTA
      {
        PivHdr h;
        h.row = PIV_NONE;
        h.hi = h.lo = 0;
        if (lane < S) h = hdr[par][lane];
        uint32_t mj = h.row != PIV_NONE ? piv_major(o, h.hi, h.lo) : 0u;
        int slot = lane;
        if (S > 32) {
          const int q = lane + 32;
          PivHdr h2;
          h2.row = PIV_NONE;
          if (q < S) h2 = hdr[par][q];
          const uint32_t m2 = h2.row != PIV_NONE ? piv_major(o, h2.hi, h2.lo) : 0u;
          if (m2 > 0 &&
              piv_better(o, m2, h2.lo, (int)(h2.row & 0xffffu), mj, h.lo, (int)(h.row & 0xffffu))) {
            mj = m2;
            h = h2;
            slot = q;
          }
        }
        const int wl = piv_best_lane(o, mj, h.lo, (int)(h.row & 0xffffu));
        pv = __hiloint2double((int)__shfl_sync(0xffffffffu, h.hi, wl), (int)__shfl_sync(0xffffffffu, h.lo, wl));
        prw = __shfl_sync(0xffffffffu, h.row, wl);
        wc = __shfl_sync(0xffffffffu, slot, wl) >> lsend;
      }
      const int jp = (int)(prw & 0xffffu);
      bar_sync(BAR_UPDATED);  // the update warps are done with pivot j - 1
      const int lost = hfail[par] | rfail[par ^ 1];  // this column's candidates, the last one's row: written before it
      if (lost || !nonzero64(pv)) {
        // an exact zero pivot: BOLA's "Matrix is singular" (src/getrf2.rs:166-168)
#pragma unroll
        for (int r = 0; r < RPT; ++r)
          if (g[r] >= j) data[j * RP + tid + PIV_T * r] = a[r];
        if (tid == 0) {
          sstop = 1;
          if (lost) {
            atomicCAS(info, 0, BOLA_INFO_WAIT_EXPIRED);
          } else if (cr == 0) {
            ipiv[j] = jp + 1;
            *info = col0 + j + 1;
          }
        }
        bar_arrive(BAR_SCALED);
        break;
      }
      // -- the pivot's CTA sends the row; everyone forms the reciprocal
      if (next && wc == cr) {
        const int pil = (int)(prw >> 16), c = 2 * (tid & 15);
        const double v0 = data[c * RP + pil], v1 = data[(c + 1) * RP + pil];
        for (int d = tid >> 4; d < C; d += PIV_T / 16)
          sm100::st_async4(sm100::cluster_addr(&prow[par][c], d), (uint32_t)__double2loint(v0),
                           (uint32_t)__double2hiint(v0), (uint32_t)__double2loint(v1), (uint32_t)__double2hiint(v1),
                           sm100::cluster_addr(&rbar[par], d));
      }
      // (src/getrf2.rs:152-164, src/ger.rs:28-61)
      const double inv = recip_rn(pv);
      double an[RPT];  // column j + 1
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        if (RPT > 1 && PIV_T * r >= nr) break;
        const int il = tid + PIV_T * r;
        an[r] = next && il < nr ? data[(j + 1) * RP + il] : 0.0;
        const double x = __dmul_rn(a[r], inv);
        if (g[r] >= j) {
          if (g[r] == j || g[r] == jp) {  // the interchange of positions j and jp
            g[r] = g[r] == jp ? j : jp;
            spos[il] = g[r];
          }
          data[j * RP + il] = g[r] == j ? a[r] : x;  // the pivot stays
        }
        a[r] = x;
      }
      if (next) {
        if (!sm100::bounded_wait(&rbar[par], phase)) rfail[par] = 1;
        bar_arrive(BAR_SCALED);  // the update warps may start
        const GerStep gs = ger_step(j, nb, mp, lanes);
        const double pn = prow[par][j + 1];
        // j + 1 is ger's first column: paired with j + 2 unless it is the last
        bool touch = nonzero64(pn);
        if (gs.nun > 0) touch = touch || nonzero64(prow[par][j + 2]);
        if (touch) {
#pragma unroll
          for (int r = 0; r < RPT; ++r) {
            if (RPT > 1 && PIV_T * r >= nr) break;
            const bool body = gs.nun > 0 && g[r] - j - 1 < gs.vec_end;
            const double u = __fma_rn(a[r], -pn, an[r]);
            a[r] = __any_sync(0xffffffffu, !body && g[r] > j) && !body ? add_prod(an[r], a[r], -pn) : u;
          }
        } else {
#pragma unroll
          for (int r = 0; r < RPT; ++r) a[r] = an[r];
        }
      } else {
        bar_arrive(BAR_SCALED);
      }
      if (cr == 0 && tid == 0) ipiv[j] = jp + 1;
    }
  } else {
    // Update warps: pivot j on columns j + 2.., 32 rows of one group at a time;
    // with fewer row groups than warps a group's columns are split.
    const int uw = warp - PIV_WARPS;
    const int groups = (nr + 31) / 32;
    const int split = groups <= 1 ? 8 : groups <= 2 ? 4 : groups <= 4 ? 2 : 1;
    const int ws = uw % split;
    for (int j = 0; j < steps; ++j) {
      const GerStep gs = ger_step(j, nb, mp, lanes);
      const bool odd = (nb - j - 1) & 1;
      const int cend = odd ? nb - 1 : nb, c0 = j + 2 + ws;
      // first columns of ger's pairs
      const unsigned first = gs.nun > 0 ? (0x55555555u << ((j + 1) & 1)) & (((1u << gs.nun) - 1u) << (j + 1)) : 0u;
      const double *pr = prow[j & 1];
      bar_arrive(BAR_UPDATED);
      bar_sync(BAR_SCALED);
      if (sstop) break;
      if (j >= steps - 1) continue;
      unsigned touch = 0;
      for (int gr = uw / split; gr < groups; gr += UPD_WARPS / split) {
        const int il = min(gr * 32 + lane, nr - 1);
        const int g = gr * 32 + lane < nr ? spos[il] : -1;
        const double x = data[j * RP + il];
        constexpr int U = 4;  // independent updates in flight per warp
        for (int cb = c0; cb < cend; cb += U * split) {
          double v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = cb + u * split;
            if (c < cend) v[u] = __fma_rn(x, -pr[c], data[c * RP + il]);
          }
          if (cb == c0) {
            // the columns that ger touches: a pair with a non-zero entry, a
            // last odd column (always unfused) if non-zero
            const unsigned nz = __ballot_sync(0xffffffffu, lane < nb && nonzero64(pr[lane]));
            const unsigned pairs = (nz | nz >> 1) & first;
            touch = pairs | pairs << 1 | (odd ? nz & (1u << (nb - 1)) : 0u);
          }
          const bool body = g > j && g - j - 1 < gs.vec_end;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c = cb + u * split;
            if (c < cend && body && (touch >> c & 1u)) data[c * RP + il] = v[u];
          }
        }
        if (c0 >= cend) {  // no paired column of this warp's
          const unsigned nz = __ballot_sync(0xffffffffu, lane < nb && nonzero64(pr[lane]));
          touch = odd ? nz & (1u << (nb - 1)) : 0u;
        }
        const bool body = g > j && g - j - 1 < gs.vec_end;
        if (odd && nb - 1 >= c0 && (nb - 1 - c0) % split == 0 && (touch >> (nb - 1) & 1u)) {
          const double v = add_prod(data[(nb - 1) * RP + il], x, -pr[nb - 1]);
          if (body) data[(nb - 1) * RP + il] = v;
        }
        // rows past the vector body (fewer than `lanes` of the whole panel): a
        // lane per column, so that the other rows' warps issue only FMAs
        unsigned tail = __ballot_sync(0xffffffffu, g > j && !body);
        if (ws == split - 1 && tail) {
          const unsigned nz = __ballot_sync(0xffffffffu, lane < nb && nonzero64(pr[lane]));
          const unsigned pairs = (nz | nz >> 1) & first;
          const unsigned all = pairs | pairs << 1 | (odd ? nz & (1u << (nb - 1)) : 0u);
          do {
            const int tl = gr * 32 + __ffs(tail) - 1;
            tail &= tail - 1;
            const double v = lane < nb ? add_prod(data[lane * RP + tl], data[j * RP + tl], -pr[lane]) : 0.0;
            if (lane > j + 1 && lane < nb && (all >> lane & 1u)) data[lane * RP + tl] = v;
          } while (tail);
        }
      }
    }
  }
  __syncthreads();
  if (!sstop && cr == 0 && add_on_success != 0)
    for (int t = tid; t < steps; t += PAN_T) ipiv[t] += add_on_success;
  // every row to its position (all but the rows that pivots displaced stay
  // where they were: coalesced)
  for (int c = warp; c < nb; c += PAN_T / 32)
    for (int il = lane; il < nr; il += 32) A[spos[il] + (int64_t)c * lda] = data[c * RP + il];
  if (plan != nullptr) {
    for (int il = tid; il < nr; il += PAN_T) {
      const int was = r0 + il, is = spos[il];
      if (is < steps) plan[PLAN_SRC + is] = was;
      if (was < steps) plan[PLAN_TO + was] = is < steps ? -1 : is;
    }
  }
  cluster.sync();  // no CTA may leave while another can still push into it
  if (plan != nullptr && cr == 0 && tid == 0) plan[PLAN_STOP] = *(volatile int32_t *)info;
}

// iterative_getrf2 for a short, wide matrix (m <= 32 rows, any n): one CTA,
// data in global memory.
__global__ void __launch_bounds__(PT)
panel_lu_wide(double *A, int64_t lda, int64_t m, int64_t n, int32_t *ipiv, int32_t *info, int32_t col0,
              int lanes) {
  __shared__ Cand red[PT / 32];
  __shared__ int64_t sjp;
  if (stop_flag(info)) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t steps = imin(m, n);
  for (int64_t j = 0; j < steps; ++j) {
    Cand best = cand_none();
    for (int64_t g = j + tid; g < m; g += PT) {
      const Cand c = make_cand(A[g + j * lda], g - j, m - j, lanes);
      if (cand_better(c, best)) best = c;
    }
    best = warp_best(best);
    if (lane == 0) red[warp] = best;
    __syncthreads();
    if (tid == 0) {
      Cand b = red[0];
      for (int w = 1; w < PT / 32; ++w)
        if (cand_better(red[w], b)) b = red[w];
      sjp = (b.v < 0) ? j : j + b.idx;
      ipiv[j] = (int32_t)(sjp + 1);
    }
    __syncthreads();
    const int64_t jp = sjp;
    const double pv = A[jp + j * lda];
    if (!nonzero64(pv)) {
      if (tid == 0) *info = col0 + (int32_t)j + 1;
      return;
    }
    if (jp != j) {
      for (int64_t c = tid; c < n; c += PT) {
        const double t = A[j + c * lda];
        A[j + c * lda] = A[jp + c * lda];
        A[jp + c * lda] = t;
      }
    }
    __syncthreads();
    if (j < m - 1) {
      const double inv = 1.0 / pv;
      for (int64_t g = j + 1 + tid; g < m; g += PT) A[g + j * lda] = __dmul_rn(A[g + j * lda], inv);
    }
    __syncthreads();
    if (j < steps - 1) {
      const int64_t mr = m - j - 1, ncols = n - j - 1;
      const int64_t rows_vec = (mr / lanes) * lanes, n_unrolled = ncols - (ncols % 2);
      for (int64_t e = tid; e < mr * ncols; e += PT) {
        const int64_t ri = e % mr, ci = e / mr;
        const int64_t g = j + 1 + ri, c = j + 1 + ci;
        const double x = A[g + j * lda];
        double &a = A[g + c * lda];
        if (ci < n_unrolled) {
          const int64_t p0 = j + 1 + (ci & ~(int64_t)1);
          const double t0 = -A[j + p0 * lda], t1 = -A[j + (p0 + 1) * lda];
          if (!nonzero64(t0) && !nonzero64(t1)) continue;
          const double t = (c == p0) ? t0 : t1;
          a = fused_or_unfused(ri < rows_vec, x, t, a);
        } else {
          const double t = -A[j + c * lda];
          if (nonzero64(t)) a = add_prod(a, t, x);
        }
      }
    }
    __syncthreads();
  }
}

// The same plan from the panel's ipiv (with its offset j added), for the
// panel kernels that do not write one.  One warp.
__global__ void plan_from_ipiv(int jb, const int32_t *ipiv, int32_t j, const int32_t *info, int32_t *plan) {
  __shared__ int64_t rows[2 * PNB], src[2 * PNB];
  const int lane = threadIdx.x;
  if (lane == 0) plan[PLAN_STOP] = *info;
  if (stop_flag(info)) return;
  SwapPlan p;
  p.ix0 = 0;
  p.i1 = j + 1;
  p.i2 = j + jb;
  p.i_inc = 1;
  p.incx = 1;
  const int cnt = compose_swaps_warp(p, ipiv, rows, src);
  plan[PLAN_SRC + lane] = lane;
  plan[PLAN_TO + lane] = -1;
  __syncwarp();
  for (int t = lane; t < cnt; t += 32) {
    const int r = (int)(rows[t] - j), f = (int)(src[t] - j);
    if (r < jb) plan[PLAN_SRC + r] = f;
    else plan[PLAN_TO + f] = r;
  }
}

// One getrf block step after the panel at column j: the panel's interchanges
// applied to the columns [c0, c0 + ncols) but its own (src/getrf.rs:64-70) and,
// right of it, BOLA's unit-lower trsm base case with its daxpy
// (src/getrf.rs:78, src/trsm.rs:96-109).  A warp per column, a lane per row;
// the chain of a step (broadcast, multiply-add) is what it waits for, with the
// column's coefficients one step ahead.  Measured at n = 1024: 7 us for all
// columns (26 with the interchanges composed by every CTA and the solve's votes
// and loads inside the chain).
constexpr int SW_WARPS = 4;
__global__ void __launch_bounds__(32 * SW_WARPS)
step_swap_trsm(double *A, int64_t lda, int64_t j, int jb, int64_t c0, int64_t ncols, const int32_t *plan, int lanes) {
  sm100::grid_dependency_wait();
  __shared__ double L[PNB * PNB];
  if (stop_flag(plan + PLAN_STOP)) return;
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * SW_WARPS + (threadIdx.x >> 5);
  int64_t col = c0 + w;
  if (col >= j && c0 <= j) col += jb;  // (a range that starts at or left of the panel skips it)
  const bool on = w < ncols, right = col >= j + jb;
  double *cp = A + col * lda + j;
  double b = 0.0, mv = 0.0;
  int to = -1;
  if (on && lane < jb) {
    b = cp[plan[PLAN_SRC + lane]];
    to = plan[PLAN_TO + lane];
    if (to >= 0) mv = cp[lane];
  }
  for (int e = threadIdx.x; e < PNB * PNB; e += 32 * SW_WARPS) {
    const int r = e % PNB, c = e / PNB;
    L[e] = r < jb && c < r ? A[(j + r) + (j + c) * lda] : 0.0;
  }
  __syncthreads();
  if (!on) return;
  if (to >= 0) cp[to] = mv;
  if (right) {
    double an = L[lane];
    for (int k = 0; k < jb - 1; ++k) {
      const double a = an;
      an = L[lane + (k + 1) * PNB];
      const double bk = __shfl_sync(0xffffffffu, b, k);
      if (!nonzero64(bk)) continue;
      // daxpy over rows k + 1.. with alpha = -b_k: its last len % lanes rows are the unfused tail
      const int cut = jb - ((jb - k - 1) & (lanes - 1));
      const double f = __fma_rn(-bk, a, b);
      if (cut < jb) {
        const double t = add_prod(b, -bk, a);
        if (lane > k) b = lane < cut ? f : t;
      } else if (lane > k) {
        b = f;
      }
    }
  }
  if (lane < jb) cp[lane] = b;
}

__global__ void zero_i32(int32_t *p) { *p = 0; }

// The n row interchanges of a factorisation on the right-hand sides, in order
// (laswp with k1 = 1, k2 = n).  A CTA composes them into one permutation in
// shared memory (one thread, ~60 cycles each) while the others load its first
// column, then gathers its columns.  Bound by that chain: n = 200 in 15 us,
// n = 4000 in 136 (under the profiler's events); a thread per column walking
// the interchanges through global memory took 33 and 729 us.  Entries that name no row of b are left to that
// walk, element by element as it would go.
constexpr int GR_T = 256;
constexpr int64_t GR_MAX = 8192;  // rows: 16 bytes of shared memory each
__global__ void __launch_bounds__(GR_T)
getrs_rows(int n, int64_t nrhs, const int32_t *ipiv, double *b, int64_t ldb) {
  sm100::grid_dependency_wait();
  extern __shared__ __align__(16) unsigned char gr_raw[];
  double *x = reinterpret_cast<double *>(gr_raw);
  int32_t *p = reinterpret_cast<int32_t *>(x + n), *piv = p + n;
  bool out = false;
  for (int i = threadIdx.x; i < n; i += GR_T) {
    const int32_t t = ipiv[i] - 1;
    out = out || (uint32_t)t >= (uint32_t)n;
    piv[i] = t;
    p[i] = i;
  }
  if (__syncthreads_or(out)) {
    if (threadIdx.x == 0)
      for (int64_t c = blockIdx.x; c < nrhs; c += gridDim.x) {
        double *cp = b + c * ldb;
        for (int i = 0; i < n; ++i) {
          const double t = cp[i];
          cp[i] = cp[piv[i]];
          cp[piv[i]] = t;
        }
      }
    return;
  }
  for (int64_t c = blockIdx.x; c < nrhs; c += gridDim.x) {
    double *cp = b + c * ldb;
    const bool first = c == (int64_t)blockIdx.x;
    if (first && threadIdx.x == 0) {
#pragma unroll 4
      for (int i = 0; i < n; ++i) {
        const int t = piv[i], u = p[i], w = p[t];
        p[i] = w;
        p[t] = u;
      }
    }
    if (!first || threadIdx.x >= 32)
      for (int i = first ? (int)threadIdx.x - 32 : (int)threadIdx.x; i < n; i += first ? GR_T - 32 : GR_T) x[i] = cp[i];
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += GR_T) cp[i] = x[p[i]];
    __syncthreads();
  }
}

// Launches a panel on the largest cluster (<= 16 CTAs) the device can
// co-schedule: about 32 rows per CTA, so that the update warps stay well behind
// the pivot warps' chain; more rows per CTA once 16 CTAs are in use (1024 x 32,
// 64 rows: 52 us; 4096 x 32, 256 rows: 96 us).  Rows that do not fit
// in shared memory (mp > 12k) stay in global memory (panel_lu).
int launch_panel(cudaStream_t s, double *A, int64_t lda, int64_t mp, int nb, int32_t *ipiv, int32_t *info,
                 int32_t add_on_success, int32_t col0, int32_t *plan = nullptr, bool fresh = false) {
  double fl = 0.0;
  for (int j = 0; j < nb && j < mp; ++j) fl += (double)(mp - j - 1) * (1.0 + 2.0 * (nb - j - 1));
  ProfScope prof(s, "getrf_panel", fl, 16.0 * (double)mp * nb);
  int C = (int)imin(MAXC, imax(1, cdiv(mp, PAN_ROWS)));
  for (;; C = C > 1 ? (C + 1) / 2 : 0) {
    if (C == 0) return fail(BOLA_ERR_CUDA, "panel_lu: no cluster size could be scheduled");
    const int64_t R = cdiv(mp, C);
    const bool use_smem = panel_smem(R) <= SMEM_DATA_LIMIT;
    const size_t smem = use_smem ? panel_smem(R) : panel_base_bytes();
    void (*const cluster_kern)(double *, int64_t, int64_t, int, int32_t *, int32_t *, int32_t, int32_t, int, int64_t,
                               int32_t *, bool) = R <= PIV_T       ? panel_lu_cluster<1>
                                                  : R <= 2 * PIV_T ? panel_lu_cluster<2>
                                                  : R <= 4 * PIV_T ? panel_lu_cluster<4>
                                                                   : panel_lu_cluster<7>;
    const void *kern = use_smem ? reinterpret_cast<const void *>(cluster_kern) : reinterpret_cast<const void *>(panel_lu);
    const int ki = !use_smem ? 0 : R <= PIV_T ? 1 : R <= 2 * PIV_T ? 2 : R <= 4 * PIV_T ? 3 : 4;
    BOLA_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_DATA_LIMIT));
    BOLA_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)C, 1, 1);
    cfg.blockDim = dim3(use_smem ? PAN_T : PT, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // asked once per device, kernel and cluster size, for the largest shared memory
    int dev = 0;
    BOLA_TRY_CUDA(cudaGetDevice(&dev));
    static std::atomic<int8_t> fits[64][5][MAXC + 1];
    std::atomic<int8_t> &known = fits[dev & 63][ki][C];
    if (known.load(std::memory_order_relaxed) == 0) {
      cfg.dynamicSmemBytes = use_smem ? SMEM_DATA_LIMIT : smem;
      int nclusters = 0;
      const bool ok = cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) == cudaSuccess && nclusters >= 1;
      cudaGetLastError();
      known.store(ok ? 1 : -1, std::memory_order_relaxed);
      cfg.dynamicSmemBytes = smem;
    }
    if (known.load(std::memory_order_relaxed) < 0) continue;
    const int lanes_v = lanes();
    if (use_smem) {
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_after
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.numAttrs = 2;
      BOLA_TRY_CUDA(cudaLaunchKernelEx(&cfg, cluster_kern, A, lda, mp, nb, ipiv, info, add_on_success, col0, lanes_v, R,
                                       plan, fresh));
      return 0;
    }
    if (fresh) zero_i32<<<1, 1, 0, s>>>(info);
    BOLA_TRY_CUDA(cudaLaunchKernelEx(&cfg, panel_lu, A, lda, mp, nb, ipiv, info, add_on_success, col0, lanes_v, R));
    if (plan != nullptr) plan_from_ipiv<<<1, 32, 0, s>>>((int)imin(nb, mp), ipiv, add_on_success, info, plan);
    BOLA_CHECK_LAUNCH();
    return 0;
  }
}

// iterative_getrf2 dispatch: tall panels go to the cluster kernel, short wide
// ones to the single-CTA kernel.
int iterative(cudaStream_t s, int64_t m, int64_t n, double *A, int64_t lda, int32_t *ipiv, int32_t *info,
              int32_t col0, int32_t add_on_success) {
  if (n <= PNB) return launch_panel(s, A, lda, m, (int)n, ipiv, info, add_on_success, col0);
  ProfScope prof(s, "getrf_panel_wide", 2.0 * (double)m * m * n);
  panel_lu_wide<<<1, PT, 0, s>>>(A, lda, m, n, ipiv, info, col0, lanes());
  BOLA_CHECK_LAUNCH();
  return ipiv_add(s, ipiv, imin(m, n), add_on_success, info);
}

}  // namespace

// src/getrf2.rs:39-106; col0 is the global column of A's first column (for info).
int getrf2_rec(cudaStream_t s, int64_t m, int64_t n, double *A, int64_t lda, int32_t *ipiv, int32_t *info,
               int32_t col0) {
  if (m == 0 || n == 0) return 0;
  if (m <= PNB || n <= PNB) return iterative(s, m, n, A, lda, ipiv, info, col0, 0);
  const int64_t n1 = imin(m, n) / 2, n2 = n - n1;
  BOLA_TRY(getrf2_rec(s, m, n1, A, lda, ipiv, info, col0));
  BOLA_TRY(laswp_exact(s, n2, A + n1 * lda, lda, 1, (int32_t)n1, ipiv, 1, info));
  BOLA_TRY(trsm_exact(s, 'L', 'L', 'N', 'U', n1, n2, 1.0, A, lda, A + n1 * lda, lda, info));
  if (n1 < m) {
    BOLA_TRY(dgemm_exact(s, 'N', 'N', m - n1, n2, n1, -1.0, A + n1, lda, A + n1 * lda, lda, 1.0,
                         A + n1 + n1 * lda, lda, 64, info, 0));
    BOLA_TRY(getrf2_rec(s, m - n1, n2, A + n1 + n1 * lda, lda, ipiv + n1, info, col0 + (int32_t)n1));
  }
  BOLA_TRY(ipiv_add(s, ipiv + n1, imin(m, n) - n1, (int32_t)n1, info));
  return laswp_exact(s, n1, A, lda, (int32_t)(n1 + 1), (int32_t)imin(m, n), ipiv, 1, info);
}

// src/getrf.rs:37-101

// ---- look-ahead stream pool (shared by the blocked getrf and potrf) ----------
namespace {
std::mutex g_la_mu;
std::vector<LookAhead *> g_la_pool[64];

// The capture that stream s is part of (0: none).
unsigned long long capture_of(cudaStream_t s) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(s, &status, &id) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return status == cudaStreamCaptureStatusNone ? 0 : id;
}
}  // namespace

LookAhead *la_acquire(cudaStream_t s) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  const unsigned long long id = context_id(), capture = capture_of(s);
  {
    std::lock_guard<std::mutex> lk(g_la_mu);
    auto &pool = g_la_pool[dev & 63];
    for (size_t i = pool.size(); i-- > 0;)
      if (pool[i]->ctx_id == id && capture_of(pool[i]->sp) == capture && capture_of(pool[i]->su) == capture) {
        LookAhead *la = pool[i];
        pool.erase(pool.begin() + (std::ptrdiff_t)i);
        return la;
      }
  }
  LookAhead *la = new LookAhead();
  la->ctx_id = id;
  int least = 0, greatest = 0;
  bool ok = cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess &&
            cudaStreamCreateWithPriority(&la->sp, cudaStreamNonBlocking, greatest) == cudaSuccess &&
            cudaStreamCreateWithPriority(&la->su, cudaStreamNonBlocking, least) == cudaSuccess;
  for (cudaEvent_t &e : la->ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (!ok) return nullptr;  // (leaks the partial set; only on a failing device)
  return la;
}

void la_release(LookAhead *la) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_la_mu);
  g_la_pool[dev & 63].push_back(la);
}

// BOLA's blocked getrf (src/getrf.rs:37-101) with look-ahead.  Per step k, on
// the high-priority stream sp: the panel, then the interchanges, trsm and
// update of the next panel's 32 columns; on su, once the panel is done: the
// interchanges and trsm of all other columns and the update of those right of
// the next panel, overlapping panel k + 1 (whose columns wait for it).
// Splitting the trailing DGEMM at a column multiple of 4 keeps BOLA's 8x4
// edge-tile classification, so every element is computed exactly as in one
// call.  Everything after a panel stops on the panel's own record of *info
// (PLAN_STOP): a zero pivot found by panel k + 1 while step k's wide update
// runs must not cut that short, which BOLA completes before factoring panel
// k + 1.
int swap_columns(cudaStream_t s, double *A, int64_t lda, int64_t j, int jb, int64_t c0, int64_t ncols, int64_t nright,
                 const int32_t *plan) {
  if (ncols <= 0) return 0;
  ProfScope prof(s, "getrf_swap_trsm", (double)jb * (jb - 1) * (double)nright, 32.0 * jb * (double)ncols);
  BOLA_TRY(roomy(step_swap_trsm));
  BOLA_TRY_CUDA(launch_after(step_swap_trsm, dim3((unsigned)cdiv(ncols, SW_WARPS)), 32 * SW_WARPS, 0, s, A, lda, j, jb, c0,
                             ncols, plan, lanes()));
  BOLA_CHECK_LAUNCH();
  return 0;
}

int getrf_blocked(cudaStream_t s, int64_t m, int64_t n, double *A, int64_t lda, int32_t *ipiv, int32_t *info) {
  const int64_t min_mn = imin(m, n);
  if (m == 0 || n == 0 || PNB >= min_mn) {
    ProfScope prof(s, "info_init");
    zero_i32<<<1, 1, 0, s>>>(info);
    BOLA_CHECK_LAUNCH();
    return m == 0 || n == 0 ? 0 : getrf2_rec(s, m, n, A, lda, ipiv, info, 0);
  }
  Scratch plans;
  BOLA_TRY(plans.alloc((size_t)cdiv(min_mn, PNB) * PLAN_INTS * sizeof(int32_t), s, true));
  // look-ahead pays from a few hundred columns on; below that its events and
  // the extra launches cost more than the overlap saves
  LookAhead *la = min_mn >= LOOK_AHEAD_MIN ? la_acquire(s) : nullptr;
  cudaStream_t sp = la ? la->sp : s, su = la ? la->su : s;
  auto run = [&]() -> int {
    if (la) {
      BOLA_TRY_CUDA(cudaEventRecord(la->ev[0], s));
      BOLA_TRY_CUDA(cudaStreamWaitEvent(sp, la->ev[0], 0));
      BOLA_TRY_CUDA(cudaStreamWaitEvent(su, la->ev[0], 0));
    }
    bool wide_pending = false;
    for (int64_t j = 0, k = 0; j < min_mn; j += PNB, ++k) {
      const int jb = (int)imin(PNB, min_mn - j);
      int32_t *plan = plans.as<int32_t>() + k * PLAN_INTS, *stop = plan + PLAN_STOP;
      BOLA_TRY(launch_panel(sp, A + j + j * lda, lda, m - j, jb, ipiv + j, info, (int32_t)j, (int32_t)j, plan, j == 0));
      const int64_t m2 = m - j - jb, n2 = n - j - jb;
      const double *A21 = A + (j + jb) + j * lda, *A12 = A + j + (j + jb) * lda;
      double *A22 = A + (j + jb) + (j + jb) * lda;
      if (!la) {
        BOLA_TRY(swap_columns(s, A, lda, j, jb, 0, n - jb, n2, plan));
        if (m2 > 0 && n2 > 0)
          BOLA_TRY(dgemm_exact(s, 'N', 'N', m2, n2, jb, -1.0, A21, lda, A12, lda, 1.0, A22, lda, 64, stop, 0));
        continue;
      }
      BOLA_TRY_CUDA(cudaEventRecord(la->ev[1], sp));
      const int64_t nn = imin((int64_t)PNB, n2);  // the next panel's columns: a multiple of 4 unless all of n2
      if (n2 > 0) {
        if (wide_pending) BOLA_TRY_CUDA(cudaStreamWaitEvent(sp, la->ev[2], 0));
        BOLA_TRY(swap_columns(sp, A, lda, j, jb, j + jb, nn, nn, plan));
        if (m2 > 0)
          BOLA_TRY(dgemm_exact(sp, 'N', 'N', m2, nn, jb, -1.0, A21, lda, A12, lda, 1.0, A22, lda, 64, stop, 0));
      }
      BOLA_TRY_CUDA(cudaStreamWaitEvent(su, la->ev[1], 0));
      BOLA_TRY(swap_columns(su, A, lda, j, jb, j + jb + nn, n2 - nn, n2 - nn, plan));
      if (n2 > nn && m2 > 0)
        BOLA_TRY(dgemm_exact(su, 'N', 'N', m2, n2 - nn, jb, -1.0, A21, lda, A12 + nn * lda, lda, 1.0, A22 + nn * lda, lda,
                             64, stop, 0));
      BOLA_TRY_CUDA(cudaEventRecord(la->ev[2], su));
      wide_pending = true;
      BOLA_TRY(swap_columns(su, A, lda, j, jb, 0, j, 0, plan));  // the finished columns, read by nothing later
    }
    if (la) {
      BOLA_TRY_CUDA(cudaEventRecord(la->ev[3], su));
      BOLA_TRY_CUDA(cudaStreamWaitEvent(sp, la->ev[3], 0));
      BOLA_TRY_CUDA(cudaEventRecord(la->ev[4], sp));
      BOLA_TRY_CUDA(cudaStreamWaitEvent(s, la->ev[4], 0));
    }
    return 0;
  };
  const int st = run();
  if (la) {
    if (st != 0) {  // leave nothing of this call running on the look-ahead streams
      cudaStreamSynchronize(la->sp);
      cudaStreamSynchronize(la->su);
    }
    la_release(la);
  }
  return st;
}

}  // namespace bola

using namespace bola;

extern "C" {

int bola_dgetrf(int64_t m, int64_t n, double *a, int64_t lda, int32_t *ipiv, int32_t *info,
                bola_stream_t stream) {
  if (m < 0) return -1;
  if (n < 0) return -2;
  if (lda < imax(m, 1)) return -4;  // "Argument 4 to getrf had an illegal value" (src/getrf.rs:41-43)
  if (imin(m, n) > INT32_MAX - 1) return -1;
  if (info == nullptr) return -6;
  return getrf_blocked((cudaStream_t)stream, m, n, a, lda, ipiv, info);
}

int bola_dgetrf2(int64_t m, int64_t n, double *a, int64_t lda, int32_t *ipiv, int32_t *info,
                 bola_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (m < 0) return -1;
  if (n < 0) return -2;
  if (lda < imax(m, 1)) return -4;  // src/getrf2.rs:43-45
  if (info == nullptr) return -6;
  {
    ProfScope prof(s, "info_init");
    zero_i32<<<1, 1, 0, s>>>(info);
  }
  BOLA_CHECK_LAUNCH();
  return getrf2_rec(s, m, n, a, lda, ipiv, info, 0);
}

int bola_dgetrs(int64_t n, int64_t nrhs, const double *lu, int64_t lda, const int32_t *ipiv, double *b,
                int64_t ldb, bola_stream_t stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (n < 0) return -1;
  if (nrhs < 0) return -2;
  if (lda < imax(1, n)) return -4;
  if (ldb < imax(1, n)) return -7;
  if (n == 0 || nrhs == 0) return 0;
  if (n > 32 && n <= GR_MAX) {
    ProfScope prof(s, "laswp", 0.0, 32.0 * (double)n * nrhs);
    const size_t smem = 16 * (size_t)n;
    if (smem > 48 * 1024)
      BOLA_TRY_CUDA(cudaFuncSetAttribute(getrs_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, 16 * (int)GR_MAX));
    BOLA_TRY_CUDA(launch_after(getrs_rows, dim3((unsigned)imin(nrhs, num_sms())), GR_T, smem, s, (int)n, nrhs, ipiv, b,
                               ldb));
  } else {
    BOLA_TRY(laswp_exact(s, nrhs, b, ldb, 1, (int32_t)n, ipiv, 1, nullptr));
  }
  BOLA_TRY(trsm_exact(s, 'L', 'L', 'N', 'U', n, nrhs, 1.0, lu, lda, b, ldb, nullptr));
  return trsm_exact(s, 'L', 'U', 'N', 'N', n, nrhs, 1.0, lu, lda, b, ldb, nullptr);
}

}  // extern "C"
