// LU factorization with partial pivoting (DecomposeLU) and the row interchanges used by
// SolveLU, on the device.
//
// Reference: lu.go:173-231 (blockedLUpiv, left-looking Crout variant), lu.go:103-171
// (unblockedLUpiv), pivot.go:27-61 (swapRows/applyPivots), pivot.go:98-107 (pivotIndex:
// first row holding the strict maximum of |x|; a NaN never wins unless it sits on the
// diagonal, where the scan starts).  The factors do not depend on left- vs right-looking
// order except through rounding, so the device runs the right-looking form:
//   panel   : up to 16384 rows one thread-block cluster, rows in registers, one exchange
//             between the CTAs per column, through distributed shared memory onto an
//             mbarrier; above, a cooperative kernel whose CTAs own slices of the panel in
//             shared memory, one grid barrier per column (candidate rows are published with
//             the local argmax, so every CTA picks the pivot itself)
//   laswp   : apply the panel's interchanges to the other columns (all of them after the
//             cluster panel, which leaves its rows where they were)
//   trsm    : U12 = L11^-1 A12 (unit lower inverse + in-place GEMM)
//   update  : A22 -= L21 U12 on the FP64 tensor pipe
#include <algorithm>
#include <climits>
#include <utility>

#include "cluster.cuh"
#include "context.cuh"
#include "lu_shape.h"
#include "tri.cuh"

namespace mo {
int trtri_blocks(mo_ctx *ctx, View A, int N, bool trans, bool lower_eff, bool unit, double *inv);

namespace {

constexpr int PANEL_THREADS = 256;
constexpr int MAX_PANEL_W = 128;

struct PanelScratch {
  // double-buffered per-CTA candidates: value, index, NaN-on-diagonal flag, row values
  double *cand_val;   // [2][nblk]
  int *cand_idx;      // [2][nblk]
  double *cand_row;   // [2][nblk][W]
  double *rowj;       // [2][W]  current contents of panel row j (published by its owner)
  int *diag_nan;      // [2]
  unsigned *barrier;  // monotonically increasing arrival counter
};

__device__ __forceinline__ bool better(double v, int i, double bv, int bi) {
  return v > bv || (v == bv && i < bi);
}

// Bounded grid barrier over `nblk` co-resident CTAs (cooperative launch).  Returns false
// after recording MO_EDEVTIMEOUT.
__device__ bool grid_barrier(unsigned *counter, unsigned target, int *status, int *abort_flag) {
  __syncthreads();
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1u);
    int ok = 1;
    unsigned i = 0;
    while (true) {
      unsigned v = *(volatile unsigned *)counter;
      if (v >= target) break;
      if (*(volatile int *)abort_flag) {
        ok = 0;
        break;
      }
      if (++i > MO_SPIN_LIMIT) {
        set_status(status, MO_EDEVTIMEOUT);
        atomicExch(abort_flag, 1);
        ok = 0;
        break;
      }
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// Factor the m x W panel P (column-major, ld) in place; piv[j] = row0 + pivot position.
// Each CTA owns rows [b*R, min((b+1)*R, m)) in shared memory (row-major, stride W+1).
__global__ void __launch_bounds__(PANEL_THREADS)
    lu_panel_kernel(double *P, int64_t ld, int m, int W, int R, int64_t *piv, int64_t row0,
                    PanelScratch sc, int *status, int *abort_flag) {
  extern __shared__ double S[];
  const int nblk = gridDim.x, b = blockIdx.x;
  const int LDW = W + 1;
  const int rbeg = b * R, rend = min(m, rbeg + R), nr = max(0, rend - rbeg);
  __shared__ double s_prow[MAX_PANEL_W];
  __shared__ double s_oldj[MAX_PANEL_W];
  __shared__ double red_v[PANEL_THREADS / 32];
  __shared__ int red_i[PANEL_THREADS / 32];
  __shared__ int red_q[PANEL_THREADS / 32];

  for (int e = threadIdx.x; e < nr * W; e += blockDim.x) {
    const int r = e % nr, c = e / nr;
    S[r * LDW + c] = P[(rbeg + r) + (int64_t)c * ld];
  }
  __syncthreads();

  const int kmax = min(m, W);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // (row, column) work of the update: G consecutive lanes per row
  int G = 32;
  while (G > 1 && G * nr > (int)blockDim.x) G >>= 1;
  for (int j = 0; j < kmax; ++j) {
    const int par = j & 1;
    // (a) local argmax of |column j| over owned positions >= j; every warp then combines
    // the warps' partials itself (no second barrier)
    double bv = -1.0;
    int bi = INT_MAX;
    for (int r = threadIdx.x; r < nr; r += blockDim.x) {
      const int gi = rbeg + r;
      if (gi < j) continue;
      double v = fabs(S[r * LDW + j]);
      if (isnan(v)) v = -1.0;  // NaN never wins off the diagonal
      if (better(v, gi, bv, bi)) {
        bv = v;
        bi = gi;
      }
    }
    for (int off = 16; off > 0; off >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, bv, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      if (better(ov, oi, bv, bi)) {
        bv = ov;
        bi = oi;
      }
    }
    if (lane == 0) {
      red_v[wid] = bv;
      red_i[wid] = bi;
    }
    __syncthreads();
    bv = lane < nw ? red_v[lane] : -1.0;
    bi = lane < nw ? red_i[lane] : INT_MAX;
    for (int off = 16; off > 0; off >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, bv, off);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, off);
      if (better(ov, oi, bv, bi)) {
        bv = ov;
        bi = oi;
      }
    }
    // (b) publish the candidate and its row and, if owned here, row j
    if (threadIdx.x == 0) {
      sc.cand_val[par * nblk + b] = bv;
      sc.cand_idx[par * nblk + b] = bi;
    }
    {
      double *crow = sc.cand_row + ((size_t)par * nblk + b) * W;
      if (bi != INT_MAX)
        for (int c = threadIdx.x; c < W; c += blockDim.x) crow[c] = S[(bi - rbeg) * LDW + c];
      if (j >= rbeg && j < rend) {
        for (int c = threadIdx.x; c < W; c += blockDim.x) sc.rowj[par * W + c] = S[(j - rbeg) * LDW + c];
        if (threadIdx.x == 0) sc.diag_nan[par] = isnan(S[(j - rbeg) * LDW + j]) ? 1 : 0;
      }
    }
    if (!grid_barrier(sc.barrier, (unsigned)(j + 1) * nblk, status, abort_flag)) return;
    // (c) every CTA selects the pivot: largest value, lowest index; NaN on the diagonal wins.
    // The candidates are read in parallel (one per thread) and reduced like the local
    // argmax, so the selection costs one L2 round trip, not one per CTA.
    int p, wb;
    {
      double v = -2.0;
      int pi = INT_MAX, wq = INT_MAX;
      for (int q = threadIdx.x; q < nblk; q += blockDim.x) {
        const double cv = __ldcg(sc.cand_val + par * nblk + q);
        const int ci = __ldcg(sc.cand_idx + par * nblk + q);
        if (ci != INT_MAX && better(cv, ci, v, pi)) {
          v = cv;
          pi = ci;
          wq = q;
        }
      }
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, v, off);
        const int oi = __shfl_xor_sync(0xffffffffu, pi, off);
        const int oq = __shfl_xor_sync(0xffffffffu, wq, off);
        if (better(ov, oi, v, pi)) {
          v = ov;
          pi = oi;
          wq = oq;
        }
      }
      if (lane == 0) {
        red_v[wid] = v;
        red_i[wid] = pi;
        red_q[wid] = wq;
      }
      __syncthreads();
      v = lane < nw ? red_v[lane] : -2.0;
      pi = lane < nw ? red_i[lane] : INT_MAX;
      wq = lane < nw ? red_q[lane] : INT_MAX;
      for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, v, off);
        const int oi = __shfl_xor_sync(0xffffffffu, pi, off);
        const int oq = __shfl_xor_sync(0xffffffffu, wq, off);
        if (better(ov, oi, v, pi)) {
          v = ov;
          pi = oi;
          wq = oq;
        }
      }
      p = pi;
      wb = pi == INT_MAX ? -1 : wq;
      if (__ldcg(sc.diag_nan + par)) {
        p = j;
        wb = -1;
      }
      if (p == INT_MAX) p = j;  // no comparable candidate: keep the row
    }
    // (d) the pivot row (U row) and the old row j, into shared memory
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
      const double oj = __ldcg(sc.rowj + par * W + c);
      s_oldj[c] = oj;
      s_prow[c] = (wb >= 0) ? __ldcg(sc.cand_row + ((size_t)par * nblk + wb) * W + c) : oj;
    }
    if (b == 0 && threadIdx.x == 0) piv[j] = row0 + p;
    __syncthreads();
    // (e) interchange rows j and p (pivot.go:27-35 on the panel columns), l = a_ij / u_jj
    // (true division, mvec.go:422 InvScale) and the rank-1 update of the owned rows below j,
    // in one pass: row j takes the pivot row; the row at p is read from the old row j
    if (p != j && j >= rbeg && j < rend)
      for (int c = threadIdx.x; c < W; c += blockDim.x) S[(j - rbeg) * LDW + c] = s_prow[c];
    const double ujj = s_prow[j];
    const int r0 = max(0, j + 1 - rbeg);  // first owned row below j
    const int grp = threadIdx.x / G, gl = threadIdx.x % G;
    // the lanes of this thread's group (G divides 32; every lane of a group runs the same
    // iterations)
    const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << (lane & ~(G - 1));
    for (int r = r0 + grp; r < nr; r += blockDim.x / G) {
      double *row = S + r * LDW;
      const bool swapped = p != j && rbeg + r == p;
      const double *src = swapped ? s_oldj : row;
      const double l = src[j] / ujj;
      __syncwarp(gmask);  // the group has read src[j] before it is overwritten
      if (swapped)
        for (int c = gl; c < j; c += G) row[c] = src[c];
      if (gl == 0) row[j] = l;
      for (int c = j + 1 + gl; c < W; c += G) row[c] = fma(-l, s_prow[c], src[c]);
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < nr * W; e += blockDim.x) {
    const int r = e % nr, c = e / nr;
    P[(rbeg + r) + (int64_t)c * ld] = S[r * LDW + c];
  }
}

// ---- the panel in one thread-block cluster ---------------------------------------------
// What bounds a panel is its chain of columns: pivot search, exchange of the pivot row,
// scaling, update, and nothing of column j + 1 can start before.  A grid barrier costs
// several L2 round trips per column (5.0 us a column with the cooperative kernel above at
// 1001 and at 16384 rows); inside a cluster the candidates and the diagonal row travel through
// distributed shared memory onto one mbarrier per CTA and column (a cluster barrier comes
// only between sub-panels).  16 CTAs x 256 threads x 4 rows hold 16384 rows of a
// 16-column sub-panel in registers; the 128 columns are done left-looking, sub-panel by
// sub-panel: a thread first applies the finished columns to its rows (L from L2, U from
// shared memory), then the 16 columns are eliminated.  Every entry takes the same FMAs in
// the same order as in a right-looking panel.
//
// Rows do not move in memory: a thread holds a logical row and its physical row, an
// interchange exchanges both between two threads, and the moves that put all columns of the
// matrix (the panel's among them) in order are emitted at the end.
//
// Measured on B200, 128 columns with the interchanges applied, against the cooperative
// kernel: 128 rows 608 -> 187 us, 1001 rows 671 -> 214, 4000 rows 698 -> 264, 8000 rows 708 ->
// 320, 16000 rows 766 -> 439 (there the FP64 rate of the 16 SMs takes over).  A column takes
// about 1000 cycles in one CTA and 1600 in a cluster, half of it the argmax and the exchange:
// 65 us of the 187 and 104 of the 214.  The rest is the triangle of U by CTA 0 alone, its way
// through global memory, and the left-looking products.
constexpr int kClWarps = kClThreads / 32, kClSub = 16;
constexpr int kClByWarp = 4, kClCands = kClByWarp * kClWarps;  // (one lane per candidate)
constexpr int kClL = MAX_PANEL_W - kClSub;  // rows of U that a later sub-panel needs
constexpr int kClLd = kClL + 2;  // a row of L^T (16-byte aligned, 4 banks from the next)

struct __align__(16) ClRow {
  double x[kClSub];       // the row's columns from the current one on
  unsigned hi, lo;        // key: bits of |x_0|
  int idx, phys;          // logical and physical row
};

struct ClSmem {
  uint64_t bar[2];            // arrival of a column's packets, by column parity
  uint64_t pad[2];
  ClRow recv[2][kClCands];    // a candidate per CTA or per warp, double-buffered by column
  ClRow rowj[2];              // the row at the diagonal
  ClRow own[kClWarps];        // this CTA's (own[0]) or each warp's candidate, for sending
  ClRow ownj;                 // (CTA 0) the diagonal row, gathered for sending
  unsigned red_hi[2][kClWarps], red_lo[2][kClWarps];
  int red_idx[2][kClWarps];
  int phys[MAX_PANEL_W];      // (CTA 0) physical rows of the logical rows < W
  __align__(16) double U[kClL * kClSub];    // finished rows of the current 16 columns
  __align__(16) double L[(kClL + 1) * kClLd];  // (CTA 0) finished rows of L, transposed
};

static_assert(sizeof(ClRow) == 9 * 16, "row packet");
static_assert(kClThreads == kClSub * kClSub && kClThreads >= MAX_PANEL_W, "index splits below");

// warp-wide largest key, lowest index on ties; every lane gets the result
__device__ __forceinline__ void cl_argmax(unsigned &hi, unsigned &lo, int &idx) {
  const unsigned h = __reduce_max_sync(0xffffffffu, hi);
  const unsigned l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
  idx = (int)__reduce_min_sync(0xffffffffu, hi == h && lo == l ? (unsigned)idx : (unsigned)INT_MAX);
  hi = h;
  lo = l;
}

// BY_WARP (at most kClByWarp CTAs): every warp sends its own candidate to every CTA, which spares
// the second argmax level and a block barrier per column; more CTAs would receive more
// candidates than a warp has lanes, and many times the bytes, so there a CTA sends one.
// Panels of LU at n = 1001: 221 -> 214 us each.
template <int RPT, bool BY_WARP>
__global__ void __launch_bounds__(kClThreads, 1)
    lu_cluster_panel_kernel(double *P, int64_t ld, int m, int W, int64_t *piv, int64_t row0,
                            double *ubuf, int *mv_dst, int *mv_src, int *mv_count,
                            int *status) {
  extern __shared__ __align__(16) unsigned char cl_raw[];
  ClSmem &s = *reinterpret_cast<ClSmem *>(cl_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nctas = gridDim.x, cta = blockIdx.x;  // one cluster: the grid is the cluster
  const int rbase = cta * kClThreads * RPT + tid;  // logical rows rbase + kClThreads q
  int phys[RPT];
#pragma unroll
  for (int q = 0; q < RPT; ++q) phys[q] = rbase + kClThreads * q;
  if (cta == 0 && tid == 0) *mv_count = W;
  if (tid == 0) {
    mbar_init(&s.bar[0], 1);
    mbar_init(&s.bar[1], 1);
    fence_barrier_init();
  }
  if (nctas > 1) cl_sync();  // every CTA has started before any writes into its memory
  for (int j0 = 0; j0 < W; j0 += kClSub) {
    const int w = min(kClSub, W - j0);
    double x[RPT][kClSub];
#pragma unroll
    for (int q = 0; q < RPT; ++q)
#pragma unroll
      for (int k = 0; k < kClSub; ++k)
        x[q][k] = (rbase + kClThreads * q < m && k < w)
                      ? __ldcg(P + phys[q] + (int64_t)(j0 + k) * ld) : 0.0;
    // LB columns of L of this thread's unfinished rows
    constexpr int LB = 8 / RPT;
    double l0[RPT][LB], l1[RPT][LB];
    auto fetch = [&](int i0, double (&l)[RPT][LB]) {
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int r = rbase + kClThreads * q;
        const double *src = P + phys[q] + (int64_t)i0 * ld;
#pragma unroll
        for (int i = 0; i < LB; ++i) l[q][i] = r >= j0 && r < m ? __ldcg(src + i * ld) : 0.0;
      }
    };
    if (j0 > 0) {
      fetch(0, l0);
      // rows < j0 of these columns: U = L^-1 A by CTA 0, 16 rows at a time
      if (cta == 0) {
        {  // the 16 newest rows of L, all loads in flight at once
          const int i = j0 - kClSub + (tid & (kClSub - 1)), k1 = tid / kClSub;
          const double *src = P + s.phys[i];
          double v[kClL / kClSub];
#pragma unroll
          for (int n = 0; n < kClL / kClSub; ++n) {
            const int k = k1 + kClSub * n;
            v[n] = k < i ? __ldcg(src + (int64_t)k * ld) : 0.0;
          }
#pragma unroll
          for (int n = 0; n < kClL / kClSub; ++n) s.L[(k1 + kClSub * n) * kClLd + i] = v[n];
        }
        if (tid < j0) {
#pragma unroll
          for (int k = 0; k < kClSub; ++k) s.U[tid * kClSub + k] = x[0][k];
        }
        __syncthreads();
        const int c = tid & (kClSub - 1), i1 = tid / kClSub;
        for (int b = 0; b < j0; b += kClSub) {
          if (tid < kClSub) {  // 16 x 16 unit lower triangle, one thread per column
            double u[kClSub];
#pragma unroll
            for (int i = 0; i < kClSub; ++i) u[i] = s.U[(b + i) * kClSub + tid];
#pragma unroll
            for (int k = 0; k + 1 < kClSub; ++k) {
              const double2 *lk = reinterpret_cast<const double2 *>(s.L + (b + k) * kClLd + b);
#pragma unroll
              for (int i2 = (k + 1) / 2; i2 < kClSub / 2; ++i2) {
                const double2 v = lk[i2];
                if (2 * i2 > k) u[2 * i2] = fma(-v.x, u[k], u[2 * i2]);
                u[2 * i2 + 1] = fma(-v.y, u[k], u[2 * i2 + 1]);
              }
            }
#pragma unroll
            for (int i = 1; i < kClSub; ++i) s.U[(b + i) * kClSub + tid] = u[i];
          }
          __syncthreads();
          // the rows below it, 16 at a time by all threads, all of a thread's rows together
          // (those past j0 compute on what the padded array holds and are not stored)
          double a[kClL / kClSub - 1];
          const int nr = (j0 - b) / kClSub - 1;
#pragma unroll
          for (int j = 0; j < kClL / kClSub - 1; ++j)
            a[j] = j < nr ? s.U[(b + kClSub * (j + 1) + i1) * kClSub + c] : 0.0;
#pragma unroll
          for (int k = 0; k < kClSub; ++k) {
            const double uk = s.U[(b + k) * kClSub + c];
            const double *lk = s.L + (b + k) * kClLd + b + kClSub + i1;
#pragma unroll
            for (int j = 0; j < kClL / kClSub - 1; ++j) a[j] = fma(-lk[kClSub * j], uk, a[j]);
          }
#pragma unroll
          for (int j = 0; j < kClL / kClSub - 1; ++j)
            if (j < nr) s.U[(b + kClSub * (j + 1) + i1) * kClSub + c] = a[j];
          __syncthreads();
        }
        for (int e = tid; e < kClSub * j0; e += kClThreads) {
          const int i = e % j0, k = e / j0;
          if (k < w) P[s.phys[i] + (int64_t)(j0 + k) * ld] = s.U[i * kClSub + k];
        }
        if (nctas > 1)
          for (int e = tid; e < j0 * kClSub; e += kClThreads) ubuf[e] = s.U[e];
      }
      if (nctas > 1) {
        cl_sync();
        if (cta != 0) {
          for (int e = tid; e < j0 * kClSub; e += kClThreads) s.U[e] = __ldcg(ubuf + e);
          __syncthreads();
        }
      }
      // rows >= j0 take the finished columns, a batch of them while the next batch's L is on
      // its way (the first one was requested before U)
      auto apply = [&](int i0, const double (&l)[RPT][LB]) {
#pragma unroll
        for (int i = 0; i < LB; ++i) {
          const double2 *u = reinterpret_cast<const double2 *>(s.U + (i0 + i) * kClSub);
#pragma unroll
          for (int k = 0; k < kClSub / 2; ++k) {
            const double2 v = u[k];
#pragma unroll
            for (int q = 0; q < RPT; ++q) {
              x[q][2 * k] = fma(-l[q][i], v.x, x[q][2 * k]);
              x[q][2 * k + 1] = fma(-l[q][i], v.y, x[q][2 * k + 1]);
            }
          }
        }
      };
#pragma unroll 1
      for (int i0 = 0; i0 < j0; i0 += 2 * LB) {
        fetch(i0 + LB, l1);
        apply(i0, l0);
        if (i0 + 2 * LB < j0) fetch(i0 + 2 * LB, l0);
        apply(i0 + LB, l1);
      }
    }
    // Eliminate the columns.  The loop is rolled (the registers shift by one column per turn:
    // x[q][0] is always the current one): with the 16 columns unrolled every instruction
    // ran once per sub-panel and the fetches, not the arithmetic, set the time.  A finished
    // multiplier goes straight to its physical row in memory.
    unsigned hi = 0, lo = 0;
    int idx = INT_MAX;
    // this thread's largest |x_0| among the rows >= jc (pivot.go:98-107): first index of the
    // maximum; a NaN wins only on the diagonal, where its bits exceed every number's
    auto search = [&](int jc) {
      hi = lo = 0u;
      idx = INT_MAX;
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int r = rbase + kClThreads * q;
        const unsigned long long bits = __double_as_longlong(fabs(x[q][0]));
        const bool nan = bits > 0x7ff0000000000000ull && r != jc;
        const unsigned h2 = nan ? 0u : (unsigned)(bits >> 32), l2 = nan ? 0u : (unsigned)bits;
        if (r >= jc && r < m && (idx == INT_MAX || h2 > hi || (h2 == hi && l2 > lo))) {
          hi = h2;
          lo = l2;
          idx = r;
        }
      }
    };
    search(j0);
#pragma unroll 1
    for (int c = 0; c < w; ++c) {
      const int jc = j0 + c, par = jc & 1;
      // this column's packets: one candidate per CTA and the diagonal row
      if (nctas > 1 && tid == 0)
        mbar_arrive_expect_tx(&s.bar[par],
                              (uint32_t)((nctas * (BY_WARP ? kClWarps : 1) + 1) * sizeof(ClRow)));
      cl_argmax(hi, lo, idx);
      // the candidate row, from its owner's registers
      auto gather = [&](ClRow &to) {
        if (idx == INT_MAX && lane == 0) {  // no row left in this CTA (warp)
          to.hi = to.lo = 0u;
          to.idx = INT_MAX;
        }
#pragma unroll
        for (int q = 0; q < RPT; ++q)
          if (rbase + kClThreads * q == idx) {
#pragma unroll
            for (int k = 0; k < kClSub; ++k) to.x[k] = x[q][k];
            to.hi = hi;
            to.lo = lo;
            to.idx = idx;
            to.phys = phys[q];
          }
        __syncwarp();
      };
      if constexpr (BY_WARP) {
        gather(nctas > 1 ? s.own[warp] : s.recv[par][warp]);
        if (nctas > 1)
          cl_send<9, 32 / kClByWarp>(&s.recv[par][cta * kClWarps + warp], &s.own[warp],
                                     &s.bar[par], lane, nctas);
      } else if (lane == 0) {
        s.red_hi[par][warp] = hi;
        s.red_lo[par][warp] = lo;
        s.red_idx[par][warp] = idx;
      }
      // the diagonal row (always one of CTA 0's first rows) goes out beside the search
      if (cta == 0 && warp == jc / 32) {
        ClRow &to = nctas > 1 ? s.ownj : s.rowj[par];
        if (tid == jc) {
#pragma unroll
          for (int k = 0; k < kClSub; ++k) to.x[k] = x[0][k];
          to.phys = phys[0];
        }
        __syncwarp();
        if (nctas > 1) cl_send<9>(&s.rowj[par], &s.ownj, &s.bar[par], lane, nctas);
      }
      if constexpr (!BY_WARP) {
        __syncthreads();
        hi = s.red_hi[par][lane & (kClWarps - 1)];
        lo = s.red_lo[par][lane & (kClWarps - 1)];
        idx = s.red_idx[par][lane & (kClWarps - 1)];
        cl_argmax(hi, lo, idx);
        // this CTA's candidate to every CTA
        if (warp == (idx == INT_MAX ? 0 : (idx & (kClThreads - 1)) >> 5)) {
          gather(s.own[0]);
          cl_send<9>(&s.recv[par][cta], &s.own[0], &s.bar[par], lane, nctas);
        }
      }
      // every warp picks the pivot: largest key, lowest row
      // (a wait that runs out is recorded; the kernel goes on with what it holds)
      if (nctas > 1) mbar_wait(&s.bar[par], (jc >> 1) & 1, status);
      else __syncthreads();
      const int cands = BY_WARP ? nctas * kClWarps : nctas;
      const ClRow &cand = s.recv[par][lane < cands ? lane : 0];
      hi = cand.hi;
      lo = cand.lo;
      idx = cand.idx;
      cl_argmax(hi, lo, idx);
      const int p = min(max(idx, jc), m - 1);  // (idx itself, unless a wait ran out)
      const ClRow &pr = s.recv[par][p / (BY_WARP ? 32 : kClThreads * RPT)];
      if (cta == 0 && warp == kClWarps - 1) {  // the U row, and the pivot
        if (lane < w - c)
          P[min(max(pr.phys, 0), m - 1) + (int64_t)(jc + lane) * ld] = pr.x[lane];
        if (lane == 0) piv[jc] = row0 + p;
      }
      double u[kClSub];
#pragma unroll
      for (int k = 0; k < kClSub / 2; ++k) {
        const double2 v = reinterpret_cast<const double2 *>(pr.x)[k];
        u[2 * k] = v.x;
        u[2 * k + 1] = v.y;
      }
      if (p != jc && (warp == ((p & (kClThreads - 1)) >> 5) || warp == jc / 32)) {
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const int r = rbase + kClThreads * q;
          if (r == p) {
#pragma unroll
            for (int k = 0; k < kClSub; ++k) x[q][k] = s.rowj[par].x[k];
            phys[q] = min(max(s.rowj[par].phys, 0), m - 1);
          } else if (r == jc) {
            phys[q] = min(max(pr.phys, 0), m - 1);
          }
        }
      }
      // l = a / u (true division, mvec.go:422 InvScale) and the rank-1 update, on every row
      // (the rows <= jc hold nothing that is read again)
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const int r = rbase + kClThreads * q;
        const double l = x[q][0] / u[0];
        if (r > jc && r < m) P[phys[q] + (int64_t)jc * ld] = l;
#pragma unroll
        for (int k = 0; k + 1 < kClSub; ++k) x[q][k] = fma(-l, u[k + 1], x[q][k + 1]);
      }
      search(jc + 1);
    }
    if (cta == 0 && tid < MAX_PANEL_W) s.phys[tid] = phys[0];
    // the stores are visible to the rows' later owners
    if (nctas > 1) cl_sync();
    else __syncthreads();
  }
  // the moves: the W rows of the block in order, then every other row that changed place
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int r = rbase + kClThreads * q;
    if (r >= m) continue;
    int at = r;
    if (r >= W) {
      if (phys[q] == r) continue;
      at = atomicAdd(mv_count, 1);
    }
    mv_dst[at] = (int)row0 + r;
    mv_src[at] = (int)row0 + phys[q];
  }
}

const void *cl_kernel(int ctas, int rpt) {
  return ctas <= kClByWarp ? (const void *)lu_cluster_panel_kernel<1, true>
         : rpt == 1        ? (const void *)lu_cluster_panel_kernel<1, false>
         : rpt == 2        ? (const void *)lu_cluster_panel_kernel<2, false>
                           : (const void *)lu_cluster_panel_kernel<4, false>;
}

int cl_config(int ctas, int rpt, cudaStream_t st, cudaLaunchConfig_t *cfg,
              cudaLaunchAttribute *attr) {
  const void *fn = cl_kernel(ctas, rpt);
  if (int rc = mo_smem_attr(fn, (int)sizeof(ClSmem))) return rc;
  MO_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(ctas);
  cfg->blockDim = dim3(kClThreads);
  cfg->dynamicSmemBytes = sizeof(ClSmem);
  cfg->stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim = {(unsigned)ctas, 1, 1};
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return MO_OK;
}

// Apply interchanges rows (r0+s) <-> piv[s] (absolute rows of A), s = 0..ns-1 in order,
// to columns [0, ncols) of A; one thread per column.  Out-of-range pivots are reported.
__global__ void laswp_kernel(double *A, int64_t ld, int rows, int ncols, const int64_t *piv,
                             int ns, int64_t r0, int *status) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  double *col = A + (int64_t)c * ld;
  for (int s = 0; s < ns; ++s) {
    const int64_t p = piv[s];
    const int64_t q = r0 + s;
    if (p <= 0 || p == q) continue;  // pivot.go:57: entries <= 0 are skipped
    if (p >= rows || q >= rows) {
      if (c == 0) set_status(status, MO_EINVAL);
      continue;
    }
    const double t = col[q];
    col[q] = col[p];
    col[p] = t;
  }
}

// The net effect of the interchanges rows (r0 + s) <-> piv[s], s = 0 .. ns - 1 in order
// (pivot.go:55-61, entries <= 0 skipped) on the rows they touch: rows r0 .. r0 + ns - 1 and
// the distinct pivot rows beyond them.  One warp simulates the swaps on row labels and
// writes the moves dst[i] <- src[i] (i < *count), so that one pass of loads and one of
// stores applies all of them to any set of columns.  ns <= MAX_PANEL_W.
__global__ void __launch_bounds__(32) swap_map_kernel(const int64_t *piv, int ns, int64_t r0,
                                                      int rows, int *dst, int *src, int *count,
                                                      int *status) {
  __shared__ int lab[2 * MAX_PANEL_W];   // source row now held at each position
  __shared__ int ext[MAX_PANEL_W];       // rows beyond the block, in order of first use
  __shared__ int next;
  const int lane = threadIdx.x;
  for (int i = lane; i < ns; i += 32) lab[i] = (int)(r0 + i);
  if (lane == 0) next = 0;
  __syncwarp();
  for (int s = 0; s < ns; ++s) {
    const int64_t p = piv[s];
    const int64_t q = r0 + s;
    if (p <= 0 || p == q) continue;
    if (p >= rows || q >= rows) {
      if (lane == 0) set_status(status, MO_EINVAL);
      continue;
    }
    int pos;
    if (p < r0 + ns) {
      pos = (int)(p - r0);
    } else {
      const int ne = next;
      int found = -1;
      for (int b = 0; b < ne; b += 32) {
        const unsigned hit = __ballot_sync(0xffffffffu, b + lane < ne && ext[b + lane] == (int)p);
        if (hit) {
          found = b + __ffs(hit) - 1;
          break;
        }
      }
      if (found < 0) {
        found = ne;
        if (lane == 0) {
          ext[ne] = (int)p;
          lab[ns + ne] = (int)p;
          next = ne + 1;
        }
      }
      pos = ns + found;
    }
    __syncwarp();
    if (lane == 0) {
      const int t = lab[s];
      lab[s] = lab[pos];
      lab[pos] = t;
    }
    __syncwarp();
  }
  const int total = ns + next;
  for (int i = lane; i < total; i += 32) {
    dst[i] = i < ns ? (int)(r0 + i) : ext[i - ns];
    src[i] = lab[i];
  }
  if (lane == 0) *count = total;
}

// swap_map_kernel for panels whose rows [r0, rows) fit a shared-memory table (label per
// position, touched flag): the pivots are read in parallel, one thread applies the swaps
// to the table in order (a few shared-memory operations each, no warp-wide search), and
// the moves are written in the same form and order as swap_map_kernel's.
constexpr int kSwapTableMax = 32768;
__global__ void __launch_bounds__(256) swap_map_table_kernel(const int64_t *piv, int ns, int64_t r0,
                                                             int rows, int *dst, int *src,
                                                             int *count, int *status) {
  extern __shared__ int tb[];
  const int span = rows - (int)r0;
  int *lab = tb;                                             // [span]
  int *ext = lab + span;                                     // [MAX_PANEL_W]
  int *pv = ext + MAX_PANEL_W;                               // [MAX_PANEL_W]
  unsigned char *touched = reinterpret_cast<unsigned char *>(pv + MAX_PANEL_W);  // [span]
  __shared__ int next;
  for (int i = threadIdx.x; i < span; i += blockDim.x) {
    lab[i] = (int)r0 + i;
    touched[i] = 0;
  }
  for (int i = threadIdx.x; i < ns; i += blockDim.x) {
    const int64_t p = piv[i];
    // -1: skipped (pivot.go:57, entries <= 0, or no exchange); -2: out of range
    pv[i] = (p <= 0 || p == r0 + i) ? -1 : ((p >= rows || p < r0 || r0 + i >= rows) ? -2 : (int)(p - r0));
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int ne = 0;
    bool bad = false;
    for (int s2 = 0; s2 < ns; ++s2) {
      const int pi = pv[s2];
      if (pi == -1) continue;
      if (pi == -2) {
        bad = true;
        continue;
      }
      const int t = lab[s2];
      lab[s2] = lab[pi];
      lab[pi] = t;
      if (pi >= ns && !touched[pi]) {
        touched[pi] = 1;
        ext[ne++] = pi;
      }
    }
    if (bad) set_status(status, MO_EINVAL);
    next = ne;
  }
  __syncthreads();
  const int total = ns + next;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int pos = i < ns ? i : ext[i - ns];
    dst[i] = (int)r0 + pos;
    src[i] = lab[pos];
  }
  if (threadIdx.x == 0) *count = total;
}

// A[dst[i], c] = A_old[src[i], c] for a panel's moves, columns [0, ncols): a CTA takes 32 columns, a
// thread one move (at most 2 MAX_PANEL_W of them), all its 32 loads in flight, then a barrier,
// then the stores.  What bounds it at many columns is the scattered half of the rows, a 32-byte
// sector per element (16384 columns: 130 us); 1001 columns take 7 us, 21 with a division per element and the values
// passed through shared memory.
__global__ void __launch_bounds__(2 * MAX_PANEL_W) laswp_map_kernel(double *A, int64_t ld, int ncols,
                                                                    const int *dst, const int *src,
                                                                    const int *count) {
  const int i = threadIdx.x, c0 = blockIdx.x * 32;
  const bool mine = i < *count;
  double v[32];
  const double *from = A + (mine ? src[i] : 0) + (int64_t)c0 * ld;
#pragma unroll
  for (int c = 0; c < 32; ++c) v[c] = mine && c0 + c < ncols ? from[c * ld] : 0.0;
  __syncthreads();
  if (!mine) return;
  double *to = A + dst[i] + (int64_t)c0 * ld;
#pragma unroll
  for (int c = 0; c < 32; ++c)
    if (c0 + c < ncols) to[c * ld] = v[c];
}

// All interchanges rows s <-> piv[s] (s = 0 .. ns - 1, in order) on a few columns of B
// (SolveLU's applyPivots): one CTA per column, the column in shared memory, one thread
// applying the swaps in order.
__global__ void __launch_bounds__(256) laswp_cols_kernel(double *B, int64_t ld, int rows,
                                                         const int64_t *piv, int ns, int *status) {
  extern __shared__ double col[];
  double *g = B + (int64_t)blockIdx.x * ld;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) col[i] = g[i];
  // the pivots come through shared memory, a part at a time (read one by one from global memory
  // they set the pace: 240 cycles a swap); an entry that is not applied becomes its own row
  constexpr int kPart = 1024;
  __shared__ int part[kPart];
  for (int s0 = 0; s0 < ns; s0 += kPart) {
    const int np = min(kPart, ns - s0);
    __syncthreads();
    for (int i = threadIdx.x; i < np; i += blockDim.x) {
      const int64_t p = piv[s0 + i];
      const bool out = p > 0 && p != s0 + i && (p >= rows || s0 + i >= rows);
      if (out && blockIdx.x == 0) set_status(status, MO_EINVAL);
      part[i] = p <= 0 || out ? s0 + i : (int)p;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int i = 0; i < np; ++i) {
        const int s = s0 + i, p = part[i];
        if (p == s) continue;
        const double t = col[s];
        col[s] = col[p];
        col[p] = t;
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < rows; i += blockDim.x) g[i] = col[i];
}

// Keeps its stream busy for about ns nanoseconds (at most 1000 naps of 100 ns).
__global__ void head_start_kernel(int ns) {
  for (int i = 0; i < min(ns / 100, 1000); ++i) __nanosleep(100);
}

// piv[i] = v for i in [lo, hi)
__global__ void fill_pivots_kernel(int64_t *piv, int64_t lo, int64_t hi, int64_t v) {
  const int64_t i = lo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < hi) piv[i] = v;
}

struct CtrlView {
  int status;
  int info;
  double bad;
};

}  // namespace

int laswp(mo_ctx *ctx, View A, int c0, int c1, const int64_t *piv, int ns, int64_t r0) {
  if (c1 <= c0 || ns <= 0) return MO_OK;
  const int nc = c1 - c0;
  ProfScope ps;
  prof_begin(ctx, ps, MO_PROF_LASWP);
  laswp_kernel<<<(nc + 127) / 128, 128, 0, ctx->stream>>>(
      A.at(0, c0), A.ld, A.rows, nc, piv, ns, r0,
      &reinterpret_cast<CtrlView *>(ctx->d_status)->status);
  prof_end(ctx, ps, 0.0, 4.0 * 8.0 * ns * (double)nc);
  MO_CUDA_TRY(cudaGetLastError());
  return MO_OK;
}

// SolveLU's applyPivots(B, pivots) (lu.go:322, pivot.go:55-61)
int laswp_forward(mo_ctx *ctx, View B, const int64_t *piv, int64_t npiv) {
  if (B.rows == 0 || B.cols == 0 || npiv <= 0) return MO_OK;
  if (npiv > INT_MAX) return MO_EINVAL;
  const size_t smem = (size_t)B.rows * sizeof(double);
  if (smem > 200 * 1024) return laswp(ctx, B, 0, B.cols, piv, (int)npiv, 0);
  if (int rc = mo_smem_attr((const void *)laswp_cols_kernel, (int)smem)) return rc;
  ProfScope ps;
  prof_begin(ctx, ps, MO_PROF_LASWP);
  laswp_cols_kernel<<<B.cols, 256, smem, ctx->stream>>>(
      B.d, B.ld, B.rows, piv, (int)npiv,
      &reinterpret_cast<CtrlView *>(ctx->d_status)->status);
  prof_end(ctx, ps, 0.0, 16.0 * B.rows * (double)B.cols);
  MO_CUDA_TRY(cudaGetLastError());
  return MO_OK;
}

// the panel's interchanges on columns [c0, c1) of A through its move list
int laswp_moves(mo_ctx *ctx, View A, int c0, int c1, const int *dst, const int *src,
                const int *count) {
  if (c1 <= c0) return MO_OK;
  const int nc = c1 - c0;
  ProfScope ps;
  prof_begin(ctx, ps, MO_PROF_LASWP);
  laswp_map_kernel<<<(nc + 31) / 32, 2 * MAX_PANEL_W, 0, ctx->stream>>>(A.at(0, c0), A.ld, nc, dst,
                                                                        src, count);
  prof_end(ctx, ps, 0.0, 16.0 * 2 * MAX_PANEL_W * (double)nc);
  MO_CUDA_TRY(cudaGetLastError());
  return MO_OK;
}

int getrf(mo_ctx *ctx, View A, int64_t *piv, int64_t npiv, int ref_nb) {
  const int m = A.rows, n = A.cols, mn = min(m, n);
  int *status = &reinterpret_cast<CtrlView *>(ctx->d_status)->status;
  // panel width and rows per CTA: keep the panel slice <= ~200 KB of shared memory
  int W = MAX_PANEL_W;
  const int max_blocks = ctx->sms;
  auto rows_per_block = [&](int) {
    int nblk = min(max_blocks, max(1, (m + 63) / 64));
    return std::pair<int, int>((m + nblk - 1) / nblk, nblk);
  };
  auto smem_for = [](int R, int w) { return (size_t)R * (w + 1) * sizeof(double); };
  auto rb = rows_per_block(W);
  while (smem_for(rb.first, W) > 200 * 1024 && W > 8) {
    W /= 2;
    rb = rows_per_block(W);
  }
  if (smem_for(rb.first, W) > 200 * 1024) return MO_EINVAL;  // > ~3.2M rows
  const int R = rb.first, nblk = rb.second;
  // later (shorter) panels may use up to 64 rows per CTA
  const size_t smem = smem_for(std::max(R, 64), W);
  MO_CUDA_TRY(cudaFuncSetAttribute(lu_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)smem));
  int occ = 0;
  MO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, lu_panel_kernel, PANEL_THREADS,
                                                            smem));
  if (occ * ctx->sms < nblk) return MO_EINVAL;

  // workspace: panel scratch + L11 inverse
  const size_t sz_val = 2 * nblk * sizeof(double), sz_idx = 2 * nblk * sizeof(int);
  const size_t sz_row = (size_t)2 * nblk * W * sizeof(double), sz_rowj = 2 * W * sizeof(double);
  const size_t inv_bytes = 2 * 128 * 128 * sizeof(double);  // two panels' L11 inverses
  const size_t sz_moves = 2 * (2 * (2 * MAX_PANEL_W) * sizeof(int) + 64);  // two panels'
  const size_t sz_ubuf = (size_t)kClL * kClSub * sizeof(double);
  const size_t total =
      inv_bytes + sz_ubuf + sz_val + sz_row + sz_rowj + sz_idx + 64 + 64 + sz_moves;
  char *ws = nullptr;
  int rc = workspace(ctx, total, (void **)&ws);
  if (rc) return rc;
  double *inv = (double *)ws, *inv_b = inv + 128 * 128;
  PanelScratch sc;
  double *ubuf = (double *)(ws + inv_bytes);
  char *q = ws + inv_bytes + sz_ubuf;
  sc.cand_val = (double *)q;
  q += sz_val;
  sc.cand_row = (double *)q;
  q += sz_row;
  sc.rowj = (double *)q;
  q += sz_rowj;
  sc.cand_idx = (int *)q;
  q += sz_idx;
  sc.diag_nan = (int *)q;
  q += 16;
  sc.barrier = (unsigned *)q;
  q += 16;
  int *abort_flag = (int *)q;
  q += 32;
  // the moves of a pair's two panels; own: the panel's own columns are still to be put in order
  struct Moves {
    int *dst, *src, *count;
    bool own;
  } mv[2];
  for (Moves &v : mv) {
    v.dst = (int *)q;
    v.src = v.dst + 2 * MAX_PANEL_W;
    v.count = v.src + 2 * MAX_PANEL_W;
    v.own = false;
    q += 2 * (2 * MAX_PANEL_W) * sizeof(int) + 64;
  }

  // CTAs and rows up to which a panel may run in one cluster.  More than 8 CTAs are not portable
  // (a part of a device may not place them): ask, once per context, where they would be used.
  int cl_ctas = kClPortable;
  if (m > kClThreads * kClPortable) {
    if (ctx->lu_ctas == 0) {
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute attr;
      int clusters = 0;
      if ((rc = cl_config(kClMaxCtas, kClMaxRpt, ctx->stream, &cfg, &attr))) return rc;
      if (cudaOccupancyMaxActiveClusters(&clusters, cl_kernel(kClMaxCtas, kClMaxRpt), &cfg) ==
              cudaSuccess &&
          clusters > 0) {
        ctx->lu_ctas = kClMaxCtas;
      } else {
        cudaGetLastError();
        ctx->lu_ctas = kClPortable;
      }
    }
    cl_ctas = ctx->lu_ctas;
  }
  const int cl_rows = cl_max_rows(cl_ctas);
  // one panel: factor A[k:m, k:k+b] and list its interchanges
  auto panel = [&](int k, int b, Moves &v) -> int {
    v.own = m - k <= cl_rows;
    if (v.own) {
      int rpt;
      const int ctas = cl_shape(m - k, cl_ctas, &rpt);
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute attr;
      int r2 = cl_config(ctas, rpt, ctx->stream, &cfg, &attr);
      if (r2) return r2;
      ProfScope ps;
      prof_begin(ctx, ps, MO_PROF_PANEL);
      double *Pd = A.at(k, k);
      int64_t pld = A.ld, *pv = piv + k, row0 = k;
      int pm = m - k, pw = b;
      void *args[] = {&Pd, &pld, &pm, &pw, &pv, &row0, &ubuf, &v.dst, &v.src, &v.count, &status};
      const cudaError_t e = cudaLaunchKernelExC(&cfg, cl_kernel(ctas, rpt), args);
      prof_end(ctx, ps, (double)(m - k) * b * b - (double)b * b * b / 3.0, 16.0 * (m - k) * b);
      MO_CUDA_TRY(e);
      return MO_OK;
    }
    MO_CUDA_TRY(cudaMemsetAsync(sc.barrier, 0, 32, ctx->stream));  // barrier + abort flag
    View Pv = A.sub(k, k, m - k, b);
    const int pm = m - k;
    int pblk = min(nblk, max(1, (pm + 63) / 64));
    int pR = (pm + pblk - 1) / pblk;
    int64_t *pv = piv + k;
    int64_t row0 = k;
    double *pd = Pv.d;
    int64_t pld = Pv.ld;
    int pw = b;
    void *args[] = {&pd, &pld, (void *)&pm, &pw, &pR, &pv, &row0, &sc, &status, &abort_flag};
    ProfScope ps;
    prof_begin(ctx, ps, MO_PROF_PANEL);
    MO_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)lu_panel_kernel, dim3(pblk),
                                            dim3(PANEL_THREADS), args, smem, ctx->stream));
    prof_end(ctx, ps, (double)pm * b * b - (double)b * b * b / 3.0, 16.0 * pm * b);
    if (n <= b) return MO_OK;  // no other columns to interchange rows in
    ProfScope pms;
    prof_begin(ctx, pms, MO_PROF_LASWP);
    if (m - k <= kSwapTableMax) {
      const size_t tsm = (size_t)(m - k) * 5 + 2 * MAX_PANEL_W * sizeof(int) + 16;
      int r2 = mo_smem_attr((const void *)swap_map_table_kernel, (int)tsm);
      if (r2) return r2;
      swap_map_table_kernel<<<1, 256, tsm, ctx->stream>>>(piv + k, b, k, m, v.dst, v.src, v.count,
                                                          status);
    } else {
      swap_map_kernel<<<1, 32, 0, ctx->stream>>>(piv + k, b, k, m, v.dst, v.src, v.count, status);
    }
    prof_end(ctx, pms, 0.0, 8.0 * b);
    MO_CUDA_TRY(cudaGetLastError());
    return MO_OK;
  };
  // a panel's interchanges on the columns [c0, c1)
  auto swap = [&](int k, int b, const Moves &v, int c0, int c1) -> int {
    if (v.own) return laswp_moves(ctx, A, c0, c1, v.dst, v.src, v.count);
    int r2 = laswp_moves(ctx, A, c0, std::min(c1, k), v.dst, v.src, v.count);
    if (!r2) r2 = laswp_moves(ctx, A, std::max(c0, k + b), c1, v.dst, v.src, v.count);
    return r2;
  };
  // Panels in pairs: the first is factored, the second one's columns are brought up to date with
  // it (U01 = inv0 A01, A[k2:m, P1] -= L[k2:m, P0] U01), the second is factored.  The
  // interchanges are applied to the columns [c0, c1).
  auto pair = [&](int k, int b0, int b1, int c0, int c1, const GemmOpts &o) -> int {
    const int k2 = k + b0;
    int r = panel(k, b0, mv[0]);
    if (!r) r = swap(k, b0, mv[0], c0, c1);
    if (!r && n > k2) r = trtri_blocks(ctx, A.sub(k, k, b0, b0), b0, false, true, true, inv);
    if (r || b1 == 0) return r;
    View U01 = A.sub(k, k2, b0, b1);
    r = gemm_ex(ctx, U01, View{inv, b0, b0, 128}, false, U01, false, 1.0, 0.0, o);
    if (!r)
      r = gemm_ex(ctx, A.sub(k2, k2, m - k2, b1), A.sub(k2, k, m - k2, b0), false, U01, false, -1.0,
                  1.0, o);
    if (!r) r = panel(k2, b1, mv[1]);
    if (!r) r = swap(k2, b1, mv[1], c0, c1);
    if (!r && n > k2 + b1)
      r = trtri_blocks(ctx, A.sub(k2, k2, b1, b1), b1, false, true, true, inv_b);
    return r;
  };
  // Then the rows of the pair right of it become U (two small products and one b1-row update
  // between them) and the rest of the matrix takes one update with K = b0 + b1, so the
  // trailing matrix is read and written once per pair.
  //
  // Look-ahead: a pair is a chain of columns on one cluster (up to 16 SMs) and took as long as
  // half of the update it waited for.  While the rest is wide, the next pair's columns are
  // updated first and the pair is factored on the auxiliary stream, its interchanges applied
  // to its own columns only, beside the update of the rest on the other SMs; the
  // interchanges of the other columns follow.  The update is enqueued behind an event of the
  // auxiliary stream that precedes the panel and a 5 us nap, so that the panel's cluster, which
  // needs 16 free SMs in one part of the chip, is placed before the update fills it (without
  // the nap the update mostly came first and the panel waited for its end).  Measured on B200,
  // DecomposeLU: n = 16384 159.8 -> 130.1 ms, 8000 33.7 -> 26.6, 4000 10.8 -> 10.0, 3000 7.6 -> 7.3;
  // below 1024 rows or columns of rest there is nothing to hide behind (n = 2000: no change).
  constexpr int kAheadMin = 1024;
  cudaStream_t s1 = nullptr;
  bool ahead = false;  // the pair at k is being factored on the auxiliary stream
  for (int k = 0; k < mn; k += 2 * W) {
    const int b0 = min(W, mn - k);
    const int k2 = k + b0;
    const int b1 = k2 < mn ? min(W, mn - k2) : 0;
    const int kc = k2 + b1;
    const int c_rest = n - kc;  // columns right of the pair
    if (ahead) {
      if ((rc = stream_wait(ctx, ctx->stream, s1, ctx->ev_join))) return rc;
      if ((rc = swap(k, b0, mv[0], 0, k)) || (rc = swap(k, b0, mv[0], kc, n))) return rc;
      if (b1 > 0 && ((rc = swap(k2, b1, mv[1], 0, k)) || (rc = swap(k2, b1, mv[1], kc, n)))) return rc;
      ahead = false;
    } else if ((rc = pair(k, b0, b1, 0, n, GemmOpts()))) {
      return rc;
    }
    if (c_rest <= 0) continue;
    // rows k..k2 of the columns right of the pair: U0T = inv0 A0T
    View U0T = A.sub(k, kc, b0, c_rest);
    if ((rc = gemm(ctx, U0T, View{inv, b0, b0, 128}, false, U0T, false, 1.0, 0.0))) return rc;
    if (b1 > 0) {
      // rows k2..kc: A1T -= L10 U0T, then U1T = inv1 A1T
      View U1T = A.sub(k2, kc, b1, c_rest);
      if ((rc = gemm(ctx, U1T, A.sub(k2, k, b1, b0), false, U0T, false, -1.0, 1.0))) return rc;
      if ((rc = gemm(ctx, U1T, View{inv_b, b1, b1, 128}, false, U1T, false, 1.0, 0.0))) return rc;
    }
    // the rest: A[kc:m, kc:n] -= L[kc:m, k:kc] U[k:kc, kc:n]  (K = b0 + b1)
    const int rest_r = m - kc;
    if (rest_r <= 0) continue;
    const View Lp = A.sub(kc, k, rest_r, b0 + b1);
    auto update = [&](int c0, int nc, const GemmOpts &o) {
      return gemm_ex(ctx, A.sub(kc, c0, rest_r, nc), Lp, false, A.sub(k, c0, b0 + b1, nc), false, -1.0,
                     1.0, o);
    };
    const int nb0 = kc < mn ? min(W, mn - kc) : 0;
    const int nb1 = kc + nb0 < mn ? min(W, mn - kc - nb0) : 0;
    const int nn = nb0 + nb1;
    ahead = nb1 > 0 && rest_r <= cl_rows && c_rest - nn >= kAheadMin && rest_r >= kAheadMin;
    if (!ahead) {
      if ((rc = update(kc, c_rest, GemmOpts()))) return rc;
      continue;
    }
    if ((rc = update(kc, nn, GemmOpts()))) return rc;
    cudaStream_t s0 = ctx->stream;
    if (!s1 && (rc = aux_stream(ctx, &s1))) return rc;
    if ((rc = stream_wait(ctx, s1, s0, ctx->ev_fork))) return rc;
    if ((rc = stream_wait(ctx, s0, s1, ctx->ev_join))) return rc;
    {
      StreamSwap sw(ctx, s1);
      GemmOpts o;
      o.stream_k = false;  // the stream-K scratch is the main stream's
      o.max_ctas = kClMaxCtas;
      if ((rc = pair(kc, nb0, nb1, kc, kc + nn, o))) return rc;
    }
    head_start_kernel<<<1, 1, 0, s0>>>(5000);
    MO_CUDA_TRY(cudaGetLastError());
    GemmOpts o;
    o.max_ctas = ctx->sms - kClMaxCtas;
    if ((rc = update(kc + nn, c_rest - nn, o))) return rc;
  }
  // The reference's blocked path (mlen > nb, nb != 0) leaves the pivot entries past
  // min(rows, cols) inside the last block equal to that block's start row (lu.go:216-219).
  if (ref_nb > 0 && mn > ref_nb && npiv > mn) {
    int64_t k_last = 0;
    for (int64_t k = 0; k < m && k < n;) {
      k_last = k;
      k += (k + ref_nb > n) ? n - k : ref_nb;
    }
    const int64_t hi = std::min<int64_t>(npiv, k_last + ref_nb);
    if (hi > mn) {
      ProfScope ps;
      prof_begin(ctx, ps, MO_PROF_OTHER);
      fill_pivots_kernel<<<(unsigned)((hi - mn + 255) / 256), 256, 0, ctx->stream>>>(piv, mn, hi,
                                                                                     k_last);
      prof_end(ctx, ps, 0.0, 8.0 * (hi - mn));
    }
    MO_CUDA_TRY(cudaGetLastError());
  }
  return MO_OK;
}

}  // namespace mo
