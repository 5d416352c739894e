// Batched Cholesky / LU factor + solve of many small FP64 systems of uneven order
// (n <= MO_BATCH_MAX_N) in one persistent launch per schedule group, replayed from a CUDA
// graph.  The reference factors one matrix per call (DecomposeCHOL chol.go:116,
// DecomposeLU lu.go:257, SolveCHOL chol.go:147, SolveLU lu.go:320); here each CTA takes
// whole matrices from a work queue ordered by decreasing n^3 (longest job first) and
// runs, for each one:
//
//   Cholesky (lower, left-looking, 32-column panels): every warp takes 32 x 32 tiles of the
//     panel, C - L(rows, 0:j) L(j:j+32, 0:j)^T with the accumulators kept in registers; one
//     warp factors and inverts the diagonal tile (a NaN pivot stops the matrix with info =
//     column + 1, where the reference panics, chol.go:33-36); the other tiles are multiplied by
//     the inverse straight from their accumulators and stored, so a panel is read and written
//     once.
//   LU (partial pivoting, 64-column blocks):
//     panel  : 16-column sub-panels with the rows in registers, left-looking inside the block
//              (the scheme of the single-matrix panel, one CTA): per column an argmax of |a|
//              with ties to the lowest row (pivotIndex, pivot.go:98-107), the pivot row
//              through shared memory, true division by the pivot
//     swaps  : an interchange exchanges two rows' labels; rows are put in order once, at the
//              end
//     U12    : by 32 rows with the inverses of L11's diagonal blocks, a warp per 32 columns;
//              also written row-major to the CTA's scratch for the update
//     update : A22 -= L21 U12, a warp per 16 rows, L21 in registers, U12 in shared memory
//   solve (when B is given): forward and backward substitution per right-hand side, 32-row
//     blocks: a warp solves the diagonal block by shuffles, the other rows are updated in
//     axpy form (columns of the factor are read contiguously)
//
// All products run on the FP64 tensor pipe (mma.sync m16n8k4), most fragments loaded straight
// from global memory: a fragment row is 8 consecutive elements of four columns.
//
// What bounds it: the chain of columns and blocks of each matrix, so many matrices have to be
// in flight per SM -- four CTAs of 128 threads or two of 256 -- and every step that only a
// few warps can do is kept short.  Measured on B200, 4096 systems n ~ U{16..512}, 1 RHS,
// against right-looking 32-column panels with shared-memory staging (diagonal block, panel
// substitution and solve by division chains; LU panels unrolled over 32 columns):
// Cholesky 9.8 -> 5.8 ms, LU 42.7 -> 16.9; 512 x n = 256 Cholesky 0.60 -> 0.29 ms, LU 3.5 -> 1.3;
// 1024 x n = 128 Cholesky 0.38 -> 0.13, LU 2.28 -> 0.57.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "context.cuh"

namespace mo {
namespace {

constexpr int MAXN = MO_BATCH_MAX_N;
constexpr int CB = 32;     // Cholesky panel, and the blocks of the solves
constexpr int LB = 64;     // LU block
constexpr int SB = 16;     // LU sub-panel
// row stride of the LU scratch: 33 lines of 128 bytes (512 elements apart, a fragment's rows
// would meet in the same L1 sets)
constexpr int UTLD = MAXN + 16;
constexpr int ULD = 36;    // row stride of a U12 tile in shared memory (fragments: no conflicts)

struct BatchParams {
  int count;                 // matrices in this group's queue
  const int *order;          // queue: indices into the arrays below
  int *counter;              // next queue position (reset to 0 before each launch)
  const int *n;              // order of each matrix
  double *const *A;          // device pointers to the matrices
  const int64_t *lda;
  double *const *B;          // right-hand sides (nullptr: factor only)
  const int64_t *ldb;
  int nrhs;
  int64_t *const *piv;       // LU pivots (0-based absolute row, LAPACK convention)
  int *info;                 // per matrix: 0 or column + 1 of the failing pivot
  double *ut;                // LU: per-CTA scratch, LB x UTLD doubles each
};

struct CholSmem {
  double D[CB][CB + 1];      // diagonal tile: updated, then its factor
  double It[CB][CB + 2];     // transposed inverse, It[k][n] = Linv(n, k)
  double col[16][16];        // columns of a 16 x 16 factor, zero on and above the diagonal
  double vec[MAXN];          // solve vector
  int idx, info;
};
// LARGE (orders above 128): with the running C of the tile that each tile warp has in hand, in
// fragment order
template <int T, bool LARGE>
struct CholTiles : CholSmem {
  double C[LARGE ? T / 32 * 3 / 4 : 1][LARGE ? CB * CB : 1];
};

static_assert(2 * LB * ULD <= (LB + 6) * (LB + 2), "two U12 tiles fit where L11 was");
struct LuRow {
  double x[SB];
  int phys;
};
struct LuSmem {
  double U[(LB - SB) * SB];       // finished rows of the current 16 columns
  // L11 transposed, L[k][i] = L11(i, k); its 32 x 32 diagonal blocks become their inverses
  // for U12 (also the buffer of the final row order, and the solve's block and vector)
  __align__(16) double L[LB + 6][LB + 2];
  LuRow prow[2];                  // pivot row, by column parity
  unsigned red_hi[2][16], red_lo[2][16];
  int red_idx[2][16];
  int label[MAXN];                // physical row -> logical row
  int perm[MAXN];                 // logical row -> physical row (finished rows; at the end all)
  int act[MAXN];                  // unfinished physical rows, ascending
  int idx, info, swapped;
};

__device__ __forceinline__ double neg(double x) { return -x; }

// acc (32 x 32: rows 16 mi + g + 8 h, columns 8 ni + 2 t + e at acc[mi][ni][2 h + e]) +=
// sum over k of P(row, k) Q(column, k), K a multiple of 4, P and Q read from global memory in
// fragment layout: `pa`, `pb` point at this lane's first element (row g, column g; k = t4).
// fold() after every FOLD columns but the last ones.
template <int FOLD, typename F>
__device__ __forceinline__ void tile_mma(double (&acc)[2][4][4], const double *pa, const double *pb,
                                         int64_t ld, int K, F &&fold) {
  double a[2][2][2], b[2][4];
  const int64_t step = 4 * ld;
  auto load = [&](int s) {
#pragma unroll
    for (int mi = 0; mi < 2; ++mi) {
      a[s][mi][0] = pa[16 * mi];
      a[s][mi][1] = pa[16 * mi + 8];
    }
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) b[s][ni] = pb[8 * ni];
    pa += step;
    pb += step;
  };
  auto mma = [&](int s) {
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
        dmma_16x8x4(acc[mi][ni], a[s][mi][0], a[s][mi][1], b[s][ni]);
  };
  if (K <= 0) return;
  load(0);
#pragma unroll 1
  for (int k = 0; k < K; k += 8) {  // K is a multiple of 8 (of a panel's 32 columns)
    load(1);
    mma(0);
    if (k + 8 < K) load(0);
    mma(1);
    if ((k & (FOLD - 1)) == FOLD - 8 && k + 8 < K) fold();
  }
}

// Cholesky factor and inverse of the 16 x 16 block of s.D at (b, b) by one warp: lane i (and
// lane i + 16) holds row i, then column i of the inverse.  Two columns per step, every lane
// factoring the 2 x 2 pivot block itself.  Leaves the factor in s.D and its transposed inverse
// in s.It (`inverse`); returns the block's first NaN pivot or -1.
__device__ __forceinline__ int chol_diag16(CholSmem &s, int b, bool inverse) {
  const int lane = threadIdx.x & 31, i16 = lane & 15;
  double r[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) r[k] = k <= i16 ? s.D[b + i16][b + k] : 0.0;
  double pivot = 1.0, rd = 1.0;  // this lane's diagonal entry before its root, and 1 / root
#pragma unroll
  for (int k = 0; k < 16; k += 2) {
    const double a = __shfl_sync(0xffffffffu, r[k], k);
    const double m = __shfl_sync(0xffffffffu, r[k], k + 1);
    const double c = __shfl_sync(0xffffffffu, r[k + 1], k + 1);
    const double rs1 = rsqrt(a), l21 = m * rs1, d = fma(-l21, l21, c), rs2 = rsqrt(d);
    const double x1 = i16 > k ? r[k] * rs1 : 0.0;
    const double x2 = i16 > k + 1 ? fma(-x1, l21, r[k + 1]) * rs2 : 0.0;
    if (i16 == k) {
      pivot = a;
      rd = rs1;
    }
    if (i16 == k + 1) {
      pivot = d;
      rd = rs2;
    }
    if (lane < 16) {
      s.col[k][lane] = x1;
      s.col[k + 1][lane] = x2;
    }
    __syncwarp();
#pragma unroll
    for (int j = k + 2; j < 16; ++j)
      r[j] = fma(-x2, s.col[k + 1][j], fma(-x1, s.col[k][j], r[j]));
    r[k] = x1;
    r[k + 1] = x2;
  }
  const double dg = sqrt(pivot);
  const unsigned bad = __ballot_sync(0xffffffffu, isnan(dg));
  if (bad) return __ffs(bad) - 1;
  if (lane < 16) {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k <= i16) s.D[b + i16][b + k] = k == i16 ? dg : r[k];
  }
  if (!inverse) {
    __syncwarp();
    return -1;
  }
  // column i16 of the inverse: L x = e
  double x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    double s0 = i == i16 ? 1.0 : 0.0, s1 = 0.0;
#pragma unroll
    for (int m = 0; m + 1 < i; m += 2) {
      s0 = fma(-s.col[m][i], x[m], s0);
      s1 = fma(-s.col[m + 1][i], x[m + 1], s1);
    }
    if (i & 1) s0 = fma(-s.col[i - 1][i], x[i - 1], s0);
    x[i] = (s0 + s1) * __shfl_sync(0xffffffffu, rd, i);
  }
  if (lane < 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) s.It[b + lane][b + i] = i < lane ? 0.0 : x[i];
  }
  __syncwarp();
  return -1;
}

// Factor the updated diagonal tile s.D at column j (padded with the identity here) by one warp,
// write it to Ad and, unless it is the matrix's last, leave its transposed inverse in s.It: two
// 16 x 16 blocks on FP64 FMAs and the rest as DMMA products.  (One 32 x 32 block in registers had
// to give up either its loads in flight or its registers under the 128 of this kernel: 36 to
// 41 K cycles.)
__device__ __noinline__ void chol_diag(CholSmem &s, double *Ad, int64_t ld, int j, int n) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int jb = min(CB, n - j);
  if (jb < CB) {
    for (int k = 0; k < CB; ++k)
      if (lane >= jb || k >= jb) s.D[lane][k] = lane == k ? 1.0 : 0.0;
    __syncwarp();
  }
  // The last tile's inverse is not needed, and an order up to 64 that ends in at most 16 columns is
  // done with its first block (with the padding behind it a zero last pivot in its column 16
  // would be 0 times infinity).  One matrix per launch: order 8 10.3 -> 8.3 us, order 33 (with a
  // copy of it) 29.1 -> 25.0.
  const bool last = j + CB >= n, one = jb <= 16 && j + jb <= 64;
  int bad = chol_diag16(s, 0, !one);
  if (bad < 0 && !one) {
    // C (16 x 16, fragments) += sign P Q, element functions of (row, k) and (k, column)
    auto mm = [&](double (&c)[2][4], auto &&P, auto &&Q) {
#pragma unroll
      for (int k = t4; k < 16; k += 4) {
        const double a0 = P(g, k), a1 = P(g + 8, k);
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) dmma_16x8x4(c[ni], a0, a1, Q(k, 8 * ni + g));
      }
      __syncwarp();
    };
    auto put = [&](const double (&c)[2][4], auto &&at) {
#pragma unroll
      for (int ni = 0; ni < 2; ++ni)
#pragma unroll
        for (int q = 0; q < 4; ++q) at(g + 8 * (q >> 1), 8 * ni + 2 * t4 + (q & 1), c[ni][q]);
      __syncwarp();
    };
    {  // L21 = A21 X11^T
      double c[2][4] = {};
      mm(c, [&](int i, int k) { return s.D[16 + i][k]; }, [&](int k, int n) { return s.It[k][n]; });
      put(c, [&](int i, int n, double v) { s.D[16 + i][n] = v; });
    }
    {  // A22 -= L21 L21^T
      double c[2][4] = {};
      mm(c, [&](int i, int k) { return s.D[16 + i][k]; },
         [&](int k, int n) { return s.D[16 + n][k]; });
      put(c, [&](int i, int n, double v) { s.D[16 + i][16 + n] -= v; });
    }
    bad = chol_diag16(s, 16, !last);
    if (bad >= 0) {
      bad += 16;
    } else if (!last) {
      {  // M = L21 X11, into the unused upper right block
        double c[2][4] = {};
        mm(c, [&](int i, int k) { return s.D[16 + i][k]; },
           [&](int k, int n) { return s.It[n][k]; });
        put(c, [&](int i, int n, double v) { s.D[i][16 + n] = v; });
      }
      {  // X21 = -X22 M
        double c[2][4] = {};
        mm(c, [&](int i, int k) { return s.It[16 + k][16 + i]; },
           [&](int k, int n) { return s.D[k][16 + n]; });
        put(c, [&](int i, int n, double v) { s.It[n][16 + i] = neg(v); });
      }
    }
  }
  if (bad >= 0) {
    if (lane == 0) s.info = j + bad + 1;
    return;
  }
#pragma unroll 4
  for (int k = 0; k < jb; ++k)
    if (lane >= k && lane < jb) Ad[lane + (int64_t)k * ld] = s.D[lane][k];
}

// In-place lower Cholesky of one n x n matrix; returns 0 or info = column + 1.  Warp 0 factors
// and inverts the diagonal tiles; the warps of the other three schedulers hold the panel's
// tiles, and the first of them also updates the next diagonal tile as soon as its own tile
// (the same rows) is stored, so that warp 0 works on it while the others apply the finished
// columns to their tiles of the next panel.  No tile warp shares warp 0's scheduler: beside
// one warp of DMMAs a chain of FP64 FMAs is starved (512 of them take 200 K cycles instead
// of 4.3 K; 1.5 M beside three).
template <int T, bool LARGE>
__device__ int chol_matrix(CholTiles<T, LARGE> &s, double *A, int64_t ld, int n) {
  constexpr int NT = T / 32 * 3 / 4;  // warps with panel tiles
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tw = warp % 4 ? warp - warp / 4 : 0;  // 1 .. NT: tile warps; 0: diagonal or idle
  const int g = lane >> 2, t4 = lane & 3;
  if (tid == 0) s.info = 0;
  // f(index in fragment order, row and column in the tile, accumulator)
  auto each = [&](double (&acc)[2][4][4], auto &&f) {
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          f(((mi * 4 + ni) * 4 + q) * 32 + lane, 16 * mi + g + 8 * (q >> 1),
            8 * ni + 2 * t4 + (q & 1), acc[mi][ni][q]);
  };
  // acc = L(rows r0.., 0 .. K) L(j .. j + 32, 0 .. K)^T, added up from zero.  LARGE: take(acc) takes the
  // sum of every 32 columns but the last from the running C, so that C is rounded once per
  // panel and shrinks from panel to panel, as in a right-looking factorization.  Error of L
  // against one (geometric means), at diagonally dominant matrices of order 256 and 400, and
  // at a condition of 1e6: with C in the accumulators, rounded by every product, 1.24 1.51,
  // 1.55 1.93; all products from zero 0.75 0.76, 1.98 2.57; this way 0.73 0.76, 0.94 0.91.
  // Times are the same as with C in the accumulators (512 x 256 0.29 ms, 600 x 512 3.1 -> 3.0); up to
  // 128 columns the plain sum is 8 % faster and the difference small (order 128: 0.73, 1.38).
  constexpr int kFold = LARGE ? CB : MAXN;
  auto apply = [&](double (&acc)[2][4][4], int r0, int j, int K, auto &&take) {
    // (rows past n: the reads stay inside the matrix, since k < j < n and ld > 31 here, and
    // what they bring is not stored)
    const double *base = A + g + (int64_t)t4 * ld;
    each(acc, [](int, int, int, double &v) { v = 0.0; });
    tile_mma<kFold>(acc, base + r0, base + j, ld, K, [&] {
      take(acc);
      each(acc, [](int, int, int, double &v) { v = 0.0; });
    });
  };
  // the diagonal tile's C, on its way to s.D meanwhile
  auto fetch_d = [&](int r0) {
#pragma unroll 4
    for (int c = 0; c < CB; ++c) {
      const bool in = r0 + lane < n && lane >= c;
      cp_async_8(&s.D[lane][c], in ? A + r0 + lane + (int64_t)(r0 + c) * ld : A, in ? 8 : 0);
    }
  };
  if (tw == 1) {
    fetch_d(0);
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  for (int j = 0; j < n; j += CB) {
    const int nt = (n - j + CB - 1) / CB;  // 32-row tiles of the panel, tile 0 diagonal
    __syncthreads();                       // the previous panel is stored, the diagonal tile ready
    if (tw == 0) {
      if (warp == 0) chol_diag(s, A + j + (int64_t)j * ld, ld, j, n);
      __syncthreads();
      if (s.info) return s.info;
      continue;
    }
    bool waited = false;
    for (int t = tw; t < nt || !waited; t += NT) {
      double acc[2][4][4];
      const int r0 = j + t * CB;
      if (t < nt) {
        // acc = L L^T - C; the panel becomes -acc L11^-T
        double *At = A + r0 + (int64_t)j * ld;
        auto in = [&](int r, int c) { return r0 + r < n && j + c < n && r0 + r >= j + c; };
        const bool folds = LARGE && j > kFold;
        double *C = s.C[LARGE ? tw - 1 : 0];
        if (folds)
          each(acc, [&](int e, int r, int c, double &) {
            cp_async_8(C + e, in(r, c) ? At + r + (int64_t)c * ld : A, in(r, c) ? 8 : 0);
          });
        apply(acc, r0, j, j, [&](double (&d)[2][4][4]) {
          asm volatile("cp.async.wait_all;" ::: "memory");
          each(d, [&](int e, int, int, double &v) { C[e] -= v; });
        });
        if (folds) {
          asm volatile("cp.async.wait_all;" ::: "memory");
          each(acc, [&](int e, int, int, double &v) { v -= C[e]; });
        } else {
          each(acc, [&](int, int r, int c, double &v) {
            if (in(r, c)) v -= At[r + (int64_t)c * ld];
          });
        }
      }
      if (!waited) {
        waited = true;
        __syncthreads();
        if (s.info) return s.info;
      }
      if (t >= nt) continue;
      // X = -acc L11^-T: the accumulators are A fragments as they stand (lane t4 holds the
      // columns 8 ni + 2 t4 + e, so a k-step takes k = 8 ni + 2 t4 + e, e = 0 or 1)
#pragma unroll
      for (int mi = 0; mi < 2; ++mi) {
        double x[4][4] = {};
#pragma unroll
        for (int nk = 0; nk < 4; ++nk)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const double *it = s.It[8 * nk + 2 * t4 + e];
#pragma unroll
            for (int ni = nk; ni < 4; ++ni)
              dmma_16x8x4(x[ni], acc[mi][nk][e], acc[mi][nk][2 + e], it[8 * ni + g]);
          }
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int r = r0 + 16 * mi + g + 8 * (q >> 1);
            if (r < n) A[r + (int64_t)(j + 8 * ni + 2 * t4 + (q & 1)) * ld] = neg(x[ni][q]);
          }
      }
      if (t == 1) {  // the next diagonal tile: these rows, and the columns just stored too
        __syncwarp();
        fetch_d(r0);
        auto take = [&](double (&d)[2][4][4]) {
          asm volatile("cp.async.wait_all;" ::: "memory");
          __syncwarp();
          each(d, [&](int, int r, int c, double &v) { s.D[r][c] -= v; });
        };
        apply(acc, r0, r0, r0, take);
        take(acc);
      }
    }
  }
  __syncthreads();
  return 0;
}

// warp-wide largest key, lowest index on ties
__device__ __forceinline__ void warp_argmax(unsigned &hi, unsigned &lo, int &idx) {
  const unsigned h = __reduce_max_sync(0xffffffffu, hi);
  const unsigned l = __reduce_max_sync(0xffffffffu, hi == h ? lo : 0u);
  idx = (int)__reduce_min_sync(0xffffffffu, hi == h && lo == l ? (unsigned)idx : 0x7fffffffu);
  hi = h;
  lo = l;
}

// s.act = the physical rows whose label is >= lo, ascending (one warp)
__device__ __forceinline__ void lu_compact(LuSmem &s, int n, int lo) {
  const int lane = threadIdx.x & 31;
  int at = 0;
  for (int r0 = 0; r0 < n; r0 += 32) {
    const bool in = r0 + lane < n && s.label[r0 + lane] >= lo;
    const unsigned m = __ballot_sync(0xffffffffu, in);
    if (in) s.act[at + __popc(m & ((1u << lane) - 1u))] = r0 + lane;
    at += __popc(m);
  }
}

// The unit lower 32 x 32 triangle at (jo, jo) on the rows of ut, 32 columns from c0, by forward
// substitution, a lane per column, the result also to A (one warp): for right-hand sides with
// an infinity or a NaN, which the zeros of an inverse would carry into the rows above
__device__ __noinline__ void lu_substitute(const int *perm, double *A, int64_t ld, int n, int jo,
                                           double *ut, int c0) {
  const int c = c0 + (threadIdx.x & 31);
  for (int i = 0; i < CB; ++i) {
    double v = ut[(int64_t)i * UTLD + c];
    const double *l = A + perm[jo + i] + (int64_t)jo * ld;
    for (int k = 0; k < i; ++k) v = fma(-l[(int64_t)k * ld], ut[(int64_t)k * UTLD + c], v);
    ut[(int64_t)i * UTLD + c] = v;
    if (c < n) A[perm[jo + i] + (int64_t)c * ld] = v;
  }
  __syncwarp();
}

// U12 = L11^-1 A12 for the 64-row block at jo, by 32 rows: U_0 = inv(L_00) A_0, U_1 = inv(L_11)
// (A_1 - L_10 U_0), a warp per 32 columns; written to the rows' physical places and row-major
// into ut
template <int T>
__device__ __noinline__ void lu_u12(LuSmem &s, double *A, int64_t ld, int n, int jo, double *ut) {
  constexpr int NW = T / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  for (int c0 = jo + LB + CB * warp; c0 < n; c0 += CB * NW) {
    auto zero = [&](double (&acc)[2][4][4]) {
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[mi][ni][q] = 0.0;
    };
    // acc += M^T-stored (mt[k][i], row stride `lm`) times the 32 x 32 block whose element
    // (k, column 8 ni + g) is b(k, ni)
    auto product = [&](double (&acc)[2][4][4], const double *mt, int lm, auto &&b) {
#pragma unroll 4
      for (int k = t4; k < CB; k += 4) {
        double bv[4];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) bv[ni] = b(k, ni);
#pragma unroll
        for (int mi = 0; mi < 2; ++mi) {
          const double a0 = mt[k * lm + 16 * mi + g], a1 = mt[k * lm + 16 * mi + g + 8];
#pragma unroll
          for (int ni = 0; ni < 4; ++ni) dmma_16x8x4(acc[mi][ni], a0, a1, bv[ni]);
        }
      }
    };
    // the block's rows h .. h + 31: to A and to ut
    auto store = [&](const double (&acc)[2][4][4], int h, double sign, bool out) {
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
          const int i = h + 16 * mi + g + 8 * hh;
          const int64_t phys = s.perm[jo + i];
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int c = c0 + 8 * ni + 2 * t4 + e;
              const double v = sign * acc[mi][ni][2 * hh + e];
              ut[(int64_t)i * UTLD + c] = v;  // (columns past n stay within the scratch row)
              if (out && c < n) A[phys + (int64_t)c * ld] = v;
            }
        }
      __syncwarp();
    };
    auto from_ut = [&](int h) {
      return [=](int k, int ni) { return ut[(int64_t)(h + k) * UTLD + c0 + 8 * ni + g]; };
    };
    double acc[2][4][4];
    int top = 0;  // largest exponent among the right-hand sides in hand
    auto seen = [&](double v) {
      top = max(top, __double2hiint(v) & 0x7fffffff);
      return v;
    };
    auto odd = [&] { return __any_sync(0xffffffffu, top >= 0x7ff00000); };
    zero(acc);
    product(acc, &s.L[0][0], LB + 2, [&](int k, int ni) {
      return seen(A[s.perm[jo + k] + (int64_t)min(c0 + 8 * ni + g, n - 1) * ld]);
    });
    if (odd()) {
      const int c = min(c0 + lane, n - 1);
      for (int i = 0; i < CB; ++i)
        ut[(int64_t)i * UTLD + c0 + lane] = A[s.perm[jo + i] + (int64_t)c * ld];
      __syncwarp();
      lu_substitute(s.perm, A, ld, n, jo, ut, c0);
      top = 0;
    } else {
      store(acc, 0, 1.0, true);
    }
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int q = 0; q < 4; ++q)
          acc[mi][ni][q] = neg(A[s.perm[jo + CB + 16 * mi + g + 8 * (q >> 1)] +
                                 (int64_t)min(c0 + 8 * ni + 2 * t4 + (q & 1), n - 1) * ld]);
    product(acc, &s.L[0][CB], LB + 2, from_ut(0));
#pragma unroll
    for (int mi = 0; mi < 2; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int q = 0; q < 4; ++q) seen(acc[mi][ni][q]);
    store(acc, CB, -1.0, false);
    if (odd()) {
      lu_substitute(s.perm, A, ld, n, jo + CB, ut + (int64_t)CB * UTLD, c0);
      continue;
    }
    zero(acc);
    product(acc, &s.L[CB][CB], LB + 2, from_ut(CB));
    __syncwarp();  // every lane has read ut's rows before they are replaced
    store(acc, CB, 1.0, true);
  }
}

// In-place LU with partial pivoting of one n x n matrix, n <= T RPT.  piv[k] receives the
// 0-based row exchanged with row k.  Returns 0 or the first column + 1 whose pivot is exactly
// zero (the factorization still completes, as LAPACK's dgetrf does; the reference does not
// check).  A NaN is never chosen as a pivot; a column without a comparable entry keeps its
// row.  On return s.perm holds the row map (logical row r came from physical row perm[r] of
// the input).
//
// Rows never move before the end: an interchange exchanges two rows' labels.  A thread keeps
// its physical rows (ascending, so that neighbours read neighbours) for a whole block, and the
// update runs over the unfinished physical rows in ascending order.
template <int T, int RPT>
__device__ int lu_matrix(LuSmem &s, double *A, int64_t ld, int n, int64_t *piv, double *ut) {
  constexpr int NW = T / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  for (int r = tid; r < n; r += T) s.label[r] = s.act[r] = r;
  if (tid == 0) {
    s.info = 0;
    s.swapped = 0;
  }
  __syncthreads();
  for (int jo = 0; jo < n; jo += LB) {
    const int W = min(LB, n - jo), m = n - jo;
    int phys[RPT], lab[RPT];  // this thread's rows; label -1: none
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int i = tid + T * q;
      phys[q] = i < m ? s.act[i] : 0;
      lab[q] = i < m ? s.label[phys[q]] : -1;
    }
    for (int j0 = jo; j0 < jo + W; j0 += SB) {
      const int w = min(SB, jo + W - j0), s0 = j0 - jo;
      double x[RPT][SB];
#pragma unroll
      for (int q = 0; q < RPT; ++q)
#pragma unroll
        for (int k = 0; k < SB; ++k)
          x[q][k] = (lab[q] >= j0 && k < w) ? A[phys[q] + (int64_t)(j0 + k) * ld] : 0.0;
      if (s0 > 0) {
        // the finished rows jo .. j0 of these columns: U = L^-1 A, 16 rows at a time
#pragma unroll 4
        for (int e = tid; e < SB * s0; e += T) {
          const int i = e % s0, k = e / s0;
          s.U[i * SB + k] = k < w ? A[s.perm[jo + i] + (int64_t)(j0 + k) * ld] : 0.0;
          const int i2 = s0 - SB + (e & (SB - 1)), k2 = e / SB;
          if (k2 < i2) s.L[k2][i2] = A[s.perm[jo + i2] + (int64_t)(jo + k2) * ld];
        }
        __syncthreads();
        for (int b = 0; b < s0; b += SB) {
          if (tid < SB) {
            double u[SB];
#pragma unroll
            for (int i = 0; i < SB; ++i) u[i] = s.U[(b + i) * SB + tid];
#pragma unroll
            for (int k = 0; k + 1 < SB; ++k)
#pragma unroll
              for (int i = k + 1; i < SB; ++i) u[i] = fma(-s.L[b + k][b + i], u[k], u[i]);
#pragma unroll
            for (int i = 1; i < SB; ++i) s.U[(b + i) * SB + tid] = u[i];
          }
          __syncthreads();
          for (int e = tid; e < (s0 - b - SB) * SB; e += T) {
            const int i = b + SB + e / SB, c = e & (SB - 1);
            double a = s.U[i * SB + c];
#pragma unroll
            for (int k = 0; k < SB; ++k) a = fma(-s.L[b + k][i], s.U[(b + k) * SB + c], a);
            s.U[i * SB + c] = a;
          }
          __syncthreads();
        }
        for (int e = tid; e < SB * s0; e += T) {
          const int i = e % s0, k = e / s0;
          if (k < w) A[s.perm[jo + i] + (int64_t)(j0 + k) * ld] = s.U[i * SB + k];
        }
        // the unfinished rows take the finished columns of the block
#pragma unroll 1
        for (int i0 = 0; i0 < s0; i0 += 8) {
          double l[RPT][8];
#pragma unroll
          for (int q = 0; q < RPT; ++q) {
            const double *src = A + phys[q] + (int64_t)(jo + i0) * ld;
#pragma unroll
            for (int i = 0; i < 8; ++i) l[q][i] = lab[q] >= j0 ? src[i * ld] : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int k = 0; k < SB; ++k) {
              const double u = s.U[(i0 + i) * SB + k];
#pragma unroll
              for (int q = 0; q < RPT; ++q) x[q][k] = fma(-l[q][i], u, x[q][k]);
            }
        }
      }
      // Eliminate the columns; rolled, the registers shifting by one column per turn (x[q][0]
      // is the current one), so that the instructions stay in the cache.  A finished
      // multiplier goes straight to its physical row in memory.
      unsigned hi = 0, lo = 0;
      int idx = 0x7fffffff;
      auto search = [&](int jc) {
        hi = lo = 0u;
        idx = 0x7fffffff;
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const unsigned long long bits = __double_as_longlong(fabs(x[q][0]));
          const unsigned h2 = (unsigned)(bits >> 32), l2 = (unsigned)bits;
          if (lab[q] >= jc && bits <= 0x7ff0000000000000ull &&
              (h2 > hi || (h2 == hi && (l2 > lo || (l2 == lo && lab[q] < idx))))) {
            hi = h2;
            lo = l2;
            idx = lab[q];
          }
        }
      };
      search(j0);
#pragma unroll 1
      for (int c = 0; c < w; ++c) {
        const int jc = j0 + c, par = jc & 1;
        warp_argmax(hi, lo, idx);
        if (lane == 0) {
          s.red_hi[par][warp] = hi;
          s.red_lo[par][warp] = lo;
          s.red_idx[par][warp] = idx;
        }
        __syncthreads();
        hi = s.red_hi[par][lane & (NW - 1)];
        lo = s.red_lo[par][lane & (NW - 1)];
        idx = s.red_idx[par][lane & (NW - 1)];
        warp_argmax(hi, lo, idx);
        const int p = idx == 0x7fffffff ? jc : idx;
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          if (lab[q] == p) {
#pragma unroll
            for (int k = 0; k < SB; ++k) s.prow[par].x[k] = x[q][k];
            s.prow[par].phys = phys[q];
            lab[q] = jc;
          } else if (lab[q] == jc) {
            lab[q] = p;
          }
        }
        __syncthreads();
        double u[SB];
#pragma unroll
        for (int k = 0; k < SB; ++k) u[k] = s.prow[par].x[k];
        if (warp == NW - 1) {
          const int64_t pr = s.prow[par].phys;
          if (lane < w - c) A[pr + (int64_t)(jc + lane) * ld] = s.prow[par].x[lane];
          if (lane == 0) {
            piv[jc] = p;
            s.perm[jc] = (int)pr;
            if (p != jc) s.swapped = 1;
            if (u[0] == 0.0 && s.info == 0) s.info = jc + 1;
          }
        }
#pragma unroll
        for (int q = 0; q < RPT; ++q) {
          const double l = x[q][0] / u[0];
          if (lab[q] > jc) A[phys[q] + (int64_t)jc * ld] = l;
#pragma unroll
          for (int k = 0; k + 1 < SB; ++k) x[q][k] = fma(-l, u[k + 1], x[q][k + 1]);
        }
        search(jc + 1);
      }
      __syncthreads();
    }
    const int j1 = jo + LB, m2 = n - j1;
    if (m2 <= 0) break;
#pragma unroll
    for (int q = 0; q < RPT; ++q)
      if (lab[q] >= 0) s.label[phys[q]] = lab[q];
#pragma unroll 4
    for (int e = tid; e < LB * LB; e += T) {
      const int i = e & (LB - 1), k = e / LB;
      if (k < i) s.L[k][i] = A[s.perm[jo + i] + (int64_t)(jo + k) * ld];
    }
    __syncthreads();
    if (warp < 2) {
      // inverse of a unit lower 32 x 32 block in place, lane c its column c (rolled, shifting):
      // turn k writes inv(k, c) to L[c][k], and L11's column c was read at turn c <= k
      const int b = CB * warp;
      double r[CB];
#pragma unroll
      for (int i = 0; i < CB; ++i) r[i] = i == lane ? 1.0 : 0.0;
#pragma unroll 1
      for (int k = 0; k < CB; ++k) {
        const double xk = r[0];
        const double *col = s.L[b + k] + b;
#pragma unroll
        for (int i = 0; i + 1 < CB; ++i) r[i] = fma(-col[k + 1 + i], xk, r[i + 1]);
        __syncwarp();
        s.L[b + lane][b + k] = xk;  // (zero while k < lane)
      }
    } else if (warp == 2) {
      lu_compact(s, n, j1);
    }
    __syncthreads();
    lu_u12<T>(s, A, ld, n, jo, ut);
    __syncthreads();
    // A22 -= L21 U12: a warp takes 16 unfinished rows at a time, holds their 64 columns of L21
    // as fragments and goes along the columns, 32 at a time, all warps together: U12's 64 x 32
    // tile is copied to shared memory (where L11 was) one tile ahead of its use
    auto stage = [&](int c0, int buf) {
      for (int e = tid; e < LB * 16; e += T) {
        const int k = e >> 4, c = 2 * (e & 15);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(
                         &s.L[0][0] + buf * (LB * ULD) + k * ULD + c)),
                     "l"(ut + (int64_t)k * UTLD + c0 + c)
                     : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int ib = 0; ib < m2; ib += 16 * NW) {
      const int i0 = ib + 16 * warp;
      stage(j1, 0);
      double a[LB / 4][2];
      double *row[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        row[h] = A + s.act[min(i0 + g + 8 * h, m2 - 1)];
        const double *src = row[h] + (int64_t)(jo + t4) * ld;
#pragma unroll
        for (int k = 0; k < LB / 4; ++k) a[k][h] = src[(int64_t)(4 * k) * ld];
      }
      const bool in0 = i0 + g < m2, in1 = i0 + g + 8 < m2;
      int buf = 0;
#pragma unroll 1
      for (int c0 = j1; c0 < n; c0 += 32, buf ^= 1) {
        if (c0 + 32 < n) {
          stage(c0 + 32, buf ^ 1);
          asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        double acc[4][4];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int c = c0 + 8 * ni + 2 * t4 + (q & 1);
            acc[ni][q] = (q >> 1 ? in1 : in0) && c < n ? neg(row[q >> 1][(int64_t)c * ld]) : 0.0;
          }
        if (c0 + 32 + lane < n) {  // the next 32 columns of these rows, one column per lane
          asm volatile("prefetch.global.L2 [%0];" ::"l"(row[0] + (int64_t)(c0 + 32 + lane) * ld));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(row[1] + (int64_t)(c0 + 32 + lane) * ld));
        }
        __syncthreads();
        const double *pb = &s.L[0][0] + buf * (LB * ULD) + t4 * ULD + g;
#pragma unroll
        for (int k = 0; k < LB / 4; ++k)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni)
            dmma_16x8x4(acc[ni], a[k][0], a[k][1], pb[4 * k * ULD + 8 * ni]);
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int c = c0 + 8 * ni + 2 * t4 + (q & 1);
            if ((q >> 1 ? in1 : in0) && c < n) row[q >> 1][(int64_t)c * ld] = neg(acc[ni][q]);
          }
        __syncthreads();
      }
    }
    __syncthreads();
  }
  // put the rows in their final order through shared memory, a few columns at a time:
  // physical row r holds logical row label
  if (s.swapped) {
    double *buf = &s.L[0][0];
    constexpr int CH = (int)(sizeof(s.L) / (MAXN * sizeof(double)));
    for (int r = tid; r < n; r += T) s.label[s.perm[r]] = r;
    __syncthreads();
    for (int c0 = 0; c0 < n; c0 += CH) {
      const int nc = min(CH, n - c0);
      for (int r = tid; r < n; r += T) {
        const int to = s.label[r];
        double v[CH];
#pragma unroll
        for (int c = 0; c < CH; ++c) v[c] = c < nc ? A[r + (int64_t)(c0 + c) * ld] : 0.0;
#pragma unroll
        for (int c = 0; c < CH; ++c) buf[c * MAXN + to] = v[c];
      }
      __syncthreads();
      for (int r = tid; r < n; r += T)
        for (int c = 0; c < nc; ++c) A[r + (int64_t)(c0 + c) * ld] = buf[c * MAXN + r];
      __syncthreads();
    }
  }
  return s.info;
}

// Solve with the factor of one matrix, right-hand side by right-hand side, in 32-row
// blocks.  CHOL: L L^T x = b (SolveCHOL LOWER, chol.go:147-158).  LU: P A = L U, x = U^-1
// L^-1 P b (SolveLU, lu.go:320-334; P b gathered through the row map perm).  The next
// diagonal block is copied into shared memory (D, padded with zeros) while a block's rows
// are updated; a warp solves a block with one shuffle per row.
template <bool LU, int T>
__device__ __noinline__ void solve_matrix(double *y, double (*D)[CB + 1], const int *perm,
                                          const double *A, int64_t ld, int n, double *B,
                                          int64_t ldb, int nrhs) {
  constexpr int NW = T / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int last = ((n - 1) / CB) * CB;
  // block at j of the stored matrix: D[i][c] = A(j + i, j + c)
  auto fetch = [&](int j) {
#pragma unroll
    for (int e = 0; e < CB / NW; ++e) {
      const int c = warp + e * NW;
      D[lane][c] = j + lane < n && j + c < n ? A[(j + lane) + (int64_t)(j + c) * ld] : 0.0;
    }
  };
  // y_r -= A(r, j .. j + jb) x over the rows [lo, hi)
  auto axpy = [&](int lo, int hi, int j, int jb) {
    for (int r = lo + tid; r < hi; r += T) {
      double t0 = y[r], t1 = 0.0;
      const double *src = A + r + (int64_t)j * ld;
      if (jb == CB) {
#pragma unroll
        for (int c = 0; c < CB; c += 2) {
          t0 = fma(-src[c * ld], y[j + c], t0);
          t1 = fma(-src[(c + 1) * ld], y[j + c + 1], t1);
        }
      } else {
        for (int c = 0; c < jb; ++c) t0 = fma(-src[c * ld], y[j + c], t0);
      }
      y[r] = t0 + t1;
    }
  };
  for (int rc = 0; rc < nrhs; ++rc) {
    double *b = B + (int64_t)rc * ldb;
    for (int r = tid; r < n; r += T) y[r] = LU ? b[perm[r]] : b[r];
    fetch(0);
    __syncthreads();
    for (int j = 0; j < n; j += CB) {
      const int jb = min(CB, n - j);
      if (warp == 0) {
        double yi = lane < jb ? y[j + lane] : 0.0;
        const double inv = LU ? 1.0 : 1.0 / D[lane][lane];
#pragma unroll 8
        for (int c = 0; c < jb; ++c) {
          const double yc = __shfl_sync(0xffffffffu, LU ? yi : yi * inv, c);
          yi = lane > c ? fma(-D[lane][c], yc, yi) : (lane == c ? yc : yi);
        }
        if (lane < jb) y[j + lane] = yi;
      }
      __syncthreads();
      if (j + CB < n) fetch(j + CB);
      axpy(j + CB, n, j, jb);
      __syncthreads();
    }
    fetch(last);
    __syncthreads();
    for (int j = last; j >= 0; j -= CB) {
      const int jb = min(CB, n - j);
      if (!LU && j + CB < n) {
        // y_j -= L(j+32.., j..j+32)^T y(j+32..): a warp takes 32 / NW columns, lanes stride
        // over the rows
        double t[CB / NW] = {};
#pragma unroll 2
        for (int r = j + CB + lane; r < n; r += 32) {
          const double yr = y[r];
          const double *src = A + r + (int64_t)(j + warp) * ld;
#pragma unroll
          for (int u = 0; u < CB / NW; ++u) t[u] = fma(src[(int64_t)u * NW * ld], yr, t[u]);
        }
#pragma unroll
        for (int u = 0; u < CB / NW; ++u) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t[u] += __shfl_xor_sync(0xffffffffu, t[u], o);
          if (lane == 0) y[j + warp + u * NW] -= t[u];
        }
        __syncthreads();
      }
      if (warp == 0) {
        double xi = lane < jb ? y[j + lane] : 0.0;
        const double d = lane < jb ? D[lane][lane] : 1.0, inv = 1.0 / d;
        // (where the reciprocal of a tiny pivot overflows, the quotient is taken)
        const bool big = __any_sync(0xffffffffu, isinf(inv));
#pragma unroll 8
        for (int c = jb - 1; c >= 0; --c) {
          const double xc = __shfl_sync(0xffffffffu, big ? xi / d : xi * inv, c);
          const double a = LU ? D[lane][c] : D[c][lane];
          xi = lane < c ? fma(-a, xc, xi) : (lane == c ? xc : xi);
        }
        if (lane < jb) y[j + lane] = xi;
      }
      __syncthreads();
      if (j > 0) fetch(j - CB);
      if (LU) axpy(0, j, j, jb);
      __syncthreads();
    }
    for (int r = tid; r < n; r += T) b[r] = y[r];
    __syncthreads();
  }
}

template <int T, int MINB, bool LARGE>
__global__ void __launch_bounds__(T, MINB) batch_chol_kernel(BatchParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto &s = *reinterpret_cast<CholTiles<T, LARGE> *>(smem_raw);
  for (;;) {
    if (threadIdx.x == 0) s.idx = atomicAdd(p.counter, 1);
    __syncthreads();
    const int q = s.idx;
    __syncthreads();
    if (q >= p.count) break;
    const int m = p.order[q], n = p.n[m];
    const int info = chol_matrix<T, LARGE>(s, p.A[m], p.lda[m], n);
    if (threadIdx.x == 0) p.info[m] = info;
    if (p.B != nullptr && info == 0)
      solve_matrix<false, T>(s.vec, s.D, nullptr, p.A[m], p.lda[m], n, p.B[m], p.ldb[m], p.nrhs);
    __syncthreads();
  }
}

template <int T, int RPT, int MINB>
__global__ void __launch_bounds__(T, MINB) batch_lu_kernel(BatchParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  LuSmem &s = *reinterpret_cast<LuSmem *>(smem_raw);
  double *ut = p.ut + (size_t)blockIdx.x * LB * UTLD;
  for (;;) {
    if (threadIdx.x == 0) s.idx = atomicAdd(p.counter, 1);
    __syncthreads();
    const int q = s.idx;
    __syncthreads();
    if (q >= p.count) break;
    const int m = p.order[q], n = p.n[m];
    const int info = lu_matrix<T, RPT>(s, p.A[m], p.lda[m], n, p.piv[m], ut);
    if (threadIdx.x == 0) p.info[m] = info;
    if (p.B != nullptr)
      solve_matrix<true, T>(&s.L[0][0], reinterpret_cast<double(*)[CB + 1]>(&s.L[0][0] + MAXN), s.perm, p.A[m], p.lda[m], n, p.B[m], p.ldb[m], p.nrhs);
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------
// host side: kernel configurations, schedule groups, CUDA graph, autotuner
// ---------------------------------------------------------------------------------------

constexpr int NBUCKETS = MO_BATCH_BUCKETS;
constexpr int NCFG = 2;
const int kBucketMax[NBUCKETS] = {64, 128, 256, MAXN};

struct KernelCfg {
  int threads;
  const void *fn;
  size_t smem;
};

template <int T, int MINB, bool LARGE>
KernelCfg chol_cfg() {
  return KernelCfg{T, (const void *)batch_chol_kernel<T, MINB, LARGE>, sizeof(CholTiles<T, LARGE>)};
}
template <int T, int RPT, int MINB>
KernelCfg lu_cfg() {
  return KernelCfg{T, (const void *)batch_lu_kernel<T, RPT, MINB>, sizeof(LuSmem)};
}

// configuration c of a kind for the orders of bucket b: 0 = 256 threads per matrix, two CTAs
// per SM; 1 = 128 threads, four CTAs per SM.  LU above 256 rows, where a thread holds at most
// two rows: 0 = 512 threads, one CTA per SM, 1 = 256 threads, two CTAs per SM
KernelCfg kernel_cfg(int kind, int b, int c) {
  if (kind == MO_BATCH_CHOL) {
    if (b >= NBUCKETS - 2) return c == 0 ? chol_cfg<256, 2, true>() : chol_cfg<128, 4, true>();
    return c == 0 ? chol_cfg<256, 2, false>() : chol_cfg<128, 4, false>();
  }
  if (b == NBUCKETS - 1) return c == 0 ? lu_cfg<512, 1, 1>() : lu_cfg<256, 2, 2>();
  if (c == 0) return lu_cfg<256, 1, 2>();
  return b == NBUCKETS - 2 ? lu_cfg<128, 2, 4>() : lu_cfg<128, 1, 4>();
}

int bucket_of(int n) {
  for (int b = 0; b < NBUCKETS; ++b)
    if (n <= kBucketMax[b]) return b;
  return NBUCKETS - 1;
}

double work_of(int kind, int n) { return (kind == MO_BATCH_LU ? 2.0 : 1.0) * n * (double)n * n / 3.0; }

int prepare_kernel(const KernelCfg &k, int device, int *occ) {
  MO_CUDA_TRY(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem));
  MO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k.fn, k.threads, k.smem));
  (void)device;
  if (*occ < 1) return MO_ENOKERNEL;
  return MO_OK;
}

}  // namespace
}  // namespace mo

struct mo_batch {
  mo_ctx *ctx = nullptr;
  int kind = 0, count = 0, nrhs = 0;
  std::vector<int> n;          // orders (host copy)
  int cfg[MO_BATCH_BUCKETS] = {0, 0, 0, 0};
  int *d_n = nullptr;          // orders
  int *d_order = nullptr;      // queues of all groups, back to back
  int *d_counters = nullptr;   // one per group
  double *d_ut = nullptr;      // LU scratch (LB x UTLD doubles per CTA)
  size_t ut_bytes = 0;
  struct Group {
    mo::KernelCfg k;
    int count, offset, grid;
    size_t ut_off;  // doubles
  };
  std::vector<Group> groups;
  double flops = 0.0, bytes = 0.0;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  std::vector<cudaGraphNode_t> knodes;
  std::vector<mo::BatchParams> params;
  bool dirty = true;
};

namespace mo {
namespace {

void release_graph(mo_batch *b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->exec = nullptr;
  b->graph = nullptr;
  b->knodes.clear();
}

// groups from the per-bucket configuration: one queue per kernel in use, ordered by
// decreasing n, each with a full persistent grid
int build_groups(mo_batch *b) {
  mo_ctx *ctx = b->ctx;
  std::vector<KernelCfg> kern;
  std::vector<std::vector<int>> idx;
  for (int bk = NBUCKETS - 1; bk >= 0; --bk) {
    const KernelCfg k = kernel_cfg(b->kind, bk, b->cfg[bk]);
    size_t g = 0;
    while (g < kern.size() && kern[g].fn != k.fn) ++g;
    if (g == kern.size()) {
      kern.push_back(k);
      idx.emplace_back();
    }
    for (int i = 0; i < b->count; ++i)
      if (bucket_of(b->n[i]) == bk) idx[g].push_back(i);
  }
  std::vector<int> order;
  b->groups.clear();
  size_t ut_total = 0;
  for (size_t g = 0; g < kern.size(); ++g) {
    if (idx[g].empty()) continue;
    std::stable_sort(idx[g].begin(), idx[g].end(),
                     [&](int x, int y) { return b->n[x] > b->n[y]; });
    int occ = 0;
    int rc = prepare_kernel(kern[g], ctx->device, &occ);
    if (rc) return rc;
    const int grid = std::max(1, std::min(ctx->sms * occ, (int)idx[g].size()));
    mo_batch::Group gr{kern[g], (int)idx[g].size(), (int)order.size(), grid, ut_total};
    ut_total += (size_t)grid * LB * UTLD;
    b->groups.push_back(gr);
    order.insert(order.end(), idx[g].begin(), idx[g].end());
  }
  // the group holding the largest matrices runs first
  std::stable_sort(b->groups.begin(), b->groups.end(), [&](const mo_batch::Group &x,
                                                          const mo_batch::Group &y) {
    return b->n[order[x.offset]] > b->n[order[y.offset]];
  });
  if (b->d_order) cudaFree(b->d_order);
  if (b->d_counters) cudaFree(b->d_counters);
  b->d_order = nullptr;
  b->d_counters = nullptr;
  MO_CUDA_TRY(cudaMalloc(&b->d_order, sizeof(int) * std::max<size_t>(1, order.size())));
  MO_CUDA_TRY(cudaMalloc(&b->d_counters, sizeof(int) * NBUCKETS));
  MO_CUDA_TRY(cudaMemcpy(b->d_order, order.data(), sizeof(int) * order.size(), cudaMemcpyHostToDevice));
  const size_t need = b->kind == MO_BATCH_LU ? ut_total * sizeof(double) : 0;
  if (need > b->ut_bytes) {
    if (b->d_ut) cudaFree(b->d_ut);
    b->d_ut = nullptr;
    b->ut_bytes = 0;
    MO_CUDA_TRY(cudaMalloc(&b->d_ut, need));
    b->ut_bytes = need;
  }
  return MO_OK;
}

BatchParams group_params(mo_batch *b, const mo_batch::Group &g, double *const *A,
                         const int64_t *lda, double *const *B, const int64_t *ldb,
                         int64_t *const *piv, int *info) {
  BatchParams p;
  p.count = g.count;
  p.order = b->d_order + g.offset;
  p.counter = b->d_counters + (&g - b->groups.data());
  p.n = b->d_n;
  p.A = A;
  p.lda = lda;
  p.B = B;
  p.ldb = ldb;
  p.nrhs = b->nrhs;
  p.piv = piv;
  p.info = info;
  p.ut = b->d_ut ? b->d_ut + g.ut_off : nullptr;
  return p;
}

bool same_args(const BatchParams &x, const BatchParams &y) {
  return x.A == y.A && x.lda == y.lda && x.B == y.B && x.ldb == y.ldb && x.piv == y.piv &&
         x.info == y.info;
}

// graph: memset(queue counters) -> one persistent kernel node per group, all after the memset
// (the first group's kernel fills the GPU; the next one's CTAs start as its CTAs run out of
// work, and no group waits for another's last matrix)
int build_graph(mo_batch *b, const std::vector<BatchParams> &params) {
  release_graph(b);
  MO_CUDA_TRY(cudaGraphCreate(&b->graph, 0));
  cudaMemsetParams ms = {};
  ms.dst = b->d_counters;
  ms.value = 0;
  ms.elementSize = sizeof(int);
  ms.width = NBUCKETS;
  ms.height = 1;
  ms.pitch = 0;
  cudaGraphNode_t mnode;
  MO_CUDA_TRY(cudaGraphAddMemsetNode(&mnode, b->graph, nullptr, 0, &ms));
  for (size_t gi = 0; gi < b->groups.size(); ++gi) {
    const KernelCfg k = b->groups[gi].k;
    cudaKernelNodeParams kp = {};
    kp.func = const_cast<void *>(k.fn);
    kp.gridDim = dim3(b->groups[gi].grid);
    kp.blockDim = dim3(k.threads);
    kp.sharedMemBytes = (unsigned)k.smem;
    void *args[] = {const_cast<BatchParams *>(&params[gi])};
    kp.kernelParams = args;
    cudaGraphNode_t kn;
    MO_CUDA_TRY(cudaGraphAddKernelNode(&kn, b->graph, &mnode, 1, &kp));
    // One group of at most one CTA per SM: shared memory for that one CTA, the rest to L1, where
    // the solves find the factor (the driver would set room for as many CTAs as fit: 8 x 129
    // Cholesky with 32 right-hand sides 1.25 -> 0.81 ms, 1 x 129 with one 123 -> 106 us)
    if (b->groups.size() == 1 && b->groups[gi].grid <= b->ctx->sms) {
      cudaKernelNodeAttrValue v = {};
      v.sharedMemCarveout = (unsigned)((k.smem + 2048) * 100 / (228 * 1024) + 1);
      MO_CUDA_TRY(cudaGraphKernelNodeSetAttribute(
          kn, cudaKernelNodeAttributePreferredSharedMemoryCarveout, &v));
    }
    b->knodes.push_back(kn);
  }
  MO_CUDA_TRY(cudaGraphInstantiate(&b->exec, b->graph, 0));
  b->params = params;
  b->dirty = false;
  return MO_OK;
}

int update_graph(mo_batch *b, const std::vector<BatchParams> &params) {
  for (size_t gi = 0; gi < b->groups.size(); ++gi) {
    const KernelCfg k = b->groups[gi].k;
    cudaKernelNodeParams kp = {};
    kp.func = const_cast<void *>(k.fn);
    kp.gridDim = dim3(b->groups[gi].grid);
    kp.blockDim = dim3(k.threads);
    kp.sharedMemBytes = (unsigned)k.smem;
    void *args[] = {const_cast<BatchParams *>(&params[gi])};
    kp.kernelParams = args;
    MO_CUDA_TRY(cudaGraphExecKernelNodeSetParams(b->exec, b->knodes[gi], &kp));
  }
  b->params = params;
  return MO_OK;
}

int batch_run(mo_batch *b, double *const *A, const int64_t *lda, double *const *B,
              const int64_t *ldb, int64_t *const *piv, int *info) {
  mo_ctx *ctx = b->ctx;
  int rc;
  if (b->dirty || b->groups.empty()) {
    if ((rc = build_groups(b))) return rc;
    release_graph(b);
  }
  std::vector<BatchParams> params;
  for (const auto &g : b->groups) params.push_back(group_params(b, g, A, lda, B, ldb, piv, info));
  if (!b->exec) {
    if ((rc = build_graph(b, params))) return rc;
  } else {
    bool same = true;
    for (size_t i = 0; i < params.size(); ++i) same = same && same_args(params[i], b->params[i]);
    if (!same && (rc = update_graph(b, params))) return rc;
  }
  ProfScope ps;
  prof_begin(ctx, ps, MO_PROF_BATCH);
  MO_CUDA_TRY(cudaGraphLaunch(b->exec, ctx->stream));
  prof_end(ctx, ps, b->flops, b->bytes);
  return MO_OK;
}

// synthetic matrices for the autotuner: uniform[-1, 1] entries from a hash of (matrix,
// row, column); symmetric with n added to the diagonal (positive definite) for Cholesky
__global__ void tune_fill_kernel(double *buf, const int64_t *off, const int *n, int kind) {
  const int m = blockIdx.y;
  const int nm = n[m];
  double *A = buf + off[m];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)nm * nm;
       e += (int64_t)gridDim.x * blockDim.x) {
    int i = (int)(e % nm), j = (int)(e / nm);
    if (kind == MO_BATCH_CHOL && i < j) {
      const int t = i;
      i = j;
      j = t;
    }
    uint64_t h = ((uint64_t)m * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)i << 32 | (uint32_t)j);
    h ^= h >> 33;
    h *= 0xff51afd7ed558ccdull;
    h ^= h >> 33;
    h *= 0xc4ceb9fe1a85ec53ull;
    h ^= h >> 33;
    double v = (double)(h >> 11) * 0x1.0p-53 * 2.0 - 1.0;
    if (kind == MO_BATCH_CHOL && i == j) v += nm;
    A[e] = v;
  }
}

// Time every configuration on a sample of each size bucket of the plan (synthetic
// matrices of the plan's own orders) and keep the fastest per bucket.
int batch_tune(mo_batch *b, int reps, double *ms_out) {
  mo_ctx *ctx = b->ctx;
  cudaStream_t st = ctx->stream;
  reps = std::max(1, reps);
  for (int bk = 0; bk < NBUCKETS; ++bk) {
    std::vector<int> sizes;
    for (int i = 0; i < b->count; ++i)
      if (bucket_of(b->n[i]) == bk) sizes.push_back(b->n[i]);
    if (sizes.empty()) continue;
    std::sort(sizes.begin(), sizes.end(), [](int x, int y) { return x > y; });
    const int S = std::min<int>((int)sizes.size(), 4 * ctx->sms);
    std::vector<int> ns(S);
    for (int s = 0; s < S; ++s) ns[s] = sizes[(size_t)s * sizes.size() / S];
    std::vector<int64_t> off(S), lds(S), boff(S);
    int64_t tot = 0, btot = 0;
    for (int s = 0; s < S; ++s) {
      off[s] = tot;
      lds[s] = ns[s];
      tot += (int64_t)ns[s] * ns[s];
      boff[s] = btot;
      btot += (int64_t)ns[s] * std::max(1, b->nrhs);
    }
    std::vector<int> order(S);
    for (int s = 0; s < S; ++s) order[s] = s;
    // device buffers: pristine + work matrices, B, pivots, pointer arrays, scratch
    size_t ut_need = 0;
    int occs[NCFG];
    for (int c = 0; c < NCFG; ++c) {
      const KernelCfg k = kernel_cfg(b->kind, bk, c);
      int rc = prepare_kernel(k, ctx->device, &occs[c]);
      if (rc) return rc;
      ut_need = std::max(ut_need, (size_t)std::min(S, ctx->sms * occs[c]) * LB * UTLD);
    }
    char *mem = nullptr;
    const size_t bytes = 2 * tot * 8 + btot * 8 + tot * 8 /*piv*/ + S * (3 * 8 + 8 + 8 + 4 + 4 + 4) +
                         ut_need * 8 + 4096;
    MO_CUDA_TRY(cudaMalloc(&mem, bytes));
    int rc = MO_OK;
    do {
      char *p = mem;
      auto take = [&](size_t nb) {
        char *r = p;
        p += (nb + 255) & ~(size_t)255;
        return r;
      };
      double *pristine = (double *)take(tot * 8), *work = (double *)take(tot * 8);
      double *Bbuf = (double *)take(btot * 8);
      int64_t *pivbuf = (int64_t *)take(tot * 8);
      double **dA = (double **)take(S * 8), **dB = (double **)take(S * 8);
      int64_t **dP = (int64_t **)take(S * 8);
      int64_t *dlda = (int64_t *)take(S * 8), *doff = (int64_t *)take(S * 8);
      int *dn = (int *)take(S * 4), *dorder = (int *)take(S * 4), *dinfo = (int *)take(S * 4);
      int *dcounter = (int *)take(4);
      double *dut = (double *)take(ut_need * 8);
      std::vector<double *> hA(S), hB(S);
      std::vector<int64_t *> hP(S);
      for (int s = 0; s < S; ++s) {
        hA[s] = work + off[s];
        hB[s] = Bbuf + boff[s];
        hP[s] = pivbuf + off[s];
      }
      if (cudaMemcpy(dA, hA.data(), S * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
          cudaMemcpy(dB, hB.data(), S * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
          cudaMemcpy(dP, hP.data(), S * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
          cudaMemcpy(dlda, lds.data(), S * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
          cudaMemcpy(doff, off.data(), S * 8, cudaMemcpyHostToDevice) != cudaSuccess ||
          cudaMemcpy(dn, ns.data(), S * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
          cudaMemcpy(dorder, order.data(), S * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
        rc = MO_ECUDA;
        break;
      }
      tune_fill_kernel<<<dim3(16, S), 256, 0, st>>>(pristine, doff, dn, b->kind);
      cudaEvent_t e0, e1;
      cudaEventCreate(&e0);
      cudaEventCreate(&e1);
      double best = INFINITY;
      int best_c = b->cfg[bk];
      for (int c = 0; c < NCFG && !rc; ++c) {
        const KernelCfg k = kernel_cfg(b->kind, bk, c);
        BatchParams prm;
        prm.count = S;
        prm.order = dorder;
        prm.counter = dcounter;
        prm.n = dn;
        prm.A = dA;
        prm.lda = dlda;
        prm.B = b->nrhs > 0 ? dB : nullptr;
        prm.ldb = dlda;
        prm.nrhs = b->nrhs;
        prm.piv = dP;
        prm.info = dinfo;
        prm.ut = dut;
        const int grid = std::min(S, ctx->sms * occs[c]);
        double t_min = INFINITY;
        for (int r = 0; r <= reps && !rc; ++r) {
          cudaMemcpyAsync(work, pristine, tot * 8, cudaMemcpyDeviceToDevice, st);
          cudaMemsetAsync(Bbuf, 0, btot * 8, st);
          cudaMemsetAsync(dcounter, 0, 4, st);
          cudaEventRecord(e0, st);
          void *args[] = {&prm};
          if (cudaLaunchKernel(k.fn, dim3(grid), dim3(k.threads), args, k.smem, st) != cudaSuccess) {
            rc = MO_ECUDA;
            break;
          }
          cudaEventRecord(e1, st);
          if (cudaEventSynchronize(e1) != cudaSuccess) {
            rc = MO_ECUDA;
            break;
          }
          float ms = 0.f;
          cudaEventElapsedTime(&ms, e0, e1);
          if (r > 0) t_min = std::min(t_min, (double)ms);
        }
        if (ms_out) ms_out[bk * NCFG + c] = t_min;
        if (t_min < best) {
          best = t_min;
          best_c = c;
        }
      }
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      b->cfg[bk] = best_c;
    } while (false);
    cudaStreamSynchronize(st);
    cudaFree(mem);
    if (rc) return rc;
  }
  b->dirty = true;
  return MO_OK;
}

}  // namespace
}  // namespace mo

using namespace mo;

extern "C" int mo_batch_create(mo_ctx *ctx, int kind, int count, const int32_t *n, int nrhs,
                               mo_batch **out) {
  int rc = enter(ctx);
  if (rc) return rc;
  if (!out || count < 0 || nrhs < 0 || (count > 0 && !n)) return MO_EINVAL;
  if (kind != MO_BATCH_CHOL && kind != MO_BATCH_LU) return MO_EINVAL;
  for (int i = 0; i < count; ++i)
    if (n[i] < 1 || n[i] > MO_BATCH_MAX_N) return MO_EBATCHN;
  mo_batch *b = new mo_batch;
  b->ctx = ctx;
  b->kind = kind;
  b->count = count;
  b->nrhs = nrhs;
  b->n.assign(n, n + count);
  for (int i = 0; i < count; ++i) {
    const double ni = n[i];
    b->flops += work_of(kind, n[i]) + (nrhs ? 2.0 * ni * ni * nrhs : 0.0);
    b->bytes += 16.0 * ni * ni + 16.0 * ni * nrhs;
  }
  // default schedule (the autotuner may change it): more and smaller CTAs per SM, measured on
  // 4096 systems of 16 to 512 unknowns: Cholesky 5.8 ms against 7.1, LU 16.9 against 19.8.
  // (Only the order 257 to 512 of Cholesky, by 0: 200 x 512 1.05 ms against 1.27, 300 x 512 1.78
  // against 1.47, the 4096 systems 6.9.)
  // LU from 129 to 256 rows: 256 threads (512 matrices of 256: 1.46 ms against 1.69)
  for (int &c : b->cfg) c = 1;
  if (kind == MO_BATCH_LU) b->cfg[2] = 0;
  if (cudaMalloc(&b->d_n, sizeof(int) * std::max(1, count)) != cudaSuccess ||
      (count > 0 && cudaMemcpy(b->d_n, n, sizeof(int) * count, cudaMemcpyHostToDevice) != cudaSuccess)) {
    if (b->d_n) cudaFree(b->d_n);
    delete b;
    return MO_ENOMEM;
  }
  *out = b;
  return MO_OK;
}

extern "C" int mo_batch_destroy(mo_batch *b) {
  if (!b) return MO_EINVAL;
  enter(b->ctx);
  cudaStreamSynchronize(b->ctx->stream);
  release_graph(b);
  if (b->d_n) cudaFree(b->d_n);
  if (b->d_order) cudaFree(b->d_order);
  if (b->d_counters) cudaFree(b->d_counters);
  if (b->d_ut) cudaFree(b->d_ut);
  delete b;
  return MO_OK;
}

extern "C" int mo_batch_run(mo_batch *b, double *const *A, const int64_t *lda, double *const *B,
                            const int64_t *ldb, int64_t *const *piv, int *info) {
  if (!b) return MO_EINVAL;
  int rc = enter(b->ctx);
  if (rc) return rc;
  if (b->count == 0) return MO_OK;
  if (!A || !lda || !info || (b->kind == MO_BATCH_LU && !piv)) return MO_EINVAL;
  if (B && !ldb) return MO_EINVAL;
  if (b->nrhs == 0) B = nullptr;
  return batch_run(b, A, lda, B, B ? ldb : nullptr, piv, info);
}

extern "C" int mo_batch_tune(mo_batch *b, int reps, double *ms) {
  if (!b) return MO_EINVAL;
  int rc = enter(b->ctx);
  if (rc) return rc;
  if (ms)
    for (int i = 0; i < MO_BATCH_BUCKETS * NCFG; ++i) ms[i] = -1.0;
  return batch_tune(b, reps, ms);
}

extern "C" int mo_batch_schedule(mo_batch *b, int *cfg, int set) {
  if (!b || !cfg) return MO_EINVAL;
  if (set) {
    for (int i = 0; i < MO_BATCH_BUCKETS; ++i)
      if (cfg[i] < 0 || cfg[i] >= NCFG) return MO_EINVAL;
    for (int i = 0; i < MO_BATCH_BUCKETS; ++i) b->cfg[i] = cfg[i];
    b->dirty = true;
  } else {
    for (int i = 0; i < MO_BATCH_BUCKETS; ++i) cfg[i] = b->cfg[i];
  }
  return MO_OK;
}
