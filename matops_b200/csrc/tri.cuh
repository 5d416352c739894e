// Diagonal blocks (order <= 128) in shared memory: Cholesky factor and lower-triangular
// inverse by 16 x 16 sub-blocks, FP64, one CTA of 256 threads.
//
// Layout: S[i * LDS + j] = element (i, j), row length LDS = 132 (4 mod 16 doubles, so that DMMA
// fragment loads by rows and by columns touch every bank once).  A block of order n is padded
// to NP = roundup(n, 32) with the identity.  The lower triangle of S holds the block, then
// its factor L; the inverse X = L^-1 goes to the part above the diagonal blocks, transposed
// (X(i, j) at S[j * LDS + i] for i, j in different sub-blocks), and its diagonal sub-blocks to
// Xd, transposed too (X(b, b)(r, c) at Xd[(16 b + c) * XLD + r]).
//
// What bounds it is the chain of columns.  Per sub-block: one warp factors and inverts the 16 x
// 16 diagonal block (two columns per step, registers and shuffles), multiplies the tile below
// it by that inverse, updates the next diagonal block and goes on to it; meanwhile the other
// warps do the other tiles (DMMA products), the rest of the update and the finished block row
// of the inverse.  They stay off the first warp's scheduler: beside a warp of DMMAs its FP64
// FMAs would starve.  Measured on B200, one 128 x 128 block with its inverse, against 32-column
// leaves, one thread per row below them and FMA updates, the inverse after the factor:
// DecomposeCHOL's kernel 88 -> 38 us, the inverse alone 35 -> 24 us, the mixed factorization's
// block 68 -> 43 us (of the 38, 16 us are the eight 16 x 16 blocks, 6 us loads and stores).
#pragma once
#include "common.cuh"

namespace mo {

constexpr int TRI_MAX = 128;
constexpr int LDS = TRI_MAX + 4;
constexpr int XLD = 20;
constexpr int TRI_THREADS = 256;  // two threads per row of a block
// shared memory: the block, the inverse's diagonal sub-blocks, a 16 x 16 scratch per warp, and
// the columns of the sub-block being factored
constexpr int TRI_SMEM_DBL = TRI_MAX * LDS + TRI_MAX * XLD + 8 * 16 * XLD + 16 * 16;
constexpr int TRI_SMEM_BYTES = TRI_SMEM_DBL * 8;
struct TriSmem {
  double *S, *Xd, *M, *col;
  __device__ explicit TriSmem(double *sm)
      : S(sm), Xd(sm + TRI_MAX * LDS), M(Xd + TRI_MAX * XLD), col(M + 8 * 16 * XLD) {}
};

__device__ __forceinline__ int round_up32(int n) { return (n + 31) & ~31; }

// Load the n x n block at G (column-major, ld) into S as a LOWER triangle:
//   transpose == false: S(i,j) = G(i,j) for i >= j
//   transpose == true : S(i,j) = G(j,i) for i >= j   (reads the upper triangle of G)
// The strict upper part of S is zeroed; rows/cols n..NP-1 become the identity.
// unit_diag forces S(i,i) = 1.  A thread keeps to one row of G (128 rows x 2 columns per pass: no
// divisions) and has 16 loads in flight before its shared-memory stores.
template <typename T>
__device__ inline void tri_load_lower(double *S, const T *G, int64_t ld, int n, bool transpose,
                                      bool unit_diag) {
  const int NP = round_up32(n);
  const int i = threadIdx.x & (TRI_MAX - 1);
  for (int j0 = threadIdx.x / TRI_MAX; j0 < NP; j0 += 32) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int j = j0 + 2 * u;
      // element of the lower triangle that G(i, j) feeds: (si, sj)
      const int si = transpose ? j : i, sj = transpose ? i : j;
      v[u] = (si == sj) ? 1.0 : 0.0;
      if (si < n && sj < n && si >= sj && !(unit_diag && si == sj))
        v[u] = (double)G[i + (int64_t)j * ld];
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int j = j0 + 2 * u;
      if (i < NP && j < NP) S[(transpose ? j : i) * LDS + (transpose ? i : j)] = v[u];
    }
  }
}

// Store the lower triangle of S (n x n) to G: transpose == false -> G(i,j) = S(i,j) for
// i >= j; transpose == true -> G(j,i) = S(i,j) (upper triangle of G).
template <typename T>
__device__ inline void tri_store_lower(const double *S, T *G, int64_t ld, int n, bool transpose) {
  const int i = threadIdx.x & (TRI_MAX - 1);
  if (i >= n) return;
#pragma unroll 8
  for (int j = threadIdx.x / TRI_MAX; j < n; j += 2)
    if (transpose ? j >= i : i >= j)
      G[i + (int64_t)j * ld] = (T)(transpose ? S[j * LDS + i] : S[i * LDS + j]);
}

// element (i, j) of the inverse, zero above the diagonal
__device__ __forceinline__ double tri_inv_at(const TriSmem &t, int i, int j) {
  if (i < j) return 0.0;
  return (i >> 4) == (j >> 4) ? t.Xd[j * XLD + (i & 15)] : t.S[j * LDS + i];
}

// Store the inverse (n x n) to G with zeros in its other triangle; transpose: G = X^T
__device__ inline void tri_store_inverse(const TriSmem &t, double *G, int64_t ld, int n,
                                         bool transpose) {
  const int i = threadIdx.x & (TRI_MAX - 1);
  if (i >= n) return;
#pragma unroll 8
  for (int j = threadIdx.x / TRI_MAX; j < n; j += 2)
    G[i + (int64_t)j * ld] = transpose ? tri_inv_at(t, j, i) : tri_inv_at(t, i, j);
}

// c (16 x 16 in fragments: rows g + 8 h, columns 8 ni + 2 t + e at c[ni][2 h + e]) += P Q with
// P(r, k) = p[r * pr + k * pk] and Q(k, n) = q[n * qn + k * qk], one warp
__device__ __forceinline__ void tri_mm16(double (&c)[2][4], const double *p, int pr, int pk,
                                         const double *q, int qn, int qk) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  p += g * pr + t * pk;
  q += g * qn + t * qk;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double a0 = p[4 * k * pk], a1 = p[8 * pr + 4 * k * pk];
#pragma unroll
    for (int ni = 0; ni < 2; ++ni) dmma_16x8x4(c[ni], a0, a1, q[8 * ni * qn + 4 * k * qk]);
  }
}
// d(r, n) = sign * c (+ d when add), at d[r * dr + n * dn]; one warp, ordered before its later
// reads
__device__ __forceinline__ void tri_put16(const double (&c)[2][4], double *d, int dr, int dn,
                                          double sign, bool add) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  __syncwarp();  // every lane has read what this replaces
#pragma unroll
  for (int ni = 0; ni < 2; ++ni)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      double *at = d + (g + 8 * (q >> 1)) * dr + (8 * ni + 2 * t + (q & 1)) * dn;
      *at = add ? fma(sign, c[ni][q], *at) : sign * c[ni][q];
    }
  __syncwarp();
}

// Column c = lane % 16 of the inverse of a 16 x 16 lower triangle: L(i, m) for m < i through
// l(i, m), reciprocal diagonal rd of row lane % 16; X(i, c) to Xd[c * ldc + i * ldi]
template <typename F>
__device__ __forceinline__ void tri_inv16(double *Xd, int ldc, int ldi, double rd, F &&l) {
  const int lane = threadIdx.x & 31, c = lane & 15;
  double x[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    double s0 = i == c ? 1.0 : 0.0, s1 = 0.0;
#pragma unroll
    for (int m = 0; m + 1 < i; m += 2) {
      s0 = fma(-l(i, m), x[m], s0);
      s1 = fma(-l(i, m + 1), x[m + 1], s1);
    }
    if (i & 1) s0 = fma(-l(i, i - 1), x[i - 1], s0);
    const double r = __shfl_sync(0xffffffffu, rd, i);
    // zero above the diagonal also where the row has a zero pivot (0 times infinity): the
    // columns right of it are those of a regular triangle
    x[i] = i < c ? 0.0 : (s0 + s1) * r;
  }
  if (lane < 16) {
#pragma unroll
    for (int i = 0; i < 16; ++i) Xd[c * ldc + i * ldi] = x[i];
  }
}

// Factor the 16 x 16 block at B (row length LDS) and invert it into Xd, by one warp: lane i (and
// i + 16) holds row i; two columns per step, every lane factoring the 2 x 2 pivot block itself
// (l11 = sqrt(a), l21 = b / l11, l22 = sqrt(c - l21^2)) and the multipliers passed through `col`.
// The reference divides by the square root (calgo/dvec_util.c:230-246); here columns are
// multiplied by reciprocal square roots, equal to rounding.  Returns the first column whose
// pivot has no real root (its value in *badv), or -1.
__device__ __forceinline__ int tri_potrf16(double *B, double *Xd, double *col, double *badv) {
  const int lane = threadIdx.x & 31, i16 = lane & 15;
  double r[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) r[k] = k <= i16 ? B[i16 * LDS + k] : 0.0;
  double pivot = 1.0, rd = 1.0;  // this lane's diagonal entry before its root, and 1 / root
#pragma unroll
  for (int k = 0; k < 16; k += 2) {
    const double a = __shfl_sync(0xffffffffu, r[k], k);
    const double b = __shfl_sync(0xffffffffu, r[k], k + 1);
    const double c = __shfl_sync(0xffffffffu, r[k + 1], k + 1);
    const double rs1 = rsqrt(a), l21 = b * rs1, d = fma(-l21, l21, c), rs2 = rsqrt(d);
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
      col[16 * k + lane] = x1;
      col[16 * k + 16 + lane] = x2;
    }
    __syncwarp();
#pragma unroll
    for (int j = k + 2; j < 16; ++j)
      r[j] = fma(-x2, col[16 * k + 16 + j], fma(-x1, col[16 * k + j], r[j]));
    r[k] = x1;
    r[k + 1] = x2;
  }
  const double dg = sqrt(pivot);
  const unsigned bad = __ballot_sync(0xffffffffu, isnan(dg));
  if (bad) {
    const int at = __ffs(bad) - 1;
    *badv = __shfl_sync(0xffffffffu, pivot, at);
    return at;
  }
  if (lane < 16) {
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k <= i16) B[i16 * LDS + k] = k == i16 ? dg : r[k];
  }
  tri_inv16(Xd, XLD, 1, rd, [&](int i, int m) { return col[16 * m + i]; });
  __syncwarp();
  return -1;
}

// Block row i of the inverse, X(i, j) = -X(i, i) sum_{k = j}^{i-1} L(i, k) X(k, j), tiles j = w, w +
// nw, ... by this warp (scratch M: 16 x XLD)
__device__ __forceinline__ void tri_inv_row(const TriSmem &t, double *M, int i, int w, int nw) {
  for (int j = w; j < i; j += nw) {
    double c[2][4] = {};
    // X(j, j)(k, n) at Xd[(16 j + n) * XLD + k], X(k, j)(kk, n) at S[(16 j + n) * LDS + 16 k + kk]
    tri_mm16(c, t.S + 16 * i * LDS + 16 * j, LDS, 1, t.Xd + 16 * j * XLD, XLD, 1);
    for (int k = j + 1; k < i; ++k)
      tri_mm16(c, t.S + 16 * i * LDS + 16 * k, LDS, 1, t.S + 16 * j * LDS + 16 * k, LDS, 1);
    tri_put16(c, M, XLD, 1, 1.0, false);
    double x[2][4] = {};
    tri_mm16(x, t.Xd + 16 * i * XLD, 1, XLD, M, 1, XLD);
    tri_put16(x, t.S + 16 * j * LDS + 16 * i, 1, LDS, -1.0, false);
  }
}

// In-place Cholesky of the lower triangle of S (order NP, a multiple of 32) and the inverse of
// the factor.  All threads of the block (256).  Returns the first column whose pivot is
// negative or NaN, with its value in *bad_val (then the factorization stops there), or -1.
__device__ inline int tri_potrf_inverse(const TriSmem &t, int NP, double *bad_val) {
  // the failing column by parity of the block that set it: warp 0 writes block b + 1's word
  // while the others may still be reading block b's
  __shared__ int s_bad[2];
  __shared__ double s_badv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = NP / 16;
  // warps 1-3 and 5-7 (never warp 0's scheduler) work beside warp 0
  const int w6 = warp < 4 ? warp - 1 : warp - 2;
  double *M = t.M + warp * 16 * XLD;
  auto blk = [&](int i, int j) { return t.S + 16 * i * LDS + 16 * j; };
  // L(i, b) = A(i, b) X(b, b)^T
  auto panel = [&](int i, int b) {
    double c[2][4] = {};
    tri_mm16(c, blk(i, b), LDS, 1, t.Xd + 16 * b * XLD, 1, XLD);
    tri_put16(c, blk(i, b), LDS, 1, 1.0, false);
  };
  // A(i, j) -= L(i, b) L(j, b)^T
  auto update = [&](int i, int j, int b) {
    double c[2][4] = {};
    tri_mm16(c, blk(i, b), LDS, 1, blk(j, b), LDS, 1);
    tri_put16(c, blk(i, j), LDS, 1, -1.0, true);
  };
  auto diag = [&](int b) {
    double bv = 0.0;
    const int bad = tri_potrf16(blk(b, b), t.Xd + 16 * b * XLD, t.col, &bv);
    if (bad >= 0 && lane == 0) {
      s_bad[b & 1] = 16 * b + bad;
      s_badv = bv;
    }
  };
  if (threadIdx.x == 0) s_bad[0] = s_bad[1] = -1;
  __syncthreads();
  if (warp == 0) diag(0);
  __syncthreads();
  int bad = -1;
  for (int b = 0; b < nb; ++b) {
    bad = s_bad[b & 1];
    if (bad >= 0) break;  // the same for all threads
    if (warp == 0) {
      if (b + 1 < nb) panel(b + 1, b);
      asm volatile("bar.arrive 1, 256;" ::: "memory");
      if (b + 1 < nb) {
        update(b + 1, b + 1, b);
        diag(b + 1);
      }
    } else {
      if (warp != 4)
        for (int i = b + 2 + w6; i < nb; i += 6) panel(i, b);
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (warp != 4) {
        // the tiles (i, j) of the trailing triangle but its first, row by row
        int q = 0;
        for (int i = b + 2; i < nb; ++i)
          for (int j = b + 1; j <= i; ++j, ++q)
            if (q % 6 == w6) update(i, j, b);
        tri_inv_row(t, M, b, 5 - w6, 6);
      }
    }
    __syncthreads();
  }
  if (bad >= 0) *bad_val = s_badv;
  return bad;
}

// The inverse of the lower-triangular S (order NP, a multiple of 32, non-singular diagonal),
// all threads of the block (256).
__device__ inline void tri_inverse_lower(const TriSmem &t, int NP) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = NP / 16;
  if (warp < nb) {
    const double *B = t.S + 16 * warp * (LDS + 1);
    const double rd = 1.0 / B[(lane & 15) * (LDS + 1)];
    tri_inv16(t.Xd + 16 * warp * XLD, XLD, 1, rd, [&](int i, int m) { return B[i * LDS + m]; });
  }
  __syncthreads();
  for (int i = 1; i < nb; ++i) {
    tri_inv_row(t, t.M + warp * 16 * XLD, i, warp, 8);
    __syncthreads();
  }
}

}  // namespace mo
