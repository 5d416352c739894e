// QR factorization in the compact WY form and its applications (qrwy.go, qrwym.go,
// house.go): DecomposeQRT, BuildT, MultQT and SolveQRT on the device.
//
// Reference semantics: A (m x n) = Q R with Q = H(0) H(1) ... H(k-1), k = min(m, n),
// H(j) = I - tau_j v_j v_j^T (LAPACK dlarfg: v_j(j) = 1, beta = -sign(alpha) ||(alpha, x)||,
// tau = (beta - alpha) / beta, house.go:55-78), and Q = I - Y T Y^T with Y the unit lower
// trapezoid of the reflectors and T the k x k upper triangular block reflector built by
// the dlarft recurrence T(0:j, j) = -tau_j T(0:j, 0:j) Y(:, 0:j)^T v_j (qrwy.go:61-70,
// 121-129, 433-453).  A holds R on and above its diagonal and the reflectors below it.
//
// Device form, per 128-column block of A:
//   * four 32-column panels, each factored by one kernel: up to 8192 rows one thread-block
//     cluster with the rows in registers (below); above, a cooperative kernel whose CTAs
//     keep slices of the panel's rows in shared memory; per column the CTAs publish their
//     partial products of the column with all panel columns (which give the norm below
//     the diagonal and, after the scaling, both the reflector's effect on the columns to
//     its right and the dlarft vector for the columns to its left), one grid barrier, and
//     every CTA reduces the partials in the same fixed order, so all of them hold the same
//     tau, beta and update row.  CTA 0 builds the panel's 32 x 32 T block.  The kernel also
//     writes the reflectors as an explicit unit lower trapezoid Y (zeros above) and the T
//     block with zeros below its diagonal, so that every later product is a plain GEMM;
//   * after each panel: the rest of the 128-column block takes the panel's reflectors
//     (W = C^T Y_p, its K split over the device, W = W T_p, C -= Y_p W^T);
//   * after each block: its T (the four panel T blocks joined through Y_b^T Y_b by one CTA),
//     T's rows above it, -T(0:kb,0:kb) (Y(:,0:kb)^T Y_b) T_b, and the columns to its right
//     take Q_b^T in three products with K = 128 (W = C^T Y_b, W = W T_b, C -= Y_b W^T).
// The products run on the FP64 DMMA engine.  T is kept dense (zeros below the diagonal)
// in workspace and copied to the caller's upper triangle at the end.
//
// One deliberate difference: the reference's transposed matrix-vector product
// (calgo/dmvec_gemv.c:368-395) scales y by beta once per 68-row block of A instead of
// once, and unblockedQRT / BuildT call it with beta = -tau (qrwy.go:66, :125), so the
// reference's T is the dlarft T only while at most 68 rows lie below each column; with
// more rows its T, and in the blocked factorization the trailing updates that use it,
// differ from the LAPACK definitions that its documentation names (DGEQRT, DLARFT).
// This implementation computes the LAPACK quantities at every size (bit-for-bit the same
// algorithm as the reference wherever that GEMV takes one block).
#include <algorithm>

#include "cluster.cuh"
#include "context.cuh"
#include "tri.cuh"

namespace mo {
namespace {

constexpr int kQrPanel = 32;    // columns of a Householder panel (one warp lane each)
constexpr int kQrBlock = 128;   // columns per trailing update (the K of its products)
constexpr int kQrThreads = 256;
constexpr int kQrRowsPerCta = 256;  // panel rows per CTA aimed at
constexpr int kQrMaxSmem = 220 * 1024;
constexpr int kQrApply = 256;   // reflectors per block when Q is applied to a matrix

struct QrScratch {
  double *part;        // [2][grid][32]: per-CTA column products, double-buffered by column
  double *prow;        // [2][32]: the pivot row's current values, published by its owner
  unsigned *bar;       // arrival counter of the grid barrier (zeroed before each launch)
  int *abort_flag;     // set by a CTA whose barrier wait gave up
};

// Bounded grid barrier over the co-resident CTAs of a cooperative launch.  Returns false
// (after recording MO_EDEVTIMEOUT, or when another CTA did) instead of waiting forever.
__device__ bool qr_grid_barrier(unsigned *counter, unsigned target, int *status,
                                int *abort_flag) {
  __syncthreads();
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(counter, 1u);
    int ok = 1;
    for (unsigned i = 0;; ++i) {
      if (*(volatile unsigned *)counter >= target) break;
      if (*(volatile int *)abort_flag) {
        ok = 0;
        break;
      }
      if (i > MO_SPIN_LIMIT) {
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

// sqrt(x^2 + y^2) without needless overflow (house.go:18-32, LAPACK dlapy2)
__device__ __forceinline__ double qr_hypot(double x, double y) {
  const double xa = fabs(x), ya = fabs(y);
  double w = xa, z = xa;
  if (ya > w) w = ya;
  if (ya < z) z = ya;
  if (z == 0.0) return w;
  const double q = z / w;
  return w * sqrt(1.0 + q * q);
}

// Dynamic shared memory of the panel kernel for `rpc` rows per CTA.
__host__ __device__ constexpr size_t qr_panel_smem(int rpc) {
  return (size_t)kQrPanel * (rpc | 1) * sizeof(double) + 8 * 32 * sizeof(double);
}

// Factor the R x w panel P (w <= 32, column-major, ld ldp) in place: kmax = min(R, w)
// reflectors.  Writes Y (R x w, explicit unit lower trapezoid, zeros above) and Tb (w x w,
// the panel's T with zeros below the diagonal).  Grid: cooperative, rpc rows per CTA.
__global__ void __launch_bounds__(kQrThreads, 1)
    qr_panel_kernel(double *P, int64_t ldp, int R, int w, int rpc, double *Y, int64_t ldy,
                    double *Tb, int64_t ldt, QrScratch sc, int *status) {
  extern __shared__ double smem[];
  const int S = rpc | 1;  // odd column stride: lanes that read one row of 32 columns hit
                          // 32 different banks
  double *slab = smem;    // [w][S]
  double *red = smem + (size_t)kQrPanel * S;  // [8][32] per-warp partial sums
  __shared__ double s_w[32], s_z[32], s_t[32 * 33], s_scal[4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x, cta = blockIdx.x;
  const int r0 = cta * rpc, nr = max(0, min(rpc, R - r0));
  const int kmax = min(R, w);

  for (int e = tid; e < w * rpc; e += kQrThreads) {
    const int c = e / rpc, r = e - c * rpc;
    slab[c * S + r] = r < nr ? P[(r0 + r) + (int64_t)c * ldp] : 0.0;
  }
  if (cta == 0)
    for (int e = tid; e < 32 * 33; e += kQrThreads) s_t[e] = 0.0;
  __syncthreads();

  // column products of column j with every panel column over this CTA's rows below row j
  // (q_j is the squared norm below the diagonal), and the pivot row from its owner
  auto publish = [&](int j) {
    const int par = j & 1;
    double acc0 = 0.0, acc1 = 0.0;
    const int lo = max(0, j + 1 - r0);
    if (lane < w) {
      const double *x = slab + j * S, *pc = slab + lane * S;
      int r = lo + warp;
      for (; r + 8 < nr; r += 16) {
        acc0 = fma(x[r], pc[r], acc0);
        acc1 = fma(x[r + 8], pc[r + 8], acc1);
      }
      if (r < nr) acc0 = fma(x[r], pc[r], acc0);
    }
    red[warp * 32 + lane] = acc0 + acc1;
    __syncthreads();
    if (tid < 32) {
      double s = 0.0;
#pragma unroll
      for (int g = 0; g < 8; ++g) s += red[g * 32 + tid];
      sc.part[((size_t)par * G + cta) * 32 + tid] = s;
      if (j >= r0 && j < r0 + nr) sc.prow[par * 32 + tid] = tid < w ? slab[tid * S + (j - r0)] : 0.0;
    }
  };

  if (kmax > 0) publish(0);
  for (int j = 0; j < kmax; ++j) {
    const int par = j & 1;
    if (!qr_grid_barrier(sc.bar, (unsigned)(j + 1) * G, status, sc.abort_flag)) return;
    // sum the CTAs' partials in one fixed order (every CTA gets the same values); warp 0
    // fetches the pivot row in the same round trip
    {
      double acc = 0.0;
      for (int g = warp; g < G; g += 8) acc += __ldcg(&sc.part[((size_t)par * G + g) * 32 + lane]);
      red[warp * 32 + lane] = acc;
    }
    const double prc = warp == 0 ? __ldcg(&sc.prow[par * 32 + lane]) : 0.0;
    __syncthreads();
    if (warp == 0) {
      double q = 0.0;
#pragma unroll
      for (int g = 0; g < 8; ++g) q += red[g * 32 + lane];
      // computeHouseholder (house.go:55-78) on [alpha; x] with ||x||^2 = q_j, in every lane
      const double s = __shfl_sync(0xffffffffu, q, j), alpha = __shfl_sync(0xffffffffu, prc, j);
      double tau = 0.0, denom = 1.0, beta = alpha;
      if (s != 0.0) {
        const double sign = signbit(alpha) ? -1.0 : 1.0;
        beta = -sign * qr_hypot(alpha, sqrt(s));
        denom = alpha - beta;
        tau = (beta - alpha) / beta;
      }
      // p_c = row j + v^T (rows below j) of column c, with v = x / denom
      const double p = lane < w ? prc + q / denom : 0.0;
      s_w[lane] = tau * p;   // applyHouseholder's w1 (columns right of j)
      s_z[lane] = -tau * p;  // the dlarft vector (columns left of j)
      if (lane == 0) {
        s_scal[0] = tau;
        s_scal[1] = denom;
        s_scal[2] = beta;
      }
    }
    __syncthreads();
    const double tau = s_scal[0], denom = s_scal[1], beta = s_scal[2];
    if (tau != 0.0) {
      // H(j) applied to this CTA's rows: v = x / denom, rows below j lose v_i w, row j
      // loses w and takes beta on the diagonal
      for (int r = tid; r < nr; r += kQrThreads) {
        const int i = r0 + r;
        if (i < j) continue;
        if (i == j) {
          for (int c = j + 1; c < w; ++c) slab[c * S + r] -= s_w[c];
          slab[j * S + r] = beta;
        } else {
          const double v = slab[j * S + r] / denom;
          slab[j * S + r] = v;
          for (int c = j + 1; c < w; ++c) slab[c * S + r] = fma(-v, s_w[c], slab[c * S + r]);
        }
      }
    }
    if (cta == 0 && tid < 32) {
      // T(0:j, j) = T(0:j, 0:j) z, T(j, j) = tau (zero column when tau == 0)
      double t = 0.0;
      if (tau != 0.0 && tid < j)
        for (int c = tid; c < j; ++c) t = fma(s_t[c * 33 + tid], s_z[c], t);
      __syncwarp();
      if (tid < j) s_t[j * 33 + tid] = t;
      if (tid == j) s_t[j * 33 + j] = tau;
    }
    __syncthreads();
    if (j + 1 < kmax) publish(j + 1);
  }
  __syncthreads();
  // write back: R and the reflectors into P, the explicit Y, the T block
  for (int e = tid; e < w * rpc; e += kQrThreads) {
    const int c = e / rpc, r = e - c * rpc;
    if (r >= nr) continue;
    const int i = r0 + r;
    const double v = slab[c * S + r];
    P[i + (int64_t)c * ldp] = v;
    Y[i + (int64_t)c * ldy] = i > c ? v : (i == c ? 1.0 : 0.0);
  }
  if (cta == 0)
    for (int e = tid; e < w * w; e += kQrThreads) {
      const int c = e / w, r = e - c * w;
      Tb[r + (int64_t)c * ldt] = r <= c ? s_t[c * 33 + r] : 0.0;
    }
}

// ---- the panel in one thread-block cluster ---------------------------------------------
// The panel is a chain of columns; with a grid barrier and two L2 round trips a column costs 4.6
// us (8000 rows).  Here up to 16 CTAs x 256 threads x 2 rows hold the panel in registers and
// exchange a column's products through distributed shared memory: every CTA sends its 32 sums,
// and CTA 0 the pivot row, onto the others' mbarriers, and every CTA adds the sums in the same
// order.  The loop over the columns is rolled and the registers rotate by one column per turn
// (x[q][0] is the current one, finished columns come to the end), so that its instructions
// stay in the cache; finished columns take part in the products (the dlarft vector) with a
// zero update.  T follows from the kept vectors when the columns are done.
// Measured on B200, 32 columns of 8000 to 6000 rows: 148 -> 93 us (of a column's 4.7 K cycles the
// products and their warp sums take 1.3 K, the exchange 1.7 K, the scalars 0.5 K, the update 0.6 K).
constexpr int kClThreads = 256, kClWarps = kClThreads / 32, kClMaxCtas = 16;
constexpr int kClMaxRows = kClThreads * kClMaxCtas * 2;

struct ClQr {
  uint64_t bar[2];                 // arrival of a column's sums, by column parity
  __align__(16) double sum[2][kClMaxCtas][32];
  __align__(16) double prow[2][32];
  __align__(16) double own[32], ownrow[32];  // gathered for sending
  double red[2][kClWarps][32];     // each warp's sums, by column parity: one barrier per column
                                   // does not keep a fast warp from writing the next column's
  __align__(16) double w[kClWarps][32];      // each warp's copy of the update row
  double z[32][33];                // dlarft vectors: z[j][c] = -tau_j v_c^T v_j, c < j
  double tau[32];
  double t[32][33];                // T, column j at t[j]
};

template <int RPT>
__global__ void __launch_bounds__(kClThreads, 1)
    qr_cluster_panel_kernel(double *P, int64_t ldp, int R, int w, double *Y, int64_t ldy, double *Tb,
                            int64_t ldt, int *status) {
  __shared__ ClQr s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nctas = gridDim.x, cta = blockIdx.x;  // one cluster: the grid is the cluster
  const int rbase = cta * kClThreads * RPT + tid;  // rows rbase + kClThreads q
  const int kmax = min(R, w);
  double x[RPT][32];
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int r = rbase + kClThreads * q;
#pragma unroll
    for (int k = 0; k < 32; ++k) x[q][k] = r < R && k < w ? P[r + (int64_t)k * ldp] : 0.0;
  }
  if (tid == 0) {
    mbar_init(&s.bar[0], 1);
    mbar_init(&s.bar[1], 1);
    fence_barrier_init();
  }
  if (nctas > 1) cl_sync();  // every CTA has started before any writes into its memory
  else __syncthreads();
#pragma unroll 1
  for (int j = 0; j < kmax; ++j) {
    const int par = j & 1;
    // products of the current column with all 32 over the rows below j
    double acc[32];
#pragma unroll
    for (int k = 0; k < 32; ++k) acc[k] = 0.0;
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int r = rbase + kClThreads * q;
      if (r > j && r < R) {  // (rows past R hold zeros only while no NaN is about)
#pragma unroll
        for (int k = 0; k < 32; ++k) acc[k] = fma(x[q][0], x[q][k], acc[k]);
      }
    }
    // the warp's 32 sums over its 32 lanes: lane l ends with column l's
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
      for (int k = 0; k < o; ++k) {
        const bool up = lane & o;
        const double give = up ? acc[k] : acc[k + o], keep = up ? acc[k + o] : acc[k];
        acc[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
      }
    }
    s.red[par][warp][lane] = acc[0];
    if (nctas > 1 && tid == 0)
      mbar_arrive_expect_tx(&s.bar[par], (uint32_t)((nctas + 1) * 32 * sizeof(double)));
    // the pivot row (one of CTA 0's first 32) goes out beside the sums
    if (cta == 0 && warp == 0) {
      double *to = nctas > 1 ? s.ownrow : s.prow[par];
      if (tid == j) {
#pragma unroll
        for (int k = 0; k < 32; ++k) to[k] = x[0][k];
      }
      __syncwarp();
      if (nctas > 1) cl_send<16>(s.prow[par], s.ownrow, &s.bar[par], lane, nctas);
    }
    __syncthreads();
    double qv = 0.0;  // column `lane` (rotated index) over all rows below j
    if (nctas > 1) {
      if (warp == 1) {
#pragma unroll
        for (int g = 0; g < kClWarps; ++g) qv += s.red[par][g][lane];
        s.own[lane] = qv;
        __syncwarp();
        cl_send<16>(s.sum[par][cta], s.own, &s.bar[par], lane, nctas);
      }
      // (a wait that runs out is recorded; the kernel goes on with what it holds)
      mbar_wait(&s.bar[par], (j >> 1) & 1, status);
      double part[kClMaxCtas];  // all loads in flight, added in order
#pragma unroll
      for (int g = 0; g < kClMaxCtas; ++g) part[g] = g < nctas ? s.sum[par][g][lane] : 0.0;
      qv = 0.0;
#pragma unroll
      for (int g = 0; g < kClMaxCtas; ++g) qv += part[g];
    } else {
#pragma unroll
      for (int g = 0; g < kClWarps; ++g) qv += s.red[par][g][lane];
    }
    const double prc = s.prow[par][lane];
    // computeHouseholder (house.go:55-78) on [alpha; x] with ||x||^2 = q_0, in every lane
    const double nrm2 = __shfl_sync(0xffffffffu, qv, 0), alpha = __shfl_sync(0xffffffffu, prc, 0);
    double tau = 0.0, denom = 1.0, beta = alpha;
    if (nrm2 != 0.0) {
      // (the plain root of the sum where neither square leaves the normal range: the scaled
      // one is two roots and a quotient, 500 cycles, on the chain)
      const double a2 = alpha * alpha, ss = a2 + nrm2;
      const double nrm = ss < 1e300 && nrm2 > 1e-280 ? sqrt(fma(alpha, alpha, nrm2))
                                                     : qr_hypot(alpha, sqrt(nrm2));
      beta = signbit(alpha) ? nrm : -nrm;
      denom = alpha - beta;
      tau = (beta - alpha) / beta;
    }
    // p_c = row j + v^T (rows below j) of column c, with v = x / denom; rotated index k is
    // column j + k, finished ones (columns < j) at k >= 32 - j
    const double p = tau != 0.0 ? tau * (prc + qv / denom) : 0.0;
    s.w[warp][lane] = lane < 32 - j ? p : 0.0;
    if (cta == 0 && warp == 2) {
      if (lane >= 32 - j) s.z[j][lane - (32 - j)] = -p;
      if (lane == 0) s.tau[j] = tau;
    }
    // with an infinity or a NaN about, finished rows and columns must not meet it even times zero
    const bool odd = __any_sync(0xffffffffu, !isfinite(p) || !isfinite(qv));
    __syncwarp();
    // H(j) on this thread's rows: v = x / denom, rows below j lose v w, row j loses w and
    // takes beta; the registers rotate
    double v[RPT], last[RPT];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      const int r = rbase + kClThreads * q;
      const double xv = tau != 0.0 ? x[q][0] / denom : x[q][0];
      v[q] = r > j ? xv : (r == j ? 1.0 : 0.0);
      last[q] = r > j ? xv : (r == j ? beta : x[q][0]);
    }
    if (odd) {
#pragma unroll
      for (int k = 1; k < 32; ++k)
#pragma unroll
        for (int q = 0; q < RPT; ++q)
          x[q][k - 1] = k < 32 - j && rbase + kClThreads * q >= j ? fma(-v[q], s.w[warp][k], x[q][k])
                                                                : x[q][k];
    } else
#pragma unroll
    for (int k = 0; k < 32; k += 2) {
      const double2 wk = *reinterpret_cast<const double2 *>(&s.w[warp][k]);
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        if (k > 0) x[q][k - 1] = fma(-v[q], wk.x, x[q][k]);
        x[q][k] = fma(-v[q], wk.y, x[q][k + 1]);
      }
    }
#pragma unroll
    for (int q = 0; q < RPT; ++q) x[q][31] = last[q];
  }
  // write back: R and the reflectors into P, the explicit Y (register k: column (k + kmax) % 32)
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int r = rbase + kClThreads * q;
    if (r >= R) continue;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const int c = (k + kmax) & 31;
      if (c >= w) continue;
      P[r + (int64_t)c * ldp] = x[q][k];
      Y[r + (int64_t)c * ldy] = r > c ? x[q][k] : (r == c ? 1.0 : 0.0);
    }
  }
  __syncthreads();
  if (cta == 0 && warp == 0) {
    // T(0:j, j) = T(0:j, 0:j) z_j, T(j, j) = tau_j (zero column when tau == 0)
    for (int j = 0; j < 32; ++j) {
      double t = 0.0;
      const double tau = j < kmax ? s.tau[j] : 0.0;
      if (tau != 0.0 && lane < j)
        for (int c = lane; c < j; ++c) t = fma(s.t[c][lane], s.z[j][c], t);
      s.t[j][lane] = lane < j ? t : (lane == j ? tau : 0.0);
      __syncwarp();
    }
    for (int c = 0; c < w; ++c)
      if (lane < w) Tb[lane + (int64_t)c * ldt] = s.t[c][lane];
  }
  if (nctas > 1) cl_sync();  // no CTA leaves while another may still write into its memory
}

// The 128-column block's T from its four 32 x 32 panel blocks (on the diagonal of Tb, ld
// ldt, zeros below) and the Gram matrix Zin = Y_b^T Y_b (ld ldz): for panel p the rows above
// it are T(0:32p, p) = -T(0:32p, 0:32p) Zin(0:32p, p) T_pp (qrwy.go:433-453 at panel
// granularity).  One CTA; the block lives in shared memory.
// Both products run as 16 x 16 tiles on the FP64 tensor pipe, a warp per tile: 78 us a block with
// one FMA chain per element, 41 us this way.
constexpr int kTbLd = 132;  // T(r, c) at r * kTbLd + c (4 mod 16: fragments without conflicts)
constexpr int kQrTBlockSmem = (128 * kTbLd + 96 * 36) * 8;
__global__ void __launch_bounds__(256) qr_t_block_kernel(double *Tb, int64_t ldt,
                                                         const double *Zin, int64_t ldz, int bo) {
  extern __shared__ double sm[];
  double *T = sm;                  // [128][kTbLd], zeros outside bo x bo and below the diagonal
  double *M1 = sm + 128 * kTbLd;   // [96][36]
  const int tid = threadIdx.x, warp = tid >> 5;
  bool odd = false;
#pragma unroll 16
  for (int e = tid; e < 128 * 128; e += 256) {
    const int r = e & 127, c = e >> 7;
    const bool own = r < bo && c < bo && r <= c && r / kQrPanel == c / kQrPanel;
    // above the diagonal panels: the Gram matrix, replaced block column by block column
    const bool gram = r < bo && c < bo && r / kQrPanel < c / kQrPanel;
    const double v = own ? Tb[r + (int64_t)c * ldt] : gram ? Zin[r + (int64_t)c * ldz] : 0.0;
    T[r * kTbLd + c] = v;
    odd |= !isfinite(v);
  }
  // with an infinity or a NaN about, the zeros below T's diagonal must not meet it: sums over
  // T's upper triangle only, element by element, so that the columns left of it stay right
  odd = __syncthreads_or(odd);
  for (int p0 = kQrPanel; odd && p0 < bo; p0 += kQrPanel) {
    const int w = min(kQrPanel, bo - p0);
    for (int e = tid; e < p0 * w; e += 256) {
      const int c = e / p0, r = e - c * p0;
      double acc = 0.0;
      for (int l = 0; l <= c; ++l)
        acc = fma(T[r * kTbLd + p0 + l], T[(p0 + l) * kTbLd + p0 + c], acc);
      M1[r * 36 + c] = acc;
    }
    __syncthreads();
    for (int e = tid; e < p0 * w; e += 256) {
      const int c = e / p0, r = e - c * p0;
      double acc = 0.0;
      for (int l = r; l < p0; ++l) acc = fma(T[r * kTbLd + l], M1[l * 36 + c], acc);
      T[r * kTbLd + p0 + c] = -acc;
    }
    __syncthreads();
  }
  for (int p0 = kQrPanel; !odd && p0 < bo; p0 += kQrPanel) {
    const int nt = p0 / 16;  // 16-row tiles above the panel, two columns of them
    // M1 = Zin(0:p0, p0:p0+32) T(p0:p0+32, p0:p0+32)
    for (int t = warp; t < 2 * nt; t += 8) {
      const int i = 16 * (t >> 1), j = 16 * (t & 1);
      double c[2][4] = {};
      for (int k = 0; k < kQrPanel; k += 16)
        tri_mm16(c, T + i * kTbLd + p0 + k, kTbLd, 1, T + (p0 + k) * kTbLd + p0 + j, 1, kTbLd);
      tri_put16(c, M1 + i * 36 + j, 36, 1, 1.0, false);
    }
    __syncthreads();
    // T(0:p0, p0:p0+32) = -T(0:p0, 0:p0) M1  (T upper triangular)
    for (int t = warp; t < 2 * nt; t += 8) {
      const int i = 16 * (t >> 1), j = 16 * (t & 1);
      double c[2][4] = {};
      for (int k = i; k < p0; k += 16)
        tri_mm16(c, T + i * kTbLd + k, kTbLd, 1, M1 + k * 36 + j, 1, 36);
      tri_put16(c, T + i * kTbLd + p0 + j, kTbLd, 1, -1.0, false);
    }
    __syncthreads();
  }
  for (int e = tid; e < 128 * 128; e += 256) {
    const int r = e & 127, c = e >> 7;
    if (c < bo && r < (c / kQrPanel) * kQrPanel) Tb[r + (int64_t)c * ldt] = T[r * kTbLd + c];
  }
}

// Y (m x k) = the explicit unit lower trapezoid of A's reflectors (zeros above)
__global__ void __launch_bounds__(256) qr_expand_y_kernel(const double *A, int64_t lda, int m,
                                                          int k, double *Y, int64_t ldy) {
  const int i = blockIdx.x * 256 + threadIdx.x, c = blockIdx.y;
  if (i >= m || c >= k) return;
  Y[i + (int64_t)c * ldy] = i > c ? A[i + (int64_t)c * lda] : (i == c ? 1.0 : 0.0);
}

// Tw (k x k) = T's upper triangle with zeros below
__global__ void __launch_bounds__(256) qr_expand_t_kernel(const double *T, int64_t ldt, int k,
                                                          double *Tw, int64_t ldw) {
  const int i = blockIdx.x * 256 + threadIdx.x, c = blockIdx.y;
  if (i >= k || c >= k) return;
  Tw[i + (int64_t)c * ldw] = i <= c ? T[i + (int64_t)c * ldt] : 0.0;
}

// T's upper triangle (k x k) <- Tw; with tau, columns whose tau is zero are left as they
// are (qrwy.go:60 writes nothing for them)
__global__ void __launch_bounds__(256) qr_t_out_kernel(const double *Tw, int64_t ldw, int k,
                                                       double *T, int64_t ldt, const double *tau) {
  const int i = blockIdx.x * 256 + threadIdx.x, c = blockIdx.y;
  if (i >= k || c >= k || i > c) return;
  if (tau && tau[c] == 0.0) return;
  T[i + (int64_t)c * ldt] = Tw[i + (int64_t)c * ldw];
}

// BuildT's diagonal blocks: for each 32-column panel p (one CTA), T_p from the panel's Gram
// matrix Gm = Y_p^T Y_p (in Tw's block, overwritten) and tau: column j is
// T_p(0:j, j) = T_p(0:j, 0:j) (-tau_j Gm(0:j, j)), T_p(j, j) = tau_j (qrwy.go:29-84)
__global__ void __launch_bounds__(32) qr_buildt_diag_kernel(double *Tw, int64_t ldw, int k,
                                                            const double *tau) {
  __shared__ double s_t[32 * 33], s_z[32];
  const int p0 = blockIdx.x * kQrPanel, w = min(kQrPanel, k - p0), lane = threadIdx.x;
  double *B = Tw + p0 + (int64_t)p0 * ldw;
  for (int c = 0; c < 32; ++c) s_t[c * 33 + lane] = 0.0;
  __syncwarp();
  for (int j = 0; j < w; ++j) {
    const double tj = tau[p0 + j];
    if (lane < j) s_z[lane] = -tj * B[lane + (int64_t)j * ldw];
    __syncwarp();
    double t = 0.0;
    if (tj != 0.0 && lane < j)
      for (int c = lane; c < j; ++c) t = fma(s_t[c * 33 + lane], s_z[c], t);
    __syncwarp();
    if (lane < j) s_t[j * 33 + lane] = t;
    if (lane == j) s_t[j * 33 + j] = tj;
    __syncwarp();
  }
  for (int c = 0; c < w; ++c)
    if (lane < w) B[lane + (int64_t)c * ldw] = lane <= c ? s_t[c * 33 + lane] : 0.0;
}

// rows i >= r0 of the columns of B (rows x cols, ld) set to zero
__global__ void __launch_bounds__(256) qr_zero_rows_kernel(double *B, int64_t ld, int r0,
                                                           int rows) {
  const int i = r0 + blockIdx.x * 256 + threadIdx.x, c = blockIdx.y;
  if (i < rows) B[i + (int64_t)c * ld] = 0.0;
}

// one thread per element of an rows x cols grid (cols <= 65535)
template <typename F>
int launch_grid2(int rows, int cols, F &&launch) {
  if (rows <= 0 || cols <= 0) return MO_OK;
  launch(dim3((rows + 255) / 256, cols));
  MO_CUDA_TRY(cudaGetLastError());
  return MO_OK;
}

constexpr int kQrMaxCols = 65535;  // reflectors per call (one grid row of columns)

struct QrWork {
  double *Y = nullptr;   // m x k explicit reflectors (ld m)
  double *Tw = nullptr;  // k x k dense T, zeros below the diagonal (ld k)
  double *W = nullptr;   // products' scratch, wsize doubles each
  double *W2 = nullptr;
  double *Z = nullptr;   // k x 128
  double *X = nullptr;   // k x 128
  QrScratch sc{};
  int cl_rows = 0;       // rows up to which a panel runs in one cluster
};

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// bytes of the buffers below (panel scratch for `grid` CTAs)
size_t qr_workspace_bytes(int m, int k, int64_t wsize, int grid) {
  const size_t by = align256((size_t)m * k * 8), bt = align256((size_t)k * k * 8);
  const size_t bw = align256((size_t)wsize * 8), bz = align256((size_t)k * kQrBlock * 8);
  const size_t bp = align256((size_t)2 * grid * 32 * 8), br = align256(2 * 32 * 8);
  return by + bt + 2 * bw + 2 * bz + bp + br + 256;
}

// Carve the context workspace into the buffers above (panel scratch for `grid` CTAs).
int qr_workspace(mo_ctx *ctx, int m, int k, int64_t wsize, int grid, QrWork &q) {
  const size_t by = align256((size_t)m * k * 8), bt = align256((size_t)k * k * 8);
  const size_t bw = align256((size_t)wsize * 8), bz = align256((size_t)k * kQrBlock * 8);
  const size_t bp = align256((size_t)2 * grid * 32 * 8), br = align256(2 * 32 * 8);
  char *ws = nullptr;
  int rc = workspace(ctx, qr_workspace_bytes(m, k, wsize, grid), (void **)&ws);
  if (rc) return rc;
  q.Y = (double *)ws;
  ws += by;
  q.Tw = (double *)ws;
  ws += bt;
  q.W = (double *)ws;
  ws += bw;
  q.W2 = (double *)ws;
  ws += bw;
  q.Z = (double *)ws;
  ws += bz;
  q.X = (double *)ws;
  ws += bz;
  q.sc.part = (double *)ws;
  ws += bp;
  q.sc.prow = (double *)ws;
  ws += br;
  q.sc.bar = (unsigned *)ws;
  q.sc.abort_flag = (int *)(ws + 64);
  return MO_OK;
}

// CTAs and rows per CTA of the panel kernel for R rows
void panel_shape(mo_ctx *ctx, int R, int &grid, int &rpc) {
  grid = max(1, min(ctx->sms, (R + kQrRowsPerCta - 1) / kQrRowsPerCta));
  rpc = (R + grid - 1) / grid;
}

// the most rows a panel may have: every CTA's slice must fit in shared memory
int max_panel_rows(mo_ctx *ctx) {
  const int rpc = (int)((kQrMaxSmem - 8 * 32 * 8) / (kQrPanel * 8)) - 1;
  return rpc * ctx->sms;
}

const void *cl_kernel(int rpt) {
  return rpt == 1 ? (const void *)qr_cluster_panel_kernel<1> : (const void *)qr_cluster_panel_kernel<2>;
}

int cl_config(int ctas, int rpt, cudaStream_t st, cudaLaunchConfig_t *cfg,
              cudaLaunchAttribute *attr) {
  MO_CUDA_TRY(cudaFuncSetAttribute(cl_kernel(rpt), cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(ctas);
  cfg->blockDim = dim3(kClThreads);
  cfg->stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim = {(unsigned)ctas, 1, 1};
  cfg->attrs = attr;
  cfg->numAttrs = 1;
  return MO_OK;
}

// rows up to which a panel may run in one cluster (16 CTAs are not portable: ask)
int cluster_rows(mo_ctx *ctx, int m, int *rows) {
  *rows = kClThreads * 8;
  if (m <= *rows) return MO_OK;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  int clusters = 0;
  if (int rc = cl_config(kClMaxCtas, 2, ctx->stream, &cfg, &attr)) return rc;
  if (cudaOccupancyMaxActiveClusters(&clusters, cl_kernel(2), &cfg) == cudaSuccess && clusters > 0)
    *rows = kClMaxRows;
  else
    cudaGetLastError();
  return MO_OK;
}

// factor A[kp:m, kp:kp+bp]; its reflectors go to Y's and its T block to Tw's columns kp..
int panel(mo_ctx *ctx, View A, int kp, int bp, QrWork &q, int k) {
  const int m = A.rows, R = m - kp;
  if (R <= q.cl_rows) {
    // one row per thread while 16 CTAs suffice
    const int rpt = R > kClThreads * kClMaxCtas ? 2 : 1;
    int ctas = 1;
    while (ctas * kClThreads * rpt < R) ctas *= 2;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    if (int rc = cl_config(ctas, rpt, ctx->stream, &cfg, &attr)) return rc;
    double *P = A.at(kp, kp), *Y = q.Y + kp + (int64_t)kp * m, *Tb = q.Tw + kp + (int64_t)kp * k;
    int64_t ldp = A.ld, ldy = m, ldt = k;
    int rows = R, w = bp, *status = &control(ctx)->status;
    void *args[] = {&P, &ldp, &rows, &w, &Y, &ldy, &Tb, &ldt, &status};
    ProfScope ps;
    prof_begin(ctx, ps, MO_PROF_PANEL);
    const cudaError_t e = cudaLaunchKernelExC(&cfg, cl_kernel(rpt), args);
    prof_end(ctx, ps, 4.0 * R * (double)bp * bp, 8.0 * 3 * R * (double)bp);
    MO_CUDA_TRY(e);
    return MO_OK;
  }
  int grid = 0, rpc = 0;
  panel_shape(ctx, R, grid, rpc);
  const size_t smem = qr_panel_smem(rpc);
  if (smem > (size_t)kQrMaxSmem) return MO_EINVAL;
  int rc = mo_smem_attr((const void *)qr_panel_kernel, (int)smem);
  if (rc) return rc;
  MO_CUDA_TRY(cudaMemsetAsync(q.sc.bar, 0, 128, ctx->stream));
  double *P = A.at(kp, kp);
  int64_t ldp = A.ld;
  int w = bp;
  double *Y = q.Y + kp + (int64_t)kp * m;
  int64_t ldy = m;
  double *Tb = q.Tw + kp + (int64_t)kp * k;
  int64_t ldt = k;
  QrScratch sc = q.sc;
  int *status = &control(ctx)->status;
  void *args[] = {&P, &ldp, (void *)&R, &w, &rpc, &Y, &ldy, &Tb, &ldt, &sc, &status};
  ProfScope ps;
  prof_begin(ctx, ps, MO_PROF_PANEL);
  MO_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)qr_panel_kernel, dim3(grid),
                                          dim3(kQrThreads), args, smem, ctx->stream));
  prof_end(ctx, ps, 4.0 * R * (double)bp * bp, 8.0 * 3 * R * (double)bp);
  MO_CUDA_TRY(cudaGetLastError());
  return MO_OK;
}

// T(0:kp, kp:kp+bp) = -T(0:kp, 0:kp) Z T(kp:kp+bp, kp:kp+bp) with Z = Y(:, 0:kp)^T
// Y(:, kp:kp+bp) (qrwy.go:433-453); Z is read from Zsrc (kp x bp, ld ldz), which may be T's
// own block (BuildT) because the result goes through X first
int t_columns(mo_ctx *ctx, int k, int kp, int bp, View Zsrc, QrWork &q) {
  if (kp == 0) return MO_OK;
  const View Tv{q.Tw, k, k, k}, Xv{q.X, kp, bp, kp};
  int rc = gemm(ctx, Xv, Zsrc, false, Tv.sub(kp, kp, bp, bp), false, 1.0, 0.0);
  if (!rc) rc = gemm(ctx, Tv.sub(0, kp, kp, bp), Tv.sub(0, 0, kp, kp), false, Xv, false, -1.0, 0.0);
  return rc;
}

// C (rows s.. of A's columns right of a block) = Q_b^T C for the block's reflectors:
// W = C^T Y_b, W = W T_b, C -= Y_b W^T (qrwy.go:266-303 with transpose)
int apply_left_t(mo_ctx *ctx, View C, const View &Yb, const View &Tb, QrWork &q) {
  const int nc = C.cols, b = Yb.cols;
  if (nc <= 0 || b <= 0) return MO_OK;
  const View W{q.W, nc, b, nc}, W2{q.W2, nc, b, nc};
  int rc = gemm(ctx, W, C, true, Yb, false, 1.0, 0.0);
  if (!rc) rc = gemm(ctx, W2, W, false, Tb, false, 1.0, 0.0);
  if (!rc) rc = gemm(ctx, C, Yb, false, W2, true, -1.0, 1.0);
  return rc;
}

int t_out(mo_ctx *ctx, const QrWork &q, int k, View T, const double *tau_mask) {
  return launch_grid2(k, k, [&](dim3 g) {
    qr_t_out_kernel<<<g, 256, 0, ctx->stream>>>(q.Tw, k, k, T.d, T.ld, tau_mask);
  });
}

// tau (k entries, stride) <- T's diagonal
__global__ void qr_tau_out_kernel(const double *Tw, int64_t ldw, int k, double *tau,
                                  int64_t inc) {
  const int j = blockIdx.x * 256 + threadIdx.x;
  if (j < k) tau[j * inc] = Tw[j + (int64_t)j * ldw];
}

// tau (k entries, stride) -> a contiguous copy
__global__ void qr_tau_in_kernel(const double *tau, int64_t inc, int k, double *out) {
  const int j = blockIdx.x * 256 + threadIdx.x;
  if (j < k) out[j] = tau[j * inc];
}

}  // namespace

// One 128-column block [kb, kb + bo): its 32-column panels, the rest of the block after each
// panel, the block's T (the panels' T blocks joined through Y_b^T Y_b) and T's rows above
// it, all on the context's stream.
int factor_block(mo_ctx *ctx, View A, int kb, int bo, int k, QrWork &q) {
  const int m = A.rows;
  const View Yv{q.Y, m, k, m}, Tv{q.Tw, k, k, k};
  int rc;
  for (int kp = kb; kp < kb + bo; kp += kQrPanel) {
    const int bp = min(kQrPanel, kb + bo - kp);
    if ((rc = panel(ctx, A, kp, bp, q, k))) return rc;
    // the rest of the block takes the panel's reflectors
    const int c0 = kp + bp, rest = kb + bo - c0;
    if (rest > 0 &&
        (rc = apply_left_t(ctx, A.sub(kp, c0, m - kp, rest), Yv.sub(kp, kp, m - kp, bp),
                           Tv.sub(kp, kp, bp, bp), q)))
      return rc;
  }
  const View Yb = Yv.sub(kb, kb, m - kb, bo), Tb = Tv.sub(kb, kb, bo, bo);
  if (bo > kQrPanel) {
    const View Zin{q.W2, bo, bo, bo};
    if ((rc = gemm(ctx, Zin, Yb, true, Yb, false, 1.0, 0.0))) return rc;
    if ((rc = mo_smem_attr((const void *)qr_t_block_kernel, kQrTBlockSmem))) return rc;
    qr_t_block_kernel<<<1, 256, kQrTBlockSmem, ctx->stream>>>(Tb.d, k, q.W2, bo, bo);
    MO_CUDA_TRY(cudaGetLastError());
  }
  if (kb > 0) {
    // T's rows above the block: -T(0:kb, 0:kb) (Y(kb:m, 0:kb)^T Y_b) T_b
    const View Z{q.Z, kb, bo, kb};
    if ((rc = gemm(ctx, Z, Yv.sub(kb, 0, m - kb, kb), true, Yb, false, 1.0, 0.0))) return rc;
    if ((rc = t_columns(ctx, k, kb, bo, Z, q))) return rc;
  }
  return MO_OK;
}

// The device part of DecomposeQRT / DecomposeQR: A (m x n) factored in place; T's upper
// k x k triangle written when T.d, tau (k entries, stride tau_inc) when tau.  (Factoring
// the next block on a second stream beside the trailing update was slower with the
// cooperative panel, which takes as many SMs as it has slices, and with the T products
// without stream-K; with the cluster panel and its 16 SMs it has not been measured.)
int qr_factor(mo_ctx *ctx, View A, View T, double *tau, int64_t tau_inc) {
  const int m = A.rows, n = A.cols, k = min(m, n);
  if (k == 0) return MO_OK;
  if (m > max_panel_rows(ctx) || k > kQrMaxCols) return MO_EINVAL;
  int grid = 0, rpc = 0;
  panel_shape(ctx, m, grid, rpc);
  QrWork q;
  int rc = qr_workspace(ctx, m, k, (int64_t)max(n, 1) * kQrBlock, grid, q);
  if (rc) return rc;
  if ((rc = cluster_rows(ctx, m, &q.cl_rows))) return rc;
  const View Yv{q.Y, m, k, m}, Tv{q.Tw, k, k, k};
  // the products read T's blocks below the diagonal and Y's rows above each panel inside
  // a 128-column block as zeros (the panels write only their own rows and T blocks)
  MO_CUDA_TRY(cudaMemsetAsync(q.Tw, 0, (size_t)k * k * sizeof(double), ctx->stream));
  MO_CUDA_TRY(cudaMemsetAsync(q.Y, 0, (size_t)m * k * sizeof(double), ctx->stream));
  for (int kb = 0; kb < k; kb += kQrBlock) {
    const int bo = min(kQrBlock, k - kb);
    if ((rc = factor_block(ctx, A, kb, bo, k, q))) return rc;
    const int c0 = kb + bo, nt = n - c0;
    if (nt > 0 && (rc = apply_left_t(ctx, A.sub(kb, c0, m - kb, nt), Yv.sub(kb, kb, m - kb, bo),
                                     Tv.sub(kb, kb, bo, bo), q)))
      return rc;
  }
  if (T.d && (rc = t_out(ctx, q, k, T, nullptr))) return rc;
  if (tau) {
    qr_tau_out_kernel<<<(k + 255) / 256, 256, 0, ctx->stream>>>(q.Tw, k, k, tau, tau_inc);
    MO_CUDA_TRY(cudaGetLastError());
  }
  return MO_OK;
}

// The dense block reflector of A's first k reflectors and tau into q.Tw (BuildT,
// qrwy.go:29-84): Tw = the upper triangle of Y^T Y, each 32 x 32 diagonal block replaced by
// its dlarft recurrence, then the blocks above the diagonal by t_columns in column order.
// q.Y must hold the expanded reflectors.
int qr_build_t(mo_ctx *ctx, int m, int k, const double *tau_c, QrWork &q) {
  const View Yv{q.Y, m, k, m}, Tv{q.Tw, k, k, k};
  MO_CUDA_TRY(cudaMemsetAsync(q.Tw, 0, (size_t)k * k * 8, ctx->stream));
  int rc = syrk(ctx, Tv, Yv, true, true, 1.0, 0.0, 0);
  if (rc) return rc;
  qr_buildt_diag_kernel<<<(k + kQrPanel - 1) / kQrPanel, 32, 0, ctx->stream>>>(q.Tw, k, k, tau_c);
  MO_CUDA_TRY(cudaGetLastError());
  for (int kp = kQrPanel; kp < k; kp += kQrPanel) {
    const int bp = min(kQrPanel, k - kp);
    if ((rc = t_columns(ctx, k, kp, bp, Tv.sub(0, kp, kp, bp), q))) return rc;
  }
  return MO_OK;
}

// C = Q C, Q^T C (MO_TRANS), C Q (MO_RIGHT), C Q^T (MO_RIGHT|MO_TRANS) with Q = I - Y T Y^T
// of k reflectors (q.Y, q.Tw), in blocks of nb reflectors in the order qrwym.go:382-566
// takes them: forward for Q^T C and C Q, backward (aligned at k) for Q C and C Q^T.  Each
// block reads only its reflectors' rows s..m, so blocks of a few hundred reflectors take
// about a third of the flops of one block of all k (which multiplies the zeros above Y's
// diagonal and the whole of T).
int qr_apply(mo_ctx *ctx, View C, int m, int k, int flags, int nb, QrWork &q) {
  const bool right = (flags & MO_RIGHT) != 0, trans = (flags & MO_TRANS) != 0;
  const bool forward = right ? !trans : trans;
  const View Yv{q.Y, m, k, m}, Tv{q.Tw, k, k, k};
  int rc = MO_OK;
  auto block = [&](int s, int b) -> int {
    const View Yb = Yv.sub(s, s, m - s, b), Tb = Tv.sub(s, s, b, b);
    if (!right) {
      const int nc = C.cols;
      const View Cs = C.sub(s, 0, m - s, nc), W{q.W, nc, b, nc}, W2{q.W2, nc, b, nc};
      int r = gemm(ctx, W, Cs, true, Yb, false, 1.0, 0.0);
      if (!r) r = gemm(ctx, W2, W, false, Tb, !trans, 1.0, 0.0);
      if (!r) r = gemm(ctx, Cs, Yb, false, W2, true, -1.0, 1.0);
      return r;
    }
    const int nr = C.rows;
    const View Cs = C.sub(0, s, nr, m - s), W{q.W, nr, b, nr}, W2{q.W2, nr, b, nr};
    int r = gemm(ctx, W, Cs, false, Yb, false, 1.0, 0.0);
    if (!r) r = gemm(ctx, W2, W, false, Tb, trans, 1.0, 0.0);
    if (!r) r = gemm(ctx, Cs, W2, false, Yb, true, -1.0, 1.0);
    return r;
  };
  if (forward) {
    for (int s = 0; s < k && !rc; s += nb) rc = block(s, min(nb, k - s));
  } else {
    for (int e = k; e > 0 && !rc; e -= nb) {
      const int b = min(nb, e);
      rc = block(e - b, b);
    }
  }
  return rc;
}

// expand A's reflectors (and, when T.d, T's upper triangle) into q for k reflectors, with
// W buffers of wsize doubles
int qr_prepare(mo_ctx *ctx, View A, int k, View T, int64_t wsize, QrWork &q) {
  const int m = A.rows;
  int rc = qr_workspace(ctx, m, k, wsize, 1, q);
  if (rc) return rc;
  if ((rc = launch_grid2(m, k, [&](dim3 g) {
         qr_expand_y_kernel<<<g, 256, 0, ctx->stream>>>(A.d, A.ld, m, k, q.Y, m);
       })))
    return rc;
  if (T.d)
    rc = launch_grid2(k, k, [&](dim3 g) {
      qr_expand_t_kernel<<<g, 256, 0, ctx->stream>>>(T.d, T.ld, k, q.Tw, k);
    });
  return rc;
}

// contiguous copy of tau (k entries, stride inc)
void qr_tau_copy(mo_ctx *ctx, const double *tau, int64_t inc, int k, double *out) {
  qr_tau_in_kernel<<<(k + 255) / 256, 256, 0, ctx->stream>>>(tau, inc, k, out);
}

// T's upper triangle <- q.Tw, columns with tau == 0 left untouched
int qr_t_store(mo_ctx *ctx, const QrWork &q, int k, View T, const double *tau_c) {
  return t_out(ctx, q, k, T, tau_c);
}

// rows r0.. of B set to zero
void qr_zero_rows(mo_ctx *ctx, View B, int r0) {
  if (B.rows <= r0 || B.cols <= 0) return;
  for (int c0 = 0; c0 < B.cols; c0 += 65535) {
    const dim3 g((B.rows - r0 + 255) / 256, std::min(65535, B.cols - c0));
    qr_zero_rows_kernel<<<g, 256, 0, ctx->stream>>>(B.at(0, c0), B.ld, r0, B.rows);
  }
}

// A (m x n) := the first n columns of the identity
__global__ void __launch_bounds__(256) qr_eye_kernel(double *A, int64_t lda, int m) {
  const int i = blockIdx.x * 256 + threadIdx.x, c = blockIdx.y;
  if (i < m) A[i + (int64_t)c * lda] = i == c ? 1.0 : 0.0;
}

// BuildQ / BuildQT's device part: A (m x n, m >= n) := Q [I_n; 0] with Q from A's n
// reflectors and T (or tau)
int qr_build_q(mo_ctx *ctx, View A, View T, const double *tau, int64_t tau_inc) {
  const int m = A.rows, n = A.cols;
  if (n == 0 || m == 0) return MO_OK;
  if (n > kQrMaxCols) return MO_EINVAL;
  const int b = std::min(kQrApply, n);
  QrWork q;
  int rc = qr_prepare(ctx, A, n, T, std::max((int64_t)n * b, (int64_t)n), q);
  if (rc) return rc;
  if (!T.d) {
    qr_tau_copy(ctx, tau, tau_inc, n, q.W2);
    if ((rc = qr_build_t(ctx, m, n, q.W2, q))) return rc;
  }
  if ((rc = launch_grid2(m, n, [&](dim3 g) {
         qr_eye_kernel<<<g, 256, 0, ctx->stream>>>(A.d, A.ld, m);
       })))
    return rc;
  return qr_apply(ctx, A, m, n, MO_LEFT, b, q);
}

}  // namespace mo

using mo::View;

namespace {

// W as the reference's optional workspace: data == NULL stands for a nil matrix
bool is_nil(const mo_matrix &W) { return W.data == nullptr; }

// tau as a column vector view of at least k entries: pointer and stride
int tau_view(const mo_matrix &tau, int k, double **p, int64_t *inc) {
  if (tau.rows < 0 || tau.cols < 0) return MO_EINVAL;
  const int64_t len = tau.rows * tau.cols;
  if (len < k || (tau.rows != 1 && tau.cols != 1 && k > 0)) return MO_EINVAL;
  if (k > 0 && !tau.data) return MO_EINVAL;
  *p = tau.data;
  *inc = tau.cols == 1 ? 1 : tau.ld;  // a row vector steps by its leading index
  return MO_OK;
}

// the checks of MultQT / MultQ (qrwym.go:646-671, 573-600) shared by both
int mult_checks(const View &C, const View &A, const mo_matrix &Wm, int flags, int nb,
                bool need_w) {
  if (need_w && is_nil(Wm)) return MO_ENOWORK;
  if (flags & MO_RIGHT) {
    if (C.cols != A.rows) return MO_ECQSIZE;
    if (need_w && (Wm.cols < nb || Wm.rows < C.rows)) return MO_EWORKSMALL;
  } else {
    if (need_w && (Wm.cols < nb || Wm.rows < C.cols)) return MO_EWORKSMALL;
    // the reference leaves this unchecked and then updates with mismatched operands
    if (C.rows != A.rows && C.rows > 0 && C.cols > 0) return MO_EABSIZE;
  }
  return MO_OK;
}

int apply_q(mo_ctx *ctx, View C, View A, View T, const double *tau, int64_t tau_inc, int flags,
            int nb) {
  const int m = A.rows, k = std::min(A.rows, A.cols);
  if (k == 0 || C.rows == 0 || C.cols == 0) return MO_OK;
  if (k > 65535) return MO_EINVAL;
  // the device's own blocking (results agree with any nb to rounding)
  nb = std::min(mo::kQrApply, k);
  const int64_t wsize = std::max((int64_t)std::max(C.rows, C.cols) * nb, (int64_t)k);
  mo::QrWork q;
  int rc = mo::qr_prepare(ctx, A, k, T, wsize, q);
  if (rc) return rc;
  if (!T.d) {
    double *tc = q.W2;  // contiguous tau, consumed by qr_build_t before W2 is used
    mo::qr_tau_copy(ctx, tau, tau_inc, k, tc);
    if ((rc = mo::qr_build_t(ctx, m, k, tc, q))) return rc;
  }
  return mo::qr_apply(ctx, C, m, k, flags, nb, q);
}

// SolveQRT / SolveQR (qrwym.go:784-819, 717-760) on Q from (T) or (tau)
int solve_q(mo_ctx *ctx, View B, View A, View T, const double *tau, int64_t tau_inc,
            const mo_matrix &Wm, int flags, int nb, bool need_w) {
  const int n = A.cols;
  if (A.rows < n || B.rows < n) return MO_EABSIZE;
  const View R = A.sub(0, 0, n, n), BT = B.sub(0, 0, n, B.cols);
  int rc;
  if (flags & MO_TRANS) {
    // minimum-norm solution of A^T X = B: B' = R^-T B, rows below n cleared, X = Q B'
    if ((rc = mult_checks(B, A, Wm, MO_LEFT, nb, need_w))) return rc;
    if ((rc = mo::trsm(ctx, BT, R, MO_LEFT | MO_UPPER | MO_TRANSA, 1.0))) return rc;
    if (B.rows > n) {
      mo::qr_zero_rows(ctx, B, n);
    }
    return apply_q(ctx, B, A, T, tau, tau_inc, MO_LEFT, nb);
  }
  // least squares min ||A X - B||: B' = Q^T B, X = R^-1 B'(0:n)
  if ((rc = mult_checks(B, A, Wm, MO_LEFT | MO_TRANS, nb, need_w))) return rc;
  if ((rc = apply_q(ctx, B, A, T, tau, tau_inc, MO_LEFT | MO_TRANS, nb))) return rc;
  return mo::trsm(ctx, BT, R, MO_LEFT | MO_UPPER, 1.0);
}

}  // namespace

extern "C" {

// qrwy.go:517-538
int mo_decompose_qrt(mo_ctx *ctx, mo_matrix Am, mo_matrix Tm, mo_matrix Wm, int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View A, T;
  if ((rc = mo::to_view(Am, A)) || (rc = mo::to_view(Tm, T))) return rc;
  if (!(nb == 0 || A.cols <= nb) && !is_nil(Wm) && (Wm.cols < nb || Wm.rows < A.cols))
    return MO_EWORKSMALL;
  const int k = std::min(A.rows, A.cols);
  if (T.rows < k || T.cols < k) return MO_ETSMALL;
  if (k > 0 && !T.d) return MO_EINVAL;
  return mo::qr_factor(ctx, A, T, nullptr, 0);
}

// qrwy.go:474-497
int mo_decompose_qr(mo_ctx *ctx, mo_matrix Am, mo_matrix taum, mo_matrix Wm, int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View A;
  if ((rc = mo::to_view(Am, A))) return rc;
  const int k = std::min(A.rows, A.cols);
  double *tau = nullptr;
  int64_t inc = 1;
  if ((rc = tau_view(taum, k, &tau, &inc))) return rc;
  if (!(nb == 0 || A.cols <= nb) && !is_nil(Wm) && (Wm.cols < nb || Wm.rows < A.cols))
    return MO_EWORKSMALL;
  return mo::qr_factor(ctx, A, View{nullptr, 0, 0, 1}, tau, inc);
}

// qrwy.go:546-556
int mo_build_t(mo_ctx *ctx, mo_matrix Tm, mo_matrix Am, mo_matrix taum) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View T, A;
  if ((rc = mo::to_view(Tm, T)) || (rc = mo::to_view(Am, A))) return rc;
  if (T.cols < A.cols || T.rows < A.cols) return MO_ETSMALL;
  const int m = A.rows;
  int k = std::min(A.rows, A.cols);
  double *tau = nullptr;
  int64_t inc = 1;
  if (taum.rows * taum.cols < k) k = (int)(taum.rows * taum.cols);
  if ((rc = tau_view(taum, k, &tau, &inc))) return rc;
  if (k == 0) return MO_OK;
  if (k > 65535) return MO_EINVAL;
  mo::QrWork q;
  if ((rc = mo::qr_prepare(ctx, A, k, View{nullptr, 0, 0, 1}, k, q))) return rc;
  double *tc = q.W2;
  mo::qr_tau_copy(ctx, tau, inc, k, tc);
  if ((rc = mo::qr_build_t(ctx, m, k, tc, q))) return rc;
  return mo::qr_t_store(ctx, q, k, T, tc);
}

// qrwym.go:646-688
int mo_mult_qt(mo_ctx *ctx, mo_matrix Cm, mo_matrix Am, mo_matrix Tm, mo_matrix Wm, int flags,
               int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View C, A, T;
  if ((rc = mo::to_view(Cm, C)) || (rc = mo::to_view(Am, A)) || (rc = mo::to_view(Tm, T)))
    return rc;
  if (nb == 0) nb = T.cols;
  if ((rc = mult_checks(C, A, Wm, flags, nb, true))) return rc;
  const int k = std::min(A.rows, A.cols);
  if (T.rows < k || T.cols < k) return MO_ETSMALL;
  if (k > 0 && !T.d) return MO_EINVAL;
  return apply_q(ctx, C, A, T, nullptr, 0, flags, nb);
}

// qrwym.go:573-630
int mo_mult_q(mo_ctx *ctx, mo_matrix Cm, mo_matrix Am, mo_matrix taum, mo_matrix Wm, int flags,
              int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View C, A;
  if ((rc = mo::to_view(Cm, C)) || (rc = mo::to_view(Am, A))) return rc;
  if ((rc = mult_checks(C, A, Wm, flags, nb, nb != 0))) return rc;
  const int k = std::min(A.rows, A.cols);
  double *tau = nullptr;
  int64_t inc = 1;
  if ((rc = tau_view(taum, k, &tau, &inc))) return rc;
  return apply_q(ctx, C, A, View{nullptr, 0, 0, 1}, tau, inc, flags, nb);
}

// qrwym.go:784-819
int mo_solve_qrt(mo_ctx *ctx, mo_matrix Bm, mo_matrix Am, mo_matrix Tm, mo_matrix Wm, int flags,
                 int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View B, A, T;
  if ((rc = mo::to_view(Bm, B)) || (rc = mo::to_view(Am, A)) || (rc = mo::to_view(Tm, T)))
    return rc;
  if (nb == 0) nb = T.cols;
  const int k = std::min(A.rows, A.cols);
  if (T.rows < k || T.cols < k) return MO_ETSMALL;
  if (k > 0 && !T.d) return MO_EINVAL;
  return solve_q(ctx, B, A, T, nullptr, 0, Wm, flags, nb, true);
}

// qrwym.go:717-760
int mo_solve_qr(mo_ctx *ctx, mo_matrix Bm, mo_matrix Am, mo_matrix taum, mo_matrix Wm, int flags,
                int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View B, A;
  if ((rc = mo::to_view(Bm, B)) || (rc = mo::to_view(Am, A))) return rc;
  const int k = std::min(A.rows, A.cols);
  double *tau = nullptr;
  int64_t inc = 1;
  if ((rc = tau_view(taum, k, &tau, &inc))) return rc;
  return solve_q(ctx, B, A, View{nullptr, 0, 0, 1}, tau, inc, Wm, flags, nb, nb != 0);
}

// qrwyk.go:232-267
int mo_build_q(mo_ctx *ctx, mo_matrix Am, mo_matrix taum, mo_matrix Wm, int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View A;
  if ((rc = mo::to_view(Am, A))) return rc;
  if (nb != 0 && is_nil(Wm)) return MO_ENOWORK;
  if (nb != 0 && (Wm.cols < nb || Wm.rows < A.cols)) return MO_EWORKSMALL;
  if (A.rows < A.cols) return MO_EABSIZE;
  double *tau = nullptr;
  int64_t inc = 1;
  if ((rc = tau_view(taum, A.cols, &tau, &inc))) return rc;
  return mo::qr_build_q(ctx, A, View{nullptr, 0, 0, 1}, tau, inc);
}

// qrwyk.go:278-293
int mo_build_qt(mo_ctx *ctx, mo_matrix Am, mo_matrix Tm, mo_matrix Wm, int nb) {
  int rc = mo::enter(ctx);
  if (rc) return rc;
  View A, T;
  if ((rc = mo::to_view(Am, A)) || (rc = mo::to_view(Tm, T))) return rc;
  if (nb == 0) nb = A.cols;
  if (is_nil(Wm)) return MO_ENOWORK;
  if (Wm.cols < nb || Wm.rows < A.cols) return MO_EWORKSMALL;
  if (A.rows < A.cols) return MO_EABSIZE;
  if (T.rows < A.cols || T.cols < A.cols) return MO_ETSMALL;
  if (A.cols > 0 && !T.d) return MO_EINVAL;
  return mo::qr_build_q(ctx, A, T, nullptr, 0);
}

}  // extern "C"
