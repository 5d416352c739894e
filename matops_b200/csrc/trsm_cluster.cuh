// The few-right-hand-side triangular solve in one thread-block cluster, for orders up to 2048
// (included by trsm_few.cu, whose FewArgs it takes).
//
// A solve with few right-hand sides is a chain of diagonal blocks.  As CTAs that publish 64-row
// steps through flags in L2 a 64-row step costs 4.6 us; here CTA c of a cluster of up to 16
// owns the 128 rows of step c, keeps the inverse of its diagonal block in shared memory and
// the next 128 x 128 block of op(A) in registers, adds up op(A) x for every step's x as it
// arrives, and sends its own x to the later CTAs' shared memory (st.async onto an mbarrier per
// step).  Each cluster takes up to 4 right-hand sides.
// What bounds it: per 128 rows the exchange (about 800 cycles), 64 FMAs per thread and
// right-hand side on the newest x, and the product with the inverse, whose 128 KB come from
// shared memory.  Measured on B200, this kernel against the flag-passing one: n = 500, one
// right-hand side 15 us (36 us); n = 1001, three 45 us (93 us).  SolveTrm as a whole, block
// inverses (24 us) included: n = 2048, one right-hand side 170 -> 55 us, 16: 168 -> 89 us.
#pragma once
#include <type_traits>

#include "cluster.cuh"

namespace mo {
namespace {

constexpr int kTcThreads = 256, kTcBlock = 128, kTcMax = 16, kTcLd = kTcBlock + 1;

template <int NR>
struct TcSmem {
  uint64_t bar[kTcMax];                              // arrival of step s's x
  int late;                                          // a wait of this CTA ran out
  __align__(16) double x[kTcMax][NR * kTcBlock];     // x of the earlier steps, by right-hand side
  __align__(16) double own[NR * kTcBlock];           // this CTA's x, and b before it
  double part[NR * kTcBlock];
  double inv[kTcBlock * kTcLd];                      // inv[k * kTcLd + i] = inverse(i, k)
};

// The wait for step t's x (every thread waits for itself).  False, and the timeout recorded, when
// the polls that the context allows (mo_set_spin_limit) run out.
__device__ __forceinline__ bool tc_wait(uint64_t *bar, const FewArgs &p) {
  if (p.spin_limit >= MO_SPIN_LIMIT) return mbar_wait(bar, 0, p.status);
  for (uint32_t it = 0; it <= p.spin_limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred q;\n\tmbarrier.test_wait.parity.shared::cta.b64 q, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar))
        : "memory");
    if (done) return true;
  }
  set_status(p.status, MO_EDEVTIMEOUT);
  return false;
}

template <typename TA, bool TRANS, int NR, bool UNIT>
__global__ void __launch_bounds__(kTcThreads, 1) trsm_cluster_kernel(const FewArgs p) {
  extern __shared__ __align__(16) unsigned char tc_raw[];
  TcSmem<NR> &s = *reinterpret_cast<TcSmem<NR> *>(tc_raw);
  if (p.skip && *(volatile const int *)p.skip) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (p.N + kTcBlock - 1) / kTcBlock;
  const int c = blockIdx.x, rhs0 = blockIdx.y * NR, nr = min(NR, p.nrhs - rhs0);
  const int r = tid & (kTcBlock - 1), h = tid >> 7;  // row, and which 64 of 128 columns
  auto block = [&](int step) { return p.lower_eff ? step : nblk - 1 - step; };
  const int rb = block(c), r0 = rb * kTcBlock;
  const int nrow = c < nblk ? min(kTcBlock, p.N - r0) : 0;
  const TA *A = static_cast<const TA *>(p.A);
  // 64 elements of the 128 x 128 block of op(A) for step `step`: !TRANS: row r, columns 64 h + k at
  // a[k]; TRANS: rows 16 warp + i, columns lane + 32 j at a[4 i + j] (contiguous along lanes)
  TA a[64];
  auto fetch = [&](int step) {
    const int c0 = block(step) * kTcBlock, nc = min(kTcBlock, p.N - c0);
    if constexpr (!TRANS) {
      const TA *src = A + r0 + r + (int64_t)(c0 + 64 * h) * p.lda;
#pragma unroll
      for (int k = 0; k < 64; ++k) a[k] = r < nrow && 64 * h + k < nc ? src[k * p.lda] : TA(0);
    } else {
      const TA *src = A + c0 + lane + (int64_t)(r0 + 16 * warp) * p.lda;
#pragma unroll
      for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          a[4 * i + j] =
              16 * warp + i < nrow && lane + 32 * j < nc ? src[i * p.lda + 32 * j] : TA(0);
    }
  };
  if (c > 0 && c < nblk) fetch(0);
  if (tid == 0) {
    s.late = 0;
    for (int t = 0; t < kTcMax; ++t) mbar_init(&s.bar[t], 1);
    fence_barrier_init();
    for (int t = 0; t < c && c < nblk; ++t)
      mbar_arrive_expect_tx(&s.bar[t], (uint32_t)(NR * kTcBlock * sizeof(double)));
  }
  if (c < nblk) {
    const double *iv = p.inv + (size_t)rb * kTcBlock * kTcBlock;
#pragma unroll 16
    for (int e = tid; e < kTcBlock * kTcBlock; e += kTcThreads) {
      const int u = e & (kTcBlock - 1), w = e >> 7;
      const double v = u < nrow && w < nrow ? iv[e] : 0.0;
      if (p.inv_t) s.inv[u * kTcLd + w] = v;
      else s.inv[w * kTcLd + u] = v;
    }
    if constexpr (UNIT) {
      // op(A) itself between the two 64 x 64 diagonal blocks (see below)
      __syncthreads();
      const int i0 = p.lower_eff ? 64 : 0, k0 = 64 - i0;
#pragma unroll 8
      for (int e = tid; e < 64 * 64; e += kTcThreads) {
        const int i = i0 + (TRANS ? e >> 6 : e & 63), k = k0 + (TRANS ? e & 63 : e >> 6);
        const int64_t at = TRANS ? r0 + k + (int64_t)(r0 + i) * p.lda
                                 : r0 + i + (int64_t)(r0 + k) * p.lda;
        s.inv[k * kTcLd + i] = i < nrow && k < nrow ? (double)A[at] : 0.0;
      }
    }
  }
  cl_sync();  // every CTA's barriers are armed before any x is sent
  double acc[NR];
#pragma unroll
  for (int q = 0; q < NR; ++q) acc[q] = 0.0;
  double sum[16 * NR];  // TRANS: this lane's part of the rows 16 warp + i
  if constexpr (TRANS) {
#pragma unroll
    for (int i = 0; i < 16 * NR; ++i) sum[i] = 0.0;
  }
  if (c < nblk) {
    for (int t = 0; t < c; ++t) {
      if (!tc_wait(&s.bar[t], p)) {
        s.late = 1;
        break;
      }
      if constexpr (!TRANS) {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          const double2 *x = reinterpret_cast<const double2 *>(s.x[t] + q * kTcBlock + 64 * h);
          double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
#pragma unroll
          for (int k = 0; k < 64; k += 4) {
            const double2 xa = x[k / 2], xb = x[k / 2 + 1];
            v0 = fma((double)a[k], xa.x, v0);
            v1 = fma((double)a[k + 1], xa.y, v1);
            v2 = fma((double)a[k + 2], xb.x, v2);
            v3 = fma((double)a[k + 3], xb.y, v3);
          }
          acc[q] += (v0 + v1) + (v2 + v3);
        }
      } else {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
          double x[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) x[j] = s.x[t][q * kTcBlock + lane + 32 * j];
#pragma unroll
          for (int i = 0; i < 16; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
              sum[16 * q + i] = fma((double)a[4 * i + j], x[j], sum[16 * q + i]);
        }
      }
      if (t + 1 < c) fetch(t + 1);
    }
    // b = alpha B - sum, complete in s.own
    if constexpr (!TRANS) {
      if (h == 1) {
#pragma unroll
        for (int q = 0; q < NR; ++q) s.part[q * kTcBlock + r] = acc[q];
      }
    } else {
      // 16 rows over 32 lanes: lane l ends with row l / 2 of the warp's
#pragma unroll
      for (int q = 0; q < NR; ++q) {
#pragma unroll
        for (int o = 16; o > 1; o >>= 1) {
#pragma unroll
          for (int k = 0; k < o / 2; ++k) {
            const bool up = lane & o;
            const double give = up ? sum[16 * q + k] : sum[16 * q + k + o / 2];
            const double keep = up ? sum[16 * q + k + o / 2] : sum[16 * q + k];
            sum[16 * q + k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
          }
        }
        const double v = sum[16 * q] + __shfl_xor_sync(0xffffffffu, sum[16 * q], 1);
        if (!(lane & 1)) s.part[q * kTcBlock + 16 * warp + (lane >> 1)] = v;
      }
    }
    __syncthreads();
    if (h == 0) {
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const double b = r < nrow && q < nr ? p.alpha * p.B[(int64_t)(r0 + r) * p.brs +
                                                           (int64_t)(rhs0 + q) * p.bcs]
                                            : 0.0;
        s.own[q * kTcBlock + r] = b - (TRANS ? s.part[q * kTcBlock + r]
                                             : acc[q] + s.part[q * kTcBlock + r]);
      }
    }
    __syncthreads();
    // x = inverse b, or for a unit diagonal by 64 rows: the inverse of a unit triangle grows
    // with its order, and with it the error (n = 1001, L of a partially pivoted LU, against 64
    // bits: 9.2e-15 by 128 rows, 6.6e-15 by 64; other factors by 128 rows are the closer ones)
    double x[NR];
#pragma unroll
    for (int q = 0; q < NR; ++q) x[q] = 0.0;
    if constexpr (UNIT) {
      const int first = p.lower_eff ? 0 : 1;
      // rows 64 ra .. times columns 64 ca .. of s.inv and s.own, 32 columns by each h; for h = 0
      // in x
      auto product = [&](int ra, int ca) {
#pragma unroll
        for (int q = 0; q < NR; ++q) x[q] = 0.0;
        const int k0 = 64 * ca + 32 * h;
        if ((r >> 6) == ra) {
#pragma unroll 8
          for (int k = k0; k < k0 + 32; ++k) {
            const double v = s.inv[k * kTcLd + r];
#pragma unroll
            for (int q = 0; q < NR; ++q) x[q] = fma(v, s.own[q * kTcBlock + k], x[q]);
          }
          if (h == 1) {
#pragma unroll
            for (int q = 0; q < NR; ++q) s.part[q * kTcBlock + r] = x[q];
          }
        }
        __syncthreads();
        if ((r >> 6) == ra && h == 0) {
#pragma unroll
          for (int q = 0; q < NR; ++q) x[q] += s.part[q * kTcBlock + r];
        }
      };
      for (int step = 0; step < 3; ++step) {
        const int ra = step == 0 ? first : 1 - first, ca = step == 2 ? 1 - first : first;
        product(ra, ca);
        if ((r >> 6) == ra && h == 0) {
#pragma unroll
          for (int q = 0; q < NR; ++q) {
            double &to = s.own[q * kTcBlock + r];
            to = step == 1 ? to - x[q] : x[q];
          }
        }
        __syncthreads();
      }
      // (as the sum of the two halves below)
#pragma unroll
      for (int q = 0; q < NR; ++q) x[q] = h == 0 ? s.own[q * kTcBlock + r] : 0.0;
    } else {
      const double *iv = s.inv + 64 * h * kTcLd + r;
      // (the inverse's 64 x 64 block of zeros is left out: an infinity in b stays on its side)
      if (h == (r >> 6) || (h == 0) == (p.lower_eff != 0)) {
#pragma unroll 16
        for (int k = 0; k < 64; ++k) {
          const double v = iv[k * kTcLd];
#pragma unroll
          for (int q = 0; q < NR; ++q) x[q] = fma(v, s.own[q * kTcBlock + 64 * h + k], x[q]);
        }
      }
    }
    if (h == 1) {
#pragma unroll
      for (int q = 0; q < NR; ++q) s.part[q * kTcBlock + r] = x[q];
    }
    __syncthreads();
    // A CTA that gave up leaves its rows as they are and sends NaN instead of x, so that the others'
    // waits end; its own memory is written until their x is here (waited for below).
    const bool late = s.late;
    if (h == 0) {
#pragma unroll
      for (int q = 0; q < NR; ++q) {
        const double v = r < nrow ? x[q] + s.part[q * kTcBlock + r] : 0.0;
        s.own[q * kTcBlock + r] = late ? __longlong_as_double(0x7ff8000000000000ll) : v;
        if (r < nrow && q < nr && !late)
          p.B[(int64_t)(r0 + r) * p.brs + (int64_t)(rhs0 + q) * p.bcs] = v;
      }
    }
    __syncthreads();
    // to the later CTAs, a warp per CTA
    for (int d = c + 1 + warp; d < nblk; d += kTcThreads / 32) {
      const uint32_t to = cl_map(s.x[c], d), mb = cl_map(&s.bar[c], d);
      const double2 *src = reinterpret_cast<const double2 *>(s.own);
#pragma unroll
      for (int e = lane; e < NR * kTcBlock / 2; e += 32) {
        const double2 v = src[e];
        asm volatile(
            "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(
                to + 16 * e),
            "d"(v.x), "d"(v.y), "r"(mb)
            : "memory");
      }
    }
    if (late)
      for (int t = 0; t < c; ++t) mbar_wait(&s.bar[t], 0, p.status);
  }
  cl_sync();  // no CTA leaves while another may still write into its memory
}

template <typename TA, bool TRANS, int NR, bool UNIT>
int tc_launch(mo_ctx *ctx, const FewArgs &p, int ctas, int groups) {
  const void *fn = (const void *)trsm_cluster_kernel<TA, TRANS, NR, UNIT>;
  if (int rc = mo_smem_attr(fn, (int)sizeof(TcSmem<NR>))) return rc;
  MO_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, groups);
  cfg.blockDim = dim3(kTcThreads);
  cfg.dynamicSmemBytes = sizeof(TcSmem<NR>);
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim = {(unsigned)ctas, 1, 1};
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (ctas > 8) {  // not portable: ask
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, trsm_cluster_kernel<TA, TRANS, NR, UNIT>, &cfg) != cudaSuccess ||
        clusters < 1) {
      cudaGetLastError();
      return 1;
    }
  }
  void *args[] = {const_cast<FewArgs *>(&p)};
  ProfScope ps;
  prof_begin(ctx, ps, sizeof(TA) == 4 ? MO_PROF_IR : MO_PROF_GEMM);
  const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
  prof_end(ctx, ps, (double)p.N * p.N * p.nrhs,
           sizeof(TA) * (double)p.N * p.N / 2 + 8.0 * 2.0 * p.N * p.nrhs);
  MO_CUDA_TRY(e);
  return MO_OK;
}

// MO_OK, an error, or 1: not for the cluster (more than 16 blocks of 128, or more than 128 CTAs,
// which would run in several waves; the FP64 callers cut their blocks to fit, few_sweep)
template <typename TA>
int tc_run(mo_ctx *ctx, const FewArgs &p) {
  const int nblk = (p.N + kTcBlock - 1) / kTcBlock;
  if (nblk > kTcMax) return 1;
  int ctas = 1;
  while (ctas < nblk) ctas *= 2;
  const int per = p.nrhs > 2 ? 4 : p.nrhs, groups = (p.nrhs + per - 1) / per;
  if (groups * ctas > 128) return 1;
  auto go = [&](auto trans, auto unit) {
    constexpr bool T = decltype(trans)::value, U = decltype(unit)::value;
    return per == 1   ? tc_launch<TA, T, 1, U>(ctx, p, ctas, groups)
           : per == 2 ? tc_launch<TA, T, 2, U>(ctx, p, ctas, groups)
                      : tc_launch<TA, T, 4, U>(ctx, p, ctas, groups);
  };
  constexpr std::true_type yes{};
  constexpr std::false_type no{};
  if constexpr (sizeof(TA) == 8)  // (the mixed factor's triangles have no unit diagonal)
    if (p.unit) return p.trans ? go(yes, yes) : go(no, yes);
  return p.trans ? go(yes, no) : go(no, no);
}

}  // namespace
}  // namespace mo
