// FP64 GEMM / SYRK engine for sm_100a.
//
// A unit of work is one 128x64 tile of C, computed by one consumer warpgroup (2 x 2 warps
// of 64 x 32) on the FP64 tensor pipe through mma.sync.m16n8k4.f64.  A CTA (one per SM)
// runs two such warpgroups, each with its own list of units and its own 4-stage
// shared-memory ring of 16-wide k-slabs of op(A) and op(B), filled by 2-D TMA (128-byte
// swizzle, OOB zero fill) or, where the base or leading dimension breaks TMA's 16-byte
// rules (arbitrary FloatMatrix views, e.g. an odd order), by 8-byte cp.async from two
// producer warps per ring into the identical swizzled layout.
//
// Two independent warpgroups, because an epilogue (C read, scaled, written) leaves the
// FP64 pipe idle: while one warpgroup writes its tile the other keeps multiplying.  A lone
// warp per scheduler reaches about 0.85 of the pipe's rate, two reach 0.98, so both
// multiply at once most of the time, the second one started half a tile late so that their
// epilogues do not coincide.
//
// What bounds it: the FP64 pipe (37.0 TFLOP/s measured), plus per tile the C traffic, which
// at K = 128 is a third of the tile's time.  Measured on B200, C -= A B, against one 128x128
// tile per CTA shared by both warpgroups with a per-element epilogue: 8192^2 x K = 128 24.0 ->
// 29.3 TFLOP/s, K = 256 28.6 -> 32.0; 16384^2 x 256 29.1 -> 32.7; 2048^3 33.2 -> 33.7;
// 3001 x 1777 x 2503 with odd leading dimensions, op(A) = A^T, 12.8 -> 30.9 (one producer
// warp before).
//
// Tiles are 64x128 (warps 1 x 4) where C is op(A) itself (in-place products from the right:
// a tile must cover all its columns) or has at most 64 rows.
//
// Arithmetic (calgo/dmmat_gemm.c:364-415 semantics): C = beta*C + alpha*sum_k, with
// beta == 0 never reading C.  SYRK modes restrict tiles and elements to one triangle and
// can apply beta only on diagonal blocks (calgo/dmmat_rank.c:62-127).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "gemm.cuh"

namespace mo {
namespace {

constexpr int BK = 16, STAGES = 4;  // stages per warpgroup
constexpr int GROUP_WARPS = 4;  // warps of one consumer warpgroup
// warpgroup 0 = producers (one warp per ring issues TMA loads, or two its cp.async copies),
// warpgroups 1-2 = consumers.
// Register split via setmaxnreg: launch 384 x 168 = 64512 = 128 x 40 + 256 x 232.
constexpr int THREADS = 384;
constexpr int PRODUCER_REGS = 40, CONSUMER_REGS = 232;
static_assert(THREADS * 168 >= 128 * PRODUCER_REGS + 256 * CONSUMER_REGS, "register split");
// Tile geometry of one instantiation: TALL 128 x 64, WIDE 64 x 128; warp tiles of 64 x 32.
template <bool WIDE>
struct Geo {
  static constexpr int TBM = WIDE ? 64 : 128, TBN = WIDE ? 128 : 64;
  static constexpr int WN = TBN / 32;  // warp columns of a warpgroup
};
constexpr int STAGE_DBL = (128 + 64) * BK;
constexpr uint32_t STAGE_BYTES = STAGE_DBL * 8;
constexpr int SMEM_BYTES = 2 * STAGES * STAGE_BYTES + 1024 + (4 * STAGES + 1) * 8;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
constexpr int TILE_DBL = 128 * 64;  // elements of a tile (a stream-K partial)

// Swizzled shared-memory layouts (TMA SWIZZLE_128B: 16-byte chunk ^= 128-byte row % 8).
// K-major slab: 128 rows (m or n) of 16 k-values (128 B per row).
__device__ __forceinline__ int kmaj_off(int mn, int k) {
  return mn * 16 + ((((k >> 1) ^ (mn & 7))) << 1) + (k & 1);
}
// MN-major slab: 8 boxes of [16 k-rows x 16 mn-values].
__device__ __forceinline__ int mnmaj_off(int mn, int k) {
  return (mn >> 4) * 256 + k * 16 + (((((mn & 15) >> 1) ^ (k & 7))) << 1) + (mn & 1);
}

struct KParams {
  int M, N, K;
  double alpha, beta;
  const double *A;
  int64_t lda;
  const double *B;
  int64_t ldb;
  double *C;
  int64_t ldc;
  int mode, beta_block;
  int *status;
  const int *skip;
  int tiles_m, tiles_n;
  int total_tiles;  // tiles of C (the triangle's tiles in SYRK modes)
  int kt;           // k-slabs per tile
  int workers;      // warpgroups with work of their own: 2 per CTA
  int dp_tiles;     // tiles [0, dp_tiles) are processed whole, round-robin over workers
  int sk_iters;     // stream-K iterations over the remaining tiles
  int sk_chunk;     // stream-K iterations per worker
  double *partial;  // [workers][TILE_DBL] stream-K partial accumulators
  int *flags;       // [workers] epoch stamps of published partials
  int epoch;
};

// cp.async producer for one ROWS x 16 slab (ROWS = 64 or 128) of an operand whose element
// (mn, k) lives at src[k + mn*ld] (KMAJ) or src[mn + k*ld] (!KMAJ); out-of-range elements
// are zero-filled.  The two producer warps take half of the slab each (pw = 0, 1).
template <bool KMAJ, int ROWS>
__device__ __forceinline__ void load_slab_cpasync(double *dst, const double *src, int64_t ld,
                                                  int mn0, int k0, int MN, int K, int pw,
                                                  int lane) {
  if constexpr (KMAJ) {
    // 16 lanes along k, two rows per instruction; 8 rows later the swizzle repeats
    const int k = lane & 15, mn1 = (ROWS / 2) * pw + (lane >> 4);
    const double *s = src + (k0 + k) + (int64_t)(mn0 + mn1) * ld;
    const int left = k0 + k < K ? MN - mn0 - mn1 : 0;  // rows of this lane's column in range
    uint32_t d[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) d[j] = smem_u32(dst + kmaj_off(mn1 + 2 * j, k));
    const int64_t ld2 = 2 * ld;
#pragma unroll 1
    for (int i = 0; i < ROWS / 4; i += 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const bool ok = 2 * (i + j) < left;
        cp_async_8(d[j] + i * (2 * 16 * 8), ok ? s : src, ok ? 8u : 0u);
        s += ld2;
      }
    }
  } else {
    const int left = MN - mn0 - lane;
    const double *s = src + (mn0 + lane) + (int64_t)(k0 + 8 * pw) * ld;
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
      const int k = 8 * pw + i;
      const int lim = k0 + k < K ? left : 0;
#pragma unroll
      for (int j = 0; j < ROWS / 32; ++j) {
        const bool ok = 32 * j < lim;
        cp_async_8(smem_u32(dst + mnmaj_off(32 * j + lane, k)), ok ? s + 32 * j : src, ok ? 8u : 0u);
      }
      s += ld;
    }
  }
}

__device__ __forceinline__ void tile_coords(const KParams &p, int t, int &tm, int &tn) {
  if (p.mode == kGemm || p.mode == kGemmLower || p.mode == kGemmUpper) {
    // groups of GROUP_M tile rows, column-major inside a group: a wave of persistent CTAs
    // touches GROUP_M row panels of A and a narrow band of B, which stay in L2
    constexpr int GROUP_M = 8;
    const int per_group = GROUP_M * p.tiles_n;
    const int grp = t / per_group, r = t % per_group;
    const int m_first = grp * GROUP_M;
    const int gm = min(GROUP_M, p.tiles_m - m_first);
    tm = m_first + r % gm;
    tn = r / gm;
    return;
  }
  // t / 2 enumerates the triangle of 128 x 128 squares row by row, (r, c) with c <= r, and
  // t & 1 the square's two tiles (the second one of a diagonal square may lie past N)
  const int half = t & 1;
  t >>= 1;
  int r = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while ((r + 1) * (r + 2) / 2 <= t) ++r;
  while (r * (r + 1) / 2 > t) --r;
  const int c = t - r * (r + 1) / 2;
  if (p.mode == kSyrkLower) {
    tm = r;
    tn = 2 * c + half;
  } else {
    tm = c;
    tn = 2 * r + half;
  }
}

// The worker index of a CTA's warpgroup: the first gridDim.x workers are the CTAs'
// warpgroups 0, so that every SM has one before any has two.  A stream-K worker publishes its
// own partial sum before it waits for those of lower-numbered workers, and these are in CTAs
// that started before its own, but for one worker per launch: the owner of the tile that
// spans the last warpgroup 0 and the first warpgroup 1 waits for CTAs that other work may
// still keep from being placed.  All others go on and end, so they are placed in time.  (Stream-K
// ranges numbered CTA by CTA would spare that wait and cost 3 to 5 % with odd leading
// dimensions: 3001 x 1777 x 2503 862 -> 893 us, 1500^3 231 -> 245.)
__device__ __forceinline__ int worker_of(const KParams &p, int grp) {
  return grp * gridDim.x + blockIdx.x;
}

// One unit of work: k-slabs [k0, k1) of tile `tile`.  owner: this worker finishes the tile
// (adds the partials of workers [first_contrib, w) and writes C); otherwise it publishes
// its partial sum.
struct Unit {
  int tile, k0, k1;
  bool owner;
  int first_contrib;
};

// Worker w's units in processing order: whole tiles first, then its stream-K range from the
// highest tile down (so that a partial is published before this worker waits for the
// partials of lower-numbered ones).  Returns false past the last unit; fills u otherwise.
__device__ __forceinline__ bool unit_at(const KParams &p, int w, int idx, Unit &u) {
  const int P = p.workers;
  if (w >= P) return false;
  const int ndp = (p.dp_tiles > w) ? (p.dp_tiles - w + P - 1) / P : 0;
  if (idx < ndp) {
    u.tile = w + idx * P;
    u.k0 = 0;
    u.k1 = p.kt;
    u.owner = true;
    u.first_contrib = w;
    return true;
  }
  idx -= ndp;
  if (p.sk_iters <= 0) return false;
  const int s = w * p.sk_chunk, e = min(s + p.sk_chunk, p.sk_iters);
  if (s >= e) return false;
  const int first = s / p.kt, last = (e - 1) / p.kt;
  const int t = last - idx;
  if (t < first) return false;
  const int ts = t * p.kt, te = ts + p.kt;
  u.tile = p.dp_tiles + t;
  u.k0 = max(s, ts) - ts;
  u.k1 = min(e, te) - ts;
  u.owner = (e >= te);
  u.first_contrib = ts / p.sk_chunk;
  return true;
}

__device__ __forceinline__ void group_bar(int g) {
  if (g == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}

template <bool A_KMAJ, bool B_KMAJ, bool USE_TMA, bool WIDE>
__global__ void __launch_bounds__(THREADS, 1)
    dgemm_tile_kernel(const __grid_constant__ CUtensorMap tmA,
                      const __grid_constant__ CUtensorMap tmB, const KParams p) {
  using G = Geo<WIDE>;
  extern __shared__ unsigned char smem_raw[];
  const uintptr_t base = (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023);
  uint64_t *bars = reinterpret_cast<uint64_t *>(base + 2 * STAGES * STAGE_BYTES);
  uint64_t *late = bars + 4 * STAGES;  // warpgroup 0 is halfway through its first unit
  __shared__ int s_abort[2];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (p.skip && *(volatile const int *)p.skip) return;
  if (threadIdx.x == 0) {
    for (int r = 0; r < 2; ++r)
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(&bars[2 * STAGES * r + s], USE_TMA ? 1u : 64u);             // full
        mbar_init(&bars[2 * STAGES * r + STAGES + s], GROUP_WARPS);           // empty
      }
    mbar_init(late, GROUP_WARPS);
    s_abort[0] = s_abort[1] = 0;
    fence_barrier_init();
  }
  __syncthreads();

  if (warp < 4) {
    // ------------------------------ producer warpgroup ------------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGS));
    const int grp = USE_TMA ? warp : warp >> 1;  // ring
    if (grp > 1) return;
    uint64_t *full = bars + 2 * STAGES * grp, *empty = full + STAGES;
    double *tiles = reinterpret_cast<double *>(base) + grp * STAGES * STAGE_DBL;
    const int w = worker_of(p, grp);
    int it = 0;  // ring position, continues across units
    Unit u;
    for (int ui = 0; unit_at(p, w, ui, u); ++ui) {
      int tm, tn;
      tile_coords(p, u.tile, tm, tn);
      const int m0 = tm * G::TBM, n0 = tn * G::TBN;
      for (int kt = u.k0; kt < u.k1; ++kt, ++it) {
        const int s = it % STAGES;
        const uint32_t ph = (it / STAGES) & 1;
        if (!mbar_wait(&empty[s], ph ^ 1u, p.status)) {
          if constexpr (!USE_TMA) asm volatile("cp.async.wait_all;" ::: "memory");
          return;
        }
        double *As = tiles + s * STAGE_DBL;
        double *Bs = As + G::TBM * BK;
        const int k0 = kt * BK;
        if constexpr (USE_TMA) {
          if (lane == 0) {
            mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
            // K-major maps carry boxes of the tile's rows, MN-major maps 16 x 16 boxes
            if (A_KMAJ) {
              tma_load_2d(As, &tmA, &full[s], k0, m0);
            } else {
#pragma unroll
              for (int bb = 0; bb < G::TBM / 16; ++bb)
                tma_load_2d(As + bb * 256, &tmA, &full[s], m0 + 16 * bb, k0);
            }
            if (B_KMAJ) {
              tma_load_2d(Bs, &tmB, &full[s], k0, n0);
            } else {
#pragma unroll
              for (int bb = 0; bb < G::TBN / 16; ++bb)
                tma_load_2d(Bs + bb * 256, &tmB, &full[s], n0 + 16 * bb, k0);
            }
          }
          __syncwarp();
        } else {
          load_slab_cpasync<A_KMAJ, G::TBM>(As, p.A, p.lda, m0, k0, p.M, p.K, warp & 1, lane);
          load_slab_cpasync<B_KMAJ, G::TBN>(Bs, p.B, p.ldb, n0, k0, p.N, p.K, warp & 1, lane);
          cp_async_arrive_noinc(&full[s]);
        }
      }
    }
    if constexpr (!USE_TMA) asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }

  // ------------------------------ consumer warpgroups ------------------------------
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONSUMER_REGS));
  const int grp = (warp - 4) >> 2;     // consumer warpgroup, and its ring
  const int ct = threadIdx.x & 127;     // thread of the warpgroup
  const int cw = warp & 3;
  const int w = worker_of(p, grp);
  uint64_t *full = bars + 2 * STAGES * grp, *empty = full + STAGES;
  const double *tiles = reinterpret_cast<const double *>(base) + grp * STAGES * STAGE_DBL;
  const int wm = cw / G::WN, wn = cw % G::WN;  // 64 x 32 warp tile of the unit's tile
  const int g = lane >> 2, t = lane & 3;
  // Which row (column) of a 16-wide block of the slab a fragment's index stands for: any
  // permutation gives the same products as long as the epilogue uses it too, and these make
  // every fragment load touch all 32 banks once (in plain order two rows 128 bytes apart
  // meet in the same 16-byte chunk: a two-way conflict on every load).  Index i = 0..7 of
  // the fragment, h = 0, 1 (rows i and i + 8 of A's fragment; the two 8-column tiles of B):
  //   K-major : 2 (i & 3) + (i >> 2) + 8 h        MN-major : (i & 1) + 8 (i >> 1 & 1) + 2 (i >> 2) + 4 h
  // Element (mn, k), k = kk + t, K-major: mn*16 + 2*((k>>1) ^ (mn&7)) + (k&1);
  // MN-major: (mn>>4)*256 + k*16 + 2*(((mn&15)>>1) ^ (k&7)) + (mn&1).  The offsets are split
  // into a per-thread part computed once and compile-time constants (mt, nt, kk).
  const int rk = 2 * (g & 3) + (g >> 2);
  int kv[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) kv[q] = 2 * ((2 * q + (t >> 1)) ^ (rk & 7)) + (t & 1);
  int xa[2][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int q2 = 0; q2 < 2; ++q2)
      xa[h][q2] = 2 * ((4 * ((g >> 1) & 1) + (g >> 2) + 2 * h) ^ (4 * q2 + t));
  const int a_base = A_KMAJ ? (wm * 64 + rk) * 16 : (wm * 4) * 256 + t * 16 + (g & 1);
  const int b_base =
      G::TBM * BK + (B_KMAJ ? (wn * 32 + rk) * 16 : (wn * 2) * 256 + t * 16 + (g & 1));
  // the element of the warp's part of C in accumulator [mt][nt][r]: row fr + 16 mt + RH (r >> 1),
  // column fc + 16 (nt >> 1) + CH (nt & 1) + CE (r & 1)
  constexpr int RH = A_KMAJ ? 8 : 4, CH = B_KMAJ ? 8 : 4, CE = B_KMAJ ? 2 : 1;
  const int fr = A_KMAJ ? rk : (g & 1) + 8 * ((g >> 1) & 1) + 2 * (g >> 2);
  const int fc = B_KMAJ ? 4 * (t & 1) + (t >> 1) : 8 * (t & 1) + 2 * (t >> 1);
  int it = 0;
  Unit u;
  for (int ui = 0; unit_at(p, w, ui, u); ++ui) {
    int tm, tn;
    tile_coords(p, u.tile, tm, tn);
    const int m0 = tm * G::TBM, n0 = tn * G::TBN;
    // warm L2 with this warp's C sub-tile (64 rows x 32 cols: 4 lines of 128 B per column)
    if (u.owner && (p.beta != 0.0 || p.beta_block > 0)) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int col = n0 + wn * 32 + lane;
        const int row = m0 + wm * 64 + 16 * q;
        if (col < p.N && row < p.M)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.C + row + (int64_t)col * p.ldc));
      }
    }
    double acc[4][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;

    // a warp whose 32 columns all lie past N (narrow C, e.g. a residual with few
    // right-hand sides) keeps the stage hand-shake but issues no loads or MMAs
    const bool idle = n0 + wn * 32 >= p.N || m0 + wm * 64 >= p.M;
    // fragments of k-step kk = 4 q of the slab at `st`
    auto load_frag = [&](const double *st, int q, double (&a)[4][2], double (&b)[4]) {
      const int q2 = q & 1, kk = 4 * q;
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        if constexpr (A_KMAJ) {
          a[mt][0] = st[a_base + kv[q] + mt * 256];
          a[mt][1] = st[a_base + kv[q] + mt * 256 + 128];
        } else {
          a[mt][0] = st[a_base + xa[0][q2] + mt * 256 + kk * 16];
          a[mt][1] = st[a_base + xa[1][q2] + mt * 256 + kk * 16];
        }
      }
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        if constexpr (B_KMAJ)
          b[nt] = st[b_base + kv[q] + nt * 128];
        else
          b[nt] = st[b_base + xa[nt & 1][q2] + (nt >> 1) * 256 + kk * 16];
      }
    };
    const int nk = u.k1 - u.k0;
    // two or more whole tiles each: warpgroup 1 starts half a tile after warpgroup 0
    const bool stagger = ui == 0 && p.dp_tiles > p.workers && nk > 0;
    if (stagger && grp == 1 && !mbar_wait(late, 0, p.status)) return;
    const int half = stagger && grp == 0 ? nk / 2 : -1;
    if (idle) {
      for (int kt = 0; kt < nk; ++kt, ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(&full[s], (it / STAGES) & 1, p.status)) return;
        if (lane == 0) {
          mbar_arrive(&empty[s]);
          if (kt == half) mbar_arrive(late);
        }
      }
    } else {
      for (int kt = 0; kt < nk; ++kt, ++it) {
        const int s = it % STAGES;
        if (!mbar_wait(&full[s], (it / STAGES) & 1, p.status)) return;
        const double *st = tiles + s * STAGE_DBL;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          double a[4][2], b[4];
          load_frag(st, q, a, b);
#pragma unroll
          for (int mt = 0; mt < 4; ++mt)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) dmma_16x8x4(acc[mt][nt], a[mt][0], a[mt][1], b[nt]);
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&empty[s]);
          if (kt == half) mbar_arrive(late);
        }
      }
    }

    if (!u.owner) {
      // publish the partial sum (fragment order: register r of thread ct at
      // [r * 128 + ct], coalesced per warp), then stamp this worker's flag
      double *slot = p.partial + (size_t)w * TILE_DBL;
#pragma unroll
      for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r) slot[((mt * 4 + nt) * 4 + r) * 128 + ct] = acc[mt][nt][r];
      __threadfence();
      group_bar(grp);
      if (ct == 0) atomicExch(&p.flags[w], p.epoch);
      continue;
    }
    if (u.first_contrib < w) {
      // add the partials of the lower-numbered workers that computed the tile's first slabs
      for (int c = u.first_contrib; c < w; ++c) {
        if (ct == 0) {
          uint32_t i = 0;
          while (atomicAdd(&p.flags[c], 0) != p.epoch) {
            if (++i > MO_SPIN_LIMIT) {
              set_status(p.status, MO_EDEVTIMEOUT);
              s_abort[grp] = 1;
              break;
            }
          }
          __threadfence();
        }
        group_bar(grp);
        if (s_abort[grp]) return;
        const double *slot = p.partial + (size_t)c * TILE_DBL;
#pragma unroll
        for (int mt = 0; mt < 4; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r)
              acc[mt][nt][r] += __ldcg(slot + ((mt * 4 + nt) * 4 + r) * 128 + ct);
      }
    }

    // ------------------------------ epilogue ------------------------------
    // C is read unless beta == 0 everywhere (with diagonal-block beta, off-block
    // elements use beta = 1).  All loads of a batch are issued before any store, so the L2
    // round trips overlap (stores may alias later loads, which would otherwise serialize
    // them).
    const bool need_c = p.beta != 0.0 || p.beta_block > 0;
    const int wr = m0 + wm * 64, wc = n0 + wn * 32;  // the warp's 64 x 32 part of C
    bool whole = wr + 64 <= p.M && wc + 32 <= p.N && p.beta_block == 0;
    if (p.mode == kSyrkLower || p.mode == kGemmLower) whole = whole && wr >= wc + 31;
    if (p.mode == kSyrkUpper || p.mode == kGemmUpper) whole = whole && wr + 63 <= wc;
    if (whole) {
      // every element is kept and has the same beta: no tests per element.  (With the tests
      // and their branches on all 64 elements the epilogue took as long as 85 columns of K.)
      const double alpha = p.alpha, beta = p.beta;
      double *cp[4];
      cp[0] = p.C + (wr + fr) + (int64_t)(wc + fc) * p.ldc;
      cp[1] = cp[0] + CH * p.ldc;
      cp[2] = cp[0] + 16 * p.ldc;
      cp[3] = cp[2] + CH * p.ldc;
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        if (beta != 0.0) {
          double cv[4][4];
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r)
              cv[nt][r] = __ldcg(cp[nt] + mt * 16 + RH * (r >> 1) + CE * (r & 1) * p.ldc);
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r)
              cp[nt][mt * 16 + RH * (r >> 1) + CE * (r & 1) * p.ldc] =
                  fma(beta, cv[nt][r], alpha * acc[mt][nt][r]);
        } else {
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r)
              cp[nt][mt * 16 + RH * (r >> 1) + CE * (r & 1) * p.ldc] = alpha * acc[mt][nt][r];
        }
      }
      continue;
    }
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
#pragma unroll
      for (int nh = 0; nh < 4; nh += 2) {
        double cv[2][4];
        const int row0 = wr + fr + mt * 16, col0 = wc + fc + nh * 8;
        double *c0 = p.C + row0 + (int64_t)col0 * p.ldc;
        unsigned keep = 0;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const int row = row0 + RH * (r >> 1), col = col0 + CH * nt + CE * (r & 1);
            bool k = row < p.M && col < p.N;
            if ((p.mode == kSyrkLower || p.mode == kGemmLower) && row < col) k = false;
            if ((p.mode == kSyrkUpper || p.mode == kGemmUpper) && row > col) k = false;
            keep |= (k ? 1u : 0u) << (nt * 4 + r);
            cv[nt][r] = (k && need_c)
                            ? __ldcg(c0 + RH * (r >> 1) + (int64_t)(CH * nt + CE * (r & 1)) * p.ldc)
                            : 0.0;
          }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            if (!(keep >> (nt * 4 + r) & 1u)) continue;
            const int row = row0 + RH * (r >> 1), col = col0 + CH * nt + CE * (r & 1);
            double bet = p.beta;
            if (p.beta_block > 0 && (row / p.beta_block) != (col / p.beta_block)) bet = 1.0;
            double v = p.alpha * acc[mt][nh + nt][r];
            if (bet != 0.0) v = fma(bet, cv[nt][r], v);
            c0[RH * (r >> 1) + (int64_t)(CH * nt + CE * (r & 1)) * p.ldc] = v;
          }
      }
    }
  }
}

// ---- few small tiles -------------------------------------------------------------------
// A product with a short K whose 128 x 64 tiles would occupy a fraction of the SMs (a panel
// of a factorization, a small user matrix) runs on 32 x 32 tiles instead, one CTA of four
// warps each: four to eight times the CTAs, no tensor maps, and little padding.  In-place
// products keep one CTA per strip that is both read and written: 32 x 128 tiles where C is
// op(A) (N <= 128), 128 x 32 where C is op(B) (M <= 128).  Operands of any alignment come by
// 8-byte cp.async into a ring of 16-wide slabs, k-row by k-row with a row stride of 4 mod 16
// doubles, so the fragment loads touch every bank once.
template <int TM, int TN>
struct SmallGeo {
  static constexpr int STAGES = TM * TN > 2048 ? 4 : 6;
  static constexpr int LA = TM + 4, LBS = TN + 4;
  static constexpr int STAGE = 16 * (LA + LBS);
  static constexpr int SMEM = STAGES * STAGE * 8;
};

template <bool A_KMAJ, bool B_KMAJ, int TM, int TN, int WM, int WN>
__global__ void __launch_bounds__(WM *WN * 32) dgemm_small_kernel(const KParams p) {
  using G = SmallGeo<TM, TN>;
  constexpr int NT = WM * WN * 32, FM = TM / WM / 16, FN = TN / WN / 8, STG = G::STAGES;
  extern __shared__ double small_smem[];
  const int m0 = blockIdx.x * TM, n0 = blockIdx.y * TN;
  if ((p.mode == kSyrkLower || p.mode == kGemmLower) && m0 + TM - 1 < n0) return;
  if ((p.mode == kSyrkUpper || p.mode == kGemmUpper) && m0 > n0 + TN - 1) return;
  if (p.skip && *(volatile const int *)p.skip) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int wr = (warp % WM) * (TM / WM), wc = (warp / WM) * (TN / WN);

  // one operand's slab: ROWS x 16 at s[k * ld + mn]
  auto fetch = [&](auto kmaj, auto rows, double *s, int ls, const double *src, int64_t ld, int mn0,
                   int MN, int k0) {
    constexpr bool KM = decltype(kmaj)::value;
    constexpr int ROWS = decltype(rows)::value;
#pragma unroll
    for (int e = tid; e < ROWS * 16; e += NT) {
      const int k = KM ? e & 15 : e / ROWS, mn = KM ? e >> 4 : e % ROWS;
      const bool ok = mn0 + mn < MN && k0 + k < p.K;
      const double *q = KM ? src + (k0 + k) + (int64_t)(mn0 + mn) * ld
                           : src + (mn0 + mn) + (int64_t)(k0 + k) * ld;
      cp_async_8(s + k * ls + mn, ok ? q : src, ok ? 8u : 0u);
    }
  };
  auto load = [&](int kt, int end) {
    if (kt < end) {
      double *s = small_smem + (kt % STG) * G::STAGE;
      fetch(std::integral_constant<bool, A_KMAJ>{}, std::integral_constant<int, TM>{}, s, G::LA, p.A,
            p.lda, m0, p.M, kt * BK);
      fetch(std::integral_constant<bool, B_KMAJ>{}, std::integral_constant<int, TN>{},
            s + 16 * G::LA, G::LBS, p.B, p.ldb, n0, p.N, kt * BK);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // this CTA's slabs: all of them, or a chunk of K (blockIdx.z) whose sums go to p.partial
  const int kt0 = blockIdx.z * p.sk_chunk, kt1 = min(p.kt, kt0 + p.sk_chunk);
  double acc[FM][FN][4] = {};
#pragma unroll
  for (int s = 0; s < STG - 1; ++s) load(kt0 + s, kt1);
  for (int kt = kt0; kt < kt1; ++kt) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STG - 2) : "memory");
    __syncthreads();
    load(kt + STG - 1, kt1);
    const double *sa = small_smem + (kt % STG) * G::STAGE + t * G::LA + wr + g;
    const double *sb = small_smem + (kt % STG) * G::STAGE + 16 * G::LA + t * G::LBS + wc + g;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      double a[FM][2], b[FN];
#pragma unroll
      for (int i = 0; i < FM; ++i) {
        a[i][0] = sa[4 * q * G::LA + 16 * i];
        a[i][1] = sa[4 * q * G::LA + 16 * i + 8];
      }
#pragma unroll
      for (int j = 0; j < FN; ++j) b[j] = sb[4 * q * G::LBS + 8 * j];
#pragma unroll
      for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < FN; ++j) dmma_16x8x4(acc[i][j], a[i][0], a[i][1], b[j]);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (gridDim.z > 1) {
    double *out = p.partial + ((size_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x * (TM * TN) +
                  (size_t)blockIdx.x * (TM * TN);
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
      for (int j = 0; j < FN; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r)
          out[(wr + 16 * i + g + 8 * (r >> 1)) + (wc + 8 * j + 2 * t + (r & 1)) * TM] = acc[i][j][r];
    return;
  }
  // epilogue, as the engine's general one: every C is read before any is written
  const bool need_c = p.beta != 0.0 || p.beta_block > 0;
#pragma unroll
  for (int i = 0; i < FM; ++i) {
    double cv[FN][4];
    unsigned keep = 0;
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = m0 + wr + 16 * i + g + 8 * (r >> 1), col = n0 + wc + 8 * j + 2 * t + (r & 1);
        bool k = row < p.M && col < p.N;
        if ((p.mode == kSyrkLower || p.mode == kGemmLower) && row < col) k = false;
        if ((p.mode == kSyrkUpper || p.mode == kGemmUpper) && row > col) k = false;
        keep |= (k ? 1u : 0u) << (4 * j + r);
        cv[j][r] = (k && need_c) ? __ldcg(p.C + row + (int64_t)col * p.ldc) : 0.0;
      }
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (!(keep >> (4 * j + r) & 1u)) continue;
        const int row = m0 + wr + 16 * i + g + 8 * (r >> 1), col = n0 + wc + 8 * j + 2 * t + (r & 1);
        double bet = p.beta;
        if (p.beta_block > 0 && (row / p.beta_block) != (col / p.beta_block)) bet = 1.0;
        double v = p.alpha * acc[i][j][r];
        if (bet != 0.0) v = fma(bet, cv[j][r], v);
        p.C[row + (int64_t)col * p.ldc] = v;
      }
  }
}

// C = alpha * (the K chunks' partial 32 x 32 tiles, added in order) + beta * C
__global__ void __launch_bounds__(256) small_reduce_kernel(const KParams p, int chunks) {
  const int tiles_m = (p.M + 31) / 32, tiles = tiles_m * ((p.N + 31) / 32);
  const int64_t e = blockIdx.x * (int64_t)256 + threadIdx.x;
  if (e >= (int64_t)p.M * p.N || (p.skip && *(volatile const int *)p.skip)) return;
  const int row = (int)(e % p.M), col = (int)(e / p.M);
  const double *src = p.partial + ((size_t)(col >> 5) * tiles_m + (row >> 5)) * 1024 + (row & 31) +
                      32 * (col & 31);
  double sum = 0.0;
#pragma unroll 8
  for (int c = 0; c < chunks; ++c) sum += __ldcg(src + (size_t)c * tiles * 1024);
  double *dst = p.C + row + (int64_t)col * p.ldc;
  const double v = p.alpha * sum;
  *dst = p.beta != 0.0 ? fma(p.beta, *dst, v) : v;
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// 2-D map over a column-major matrix whose contiguous dimension has `inner` elements.
bool make_tmap(CUtensorMap *tm, const double *ptr, uint64_t inner, uint64_t outer, int64_t ld,
               uint32_t box_inner, uint32_t box_outer) {
  auto fn = encode_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {inner < 1 ? 1 : inner, outer < 1 ? 1 : outer};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 8};
  cuuint32_t box[2] = {box_inner, box_outer};
  cuuint32_t es[2] = {1, 1};
  CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double *>(ptr), dims, strides,
                  box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <bool AK, bool BKM, bool TMA, bool WIDE>
int launch_inst(const KParams &kp, const CUtensorMap &ta, const CUtensorMap &tb, int grid,
                cudaStream_t st) {
  auto kern = dgemm_tile_kernel<AK, BKM, TMA, WIDE>;
  // setmaxnreg.inc only draws on the registers the CTA was launched with: refuse to launch
  // (instead of waiting forever) if the build did not keep the 168-register split (a
  // property of the binary, checked once)
  static std::atomic<int> regs_ok{0};
  if (!regs_ok.load()) {
    cudaFuncAttributes fa;
    MO_CUDA_TRY(cudaFuncGetAttributes(&fa, kern));
    if (fa.numRegs * THREADS < 128 * PRODUCER_REGS + 256 * CONSUMER_REGS) return MO_ENOKERNEL;
    regs_ok.store(1);
  }
  // the shared-memory limit is set on every launch (a cheap host call), so that it holds
  // after a context reset
  if (int rc = mo_smem_attr((const void *)kern, SMEM_BYTES)) return rc;
  kern<<<grid, THREADS, SMEM_BYTES, st>>>(ta, tb, kp);
  MO_CUDA_TRY(cudaGetLastError());
  return MO_OK;
}

template <bool TMA, bool WIDE>
int dispatch(bool ak, bool bk, const KParams &kp, const CUtensorMap &ta, const CUtensorMap &tb,
             int grid, cudaStream_t st) {
  if (ak) return bk ? launch_inst<true, true, TMA, WIDE>(kp, ta, tb, grid, st)
                    : launch_inst<true, false, TMA, WIDE>(kp, ta, tb, grid, st);
  return bk ? launch_inst<false, true, TMA, WIDE>(kp, ta, tb, grid, st)
            : launch_inst<false, false, TMA, WIDE>(kp, ta, tb, grid, st);
}

template <int TM, int TN, int WM, int WN>
int launch_small(bool ak, bool bk, const KParams &kp, cudaStream_t st, int chunks = 1) {
  constexpr int SMEM = SmallGeo<TM, TN>::SMEM;
  const dim3 grid((kp.M + TM - 1) / TM, (kp.N + TN - 1) / TN, chunks);
  auto go = [&](auto kern) -> int {
    if (SMEM > 48 * 1024)
      if (int rc = mo_smem_attr((const void *)kern, SMEM)) return rc;
    kern<<<grid, WM * WN * 32, SMEM, st>>>(kp);
    MO_CUDA_TRY(cudaGetLastError());
    return MO_OK;
  };
  if (ak) return bk ? go(dgemm_small_kernel<true, true, TM, TN, WM, WN>)
                    : go(dgemm_small_kernel<true, false, TM, TN, WM, WN>);
  return bk ? go(dgemm_small_kernel<false, true, TM, TN, WM, WN>)
            : go(dgemm_small_kernel<false, false, TM, TN, WM, WN>);
}

}  // namespace

bool gemm_tma_ok(const GemmArgs &a) {
  auto al = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15u) == 0; };
  return al(a.A) && al(a.B) && (a.lda % 2 == 0) && (a.ldb % 2 == 0) && encode_fn() != nullptr;
}

size_t gemm_partial_bytes(int sms) { return 2 * (size_t)sms * TILE_DBL * sizeof(double); }

// Whether a product goes to the small-tile kernel, and in how many chunks of K (0: the engine).
// Up to 2^27 multiply-adds the engine's start (barriers, tensor maps, the first slabs) and its
// large tiles on a few SMs cost more than the small tiles' extra operand traffic.  Measured,
// engine / small tiles in us: 64^3 12.3 / 4.1, 512 x 128 x 128 18.4 / 6.2, 1000 x 1000 x 128 24.6 /
// 19.3, 500^3 32.8 / 18.4; above, 1500 x 1500 x 128 28.8 / 35.4, 800^3 51.2 / 61.6.  With A
// transposed and B not, both operands' loads run across their columns, and past 1500 tiles the
// small ones lose where there is more than one slab and the engine's tiles fit C: 1414 x 1414 x
// 16 10.9 / 10.4, x 30 14.4 / 16.5, x 68 20.6 / 26.7; 24000 x 128 x 30 16.5 / 20.6; but 160 x 10880 x
// 30 26.8 / 12.7 and 96 x 32000 x 30 28.7 / 20.7 (tiles of 128 rows filled to 5/8 and 3/4), 54400
// x 16 x 30 27.0 / 12.4; with more of K to hide the padding 200 x 8704 x 68 20.6 / 26.7.
// 1000 x 1000 x 30, 1024 tiles, 12.5 / 10.3.
// A C of a few small tiles with a long K is split along K, two CTAs per SM with at least 128
// rows of K each, and the partial tiles are added in order by a second kernel: up to 2^29
// multiply-adds, 128 x 128 x 8000 219 / 21, 512 x 128 x 8000 103 / 62, 1000 x 128 x 8000 101 / 119;
// up to 2^31 for at most 16 tiles, where the engine has one owner adding most SMs' partial
// sums: 64 x 64 x 200000 575 / 96, 128 x 128 x 100000 335 / 171, 100 x 100 x 200000 439 / 341
// (with odd leading dimensions 453 / 432), above it 128 x 128 x 200000 434 / 330 and 449 / 512.
static int small_chunks(const GemmArgs &a, int sms) {
  const double tri = a.mode == kSyrkLower || a.mode == kSyrkUpper ? 0.5 : 1.0;
  const double work = tri * a.M * (double)a.N * a.K;
  if (a.force_fallback || a.N > 65535 * 32) return 0;
  const long long tiles = (long long)((a.M + 31) / 32) * ((a.N + 31) / 32);
  if (a.mode == kGemm && a.sk_partial && a.C != a.A && a.C != a.B && a.K >= 512 && tiles < sms &&
      work <= (tiles <= 16 ? 2147483648.0 : 536870912.0)) {
    const int chunks = (int)std::min<long long>(a.K / 128, 2 * sms / tiles);
    if (chunks > 1) return chunks;
  }
  if (a.transA && !a.transB && a.C != a.B && tri * tiles > 1500 && a.K > BK) {
    auto up = [](double n, int t) { return std::ceil(n / t) * t; };
    const bool wide = a.M <= 64 && a.N > 64;
    const double padded = wide ? up(a.M, 64) * up(a.N, 128) : up(a.M, 128) * up(a.N, 64);
    if (padded <= (a.K > 48 ? 1.4 : 1.25) * a.M * a.N) return 0;
  }
  return a.K <= 4096 && work <= 134217728.0 ? 1 : 0;
}

int launch_gemm(const GemmArgs &a, cudaStream_t stream) {
  if (a.M <= 0 || a.N <= 0) return MO_OK;
  KParams kp;
  kp.M = a.M;
  kp.N = a.N;
  kp.K = a.K < 0 ? 0 : a.K;
  kp.alpha = a.alpha;
  kp.beta = a.beta;
  kp.A = a.A;
  kp.lda = a.lda;
  kp.B = a.B;
  kp.ldb = a.ldb;
  kp.C = a.C;
  kp.ldc = a.ldc;
  kp.mode = a.mode;
  kp.beta_block = a.beta_block;
  kp.status = a.status;
  kp.skip = a.skip;
  // 64 x 128 tiles for C = op(A) itself (each tile then reads and writes its own rows
  // only; N <= 128 there) and for a C of at most 64 rows; 128 x 64 otherwise, which also
  // is the shape of in-place products from the left (C = op(B), M <= 128)
  const bool wide =
      a.mode == kGemm && (a.C == a.A || (a.M <= 64 && a.N > 64 && a.C != a.B));
  const int tbm = wide ? Geo<true>::TBM : Geo<false>::TBM;
  const int tbn = wide ? Geo<true>::TBN : Geo<false>::TBN;
  const int tiles_m = (a.M + tbm - 1) / tbm, tiles_n = (a.N + tbn - 1) / tbn;
  kp.tiles_m = tiles_m;
  kp.tiles_n = tiles_n;
  long long T;
  if (a.mode == kGemm || a.mode == kGemmLower || a.mode == kGemmUpper) {
    T = (long long)tiles_m * tiles_n;
  } else {
    if (a.M != a.N) return MO_EINVAL;
    T = (long long)tiles_m * (tiles_m + 1);  // two tiles per 128 x 128 square
  }
  if (T <= 0 || T > 0x7fffffffLL) return MO_EINVAL;
  kp.total_tiles = (int)T;
  kp.kt = (kp.K + BK - 1) / BK;
  int sms = a.sms > 0 ? a.sms : 148;
  if (a.max_ctas > 0 && a.max_ctas < sms) sms = a.max_ctas;
  // few tiles: 32 x 32 ones (or strips, in place), perhaps in chunks of K
  if (int chunks = small_chunks(a, sms)) {
    const bool ak = a.transA, bk = !a.transB;
    kp.sk_chunk = (kp.kt + chunks - 1) / chunks;
    if (a.C == a.A) return launch_small<32, 128, 2, 4>(ak, bk, kp, stream);
    if (a.C == a.B) return launch_small<128, 32, 4, 2>(ak, bk, kp, stream);
    kp.partial = a.sk_partial;
    chunks = kp.sk_chunk > 0 ? (kp.kt + kp.sk_chunk - 1) / kp.sk_chunk : 1;
    const int rc = launch_small<32, 32, 2, 2>(ak, bk, kp, stream, chunks);
    if (rc || chunks == 1) return rc;
    small_reduce_kernel<<<(unsigned)(((int64_t)a.M * a.N + 255) / 256), 256, 0, stream>>>(kp, chunks);
    MO_CUDA_TRY(cudaGetLastError());
    return MO_OK;
  }
  // Schedule: whole tiles round-robin over the workers (two per CTA) of a persistent grid;
  // when a GEMM has only a few, unequal waves (e.g. 512 tiles on 2 x 148 workers), the last
  // one or two waves are split along K evenly over all workers (stream-K) and finished by
  // the worker holding each tile's last slab.
  const int slots = 2 * sms;
  kp.workers = (int)std::min<long long>(T, slots);
  kp.dp_tiles = (int)T;
  kp.sk_iters = 0;
  kp.sk_chunk = 1;
  kp.partial = a.sk_partial;
  kp.flags = a.sk_flags;
  kp.epoch = a.sk_epoch;
  const long long waves = T / slots, rem = T % slots;
  if (a.mode == kGemm && a.sk_partial && a.sk_flags && rem != 0 && waves < 4 && kp.kt >= 8) {
    const long long dp = (waves >= 1 ? waves - 1 : 0) * slots;
    kp.dp_tiles = (int)dp;
    kp.sk_iters = (int)((T - dp) * kp.kt);
    kp.workers = slots;
    kp.sk_chunk = (kp.sk_iters + slots - 1) / slots;
    if (kp.sk_chunk < 4) {
      // too little work for every worker: fewer workers with 4 slabs each when that still
      // uses more of them than whole tiles would (a few tiles with a long K, e.g. one
      // 128 x 128 block with K in the thousands), else data-parallel
      const long long g2 = kp.sk_iters / 4;
      if (kp.kt >= 32 && g2 > T) {
        kp.workers = (int)std::min<long long>(g2, slots);
        kp.sk_chunk = (kp.sk_iters + kp.workers - 1) / kp.workers;
      } else {
        kp.dp_tiles = (int)T;
        kp.sk_iters = 0;
        kp.sk_chunk = 1;
        kp.workers = (int)std::min<long long>(T, slots);
      }
    }
  }
  const int grid = std::min(kp.workers, sms);

  const bool ak = a.transA;   // op(A) stored K-major when A is transposed
  const bool bk = !a.transB;  // op(B) stored K-major when B is not transposed
  CUtensorMap ta, tb;
  const bool use_tma = !a.force_fallback && kp.K > 0 && gemm_tma_ok(a);
  if (use_tma) {
    bool okA = ak ? make_tmap(&ta, a.A, kp.K, a.M, a.lda, 16, (uint32_t)tbm)
                  : make_tmap(&ta, a.A, a.M, kp.K, a.lda, 16, 16);
    bool okB = bk ? make_tmap(&tb, a.B, kp.K, a.N, a.ldb, 16, (uint32_t)tbn)
                  : make_tmap(&tb, a.B, a.N, kp.K, a.ldb, 16, 16);
    if (okA && okB)
      return wide ? dispatch<true, true>(ak, bk, kp, ta, tb, grid, stream)
                    : dispatch<true, false>(ak, bk, kp, ta, tb, grid, stream);
  }
  memset(&ta, 0, sizeof(ta));
  memset(&tb, 0, sizeof(tb));
  return wide ? dispatch<false, true>(ak, bk, kp, ta, tb, grid, stream)
                : dispatch<false, false>(ak, bk, kp, ta, tb, grid, stream);
}

}  // namespace mo
