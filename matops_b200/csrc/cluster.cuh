// Exchange between the CTAs of one thread-block cluster through distributed shared memory
// (the LU and QR panels; the triangular solves map addresses with it too).
#pragma once
#include "common.cuh"

namespace mo {

__device__ __forceinline__ uint32_t cl_map(const void *p, int cta) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(cta));
  return a;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}

// PIECES x 16 bytes at `src` (this CTA's shared memory, 16-byte aligned) to the same place `dst`
// of every CTA of the cluster (at most 32 / LANES), the bytes counted on that CTA's barrier `bar`:
// lanes LANES c, ... of the calling warp write CTA c's copy.  (Plain remote stores need a
// cluster barrier with release semantics, which also waits for the panel's global stores: 1330
// cycles a column of the LU panel, 850 this way.)
template <int PIECES, int LANES = 2>
__device__ __forceinline__ void cl_send(void *dst, const void *src, uint64_t *bar, int lane,
                                        int nctas) {
  const int c = lane / LANES;
  if (c >= nctas) return;
  const uint32_t to = cl_map(dst, c), mb = cl_map(bar, c);
  const double2 *s = reinterpret_cast<const double2 *>(src);
#pragma unroll
  for (int i = 0; i < (PIECES + LANES - 1) / LANES; ++i) {
    const int p = LANES * i + lane % LANES;
    if (p < PIECES) {
      const double2 v = s[p];
      asm volatile(
          "st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(
              to + 16 * p),
          "d"(v.x), "d"(v.y), "r"(mb)
          : "memory");
    }
  }
}

}  // namespace mo
