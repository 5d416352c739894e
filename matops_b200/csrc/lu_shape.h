// How many CTAs, and rows per thread, the LU panel's thread-block cluster takes (host code; no
// CUDA headers, so that a host compiler can check the rule).
#pragma once

namespace mo {

constexpr int kClThreads = 256;   // threads of a CTA of the cluster
constexpr int kClPortable = 8;    // CTAs that every device can place as one cluster
constexpr int kClMaxCtas = 16;    // CTAs that a whole B200 can place; a part of one may not
constexpr int kClMaxRpt = 4;      // rows per thread

// rows that a panel may have in one cluster of at most max_ctas CTAs
inline int cl_max_rows(int max_ctas) { return kClThreads * max_ctas * kClMaxRpt; }

// The cluster for m <= cl_max_rows(max_ctas) rows, max_ctas 8 or 16: one row per thread while
// max_ctas suffice (a second and a fourth row per thread cost 50 and 130 us a panel at 1001
// rows, more CTAs 1 to 10 us; the step from one CTA to a cluster costs 65 us, a row more per
// thread the same).
inline int cl_shape(int m, int max_ctas, int *rpt) {
  int c = 1, r = 1;
  while (c * kClThreads * r < m) {
    if (c < max_ctas) c *= 2;
    else r *= 2;
  }
  *rpt = r;
  return c;
}

}  // namespace mo
