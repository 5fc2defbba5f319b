// Host build of the sanity check's comparison |a| > b (spin-tracking_gb300/csrc/
// st_softfp.cuh) for tests, against the host's own: every pair of a list of special
// values, limits below zero, infinite and NaN among them.  Prints the number that differ.
#include <cmath>
#include <cstdint>
#include <cstdio>

#define __device__
#define __constant__ const
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#include "st_softfp.cuh"

int main() {
  const double v[] = {0.0, -0.0, 0.2, -0.2, 0.05, -0.05, 0x1p-1074, -0x1p-1074, 0x1.fffffffffffffp1023, -0x1.fffffffffffffp1023,
                      INFINITY, -INFINITY, NAN, -NAN};
  long wrong = 0;
  for (double a : v)
    for (double b : v) wrong += st::sfp::abs_gt(a, b) != (std::fabs(a) > b);
  std::printf("%ld\n", wrong);
  return 0;
}
