// Host build of the integer division, square root, draws and comparisons
// (spin-tracking_gb300/csrc/st_softfp.cuh) for tests, against the host's own
// correctly rounded operations: n random operands of each kind (uniform bits,
// near-equal significands, trajectory-sized values) and every pair of a list of special
// values.  The seeds are spoiled to the accuracy the device's instructions give.
// Prints the number of differing results per function.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#define __device__
#define __constant__ const
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#include "st_softfp.cuh"

using namespace st::sfp;

static uint64_t g_state;
static uint64_t bits() {
  g_state ^= g_state >> 12;
  g_state ^= g_state << 25;
  g_state ^= g_state >> 27;
  return g_state * 0x2545F4914F6CDD1Dull;
}
static double uniform() { return (double)(bits() >> 11) * 0x1p-53; }
static bool same(double a, double b) { return (std::isnan(a) && std::isnan(b)) || f64_bits(a) == f64_bits(b); }

int main(int argc, char** argv) {
  const long n = std::atol(argv[1]);
  g_state = std::strtoull(argv[2], nullptr, 10) * 2 + 1;
  long div = 0, root = 0, unit = 0, cmp = 0;
  auto one = [&](double a, double b) {
    volatile double va = a, vb = b;
    div += !same(div_rn(a, b), va / vb);
    root += !same(sqrt_rn(a), std::sqrt(va));
    div += !same(div_g(a), va / -9.81);
    cmp += negative(a) != (a < 0.0);
    cmp += is_finite(a) != std::isfinite(a);
    cmp += lt(a, b) != (a < b);
    cmp += le(a, b) != (a <= b);
    cmp += eq(a, b) != (a == b);
    cmp += is_nan(a) != std::isnan(a);
    cmp += is_inf(a) != std::isinf(a);
    cmp += abs_gt(a, std::fabs(b)) != (std::fabs(a) > std::fabs(b)) && !std::isnan(b);
  };
  const double special[] = {0.0, -0.0, 1.0, -1.0, 2.0, 3.0, 0x1p-1022, 0x1p-1074, 0x1.fffffffffffffp1023, INFINITY,
                            -INFINITY, NAN, 0x1.fffffffffffffp0, 0x1.0000000000001p0, 0x1p-1000, 0x1p1000, 4.0, 0x1.fffffffffffffp-1};
  for (double a : special)
    for (double b : special) one(a, b);
  for (long i = 0; i < n; ++i) {
    one(bits_f64(bits()), bits_f64(bits()));
    const uint64_t m = bits() & kFrac;
    const double a = bits_f64(m | 0x3ff0000000000000ull);
    one(a, bits_f64(((m + (bits() % 5) - 2) & kFrac) | 0x3ff0000000000000ull));  // quotients next to 1
    one(bits_f64((m & ~0x3ffull) | 0x3ff0000000000000ull), a);                   // short operands
    one((uniform() - 0.5) * 0.1, (uniform() - 0.5) * 8.0);
    one(uniform() * 20.0, -9.81);
    const double s = bits_f64((bits() & kFrac & ~0x7ffffffull) | 0x3ff0000000000000ull);
    one(s * s, s);                                                                // exact squares and quotients
    one(std::nextafter(s * s, 0.0), s);
    one(std::nextafter(s * s, 8.0), s);
    const uint64_t u = bits() >> (bits() & 63);
    unit += !same(unit_53(u), (double)(u >> 11) * 0x1p-53);
    volatile double two = (double)(u >> 11) * 0x1p-53 * 2.0;
    unit += !same(signed_unit_53(u), two + -1.0);
  }
  std::printf("div %ld sqrt %ld unit %ld compare %ld\n", div, root, unit, cmp);
  return 0;
}
