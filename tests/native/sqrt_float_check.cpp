// Host check of sqrt_to_float (perigrain_gb300/csrc/pg_sqrt_float.cuh): its bits must equal those of
// (float)sqrt(x) for squares of the halfway points between floats and their neighbours, around the
// margins in which the FP64 root decides, at binade edges, at the ends of the range it serves, and for
// random operands of every exponent, zeros, subnormals, negatives, infinities and NaN. Prints "bad 0".
#include <cfloat>
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "pg_sqrt_float.cuh"

static uint64_t bad = 0, checked = 0;
static void check(double x) {
  ++checked;
  const float want = (float)std::sqrt(x), got = pg::sqrt_to_float(x);
  if (std::isnan(want) && std::isnan(got)) return;
  if (std::memcmp(&want, &got, 4) && bad++ < 10) std::printf("x %a: want %a got %a\n", x, want, got);
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 500000;
  std::mt19937_64 rng(argc > 2 ? std::strtoull(argv[2], nullptr, 10) : 1);
  auto around = [](double x, int k) {  // x and its k neighbours on each side
    double lo = x, hi = x;
    check(x);
    for (int i = 0; i < k; ++i) {
      lo = std::nextafter(lo, 0.0);
      hi = std::nextafter(hi, INFINITY);
      check(lo);
      check(hi);
    }
  };
  // roots r + (1/2 + e) ulp(r): e around 0 and around the margins
  const double es[] = {0, 1e-9, -1e-9, 1e-7, -1e-7, 1.9e-6, 2.0e-6, 2.1e-6, -1.9e-6, -2.0e-6, -2.1e-6, 3.8e-6, -3.8e-6,
                       1e-4, -1e-4, 0.25, -0.25, 0.499, -0.499};
  for (long k = 0; k < n; ++k) {
    const uint32_t frac = k % 5 == 0 ? (uint32_t)(rng() % 4) : k % 5 == 1 ? 0x7fffffu - (uint32_t)(rng() % 4)
                                                                       : (uint32_t)(rng() & 0x7fffffu);
    const uint32_t rb = ((uint32_t)(70 + rng() % 115) << 23) | frac;
    float r, u;
    std::memcpy(&r, &rb, 4);
    const uint32_t ub = rb + 1;
    std::memcpy(&u, &ub, 4);
    for (double e : es) {
      const double root = (double)r + (0.5 + e) * ((double)u - (double)r);
      around(root * root, 2);
    }
    around((double)r * (double)r, 2);
  }
  for (double x : {1e-30, 1e30, 1e-45, 1e-38, 1e38, 3.4e38, 3.5e38, 1e300, 1e-300, 0.0, -0.0, -1.0, 4.9e-324, DBL_MAX,
                   (double)INFINITY, (double)-INFINITY, (double)NAN, 1.0, 2.0, 4.0, 0.25})
    around(x, 3);
  for (long k = 0; k < n; ++k) {
    const uint64_t b = rng();
    double x;
    std::memcpy(&x, &b, 8);
    check(x);
    check(std::ldexp(1.0 + (double)(b >> 12) * 0x1p-52, (int)(b % 200) - 100));
  }
  std::printf("checked %" PRIu64 " bad %" PRIu64 "\n", checked, bad);
}
