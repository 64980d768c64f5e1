// cos2pi_box against cos2pi (pps_device.cuh), both compiled for the host: argv
// first, last, step of the bit patterns; prints the number of mismatches.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>

#define __device__
#define __forceinline__ inline
static float __uint_as_float(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static uint32_t __float_as_uint(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
#include "cosines.inc"  // the two functions, cut out of the header by the test

int main(int argc, char** argv) {
  (void)argc;
  const uint64_t first = strtoull(argv[1], nullptr, 0), last = strtoull(argv[2], nullptr, 0), step = strtoull(argv[3], nullptr, 0);
  unsigned long long bad = 0, count = 0;
  for (uint64_t u = first; u < last; u += step, ++count) {
    for (uint32_t sign : {0u, 0x80000000u}) {
      const float x = __uint_as_float((uint32_t)u | sign);
      if (__float_as_uint(cos2pi(x)) != __float_as_uint(cos2pi_box(x))) ++bad;
    }
  }
  printf("%llu %llu\n", count, bad);
  return 0;
}
