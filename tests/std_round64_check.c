// Compares csrc/std_round64.h with a __float128 reference: the error of
// sqrt(N) / n in ulps of the float64 result, over random N of every length,
// edge values and perfect squares, all window counts.  Prints the number of
// cases, the largest error in thousandths of an ulp and the exact squares
// that did not come out exactly.
#include <stdio.h>
#include <stdlib.h>
#include <math.h>
static float pert = 1.0f;  // the device's rsqrtf is within 2 ulps: the error must not depend on it
#define VSR_S64_RSQRT(f) (1.0f / sqrtf(f) * pert)
#include "std_round64.h"

static uint64_t s = 88172645463325252ull;
static uint64_t rnd(void) {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}
// sqrt of a __float128 by Newton steps from the long double root
static __float128 qsqrt(__float128 v) {
  __float128 x = sqrtl((long double)v);
  for (int i = 0; i < 3; ++i) x = (x + v / x) / 2;
  return x;
}

int main(int argc, char** argv) {
  const long count = argc > 1 ? atol(argv[1]) : 1000000;
  double worst = 0;
  long cases = 0, bad = 0;
  for (long i = 0; i < count; ++i) {
    uint64_t nh = 0, nl = rnd() >> (rnd() % 64);
    const int kind = i % 8;
    pert = 1.0f + (float)((int)(rnd() % 9) - 4) * 1.1920929e-7f;
    if (kind == 1) nh = rnd() >> (rnd() % 64);
    if (kind == 2) nl = ~0ull >> (rnd() % 64);
    if (kind == 3) nl = 1ull << (rnd() % 64);
    if (kind == 4) nh = ~0ull >> (rnd() % 64), nl = ~0ull;
    if (kind == 5) nh = 1ull << (rnd() % 64), nl = 0;
    const uint32_t n = 1 + rnd() % 225;
    uint64_t root = 0;
    if (kind >= 6) {  // (n r)^2: the exact result is r
      root = rnd() >> (33 + rnd() % 31);
      if (!root) root = 1;
      const unsigned __int128 p = (unsigned __int128)(root * n) * (root * n);
      nh = (uint64_t)(p >> 64);
      nl = (uint64_t)p;
    }
    if (!(nh | nl)) continue;
    int L = 0;
    while ((n >> L) > 1u) ++L;
    const int u = (int)(rnd() % 200) - 100;
    const uint64_t b = vsr_s64_std128(nh, nl, u, vsr_s64_recip(n), L);
    double got;
    memcpy(&got, &b, 8);
    const __float128 N = (__float128)nh * 18446744073709551616.0Q + (__float128)nl;
    const __float128 ref = qsqrt(N) / n;
    const __float128 g = (__float128)ldexp(got, -u);
    const double ulp = ldexp(1.0, ilogb((double)ref) - 52);
    __float128 err = (g - ref) / ulp;
    if (err < 0) err = -err;
    if ((double)err > worst) worst = (double)err;
    if (kind >= 6 && g != (__float128)root) ++bad;
    ++cases;
  }
  printf("%ld %ld %ld\n", cases, (long)(worst * 1000), bad);
  return 0;
}
