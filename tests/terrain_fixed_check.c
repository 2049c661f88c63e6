// csrc/terrain_fixed.h in 128-bit floating point: curvature factors and the
// product -(a kx + b ky) 2^u, over random, cancelling, short and zero sums,
// factors alike and up to 2^14 apart.  Prints the number of products, of those
// beyond the bound (0.5 ulp, half a unit of 2^-s per factor, one for the ones'
// complement), of cell sizes refused, and of refusals that are not due; then
// of 64-bit integers scaled and of those that are not the rounded value.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "terrain_fixed.h"

typedef _Float128 quad;
static uint64_t s = 88172645463325252ull;
static uint64_t rnd(void) {
  s ^= s << 13;
  s ^= s >> 7;
  s ^= s << 17;
  return s;
}
static double unit(void) { return (double)(rnd() >> 11) * 0x1p-53; }
static quad qabs(quad v) { return v < 0 ? -v : v; }
static quad pow2(int e) {
  quad v = 1;
  for (; e > 0; --e) v *= 2;
  for (; e < 0; ++e) v /= 2;
  return v;
}

int main(int argc, char** argv) {
  const long count = argc > 1 ? atol(argv[1]) : 1000000;
  long cases = 0, bad = 0, refused = 0, undue = 0;
  for (long i = 0; i < count; ++i) {
    const double cx = exp2(20.0 * unit() - 10.0), ratio = exp2(16.0 * unit() - 8.0);
    const double cy = i % 5 == 0 ? cx : cx * ratio, cx2 = cx * cx, cy2 = cy * cy;
    const vsr_curv_k k = vsr_curv_factors(cx2, cy2);
    if (!k.ok) {
      ++refused;
      undue += fabs(log2(cx2 / cy2)) < 13.999;
      continue;
    }
    for (int j = 0; j < 8; ++j) {
      const int len = 1 + (int)(rnd() % 29);
      int32_t a = (int32_t)(rnd() & ((1u << len) - 1)), b = (int32_t)(rnd() & ((1u << len) - 1));
      if (j & 1) a = -a;
      if (j & 2) b = -b;
      if (j == 4) b = -a;                                  // cancels where the factors are alike
      if (j == 5) {                                        // nearly cancels
        const double t = -(double)a * cy2 / cx2;
        if (fabs(t) >= 0x1p29) continue;
        b = (int32_t)t;
      }
      if (j == 6 && (rnd() & 1)) a = 0;
      if (j == 7 && (rnd() & 1)) b = 0;
      const int u = (int)(rnd() % 129) - 88;
      const uint64_t bits = vsr_curv_bits(a, b, &k, u);
      double got;
      memcpy(&got, &bits, 8);
      const quad ref = -100 * ((quad)a / cx2 + (quad)b / cy2) * pow2(u);
      const double ulp = got == 0.0 ? 0.0 : ldexp(1.0, ilogb(got) - 52);
      const quad bound = (quad)ulp / 2 + ((quad)(abs(a) + (double)abs(b)) / 2 + 1) * pow2(u - k.s);
      bad += qabs((quad)got - ref) > bound;
      ++cases;
    }
  }
  printf("%ld %ld %ld %ld ", cases, bad, refused, undue);
  cases = bad = 0;
  for (long i = 0; i < 10 * count; ++i) {
    int64_t v = (int64_t)rnd() >> (1 + i % 63);
    if (i % 7 == 0) v = (int64_t)((rnd() >> 11) | 1) << (i % 9);  // 53 bits and fewer, halfway cases
    if (i % 11 == 0) v &= ~((1ll << (i % 40)) - 1);
    if (i % 13 == 0) v = 0;
    const int e = (int)(i % 130) - 89;
    const uint64_t bits = vsr_wide_bits(v, e);
    double got;
    memcpy(&got, &bits, 8);
    bad += got != ldexp((double)v, e);
    ++cases;
  }
  printf("%ld %ld\n", cases, bad);
  return 0;
}
