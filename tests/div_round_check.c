// csrc/div_round.h over the quotients nearest to halfway cases: for every 24-bit
// W, the 24-bit N with N / W = M / 2^E + c / (W 2^E), M odd (halfway between two
// floats), |c| <= 6, the estimate of 1 / W off by -2 .. 2 ulps (in turn where
// the reciprocal is the rounded one all the same); then random pairs.  Prints the number of quotients, of those that are not the
// rounded one, of those of them where the reciprocal is the rounded one, and
// the largest error beyond half an ulp in units of 2^-24 ulp (rounded up).
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
static int pert;
static float off(float w);
#define VSR_DR_ESTIMATE(w) off(w)
#include "div_round.h"

static float off(float w) {
  float r = 1.0f / w;
  for (int i = 0; i < abs(pert); ++i) r = nextafterf(r, pert < 0 ? 0.0f : 1e30f);
  return r;
}

static long cases, differ, wrong;
static double worst;

static void check(float n, float w, float r, int rounded) {
  const float q = vsr_div_quot(n, w, r, n * r);
  ++cases;
  if (q == n / w) return;
  ++differ;
  wrong += rounded;
  const double exact = (double)n / w, ulp = ldexp(1.0, ilogb(exact) - 23);
  const double e = fabs(q - exact) / ulp - 0.5;
  if (e > worst) worst = e;
}

int main(void) {
  for (uint32_t m = 0; m < (1u << 23); ++m) {
    const uint32_t W = (1u << 23) | m;
    const int j = __builtin_ctz(W);
    if (j > 2) continue;  // c is a multiple of 2^j: the halfway cases of an odd divisor
    const uint32_t Wo = W >> j;
    const float w = (float)W, rn = (float)(1.0 / (double)w);
    for (int E = 24; E <= 25; ++E) {  // N >= W: quotients in [1, 2); N < W: in (1/2, 1)
      uint64_t inv = 1 % Wo;          // 2^-(E - j) mod Wo
      for (int i = 0; i < E - j; ++i) inv = (inv & 1) ? (inv + Wo) >> 1 : inv >> 1;
      for (int c = -6; c <= 6; ++c) {
        if (!c) continue;
        int64_t n0 = (int64_t)c * (int64_t)inv % Wo;
        if (n0 < 0) n0 += Wo;
        for (int64_t N = n0; N < (1 << 24); N += Wo) {
          if (N < (1 << 23) || (E == 25) != (N < W)) continue;
          if (!((((N << E) - ((int64_t)c << j)) / W) & 1)) continue;  // not a halfway case
          for (pert = -2; pert <= 2; ++pert) {
            const float r = vsr_div_recip(w);
            if (r != rn || (m + c + pert) % 5 == 0) check((float)N, w, r, r == rn);
          }
        }
      }
    }
  }
  uint64_t s = 88172645463325252ull;
  for (long i = 0; i < 20000000; ++i) {
    s ^= s << 13;
    s ^= s >> 7;
    s ^= s << 17;
    const float n = ldexpf((float)(s & 0xffffff), (int)((s >> 48) % 60) - 30);
    const float w = ldexpf((float)(0x800000 | ((s >> 24) & 0x7fffff)), (int)((s >> 56) % 40) - 40);
    if (n == 0.0f) continue;
    pert = (int)(i % 5) - 2;
    const float r = vsr_div_recip(w);
    check(n, w, r, r == (float)(1.0 / (double)w));
  }
  printf("%ld %ld %ld %ld\n", cases, differ, wrong, (long)ceil(worst * 16777216.0));
  return 0;
}
