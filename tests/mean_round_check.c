// csrc/mean_round.h against the compiler's division: every count up to 81 and
// every sum of that many 16-bit values, signed and unsigned.  Prints the number
// of quotients and of those that differ.
#include <stdint.h>
#include <stdio.h>
#include "mean_round.h"

int main(void) {
  long cases = 0, bad = 0;
  for (int n = 1; n <= 81; ++n) {
    const double nn = -(double)n, r = 1.0 / n;
    for (int32_t s = -32768 * n; s <= 65535 * n; ++s) {
      const double v = s;
      bad += vsr_mean_quot(v, nn, r) != v / n;
      ++cases;
    }
  }
  printf("%ld %ld\n", cases, bad);
  return 0;
}
