// sum / n as a float64 from the rounded reciprocal of n: q0 = s r and Markstein's
// residual correction (div_round.h).  Equal to the division for every window
// count and sum of 8/16-bit values that the register kernel forms (n <= 81),
// which the host test goes through one by one.
//
// Three operations on the narrow FP64 pipe, where a division takes about nine:
// uint16 3 x 3 mean with float64 output at 7760^2 1433 -> 499 us.
//
// Plain C so that the host test compiles it with gcc; CUDA includes it as
// device functions.
#ifndef VSR_MEAN_ROUND_H
#define VSR_MEAN_ROUND_H

#if defined(__CUDACC__)
#define VSR_MR_FN __device__ __forceinline__
#else
#include <math.h>
#define VSR_MR_FN static inline
#endif

// s / n; nn = -n, r = 1 / n rounded to nearest
VSR_MR_FN double vsr_mean_quot(double s, double nn, double r) {
  const double q0 = s * r;
  return fma(fma(nn, q0, s), r, q0);
}

#endif
