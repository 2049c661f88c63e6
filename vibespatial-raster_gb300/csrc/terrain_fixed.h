// Terrain derivatives from integer elevations: curvature as a 96-bit
// fixed-point product, rounded once to float64.
//
// With the window's values n_i 2^u, profile curvature is
//   -100 (a / cx^2 + b / cy^2) 2^u,  a = n3 + n5 - 2 n4,  b = n1 + n7 - 2 n4.
// The factors 100 / cx^2 and 100 / cy^2 are kept as 60-bit integers in one
// unit (two limbs of 29 and 31 bits), so both products and their sum are exact
// and the only roundings are those of the factors (2^-60 of the larger) and of
// the result: the float64 formula rounds five times.  No FP64 operation: an
// SM starts two per clock.
//
// Plain C so that a host program can check it; CUDA includes it as device code.
#ifndef VSR_TERRAIN_FIXED_H
#define VSR_TERRAIN_FIXED_H

#include <stdint.h>

#if defined(__CUDACC__)
#define VSR_TF_FN __host__ __device__ __forceinline__
#else
#define VSR_TF_FN static inline
#endif

// Curvature factors: mh 2^31 + ml in units of 2^-s.
typedef struct {
  int32_t xh, xl, yh, yl;
  int32_t s;
  int32_t ok;  // 0: the factors are more than 2^14 apart (the smaller would lose bits)
} vsr_curv_k;

VSR_TF_FN int vsr_tf_clz32(uint32_t v) {  // v != 0
#if defined(__CUDA_ARCH__)
  return __clz((int)v);
#else
  return __builtin_clz(v);
#endif
}

// float64 bits of -(a kx + b ky) 2^u; |a|, |b| < 2^29 and a normal result.
VSR_TF_FN uint64_t vsr_curv_bits(int32_t a, int32_t b, const vsr_curv_k* k, int u) {
  const int64_t sl = (int64_t)a * k->xl + (int64_t)b * k->yl;  // < 2^61
  const int64_t sh = (int64_t)a * k->xh + (int64_t)b * k->yh;  // < 2^59
  int64_t vh = sh + (sl >> 31);
  uint32_t vl = (uint32_t)sl & 0x7fffffffu;  // value = vh 2^31 + vl
  const uint32_t neg = vh < 0;
  if (neg) {
    vh = ~vh + (vl == 0u);
    vl = (0u - vl) & 0x7fffffffu;
  }
  uint64_t m = (uint64_t)vh, r = (uint64_t)vl << 33;  // m.r, r the fraction bits left-aligned
  int e = 63 + 31;
  if (m == 0u) {
    m = r;
    r = 0u;
    e -= 64;
    if (m == 0u) return 0u;
  }
  if ((uint32_t)(m >> 32) == 0u) {
    m = (m << 32) | (r >> 32);
    r <<= 32;
    e -= 32;
  }
  const int z = vsr_tf_clz32((uint32_t)(m >> 32));
  m = z ? (m << z) | (r >> (64 - z)) : m;
  const uint64_t mant = (m >> 11) + ((m >> 10) & 1u);
  const uint32_t be = (uint32_t)(e - z + u - k->s + 1023 - 1);
  return ((uint64_t)((neg ^ 1u) << 31 | be << 20) << 32) + mant;
}

#endif
