// Terrain derivatives from integer elevations: curvature as a 96-bit
// fixed-point product, rounded once to float64.
//
// With the window's values n_i 2^u, profile curvature is
//   -100 (a / cx^2 + b / cy^2) 2^u,  a = n3 + n5 - 2 n4,  b = n1 + n7 - 2 n4.
// The factors 100 / cx^2 and 100 / cy^2 are kept as 60-bit integers in one
// unit (two limbs of 29 and 31 bits), so both products and their sum are exact
// and the only roundings are those of the factors (2^-60 of the larger) and of
// the result: the float64 formula rounds five times.  No FP64 operation, as
// that pipe is narrow.
//
// Plain C so that the host test compiles it with gcc; CUDA includes it as device
// code (the factors as host code).
#ifndef VSR_TERRAIN_FIXED_H
#define VSR_TERRAIN_FIXED_H

#include <math.h>
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
  int32_t ok;  // 0: no integer form
} vsr_curv_k;

// 100 / cx2 and 100 / cy2 to 106 bits as integers in one unit of 2^-s, the
// larger in [2^59, 2^60].  No integer form where the factors are more than 2^14
// apart (the smaller would lose bits) or near the ends of the exponent range
// (the scaled results would not be normal).
static inline vsr_curv_k vsr_curv_factors(double cx2, double cy2) {
  vsr_curv_k k = {0, 0, 0, 0, 0, 0};
  const double qx = 100.0 / cx2, qy = 100.0 / cy2;
  const double rx = fma(-qx, cx2, 100.0) / cx2, ry = fma(-qy, cy2, 100.0) / cy2;
  const double most = qx > qy ? qx : qy, least = qx > qy ? qy : qx;
  if (!(least > 0.0) || !(most < 1.0e300)) return k;
  int e = 0;
  frexp(most, &e);
  k.s = 60 - e;
  k.ok = least >= ldexp(most, -14) && e > -400 && e < 400;
  if (!k.ok) return k;
  const double tx = ldexp(qx, k.s), ty = ldexp(qy, k.s);  // (the smaller may have a fraction)
  const int64_t mx = (int64_t)tx + (int64_t)llrint(tx - floor(tx) + ldexp(rx, k.s));
  const int64_t my = (int64_t)ty + (int64_t)llrint(ty - floor(ty) + ldexp(ry, k.s));
  k.xh = (int32_t)(mx >> 31);
  k.xl = (int32_t)(mx & 0x7fffffff);
  k.yh = (int32_t)(my >> 31);
  k.yl = (int32_t)(my & 0x7fffffff);
  return k;
}

VSR_TF_FN int vsr_tf_clz32(uint32_t v) {  // v != 0
#if defined(__CUDA_ARCH__)
  return __clz((int)v);
#else
  return __builtin_clz(v);
#endif
}

VSR_TF_FN uint32_t vsr_tf_shl(uint32_t hi, uint32_t lo, int z) {  // high word of (hi, lo) << z, 0 <= z < 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, z);
#else
  return z ? (hi << z) | (lo >> (32 - z)) : hi;
#endif
}

// float64 bits of s 2^e, rounded to nearest (to even); |s| < 2^63 and a normal
// result.  (A conversion would run on the narrow FP64 pipe.)
VSR_TF_FN uint64_t vsr_wide_bits(int64_t s, int e) {
  const uint64_t neg = (uint64_t)(s >> 63), m = ((uint64_t)s ^ neg) - neg;
  const int w = (m >> 32) == 0u;  // a low word only
  const uint32_t x0 = w ? (uint32_t)m : (uint32_t)(m >> 32), x1 = w ? 0u : (uint32_t)m;
  const int z = vsr_tf_clz32(x0 | 1u);
  const uint32_t f0 = vsr_tf_shl(x0, x1, z), f1 = x1 << z;  // the leading bit on top
  const uint64_t mant = (uint64_t)(f0 >> 11) << 32 | vsr_tf_shl(f0, f1, 21);  // 53 bits
  const uint64_t r = mant + (((f1 & 0x7ffu) + 0x3ffu + ((uint32_t)mant & 1u)) >> 11);  // (2^53 when it carries)
  const uint32_t ex = (uint32_t)(1023 + 63 - 1 - z - (w ? 32 : 0) + e);
  return x0 ? r + ((uint64_t)((ex << 20) | ((uint32_t)neg & 0x80000000u)) << 32) : 0u;
}

// float64 bits of -(a kx + b ky) 2^u; |a|, |b| < 2^29 and a normal result.
// Without branches: lanes differ in sign and length.  A negative value is
// taken as its ones' complement, one unit of 2^-s (2^-59 of a factor) off.
VSR_TF_FN uint64_t vsr_curv_bits(int32_t a, int32_t b, const vsr_curv_k* k, int u) {
  const int64_t sl = (int64_t)a * k->xl + (int64_t)b * k->yl;                // < 2^61
  const int64_t vh = (int64_t)a * k->xh + (int64_t)b * k->yh + (sl >> 31);   // < 2^60
  const uint32_t neg = (uint32_t)(int32_t)(vh >> 63);  // all ones when negative
  // |value| = (x0, x1, x2 / 2^32) 2^31
  uint32_t x0 = (uint32_t)((uint64_t)vh >> 32) ^ neg, x1 = (uint32_t)vh ^ neg, x2 = ((uint32_t)sl ^ neg) << 1;
  int e = 63 + 31 + 1023 - 1 + u - k->s;
  const int s1 = x0 == 0u;
  x0 = s1 ? x1 : x0;
  x1 = s1 ? x2 : x1;
  x2 = s1 ? 0u : x2;
  const int s2 = x0 == 0u;
  x0 = s2 ? x1 : x0;
  x1 = s2 ? x2 : x1;
  e -= (s1 ? 32 : 0) + (s2 ? 32 : 0);
  const int z = vsr_tf_clz32(x0 | 1u);
  const uint32_t f0 = vsr_tf_shl(x0, x1, z), f1 = vsr_tf_shl(x1, s2 ? 0u : x2, z);
  const uint64_t m = ((uint64_t)(f0 >> 11) << 32 | vsr_tf_shl(f0, f1, 21)) + ((f1 >> 10) & 1u);
  const uint64_t r = m + ((uint64_t)((uint32_t)(e - z) << 20 | (~neg & 0x80000000u)) << 32);
  return x0 ? r : 0u;
}

#endif
