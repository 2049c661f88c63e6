// sqrt(N) / n as a float64 with integer arithmetic, for the focal standard
// deviation (N = n sum x^2 - (sum x)^2 formed exactly, std = sqrt(N) / n).
//
// The FP64 pipe of a GB300's SM is narrow, and a float64 square root and a
// division take about 25 operations on it.  Here the root is a 64-bit
// fixed-point number: a float estimate, two Newton corrections whose
// residuals are exact (mod 2^64) integer products, then one 64 x 64-bit
// product with the reciprocal of n.  The error before the final rounding is
// below 2^-58 of the value, so the result lies within 0.52 ulp; sqrt() and a
// division, each rounded, reach 1 ulp.
//
// Plain C so that the host test compiles it with gcc and checks it against a
// wider type; CUDA includes it as device functions.
#ifndef VSR_STD_ROUND64_H
#define VSR_STD_ROUND64_H

#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define VSR_S64_FN __device__ __forceinline__
#define VSR_S64_MULHI32(a, b) __umulhi((a), (b))
#define VSR_S64_CLZ(a) __clz((int)(a))
#define VSR_S64_RSQRT(f) vsr_s64_rsqrt(f)
#define VSR_S64_F2U(f) __float2uint_rz(f) /* saturates at 2^32 - 1 */
#define VSR_S64_F2I(f) __float2int_rn(f)
#else
#include <math.h>
#define VSR_S64_FN static inline
#define VSR_S64_MULHI32(a, b) ((uint32_t)(((uint64_t)(a) * (b)) >> 32))
#define VSR_S64_CLZ(a) __builtin_clz(a)
#if !defined(VSR_S64_RSQRT)
#define VSR_S64_RSQRT(f) (1.0f / sqrtf(f))
#endif
#define VSR_S64_F2U(f) ((f) >= 4294967296.0f ? 0xffffffffu : (uint32_t)(f))
#define VSR_S64_F2I(f) ((int32_t)lrintf(f))
#endif

#if defined(__CUDACC__)
__device__ __forceinline__ float vsr_s64_rsqrt(float f) {  // f in [2^30, 2^32]: no subnormals to care for
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return r;
}
#endif

// The reciprocal of n >= 1 as a 64-bit fraction: ceil(2^(63 + L) / n) with
// L = floor(log2 n), in (2^62, 2^63].
#if defined(__cplusplus)
constexpr
#else
static inline
#endif
    uint64_t
    vsr_s64_recip(uint32_t n) {
  int L = 0;
  while ((n >> L) > 1u) ++L;
  const uint64_t one = (uint64_t)1 << 63;
  const uint64_t q = one / n, r = one % n;
  const uint64_t t = r << L;  // r < n < 2^32
  return (q << L) + t / n + (t % n ? 1 : 0);
}

// sqrt(M 2^(2 h)) / n as float64 bits: M in [2^62, 2^64), recip =
// vsr_s64_recip(n) and L = floor(log2 n); the result must be a normal number.
VSR_S64_FN uint64_t vsr_s64_bits(uint64_t M, int h, uint64_t recip, int L) {
  const float f = (float)(uint32_t)(M >> 32);  // 2^-32 M to 24 bits
  const float y = VSR_S64_RSQRT(f);            // 2^16 / sqrt(M)
  const uint32_t x0 = VSR_S64_F2U(f * y * 65536.0f);  // sqrt(M) within 2^11
  // e0 = M - x0^2, |e0| < 2^45: sqrt(M) = x0 + e0 / (2 sqrt M) - ..., to 2^-9
  const int64_t e0 = (int64_t)(M - (uint64_t)x0 * x0);
  const float d0 = (float)(int32_t)(e0 >> 14) * (y * 8192.0f);  // 2^16 e0 / (2 sqrt M)
  const uint64_t x1 = ((uint64_t)x0 << 16) + (uint64_t)(int64_t)VSR_S64_F2I(d0);  // units of 2^-16
  // e1 = 2^32 M - x1^2 (mod 2^64; |e1| < 2^57), the second correction to 2^-30
  const uint32_t xl = (uint32_t)x1, xh = (uint32_t)(x1 >> 32);
  const uint64_t sq = (uint64_t)xl * xl + ((uint64_t)(xl * xh) << 33);
  const int64_t e1 = (int64_t)(((uint64_t)(uint32_t)M << 32) - sq);
  const float d1 = (float)(int32_t)(e1 >> 26) * (y * 64.0f);  // 2^13 e1 / (2 x1), 1 / x1 = 2^-32 y
  const uint64_t x2 = (x1 << 13) + (uint64_t)(int64_t)VSR_S64_F2I(d1);  // units of 2^-29, in [2^60, 2^61]
  // x2 / n: hi(4 x2, recip) 2^(64 - 2 - 63 - L); the product of the low halves is left out (2^-60)
  const uint64_t t = x2 << 2;
  const uint32_t th = (uint32_t)(t >> 32), rh = (uint32_t)(recip >> 32);
  const uint64_t q = (uint64_t)th * rh + VSR_S64_MULHI32(th, (uint32_t)recip) + VSR_S64_MULHI32((uint32_t)t, rh);
  const int z = VSR_S64_CLZ((uint32_t)(q >> 32));
  const uint64_t qn = q << z, mant = (qn >> 11) + ((qn >> 10) & 1u);  // 53 bits (2^53 when it carries)
  // top bit of q: 2^(63 - z), times 2^(-1 - L) 2^-29 2^h; the leading bit adds 1 to the exponent
  const uint32_t e = (uint32_t)(1023 + 63 - z - 1 - L - 29 + h - 1);
  return ((uint64_t)(e << 20) << 32) + mant;
}

// N 2^(2 u) of a 64-bit N > 0.
VSR_S64_FN uint64_t vsr_s64_std(uint64_t N, int u, uint64_t recip, int L) {
  const int w = (uint32_t)(N >> 32) == 0u;  // shift a low word up first
  const uint64_t v = w ? N << 32 : N;
  const int z = VSR_S64_CLZ((uint32_t)(v >> 32)) & ~1;
  return vsr_s64_bits(v << z, u - (z >> 1) - 16 * w, recip, L);
}

// N 2^(2 u) of a 128-bit N = nh 2^64 + nl > 0.
VSR_S64_FN uint64_t vsr_s64_std128(uint64_t nh, uint64_t nl, int u, uint64_t recip, int L) {
  if (nh == 0) return vsr_s64_std(nl, u, recip, L);
  const int w = (uint32_t)(nh >> 32) == 0u;
  const uint64_t v = w ? (nh << 32) | (nl >> 32) : nh, r = w ? nl << 32 : nl;
  const int z = VSR_S64_CLZ((uint32_t)(v >> 32)) & ~1;  // 0 .. 30
  const uint64_t M = z ? (v << z) | (r >> (64 - z)) : v;
  return vsr_s64_bits(M, u + 32 - (z >> 1) - 16 * w, recip, L);
}

#endif
