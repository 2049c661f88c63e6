// Terrain derivatives of one pixel (terrain.cu, terrain_strip.cu): the formulas,
// the integer forms and the double-float arithmetic.
//
// GB300's FP64 rate is a small fraction of its FP32 rate, so 8/16-bit and
// float32 elevations are taken as integers in one unit per window (32 or 64
// bits): TRI and TPI are exact and rounded once.  Windows that no unit holds are
// evaluated in double-float FP32: every neighbour difference is formed
// error-free (TwoDiff), sums are compensated (TwoSum) and products use FMA, so
// results carry ~44 significant bits before the single conversion to the
// output type.  A formula whose inputs include NaN or +-inf takes the plain
// float form (the special values propagate as in the reference).
#pragma once

#include <cmath>
#include <type_traits>

#include "df_round.h"
#include "terrain_exact.h"
#include "terrain_fixed.h"
#include "vsr_internal.cuh"

namespace vsr {

struct DerivParams {
  int64_t H, W, pitch, out_pitch;
  int64_t band_stride, out_band_stride;  // band blockIdx.z of a band-first stack
  int nd_kind;      // resolved VSR_NODATA_*
  double nd_in;     // nodata value of the raster (element value, as double)
  double nd_out;    // value written to nodata / border pixels
  double cx2, cy2;                  // cx^2, cy^2 (FP64 path: the reference divides)
  float icx2_hi, icx2_lo, icy2_hi, icy2_lo;  // the same as float pairs
  void *tri, *tpi, *curv;
  int out_dtype;
  double kx, ky;    // the curvature factors 100 / cx^2, 100 / cy^2
  vsr_curv_k ck;    // the same as integers (terrain_fixed.h)
};

// Binades of the values of a 32-bit unit: |n| < 2^27, or 2^28 where no value is
// negative; differences stay below 2^28, the sums of eight below 2^31.
constexpr uint32_t kTdSpan = 4, kTdSpanPos = 5;
// ... of a 64-bit unit: |n| < 2^58, the sums of eight differences below 2^62.
constexpr uint32_t kTdSpanWide = 35;
// Exponents of values whose scaled results are normal float64 numbers.
constexpr uint32_t kTdExpMin = 64u, kTdExpMax = 190u;

// ---- double-float helpers: value = hi + lo with |lo| <= ulp(hi)/2
struct DF {
  float hi, lo;
};
__device__ __forceinline__ DF two_diff_df(float a, float b) {  // a - b exactly
  const float s = __fsub_rn(a, b);
  const float z = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), -__fadd_rn(b, z))};
}
__device__ __forceinline__ DF two_sum_df(float a, float b) {  // a + b exactly
  const float s = __fadd_rn(a, b);
  const float z = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z))};
}
__device__ __forceinline__ DF fast_two_sum_df(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ DF df_add(DF a, DF b) {
  const DF s = two_sum_df(a.hi, b.hi);
  return fast_two_sum_df(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ DF df_mul(DF a, DF b) {
  const float p = __fmul_rn(a.hi, b.hi);
  float e = __fmaf_rn(a.hi, b.hi, -p);
  e = __fmaf_rn(a.hi, b.lo, e);
  e = __fmaf_rn(a.lo, b.hi, e);
  return fast_two_sum_df(p, e);
}
__device__ __forceinline__ DF df_mul_f(DF a, float c) {
  const float p = __fmul_rn(a.hi, c);
  const float e = __fmaf_rn(a.lo, c, __fmaf_rn(a.hi, c, -p));
  return fast_two_sum_df(p, e);
}
__device__ __forceinline__ DF df_neg(DF a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ DF df_abs(DF a) { return a.hi < 0.0f ? df_neg(a) : a; }
__device__ __forceinline__ DF df_scale(DF a, float p2) { return {a.hi * p2, a.lo * p2}; }  // p2 a power of two

template <typename T>
__device__ __forceinline__ void store_out(void* base, int out_dtype, int64_t i, T v) {
  if (out_dtype == VSR_F64) static_cast<double*>(base)[i] = static_cast<double>(v);
  else static_cast<float*>(base)[i] = static_cast<float>(v);
}
// hi + lo as a double: both floats widened with integer operations
// (vsr_f32_widen), one FP64 add; subnormal or non-finite parts convert in FP64.
__device__ __forceinline__ double df_to_double(float hi, float lo) {
  const uint32_t hb = __float_as_uint(hi), lb = __float_as_uint(lo);
  if (!(vsr_f32_widen_ok(hb) && vsr_f32_widen_ok(lb))) return static_cast<double>(hi) + static_cast<double>(lo);
  uint32_t hh, hl, lh, ll;
  vsr_f32_widen(hb, &hh, &hl);
  vsr_f32_widen(lb, &lh, &ll);
  return __hiloint2double(static_cast<int>(hh), static_cast<int>(hl)) +
         __hiloint2double(static_cast<int>(lh), static_cast<int>(ll));
}

// s 2^e (exact, |s| < 2^31) as the output: float64 bits written directly,
// float32 rounded once.
__device__ __forceinline__ void store_int_scaled(void* base, int out_dtype, int64_t i, int32_t s, int e) {
  const double v = __longlong_as_double(static_cast<long long>(vsr_int_scaled_bits(s, e)));
  if (out_dtype == VSR_F64) static_cast<double*>(base)[i] = v;
  else static_cast<float*>(base)[i] = static_cast<float>(v);
}

__device__ __forceinline__ void store_df(void* base, int out_dtype, int64_t i, DF v) {
  if (out_dtype == VSR_F64) static_cast<double*>(base)[i] = df_to_double(v.hi, v.lo);
  else static_cast<float*>(base)[i] = v.hi + v.lo;
}

// The reference's formulas in the operation order of algebra.py:3394-3412
// (double for FP64 DEMs; float where a window holds NaN or +-inf, whose
// special values propagate the same way in either precision).
template <typename C>
__device__ __forceinline__ C plain_tri(const C z[9]) {
  return (fabs(z[0] - z[4]) + fabs(z[1] - z[4]) + fabs(z[2] - z[4]) + fabs(z[3] - z[4]) + fabs(z[5] - z[4]) +
          fabs(z[6] - z[4]) + fabs(z[7] - z[4]) + fabs(z[8] - z[4])) /
         C(8);
}
template <typename C>
__device__ __forceinline__ C plain_tpi(const C z[9]) {
  return z[4] - (z[0] + z[1] + z[2] + z[3] + z[5] + z[6] + z[7] + z[8]) / C(8);
}
template <typename C>
__device__ __forceinline__ C plain_curv(const C z[9], const DerivParams& P) {
  const C D = ((z[3] + z[5]) / C(2) - z[4]) / static_cast<C>(P.cx2);
  const C E = ((z[1] + z[7]) / C(2) - z[4]) / static_cast<C>(P.cy2);
  return C(-2) * (D + E) * C(100);
}

// float64 bits of s 2^e, e20 = e 2^20: s + 2^31 as the low word of 2^52 + .,
// one FP64 subtraction.
__device__ __forceinline__ uint64_t scaled_bits(int32_t s, uint32_t e20) {
  const double d = __hiloint2double(0x43300000, s ^ static_cast<int32_t>(0x80000000u)) -
                   (4503599627370496.0 + 2147483648.0);
  return static_cast<uint64_t>(__double_as_longlong(
      __hiloint2double(__double2hiint(d) + static_cast<int32_t>(s ? e20 : 0u), __double2loint(d))));
}
template <typename B>
__device__ __forceinline__ B out_bits(uint64_t b64) {
  if constexpr (sizeof(B) == 8) return b64;
  else return __float_as_uint(static_cast<float>(__longlong_as_double(static_cast<long long>(b64))));
}

// A finite float as an integer in units of 2^(e0 - 150), e0 its unit's lowest
// exponent.
__device__ __forceinline__ long long wide_int(float v, uint32_t e0) {
  const uint32_t b = __float_as_uint(v);
  const long long m = static_cast<long long>((b & 0x7fffffu) | 0x800000u) << ((((b >> 23) & 0xffu) - e0) & 63u);
  return (b << 1) == 0u ? 0ll : (b >> 31 ? -m : m);
}

// Eight times TRI and TPI in the values' unit: exact.
__device__ __forceinline__ int32_t abs_of(int32_t v) { return abs(v); }
__device__ __forceinline__ long long abs_of(long long v) { return llabs(v); }
template <typename N>
__device__ __forceinline__ N tri8_of(N tl, N tc, N tr, N ml, N c, N mr, N bl, N bc, N br) {
  return (abs_of(tl - c) + abs_of(tc - c)) + (abs_of(tr - c) + abs_of(ml - c)) + (abs_of(mr - c) + abs_of(bl - c)) +
         (abs_of(bc - c) + abs_of(br - c));
}
template <typename N>
__device__ __forceinline__ N tpi8_of(N tl, N tc, N tr, N ml, N c, N mr, N bl, N bc, N br) {
  return 8 * c - ((tl + tc + tr) + (ml + mr) + (bl + bc + br));
}

// Curvature from the exact neighbour sums a and b as doubles: what the integer
// product does not take (values of more binades, factors far apart).  Errors:
// the factors', one rounding per product and sum, against five roundings of the
// float64 formula.
__device__ __forceinline__ uint64_t curv_bits_f64(uint64_t a, uint64_t b, const DerivParams& P) {
  const double da = __longlong_as_double(static_cast<long long>(a)), db = __longlong_as_double(static_cast<long long>(b));
  return static_cast<uint64_t>(__double_as_longlong(-fma(da, P.kx, db * P.ky)));
}
__device__ __forceinline__ uint64_t curv_bits_f64(int32_t a, int32_t b, int u, const DerivParams& P) {
  return curv_bits_f64(vsr_int_scaled_bits(a, u), vsr_int_scaled_bits(b, u), P);
}

__device__ __forceinline__ void put_bits(void* base, int out_dtype, int64_t i, uint64_t b) {
  if (out_dtype == VSR_F64) static_cast<uint64_t*>(base)[i] = b;
  else static_cast<uint32_t*>(base)[i] = out_bits<uint32_t>(b);
}

// One pixel from its window's integers in units of 2^u.
__device__ __forceinline__ void deriv_ints(const int32_t n[9], int u, int64_t o, const DerivParams& P) {
  const uint32_t e20 = static_cast<uint32_t>(u - 3) << 20;
  const int32_t a = n[3] + n[5] - 2 * n[4], b = n[1] + n[7] - 2 * n[4];
  if (P.tri)
    put_bits(P.tri, P.out_dtype, o, scaled_bits(tri8_of(n[0], n[1], n[2], n[3], n[4], n[5], n[6], n[7], n[8]), e20));
  if (P.tpi)
    put_bits(P.tpi, P.out_dtype, o, scaled_bits(tpi8_of(n[0], n[1], n[2], n[3], n[4], n[5], n[6], n[7], n[8]), e20));
  if (P.curv)
    put_bits(P.curv, P.out_dtype, o, P.ck.ok ? vsr_curv_bits(a, b, &P.ck, u) : curv_bits_f64(a, b, u, P));
}
__device__ __forceinline__ void deriv_ints(const long long n[9], int u, int64_t o, const DerivParams& P) {
  if (P.tri)
    put_bits(P.tri, P.out_dtype, o, vsr_wide_bits(tri8_of(n[0], n[1], n[2], n[3], n[4], n[5], n[6], n[7], n[8]), u - 3));
  if (P.tpi)
    put_bits(P.tpi, P.out_dtype, o, vsr_wide_bits(tpi8_of(n[0], n[1], n[2], n[3], n[4], n[5], n[6], n[7], n[8]), u - 3));
  if (P.curv)
    put_bits(P.curv, P.out_dtype, o,
             curv_bits_f64(vsr_wide_bits(n[3] + n[5] - 2 * n[4], u), vsr_wide_bits(n[1] + n[7] - 2 * n[4], u), P));
}

// A pixel from a window that no unit holds (more than 35 binades, values of
// extreme exponents, infinities, NaN): double-float, or integers without the
// curvature where exponents are extreme but alike.
struct Window {
  float z[9];
};
static __device__ __noinline__ void deriv_df(const Window w, int64_t o, const DerivParams& P) {
  const float* z = w.z;
  // finiteness of the values each formula reads: TRI and TPI all nine,
  // curvature the centre and its four edge neighbours
  bool f5 = true, f9;
#pragma unroll
  for (int k = 1; k < 9; k += 2) f5 &= fabs(z[k]) <= 3.4e38f;
  f5 &= fabs(z[4]) <= 3.4e38f;
  f9 = f5 && fabs(z[0]) <= 3.4e38f && fabs(z[2]) <= 3.4e38f &&
     fabs(z[6]) <= 3.4e38f && fabs(z[8]) <= 3.4e38f;
  // TRI and TPI as exact integers when the window's values share a narrow
  // binade range (terrain_exact.h): the reference's float64 results bit for
  // bit, no double-float arithmetic
  uint32_t bits[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) bits[k] = __float_as_uint(z[k]);
  int32_t t8 = 0, p8 = 0;
  int e2 = 0;
  if ((P.tri || P.tpi) && vsr_tt_exact(bits, &t8, &p8, &e2)) {
    if (P.tri) store_int_scaled(P.tri, P.out_dtype, o, t8, e2 - 3);
    if (P.tpi) store_int_scaled(P.tpi, P.out_dtype, o, p8, e2 - 3);
    if (P.curv) {
      if (f5) {
        const float z4 = z[4];
        const DF dw = two_diff_df(static_cast<float>(z[3]), z4), de = two_diff_df(static_cast<float>(z[5]), z4);
        const DF dn = two_diff_df(static_cast<float>(z[1]), z4), ds = two_diff_df(static_cast<float>(z[7]), z4);
        const DF dx = df_scale(df_add(dw, de), 0.5f), dy = df_scale(df_add(dn, ds), 0.5f);
        const DF e = df_add(df_mul(dx, DF{P.icx2_hi, P.icx2_lo}), df_mul(dy, DF{P.icy2_hi, P.icy2_lo}));
        store_df(P.curv, P.out_dtype, o, df_mul_f(e, -200.0f));
      } else {
        store_out(P.curv, P.out_dtype, o, plain_curv(z, P));
      }
    }
    return;
  }
  // error-free neighbour differences d_i = z_i - z4 (i = 0..3, 5..8)
  DF d[8];
#pragma unroll
  for (int k = 0, i = 0; k < 9; ++k)
    if (k != 4) d[i++] = two_diff_df(z[k], z[4]);
  if (P.tri) {
    if (f9) {
      DF s = df_abs(d[0]);
#pragma unroll
      for (int i = 1; i < 8; ++i) s = df_add(s, df_abs(d[i]));
      store_df(P.tri, P.out_dtype, o, df_scale(s, 0.125f));
    } else {
      store_out(P.tri, P.out_dtype, o, plain_tri(z));
    }
  }
  if (P.tpi) {
    if (f9) {
      DF s = d[0];
#pragma unroll
      for (int i = 1; i < 8; ++i) s = df_add(s, d[i]);
      store_df(P.tpi, P.out_dtype, o, df_scale(df_neg(s), 0.125f));  // z4 - mean = -(sum d_i) / 8
    } else {
      store_out(P.tpi, P.out_dtype, o, plain_tpi(z));
    }
  }
  if (P.curv) {
    if (f5) {
      // (z3 + z5)/2 - z4 = (d_w + d_e) / 2, (z1 + z7)/2 - z4 = (d_n + d_s) / 2
      const DF dx = df_scale(df_add(d[3], d[4]), 0.5f), dy = df_scale(df_add(d[1], d[6]), 0.5f);
      const DF e = df_add(df_mul(dx, DF{P.icx2_hi, P.icx2_lo}), df_mul(dy, DF{P.icy2_hi, P.icy2_lo}));
      store_df(P.curv, P.out_dtype, o, df_mul_f(e, -200.0f));
    } else {
      store_out(P.curv, P.out_dtype, o, plain_curv(z, P));
    }
  }
}

// The unit that holds a window, its lowest exponent and the integers' size.
enum { kUnit32, kUnit64, kUnitNone };
struct WindowUnit {
  uint32_t e;
  int size;
};
__device__ __forceinline__ WindowUnit window_unit(const float z[9]) {
  uint32_t lo = 0xffffffffu, hi = 0u, sign = 0u;
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const uint32_t b = __float_as_uint(z[k]), m = b & 0x7fffffffu;
    lo = min(lo, m - 1u);  // zeros last
    hi = max(hi, m);
    sign |= m ? b : 0u;
  }
  const uint32_t eh = hi ? hi >> 23 : 127u, el = hi ? (lo + 1u) >> 23 : 127u;  // zeros only: any unit
  if (el < kTdExpMin || eh > kTdExpMax || eh - el >= kTdSpanWide) return {el, kUnitNone};
  return {el, eh - el < (sign >> 31 ? kTdSpan : kTdSpanPos) ? kUnit32 : kUnit64};
}

// One pixel of a float32 DEM from its window.
__device__ __forceinline__ void deriv_pixel(const float z[9], WindowUnit w, int64_t o, const DerivParams& P) {
  if (w.size == kUnit32) {
    const float scale = __uint_as_float((277u - w.e) << 23);  // 2^(150 - e)
    int32_t n[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) n[k] = __float2int_rn(z[k] * scale);
    deriv_ints(n, static_cast<int>(w.e) - 150, o, P);
  } else if (w.size == kUnit64) {
    long long n[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) n[k] = wide_int(z[k], w.e);
    deriv_ints(n, static_cast<int>(w.e) - 150, o, P);
  } else {
    deriv_df(Window{z[0], z[1], z[2], z[3], z[4], z[5], z[6], z[7], z[8]}, o, P);
  }
}

// Derivatives of 8/16-bit and float32 DEMs (terrain_strip.cu); -1: too few
// strips to fill the GPU.
int run_terrain_strip(const void* dem, int dtype, const DerivParams& P, int bands, cudaStream_t st);

}  // namespace vsr
