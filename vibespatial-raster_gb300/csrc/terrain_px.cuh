// Terrain derivatives of one pixel (terrain.cu, terrain_strip.cu): the formulas
// and the double-float arithmetic.
//
// GB300's FP64 rate is a small fraction of its FP32 rate, so windows of
// 8/16-bit and float32 elevations that the integer forms do not take are
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
  vsr_curv_k ck;    // the curvature factors as integers (terrain_fixed.h)
};

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

// One pixel of a float32-exact DEM from its window, in double-float where the
// exact integers do not apply.
__device__ __forceinline__ void deriv_pixel(const float z[9], int64_t o, const DerivParams& P) {
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

// Derivatives of 8/16-bit and float32 DEMs (terrain_strip.cu).
int run_terrain_strip(const void* dem, int dtype, const DerivParams& P, int bands, cudaStream_t st);

}  // namespace vsr
