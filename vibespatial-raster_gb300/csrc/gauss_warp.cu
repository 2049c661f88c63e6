// Separable Gaussian for kernels of 3 to 17 taps, in registers.
//
// Semantics as sep_strip (focal.cu): out = sum g g v valid / sum g g valid over
// the in-raster taps, both sums separable; the row pass first, then the column
// pass, taps in ascending order, FP32.
//
// Warp strips (warp_strip.cuh): a lane takes its neighbours' columns by
// shuffles and forms the row sums of its 4 columns; the column pass keeps the
// 2R partial sums of the output rows in flight, and adding a row's term moves
// each sum one place (acc[j] = g h + acc[j + 1]: an FMA's result may go to
// another register, so the shift is free).  Column pairs share packed FMAs.
// No shared memory but for unaligned stores, no barriers.
//
// The weight sum is a constant while all taps of the strip's last 2R+1 rows
// are valid (the warp votes once per row); otherwise its partial sums run
// along, started from the constants when a row with a gap enters.
//
// The weights are formed in float64 on the host and travel as kernel
// arguments: FMAs read them from the constant bank, and the call is one
// launch.
//
// Bound by instruction issue (FMA and shuffles), close to HBM.
#include <cmath>

#include "df_round.h"
#include "vsr_internal.cuh"
#include "warp_strip.cuh"

namespace vsr {
namespace {

constexpr int kGwMaxR = 8;
#ifndef GW_STRIP
#define GW_STRIP 64
#endif
#ifndef GW_AHEAD
#define GW_AHEAD 2
#endif
constexpr int kGwAhead = GW_AHEAD;  // rows loaded ahead

struct GwArgs {
  const void* src;
  int64_t H, W, pitch, band_stride;
  int kind;
  double ndv;
  double nd_out;
  void* dst;
  int64_t out_pitch, out_band_stride;
  bool vin, vout;
  int strip;
  float g[kGwMaxR + 1];  // g[d]: the weight d from the centre
};

// A float's float64 bits (exact).
__device__ __forceinline__ uint64_t widen_bits(float v) {
  const uint32_t b = __float_as_uint(v);
  if (!vsr_f32_widen_ok(b)) return static_cast<uint64_t>(__double_as_longlong(static_cast<double>(v)));
  uint32_t hi, lo;
  vsr_f32_widen(b, &hi, &lo);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}

template <typename T>
__device__ __forceinline__ float value_of(uint32_t b) {
  if constexpr (std::is_same<T, float>::value) return __uint_as_float(b);
  else return static_cast<float>(static_cast<T>(b));
}

template <int R>
struct GwGeom {
  static constexpr int K = 2 * R + 1, HL = (R + 3) / 4, kCols = 128 - 8 * HL, kWin = 4 * (2 * HL + 1);
};

// Row sums of a lane's 4 columns.
template <int R>
__device__ __forceinline__ void row_sums(const float own[4], const float* g, float h[4]) {
  constexpr int HL = GwGeom<R>::HL, C0 = 4 * HL;
  float w[GwGeom<R>::kWin];
#pragma unroll
  for (int e = 0; e < 4; ++e) w[C0 + e] = own[e];
#pragma unroll
  for (int q = 1; q <= HL; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (4 * q - e <= R) w[C0 - 4 * q + e] = __shfl_up_sync(0xffffffffu, own[e], q);
      if (4 * q + e - 3 <= R) w[C0 + 4 * q + e] = __shfl_down_sync(0xffffffffu, own[e], q);
    }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    float s = g[R] * w[C0 + c - R];
#pragma unroll
    for (int t = 1; t < 2 * R + 1; ++t) s = fmaf(g[t < R ? R - t : t - R], w[C0 + c - R + t], s);
    h[c] = s;
  }
}

// Add a row's terms to the partial sums of the 2R rows in flight; the row
// that it completes comes back.
template <int R>
__device__ __forceinline__ float2 column_step(float2 acc[2 * R], const float* g, float2 h) {
  auto gg = [&](int t) { const float v = g[t < R ? R - t : t - R]; return make_float2(v, v); };
  const float2 out = __ffma2_rn(gg(2 * R), h, acc[0]);
#pragma unroll
  for (int j = 0; j < 2 * R - 1; ++j) acc[j] = __ffma2_rn(gg(2 * R - 1 - j), h, acc[j + 1]);
  acc[2 * R - 1] = __fmul2_rn(gg(0), h);
  return out;
}

template <int R, typename T, typename B>
__global__ void __launch_bounds__(32) gauss_warp(const __grid_constant__ GwArgs a) {
  using G = GwGeom<R>;
  constexpr bool kFloat = std::is_same<T, float>::value;
  __shared__ __align__(16) B obuf[128];
  const int lane = threadIdx.x;
  const int64_t xw = static_cast<int64_t>(blockIdx.x) * G::kCols - 4 * G::HL;
  const int64_t xs = xw + 4 * lane, ys = static_cast<int64_t>(blockIdx.y) * a.strip;
  const int nout = static_cast<int>(a.H - ys < a.strip ? a.H - ys : static_cast<int64_t>(a.strip));
  const int nin = nout + 2 * R;
  uint32_t inm = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) inm |= static_cast<uint32_t>(xs + e >= 0 && xs + e < a.W) << e;
  const T* src = static_cast<const T*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride;
  const T* lp = src + (ys - R) * a.pitch + xs;
  // input rows [r0, r1) of the strip lie in the raster
  const int r0 = ys < R ? static_cast<int>(R - ys) : 0;
  const int r1 = a.H - (ys - R) < nin ? static_cast<int>(a.H - (ys - R)) : nin;
  auto load = [&](int i, uint32_t e[4]) {
    if (i >= r0 && i < r1) strip_load4<T, true>(lp, inm, a.vin, e);
    lp += a.pitch;
  };
  const bool has_nd = a.kind == VSR_NODATA_VALUE, nd_nan = a.kind == VSR_NODATA_NAN;
  const T ndq = static_cast<T>(a.ndv);
  constexpr int lo = 4 * G::HL;
  const int hi = static_cast<int>(a.W - xw < 128 - 4 * G::HL ? a.W - xw : static_cast<int64_t>(128 - 4 * G::HL));
  B* orow = static_cast<B*>(a.dst) + static_cast<int64_t>(blockIdx.z) * a.out_band_stride + ys * a.out_pitch + xw;
  // sums of weights of a row and of a window without gaps
  float rd = a.g[R];
#pragma unroll
  for (int t = 1; t < 2 * R + 1; ++t) rd += a.g[t < R ? R - t : t - R];
  float wd = a.g[R] * rd;
#pragma unroll
  for (int t = 1; t < 2 * R + 1; ++t) wd = fmaf(a.g[t < R ? R - t : t - R], rd, wd);

  uint32_t pre[kGwAhead][4];
#pragma unroll
  for (int u = 0; u < kGwAhead; ++u) {
#pragma unroll
    for (int e = 0; e < 4; ++e) pre[u][e] = 0u;
    load(u, pre[u]);
  }
  float2 num[2][2 * R], den[2][2 * R];
#pragma unroll
  for (int j = 0; j < 2 * R; ++j) num[0][j] = num[1][j] = den[0][j] = den[1][j] = make_float2(0.0f, 0.0f);
  int gaps = 0;     // rows until the last row with a gap leaves the window
  uint64_t vm = 0;  // validity of the lane's columns, 4 bits per row
  // not unrolled: two copies of the body overflowed the instruction cache
#pragma unroll 1
  for (int i = 0; i < nin; ++i) {
    float v[4];
    uint32_t ok = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = value_of<T>(pre[0][e]);
      bool good;
      if constexpr (kFloat) good = !(has_nd && v[e] == ndq) && !(nd_nan && v[e] != v[e]);
      else good = !(has_nd && static_cast<T>(pre[0][e]) == ndq);
      ok |= good ? 1u << e : 0u;
#pragma unroll
      for (int u = 0; u + 1 < kGwAhead; ++u) pre[u][e] = pre[u + 1][e];
    }
    ok &= inm;
    const bool in = i >= r0 && i < r1;
    if (!in) ok = 0u;
    load(i + kGwAhead, pre[kGwAhead - 1]);
    vm = (vm << 4) | ok;
    const bool gap = !__all_sync(0xffffffffu, ok == 0xFu);
    if (gap) {
      // v * valid, as the reference masks: a NaN stays NaN under a zero
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = in ? v[e] * ((ok >> e) & 1u ? 1.0f : 0.0f) : 0.0f;
      if (gaps == 0) {  // rows so far had none: acc[j] holds the constant terms t = 0 .. 2R - 1 - j
        float s = a.g[R] * rd;
#pragma unroll
        for (int j = 2 * R - 1; j >= 0; --j) {
          den[0][j] = den[1][j] = make_float2(s, s);
          const int t = 2 * R - j;
          s = fmaf(a.g[t < R ? R - t : t - R], rd, s);
        }
      }
      gaps = 2 * R + 1;
    }
    float h[4];
    row_sums<R>(v, a.g, h);
    const float2 o0 = column_step<R>(num[0], a.g, make_float2(h[0], h[1]));
    const float2 o1 = column_step<R>(num[1], a.g, make_float2(h[2], h[3]));
    float2 d0 = make_float2(wd, wd), d1 = d0;
    if (gaps) {
      --gaps;
      float w[4] = {rd, rd, rd, rd};
      if (gap) {
        float f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = (ok >> e) & 1u ? 1.0f : 0.0f;
        row_sums<R>(f, a.g, w);
      }
      d0 = column_step<R>(den[0], a.g, make_float2(w[0], w[1]));
      d1 = column_step<R>(den[1], a.g, make_float2(w[2], w[3]));
    }
    if (i >= 2 * R) {
      const uint32_t cm = static_cast<uint32_t>(vm >> (4 * R));
      const float n4[4] = {o0.x, o0.y, o1.x, o1.y}, w4[4] = {d0.x, d0.y, d1.x, d1.y};
      B b[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const bool nd = !((cm >> c) & 1u) || !(w4[c] > 0.0f);
        const float q = n4[c] / w4[c];
        if constexpr (sizeof(B) == 8) b[c] = nd ? static_cast<B>(__double_as_longlong(a.nd_out)) : widen_bits(q);
        else b[c] = __float_as_uint(nd ? static_cast<float>(a.nd_out) : q);
      }
      strip_store4<B>(orow, b, lane, lo, hi, a.vout, obuf);
      orow += a.out_pitch;
    }
  }
}

template <int R, typename T>
int launch_gw(GwArgs& a, int bands, bool f64, cudaStream_t st) {
  const int64_t gx = (a.W + GwGeom<R>::kCols - 1) / GwGeom<R>::kCols;
  a.strip = GW_STRIP;
  const int64_t gy = (a.H + a.strip - 1) / a.strip;
  if (gy > 65535) return fail(VSR_ERR_UNSUPPORTED, "raster too tall for the separable Gaussian grid");
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(bands));
  if (f64) gauss_warp<R, T, uint64_t><<<grid, 32, 0, st>>>(a);
  else gauss_warp<R, T, uint32_t><<<grid, 32, 0, st>>>(a);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

template <typename T>
int launch_gw_r(GwArgs& a, int r, int bands, bool f64, cudaStream_t st) {
  switch (r) {
    case 1: return launch_gw<1, T>(a, bands, f64, st);
    case 2: return launch_gw<2, T>(a, bands, f64, st);
    case 3: return launch_gw<3, T>(a, bands, f64, st);
    case 4: return launch_gw<4, T>(a, bands, f64, st);
    case 5: return launch_gw<5, T>(a, bands, f64, st);
    case 6: return launch_gw<6, T>(a, bands, f64, st);
    case 7: return launch_gw<7, T>(a, bands, f64, st);
    default: return launch_gw<8, T>(a, bands, f64, st);
  }
}

}  // namespace

// The Gaussian of an odd k in 3..17 on 8/16-bit and float32 rasters; -1 for
// anything else.  ``kind`` and ``ndv`` as resolve_nodata gives them.
int run_gauss_warp(const void* src, int dtype, int bands, int64_t band_stride, int64_t H, int64_t W, int64_t pitch,
                   double sigma, int k, int kind, double ndv, double nd_out, void* dst, int out_dtype,
                   int64_t out_band_stride, int64_t out_pitch, cudaStream_t st) {
  if (k < 3 || k > 2 * kGwMaxR + 1 || k % 2 == 0) return -1;
  const size_t es = dtype_size(dtype), os = out_dtype == VSR_F64 ? 8 : 4;
  GwArgs a{src, H, W, pitch, bands > 1 ? band_stride : 0, kind, ndv, nd_out, dst, out_pitch,
           bands > 1 ? out_band_stride : 0};
  a.vin = aligned(src, 4 * es) && pitch % 4 == 0 && a.band_stride % 4 == 0;
  a.vout = aligned(dst, 4 * os) && out_pitch % 4 == 0 && a.out_band_stride % 4 == 0;
  for (int d = 0; d <= k / 2; ++d) a.g[d] = static_cast<float>(std::exp(-0.5 * (d / sigma) * (d / sigma)));
  switch (dtype) {
    case VSR_U8: return launch_gw_r<uint8_t>(a, k / 2, bands, os == 8, st);
    case VSR_I16: return launch_gw_r<int16_t>(a, k / 2, bands, os == 8, st);
    case VSR_U16: return launch_gw_r<uint16_t>(a, k / 2, bands, os == 8, st);
    case VSR_F32: return launch_gw_r<float>(a, k / 2, bands, os == 8, st);
    default: return -1;
  }
}

}  // namespace vsr
