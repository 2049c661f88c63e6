// Dense normalised convolution with small square kernels (odd, 3 to 13), in
// registers.
//
// Semantics as conv_direct (focal.cu): out = sum w v valid / sum w valid over
// the in-raster taps; one partial sum per kernel row, added up over the rows,
// FP32; a NaN anywhere in the window gives NaN.
//
// Warp strips (warp_strip.cuh), 4 columns per lane, the neighbours' by
// shuffles.  An input row adds its K partial sums to the K output rows it
// reaches; those K sums per column live in registers and move one place per
// row (acc[j] = acc[j + 1] + part, so the shift is free).  Weights come as
// kernel arguments (FMAs read them from the constant bank): a call is one
// launch, with no copy of the weights.  The weight sum is the full one while
// all taps are valid; windows with a gap (nodata or the border) are summed
// again over the validity bits of their rows.
//
// Bound by instruction issue (5 x 5 at 4099 x 5003, 83 us: 77 % of the issue
// slots, ALU pipe 55 %, FMA 32 %, DRAM 18 %).
#include <cmath>

#include "vsr_internal.cuh"
#include "warp_strip.cuh"

namespace vsr {
namespace {

constexpr int kCwMaxK = 13;
constexpr int kCwDepth = 6;  // rows in shared memory

struct CwArgs {
  const void* src;
  int64_t H, W, pitch, band_stride;
  int kind;
  double ndv;
  double nd_out;
  void* dst;
  int64_t out_pitch, out_band_stride;
  bool vin, vout;
  int strip;
  float wsum;
  float w[kCwMaxK * kCwMaxK];  // row-major K x K
};

template <int K>
struct CwGeom {
  static constexpr int R = K / 2, HL = (R + 3) / 4, kCols = 128 - 8 * HL, C0 = 4 * HL, kWin = 4 * (2 * HL + 1);
};

template <int K, typename T, typename B>
__global__ void __launch_bounds__(32) conv_warp(const __grid_constant__ CwArgs a) {
  using G = CwGeom<K>;
  constexpr int R = G::R, HL = G::HL, C0 = G::C0;
  constexpr bool kFloat = std::is_same<T, float>::value;
  __shared__ __align__(16) B obuf[128];
  __shared__ __align__(16) unsigned char rows[RowRing<T, kCwDepth>::kBytes];
  // while a window holds a gap: the validity of its rows' columns that the
  // lane reaches, each thread reading only its own
  __shared__ uint32_t mring[K][32];
  const int lane = threadIdx.x;
  const int64_t xw = static_cast<int64_t>(blockIdx.x) * G::kCols - 4 * HL;
  const int64_t xs = xw + 4 * lane, ys = static_cast<int64_t>(blockIdx.y) * a.strip;
  const int nout = static_cast<int>(a.H - ys < a.strip ? a.H - ys : static_cast<int64_t>(a.strip));
  const int nin = nout + 2 * R;
  bool col_out[4];
  uint32_t inm = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    col_out[e] = xs + e < 0 || xs + e >= a.W;
    inm |= col_out[e] ? 0u : 1u << e;
  }
  const bool writes = lane >= HL && lane < 32 - HL && !col_out[0];
  const T* src = static_cast<const T*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride;
  // input rows [r0, r1) of the strip lie in the raster
  const int r0 = ys < R ? static_cast<int>(R - ys) : 0;
  const int r1 = a.H - (ys - R) < nin ? static_cast<int>(a.H - (ys - R)) : nin;
  const bool nd_nan = a.kind == VSR_NODATA_NAN;
  const float ndq = a.kind == VSR_NODATA_VALUE ? static_cast<float>(a.ndv) : __int_as_float(0x7fffffff);
  constexpr int lo = 4 * HL;
  const int hi = static_cast<int>(a.W - xw < 128 - 4 * HL ? a.W - xw : static_cast<int64_t>(128 - 4 * HL));
  B* orow = static_cast<B*>(a.dst) + static_cast<int64_t>(blockIdx.z) * a.out_band_stride + ys * a.out_pitch + xw;
  // bit j of a row's mask: column xs - C0 + j is valid
  auto spread = [&](uint32_t m) -> uint32_t {
    uint32_t r = m << C0;
#pragma unroll
    for (int q = 1; q <= HL; ++q) {
      r |= __shfl_up_sync(0xffffffffu, m, q) << (C0 - 4 * q);
      r |= __shfl_down_sync(0xffffffffu, m, q) << (C0 + 4 * q);
    }
    return r;
  };
  // weights of a window's row over its valid columns
  auto add_weights = [&](uint32_t m, int ky, float d[4]) {
    float f[4 + 2 * R];
#pragma unroll
    for (int j = 0; j < 4 + 2 * R; ++j) f[j] = (m >> (C0 - R + j)) & 1u ? 1.0f : 0.0f;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float p = a.w[ky * K] * f[c];
#pragma unroll
      for (int kx = 1; kx < K; ++kx) p = fmaf(a.w[ky * K + kx], f[c + kx], p);
      d[c] += p;
    }
  };
  // the weight sums where only columns of the raster's edge are missing
  const uint32_t colm = spread(inm);
  float wd[4] = {a.wsum, a.wsum, a.wsum, a.wsum}, wr[4];
  if (xw < 0 || xw + 128 > a.W) {
    float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int ky = 0; ky < K; ++ky) add_weights(colm, ky, d);
#pragma unroll
    for (int c = 0; c < 4; ++c) wd[c] = d[c];
  }
  bool odd = false;  // a weight sum whose reciprocal or quotients (numerators from 1e-30) may not be normal
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    wr[c] = vsr_div_recip(wd[c]);
    odd |= !(wd[c] > 1.0e-30f && wd[c] < 1.0e6f);
  }
  RowRing<T, kCwDepth> in_rows;
  in_rows.start(rows, src + (ys - R) * a.pitch + xw, a.pitch, xw, a.W, r0, r1, a.vin);
  float acc[K - 1][4];  // acc[j]: the output row that completes j rows on
#pragma unroll
  for (int j = 0; j < K - 1; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[j][c] = 0.0f;
  int gaps = 0, slot = 0;
#pragma unroll 1
  for (int i = 0; i < nin; ++i) {
    uint32_t raw[4];
    in_rows.take(raw);
    float w[G::kWin];
    bool good = true;
    const bool in = i >= r0 && i < r1;  // a row outside reads as zeros
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float v = strip_value<T>(raw[e]);
      w[C0 + e] = v;
      good &= ((v != ndq) & !(kFloat & nd_nan & (v != v))) | col_out[e];
    }
    if (!__all_sync(0xffffffffu, good && in)) {
      uint32_t ok = 0u;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float v = w[C0 + e];
        const bool o = in & !col_out[e] & (v != ndq) & !(kFloat & nd_nan & (v != v));
        ok |= o ? 1u << e : 0u;
        w[C0 + e] = v * (o ? 1.0f : 0.0f);  // as the reference masks: a NaN stays NaN under a zero
      }
      if (gaps == 0) {  // the rows before had none
        for (int t = 1; t < K; ++t) mring[t][lane] = colm;
        slot = 0;
      }
      mring[slot][lane] = spread(ok);
      slot = slot + 1 == K ? 0 : slot + 1;
      gaps = K;
    } else if (gaps) {
      mring[slot][lane] = colm;
      slot = slot + 1 == K ? 0 : slot + 1;
    }
#pragma unroll
    for (int q = 1; q <= HL; ++q)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (4 * q - e <= R) w[C0 - 4 * q + e] = __shfl_up_sync(0xffffffffu, w[C0 + e], q);
        if (4 * q + e - 3 <= R) w[C0 + 4 * q + e] = __shfl_down_sync(0xffffffffu, w[C0 + e], q);
      }
    float done[4];
#pragma unroll
    for (int j = 0; j < K; ++j) {  // kernel row K - 1 - j completes in j rows
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float* wt = a.w + (K - 1 - j) * K;
        float p = wt[0] * w[C0 - R + c];
#pragma unroll
        for (int kx = 1; kx < K; ++kx) p = fmaf(wt[kx], w[C0 - R + c + kx], p);
        if (j < K - 1) p += acc[j][c];
        if (j == 0) done[c] = p;
        else acc[j - 1][c] = p;
      }
    }
    if (i >= 2 * R) {
      float q[4], d[4] = {wd[0], wd[1], wd[2], wd[3]};
      uint32_t cm = 0xFu;
      bool bad = odd;
      if (gaps) {
#pragma unroll
        for (int c = 0; c < 4; ++c) d[c] = 0.0f;
#pragma unroll
        for (int t = 0; t < K; ++t) {
          const int s = slot + t >= K ? slot + t - K : slot + t;  // the row of weights t
          const uint32_t m = mring[s][lane];
          add_weights(m, t, d);
          if (t == R) cm = m >> C0;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          bad |= !(d[c] > 1.0e-30f && d[c] < 1.0e6f);
          q[c] = strip_quot(done[c], d[c], vsr_div_recip(d[c]), bad);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) q[c] = strip_quot(done[c], d[c], wr[c], bad);
      }
      if (bad && writes) {  // a lane that writes nothing may hold anything
#pragma unroll
        for (int c = 0; c < 4; ++c) q[c] = done[c] / d[c];
      }
      B b[4];
      bool nd[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) nd[c] = !((cm >> c) & 1u) | !(d[c] > 0.0f);
      if constexpr (sizeof(B) == 8) {
        widen4(q, b);
#pragma unroll
        for (int c = 0; c < 4; ++c) b[c] = nd[c] ? static_cast<B>(__double_as_longlong(a.nd_out)) : b[c];
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) b[c] = __float_as_uint(nd[c] ? static_cast<float>(a.nd_out) : q[c]);
      }
      strip_store4<B>(orow, b, lane, lo, hi, a.vout, obuf);
      orow += a.out_pitch;
    }
    if (gaps) --gaps;
  }
}

template <int K, typename T>
int launch_cw(CwArgs& a, int bands, bool f64, cudaStream_t st) {
  const int64_t gx = (a.W + CwGeom<K>::kCols - 1) / CwGeom<K>::kCols;
  // rows per strip: see gauss_warp.cu
  a.strip = 64;
  while (a.strip > 16 && gx * ((a.H + a.strip - 1) / a.strip) * bands < 32 * static_cast<int64_t>(sm_count())) a.strip /= 2;
  const int64_t gy = (a.H + a.strip - 1) / a.strip;
  if ((a.H + 31) / 32 > 65535 || gy > 65535)
    return fail(VSR_ERR_UNSUPPORTED, "raster too tall for the direct convolution grid");
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(bands));
  if (f64) conv_warp<K, T, uint64_t><<<grid, 32, 0, st>>>(a);
  else conv_warp<K, T, uint32_t><<<grid, 32, 0, st>>>(a);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

template <typename T>
int launch_cw_k(CwArgs& a, int k, int bands, bool f64, cudaStream_t st) {
  switch (k) {
    case 3: return launch_cw<3, T>(a, bands, f64, st);
    case 5: return launch_cw<5, T>(a, bands, f64, st);
    case 7: return launch_cw<7, T>(a, bands, f64, st);
    case 9: return launch_cw<9, T>(a, bands, f64, st);
    case 11: return launch_cw<11, T>(a, bands, f64, st);
    default: return launch_cw<13, T>(a, bands, f64, st);
  }
}

}  // namespace

// The convolution with a k x k kernel, k odd in 3..13, of an 8/16-bit or
// float32 raster; -1 for anything else.  ``kind`` and ``ndv`` as
// resolve_nodata gives them.
int run_conv_warp(const void* src, int dtype, int bands, int64_t band_stride, int64_t H, int64_t W, int64_t pitch,
                  const double* weights_host, int kh, int kw, int kind, double ndv, double nd_out, void* dst,
                  int out_dtype, int64_t out_band_stride, int64_t out_pitch, cudaStream_t st) {
  if (kh != kw || kh < 3 || kh > kCwMaxK || kh % 2 == 0) return -1;
  const size_t es = dtype_size(dtype), os = out_dtype == VSR_F64 ? 8 : 4;
  CwArgs a{src, H, W, pitch, bands > 1 ? band_stride : 0, kind, ndv, nd_out, dst, out_pitch,
           bands > 1 ? out_band_stride : 0};
  a.vin = aligned(src, 4 * es) && pitch % 4 == 0 && a.band_stride % 4 == 0;
  a.vout = aligned(dst, 4 * os) && out_pitch % 4 == 0 && a.out_band_stride % 4 == 0;
  double sum = 0.0;
  for (int i = 0; i < kh * kw; ++i) {
    a.w[i] = static_cast<float>(weights_host[i]);
    sum += weights_host[i];
  }
  a.wsum = static_cast<float>(sum);
  switch (dtype) {
    case VSR_U8: return launch_cw_k<uint8_t>(a, kh, bands, os == 8, st);
    case VSR_I16: return launch_cw_k<int16_t>(a, kh, bands, os == 8, st);
    case VSR_U16: return launch_cw_k<uint16_t>(a, kh, bands, os == 8, st);
    case VSR_F32: return launch_cw_k<float>(a, kh, bands, os == 8, st);
    default: return -1;
  }
}

}  // namespace vsr
