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
// No barriers.
//
// The weight sum is a constant while all taps of the strip's last 2R+1 rows
// are valid (the warp votes once per row); otherwise the rows' weight sums go
// through a small ring in shared memory and are added up per output row.
//
// The weights are formed in float64 on the host and travel as kernel
// arguments: FMAs read them from the constant bank, and the call is one
// launch.
//
// Bound by instruction issue (13 taps at 6000^2, 162 us: 74 % of the issue slots,
// ALU pipe 54 %, FMA 29 %, DRAM 21 %).
#include <cmath>

#include "vsr_internal.cuh"
#include "warp_strip.cuh"

namespace vsr {
namespace {

constexpr int kGwMaxR = 8;
constexpr int kGwDepth = 6;  // rows in shared memory

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
  constexpr int K = G::K;
  constexpr bool kFloat = std::is_same<T, float>::value;
  __shared__ __align__(16) B obuf[128];
  __shared__ __align__(16) unsigned char rows[RowRing<T, kGwDepth>::kBytes];
  // while a window holds a gap: the weight sums of its rows and the validity
  // of the lane's columns (4 bits), each thread reading only its own
  __shared__ float4 wring[K][32];
  __shared__ uint32_t oring[K][32];
  auto g_at = [&](int t) { return a.g[t < R ? R - t : t - R]; };
  const int lane = threadIdx.x;
  const int64_t xw = static_cast<int64_t>(blockIdx.x) * G::kCols - 4 * G::HL;
  const int64_t xs = xw + 4 * lane, ys = static_cast<int64_t>(blockIdx.y) * a.strip;
  const int nout = static_cast<int>(a.H - ys < a.strip ? a.H - ys : static_cast<int64_t>(a.strip));
  const int nin = nout + 2 * R;
  bool col_out[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) col_out[e] = xs + e < 0 || xs + e >= a.W;
  const bool writes = 4 * lane >= 4 * G::HL && 4 * lane < 128 - 4 * G::HL && !col_out[0];
  const T* src = static_cast<const T*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride;
  // input rows [r0, r1) of the strip lie in the raster
  const int r0 = ys < R ? static_cast<int>(R - ys) : 0;
  const int r1 = a.H - (ys - R) < nin ? static_cast<int>(a.H - (ys - R)) : nin;
  const bool nd_nan = a.kind == VSR_NODATA_NAN, nd_val = a.kind == VSR_NODATA_VALUE;
  const float ndq = nd_val ? static_cast<float>(a.ndv) : __int_as_float(0x7fffffff);  // NaN: equal to nothing
  constexpr int lo = 4 * G::HL;
  const int hi = static_cast<int>(a.W - xw < 128 - 4 * G::HL ? a.W - xw : static_cast<int64_t>(128 - 4 * G::HL));
  B* orow = static_cast<B*>(a.dst) + static_cast<int64_t>(blockIdx.z) * a.out_band_stride + ys * a.out_pitch + xw;
  // sums of weights of a row (its columns in the raster) and of K such rows
  float rd[4], wd[4], wr[4];
  {
    float f[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = col_out[e] ? 0.0f : 1.0f;
    row_sums<R>(f, a.g, rd);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      wd[c] = g_at(0) * rd[c];
#pragma unroll
      for (int t = 1; t < K; ++t) wd[c] = fmaf(g_at(t), rd[c], wd[c]);
      wr[c] = vsr_div_recip(wd[c]);
    }
  }
  RowRing<T, kGwDepth> in_rows;
  in_rows.start(rows, src + (ys - R) * a.pitch + xw, a.pitch, xw, a.W, r0, r1, a.vin);
  float2 num[2][2 * R];
#pragma unroll
  for (int j = 0; j < 2 * R; ++j) num[0][j] = num[1][j] = make_float2(0.0f, 0.0f);
  int gaps = 0;  // rows until the last row with a gap has left the window
  int slot = 0;  // ring slot of the row (while gaps > 0)
  __syncwarp();
  // not unrolled: more copies of the body outgrow the instruction cache (4
  // rows per iteration took 263 us where 1 took 192)
#pragma unroll 1
  for (int i = 0; i < nin; ++i) {
    uint32_t raw[4];
    in_rows.take(raw);
    float v[4];
    bool good = true;
    const bool in = i >= r0 && i < r1;  // a row outside reads as zeros
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = strip_value<T>(raw[e]);
      good &= ((v[e] != ndq) & !(kFloat & nd_nan & (v[e] != v[e]))) | col_out[e];
    }
    const bool gap = !__all_sync(0xffffffffu, good || !in);
    uint32_t ok = 0xFu;
    if (gap) {
      ok = 0u;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const bool o = !col_out[e] & (v[e] != ndq) & !(kFloat & nd_nan & (v[e] != v[e]));
        ok |= o ? 1u << e : 0u;
        v[e] *= o ? 1.0f : 0.0f;  // as the reference masks: a NaN stays NaN under a zero
      }
      if (gaps == 0) {  // the rows before had none
        for (int t = 1; t < K; ++t) {
          const bool ti = i - K + t >= r0 && i - K + t < r1;
          wring[t][lane] = ti ? make_float4(rd[0], rd[1], rd[2], rd[3]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          oring[t][lane] = 0xFu;
        }
        slot = 0;
      }
      gaps = K;
    }
    float h[4];
    row_sums<R>(v, a.g, h);
    const float2 o0 = column_step<R>(num[0], a.g, make_float2(h[0], h[1]));
    const float2 o1 = column_step<R>(num[1], a.g, make_float2(h[2], h[3]));
    const float n4[4] = {o0.x, o0.y, o1.x, o1.y};
    uint32_t cm = 0xFu;  // validity of the output row's columns
    float w4[4], r4[4];
    bool whole = false;
    if (gaps) {
      --gaps;
      float w[4] = {rd[0], rd[1], rd[2], rd[3]};
      if (gap) {
        float f[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) f[e] = (ok >> e) & 1u ? 1.0f : 0.0f;
        row_sums<R>(f, a.g, w);
      }
      wring[slot][lane] = in ? make_float4(w[0], w[1], w[2], w[3]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      oring[slot][lane] = ok;
      slot = slot + 1 == K ? 0 : slot + 1;
      // tap t's row is in slot (slot + t) mod K; taps in ascending order, as in
      // the numerator: rounding errors common to both sums cancel in the quotient
      float2 d0 = make_float2(0.0f, 0.0f), d1 = d0;
#pragma unroll
      for (int t = 0; t < K; ++t) {
        const int s = slot + t;
        const float4 x = wring[s >= K ? s - K : s][lane];
        const float2 gt = make_float2(g_at(t), g_at(t));
        d0 = __ffma2_rn(gt, make_float2(x.x, x.y), d0);
        d1 = __ffma2_rn(gt, make_float2(x.z, x.w), d1);
      }
      const int cs = slot + R;
      cm = oring[cs >= K ? cs - K : cs][lane];
      w4[0] = d0.x;
      w4[1] = d0.y;
      w4[2] = d1.x;
      w4[3] = d1.y;
    } else if (i - 2 * R < r0 || i >= r1) {  // rows outside: only those inside weigh
#pragma unroll
      for (int c = 0; c < 4; ++c) w4[c] = 0.0f;
#pragma unroll
      for (int t = 0; t < K; ++t) {
        const float gt = i - 2 * R + t >= r0 && i - 2 * R + t < r1 ? g_at(t) : 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) w4[c] = fmaf(gt, rd[c], w4[c]);
      }
    } else {
#pragma unroll
      for (int c = 0; c < 4; ++c) w4[c] = wd[c];
      whole = true;
    }
    if (i >= 2 * R) {
      B b[4];
      bool bad = false;
      float q[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        r4[c] = whole ? wr[c] : vsr_div_recip(w4[c]);
        bad |= !(w4[c] > 1.0e-30f);
        q[c] = strip_quot(n4[c], w4[c], r4[c], bad);
      }
      if (bad && writes) {  // a lane that writes nothing may hold anything
#pragma unroll
        for (int c = 0; c < 4; ++c) q[c] = n4[c] / w4[c];
      }
      bool nd[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) nd[c] = !((cm >> c) & 1u) | !(w4[c] > 0.0f);
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
  }
}

template <int R, typename T>
int launch_gw(GwArgs& a, int bands, bool f64, cudaStream_t st) {
  const int64_t gx = (a.W + GwGeom<R>::kCols - 1) / GwGeom<R>::kCols;
  // rows per strip: the most that gives every SM 32 warps, two rounds of what
  // fits (2R rows of a strip are read again by the next; 900 x 6000, 13 taps: 77 us at
  // 64 rows, 54 us at 32)
  a.strip = 64;
  while (a.strip > 16 && gx * ((a.H + a.strip - 1) / a.strip) * bands < 32 * static_cast<int64_t>(sm_count())) a.strip /= 2;
  const int64_t gy = (a.H + a.strip - 1) / a.strip;
  if ((a.H + 31) / 32 > 65535 || gy > 65535)
    return fail(VSR_ERR_UNSUPPORTED, "raster too tall for the separable Gaussian grid");
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
