// Terrain derivatives on the 3x3 window: TRI, TPI and profile curvature in
// one pass (any subset of the three outputs).
//
// Replaces the reference's ``terrain_derivatives`` NVRTC kernel
// (kernels/focal.py:487-647) and its launch glue (algebra.py:2854-2991): the
// float64 up-cast, the uint8 mask pass and one launch per derivative.  The
// semantics are the reference CPU/GPU ones (algebra.py:3352-3445): window
// z0..z8 (row-major, z4 the centre) with edge replication,
//   TRI  = sum |z_i - z4| / 8                      (Riley et al. 1999)
//   TPI  = z4 - sum z_i / 8
//   curv = -2 (D + E) 100,  D = ((z3 + z5)/2 - z4) / cx^2,
//                           E = ((z1 + z7)/2 - z4) / cy^2   (Zevenbergen & Thorne 1987)
// over the 8 neighbours; border pixels and pixels whose window touches a
// nodata pixel get the output nodata value.
//
// int32 and float64 DEMs are computed here in FP64 with the reference's own
// operation order; 8/16-bit and float32 DEMs in terrain_strip.cu.
#include <algorithm>
#include <cmath>

#include "terrain_px.cuh"

namespace vsr {
namespace {

constexpr int kDTW = 32, kDTH = 8;  // output tile: 32 x 8 pixels, one per thread
constexpr int kDSW = kDTW + 2, kDSH = kDTH + 2;

// One pixel per thread.  int32 and float64 DEMs in FP64 with the reference's
// formulas; 8/16-bit and float32 DEMs of too few strips in the strips' integers
// (and FP64 for the curvature) window by window.
template <typename T>
__global__ void __launch_bounds__(kDTW * kDTH) terrain_deriv_kernel(const T* __restrict__ src, const DerivParams P) {
  using C = std::conditional_t<std::is_same<T, int32_t>::value || std::is_same<T, double>::value, double,
                               std::conditional_t<std::is_same<T, float>::value, float, int32_t>>;
  __shared__ C tile[kDSH][kDSW + 1];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kDTW + tx;
  const int64_t x0 = static_cast<int64_t>(blockIdx.x) * kDTW, y0 = static_cast<int64_t>(blockIdx.y) * kDTH;
  src += static_cast<int64_t>(blockIdx.z) * P.band_stride;
  // the tile and its 1-pixel halo, coordinates clamped (edge replication)
  for (int i = tid; i < kDSH * kDSW; i += kDTW * kDTH) {
    const int r = i / kDSW, c = i - r * kDSW;
    int64_t gy = y0 - 1 + r, gx = x0 - 1 + c;
    gy = gy < 0 ? 0 : (gy >= P.H ? P.H - 1 : gy);
    gx = gx < 0 ? 0 : (gx >= P.W ? P.W - 1 : gx);
    tile[r][c] = static_cast<C>(__ldg(src + gy * P.pitch + gx));
  }
  __syncthreads();
  const int64_t x = x0 + tx, y = y0 + ty;
  const int64_t o = static_cast<int64_t>(blockIdx.z) * P.out_band_stride + y * P.out_pitch + x;
  C z[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) z[k] = tile[ty + k / 3][tx + k % 3];
  bool nd = x == 0 || y == 0 || x == P.W - 1 || y == P.H - 1;
  if (P.nd_kind == VSR_NODATA_VALUE) {
    const C ndv = static_cast<C>(P.nd_in);
#pragma unroll
    for (int k = 0; k < 9; ++k) nd |= z[k] == ndv;
  } else if (P.nd_kind == VSR_NODATA_NAN) {
#pragma unroll
    for (int k = 0; k < 9; ++k) nd |= z[k] != z[k];
  }
  WindowUnit unit{};
  if constexpr (std::is_same<C, float>::value) {
    // one size of integers per warp: what 32 bits hold, 64 hold as well
    unit = window_unit(z);
    if (nd) unit.size = kUnit32;
    if (__any_sync(0xffffffffu, unit.size == kUnit64) && unit.size == kUnit32) unit.size = kUnit64;
  }
  if (x >= P.W || y >= P.H) return;
  if (nd) {
    if (P.tri) store_out(P.tri, P.out_dtype, o, P.nd_out);
    if (P.tpi) store_out(P.tpi, P.out_dtype, o, P.nd_out);
    if (P.curv) store_out(P.curv, P.out_dtype, o, P.nd_out);
    return;
  }
  if constexpr (std::is_same<C, double>::value) {
    if (P.tri) store_out(P.tri, P.out_dtype, o, plain_tri(z));
    if (P.tpi) store_out(P.tpi, P.out_dtype, o, plain_tpi(z));
    if (P.curv) store_out(P.curv, P.out_dtype, o, plain_curv(z, P));
  } else if constexpr (std::is_same<C, float>::value) {
    deriv_pixel(z, unit, o, P);
  } else {
    deriv_ints(z, 0, o, P);
  }
}

template <typename T>
int launch_deriv(const void* src, const DerivParams& P, int bands, cudaStream_t st) {
  const dim3 grid(static_cast<unsigned>((P.W + kDTW - 1) / kDTW), static_cast<unsigned>((P.H + kDTH - 1) / kDTH),
                  static_cast<unsigned>(bands));
  if (grid.y > 65535u) return fail(VSR_ERR_UNSUPPORTED, "raster too tall for the terrain-derivative grid");
  terrain_deriv_kernel<T><<<grid, dim3(kDTW, kDTH), 0, st>>>(static_cast<const T*>(src), P);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

}  // namespace
}  // namespace vsr

using namespace vsr;

extern "C" int vsr_terrain_derivatives_bands(const void* dem, int dtype, int bands, int64_t band_stride,
                                             int64_t height, int64_t width, int64_t pitch, double cell_x,
                                             double cell_y, double nodata, int nodata_kind, double nodata_out,
                                             void* tri, void* tpi, void* curvature, int out_dtype,
                                             int64_t out_band_stride, int64_t out_pitch, void* stream) {
  if (height < 0 || width < 0) return fail(VSR_ERR_INVALID_ARG, "negative raster size");
  if (bands < 1 || bands > 65535) return fail(VSR_ERR_INVALID_ARG, "bands must be in [1, 65535]");
  if (height == 0 || width == 0 || (!tri && !tpi && !curvature)) return VSR_OK;
  if (!dem) return fail(VSR_ERR_INVALID_ARG, "dem is NULL");
  const size_t es = dtype_size(dtype);
  if (es == 0) return fail(VSR_ERR_INVALID_ARG, "unsupported dtype %d", dtype);
  if (pitch < width) return fail(VSR_ERR_INVALID_ARG, "pitch %lld < width %lld", (long long)pitch, (long long)width);
  if (out_dtype != VSR_F32 && out_dtype != VSR_F64) return fail(VSR_ERR_INVALID_ARG, "out_dtype must be VSR_F32 or VSR_F64");
  if (out_pitch < width) return fail(VSR_ERR_INVALID_ARG, "out_pitch < width");
  if (bands > 1 && (band_stride < pitch * height || out_band_stride < out_pitch * height))
    return fail(VSR_ERR_INVALID_ARG, "band strides smaller than one band");
  if (!(cell_x > 0.0) || !(cell_y > 0.0) || !std::isfinite(cell_x) || !std::isfinite(cell_y))
    return fail(VSR_ERR_INVALID_ARG, "cell sizes must be positive and finite");
  if (nodata_kind < VSR_NODATA_NONE || nodata_kind > VSR_NODATA_NAN)
    return fail(VSR_ERR_INVALID_ARG, "bad nodata_kind %d", nodata_kind);
  if (!aligned(dem, es)) return fail(VSR_ERR_INVALID_ARG, "dem not aligned to its element size");
  const size_t os = out_dtype == VSR_F64 ? 8 : 4;
  for (void* p : {tri, tpi, curvature})
    if (p && !aligned(p, os)) return fail(VSR_ERR_INVALID_ARG, "outputs not aligned to the output element size");
  DerivParams P{};
  P.H = height;
  P.W = width;
  P.pitch = pitch;
  P.out_pitch = out_pitch;
  P.band_stride = bands > 1 ? band_stride : 0;
  P.out_band_stride = bands > 1 ? out_band_stride : 0;
  P.nd_kind = resolve_nodata(dtype, nodata, nodata_kind, &P.nd_in);
  P.nd_out = nodata_out;
  P.cx2 = cell_x * cell_x;
  P.cy2 = cell_y * cell_y;
  const double icx2 = 1.0 / P.cx2, icy2 = 1.0 / P.cy2;
  P.icx2_hi = static_cast<float>(icx2);
  P.icx2_lo = static_cast<float>(icx2 - static_cast<double>(P.icx2_hi));
  P.icy2_hi = static_cast<float>(icy2);
  P.icy2_lo = static_cast<float>(icy2 - static_cast<double>(P.icy2_hi));
  P.tri = tri;
  P.tpi = tpi;
  P.curv = curvature;
  P.out_dtype = out_dtype;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  P.kx = 100.0 / P.cx2;
  P.ky = 100.0 / P.cy2;
  P.ck = vsr_curv_factors(P.cx2, P.cy2);
  const int rc = run_terrain_strip(dem, dtype, P, bands, st);
  if (rc >= 0) return rc;
  switch (dtype) {
    case VSR_U8: return launch_deriv<uint8_t>(dem, P, bands, st);
    case VSR_I16: return launch_deriv<int16_t>(dem, P, bands, st);
    case VSR_U16: return launch_deriv<uint16_t>(dem, P, bands, st);
    case VSR_I32: return launch_deriv<int32_t>(dem, P, bands, st);
    case VSR_F32: return launch_deriv<float>(dem, P, bands, st);
    default: return launch_deriv<double>(dem, P, bands, st);
  }
}

extern "C" int vsr_terrain_derivatives(const void* dem, int dtype, int64_t height, int64_t width, int64_t pitch,
                                       double cell_x, double cell_y, double nodata, int nodata_kind,
                                       double nodata_out, void* tri, void* tpi, void* curvature, int out_dtype,
                                       int64_t out_pitch, void* stream) {
  return vsr_terrain_derivatives_bands(dem, dtype, 1, 0, height, width, pitch, cell_x, cell_y, nodata, nodata_kind,
                                       nodata_out, tri, tpi, curvature, out_dtype, 0, out_pitch, stream);
}
