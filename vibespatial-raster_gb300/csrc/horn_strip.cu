// Slope, aspect and hillshade of 8/16-bit DEMs and of float32 DEMs whose rows
// the TMA kernel cannot take (horn_tma.cuh: 16-byte alignment).
//
// A warp walks down 126 columns (128 with the halo), column 32 j + lane in a
// lane's place j, so that every store instruction writes 32 adjacent outputs
// whatever the rows' alignment; rows arrive through shared memory
// (warp_strip.cuh) and the last three rows' windows stay in registers.  The
// arithmetic is horn_common.cuh's, two pixels per packed instruction: the
// generic (scalar) kernel's results bit for bit, and the TMA kernel's.  float64
// outputs are the float results widened by integer operations (a conversion
// would occupy the narrow FP64 pipe).
//
// Bound by instruction issue (int16 3601^2 with float64 outputs, 98 us: 68 % of
// the issue slots, DRAM 24 %, 14 warps per SM).
#include <type_traits>

#include "horn_common.cuh"
#include "warp_strip.cuh"

namespace vsr {
namespace horn {
namespace {

constexpr int kHsCols = 126;
constexpr int kHsDepth = 6;  // rows in shared memory
// Blocks per SM (strips of 8 rows) from which the strips are used.  With fewer,
// a block's 10 rows one after the other take longer than one pixel per thread
// (horn.cu).  us, pixels | strips: slope of int16 300^2 4.2 | 10.5, 1024^2 10.4
// | 12.4, 1230^2 14.4 | 12.9; all three of int16 725^2 8.3 | 14.5, 1230^2 16.5 |
// 17.3, 2048^2 39 | 36; float32 odd rows 300^2 4.2 | 10.6, 850^2 12.4 | 12.4,
// 1024^2 16.4 | 12.4.
template <typename T>
constexpr int kHsFew = sizeof(T) < 4 ? 8 : 6;

// The values at and beside a lane's 4 columns in one row, and the row's nodata.
struct HsRow {
  float l[4], c[4], r[4];
  uint32_t nd[4], dil[4];  // nodata at / at or beside a column, a bit per lane
};

template <typename T, typename O>
__global__ void __launch_bounds__(32) horn_strip(const T* __restrict__ src, const __grid_constant__ HornParams P,
                                                 const T ndv, const int strip, O* __restrict__ slope,
                                                 O* __restrict__ aspect, uint8_t* __restrict__ hs) {
  constexpr bool kFloat = std::is_same<T, float>::value;
  using B = std::conditional_t<sizeof(O) == 8, unsigned long long, unsigned int>;
  __shared__ __align__(16) unsigned char ring[16 + RowRing<T, kHsDepth>::kBytes + 16];
  const int lane = threadIdx.x;
  src += static_cast<int64_t>(blockIdx.z) * P.in_band_stride;
  const int64_t xw = static_cast<int64_t>(blockIdx.x) * kHsCols - 1, ys = static_cast<int64_t>(blockIdx.y) * strip;
  const int nout = static_cast<int>(P.height - ys < strip ? P.height - ys : static_cast<int64_t>(strip));
  const int nin = nout + 2;  // input row i is raster row ys - 1 + i
  const int r0 = ys == 0 ? 1 : 0, r1 = P.height - (ys - 1) < nin ? static_cast<int>(P.height - (ys - 1)) : nin;
  RowRing<T, kHsDepth> rows;
  rows.start(ring + 16, src + (ys - 1) * P.in_pitch + xw, P.in_pitch, xw, P.width, r0, r1, false);
  bool writes[4], first[4], last[4];  // an output column of the warp; the raster's first / last column
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int p = 32 * j + lane;
    writes[j] = p >= 1 && p <= kHsCols && xw + p < P.width;
    first[j] = xw + p == 0;
    last[j] = xw + p == P.width - 1;
  }
  const bool edge = xw < 0 || xw + 128 >= P.width;
  const MaskRule rule = mask_rule(P);
  // every output of a window that holds nodata is masked
  const bool skip_nd = (!slope && !aspect) || (rule.sa_any && !rule.sa_center);
  const bool nd_nan = P.nd_kind == VSR_NODATA_NAN, nd_val = P.nd_kind == VSR_NODATA_VALUE;
  const int64_t o0 = static_cast<int64_t>(blockIdx.z) * P.out_band_stride + ys * P.out_pitch + xw + lane;
  B* sp = slope ? reinterpret_cast<B*>(slope) + o0 : nullptr;
  B* ap = aspect ? reinterpret_cast<B*>(aspect) + o0 : nullptr;
  uint8_t* hp = hs ? hs + static_cast<int64_t>(blockIdx.z) * P.hs_band_stride + ys * P.hs_pitch + xw + lane : nullptr;
  B ndb;
  if constexpr (sizeof(B) == 8) ndb = static_cast<B>(__double_as_longlong(P.nd_out_d));
  else ndb = __float_as_uint(P.nd_out_f);

  HsRow t{}, m{}, b{};
#pragma unroll 1
  for (int i = 0; i < nin; ++i) {
    const T* row = reinterpret_cast<const T*>(rows.advance()) - 3 * lane;  // element ``lane`` of the 128
    if (i < r1) {
      bool nd[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const T c = row[32 * j];
        nd[j] = (nd_val & (c == ndv)) | (kFloat & nd_nan & (c != c));
        b.c[j] = static_cast<float>(c);
        b.l[j] = static_cast<float>(row[32 * j - 1]);
        b.r[j] = static_cast<float>(row[32 * j + 1]);
      }
      if (edge) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          b.l[j] = first[j] ? b.c[j] : b.l[j];
          b.r[j] = last[j] ? b.c[j] : b.r[j];
        }
      }
      if (rule.hs_any) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // (places outside the raster hold zeros: no nodata)
          const bool in = xw + 32 * j + lane >= 0 && xw + 32 * j + lane < P.width;
          b.nd[j] = __ballot_sync(0xffffffffu, nd[j] && in);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          b.dil[j] = b.nd[j] | (b.nd[j] << 1) | (b.nd[j] >> 1);
          if (j > 0) b.dil[j] |= b.nd[j - 1] >> 31;
          if (j < 3) b.dil[j] |= b.nd[j + 1] << 31;
        }
      }
    } else {
      b = m;  // below the last row: its copy
    }
    if (i == 1 && ys == 0) m = b;  // above the first row: its copy
    if (i >= 2) {
      uint32_t any = 0, dil[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        dil[j] = t.dil[j] | m.dil[j] | b.dil[j];
        any |= dil[j];
      }
      float gx[4], gy[4];
      bool plain = true;
      if constexpr (kFloat) {  // differences of values within a factor of two are exact
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float lo = min3f(min3f(t.l[j], t.c[j], t.r[j]), min3f(m.l[j], m.c[j], m.r[j]), min3f(b.l[j], b.c[j], b.r[j]));
          const float hi = max3f(max3f(t.l[j], t.c[j], t.r[j]), max3f(m.l[j], m.c[j], m.r[j]), max3f(b.l[j], b.c[j], b.r[j]));
          const bool masked = skip_nd & (dil[j] >> lane & 1u);
          plain &= masked | ((lo > 0.0f) & (hi <= 2.0f * lo)) | ((hi < 0.0f) & (lo >= 2.0f * hi)) |
                   ((lo == 0.0f) & (hi == 0.0f)) | !writes[j];
        }
        plain = __all_sync(0xffffffffu, plain);
      }
      if (plain) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          gx[j] = fmaf(2.0f, m.r[j] - m.l[j], (t.r[j] - t.l[j]) + (b.r[j] - b.l[j]));
          gy[j] = fmaf(2.0f, b.c[j] - t.c[j], (b.l[j] - t.l[j]) + (b.r[j] - t.r[j]));
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          gx[j] = grad_exact(t.l[j], t.r[j], m.l[j], m.r[j], b.l[j], b.r[j]);
          gy[j] = grad_exact(t.l[j], b.l[j], t.c[j], b.c[j], t.r[j], b.r[j]);
        }
      }
      float so[4], ao[4];
      uint32_t ho[4];
#pragma unroll
      for (int k = 0; k < 4; k += 2) {
        const float2 p = mul2(make_float2(gx[k], gx[k + 1]), f2(P.inv8cx));
        const float2 q = mul2(make_float2(gy[k], gy[k + 1]), f2(P.inv8cy));
        const float2 s = fma2(p, p, mul2(q, q));
        if (slope) {
          const float2 v = slope_deg2(s);
          so[k] = v.x;
          so[k + 1] = v.y;
        }
        if (aspect) {
          const float2 v = aspect_deg2(p, q);
          ao[k] = v.x;
          ao[k + 1] = v.y;
        }
        if (hs) hillshade_bits2(p, q, s, P, ho[k], ho[k + 1]);
      }
      auto put = [&](B* to, const float v[4]) {
        B w[4];
        if constexpr (sizeof(B) == 8) {
          uint64_t x[4];
          widen4(v, x);
#pragma unroll
          for (int j = 0; j < 4; ++j) w[j] = x[j];
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) w[j] = __float_as_uint(v[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (writes[j]) to[32 * j] = w[j];
      };
      if (slope) put(sp, so);
      if (aspect) put(ap, ao);
      if (hs) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (writes[j]) hp[32 * j] = static_cast<uint8_t>(ho[j]);
      }
      if (any) {  // nodata over what was just written
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool d = dil[j] >> lane & 1u, s = rule.sa_center ? m.nd[j] >> lane & 1u : d;
          if (slope && rule.sa_any && s && writes[j]) sp[32 * j] = ndb;
          if (aspect && rule.sa_any && s && writes[j]) ap[32 * j] = ndb;
          if (hs && d && writes[j]) hp[32 * j] = 0;
        }
      }
      if (slope) sp += P.out_pitch;
      if (aspect) ap += P.out_pitch;
      if (hs) hp += P.hs_pitch;
    }
    t = m;
    m = b;
  }
}

template <typename T, typename O>
int launch_hs(const void* src, const HornParams& P, double ndv, void* slope, void* aspect, uint8_t* hs,
              cudaStream_t st) {
  const int64_t gx = (P.width + kHsCols - 1) / kHsCols;
  if (gx * ((P.height + 7) / 8) * P.bands < kHsFew<T> * static_cast<int64_t>(sm_count())) return -1;
  int strip = 64;
  while (strip > 8 && gx * ((P.height + strip - 1) / strip) * P.bands < 32 * static_cast<int64_t>(sm_count())) strip /= 2;
  const int64_t gy = (P.height + strip - 1) / strip;
  if ((P.height + 7) / 8 > 65535 || gy > 65535)
    return fail(VSR_ERR_UNSUPPORTED, "raster height %lld too large for the generic Horn path", (long long)P.height);
  horn_strip<T, O><<<dim3(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(P.bands)), 32, 0,
                     st>>>(static_cast<const T*>(src), P, static_cast<T>(ndv), strip, static_cast<O*>(slope),
                           static_cast<O*>(aspect), hs);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

}  // namespace

// -1: not a DEM this kernel takes, or too few strips.
int run_horn_strip(int dtype, const void* src, const HornParams& P, double ndv, void* slope, void* aspect, bool f64,
                   uint8_t* hs, cudaStream_t st) {
  switch (dtype) {
    case VSR_U8:
      return f64 ? launch_hs<uint8_t, double>(src, P, ndv, slope, aspect, hs, st)
                 : launch_hs<uint8_t, float>(src, P, ndv, slope, aspect, hs, st);
    case VSR_I16:
      return f64 ? launch_hs<int16_t, double>(src, P, ndv, slope, aspect, hs, st)
                 : launch_hs<int16_t, float>(src, P, ndv, slope, aspect, hs, st);
    case VSR_U16:
      return f64 ? launch_hs<uint16_t, double>(src, P, ndv, slope, aspect, hs, st)
                 : launch_hs<uint16_t, float>(src, P, ndv, slope, aspect, hs, st);
    case VSR_F32:
      return f64 ? launch_hs<float, double>(src, P, ndv, slope, aspect, hs, st)
                 : launch_hs<float, float>(src, P, ndv, slope, aspect, hs, st);
    default: return -1;
  }
}

}  // namespace horn
}  // namespace vsr
