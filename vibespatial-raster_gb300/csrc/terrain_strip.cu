// Terrain derivatives (TRI, TPI, profile curvature) of 8/16-bit and float32
// DEMs on integers: one pass, any subset of the outputs.
//
// Semantics and formulas: terrain.cu.  Elevations that lie within four
// binades of each other (five if none is negative) are integers below 2^27
// (2^28) in one unit; TRI and TPI are
// then exact integers (terrain_exact.h: the reference's float64 results bit for
// bit) and the curvature is a fixed-point product (terrain_fixed.h).
//
// A warp walks down 126 columns (128 with the halo), column 32 j + lane in a
// lane's place j, so that every store instruction writes 256 contiguous bytes
// whatever the rows' alignment.  Rows arrive through shared memory
// (warp_strip.cuh); the lane keeps the integers of the last three rows'
// windows in registers.  The warp checks each row against the current unit
// with one vote and, when it does not fit, picks a unit for the last three
// rows; output rows whose three rows share none (values near zero beside large ones,
// infinities, NaN) take the per-pixel double-float form (terrain_px.cuh).
//
// One conversion to float64 per TRI and TPI runs on the FP64 pipe (two
// operations per clock and SM) beside the integer work; with the curvature's
// conversions there too, that pipe would be the bound.  Bound by instruction
// issue (about 100 per pixel), close to HBM (28 B/px with three float64
// outputs).
#include "terrain_px.cuh"
#include "warp_strip.cuh"

namespace vsr {
namespace {

constexpr int kTsCols = 126;
constexpr int kTsDepth = 6;  // rows in shared memory
// Binades of a unit: |n| < 2^27, or 2^28 where no value is negative: either
// way differences stay below 2^28 and the sums of eight below 2^31.
constexpr uint32_t kTsSpan = 4, kTsSpanPos = 5;

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

// A pixel whose window does not fit one unit.
template <typename T>
__device__ __noinline__ void slow_pixel(const T* __restrict__ src, const DerivParams& P, int64_t x, int64_t y) {
  float z[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int64_t gy = min(max(y + k / 3 - 1, int64_t(0)), P.H - 1), gx = min(max(x + k % 3 - 1, int64_t(0)), P.W - 1);
    z[k] = static_cast<float>(__ldg(src + gy * P.pitch + gx));
  }
  deriv_pixel(z, static_cast<int64_t>(blockIdx.z) * P.out_band_stride + y * P.out_pitch + x, P);
}

template <typename T, typename B>
__global__ void __launch_bounds__(32) terrain_strip(const T* __restrict__ src, const __grid_constant__ DerivParams P,
                                                    const int strip) {
  constexpr bool kFloat = std::is_same<T, float>::value;
  __shared__ __align__(16) unsigned char ring[16 + RowRing<T, kTsDepth>::kBytes + 16];
  __shared__ int32_t nrow[128 + 8];  // a float row's integers, from element 4
  const int lane = threadIdx.x;
  src += static_cast<int64_t>(blockIdx.z) * P.band_stride;
  const int64_t xw = static_cast<int64_t>(blockIdx.x) * kTsCols - 1, ys = static_cast<int64_t>(blockIdx.y) * strip;
  const int nout = static_cast<int>(P.H - ys < strip ? P.H - ys : static_cast<int64_t>(strip));
  const int nin = nout + 2;  // input row i is raster row ys - 1 + i
  RowRing<T, kTsDepth> rows;
  rows.start(ring + 16, src + (ys - 1) * P.pitch + xw, P.pitch, xw, P.W, ys == 0 ? 1 : 0,
             static_cast<int>(P.H - (ys - 1) < nin ? P.H - (ys - 1) : static_cast<int64_t>(nin)), false);
  // place j holds column xw + 32 j + lane: bit j of ``writes`` / ``side``: the
  // warp's output column / a border column of the raster
  uint32_t writes = 0, side = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int p = 32 * j + lane;
    writes |= static_cast<uint32_t>(p >= 1 && p <= kTsCols && xw + p < P.W) << j;
    side |= static_cast<uint32_t>(xw + p == 0 || xw + p == P.W - 1) << j;
  }
  const bool edge = xw < 0 || xw + 128 >= P.W;  // the strip has a border column
  const bool nd_nan = P.nd_kind == VSR_NODATA_NAN, nd_any = P.nd_kind != VSR_NODATA_NONE;
  const T ndv = static_cast<T>(P.nd_in);
  // a float32 DEM's nodata value, or NaN (equal to nothing)
  const float ndq = P.nd_kind == VSR_NODATA_VALUE ? static_cast<float>(P.nd_in) : __int_as_float(0x7fffffff);
  const int64_t o0 = static_cast<int64_t>(blockIdx.z) * P.out_band_stride + ys * P.out_pitch + xw + lane;
  B* tri = P.tri ? static_cast<B*>(P.tri) + o0 : nullptr;
  B* tpi = P.tpi ? static_cast<B*>(P.tpi) + o0 : nullptr;
  B* curv = P.curv ? static_cast<B*>(P.curv) + o0 : nullptr;
  const B ndb = out_bits<B>(static_cast<uint64_t>(__double_as_longlong(P.nd_out)));

  // integers left of, at and right of the lane's columns, three rows
  int32_t tl[4], tc[4], tr[4], ml[4], mc[4], mr[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) tl[j] = tc[j] = tr[j] = ml[j] = mc[j] = mr[j] = 0;
  uint32_t dt[4] = {0, 0, 0, 0}, dm[4] = {0, 0, 0, 0};  // nodata at or beside a column, a bit per lane
  uint32_t e0 = 127;       // the unit: exponent of the lowest binade, 2^(e0 - 150)
  float scale = 8388608.0f;  // 2^(150 - e0)
  uint32_t signs = 0x7fffffffu, span = kTsSpan;  // all ones: negative values do not fit
  bool shared = !kFloat;     // the last three rows are in this unit
  float vt[4] = {0.0f, 0.0f, 0.0f, 0.0f}, vm[4] = {0.0f, 0.0f, 0.0f, 0.0f};  // their values
#pragma unroll 1
  for (int i = 0; i < nin; ++i) {
    const T* row = reinterpret_cast<const T*>(rows.advance()) - 3 * lane;  // element ``lane`` of the 128
    T v[4];
    bool nd[4], fits = true;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[j] = row[32 * j];
      if constexpr (kFloat) {
        nd[j] = (v[j] == ndq) | (nd_nan & (v[j] != v[j]));
        fits &= nd[j] | (v[j] == 0.0f) | ((__float_as_uint(v[j]) & signs) - (e0 << 23) < span << 23);
      } else {
        nd[j] = nd_any & (v[j] == ndv);
      }
    }
    int32_t bl[4], bc[4], br[4];
    if constexpr (kFloat) {
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = nd[j] ? 0.0f : v[j];
      // a row's integers, left and right neighbours through shared memory
      auto convert = [&](const float f[4], int32_t l[4], int32_t c[4], int32_t r[4]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          c[j] = __float2int_rn(f[j] * scale);
          nrow[4 + 32 * j + lane] = c[j];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          l[j] = nrow[3 + 32 * j + lane];
          r[j] = nrow[5 + 32 * j + lane];
        }
      };
      if (!__all_sync(0xffffffffu, fits) || !shared) {
        // a unit for the last three rows: 64 <= exponents <= 190 (scaled
        // results are normal, infinities and NaNs fail)
        uint32_t lo = 0xffffffffu, hi = 0u;
        bool neg = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float f3[3] = {v[j], vm[j], vt[j]};
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const uint32_t m = __float_as_uint(f3[q]) & 0x7fffffffu;
            lo = min(lo, m == 0u ? 0xffffffffu : m);
            hi = max(hi, m);
            neg = neg || f3[q] < 0.0f;
          }
        }
        signs = __any_sync(0xffffffffu, neg) ? 0x7fffffffu : 0xffffffffu;
        span = signs == 0xffffffffu ? kTsSpanPos : kTsSpan;
        hi = __reduce_max_sync(0xffffffffu, hi);
        lo = hi ? __reduce_min_sync(0xffffffffu, lo) : 0x3f800000u;  // zeros only: any unit
        hi = hi ? hi : lo;
        const uint32_t el = lo >> 23, eh = hi >> 23;
        shared = el >= 64u && eh <= 190u && eh - el < span;
        if (shared) {
          e0 = el - (span - 1 - (eh - el)) / 2;
          scale = __uint_as_float((277u - e0) << 23);
          convert(vt, tl, tc, tr);
          __syncwarp();
          convert(vm, ml, mc, mr);
          __syncwarp();
        }
      }
      convert(v, bl, bc, br);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        bc[j] = v[j];
        bl[j] = row[32 * j - 1];
        br[j] = row[32 * j + 1];
      }
    }
    uint32_t db[4] = {0, 0, 0, 0};
    if (nd_any) {
      uint32_t b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = __ballot_sync(0xffffffffu, nd[j]);
      if (b[0] | b[1] | b[2] | b[3]) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          db[j] = b[j] | (b[j] << 1) | (b[j] >> 1);
          if (j > 0) db[j] |= b[j - 1] >> 31;
          if (j < 3) db[j] |= b[j + 1] << 31;
        }
      }
    }
    if (i >= 2) {
      const int64_t y = ys + i - 2;
      if (shared && P.ck.ok) {
        const int u = kFloat ? static_cast<int>(e0) - 150 : 0;
        const uint32_t e20 = static_cast<uint32_t>(u - 3) << 20;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int32_t c = mc[j];
          const bool w = writes >> j & 1u;
          if (tri) {
            const int32_t s = (abs(tl[j] - c) + abs(tc[j] - c)) + (abs(tr[j] - c) + abs(ml[j] - c)) +
                              (abs(mr[j] - c) + abs(bl[j] - c)) + (abs(bc[j] - c) + abs(br[j] - c));
            const B b = out_bits<B>(scaled_bits(s, e20));
            if (w) tri[32 * j] = b;
          }
          if (tpi) {
            const int32_t s = 8 * c - ((tl[j] + tc[j] + tr[j]) + (ml[j] + mr[j]) + (bl[j] + bc[j] + br[j]));
            const B b = out_bits<B>(scaled_bits(s, e20));
            if (w) tpi[32 * j] = b;
          }
          if (curv) {
            const B b = out_bits<B>(vsr_curv_bits(ml[j] + mr[j] - 2 * c, tc[j] + bc[j] - 2 * c, &P.ck, u));
            if (w) curv[32 * j] = b;
          }
        }
      } else {
#pragma unroll 1
        for (int j = 0; j < 4; ++j)
          if (writes >> j & 1u) slow_pixel<T>(src, P, xw + 32 * j + lane, y);
      }
      // borders and windows that touch nodata, over what was just written
      const bool border = y == 0 || y == P.H - 1;
      uint32_t any = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) any |= dt[j] | dm[j] | db[j];
      if (any || border || edge) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool f = border || (side >> j & 1u) || ((dt[j] | dm[j] | db[j]) >> lane & 1u);
          if (f && (writes >> j & 1u)) {
            if (tri) tri[32 * j] = ndb;
            if (tpi) tpi[32 * j] = ndb;
            if (curv) curv[32 * j] = ndb;
          }
        }
      }
      if (tri) tri += P.out_pitch;
      if (tpi) tpi += P.out_pitch;
      if (curv) curv += P.out_pitch;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      tl[j] = ml[j];
      tc[j] = mc[j];
      tr[j] = mr[j];
      ml[j] = bl[j];
      mc[j] = bc[j];
      mr[j] = br[j];
      dt[j] = dm[j];
      dm[j] = db[j];
      if constexpr (kFloat) {
        vt[j] = vm[j];
        vm[j] = v[j];
      }
    }
  }
}

template <typename T>
int launch_ts(const void* dem, const DerivParams& P, int bands, cudaStream_t st) {
  const int64_t gx = (P.W + kTsCols - 1) / kTsCols;
  int strip = 64;
  while (strip > 8 && gx * ((P.H + strip - 1) / strip) * bands < 32 * static_cast<int64_t>(sm_count())) strip /= 2;
  const int64_t gy = (P.H + strip - 1) / strip;
  if ((P.H + 7) / 8 > 65535 || gy > 65535)
    return fail(VSR_ERR_UNSUPPORTED, "raster too tall for the terrain-derivative grid");
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(bands));
  if (P.out_dtype == VSR_F64)
    terrain_strip<T, unsigned long long><<<grid, 32, 0, st>>>(static_cast<const T*>(dem), P, strip);
  else terrain_strip<T, unsigned int><<<grid, 32, 0, st>>>(static_cast<const T*>(dem), P, strip);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

}  // namespace

int run_terrain_strip(const void* dem, int dtype, const DerivParams& P, int bands, cudaStream_t st) {
  switch (dtype) {
    case VSR_U8: return launch_ts<uint8_t>(dem, P, bands, st);
    case VSR_I16: return launch_ts<int16_t>(dem, P, bands, st);
    case VSR_U16: return launch_ts<uint16_t>(dem, P, bands, st);
    default: return launch_ts<float>(dem, P, bands, st);
  }
}

}  // namespace vsr
