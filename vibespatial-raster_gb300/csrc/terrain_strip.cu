// Terrain derivatives (TRI, TPI, profile curvature) of 8/16-bit and float32
// DEMs on integers: one pass, any subset of the outputs.
//
// Semantics and formulas: terrain.cu.  Elevations that lie within four
// binades of each other (five if none is negative) are integers below 2^27
// (2^28) in one unit; TRI and TPI are then exact integers (the reference's
// float64 results bit for bit) and the curvature is a fixed-point product
// (terrain_fixed.h), or two FP64 products where its factors are far apart.
//
// A warp walks down 126 columns (128 with the halo), column 32 j + lane in a
// lane's place j, so that every store instruction writes 256 contiguous bytes
// whatever the rows' alignment.  Rows arrive through shared memory
// (warp_strip.cuh); the lane keeps the integers of the last three rows'
// windows in registers.  The warp checks each row against the current unit
// with one vote and, when it does not fit, picks a unit for the last three
// rows.  Output rows whose three rows share none (values through zero, several
// binades of relief) are formed in 64-bit integers of up to 35 binades, TRI and
// TPI rounded once, the curvature from its exact sums in FP64; rows with more
// binades, infinities or NaN pixel by pixel (terrain_px.cuh).
//
// One conversion to float64 per TRI and TPI runs on the narrow FP64 pipe beside
// the integer work; with the curvature's conversions there too, that pipe would
// be the bound.  Bound by instruction issue (4096 x 4097, 121 us: 186
// instructions per pixel, 68 % of the issue slots, ALU pipe 57 %, FP64 48 %, DRAM
// 43 %, 14 warps per SM).  9001 x 7201 with three float64 outputs:
// 0 .. 4500 m 442 us, -500 .. 500 m (a quarter of the pixels in 64-bit rows)
// 647; 4096 x 4097 white noise (all of them) 300; one pixel per thread in
// double-float 1052, 1078 and 320.
#include "terrain_px.cuh"
#include "warp_strip.cuh"

namespace vsr {
namespace {

constexpr int kTsCols = 126;
constexpr int kTsDepth = 6;  // rows in shared memory
// Blocks per SM (strips of 8 rows) from which the strips are used; with fewer,
// one pixel per thread (terrain.cu) is faster.  us, pixels | strips: float32 of
// 1000 .. 1500 m 300^2 6.2 | 15, 1024^2 16.6 | 18.5, 1230^2 22.8 | 20.6; int16
// 725^2 8.3 | 14.6, 1230^2 16.8 | 18.6, 1449^2 22.7 | 20.7; float32 through zero
// 1024^2 21 | 31, 1449^2 35 | 43, 2048^2 68 | 65.
constexpr int kTsFew = 10;

// A pixel whose row triple does not share a unit.
__device__ __forceinline__ void lone_pixel(const float* __restrict__ src, const DerivParams& P, int64_t x, int64_t y) {
  float z[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const int64_t gy = min(max(y + k / 3 - 1, int64_t(0)), P.H - 1), gx = min(max(x + k % 3 - 1, int64_t(0)), P.W - 1);
    z[k] = __ldg(src + gy * P.pitch + gx);
  }
  deriv_pixel(z, window_unit(z), static_cast<int64_t>(blockIdx.z) * P.out_band_stride + y * P.out_pitch + x, P);
}

// An output row whose three rows share no 32-bit unit.  Where they share a
// 64-bit one, ``e`` is its lowest exponent (values through zero, several
// binades of relief); otherwise every pixel looks for a unit of its own.  Out of
// line, as the 32-bit rows' loop is near the instruction cache's size.
struct Row3 {
  float t[4], m[4], b[4];
};
constexpr int kTsWide = 128 + 8;  // a row's 64-bit integers, from element 4
__device__ __noinline__ void odd_row(const Row3 r, uint32_t e, long long* __restrict__ buf, uint32_t writes,
                                     const float* __restrict__ src, int64_t xw, int64_t y, const DerivParams& P) {
  const int lane = threadIdx.x;
  if (!e) {
#pragma unroll 1
    for (int j = 0; j < 4; ++j)
      if (writes >> j & 1u) lone_pixel(src, P, xw + 32 * j + lane, y);
    return;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    buf[4 + 32 * j + lane] = wide_int(r.t[j], e);
    buf[kTsWide + 4 + 32 * j + lane] = wide_int(r.m[j], e);
    buf[2 * kTsWide + 4 + 32 * j + lane] = wide_int(r.b[j], e);
  }
  __syncwarp();
  const int64_t o = static_cast<int64_t>(blockIdx.z) * P.out_band_stride + y * P.out_pitch + xw + lane;
#pragma unroll 2
  for (int j = 0; j < 4; ++j) {
    long long n[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) n[k] = buf[k / 3 * kTsWide + 3 + 32 * j + lane + k % 3];
    if (writes >> j & 1u) deriv_ints(n, static_cast<int>(e) - 150, o + 32 * j, P);
  }
  __syncwarp();
}

// CK: the curvature factors have an integer form.
template <typename T, typename B, bool CK>
__global__ void __launch_bounds__(32) terrain_strip(const T* __restrict__ src, const __grid_constant__ DerivParams P,
                                                    const int strip) {
  constexpr bool kFloat = std::is_same<T, float>::value;
  __shared__ __align__(16) unsigned char ring[16 + RowRing<T, kTsDepth>::kBytes + 16];
  __shared__ int32_t nrow[128 + 8];  // a float row's integers, from element 4
  __shared__ long long wide[kFloat ? 3 * kTsWide : 1];  // three rows' in 64 bits, where 32 do not hold them
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
  uint32_t signs = 0x7fffffffu, span = kTdSpan;  // all ones: negative values do not fit
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
    uint32_t ew = 0;  // the 64-bit unit's lowest exponent, or 0
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
        // a unit for the last three rows (infinities and NaNs fail)
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
        span = signs == 0xffffffffu ? kTdSpanPos : kTdSpan;
        hi = __reduce_max_sync(0xffffffffu, hi);
        lo = __reduce_min_sync(0xffffffffu, lo);
        const uint32_t el = hi ? lo >> 23 : 127u, eh = hi ? hi >> 23 : 127u;  // zeros only: any unit
        const bool normal = el >= kTdExpMin && eh <= kTdExpMax;
        shared = normal && eh - el < span;
        ew = normal && !shared && eh - el < kTdSpanWide ? el : 0u;
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
      if (shared) {
        const int u = kFloat ? static_cast<int>(e0) - 150 : 0;
        const uint32_t e20 = static_cast<uint32_t>(u - 3) << 20;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int32_t c = mc[j];
          const bool w = writes >> j & 1u;
          if (tri) {
            const B b = out_bits<B>(scaled_bits(tri8_of(tl[j], tc[j], tr[j], ml[j], c, mr[j], bl[j], bc[j], br[j]), e20));
            if (w) tri[32 * j] = b;
          }
          if (tpi) {
            const B b = out_bits<B>(scaled_bits(tpi8_of(tl[j], tc[j], tr[j], ml[j], c, mr[j], bl[j], bc[j], br[j]), e20));
            if (w) tpi[32 * j] = b;
          }
          if (curv) {
            const int32_t ca = ml[j] + mr[j] - 2 * c, cb = tc[j] + bc[j] - 2 * c;
            const B b = out_bits<B>(CK ? vsr_curv_bits(ca, cb, &P.ck, u) : curv_bits_f64(ca, cb, u, P));
            if (w) curv[32 * j] = b;
          }
        }
      } else if constexpr (kFloat) {
        odd_row(Row3{{vt[0], vt[1], vt[2], vt[3]}, {vm[0], vm[1], vm[2], vm[3]}, {v[0], v[1], v[2], v[3]}}, ew, wide,
                writes, src, xw, y, P);
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
  if (gx * ((P.H + 7) / 8) * bands < kTsFew * static_cast<int64_t>(sm_count())) return -1;
  int strip = 64;
  while (strip > 8 && gx * ((P.H + strip - 1) / strip) * bands < 32 * static_cast<int64_t>(sm_count())) strip /= 2;
  const int64_t gy = (P.H + strip - 1) / strip;
  if ((P.H + 7) / 8 > 65535 || gy > 65535)
    return fail(VSR_ERR_UNSUPPORTED, "raster too tall for the terrain-derivative grid");
  const dim3 grid(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(bands));
  const T* src = static_cast<const T*>(dem);
  const bool f64 = P.out_dtype == VSR_F64;
  if (f64 && P.ck.ok) terrain_strip<T, unsigned long long, true><<<grid, 32, 0, st>>>(src, P, strip);
  else if (f64) terrain_strip<T, unsigned long long, false><<<grid, 32, 0, st>>>(src, P, strip);
  else if (P.ck.ok) terrain_strip<T, unsigned int, true><<<grid, 32, 0, st>>>(src, P, strip);
  else terrain_strip<T, unsigned int, false><<<grid, 32, 0, st>>>(src, P, strip);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

}  // namespace

int run_terrain_strip(const void* dem, int dtype, const DerivParams& P, int bands, cudaStream_t st) {
  switch (dtype) {
    case VSR_U8: return launch_ts<uint8_t>(dem, P, bands, st);
    case VSR_I16: return launch_ts<int16_t>(dem, P, bands, st);
    case VSR_U16: return launch_ts<uint16_t>(dem, P, bands, st);
    case VSR_F32: return launch_ts<float>(dem, P, bands, st);
    default: return -1;
  }
}

}  // namespace vsr
