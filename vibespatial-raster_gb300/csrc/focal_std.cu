// Focal standard deviation with exact integer sums: 8/16-bit and float32
// rasters, square windows of radius 1..7.
//
// The reference takes two float64 passes over every window (algebra.py:
// 3104-3122).  The FP64 pipe of a GB300's SM is narrow, so that form is bound by 150 FP64 operations per pixel at 7 x 7.  Here the
// values of a warp's strip are written as integers in one unit (the unit of
// the strip's smallest non-zero magnitude), so that sum x and sum x^2 are
// exact, slide down the rows without drift, and n^2 var = n sum x^2 -
// (sum x)^2 has no rounding; sqrt(n^2 var) / n comes from integer arithmetic
// within 0.52 ulp (std_round64.h; a float32 output of an 8/16-bit raster is
// rounded once, std_round.h).
//
// Integers fit one 32-bit word when the strip's range spans less than
// 2^32 / n units (most DEM strips: n = 49 and values above 64 m allow 670 m
// of relief), two limbs of 25 (R <= 3), 24 or 23 bits when its exponents span
// at most 26, 24 or 22 binades (limb sums stay below 2^31, products' below
// 2^60).  Other strips (wider spans, infinities, values below 2^-103) keep the
// two float64 passes.
//
// Layout: warp strips (warp_strip.cuh).  Per input row a lane adds the
// entering and subtracts the leaving row of its 4 columns (the last 2R+1 rows
// of integers wait in shared memory, each thread reading only its own), takes
// the column sums of its neighbours by shuffles and adds up the window.
//
// Bound by instruction issue and the latency of its chains (7 x 7 of float32
// 4096^2: 61 % of the issue slots, ALU pipe 58 %, 14 warps per SM; about 200
// instructions per pixel, half of them the square root and division).  7 x 7 on
// 4096^2: float32 151 us (8370 us with the two float64 passes), uint16 128 us and
// 205 us with a float32 output (404 and 586 us in 256-row strips of 128 threads
// with an FP64 root).
#include <cstring>

#include "focal_stats.cuh"
#include "std_round.h"
#include "warp_strip.cuh"

namespace vsr {
namespace {

constexpr int kSdThreads = 32;  // one warp per block: blocks of unequal strips (one word, two limbs) balance best
constexpr int kSdMaxR = 7;  // windows of at most kRecipTaps: a count fits a byte
static_assert((2 * kSdMaxR + 1) * (2 * kSdMaxR + 1) <= kRecipTaps, "reciprocal table");

// Strips of 16 rows per SM below which a raster counts as small: 8/16-bit ones
// take the shared-memory kernel (focal_stats.cu; uint16 7 x 7 at 300 x 301 8 us,
// 25 in strips), float32 ones strips of 8 rows (7 x 7 at 512^2 27 us, 45 in
// strips of 16).
constexpr int kSdFew = 2;

template <int R>
struct SdGeom {
  static constexpr int P = 2 * R + 1, kTaps = P * P;
  static constexpr int HL = (R + 3) / 4;         // lanes at each end that only supply columns
  static constexpr int kCols = 128 - 8 * HL;     // output columns per warp
  static constexpr int kWin = 4 * (2 * HL + 1);  // columns a lane sees
  // two-limb integers: kTaps limbs of kLB bits sum below 2^31
  static constexpr int kLB = R <= 3 ? 25 : (R <= 5 ? 24 : 23);
  static_assert(kTaps * ((1ll << kLB) - 1) < (1ll << 31), "limb sums overflow");
};

// Columns of the neighbours: w[4 HL + e] is this lane's element e.
template <int R, typename V>
__device__ __forceinline__ void gather(const V own[4], V w[SdGeom<R>::kWin]) {
  constexpr int HL = SdGeom<R>::HL;
#pragma unroll
  for (int e = 0; e < 4; ++e) w[4 * HL + e] = own[e];
#pragma unroll
  for (int h = 1; h <= HL; ++h)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (4 * h - e <= R) w[4 * (HL - h) + e] = __shfl_up_sync(0xffffffffu, own[e], h);
      if (4 * h + e - 3 <= R) w[4 * (HL + h) + e] = __shfl_down_sync(0xffffffffu, own[e], h);
    }
}

// Window sums of 4 adjacent columns.
template <int R, typename V>
__device__ __forceinline__ void window4(const V own[4], V out[4]) {
  constexpr int C0 = 4 * SdGeom<R>::HL;
  V w[SdGeom<R>::kWin];
  gather<R>(own, w);
  V s = w[C0 - R];
#pragma unroll
  for (int j = C0 - R + 1; j <= C0 + R; ++j) s += w[j];
  out[0] = s;
#pragma unroll
  for (int c = 1; c < 4; ++c) {
    s += w[C0 + c + R] - w[C0 + c - 1 - R];
    out[c] = s;
  }
}

// Window counts from the packed column counts (byte e: column e).
template <int R>
__device__ __forceinline__ void count4(uint32_t cw, uint32_t out[4]) {
  constexpr int HL = SdGeom<R>::HL;
  uint32_t w[2 * HL + 1];
  w[HL] = cw;
#pragma unroll
  for (int h = 1; h <= HL; ++h) {
    w[HL - h] = __shfl_up_sync(0xffffffffu, cw, h);
    w[HL + h] = __shfl_down_sync(0xffffffffu, cw, h);
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    uint32_t n = 0;
#pragma unroll
    for (int q = 0; q < 2 * HL + 1; ++q) {
      uint32_t m = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int d = 4 * (q - HL) + e - c;
        if (d >= -R && d <= R) m |= 1u << (8 * e);
      }
      if (m) n = __dp4a(w[q], m, n);
    }
    out[c] = n;
  }
}

template <typename T>
__device__ __forceinline__ T elem_of(uint32_t b) {
  if constexpr (std::is_same<T, float>::value) return __uint_as_float(b);
  else return static_cast<T>(b);
}

// The strip of one warp.
struct SdStrip {
  int64_t xw, ys;  // first column of lane 0, first output row
  int nout;
  int u;           // values are integers times 2^u
  bool inside;     // all 128 columns lie in the raster
  float ndq;       // float32 rasters: the nodata value, or NaN (equal to nothing)
  float s1, s2;    // float32 rasters: value * s1 = its integer; s2 = s1 2^-kLB
  int ref;         // subtracted from the integers (one word)
};

template <int R, typename T, int LIMBS, bool EDGE>
__device__ __forceinline__ void run_strip(const FsArgs& a, const SdStrip& S, bool vin, bool vout, int4* ring,
                                          uint32_t* flags, uint64_t* obuf) {
  using G = SdGeom<R>;
  constexpr int P = G::P;
  constexpr bool kFloat = std::is_same<T, float>::value;
  const int lane = threadIdx.x & 31, t = threadIdx.x;
  const bool has_nd = a.kind != VSR_NODATA_NONE, nd_nan = a.kind == VSR_NODATA_NAN;
  const T ndv = static_cast<T>(a.ndv);
  const int64_t xs = S.xw + 4 * lane;
  uint32_t inm = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) inm |= static_cast<uint32_t>(xs + e >= 0 && xs + e < a.W) << e;
  const T* src = static_cast<const T*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride;
  const T* lp = src + (S.ys - R) * a.pitch + xs;
  const int nin = S.nout + 2 * R;
  auto row_in = [&](int i) { return static_cast<uint64_t>(S.ys - R + i) < static_cast<uint64_t>(a.H); };
  ring += t;
  flags += t;
  for (int s = 0; s < P; ++s) {
#pragma unroll
    for (int l = 0; l < LIMBS; ++l) ring[(s * LIMBS + l) * kSdThreads] = make_int4(0, 0, 0, 0);
    flags[s * kSdThreads] = 0u;
  }
  int32_t sh[4] = {0, 0, 0, 0}, sl[4] = {0, 0, 0, 0};
  uint64_t qh[4] = {0, 0, 0, 0}, qm[4] = {0, 0, 0, 0}, ql[4] = {0, 0, 0, 0};
  uint32_t cw = 0;
  uint32_t nxt[4] = {0u, 0u, 0u, 0u};
  if (row_in(0)) strip_load4<T, EDGE>(lp, inm, vin, nxt);
  const int64_t xo = S.xw;
  constexpr int lo = 4 * G::HL;
  const int hi = static_cast<int>(a.W - xo < 128 - 4 * G::HL ? a.W - xo : static_cast<int64_t>(128 - 4 * G::HL));
  char* orow = static_cast<char*>(a.dst) +
               (static_cast<int64_t>(blockIdx.z) * a.out_band_stride + S.ys * a.out_pitch + xo) *
                   (a.out_dtype == VSR_F64 ? 8 : 4);
  int slot = 0, cslot = P - R;
#pragma unroll 1
  for (int i = 0; i < nin; ++i) {
    // integers of the entering row
    int32_t nh[4] = {0, 0, 0, 0}, nl[4] = {0, 0, 0, 0};
    uint32_t f = 0;  // byte e: 1 valid, 2 nodata
    if (row_in(i)) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const T v = elem_of<T>(nxt[e]);
        bool nd, ok;
        if constexpr (kFloat) {
          const bool eq = v == S.ndq;
          ok = !eq & (v == v);
          nd = nd_nan ? v != v : eq;
        } else {
          nd = has_nd & (v == ndv);
          ok = !nd;
        }
        if (EDGE) ok = ok & ((inm >> e) & 1u);  // nd outside the raster: never a centre that is written
        f |= ok ? 1u << (8 * e) : 0u;
        f |= nd ? 2u << (8 * e) : 0u;
        if constexpr (!kFloat) {
          nh[e] = ok ? static_cast<int32_t>(v) : 0;
        } else if constexpr (LIMBS == 1) {
          nh[e] = ok ? __float2int_rn(v * S.s1) - S.ref : 0;
        } else {
          // v = h 2^kLB + l (units), both of v's sign; the remainder is exact
          const float q = ok ? v * S.s2 : 0.0f;
          const float qt = truncf(q);
          nh[e] = __float2int_rz(qt);
          nl[e] = __float2int_rn((q - qt) * static_cast<float>(1 << G::kLB));
        }
      }
    }
    lp += a.pitch;
    if (i + 1 < nin && row_in(i + 1)) strip_load4<T, EDGE>(lp, inm, vin, nxt);
    const int4 oh = ring[(slot * LIMBS) * kSdThreads];
    ring[(slot * LIMBS) * kSdThreads] = make_int4(nh[0], nh[1], nh[2], nh[3]);
    const int32_t ph[4] = {oh.x, oh.y, oh.z, oh.w};
    const uint32_t fo = flags[slot * kSdThreads];
    flags[slot * kSdThreads] = f;
    cw += (f & 0x01010101u) - (fo & 0x01010101u);
    if constexpr (LIMBS == 1) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sh[e] += nh[e] - ph[e];
        qh[e] += static_cast<uint64_t>(static_cast<int64_t>(nh[e]) * nh[e]);
        qh[e] += static_cast<uint64_t>(static_cast<int64_t>(-ph[e]) * ph[e]);
      }
    } else {
      const int4 ol = ring[(slot * LIMBS + 1) * kSdThreads];
      ring[(slot * LIMBS + 1) * kSdThreads] = make_int4(nl[0], nl[1], nl[2], nl[3]);
      const int32_t pl[4] = {ol.x, ol.y, ol.z, ol.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sh[e] += nh[e] - ph[e];
        sl[e] += nl[e] - pl[e];
        qh[e] += static_cast<uint64_t>(static_cast<int64_t>(nh[e]) * nh[e]);
        qh[e] += static_cast<uint64_t>(static_cast<int64_t>(-ph[e]) * ph[e]);
        qm[e] += static_cast<uint64_t>(static_cast<int64_t>(nh[e]) * nl[e]);
        qm[e] += static_cast<uint64_t>(static_cast<int64_t>(-ph[e]) * pl[e]);
        ql[e] += static_cast<uint64_t>(static_cast<int64_t>(nl[e]) * nl[e]);
        ql[e] += static_cast<uint64_t>(static_cast<int64_t>(-pl[e]) * pl[e]);
      }
    }
    slot = slot + 1 == P ? 0 : slot + 1;
    if (i >= 2 * R) {
      uint32_t n4[4];
      int32_t wsh[4], wsl[4];
      uint64_t wqh[4], wqm[4], wql[4];
      count4<R>(cw, n4);
      window4<R>(sh, wsh);
      window4<R>(qh, wqh);
      if constexpr (LIMBS == 2) {
        window4<R>(sl, wsl);
        window4<R>(qm, wqm);
        window4<R>(ql, wql);
      }
      const uint32_t fc = flags[cslot * kSdThreads];  // the centre row i - R
      uint64_t o64[4];
      uint32_t o32[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint32_t n = n4[c];
        uint64_t bits = 0;
        if constexpr (LIMBS == 1) {
          const uint64_t N = n * wqh[c] - static_cast<uint64_t>(static_cast<int64_t>(wsh[c]) * wsh[c]);
          if (!kFloat && a.out_dtype == VSR_F32) {
            o32[c] = __float_as_uint(n == 0 ? 0.0f : (n < 128 ? vsr_std_f32_small(N, n) : vsr_std_f32(N, n)));
          } else if (N) {
            bits = vsr_s64_std(N, S.u, fs_recip(n), 31 - __clz(n));
          }
        } else {
          const int64_t s = (static_cast<int64_t>(wsh[c]) << G::kLB) + wsl[c];
          const __int128 q = (static_cast<__int128>(static_cast<int64_t>(wqh[c])) << (2 * G::kLB)) +
                             (static_cast<__int128>(static_cast<int64_t>(wqm[c])) << (G::kLB + 1)) +
                             static_cast<int64_t>(wql[c]);
          const unsigned __int128 N = static_cast<unsigned __int128>(q) * n -
                                      static_cast<unsigned __int128>(static_cast<__int128>(s) * s);
          const uint64_t Nh = static_cast<uint64_t>(N >> 64), Nl = static_cast<uint64_t>(N);
          if (Nh | Nl) bits = vsr_s64_std128(Nh, Nl, S.u, fs_recip(n), 31 - __clz(n));
        }
        const bool nd = (fc >> (8 * c)) & 2u;
        o64[c] = nd ? static_cast<uint64_t>(__double_as_longlong(a.nd_out)) : bits;
        if (a.out_dtype == VSR_F32) {
          if (kFloat) o32[c] = __float_as_uint(static_cast<float>(__longlong_as_double(static_cast<long long>(bits))));
          if (nd) o32[c] = __float_as_uint(static_cast<float>(a.nd_out));
        }
      }
      if (a.out_dtype == VSR_F64) strip_store4<uint64_t>(reinterpret_cast<uint64_t*>(orow), o64, lane, lo, hi, vout, obuf);
      else strip_store4<uint32_t>(reinterpret_cast<uint32_t*>(orow), o32, lane, lo, hi, vout,
                                  reinterpret_cast<uint32_t*>(obuf));
      orow += a.out_pitch * (a.out_dtype == VSR_F64 ? 8 : 4);
    }
    cslot = cslot + 1 == P ? 0 : cslot + 1;
  }
}

// Two float64 passes per window (strips whose values span too many binades
// for the integers, or hold infinities), two output rows at a time: the first
// pass adds up columns once per row, then 2R+1 columns per window; the second
// visits every tap.  Bound by the narrow FP64 pipe: 2 (2R+1)^2 + 2 (2R+1)
// operations a pixel (3 (2R+1)^2 with both passes over the taps).  11 x 11 of
// 3000 x 3001 values over 80 binades: 8.4 ms, 12.5 with both over the taps.
// ``col``, ``cnt``: 256 each, of the warp.
template <int R>
__device__ __noinline__ void slow_strip(const FsArgs& a, const SdStrip& S, double* __restrict__ col,
                                        int* __restrict__ cnt) {
  constexpr int kCols = SdGeom<R>::kCols, kHalo = 4 * SdGeom<R>::HL;
  const int lane = threadIdx.x & 31;
  const float* src = static_cast<const float*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride;
  const float ndq = S.ndq, ndv = static_cast<float>(a.ndv);  // (NaN values are invalid whatever the nodata value)
  for (int i = 0; i < S.nout; i += 2) {
    for (int c = lane; c < 256; c += 32) {
      const int64_t x = S.xw + (c & 127), y = S.ys + i + (c >> 7);
      double s = 0.0;
      int n = 0;
      if (x >= 0 && x < a.W && y < a.H) {
        const float* p = src + y * a.pitch + x;
#pragma unroll
        for (int dy = -R; dy <= R; ++dy) {
          const bool in = y + dy >= 0 && y + dy < a.H;
          const float f = in ? __ldg(p + dy * a.pitch) : __int_as_float(0x7fffffff);
          if ((f == f) & (f != ndq)) {
            s += static_cast<double>(f);
            ++n;
          }
        }
      }
      col[c] = s;
      cnt[c] = n;
    }
    __syncwarp();
    const int rows = S.nout - i < 2 ? 1 : 2;
    for (int p = lane; p < rows * kCols; p += 32) {
      const int r = p >= kCols, c = p - r * kCols + kHalo;
      const int64_t x = S.xw + c, y = S.ys + i + r;
      if (x >= a.W) continue;
      double sm = 0.0, m2 = 0.0;
      int n = 0;
#pragma unroll
      for (int d = -R; d <= R; ++d) {
        sm += col[128 * r + c + d];
        n += cnt[128 * r + c + d];
      }
      const float* const centre = src + y * a.pitch + x;
      if (n) {
        const double mean = sm / n;
        auto add = [&](float f) {
          if ((f == f) & (f != ndq)) {
            const double d = static_cast<double>(f) - mean;
            m2 = fma(d, d, m2);
          }
        };
        if (y >= R && y + R < a.H && x >= R && x + R < a.W) {
#pragma unroll
          for (int dy = -R; dy <= R; ++dy)
#pragma unroll
            for (int dx = -R; dx <= R; ++dx) add(__ldg(centre + dy * a.pitch + dx));
        } else {
          for (int dy = -R; dy <= R; ++dy)
            for (int dx = -R; dx <= R; ++dx)
              if (y + dy >= 0 && y + dy < a.H && x + dx >= 0 && x + dx < a.W) add(__ldg(centre + dy * a.pitch + dx));
        }
      }
      double out = n ? sqrt(m2 / n) : 0.0;
      if (fs_is_nd<float>(__ldg(centre), a.kind, ndv)) out = a.nd_out;
      const int64_t o = static_cast<int64_t>(blockIdx.z) * a.out_band_stride + y * a.out_pitch + x;
      if (a.out_dtype == VSR_F64) static_cast<double*>(a.dst)[o] = out;
      else static_cast<float*>(a.dst)[o] = static_cast<float>(out);
    }
    __syncwarp();
  }
}

// Range of the strip's valid values, halo included.
template <int R, bool EDGE>
__device__ __forceinline__ void scan_range(const FsArgs& a, const SdStrip& S, bool vin, uint32_t& amin, float& vmin,
                                           float& vmax) {
  const int64_t xs = S.xw + 4 * (threadIdx.x & 31);
  uint32_t inm = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) inm |= static_cast<uint32_t>(xs + e >= 0 && xs + e < a.W) << e;
  const int64_t g0 = S.ys - R < 0 ? 0 : S.ys - R, g1 = S.ys + S.nout + R < a.H ? S.ys + S.nout + R : a.H;
  const int rows = static_cast<int>(g1 - g0);
  const float* lp = static_cast<const float*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride +
                    g0 * a.pitch + xs;
#pragma unroll 4
  for (int i = 0; i < rows; ++i, lp += a.pitch) {
    uint32_t raw[4];
    strip_load4<float, EDGE>(lp, inm, vin, raw);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float v = __uint_as_float(raw[e]);
      bool ok = (v != S.ndq) & (v == v);
      if (EDGE) ok = ok & ((inm >> e) & 1u);
      amin = min(amin, ok ? (raw[e] & 0x7fffffffu) - 1u : 0xFFFFFFFFu);
      vmin = fminf(vmin, ok ? v : __int_as_float(0x7f800000));
      vmax = fmaxf(vmax, ok ? v : __int_as_float(0xff800000));
    }
  }
}

// 16 blocks per SM (128 registers); 20 blocks spill: a 7 x 7 std takes 143 us
// against 153 at 4096^2 with them, but 65 against 55 at 1000 x 4096.
template <int R, typename T>
__global__ void __launch_bounds__(kSdThreads, 16) fs_strip_std(const FsArgs a, const int strip, const bool vin,
                                                           const bool vout) {
  using G = SdGeom<R>;
  constexpr bool kFloat = std::is_same<T, float>::value;
  constexpr int kLimbs = kFloat ? 2 : 1;
  extern __shared__ __align__(16) unsigned char sd_smem[];
  uint64_t* obuf = reinterpret_cast<uint64_t*>(sd_smem);
  int4* ring = reinterpret_cast<int4*>(sd_smem + 128 * 8);
  uint32_t* flags = reinterpret_cast<uint32_t*>(ring + G::P * kLimbs * kSdThreads);
  SdStrip S{};
  S.xw = static_cast<int64_t>(blockIdx.x) * G::kCols - 4 * G::HL;
  S.ys = static_cast<int64_t>(blockIdx.y) * strip;
  S.nout = static_cast<int>(a.H - S.ys < strip ? a.H - S.ys : static_cast<int64_t>(strip));
  S.inside = S.xw >= 0 && S.xw + 128 <= a.W;
  if constexpr (!kFloat) {
    if (S.inside) run_strip<R, T, 1, false>(a, S, vin, vout, ring, flags, obuf);
    else run_strip<R, T, 1, true>(a, S, vin, vout, ring, flags, obuf);
  } else {
    // smallest non-zero magnitude and range of the strip's valid values
    S.ndq = a.kind == VSR_NODATA_VALUE ? static_cast<float>(a.ndv) : __int_as_float(0x7fffffff);
    uint32_t amin = 0xFFFFFFFFu;  // smallest non-zero magnitude's bits, less 1
    float vmin = __int_as_float(0x7f800000), vmax = -vmin;
    if (S.inside) scan_range<R, false>(a, S, vin, amin, vmin, vmax);
    else scan_range<R, true>(a, S, vin, amin, vmin, vmax);
#pragma unroll
    for (int d = 16; d; d >>= 1) {
      amin = min(amin, __shfl_xor_sync(0xffffffffu, amin, d));
      vmin = fminf(vmin, __shfl_xor_sync(0xffffffffu, vmin, d));
      vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, d));
    }
    if (amin == 0xFFFFFFFFu) {  // no value, or zeros only: any unit
      amin = 0x3f7fffffu;
      vmin = vmax = 0.0f;
    }
    ++amin;
    const int E = static_cast<int>(amin >> 23);
    const float vabs = fmaxf(fabsf(vmin), fabsf(vmax));
    const int span = static_cast<int>(__float_as_uint(vabs) >> 23) - E;
    // 24 <= E: the scales below are normal floats; infinities have exponent 255
    if (E < 24 || E > 250 || span > 2 * G::kLB - 24 || __float_as_uint(vabs) >= 0x7f800000u) {
      slow_strip<R>(a, S, reinterpret_cast<double*>(sd_smem), reinterpret_cast<int*>(sd_smem + 256 * 8));
      return;
    }
    S.u = E - 150;
    S.s1 = __uint_as_float(static_cast<uint32_t>(277 - E) << 23);  // 2^(150 - E)
    S.s2 = __uint_as_float(static_cast<uint32_t>(277 - G::kLB - E) << 23);  // 2^(150 - kLB - E)
    // one word: sums of n differences from the middle of the range stay below 2^31
    const float units = __fmul_ru(__fsub_ru(vmax, vmin), S.s1);
    if (span <= 6 && units < 4294900000.0f / static_cast<float>(G::kTaps)) {
      S.ref = __float2int_rn(vmin * S.s1) + __float2int_rn(0.5f * units);
      if (S.inside) run_strip<R, T, 1, false>(a, S, vin, vout, ring, flags, obuf);
      else run_strip<R, T, 1, true>(a, S, vin, vout, ring, flags, obuf);
    } else {
      run_strip<R, T, 2, true>(a, S, vin, vout, ring, flags, obuf);
    }
  }
}

template <int R, typename T>
int launch_strip_std(const FsArgs& a, int bands, cudaStream_t st) {
  using G = SdGeom<R>;
  constexpr int kLimbs = std::is_same<T, float>::value ? 2 : 1;
  const size_t smem = 128 * 8 + static_cast<size_t>(G::P) * kSdThreads * (16 * kLimbs + 4);
  static_assert(kLimbs == 1 || 128 * 8 + G::P * kSdThreads * (16 * kLimbs + 4) >= 256 * 12, "slow_strip's columns");
  auto kern = fs_strip_std<R, T>;
  static KernelResidency residency;
  int per_sm = 0;
  VSR_CUDA_TRY(residency.get(kern, kSdThreads, smem, &per_sm));
  const int64_t gx = (a.W + G::kCols - 1) / G::kCols;
  // rows per strip: the most that leaves every SM 32 blocks, two rounds of
  // what fits (2R rows of a strip are read again by the next one).  4096^2,
  // 11 x 11: 178 us with that, 191 us with 16 blocks per SM
  int strip = 128;
  while (strip > 16 && gx * ((a.H + strip - 1) / strip) * bands < 32 * static_cast<int64_t>(sm_count())) strip /= 2;
  if (gx * ((a.H + 15) / 16) * bands < kSdFew * static_cast<int64_t>(sm_count())) {
    if (!std::is_same<T, float>::value) return -1;
    strip = 8;
  }
  const int64_t gy = (a.H + strip - 1) / strip;
  if (gy > 65535) return -1;
  const bool vin = aligned(a.src, 4 * sizeof(T)) && a.pitch % 4 == 0 && (bands == 1 || a.band_stride % 4 == 0);
  const size_t os = a.out_dtype == VSR_F64 ? 8 : 4;
  const bool vout = aligned(a.dst, 4 * os) && a.out_pitch % 4 == 0 && (bands == 1 || a.out_band_stride % 4 == 0);
  kern<<<dim3(static_cast<unsigned>(gx), static_cast<unsigned>(gy), static_cast<unsigned>(bands)), kSdThreads, smem,
         st>>>(a, strip, vin, vout);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

template <typename T>
int launch_strip_std_r(const FsArgs& a, int bands, cudaStream_t st) {
  switch (a.ry) {
    case 1: return launch_strip_std<1, T>(a, bands, st);
    case 2: return launch_strip_std<2, T>(a, bands, st);
    case 3: return launch_strip_std<3, T>(a, bands, st);
    case 4: return launch_strip_std<4, T>(a, bands, st);
    case 5: return launch_strip_std<5, T>(a, bands, st);
    case 6: return launch_strip_std<6, T>(a, bands, st);
    default: return launch_strip_std<7, T>(a, bands, st);
  }
}

}  // namespace

int fs_std_strip(const FsArgs& a, int bands, cudaStream_t st) {
  if (a.ry != a.rx || a.ry < 1 || a.ry > kSdMaxR) return -1;
  switch (a.dtype) {
    case VSR_U8: return launch_strip_std_r<uint8_t>(a, bands, st);
    case VSR_I16: return launch_strip_std_r<int16_t>(a, bands, st);
    case VSR_U16: return launch_strip_std_r<uint16_t>(a, bands, st);
    case VSR_F32: return launch_strip_std_r<float>(a, bands, st);
    default: return -1;
  }
}

}  // namespace vsr
