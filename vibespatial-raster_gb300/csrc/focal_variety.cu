// Focal variety: the number of distinct valid values in the window
// (semantics of algebra.py:3146-3163; no cap on the count).
//
// Two forms (on a 5001 x 4999 map of 12 classes and holes, 5 x 5: 92 us, 2.4
// TB/s, against 2680 us for comparing all pairs of taps).
//
// * fs_variety_bits -- 8/16-bit rasters, square windows of radius 1..7.  A
//   block finds the set of values of its tile (with the halo) and
//   numbers them; a window's set is then the OR of its pixels' one-hot words,
//   which is separable: rows first (neighbours' words by shuffles, the
//   layout of warp_strip.cuh), then the last 2R+1 rows' results, which wait
//   in shared memory, each thread reading only its own.  32 values per pass;
//   a tile of a class map holds few, so one pass is the rule.  About 12
//   instructions per pixel and pass, against n^2 / 2 compares for n taps:
//   tiles with more than n^2 / 2 values (n^2 / 64 passes) take the second
//   form.
//
// * variety_pairs -- every other dtype, window or tile.  A tap counts when no
//   equal tap precedes it in the window (row-major).  Whether one does
//   depends on the tap's pixel p, its window column ix and row iy: let
//   first(p, ix) be the smallest dy such that row y - dy holds p's value at a
//   column inside the window (dy = 0: to the left only); the tap counts when
//   first > iy.  Each pixel compares with its 2 ry rows above once
//   ((4 rx + 1) (2 ry) + 2 rx compares) and keeps its 2 rx + 1 numbers as
//   nibbles of a 64-bit word; a window then adds up n tests.  49 taps: 84
//   compares and 49 tests instead of up to 1176 compares.
#include <type_traits>

#include "focal_stats.cuh"
#include "warp_strip.cuh"

namespace vsr {
namespace {

constexpr int kVyThreads = 128;      // block of the pairs form
constexpr int kVyMaxR = 7;           // nibbles: 2 r + 1 <= 15 columns, dy <= 14
constexpr int kVyTX = 64, kVyTY = 16;  // tile of the pairs form
constexpr int kVyStrip = 16;         // rows of a block of the bits form
constexpr int kVyOut = 258;          // output table: counts 0 .. 225, nodata at 256

__device__ __forceinline__ void vy_store(const FsArgs& a, int64_t o, double v) {
  if (a.out_dtype == VSR_F64) static_cast<double*>(a.dst)[o] = v;
  else static_cast<float*>(a.dst)[o] = static_cast<float>(v);
}

// ------------------------------------------------------------ pairs form --
// Keys: equal exactly when the values are.  8/16-bit values and float32 bit
// patterns (-0 as 0) in 32 bits, int32 and float64 as float64 bits; a NaN
// pattern marks taps that do not count (nodata, NaN, outside the raster).
template <typename T>
using VyKey = std::conditional_t<std::is_same<T, double>::value || std::is_same<T, int32_t>::value, uint64_t, uint32_t>;
template <typename K>
__device__ __forceinline__ K vy_none() { return static_cast<K>(~K(0)); }

template <typename T>
__device__ __forceinline__ VyKey<T> vy_key(T v) {
  if constexpr (std::is_same<T, float>::value) return __float_as_uint(v == 0.0f ? 0.0f : v);
  else if constexpr (std::is_same<T, double>::value)
    return static_cast<uint64_t>(__double_as_longlong(v == 0.0 ? 0.0 : v));
  else if constexpr (std::is_same<T, int32_t>::value)
    return static_cast<uint64_t>(static_cast<int64_t>(v)) & 0xffffffffu;
  else return static_cast<uint32_t>(static_cast<std::make_unsigned_t<T>>(v));
}

template <typename K>
__host__ __device__ inline size_t vy_pairs_smem(int ry, int rx) {
  const size_t SH = kVyTY + 2 * ry, SW = kVyTX + 2 * rx;
  return SH * SW * 8 + SH * (SW + 4 * rx) * sizeof(K) + kVyTX * kVyTY + 16;
}

// One 64 x 16 tile at (x0, y0) of the block's band (columns below x1) by all
// its threads.
// R > 0: a square window of that radius; R == 0: the radii of ``a``.
template <typename T, int R, int THREADS>
__device__ void variety_pairs(const FsArgs& a, int64_t x0, int64_t y0, int64_t x1, unsigned char* smem) {
  using K = VyKey<T>;
  const int ry = R ? R : a.ry, rx = R ? R : a.rx;
  const int SH = kVyTY + 2 * ry, SW = kVyTX + 2 * rx, SP = SW + 4 * rx;
  uint64_t* first = reinterpret_cast<uint64_t*>(smem);  // SH x SW
  K* key = reinterpret_cast<K*>(first + SH * SW);        // SH x SP, 2 rx columns of "none" at both ends
  unsigned char* ndc = reinterpret_cast<unsigned char*>(key + SH * SP);
  const int tid = threadIdx.x;
  const T* src = static_cast<const T*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride;
  const T ndv = static_cast<T>(a.ndv);
  for (int i = tid; i < SH * SP; i += THREADS) {
    const int r = i / SP, c = i - r * SP - 2 * rx;
    const int64_t gy = y0 - ry + r, gx = x0 - rx + c;
    K k = vy_none<K>();
    bool nd = false;
    if (c >= 0 && c < SW && gy >= 0 && gy < a.H && gx >= 0 && gx < a.W) {
      const T v = __ldg(src + gy * a.pitch + gx);
      nd = fs_is_nd<T>(v, a.kind, ndv);
      if (!nd && v == v) k = vy_key<T>(v);
    }
    key[i] = k;
    const int cr = r - ry, cc = c - rx;
    if (cr >= 0 && cr < kVyTY && cc >= 0 && cc < kVyTX) ndc[cr * kVyTX + cc] = nd;
  }
  __syncthreads();
  const int kw = 2 * rx + 1;
  for (int i = tid; i < SH * SW; i += THREADS) {
    const int r = i / SW, c = i - r * SW;
    const K* p = key + r * SP + 2 * rx + c;
    const K k = *p;
    uint64_t f = 0;  // a tap that does not count: first = 0 for every column
    if (k != vy_none<K>()) {
      f = ~uint64_t(0);
      // bit j of m: the row holds k at column offset j - 2 rx; window column
      // ix sees offsets -ix .. 2 rx - ix, bits 2 rx - ix .. 4 rx - ix
      uint32_t open = (1u << kw) - 1u;  // columns whose number is not known yet
#pragma unroll
      for (int dy = 0; dy <= 2 * ry; ++dy) {
        if (dy > r) break;
        const K* q = p - dy * SP - 2 * rx;
        const int nc = dy ? 4 * rx + 1 : 2 * rx;
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < nc; ++j) m |= static_cast<uint32_t>(q[j] == k) << j;
        if (m) {
#pragma unroll
          for (int ix = 0; ix < kw; ++ix)
            if (((m >> (2 * rx - ix)) & ((1u << kw) - 1u)) && ((open >> ix) & 1u)) {
              f ^= static_cast<uint64_t>(15 ^ dy) << (4 * ix);  // nibble 15 -> dy
              open ^= 1u << ix;
            }
          if (!open) break;
        }
      }
    }
    first[i] = f;
  }
  __syncthreads();
  const int nr = static_cast<int>(a.H - y0 < kVyTY ? a.H - y0 : int64_t(kVyTY));
  const int nc = static_cast<int>(x1 - x0 < kVyTX ? x1 - x0 : int64_t(kVyTX));
  for (int i = tid; i < kVyTX * kVyTY; i += THREADS) {
    const int r = i / kVyTX, c = i - r * kVyTX;
    if (r >= nr || c >= nc) continue;
    int cnt = 0;
#pragma unroll
    for (int iy = 0; iy <= 2 * ry; ++iy)
#pragma unroll
      for (int ix = 0; ix < kw; ++ix) {
        // the 32-bit half that holds the nibble
        const uint32_t h = reinterpret_cast<const uint32_t*>(first + (r + iy) * SW + c + ix)[ix >> 3];
        cnt += static_cast<int>((h >> (4 * (ix & 7))) & 15u) > iy;
      }
    vy_store(a, static_cast<int64_t>(blockIdx.z) * a.out_band_stride + (y0 + r) * a.out_pitch + x0 + c,
             ndc[i] ? a.nd_out : static_cast<double>(cnt));
  }
  __syncthreads();  // the staged tile may be overwritten
}

template <typename T, int R>
__global__ void __launch_bounds__(kVyThreads) fs_variety_pairs(const FsArgs a) {
  extern __shared__ __align__(16) unsigned char vy_smem[];
  variety_pairs<T, R, kVyThreads>(a, static_cast<int64_t>(blockIdx.x) * kVyTX, static_cast<int64_t>(blockIdx.y) * kVyTY, a.W,
                      vy_smem);
}

// ------------------------------------------------------------- bits form --
template <int R, typename T>
struct VyGeom {
  static constexpr int P = 2 * R + 1, kTaps = P * P;
  static constexpr int HL = (R + 3) / 4;
  static constexpr int kCols = 128 - 8 * HL;
  static constexpr bool kByte = sizeof(T) == 1;
  // 4 warps share the value table; 16 rows per block keep its set small and
  // the blocks many.  5001 x 4999, 5 x 5, rows x warps: 16 x 4 92 us, 32 x 4
  // 94, 64 x 4 127, 32 x 2 92, 32 x 1 117; 400 values in 16 bits: 595, 672, 788
  static constexpr int kWarps = 4, kThreads = 32 * kWarps;
  static constexpr int kMaxValues = kTaps * kTaps / 2;  // see above
  // shared memory, in bytes: value table, output table, transfer buffer, the
  // rows' words and nodata flags, packed counts (several passes)
  static constexpr int kTab = kByte ? 256 * 4 : 2048 * 8;
  static constexpr int kBuf = kWarps * 128 * 8, kCnt = kVyStrip * kThreads * 4;
  static constexpr int kRing = P * kThreads * 20;
  static constexpr size_t smem() { return static_cast<size_t>(kTab) + kVyOut * 8 + kBuf + kCnt + kRing; }
};

// A warp's strip of a block's tile.
struct VyStrip {
  int64_t xw, xs, ys;  // first column of lane 0, of this lane; first output row
  int nout;
  uint32_t inm;        // this lane's columns inside the raster
  bool vin, vout, has_nd;
  uint32_t ndk;        // nodata's bit pattern
};

// Mark the strip's values.  8-bit: a word per value (plain stores); 16-bit: a
// bitmap, tested before the atomic (most pixels repeat a value).  Nodata is
// taken out of the table afterwards.
template <int R, typename T, bool EDGE>
__device__ __forceinline__ void vy_scan(const FsArgs& a, const T* src, const VyStrip& S, uint32_t* lut, uint2* tab) {
  const int64_t g0 = S.ys - R < 0 ? 0 : S.ys - R, g1 = S.ys + S.nout + R < a.H ? S.ys + S.nout + R : a.H;
  const int rows = static_cast<int>(g1 - g0);
  const T* lp = src + g0 * a.pitch + S.xs;
#pragma unroll 4
  for (int i = 0; i < rows; ++i, lp += a.pitch) {
    uint32_t e4[4];
    strip_load4<T, EDGE>(lp, S.inm, S.vin, e4);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const bool in = !EDGE || ((S.inm >> e) & 1u);
      if (sizeof(T) == 1) {
        if (in) lut[e4[e]] = 1u;
      } else {
        const uint32_t b = 1u << (e4[e] & 31u);
        if (in && !(*reinterpret_cast<volatile uint32_t*>(&tab[e4[e] >> 5].x) & b)) atomicOr(&tab[e4[e] >> 5].x, b);
      }
    }
  }
}

// One pass over the strip: the counts of values 32 w .. 32 w + 31, added to
// those of the earlier passes (``cbuf``, unless the first); the last pass
// writes the outputs through ``out``: the bits of count n at n, of nodata at
// 256.
template <int R, typename T, bool EDGE>
__device__ __forceinline__ void vy_pass(const FsArgs& a, const T* src, const VyStrip& S, int w, bool last,
                                        const uint32_t* lut, const uint2* tab, const uint64_t* out, uint32_t* cbuf,
                                        uint4* ring, uint32_t* flags, uint64_t* obuf) {
  using G = VyGeom<R, T>;
  constexpr int P = G::P, HL = G::HL;
  const int t = threadIdx.x, lane = t & 31;
  const int nin = S.nout + 2 * R;
  constexpr int lo = 4 * HL;
  const int hi = static_cast<int>(a.W - S.xw < 128 - 4 * HL ? a.W - S.xw : static_cast<int64_t>(128 - 4 * HL));
  const bool f64 = a.out_dtype == VSR_F64;
  auto row_in = [&](int i) { return static_cast<uint64_t>(S.ys - R + i) < static_cast<uint64_t>(a.H); };
  const T* lp = src + (S.ys - R) * a.pitch + S.xs;
  uint32_t nxt[4] = {0u, 0u, 0u, 0u};
  if (row_in(0)) strip_load4<T, EDGE>(lp, S.inm, S.vin, nxt);
  int64_t orow = static_cast<int64_t>(blockIdx.z) * a.out_band_stride + S.ys * a.out_pitch + S.xw;
  int slot = 0, cslot = P - R;
#pragma unroll 1
  for (int i = 0; i < nin; ++i) {
    uint32_t o[4 * (2 * HL + 1)];
    uint32_t f = 0;
    if (row_in(i)) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t word;
        if (G::kByte) {
          word = lut[nxt[e]];
        } else {
          const uint2 en = tab[nxt[e] >> 5];
          const uint32_t b = 1u << (nxt[e] & 31u), rank = en.y + __popc(en.x & (b - 1u)) - 32u * w;
          word = (en.x & b) && rank < 32u ? 1u << rank : 0u;
        }
        if (EDGE && !((S.inm >> e) & 1u)) word = 0u;
        o[4 * HL + e] = word;
      }
      if (last && S.has_nd) {
#pragma unroll
        for (int e = 0; e < 4; ++e) f |= nxt[e] == S.ndk ? 1u << e : 0u;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) o[4 * HL + e] = 0u;
    }
    lp += a.pitch;
    if (i + 1 < nin && row_in(i + 1)) strip_load4<T, EDGE>(lp, S.inm, S.vin, nxt);
#pragma unroll
    for (int h = 1; h <= HL; ++h)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (4 * h - e <= R) o[4 * (HL - h) + e] = __shfl_up_sync(0xffffffffu, o[4 * HL + e], h);
        if (4 * h + e - 3 <= R) o[4 * (HL + h) + e] = __shfl_down_sync(0xffffffffu, o[4 * HL + e], h);
      }
    uint32_t hz[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      hz[c] = 0u;
#pragma unroll
      for (int j = 4 * HL + c - R; j <= 4 * HL + c + R; ++j) hz[c] |= o[j];
    }
    ring[slot * G::kThreads] = make_uint4(hz[0], hz[1], hz[2], hz[3]);
    if (S.has_nd) flags[slot * G::kThreads] = f;
    slot = slot + 1 == P ? 0 : slot + 1;
    if (i >= 2 * R) {
      // all slots hold rows of the window
#pragma unroll
      for (int s = 0; s < P; ++s) {
        const uint4 q = ring[s * G::kThreads];
        hz[0] |= q.x;
        hz[1] |= q.y;
        hz[2] |= q.z;
        hz[3] |= q.w;
      }
      uint32_t n[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) n[c] = __popc(hz[c]);
      const int j = i - 2 * R;
      if (w) {
        const uint32_t m = cbuf[j * G::kThreads];
#pragma unroll
        for (int c = 0; c < 4; ++c) n[c] += (m >> (8 * c)) & 0xFFu;
      }
      if (!last) {
        cbuf[j * G::kThreads] = n[0] | (n[1] << 8) | (n[2] << 16) | (n[3] << 24);
      } else {
        if (S.has_nd) {
          const uint32_t fc = flags[cslot * G::kThreads];
#pragma unroll
          for (int c = 0; c < 4; ++c) n[c] = (fc >> c) & 1u ? 256u : n[c];
        }
        if (f64) {
          uint64_t v[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) v[c] = out[n[c]];
          strip_store4<uint64_t>(static_cast<uint64_t*>(a.dst) + orow, v, lane, lo, hi, S.vout, obuf);
        } else {
          uint32_t v[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) v[c] = static_cast<uint32_t>(out[n[c]]);
          strip_store4<uint32_t>(static_cast<uint32_t*>(a.dst) + orow, v, lane, lo, hi, S.vout,
                                 reinterpret_cast<uint32_t*>(obuf));
        }
      }
      orow += a.out_pitch;
    }
    cslot = cslot + 1 == P ? 0 : cslot + 1;
  }
}

template <int R, typename T>
__global__ void __launch_bounds__(VyGeom<R, T>::kThreads) fs_variety_bits(const FsArgs a, const bool vin, const bool vout) {
  using G = VyGeom<R, T>;
  using U = std::make_unsigned_t<T>;
  constexpr int P = G::P, HL = G::HL;
  extern __shared__ __align__(16) unsigned char vy_smem[];
  __shared__ int wsum[G::kWarps];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  uint32_t* lut = reinterpret_cast<uint32_t*>(vy_smem);  // 8-bit: one-hot word of each value in this pass
  uint2* tab = reinterpret_cast<uint2*>(vy_smem);        // 16-bit: (bitmap word, values below it)
  uint64_t* out = reinterpret_cast<uint64_t*>(vy_smem + G::kTab);
  uint64_t* obuf = out + kVyOut + 128 * warp;
  uint4* ring = reinterpret_cast<uint4*>(vy_smem + G::kTab + kVyOut * 8 + G::kBuf) + t;
  uint32_t* flags = reinterpret_cast<uint32_t*>(ring - t + P * G::kThreads) + t;
  uint32_t* cbuf = flags + P * G::kThreads;
  const int64_t xb = static_cast<int64_t>(blockIdx.x) * G::kWarps * G::kCols;  // the block's first output column
  const T* src = static_cast<const T*>(a.src) + static_cast<int64_t>(blockIdx.z) * a.band_stride;
  VyStrip S;
  S.xw = xb + warp * G::kCols - 4 * HL;
  S.xs = S.xw + 4 * lane;
  S.ys = static_cast<int64_t>(blockIdx.y) * kVyStrip;
  S.nout = static_cast<int>(a.H - S.ys < kVyStrip ? a.H - S.ys : static_cast<int64_t>(kVyStrip));
  S.inm = 0;
#pragma unroll
  for (int e = 0; e < 4; ++e) S.inm |= static_cast<uint32_t>(S.xs + e >= 0 && S.xs + e < a.W) << e;
  S.vin = vin;
  S.vout = vout;
  S.has_nd = a.kind == VSR_NODATA_VALUE;
  S.ndk = static_cast<U>(static_cast<T>(a.ndv));
  const bool active = S.xw + 4 * HL < a.W;  // warp-uniform
  const bool inside = S.xw >= 0 && S.xw + 128 <= a.W;

  // the tile's set of values
  if (G::kByte) {
    for (int i = t; i < 256; i += G::kThreads) lut[i] = 0u;
  } else {
    for (int i = t; i < 2048; i += G::kThreads) tab[i] = make_uint2(0u, 0u);
  }
  for (int n = t; n <= 256; n += G::kThreads) {
    const double v = n == 256 ? a.nd_out : static_cast<double>(n);
    out[n] = a.out_dtype == VSR_F64 ? static_cast<uint64_t>(__double_as_longlong(v))
                                    : __float_as_uint(static_cast<float>(v));
  }
  __syncthreads();
  if (inside) vy_scan<R, T, false>(a, src, S, lut, tab);
  else if (active) vy_scan<R, T, true>(a, src, S, lut, tab);
  __syncthreads();
  if (t == 0 && S.has_nd) {
    if (G::kByte) lut[S.ndk] = 0u;
    else tab[S.ndk >> 5].x &= ~(1u << (S.ndk & 31u));
  }
  __syncthreads();
  // number the values: each thread owns a run of them
  constexpr int kOwn = (G::kByte ? 256 : 2048) / G::kThreads;  // 8-bit: values; 16-bit: bitmap words
  uint32_t own[kOwn];
  int cnt = 0;
#pragma unroll
  for (int i = 0; i < kOwn; ++i) {
    own[i] = G::kByte ? lut[t * kOwn + i] : tab[t * kOwn + i].x;
    cnt += __popc(own[i]);
  }
  int pre = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, pre, d);
    if (lane >= d) pre += v;
  }
  if (lane == 31) wsum[warp] = pre;
  __syncthreads();
  int base = pre - cnt, total = 0;
#pragma unroll
  for (int w = 0; w < G::kWarps; ++w) {
    base += w < warp ? wsum[w] : 0;
    total += wsum[w];
  }
  if (total > G::kMaxValues) {  // block-uniform
    const int64_t x1 = xb + G::kWarps * G::kCols < a.W ? xb + G::kWarps * G::kCols : a.W;
    for (int64_t y = S.ys; y < S.ys + S.nout; y += kVyTY)
      for (int64_t x = xb; x < x1; x += kVyTX) variety_pairs<T, R, G::kThreads>(a, x, y, x1, vy_smem);
    return;
  }
  if (!G::kByte) {
    int b = base;
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
      tab[t * kOwn + i].y = static_cast<uint32_t>(b);
      b += __popc(own[i]);
    }
  }
  const int passes = total > 32 ? (total + 31) / 32 : 1;
  for (int w = 0; w < passes; ++w) {
    if (G::kByte) {
      if (w) __syncthreads();  // every thread is done with the last pass's words
      int b = base - 32 * w;
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        lut[t * kOwn + i] = own[i] && static_cast<uint32_t>(b) < 32u ? 1u << b : 0u;
        b += own[i];
      }
    }
    if (w == 0 || G::kByte) __syncthreads();
    const bool last = w + 1 == passes;
    if (inside) vy_pass<R, T, false>(a, src, S, w, last, lut, tab, out, cbuf, ring, flags, obuf);
    else if (active) vy_pass<R, T, true>(a, src, S, w, last, lut, tab, out, cbuf, ring, flags, obuf);
  }
}

template <int R, typename T>
int launch_bits(const FsArgs& a, int bands, cudaStream_t st) {
  using G = VyGeom<R, T>;
  const size_t smem = std::max(G::smem(), vy_pairs_smem<VyKey<T>>(R, R));
  auto kern = fs_variety_bits<R, T>;
  static KernelResidency residency;
  int per_sm = 0;
  VSR_CUDA_TRY(residency.get(kern, G::kThreads, smem, &per_sm));
  const bool vin = aligned(a.src, 4 * sizeof(T)) && a.pitch % 4 == 0 && (bands == 1 || a.band_stride % 4 == 0);
  const size_t os = a.out_dtype == VSR_F64 ? 8 : 4;
  const bool vout = aligned(a.dst, 4 * os) && a.out_pitch % 4 == 0 && (bands == 1 || a.out_band_stride % 4 == 0);
  kern<<<dim3(static_cast<unsigned>((a.W + G::kWarps * G::kCols - 1) / (G::kWarps * G::kCols)),
              static_cast<unsigned>((a.H + kVyStrip - 1) / kVyStrip), static_cast<unsigned>(bands)),
         G::kThreads, smem, st>>>(a, vin, vout);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

template <typename T, int R>
int launch_pairs(const FsArgs& a, int bands, cudaStream_t st) {
  const size_t smem = vy_pairs_smem<VyKey<T>>(a.ry, a.rx);
  auto kern = fs_variety_pairs<T, R>;
  VSR_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  kern<<<dim3(static_cast<unsigned>((a.W + kVyTX - 1) / kVyTX), static_cast<unsigned>((a.H + kVyTY - 1) / kVyTY),
              static_cast<unsigned>(bands)),
         kVyThreads, smem, st>>>(a);
  VSR_CUDA_TRY(cudaGetLastError());
  return VSR_OK;
}

// A raster of few blocks in the bits form takes the pairs form (64 x 16 tiles): a
// block numbers its values and makes its passes, or compares the pairs of eight
// tiles, one after the other.  us, pairs | bits: 3 x 3, 16-bit with 12 values
// 300^2 10 | 21, 1449^2 25 | 29, 1740^2 33 | 29; with 250 values 512^2 9 | 47,
// 1449^2 23 | 60; 8-bit with 12 values 725^2 10 | 15, 1024^2 17 | 17, 1230^2 21 |
// 17, with 250 values 1024^2 14 | 47; 5 x 5, 16-bit with 250 values 300^2 13 | 73,
// 725^2 19 | 74, with 12 values 725^2 23 | 23, 850^2 25 | 23.
template <int R, typename T>
bool few_blocks(const FsArgs& a, int bands) {
  using G = VyGeom<R, T>;
  constexpr int kEighths = R == 1 ? (G::kByte ? 11 : 32) : (G::kByte ? 0 : 8);  // of a block per SM
  const int64_t gx = (a.W + G::kWarps * G::kCols - 1) / (G::kWarps * G::kCols), gy = (a.H + kVyStrip - 1) / kVyStrip;
  return 8 * gx * gy * bands < kEighths * static_cast<int64_t>(sm_count());
}

template <typename T>
int dispatch_t(const FsArgs& a, int bands, cudaStream_t st) {
  const bool square = a.ry == a.rx;
  if constexpr (std::is_integral<T>::value && sizeof(T) <= 2) {
    if (square) switch (a.ry) {
        case 1: return few_blocks<1, T>(a, bands) ? launch_pairs<T, 1>(a, bands, st) : launch_bits<1, T>(a, bands, st);
        case 2: return few_blocks<2, T>(a, bands) ? launch_pairs<T, 2>(a, bands, st) : launch_bits<2, T>(a, bands, st);
        case 3: return launch_bits<3, T>(a, bands, st);
        case 4: return launch_bits<4, T>(a, bands, st);
        case 5: return launch_bits<5, T>(a, bands, st);
        case 6: return launch_bits<6, T>(a, bands, st);
        case 7: return launch_bits<7, T>(a, bands, st);
        default: break;
      }
    return launch_pairs<T, 0>(a, bands, st);
  } else {
    if (square) switch (a.ry) {
        case 1: return launch_pairs<T, 1>(a, bands, st);
        case 2: return launch_pairs<T, 2>(a, bands, st);
        case 3: return launch_pairs<T, 3>(a, bands, st);
        default: break;
      }
    return launch_pairs<T, 0>(a, bands, st);
  }
}

}  // namespace

static_assert(kFsMaxVarietyRadius == kVyMaxR, "radius limit");

int fs_variety(const FsArgs& a, int bands, cudaStream_t st) {
  switch (a.dtype) {
    case VSR_U8: return dispatch_t<uint8_t>(a, bands, st);
    case VSR_I16: return dispatch_t<int16_t>(a, bands, st);
    case VSR_U16: return dispatch_t<uint16_t>(a, bands, st);
    case VSR_I32: return dispatch_t<int32_t>(a, bands, st);
    case VSR_F32: return dispatch_t<float>(a, bands, st);
    default: return dispatch_t<double>(a, bands, st);
  }
}

}  // namespace vsr
