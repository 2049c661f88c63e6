// Arguments shared by the focal-statistic kernels (focal_stats.cu and the
// warp-strip kernels that take over where they apply).
#pragma once

#include <algorithm>
#include <type_traits>

#include "std_round64.h"
#include "vsr_internal.cuh"

namespace vsr {

constexpr int kFsMaxVarietyRadius = 7;  // window up to 15 x 15 (225 taps)

struct FsArgs {
  const void* src;
  int dtype;
  int64_t H, W, pitch, band_stride;
  int kind;     // resolved VSR_NODATA_*
  double ndv;   // nodata in the element type (exact)
  int ry, rx;
  double nd_out;  // written for nodata centres and empty windows
  void* dst;
  int out_dtype;
  int64_t out_pitch, out_band_stride;
};

// Nodata test in the element type itself (the value is exact there).
template <typename TIN>
__device__ __forceinline__ bool fs_is_nd(TIN v, int kind, TIN ndv) {
  if constexpr (std::is_floating_point<TIN>::value)
    return kind == VSR_NODATA_VALUE ? v == ndv : (kind == VSR_NODATA_NAN ? v != v : false);
  else
    return kind == VSR_NODATA_VALUE && v == ndv;
}

// 2^(63 + floor(log2 n)) / n for the window counts of vsr_s64_std.
constexpr int kRecipTaps = 225;
struct RecipTable {
  uint64_t v[kRecipTaps + 1];
};
constexpr RecipTable make_recips() {
  RecipTable t{};
  for (uint32_t n = 1; n <= kRecipTaps; ++n) t.v[n] = vsr_s64_recip(n);
  return t;
}
static __device__ const RecipTable g_recip = make_recips();
__device__ __forceinline__ uint64_t fs_recip(uint32_t n) { return __ldg(&g_recip.v[n]); }

// Launch the kernel if it serves these arguments; -1 otherwise.
int fs_std_strip(const FsArgs& a, int bands, cudaStream_t st);  // focal_std.cu
int fs_variety(const FsArgs& a, int bands, cudaStream_t st);    // focal_variety.cu: every dtype and window

}  // namespace vsr
