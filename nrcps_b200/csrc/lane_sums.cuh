// lane_sums.cuh -- a warp's FP32 sums of many values, spread over its lanes.
#pragma once

#include "common.cuh"

namespace nrcps {

// Values a lane holds after reduce_scatter of `values` (padded to 32 or 64).
constexpr int lane_share(int values) { return values > 32 ? 2 : 1; }

// v[0 .. N) of every lane summed over the warp, a tree of five levels; lane l
// is left with the sums of e = lane_share(N) l + k in v[k].  The lanes halve
// the values between them at each level: about 2 N shuffles and adds per warp
// where a full reduction of each value takes 5 N.
template <int N>
__device__ __forceinline__ void reduce_scatter(float (&v)[N], int lane) {
  constexpr int FULL = N > 32 ? 64 : 32;
#pragma unroll
  for (int l = 0; l < 5; ++l) {
    const int h = FULL >> (l + 1), bit = 16 >> l;
    const bool up = lane & bit;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      if (k >= N) continue;
      const float hi = k + h < N ? v[k + h] : 0.f;  // (entries past N are zeros)
      const float keep = up ? hi : v[k], send = up ? v[k] : hi;
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
}

}  // namespace nrcps
