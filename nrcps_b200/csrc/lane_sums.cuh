// lane_sums.cuh -- a warp's FP32 sums of many values, spread over its lanes.
#pragma once

#include "common.cuh"

namespace nrcps {

// Values a lane holds after reduce_scatter of `values` (padded to 32 or 64).
constexpr int lane_share(int values) { return values > 32 ? 2 : 1; }

// v[0 .. N) of every lane summed over the warp, levels FIRST .. LAST - 1 of a
// tree of five; after all five lane l is left with the sums of e = lane_share(N) l
// + k in v[k], after LAST with (32 or 64) >> LAST values, yet to be summed over
// 32 >> LAST lanes.  The lanes halve the values between them at each level: about
// 2 N shuffles and adds per warp where a full reduction of each value takes 5 N.
template <int N, int FIRST = 0, int LAST = 5, typename V, int SIZE>
__device__ __forceinline__ void reduce_scatter(V (&v)[SIZE], int lane) {
  constexpr int FULL = N > 32 ? 64 : 32;
#pragma unroll
  for (int l = FIRST; l < LAST; ++l) {
    const int h = FULL >> (l + 1), bit = 16 >> l;
    const bool up = lane & bit;
#pragma unroll
    for (int k = 0; k < h; ++k) {
      if (k >= SIZE) continue;
      const V hi = k + h < SIZE ? v[k + h] : V(0);  // (entries past the last are zeros)
      const V keep = up ? hi : v[k], send = up ? v[k] : hi;
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
}

}  // namespace nrcps
