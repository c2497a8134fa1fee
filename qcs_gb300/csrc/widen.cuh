// widen.cuh -- floats to doubles without the FP64 pipe.
//
// That pipe (half a lane per clock and quarter of an SM: 64 cycles a warp
// instruction) also does the conversions from float, two of the four or five
// instructions of an amplitude's square.  A zero or a normal number is widened
// exactly by five integer operations instead.
#pragma once

#include "common.cuh"

namespace qcs {

// |x| as a double; PLAIN: of a zero or a normal number, by its bits.
template <bool PLAIN>
__device__ __forceinline__ double to64(float x) {
  if (!PLAIN) return fabs((double)x);
  const unsigned w = __float_as_uint(x) << 1;
  return __hiloint2double(w ? (int)((w >> 4) + 0x38000000u) : 0, (int)(w << 28));
}

// Whether all of the numbers seen are zero or normal.
struct PlainTest {
  unsigned lo = 0xffffffffu, hi = 0;  // of the bits without the sign, less one
  __device__ __forceinline__ void see(float x) {
    const unsigned w = (__float_as_uint(x) << 1) - 1u;  // zero: the largest
    lo = min(lo, w);
    hi = max(hi, w + 1u);
  }
  __device__ __forceinline__ bool plain() const { return lo >= 0xffffffu && hi < 0xff000000u; }
};

}  // namespace qcs
