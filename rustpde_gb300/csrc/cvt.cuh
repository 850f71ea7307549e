// cvt.cuh -- FP64 -> FP32 conversion in integer operations.
//
// This GPU converts between FP64 and FP32 at its FP64 rate, two per clock and
// SM; ten integer operations run at a hundred per clock.  Results are those of
// the conversion (round to nearest even); what falls outside FP32's normal
// range, other than zeros, goes through the instruction.
#pragma once
#include <cuda_runtime.h>

namespace rbc {
namespace dev {

__device__ __forceinline__ float to_f32(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const unsigned e = (hi >> 20) & 0x7ffu, s = hi & 0x80000000u;
  if (e - 897u < 254u) {
    const unsigned b = ((e - 896u) << 23) | ((hi & 0xfffffu) << 3) | (lo >> 29);
    // a carry out of the mantissa is the rounding up to the next binade (or to infinity)
    return __uint_as_float(s | (b + (((lo & 0x1fffffffu) + 0x0fffffffu + (b & 1u)) >> 29)));
  }
  if (e <= 872u) return __uint_as_float(s);  // below half of the smallest subnormal
  return (float)d;
}

}  // namespace dev
}  // namespace rbc
