// Rounding of fp32 values to tf32 operands, shared by everything that writes them.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace kxc_b200 {

// fp32 storage of a tf32 value: the low 13 mantissa bits rounded away, nearest even (infinities and NaN as they are)
__device__ __forceinline__ float tf32_rne(float x) {
    uint32_t u = __float_as_uint(x);
    if ((u & 0x7f800000u) != 0x7f800000u) u = (u + 0xfffu + ((u >> 13) & 1u)) & 0xffffe000u;
    return __uint_as_float(u);
}

// The tf32 rounding of what hi = tf32_rne(x) drops: a*b ~ a_hi*b_hi + a_hi*b_lo + a_lo*b_hi then carries about 21 bits of each
// operand instead of 11. A non-finite value lives in the high part only: inf - inf would be NaN.
__device__ __forceinline__ float tf32_low_part(float x, float hi) {
    return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u ? 0.0f : tf32_rne(__fsub_rn(x, hi));
}

}  // namespace kxc_b200
