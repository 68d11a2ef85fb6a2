// A float as a double without the FP64 pipe.
#pragma once

#include <cuda_runtime.h>

namespace lat {

// (double)f by integer instructions: a conversion takes the FP64 pipe, which bounds
// the FP32 steps with diagnostics (64 lattices of 64^3 in a batch, diagnostics at every
// step: 465 us a step with conversions, 447 without).
__device__ __forceinline__ double widen(float f)
{
    const unsigned s = __float_as_uint(f) & 0x80000000u;
    unsigned m = __float_as_uint(f) & 0x7fffffffu, bias = m >= 0x7f800000u ? 2 * 896u : 896u;   // Inf and NaN: the largest exponent
    if (m < 0x00800000u) {   // zero and subnormals, as multiples of 2^-64
        m = __float_as_uint(fabsf(f) * 0x1p64f);
        bias = m != 0 ? 896u - 64u : 0u;
    }
    return __hiloint2double((int)(s | ((m >> 3) + (bias << 20))), (int)(m << 29));
}

}  // namespace lat
