// Operands of the split precisions: a number as two 16-bit pieces, hi + lo.
#pragma once
#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace halves {

// Power-of-2 scale of an FP16 operand whose largest magnitude has the bits maxbits:
// max * scale in [0.5, 1]
__device__ __forceinline__ float fp16_scale(unsigned maxbits) {
  const float m = __uint_as_float(maxbits);
  if (!(m > 0.f)) return 1.f;
  int e;
  frexpf(m, &e);
  return ldexpf(1.f, -e);
}

// hi/lo split of v into two 16-bit values of the operand format
__device__ __forceinline__ void split16(double v, bool fp16, uint16_t* hi, uint16_t* lo) {
  if (fp16) {
    const __half h = __double2half(v);
    *hi = __half_as_ushort(h);
    *lo = __half_as_ushort(__double2half(v - (double)__half2float(h)));
  } else {
    const __nv_bfloat16 h = __double2bfloat16(v);
    *hi = __bfloat16_as_ushort(h);
    *lo = __bfloat16_as_ushort(__double2bfloat16(v - (double)__bfloat162float(h)));
  }
}

}  // namespace halves
