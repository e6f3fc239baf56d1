// x = hi + lo of two floats, both parts rounded to nearest bf16.
#pragma once

#include <cuda_bf16.h>

namespace erp {

__device__ __forceinline__ void split_pair(float a, float b, __nv_bfloat162 &hi, __nv_bfloat162 &lo) {
    hi = __floats2bfloat162_rn(a, b);
    lo = __floats2bfloat162_rn(a - __low2float(hi), b - __high2float(hi));
}

}  // namespace erp
