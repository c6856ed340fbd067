// What the CUDA-core backward kernels share about the softmax they form again from lse.
#pragma once

#include <float.h>

// p = exp(s - lse) over the window that lse was taken over adds up to 1 but for rounding: that of lse, of the logits
// beside it (both half an ulp of numbers about as large as lse) and of the exponentials.  Taken out, that rounding does
// not meet the cancellation in dP - delta.  The factor that p is multiplied by, for a row whose p add up to `sum`: a sum
// further from 1 than rounding can bring it is an lse over more than the window, whose p are what exp(s - lse) says.
__device__ __forceinline__ float na2d_row_factor(float sum, float lse) {
    return fabsf(sum - 1.f) < 4.f * FLT_EPSILON * (4.f + fabsf(lse)) ? 1.f / sum : 1.f;
}
