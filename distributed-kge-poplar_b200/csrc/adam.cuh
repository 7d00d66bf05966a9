// What the Adam steps of rows and of dense parameters share.
#pragma once

#include <cuda_runtime.h>

namespace kge {

struct AdamParams {
    float beta_m;
    float beta_v;
    float one_minus_beta_m;
    float one_minus_beta_v;
    float epsilon;
    float weight_decay;
};
// a x + b y with the first product unrounded.  Which one the addition takes in is the compiler's choice in every kernel anew
// unless it is written out, and an L1 model, whose gradients are what rounding leaves of a sum, carries a last bit on: rows
// and dense parameters have one form each in all kernels.
__device__ __forceinline__ float weighted_sum(float a, float x, float b, float y) { return __fmaf_rn(a, x, __fmul_rn(b, y)); }

}  // namespace kge
