// Shared by the two mask kernels (kernels_yolact.cu, kernels_yolact_tc.cu).
#pragma once

#include "common.cuh"

namespace fb {

#ifdef __CUDACC__
// sanitize_coordinates (yolact_mask.py:327-333) followed by "col >= x1 and col < x2" as integer bounds, both in [0, size]: a box
// outside the integers' range would saturate, and the differences that the kernels form with the bounds would wrap.
__device__ __forceinline__ void yolact_crop_range(float a, float b, int size, int& lo, int& hi) {
    float x1 = fminf(a, b);
    float x2 = fmaxf(x1, b);
    x1 = fminf(fmaxf(__fsub_rn(x1, 1.0f), 0.0f), static_cast<float>(size));
    x2 = fmaxf(fminf(__fadd_rn(x2, 1.0f), static_cast<float>(size)), 0.0f);
    lo = static_cast<int>(ceilf(x1));
    hi = static_cast<int>(ceilf(x2));
}
#endif

// masks without the logits, for thresholds in [0.001, 0.999] (kernels_yolact_tc.cu)
int launch_yolact_masks_tc(const float* proto, const float* coef, const float* boxes, int batch, int height, int width, int num_det,
                           float thr, uint8_t* masks, cudaStream_t st);

}  // namespace fb
