// Element operations of the generic group kernels (kernels_generic.cu, kernels_region.cu).
#pragma once

#include "common.cuh"

#ifdef __CUDACC__
namespace fb {

__device__ __forceinline__ float g_fetch(const void* p, int dtype, int off) {
    switch (dtype) {
        case 0: return __ldg(static_cast<const float*>(p) + off);
        case 1: return static_cast<float>(__ldg(static_cast<const uint8_t*>(p) + off));
        case 2: return static_cast<float>(__ldg(static_cast<const long long*>(p) + off));
        default: return static_cast<float>(__ldg(static_cast<const int*>(p) + off));
    }
}

__device__ __forceinline__ float g_unary(int op, float a, float imm) {
    switch (op) {
        case FB_G_EXP: return expf(a);
        case FB_G_SIGMOID: return sigmoid_f32(a);
        case FB_G_TANH: return tanhf(a);
        case FB_G_RELU: return max_nan(a, 0.0f);
        case FB_G_NEG: return -a;
        case FB_G_CLAMP_MIN: return max_nan(a, imm);
        case FB_G_CLAMP_MAX: return min_nan(a, imm);
        case FB_G_ABS: return fabsf(a);
        case FB_G_SQRT: return sqrtf(a);
        case FB_G_LOG: return logf(a);
        default: return a;
    }
}

__device__ __forceinline__ float g_binary(int op, float a, float b) {
    switch (op) {
        case FB_G_ADD: return __fadd_rn(a, b);
        case FB_G_SUB: return __fsub_rn(a, b);
        case FB_G_MUL: return __fmul_rn(a, b);
        case FB_G_DIV: return __fdiv_rn(a, b);
        case FB_G_MIN: return min_nan(a, b);
        case FB_G_MAX: return max_nan(a, b);
        case FB_G_GT: return a > b ? 1.0f : 0.0f;
        case FB_G_GE: return a >= b ? 1.0f : 0.0f;
        case FB_G_LT: return a < b ? 1.0f : 0.0f;
        case FB_G_LE: return a <= b ? 1.0f : 0.0f;
        case FB_G_EQ: return a == b ? 1.0f : 0.0f;
        case FB_G_NE: return a != b ? 1.0f : 0.0f;
        default: return a;
    }
}

}  // namespace fb
#endif
