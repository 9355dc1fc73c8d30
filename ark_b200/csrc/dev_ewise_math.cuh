// Arithmetic of the elementwise operators on N fp32 values, shared by the elementwise walkers and the row chains.
#pragma once
#include "dev_common.cuh"

namespace arkb {

// FAST: results are rounded to a 16-bit type, so the hardware exp2 / reciprocal
// approximations (relative error ~1e-6) are used for gelu / sigmoid / silu.
template <int N, bool FAST>
__device__ __forceinline__ void ewise_math(int op, float scalar, const float (&x)[N], const float (&y)[N],
                                           float (&r)[N]) {
    switch (op) {
        case EW_GELU:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = FAST ? apply_act_fast(ACT_GELU, x[i]) : gelu_f(x[i]);
            break;
        case EW_EXP:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = expf(x[i]);
            break;
        case EW_RELU:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] > 0.0f ? x[i] : 0.0f;
            break;
        case EW_RSQRT:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = 1.0f / sqrtf(x[i]);
            break;
        case EW_SIGMOID:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = FAST ? fast_sigmoid(x[i]) : sigmoid_f(x[i]);
            break;
        case EW_SILU:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] * (FAST ? fast_sigmoid(x[i]) : sigmoid_f(x[i]));
            break;
        case EW_SQRT:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = sqrtf(x[i]);
            break;
        case EW_ADD:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] + y[i];
            break;
        case EW_SUB:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] - y[i];
            break;
        case EW_MUL:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] * y[i];
            break;
        case EW_DIV:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] / y[i];
            break;
        case EW_SCALAR_ASSIGN:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = scalar;
            break;
        case EW_SCALAR_ADD:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] + scalar;
            break;
        case EW_SCALAR_MUL:
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i] * scalar;
            break;
        case EW_ROPE:
            // complex multiply on adjacent pairs (ark/include/kernels/embedding.h:14-37)
            if constexpr (N >= 2) {
#pragma unroll
                for (int i = 0; i < N; i += 2) {
                    r[i] = x[i] * y[i] - x[i + 1] * y[i + 1];
                    r[i + 1] = x[i] * y[i + 1] + x[i + 1] * y[i];
                }
            }
            break;
        default:  // EW_COPY / EW_CAST
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = x[i];
            break;
    }
}

}  // namespace arkb
