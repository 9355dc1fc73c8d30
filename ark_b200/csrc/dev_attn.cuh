// Merging the pieces of a decode attention.
#pragma once
#include "dev_common.cuh"

namespace arkb {

__device__ __forceinline__ float exp2_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Head `head` = (sequence, K/V head), query head g of its group of G: N consecutive elements from d on, un-normalised, and
// the exp-sum they are to be divided by. N = 1 or a multiple of 4.
template <int N>
__device__ __forceinline__ void merge_pieces(const AttnPieces &pc, const float *ws, int head, int G, int g, int d, float &l, float (&o)[N]) {
    const int stride = G * 132;  // records are 16-byte aligned
    int first, n;
    const float *w0;
    if (pc.span == pc.blocks) {  // every head has runs of its own
        first = head * pc.per_span;
        n = pc.per_span;
        w0 = ws + (int64_t)first * stride;
    } else {
        first = pc.run_of(head * pc.blocks);
        n = pc.run_of(head * pc.blocks + pc.blocks - 1) - first + 1;
        w0 = ws + pc.record(first, head) * stride;
    }
    // the head opens every run but the first: those records are per_run apart
    const float *w1 = ws + (int64_t)(first + 1) * pc.per_run * stride;
    const int64_t step = (int64_t)pc.per_run * stride;
    float mx = -3.402823466e+38f;
    l = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = 0.0f;
    constexpr int B = 4;  // pieces on their way together
    for (int c0 = 0; c0 < n; c0 += B) {
        float2 ml[B];
        float4 v[B][(N + 3) / 4];
#pragma unroll
        for (int c = 0; c < B; ++c) {
            if (c0 + c >= n) continue;
            const float *w = c0 + c == 0 ? w0 : w1 + (c0 + c - 1) * step;
            ml[c] = __ldcg(reinterpret_cast<const float2 *>(w + G * 128 + 2 * g));
            if constexpr (N == 1) {
                v[c][0].x = __ldcg(w + g * 128 + d);
            } else {
#pragma unroll
                for (int i = 0; i < N / 4; ++i) v[c][i] = __ldcg(reinterpret_cast<const float4 *>(w + g * 128 + d) + i);
            }
        }
        float m = mx;
#pragma unroll
        for (int c = 0; c < B; ++c)
            if (c0 + c < n) m = fmaxf(m, ml[c].x);
        if (c0 > 0) {
            const float e = exp2_fast(mx - m);
            l *= e;
#pragma unroll
            for (int i = 0; i < N; ++i) o[i] *= e;
        }
        mx = m;
#pragma unroll
        for (int c = 0; c < B; ++c) {
            if (c0 + c >= n) continue;
            const float e = exp2_fast(ml[c].x - mx);
            l += ml[c].y * e;
            if constexpr (N == 1) {
                o[0] += v[c][0].x * e;
            } else {
#pragma unroll
                for (int i = 0; i < N / 4; ++i) {
                    o[4 * i] += v[c][i].x * e;
                    o[4 * i + 1] += v[c][i].y * e;
                    o[4 * i + 2] += v[c][i].z * e;
                    o[4 * i + 3] += v[c][i].w * e;
                }
            }
        }
    }
}

}  // namespace arkb
