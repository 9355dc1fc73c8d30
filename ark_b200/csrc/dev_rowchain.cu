// Row chains: operators that follow each other on the same [rows, cols] tensor (embedding lookup, elementwise
// operators with a tensor or with one row for all, rmsnorm, layernorm, softmax, a final cast; or the sum of a matmul's
// split-K partials in front) as one stage.
//
// Each operator on its own is a pass over memory: what bounds it is HBM, and behind it stands a grid barrier. Here a
// group of warps keeps a row in registers, packed in the storage type (up to 8 16-byte vectors per lane), and applies
// the whole list to it. Every result is still rounded to the storage type and stored, so later readers, and the host,
// find what the separate stages would have left; the reads of intermediates and the barriers are gone. Groups of a CTA
// work on different rows and do not wait for one another, so one row's loads overlap another one's arithmetic.
// 8192 x 4096 bf16, embedding lookup to softmax and cast: 471 us as eight stages, 254 us so. Split-K sum, residual and norm of
// 16 rows of 8192 in a decode step: 45 -> 29 us.
#include <type_traits>

#include "dev_common.cuh"
#include "dev_ewise_math.cuh"
#include "dev_funcs.h"

namespace arkb {

namespace {

template <typename T>
struct Row {
    static constexpr int V = 16 / sizeof(T);
    static __device__ __forceinline__ void unpack(const uint4 &q, float (&f)[V]) {
        const T *e = reinterpret_cast<const T *>(&q);
#pragma unroll
        for (int i = 0; i < V; ++i) f[i] = to_f32(e[i]);
    }
    static __device__ __forceinline__ void pack(uint4 &q, const float (&f)[V]) {
        T *e = reinterpret_cast<T *>(&q);
#pragma unroll
        for (int i = 0; i < V; ++i) e[i] = from_f32<T>(f[i]);
    }
};

__device__ __forceinline__ float chain_exp(float x, bool half_type) { return half_type ? __expf(x) : expf(x); }

// N: 16-byte vectors of a row per lane. Few-row chains (a CTA per row) take the 2-vector form: it uses half the registers,
// and what a stage function uses beyond the scratch registers it saves on entry, 512 threads at a time (8-vector form
// about 3 us where the plan's matmuls leave little L1).
template <typename T, int N>
__device__ __noinline__ void rowchain_typed(const RowChainArgs &a, int p, int P) {
    using R = Row<T>;
    constexpr int V = R::V, WPC = kThreads / 32;
    constexpr bool kHalf = sizeof(T) == 2;
    __shared__ float red[2][WPC];
    const int G = a.warps, nv = a.cols / V, n_ops = a.n_ops;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = warp / G, groups = WPC / G;
    const int li = warp % G * 32 + lane, lstride = 32 * G;
    const float inv_cols = 1.0f / (float)a.cols;
    int turn = 0;  // a slot of `red` is written again only behind the barrier of the reduction in between
    auto across = [&](float v, bool is_max) -> float {
        v = is_max ? warp_max(v) : warp_sum(v);
        if (G == 1) return v;
        float *slot = red[turn];
        turn ^= 1;
        if (lane == 0) slot[warp] = v;
        named_barrier(1 + group, G * 32);
        float r = slot[group * G];
        for (int i = 1; i < G; ++i) r = is_max ? fmaxf(r, slot[group * G + i]) : r + slot[group * G + i];
        return r;
    };
    auto each = [&](auto &&f) {
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (li + j * lstride < nv) f(j, (li + j * lstride) * V);
    };
    const int64_t units = (int64_t)a.rows * a.segs;
    for (int64_t u = (int64_t)group * P + p; u < units; u += (int64_t)P * groups) {
        const int64_t row = u / a.segs, c0 = (u - row * a.segs) * a.cols;  // first column of the segment
        const int64_t off = u * a.cols;                                    // segments of a dense tensor follow each other
        uint4 x[N];
        if (a.head == RH_SUM) {
            const int64_t total = units * a.cols;
            const int splits = a.splits, act = a.act;
            const T *add = a.add ? reinterpret_cast<const T *>(a.add) + off : nullptr;
            T *out = reinterpret_cast<T *>(a.out) + off;
            const float *ws = a.ws + off;
            each([&](int j, int e) {
                // the partials in k order, several of them in flight
                constexpr int B = N == 2 ? 8 : 4;
                float f[V] = {};
                for (int s0 = 0; s0 < splits; s0 += B) {
#pragma unroll
                    for (int i = 0; i < V / 4; ++i) {
                        float4 q[B];
#pragma unroll
                        for (int s = 0; s < B; ++s)
                            if (s0 + s < splits) q[s] = __ldcg(reinterpret_cast<const float4 *>(ws + (s0 + s) * total + e) + i);
#pragma unroll
                        for (int s = 0; s < B; ++s)
                            if (s0 + s < splits) { f[i * 4] += q[s].x; f[i * 4 + 1] += q[s].y; f[i * 4 + 2] += q[s].z; f[i * 4 + 3] += q[s].w; }
                    }
                }
                if (add) {
                    float g[V];
                    load_vec<T, V>(add + e, g);
#pragma unroll
                    for (int i = 0; i < V; ++i) f[i] += g[i];
                }
#pragma unroll
                for (int i = 0; i < V; ++i) f[i] = apply_act_fast(act, f[i]);
                R::pack(x[j], f);
            });
            each([&](int j, int e) { *reinterpret_cast<uint4 *>(out + e) = x[j]; });
        } else {
            int64_t from = off;
            if (a.head == RH_GATHER) {
                int64_t r = a.idx[row];
                if (r < 0) r += a.num_emb;
                from = r * a.src_ld + c0;
            }
            const T *src = reinterpret_cast<const T *>(a.src) + from;
            each([&](int j, int e) { x[j] = ldg16_stream(src + e); });
            if (a.head == RH_GATHER) {
                T *out = reinterpret_cast<T *>(a.out) + off;
                each([&](int j, int e) { *reinterpret_cast<uint4 *>(out + e) = x[j]; });
            }
        }
        for (int k = 0; k < n_ops; ++k) {
            // An operand may be an earlier result of the chain, which this thread has just stored: the loads below, which
            // the compiler takes for reads of no memory, stay behind those stores.
            asm volatile("" ::: "memory");
            // what the loops below use is copied out of the record: their stores might alias it
            const RowChainOp &o = a.ops[k];
            const int kind = o.kind, op = o.op, mode = o.other_mode;
            const bool swapped = o.swapped != 0;
            const float scalar = o.scalar;
            T *out = reinterpret_cast<T *>(o.out) + off;
            uint4 y[N];
            if (mode == 1) {
                const T *other = reinterpret_cast<const T *>(o.other) + off;
                each([&](int j, int e) { y[j] = ldg16_stream(other + e); });
            } else if (mode == 2) {
                const T *other = reinterpret_cast<const T *>(o.other) + c0;
                each([&](int j, int e) { y[j] = *reinterpret_cast<const uint4 *>(other + e); });
            }
            if (kind == RC_CAST) {
                void *dst = o.out;
                each([&](int j, int e) {
                    float f[V];
                    R::unpack(x[j], f);
                    if (op == DT_F32) store_vec<float, V>(reinterpret_cast<float *>(dst) + off + e, f);
                    else if (op == DT_F16) store_vec<__half, V>(reinterpret_cast<__half *>(dst) + off + e, f);
                    else store_vec<__nv_bfloat16, V>(reinterpret_cast<__nv_bfloat16 *>(dst) + off + e, f);
                });
                break;  // the last operator of its chain
            }
            if (kind == RC_EWISE) {
                // one loop per operator: chosen once, not per vector
                auto run = [&](auto code) {
                    each([&](int j, int) {
                        float f[V], g[V], r[V];
                        R::unpack(x[j], f);
                        if (mode == 3) {
#pragma unroll
                            for (int i = 0; i < V; ++i) g[i] = f[i];
                        } else {
                            R::unpack(y[j], g);
                        }
                        constexpr int kOp = decltype(code)::value;
                        if ((kOp == EW_SUB || kOp == EW_DIV) && swapped) ewise_math<V, kHalf>(kOp, scalar, g, f, r);
                        else ewise_math<V, kHalf>(kOp, scalar, f, g, r);
                        R::pack(x[j], r);
                    });
                };
                switch (op) {
                    case EW_GELU: run(std::integral_constant<int, EW_GELU>()); break;
                    case EW_EXP: run(std::integral_constant<int, EW_EXP>()); break;
                    case EW_RELU: run(std::integral_constant<int, EW_RELU>()); break;
                    case EW_RSQRT: run(std::integral_constant<int, EW_RSQRT>()); break;
                    case EW_SIGMOID: run(std::integral_constant<int, EW_SIGMOID>()); break;
                    case EW_SILU: run(std::integral_constant<int, EW_SILU>()); break;
                    case EW_SQRT: run(std::integral_constant<int, EW_SQRT>()); break;
                    case EW_ADD: run(std::integral_constant<int, EW_ADD>()); break;
                    case EW_SUB: run(std::integral_constant<int, EW_SUB>()); break;
                    case EW_MUL: run(std::integral_constant<int, EW_MUL>()); break;
                    case EW_DIV: run(std::integral_constant<int, EW_DIV>()); break;
                    case EW_SCALAR_ADD: run(std::integral_constant<int, EW_SCALAR_ADD>()); break;
                    case EW_SCALAR_MUL: run(std::integral_constant<int, EW_SCALAR_MUL>()); break;
                    default: break;
                }
            } else {
                const T *wgt = reinterpret_cast<const T *>(o.weight);
                const bool wide = o.weight_f32 != 0;
                if (mode == 1) {  // rmsnorm of the sum with a residual, which is kept as well
                    T *sum = reinterpret_cast<T *>(o.out2) + off;
                    each([&](int j, int) {
                        float f[V], g[V];
                        R::unpack(x[j], f);
                        R::unpack(y[j], g);
#pragma unroll
                        for (int i = 0; i < V; ++i) f[i] += g[i];
                        R::pack(x[j], f);
                    });
                    each([&](int j, int e) { *reinterpret_cast<uint4 *>(sum + e) = x[j]; });
                }
                // the weight row is on its way while the statistics are taken
                if (wgt && !wide) each([&](int j, int e) { y[j] = *reinterpret_cast<const uint4 *>(wgt + e); });
                float mul, sub = 0.0f;
                if (kind == RC_RMSNORM) {
                    float s = 0.0f;
                    each([&](int j, int) {
                        float f[V];
                        R::unpack(x[j], f);
#pragma unroll
                        for (int i = 0; i < V; ++i) s += f[i] * f[i];
                    });
                    mul = 1.0f / sqrtf(across(s, false) * inv_cols + scalar);
                } else if (kind == RC_LAYERNORM) {
                    float s = 0.0f;
                    each([&](int j, int) {
                        float f[V];
                        R::unpack(x[j], f);
#pragma unroll
                        for (int i = 0; i < V; ++i) s += f[i];
                    });
                    sub = across(s, false) * inv_cols;
                    float var = 0.0f;
                    each([&](int j, int) {
                        float f[V];
                        R::unpack(x[j], f);
#pragma unroll
                        for (int i = 0; i < V; ++i) var += (f[i] - sub) * (f[i] - sub);
                    });
                    mul = 1.0f / sqrtf(across(var, false) * inv_cols + scalar);
                } else {
                    float m = -3.402823466e+38f;
                    each([&](int j, int) {
                        float f[V];
                        R::unpack(x[j], f);
#pragma unroll
                        for (int i = 0; i < V; ++i) m = fmaxf(m, f[i] * scalar);
                    });
                    sub = across(m, true);
                    float s = 0.0f;
                    each([&](int j, int) {
                        float f[V];
                        R::unpack(x[j], f);
#pragma unroll
                        for (int i = 0; i < V; ++i) s += chain_exp(f[i] * scalar - sub, kHalf);
                    });
                    mul = 1.0f / across(s, false);
                }
                each([&](int j, int e) {
                    float f[V];
                    R::unpack(x[j], f);
                    if (kind == RC_SOFTMAX) {
#pragma unroll
                        for (int i = 0; i < V; ++i) f[i] = chain_exp(f[i] * scalar - sub, kHalf) * mul;
                    } else {
#pragma unroll
                        for (int i = 0; i < V; ++i) f[i] = (f[i] - sub) * mul;
                        if (wgt) {
                            float g[V];
                            if (wide) load_vec_cached<float, V>(reinterpret_cast<const float *>(wgt) + e, g);
                            else R::unpack(y[j], g);
#pragma unroll
                            for (int i = 0; i < V; ++i) f[i] *= g[i];
                        }
                    }
                    R::pack(x[j], f);
                });
            }
            each([&](int j, int e) { *reinterpret_cast<uint4 *>(out + e) = x[j]; });
            if (o.copy) {
                T *copy = reinterpret_cast<T *>(o.copy) + off;
                each([&](int j, int e) { *reinterpret_cast<uint4 *>(copy + e) = x[j]; });
            }
        }
    }
}

template <typename T>
__device__ __forceinline__ void rowchain_sized(const RowChainArgs &a, int p, int P) {
    // units go to all CTAs' first groups, then to their second ones: warps without a unit do not enter
    if ((int64_t)(threadIdx.x / 32 / a.warps) * P + p >= (int64_t)a.rows * a.segs) return;
    if (a.cols <= 2 * 32 * a.warps * Row<T>::V) rowchain_typed<T, 2>(a, p, P);
    else if (a.cols <= 4 * 32 * a.warps * Row<T>::V) rowchain_typed<T, 4>(a, p, P);
    else rowchain_typed<T, 8>(a, p, P);
}

}  // namespace

__device__ __noinline__ void run_rowchain(const RowChainArgs &a, int p, int P) {
    switch (a.dtype) {
        case DT_F32: rowchain_sized<float>(a, p, P); break;
        case DT_F16: rowchain_sized<__half>(a, p, P); break;
        default: rowchain_sized<__nv_bfloat16>(a, p, P); break;
    }
}

}  // namespace arkb
