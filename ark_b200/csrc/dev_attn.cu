// Attention of one new token per sequence against a K/V cache (the decode
// step): out[b, h] = softmax(scale * q[b, h] . K[b, h / G]^T) . V[b, h / G]
// with G = Hq / Hkv query heads sharing a K/V head and a head size of 128.
// The reference builds this from two Matmuls, a scale and a softmax
// (examples/llama/model.py:336-444), i.e. several tasks with barriers between
// them; at one query row per head those tasks are nothing but a read of the
// cache, so this stage does the whole thing around that read.
//
// What bounds it is HBM. Three things used to keep it a factor of five away (16 sequences of 4096 keys, 64 / 8 heads:
// 202 us for 268 MB): the multiply-adds of 8 query heads on the CUDA cores, phases of a CTA (scores, softmax, output)
// that waited for one another with the memory idle, and whole chunks handed to CTAs, so that 160 chunks on 148 CTAs took
// two rounds. Here:
//  * The cache is a list of 16-key blocks, (sequence, K/V head) by (sequence, K/V head), cut into runs of equal length,
//    one per CTA. The pieces of a head (one from each run that holds some of it) are merged afterwards: fp32 output,
//    maximum and exp-sum per piece.
//  * Every warp works alone on every 12th block of a run: the scores of 16 keys x 8 heads and the output are 32 small
//    tensor-core products (mma.sync m16n8k16, heads as its 8 columns: there is nothing a larger tile could fill), an
//    online softmax sits in between, and no warp waits for another one until the piece is complete.
//  * Probabilities stay fp32 values: each is the sum of three 16-bit ones, see split3, smallest first. (With two parts, 2^-17 of
//    bf16, ten times as many bf16 outputs were not the nearest value of their type: 0.2 % instead of 0.02 %.) A block's
//    products are added to the output in fp32 arithmetic: the tensor core cuts off what it adds to an accumulator.
//  * K and V go through shared memory only as a queue: a lane brings in exactly the 16-byte pieces that it will use as
//    operand fragments (the head dimension may be permuted alike in K and Q, or in V and the output), a block of K and
//    one of V ahead.
// One B200, bf16: 16 sequences of 4096 keys, 64 / 8 heads 200 -> 74 us (3.6 TB/s); 5 sequences of 4096 keys, 32 heads 85 us.
#include <type_traits>

#include "dev_common.cuh"
#include "dev_funcs.h"

namespace arkb {

namespace {

constexpr int kHeadDim = 128;
constexpr int kMaxGroup = 8;                  // query heads per K/V head
constexpr int kWarps = 12;                    // warps that take part: 96 KiB of queues, with 48 to 96 KiB on their way
constexpr int kDepth = 2;                     // blocks in a warp's queue: one of K, one of V
constexpr int kBlockBytes = 16 * kHeadDim * 2;
constexpr int kRingBytes = kWarps * kDepth * kBlockBytes;
constexpr int kQBytes = kMaxGroup * kHeadDim * 2;
constexpr int kRedBytes = kWarps * kMaxGroup * kHeadDim * 4;  // warps' outputs; over the queues, which are empty by then
static_assert(kRedBytes <= kRingBytes, "the warps' outputs reuse the queues");
static_assert(kRingBytes + kQBytes + 2 * kWarps * kMaxGroup * 4 <= kDecodeAttnSmemBytes, "shared memory of the stage");

__device__ __forceinline__ void fetch16(uint32_t dst, const void *src, const void *any, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(in ? src : any), "r"(in ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void fetch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void fetch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }
__device__ __forceinline__ uint4 lds16(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}

__device__ __forceinline__ float exp2_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
template <typename T>
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (std::is_same_v<T, __nv_bfloat16>)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 8 x 8 matrix of 16-bit values, a row per four lanes, transposed across the warp
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
template <typename T>
__device__ __forceinline__ uint32_t pack2(T a, T b) {
    uint32_t r;
    T *e = reinterpret_cast<T *>(&r);
    e[0] = a;
    e[1] = b;
    return r;
}
constexpr float kLowest = -3.402823466e+38f;
constexpr float kLog2e = 1.4426950408889634f;

// Two probabilities as three 16-bit values each, packed in pairs. bf16: the 24 bits of the fp32 value cut into three times
// eight, exactly. fp16: rounded value, rounded remainder and what is left, 33 bits (of values scaled by 2^14, so that
// the remainders stay clear of the subnormals; the scale cancels in the division by the sum). bf16 needs no scale and
// gets none: outputs near the type's largest value would overflow.
template <typename T>
constexpr float kScale = std::is_same_v<T, __nv_bfloat16> ? 1.0f : 16384.0f;
template <typename T>
__device__ __forceinline__ void split3(float x, float y, uint32_t (&part)[3]) {
    if constexpr (std::is_same_v<T, __nv_bfloat16>) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            part[i] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
            x -= __uint_as_float(__float_as_uint(x) & 0xffff0000u);
            y -= __uint_as_float(__float_as_uint(y) & 0xffff0000u);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const T a = from_f32<T>(x), b = from_f32<T>(y);
            part[i] = pack2<T>(a, b);
            x -= to_f32(a);
            y -= to_f32(b);
        }
    }
}

// A warp's blocks with plain arithmetic, as the chunk form does it: for infinite or NaN operands (the parts of a probability
// may be zero, and 0 * inf is NaN) and scores or outputs beyond fp32 that scaling q first, or single products, keep inside.
// Leaves the output of head h in out[h][128], maxima and exp-sums in wm[h] and wl[h].
template <typename T>
__device__ __noinline__ void attn_plain_blocks(const DecodeAttnArgs &a, const T *kbase, const T *vbase, const T *qs, int first, int n_mine,
                                               float *out, float *wm, float *wl) {
    const int lane = threadIdx.x & 31, G = a.Hq / a.Hkv;
    for (int h = 0; h < G; ++h) {
        float q[4], m = kLowest, l = 0.0f, acc[4] = {};
#pragma unroll
        for (int e = 0; e < 4; ++e) q[e] = to_f32(qs[h * kHeadDim + lane * 4 + e]) * a.scale;
        for (int pass = 0; pass < 2; ++pass)  // the maximum; exponentials and output
            for (int i = 0; i < n_mine; ++i) {
                const int key0 = (first + i * kWarps) * 16, keys = min(16, a.T - key0);
                for (int r = 0; r < keys; ++r) {
                    float k[4], s = 0.0f;
                    load_vec<T, 4>(kbase + (int64_t)(key0 + r) * a.k_ld + lane * 4, k);
#pragma unroll
                    for (int e = 0; e < 4; ++e) s += q[e] * k[e];
                    s = warp_sum(s);
                    if (pass == 0) {
                        m = fmaxf(m, s);
                    } else {
                        const float p = __expf(s - m) * kScale<T>;
                        float v[4];
                        load_vec<T, 4>(vbase + (int64_t)(key0 + r) * a.v_ld + lane * 4, v);
                        l += p;
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[e] += p * v[e];
                    }
                }
            }
        *reinterpret_cast<float4 *>(out + h * kHeadDim + lane * 4) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        if (lane == 0) {
            wm[h] = fmaxf(m * kLog2e, kLowest);
            wl[h] = l;
        }
    }
}

template <typename T>
__device__ __noinline__ void attn_pieces(const DecodeAttnArgs &a, int p, char *smem) {
    T *qs = reinterpret_cast<T *>(smem + kRingBytes);                      // [8][128], rows of absent heads zero
    float *wm = reinterpret_cast<float *>(smem + kRingBytes + kQBytes);    // [warp][8]: maximum (log2 units), then exp-sum
    float *wl = wm + kWarps * kMaxGroup;
    float *red = reinterpret_cast<float *>(smem);                          // [warp][G][128]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;                                 // row group and place in it of the fragments
    const int G = a.Hq / a.Hkv, nb = a.pieces.blocks;
    const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem) + warp * (kDepth * kBlockBytes) + lane * 16;
    const float to_log2 = a.scale * kLog2e;
    const int run0 = a.pieces.begin(p), run1 = p + 1 < a.pieces.runs ? a.pieces.begin(p + 1) : a.B * a.Hkv * nb;
    for (int blk = run0; blk < run1;) {
        const int head = blk / nb, kb0 = blk - head * nb, kb1 = min(nb, kb0 + run1 - blk);  // blocks [kb0, kb1) of this head
        blk += kb1 - kb0;
        const int kvh = head % a.Hkv, b = head / a.Hkv;
        const T *kbase = reinterpret_cast<const T *>(a.k) + (int64_t)b * a.k_stride_b + (int64_t)kvh * a.k_stride_h;
        const T *vbase = reinterpret_cast<const T *>(a.v) + (int64_t)b * a.v_stride_b + (int64_t)kvh * a.v_stride_h;
        const int n_mine = kb1 - kb0 > warp ? (kb1 - kb0 - warp + kWarps - 1) / kWarps : 0;
        // K of a block: rows g and g + 8, 16 bytes at 32 i + 8 t. V: rows 2 t, 2 t + 1, 2 t + 8, 2 t + 9, 16 bytes at 64 h + 8 g.
        auto fetch_k = [&](int i) {
            if (i < n_mine) {
                const int key = (kb0 + warp + i * kWarps) * 16 + g;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    fetch16(ring + c * 512, kbase + (int64_t)(key + (c & 1) * 8) * a.k_ld + (c >> 1) * 32 + t * 8, kbase,
                            key + (c & 1) * 8 < a.T);
            }
            fetch_commit();
        };
        auto fetch_v = [&](int i) {
            if (i < n_mine) {
                const int key = (kb0 + warp + i * kWarps) * 16 + 2 * t;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const int r = key + (c & 1) + (c >> 1 & 1) * 8;
                    fetch16(ring + kBlockBytes + c * 512, vbase + (int64_t)r * a.v_ld + (c >> 2) * 64 + g * 8, vbase, r < a.T);
                }
            }
            fetch_commit();
        };
        named_barrier(1, kWarps * 32);  // the queues' memory is no longer read as the outputs of the piece before
        fetch_k(0);
        fetch_v(0);
        const T *qb = reinterpret_cast<const T *>(a.q) + (int64_t)b * a.q_stride_b + (int64_t)kvh * G * a.q_stride_h;
        if (tid < kMaxGroup * kHeadDim / 8) {
            const int h = tid >> 4, v = tid & 15;
            uint4 q4 = make_uint4(0, 0, 0, 0);
            if (h < G) {
                q4 = *reinterpret_cast<const uint4 *>(qb + (int64_t)h * a.q_stride_h + v * 8);
                if (a.rope) {
                    // rotary embedding of the new token's query (complex multiply of adjacent pairs with the position's
                    // (cos, sin) pairs), rounded like the separate operator would have stored it
                    float f[8], c[8];
                    unpack8<T>(q4, f);
                    unpack8<T>(*reinterpret_cast<const uint4 *>(reinterpret_cast<const T *>(a.rope) + v * 8), c);
                    T *e = reinterpret_cast<T *>(&q4);
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        e[i] = from_f32<T>(f[i] * c[i] - f[i + 1] * c[i + 1]);
                        e[i + 1] = from_f32<T>(f[i] * c[i + 1] + f[i + 1] * c[i]);
                    }
                }
            }
            *reinterpret_cast<uint4 *>(qs + h * kHeadDim + v * 8) = q4;
        }
        named_barrier(1, kWarps * 32);
        uint4 qf[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) qf[i] = *reinterpret_cast<const uint4 *>(qs + g * kHeadDim + i * 32 + t * 8);
        float o[8][4] = {};                        // [4 h + r]: elements 64 h + 8 g + 2 r (, + 1) of heads 2 t, 2 t + 1 (, and again)
        float m0 = kLowest, m1 = kLowest, l0 = 0.0f, l1 = 0.0f;  // heads 2 t and 2 t + 1
        for (int i = 0; i < n_mine; ++i) {
            fetch_wait<1>();  // K of block i; V of block i is on its way
            float c[4] = {};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint4 x = lds16(ring + k * 1024), y = lds16(ring + k * 1024 + 512);
                float u[4] = {}, v[4] = {};
                mma16816<T>(u, x.x, y.x, x.y, y.y, qf[k].x, qf[k].y);
                mma16816<T>(v, x.z, y.z, x.w, y.w, qf[k].z, qf[k].w);
#pragma unroll
                for (int e = 0; e < 4; ++e) c[e] += u[e] + v[e];
            }
            fetch_k(i + 1);
            const int key = (kb0 + warp + i * kWarps) * 16 + g;
            const bool in0 = key < a.T, in1 = key + 8 < a.T;
            const float s0 = in0 ? c[0] * to_log2 : -INFINITY, s1 = in0 ? c[1] * to_log2 : -INFINITY;
            const float s2 = in1 ? c[2] * to_log2 : -INFINITY, s3 = in1 ? c[3] * to_log2 : -INFINITY;
            float x0 = fmaxf(s0, s2), x1 = fmaxf(s1, s3);
#pragma unroll
            for (int w = 4; w < 32; w *= 2) {
                x0 = fmaxf(x0, __shfl_xor_sync(0xffffffffu, x0, w));
                x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, w));
            }
            x0 = fmaxf(x0, m0);
            x1 = fmaxf(x1, m1);
            if (__any_sync(0xffffffffu, x0 > m0 || x1 > m1)) {
                const float f0 = exp2_fast(m0 - x0), f1 = exp2_fast(m1 - x1);
                l0 *= f0;
                l1 *= f1;
                m0 = x0;
                m1 = x1;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    o[n][0] *= f0;
                    o[n][1] *= f1;
                    o[n][2] *= f0;
                    o[n][3] *= f1;
                }
            }
            // the distance to the maximum in one rounding
            const float p0 = exp2_fast(in0 ? fmaf(c[0], to_log2, -m0) : -INFINITY) * kScale<T>;
            const float p1 = exp2_fast(in0 ? fmaf(c[1], to_log2, -m1) : -INFINITY) * kScale<T>;
            const float p2 = exp2_fast(in1 ? fmaf(c[2], to_log2, -m0) : -INFINITY) * kScale<T>;
            const float p3 = exp2_fast(in1 ? fmaf(c[3], to_log2, -m1) : -INFINITY) * kScale<T>;
            l0 += p0 + p2;
            l1 += p1 + p3;
            uint32_t lo[3], hi[3];  // parts for keys g and g + 8, turned into columns of heads
            split3<T>(p0, p1, lo);
            split3<T>(p2, p3, hi);
#pragma unroll
            for (int e = 0; e < 3; ++e) {
                lo[e] = transpose8x8(lo[e]);
                hi[e] = transpose8x8(hi[e]);
            }
            fetch_wait<1>();
            const uint32_t vs = ring + kBlockBytes;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 v0 = lds16(vs + h * 2048), v1 = lds16(vs + h * 2048 + 512), v2 = lds16(vs + h * 2048 + 1024), v3 = lds16(vs + h * 2048 + 1536);
                const uint32_t r0[4] = {v0.x, v0.y, v0.z, v0.w}, r1[4] = {v1.x, v1.y, v1.z, v1.w};
                const uint32_t r2[4] = {v2.x, v2.y, v2.z, v2.w}, r3[4] = {v3.x, v3.y, v3.z, v3.w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint32_t a0 = __byte_perm(r0[r], r1[r], 0x5410), a1 = __byte_perm(r0[r], r1[r], 0x7632);
                    const uint32_t a2 = __byte_perm(r2[r], r3[r], 0x5410), a3 = __byte_perm(r2[r], r3[r], 0x7632);
                    float u[4] = {};
#pragma unroll
                    for (int e = 2; e >= 0; --e) mma16816<T>(u, a0, a1, a2, a3, lo[e], hi[e]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) o[h * 4 + r][e] += u[e];
                }
            }
            fetch_v(i + 1);
        }
        fetch_wait<0>();
#pragma unroll
        for (int w = 4; w < 32; w *= 2) {  // a warp's exp-sums are spread over its lanes
            l0 += __shfl_xor_sync(0xffffffffu, l0, w);
            l1 += __shfl_xor_sync(0xffffffffu, l1, w);
        }
        float z = l0 * 0.0f + l1 * 0.0f;  // NaN where something is not finite
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) z = fmaf(o[n][e], 0.0f, z);
        // A sum below the largest score's own 1: all scores are -inf, maybe only before their scale, or so large (2^24) that the
        // rounding of the maximum takes whole powers of two from every exponential.
        const bool lost = n_mine > 0 && fminf(l0, l1) < 0.5f * kScale<T>;
        if (__any_sync(0xffffffffu, z != z || lost)) {
            float *mine = reinterpret_cast<float *>(smem + warp * (kDepth * kBlockBytes));  // this warp's queue, empty by now
            __syncwarp();
            attn_plain_blocks<T>(a, kbase, vbase, qs, kb0 + warp, n_mine, mine, wm + warp * kMaxGroup, wl + warp * kMaxGroup);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    if (2 * t + c < G) {
                        const float *src = mine + (2 * t + c) * kHeadDim + i / 4 * 64 + 8 * g + i % 4 * 2;
                        o[i][c] = src[0];
                        o[i][c + 2] = src[1];
                    }
        } else {
            if (g == 0) {
                wm[warp * kMaxGroup + 2 * t] = m0;
                wm[warp * kMaxGroup + 2 * t + 1] = m1;
                wl[warp * kMaxGroup + 2 * t] = l0;
                wl[warp * kMaxGroup + 2 * t + 1] = l1;
            }
        }
        // the warps' pieces become one: common maximum, rescaled sums and outputs
        named_barrier(1, kWarps * 32);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int head_c = 2 * t + c;
            if (head_c >= G) continue;
            float m = kLowest;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) m = fmaxf(m, wm[w * kMaxGroup + head_c]);
            const float f = exp2_fast(wm[warp * kMaxGroup + head_c] - m);
            float4 *dst = reinterpret_cast<float4 *>(red + (warp * G + head_c) * kHeadDim + 8 * g);
#pragma unroll
            for (int i = 0; i < 4; ++i)  // elements 64 (i / 2) + 8 g + 4 (i % 2) and the three behind it
                dst[i / 2 * 16 + i % 2] = make_float4(o[2 * i][c] * f, o[2 * i][c + 2] * f, o[2 * i + 1][c] * f, o[2 * i + 1][c + 2] * f);
        }
        named_barrier(1, kWarps * 32);
        float *out = a.ws + a.pieces.record(p, head) * G * (kHeadDim + 4);
        for (int i = tid; i < G * kHeadDim; i += kWarps * 32) {
            float s = 0.0f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) s += red[w * G * kHeadDim + i];
            out[i] = s;
        }
        if (tid < G) {
            float m = kLowest, l = 0.0f;
            for (int w = 0; w < kWarps; ++w) m = fmaxf(m, wm[w * kMaxGroup + tid]);
            for (int w = 0; w < kWarps; ++w) l += wl[w * kMaxGroup + tid] * exp2_fast(wm[w * kMaxGroup + tid] - m);
            out[G * kHeadDim + 2 * tid] = m;
            out[G * kHeadDim + 2 * tid + 1] = l;
        }
    }
}

// One or two sequences: a CTA takes one (sequence, K/V head, chunk of the cache): scores of the chunk for the G query heads
// (half a warp per key, fp32), their maximum and exp-sum, and the chunk's un-normalised output. As fast as the block form
// above where each processor sees few keys (one sequence of 2048 keys, 32 heads: 16.5 us both), and it takes 11 KiB of
// shared memory instead of 102: the matmuls of such a plan stream their weights through L1, and each of them ran 1 to 4 us
// longer beside the larger one (4 layers: 537 us against 577).
template <typename T, int G>
__device__ __noinline__ void attn_chunks(const DecodeAttnArgs &a, int p, int P, char *smem) {
    constexpr int D = kHeadDim;
    float *qs = reinterpret_cast<float *>(smem);                 // [G][D], already scaled
    float *ml = qs + G * D;                                      // [G][2]: maximum, exp-sum
    float *sc = ml + 2 * kMaxGroup;                              // [G][chunk_len]
    float *red = sc + (size_t)G * a.chunk_len;                   // [16][G][D]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int hw = tid >> 4, l16 = tid & 15;                     // half-warp index 0..31, lane within it
    const int chunks = a.pieces.per_span, items = a.B * a.Hkv * chunks;
    const T *qb = reinterpret_cast<const T *>(a.q);
    const T *kb = reinterpret_cast<const T *>(a.k);
    const T *vb = reinterpret_cast<const T *>(a.v);
    for (int item = p; item < items; item += P) {
        const int c = item % chunks, bh = item / chunks;
        const int kvh = bh % a.Hkv, b = bh / a.Hkv;
        const int t0 = c * a.chunk_len, len = min(a.chunk_len, a.T - t0);
        __syncthreads();  // the previous item's shared memory is no longer read
        for (int i = tid; i < G * D / 8; i += blockDim.x) {
            const int g = i / (D / 8), v = i % (D / 8);
            const uint4 q4 = *reinterpret_cast<const uint4 *>(qb + (int64_t)b * a.q_stride_b + (int64_t)(kvh * G + g) * a.q_stride_h + v * 8);
            float f[8];
            unpack8<T>(q4, f);
            if (a.rope) {
                // rotary embedding of the new token's query (complex multiply of adjacent pairs with the position's
                // (cos, sin) pairs), rounded like the separate operator would have stored it
                float t[8];
                unpack8<T>(*reinterpret_cast<const uint4 *>(reinterpret_cast<const T *>(a.rope) + v * 8), t);
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    const float re = f[e] * t[e] - f[e + 1] * t[e + 1], im = f[e] * t[e + 1] + f[e + 1] * t[e];
                    f[e] = to_f32(from_f32<T>(re));
                    f[e + 1] = to_f32(from_f32<T>(im));
                }
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) qs[g * D + v * 8 + e] = f[e] * a.scale;
        }
        __syncthreads();
        // scores: half a warp per key, 4 keys in flight
        const T *kbase = kb + (int64_t)b * a.k_stride_b + (int64_t)kvh * a.k_stride_h + (int64_t)t0 * a.k_ld + l16 * 8;
        float qr[G][8];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int e = 0; e < 8; ++e) qr[g][e] = qs[g * D + l16 * 8 + e];
        for (int jb = 2 * warp; jb < len; jb += 32 * 4) {  // same trip count in both halves of a warp (shuffles below)
            const int j0 = jb + (hw & 1);
            uint4 k4[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + 32 * u;
                k4[u] = j < len ? ldg16_stream(kbase + (int64_t)j * a.k_ld) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + 32 * u;
                float f[8];
                unpack8<T>(k4[u], f);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    float s = 0.0f;
#pragma unroll
                    for (int e = 0; e < 8; ++e) s += qr[g][e] * f[e];
                    s += __shfl_xor_sync(0xffffffffu, s, 8);
                    s += __shfl_xor_sync(0xffffffffu, s, 4);
                    s += __shfl_xor_sync(0xffffffffu, s, 2);
                    s += __shfl_xor_sync(0xffffffffu, s, 1);
                    if (l16 == 0 && j < len) sc[(size_t)g * a.chunk_len + j] = s;
                }
            }
        }
        __syncthreads();
        // per query head: maximum, exponentials in place, their sum (warp g)
        if (warp < G) {
            float *row = sc + (size_t)warp * a.chunk_len;
            float m = -3.402823466e+38f;
            for (int j = lane; j < len; j += 32) m = fmaxf(m, row[j]);
            m = warp_max(m);
            float l = 0.0f;
            for (int j = lane; j < len; j += 32) {
                const float e = __expf(row[j] - m);
                row[j] = e;
                l += e;
            }
            l = warp_sum(l);
            if (lane == 0) {
                ml[warp * 2] = m;
                ml[warp * 2 + 1] = l;
            }
        }
        __syncthreads();
        // un-normalised output: lanes of a half-warp cover the 128 columns, the 32 half-warps interleave the keys
        const T *vbase = vb + (int64_t)b * a.v_stride_b + (int64_t)kvh * a.v_stride_h + (int64_t)t0 * a.v_ld + l16 * 8;
        float acc[G][8];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[g][e] = 0.0f;
        for (int jb = 2 * warp; jb < len; jb += 32 * 4) {
            const int j0 = jb + (hw & 1);
            uint4 v4[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + 32 * u;
                v4[u] = j < len ? ldg16_stream(vbase + (int64_t)j * a.v_ld) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int j = j0 + 32 * u;
                if (j < len) {
                    float f[8];
                    unpack8<T>(v4[u], f);
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const float pj = sc[(size_t)g * a.chunk_len + j];
#pragma unroll
                        for (int e = 0; e < 8; ++e) acc[g][e] += pj * f[e];
                    }
                }
            }
        }
        // the two half-warps of a warp hold the same columns: add them, then the 16 warps through shared memory
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[g][e] += __shfl_xor_sync(0xffffffffu, acc[g][e], 16);
        if (lane < 16) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float4 *dst = reinterpret_cast<float4 *>(red + ((size_t)warp * G + g) * D + l16 * 8);
                dst[0] = make_float4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
                dst[1] = make_float4(acc[g][4], acc[g][5], acc[g][6], acc[g][7]);
            }
        }
        __syncthreads();
        float *w = a.ws + (size_t)item * G * (D + 4);
        const int nwarps = blockDim.x >> 5;
        for (int i = tid; i < G * D; i += blockDim.x) {
            float s = 0.0f;
            for (int wi = 0; wi < nwarps; ++wi) s += red[(size_t)wi * G * D + i];
            w[i] = s;  // [g][d]
        }
        if (tid < 2 * G) w[G * D + tid] = ml[tid];  // [g][maximum, sum]
    }
}

// Block form: element d of query head g of head `head` = (sequence, K/V head), un-normalised, and the exp-sum it is to be
// divided by. Maxima are in log2 units.
__device__ __forceinline__ float merge_pieces(const AttnPieces &pc, const float *ws, int head, int G, int g, int d, float &l) {
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
    float mx = kLowest, o = 0.0f;
    l = 0.0f;
    constexpr int B = 4;  // pieces on their way together
    for (int c0 = 0; c0 < n; c0 += B) {
        float2 ml[B];
        float v[B];
#pragma unroll
        for (int c = 0; c < B; ++c) {
            if (c0 + c >= n) continue;
            const float *w = c0 + c == 0 ? w0 : w1 + (c0 + c - 1) * step;
            ml[c] = __ldcg(reinterpret_cast<const float2 *>(w + G * 128 + 2 * g));
            v[c] = __ldcg(w + g * 128 + d);
        }
        float m = mx;
#pragma unroll
        for (int c = 0; c < B; ++c)
            if (c0 + c < n) m = fmaxf(m, ml[c].x);
        if (c0 > 0) {
            const float e = exp2_fast(mx - m);
            l *= e;
            o *= e;
        }
        mx = m;
#pragma unroll
        for (int c = 0; c < B; ++c) {
            if (c0 + c >= n) continue;
            const float e = exp2_fast(ml[c].x - mx);
            l += ml[c].y * e;
            o += v[c] * e;
        }
    }
    return o;
}

// Chunk form: the same; maxima as they are.
__device__ __forceinline__ float merge_chunks(const AttnPieces &pc, const float *ws, int head, int G, int g, int d, float &l) {
    const int n = pc.per_span, stride = G * 132;
    const float *w = ws + (int64_t)head * n * stride, *ml = w + G * 128 + 2 * g;
    w += g * 128 + d;
    float m = kLowest, o = 0.0f;
#pragma unroll 4
    for (int c = 0; c < n; ++c) m = fmaxf(m, __ldcg(ml + c * stride));
    l = 0.0f;
#pragma unroll 4
    for (int c = 0; c < n; ++c, w += stride, ml += stride) {
        const float2 x = __ldcg(reinterpret_cast<const float2 *>(ml));
        const float v = __ldcg(w), f = __expf(x.x - m);
        l += x.y * f;
        o += v * f;
    }
    return o;
}

// Merges the pieces of every (sequence, query head): thread per output element.
template <typename T>
__device__ void attn_merge(const DecodeAttnArgs &a, int p, int P) {
    constexpr int D = kHeadDim;
    const int G = a.Hq / a.Hkv, rows = a.B * a.Hq;
    T *out = reinterpret_cast<T *>(a.out);
    // a row of 128 outputs per four warps
    for (int row = p * (kThreads / D) + (int)threadIdx.x / D; row < rows; row += P * (kThreads / D)) {
        const int d = threadIdx.x % D, h = row % a.Hq, b = row / a.Hq;
        float l, o;
        if (a.chunk_len > 0) o = merge_chunks(a.pieces, a.ws, b * a.Hkv + h / G, G, h % G, d, l);
        else o = merge_pieces(a.pieces, a.ws, b * a.Hkv + h / G, G, h % G, d, l);
        out[(int64_t)b * a.o_stride_b + (int64_t)h * a.o_stride_h + d] = from_f32<T>(o / l);
    }
}

template <typename T>
__device__ __forceinline__ void attn_typed(const DecodeAttnArgs &a, int p, int P, char *smem) {
    if (a.phase == 1) attn_merge<T>(a, p, P);
    else if (a.chunk_len > 0) {
        switch (a.Hq / a.Hkv) {
            case 1: return attn_chunks<T, 1>(a, p, P, smem);
            case 2: return attn_chunks<T, 2>(a, p, P, smem);
            case 4: return attn_chunks<T, 4>(a, p, P, smem);
            default: return attn_chunks<T, 8>(a, p, P, smem);
        }
    } else if (p < a.pieces.runs && threadIdx.x < kWarps * 32) attn_pieces<T>(a, p, smem);
}

}  // namespace

__device__ __noinline__ void run_decode_attn(const DecodeAttnArgs &a, int p, int P, char *smem) {
    if (a.dtype == DT_BF16) attn_typed<__nv_bfloat16>(a, p, P, smem);
    else attn_typed<__half>(a, p, P, smem);
}

}  // namespace arkb
