// Matmul on the CUDA cores, fp32 accumulation: full-precision (fp32) operands, and 16-bit operands whose rows are no
// whole 16-byte vectors, which the tensor maps of the tensor-core form cannot describe.
//
// What bounds it is the FP32 pipe (128 multiply-adds per SM and clock) and, next to it, shared memory: a thread's
// 8 x 8 block takes 4 16-byte shared loads for 64 multiply-adds, which keeps the two about even; a 4 x 4 block (packed
// fma.rn.f32x2 included) was bound by its shared loads at a third of the pipe's rate.
//  * The CTA is two groups of 256 threads that work on the same tile, one on the even, one on the odd k-blocks, with
//    buffers and barriers of their own; the second group's sums are added to the first's once per tile. So a tile is
//    half as large as 512 threads would make it, which wastes less at ragged edges and cuts more evenly.
//  * Each group has two shared-memory buffers; the next k-block arrives (fp32: by asynchronous copies, which hold no
//    registers) while one is worked on: one barrier per k-block.
//  * An even split: the k-blocks of all output tiles form one list that is cut into equal runs, one per CTA (300 rows
//    by 1024 columns are 20 tiles, an eighth of the SMs; cut by k-block every SM gets the same work). A run that covers
//    a whole tile stores it; otherwise the fp32 piece goes to the workspace and phase 1, behind a barrier, adds a
//    tile's pieces in k order. The cut depends on the shape and the grid only, so results repeat bit for bit.
// Feed-forward block of 300 tokens, 1024 -> 4096 -> 1024, fp32, on one B200: 1298 us with 64 x 64 tiles of 2 x 4 blocks on
// whole output tiles per CTA, 235 us so.
#include "dev_common.cuh"
#include "dev_funcs.h"

namespace arkb {

namespace {

constexpr int kGroup = 256;  // threads that share a k-block

// Copies of one element (or four fp32 ones) into shared memory as fp32, zeros where there is none. fp32 travels
// asynchronously, 16-bit elements are widened on the way.
__device__ __forceinline__ void put1(float *d, const float *p, const float *any, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(in ? p : any), "r"(in ? 4 : 0)
                 : "memory");
}
template <typename T>
__device__ __forceinline__ void put1(float *d, const T *p, const T *, bool in) { *d = in ? to_f32(*p) : 0.0f; }
__device__ __forceinline__ void put4(float *d, const float *p, const float *any, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(d)), "l"(in ? p : any), "r"(in ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void puts_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Brings a ROWS x TK block of an operand into shared memory, [k][row] with rows of k padded by 4 floats (neighbouring
// k of one row, which neighbouring lanes bring in, then lie 4 banks apart). row_major: element (r, k) is
// base[r * ld + k], else base[k * ld + r].
template <int ROWS, int TK>
struct Block {
    static constexpr int kPitch = ROWS + 4;
    static constexpr int kFloats = TK * kPitch;

    template <typename T>
    static __device__ __forceinline__ void put(float *s, int t, const T *base, int64_t ld, int r0, int rows, int k0, int K, bool row_major,
                                               bool vec) {
        if (row_major) {
            constexpr int kStep = kGroup / TK;
            const int k = k0 + t % TK;
            int r = r0 + t / TK;
            const T *p = base + (int64_t)r * ld + k;
            float *d = s + t % TK * kPitch + t / TK;
#pragma unroll 4
            for (int j = 0; j < ROWS / kStep; ++j) {
                put1(d, p, base, r < rows && k < K);
                r += kStep; p += kStep * ld; d += kStep;
            }
            return;
        }
        if constexpr (sizeof(T) == 4) {
            if (vec && r0 + ROWS <= rows) {
#pragma unroll 4
                for (int u = t; u < ROWS * TK / 4; u += kGroup) {
                    const int r = u % (ROWS / 4) * 4, k = u / (ROWS / 4);
                    put4(s + k * kPitch + r, base + (int64_t)(k0 + k) * ld + r0 + r, base, k0 + k < K);
                }
                return;
            }
        }
#pragma unroll 4
        for (int u = t; u < ROWS * TK; u += kGroup) {
            const int r = u % ROWS, k = u / ROWS;
            put1(s + k * kPitch + r, base + (int64_t)(k0 + k) * ld + r0 + r, base, k0 + k < K && r0 + r < rows);
        }
    }
};

// First k-block of CTA p's run: the list of k-blocks is cut into runs of run_len + 1 (the first run_rem ones) and run_len.
__device__ __forceinline__ int64_t run_begin(const GemmSimtArgs &g, int p) { return (int64_t)p * g.run_len + min(p, g.run_rem); }
// CTA whose run holds k-block b
__device__ __forceinline__ int run_of(const GemmSimtArgs &g, int64_t b) {
    const int64_t longer = (int64_t)g.run_rem * (g.run_len + 1);
    return (int)(b < longer ? b / (g.run_len + 1) : g.run_rem + (b - longer) / g.run_len);
}

// WM of a group's 8 warps along the rows, 8 / WM along the columns; a warp covers 32 rows x 64 columns.
template <typename T, int WM>
__device__ __noinline__ void simt_products(const GemmSimtArgs &g, int p, float *smem) {
    constexpr int TM = 32 * WM, TN = 512 / WM, TK = WM == 1 ? 8 : 16;
    using BlockA = Block<TM, TK>;
    using BlockB = Block<TN, TK>;
    constexpr int kBuf = BlockA::kFloats + BlockB::kFloats;
    const int grp = threadIdx.x / kGroup, t = threadIdx.x % kGroup, lane = t & 31, warp = t >> 5;
    const int mrow = warp % WM * 32 + lane / 8 * 8, ncol = warp / WM * 64 + lane % 8 * 4;
    const int tiles_n = (g.N + TN - 1) / TN, per = (g.M + TM - 1) / TM * tiles_n;
    const int kblocks = g.kblocks;
    float *buf0 = smem + grp * 2 * kBuf;
    const int64_t b0 = run_begin(g, p), b1 = run_begin(g, p + 1);
    for (int64_t b = b0; b < b1;) {
        const int64_t tile = b / kblocks;
        const int kb0 = (int)(b - tile * kblocks), kb1 = (int)min((int64_t)kblocks, kb0 + (b1 - b));
        const int batch = (int)(tile / per), r = (int)(tile % per);
        const int bc = batch % g.batch_c, bn = batch / g.batch_c;
        const int m0 = r / tiles_n * TM, n0 = r % tiles_n * TN;
        float acc[8][8] = {};
        {
            const T *A = reinterpret_cast<const T *>(g.A) + bn * g.a_stride_n + bc * g.a_stride_c;
            const T *B = reinterpret_cast<const T *>(g.B) + bn * g.b_stride_n + bc * g.b_stride_c;
            auto put = [&](float *d, int kb) {
                BlockA::put(d, t, A, g.lda, m0, g.M, kb * TK, g.K, !g.trans_a, g.vec_a);
                BlockB::put(d + BlockA::kFloats, t, B, g.ldb, n0, g.N, kb * TK, g.K, g.trans_b, g.vec_b);
            };
            __syncthreads();  // shared memory may still be read for the tile before
            if (kb0 + grp < kb1) put(buf0, kb0 + grp);
            float *cur = buf0;
            for (int kb = kb0 + grp; kb < kb1; kb += 2) {
                puts_done();
                named_barrier(1 + grp, kGroup);  // this k-block is there; the other buffer has been read
                if (kb + 2 < kb1) put(buf0 + (cur == buf0 ? kBuf : 0), kb + 2);
                const float *sa = cur + mrow, *sb = cur + BlockA::kFloats + ncol;
#pragma unroll 4
                for (int k = 0; k < TK; ++k) {
                    float av[8], bv[8];
                    *reinterpret_cast<float4 *>(av) = *reinterpret_cast<const float4 *>(sa + k * BlockA::kPitch);
                    *reinterpret_cast<float4 *>(av + 4) = *reinterpret_cast<const float4 *>(sa + k * BlockA::kPitch + 4);
                    *reinterpret_cast<float4 *>(bv) = *reinterpret_cast<const float4 *>(sb + k * BlockB::kPitch);
                    *reinterpret_cast<float4 *>(bv + 4) = *reinterpret_cast<const float4 *>(sb + k * BlockB::kPitch + 32);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
                }
                cur = buf0 + (cur == buf0 ? kBuf : 0);
            }
        }
        // the second group's sums through shared memory (64 values of 256 threads; the buffers hold at least as much)
        __syncthreads();
        if (grp == 1) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                *reinterpret_cast<float4 *>(smem + (i * kGroup + t) * 4) = *reinterpret_cast<const float4 *>(&acc[i / 2][i % 2 * 4]);
        }
        __syncthreads();
        if (grp == 0) {
            auto sums = [&](int i, float (&v)[4]) {
                const float4 o = *reinterpret_cast<const float4 *>(smem + (i * kGroup + t) * 4);
                const float w[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = acc[i / 2][i % 2 * 4 + e] + w[e];
            };
            if (kb1 - kb0 < kblocks) {
                float *piece = g.ws + ((int64_t)p * 2 + (b == b0 ? 0 : 1)) * (TM * TN) + mrow * TN + ncol;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float v[4];
                    sums(i, v);
                    *reinterpret_cast<float4 *>(piece + i / 2 * TN + i % 2 * 32) = make_float4(v[0], v[1], v[2], v[3]);
                }
            } else {
                // out of the record: the stores below might alias it (read and tested anew for every result, the activation and
                // the edges made the stores of a tile 16 us)
                const int M = g.M, N = g.N, act = g.act, vec = g.vec_c;
                const int64_t ldc = g.ldc;
                T *C = reinterpret_cast<T *>(g.C) + bn * g.c_stride_n + bc * g.c_stride_c;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int row = m0 + mrow + i / 2, col = n0 + ncol + i % 2 * 32;
                    if (row >= M || col >= N) continue;
                    float v[4];
                    sums(i, v);
                    T *c = C + (int64_t)row * ldc + col;
                    if (act != ACT_NONE) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[e] = apply_act(act, v[e]);
                    }
                    if (vec && col + 4 <= N) {
                        store_vec<T, 4>(c, v);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (col + e < N) c[e] = from_f32<T>(v[e]);
                    }
                }
            }
        }
        b += kb1 - kb0;
    }
}

// Phase 1: tiles that more than one run has a piece of; a unit is an eighth of a tile, four elements per thread.
template <typename T, int WM>
__device__ __noinline__ void simt_sums(const GemmSimtArgs &g, int p, int P) {
    constexpr int TM = 32 * WM, TN = 512 / WM, kUnits = 8, kElems = TM * TN / kUnits;
    static_assert(kElems == kThreads * 4, "four elements per thread");
    const int tiles_n = (g.N + TN - 1) / TN, per = (g.M + TM - 1) / TM * tiles_n;
    const int64_t kblocks = g.kblocks, units = (int64_t)per * g.batch_c * g.batch_n * kUnits;
    for (int64_t u = p; u < units; u += P) {
        const int64_t tile = u / kUnits, t0 = tile * kblocks;
        const int first = run_of(g, t0), last = run_of(g, t0 + kblocks - 1);
        if (first == last) continue;
        const int batch = (int)(tile / per), r = (int)(tile % per);
        const int bc = batch % g.batch_c, bn = batch / g.batch_c;
        const int e = (int)(u % kUnits) * kElems + threadIdx.x * 4, row = r / tiles_n * TM + e / TN, col = r % tiles_n * TN + e % TN;
        if (row >= g.M || col >= g.N) continue;
        // the tile opens every run but the first, where it follows another tile unless the run begins with it
        const float *piece = g.ws + ((int64_t)first * 2 + (run_begin(g, first) == t0 ? 0 : 1)) * (TM * TN) + e;
        float4 s = __ldcg(reinterpret_cast<const float4 *>(piece));
#pragma unroll 4
        for (int q = first + 1; q <= last; ++q) {
            const float4 v = __ldcg(reinterpret_cast<const float4 *>(g.ws + (int64_t)q * 2 * (TM * TN) + e));
            s = make_float4(s.x + v.x, s.y + v.y, s.z + v.z, s.w + v.w);
        }
        T *C = reinterpret_cast<T *>(g.C) + bn * g.c_stride_n + bc * g.c_stride_c + (int64_t)row * g.ldc + col;
        const float v[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (col + i < g.N) C[i] = from_f32<T>(apply_act(g.act, v[i]));
    }
}

// Small products: whole 64 x 64 tiles, 2 x 4 results per thread. A tile is a quarter of the other form's, so that few tiles
// spread over more CTAs, and costs little besides its multiply-adds; see the rule in the lowering. Not inlined: the registers
// that the caller would save for it cost the large tiles' stages 4 us each.
template <typename T>
__device__ __noinline__ void simt_small(const GemmSimtArgs &g, int p, int P, float *smem) {
    constexpr int TM = 64, TN = 64, TK = 16;
    float(*sA)[TM + 1] = reinterpret_cast<float(*)[TM + 1]>(smem);                   // [TK][TM + 1]
    float(*sB)[TN + 1] = reinterpret_cast<float(*)[TN + 1]>(smem + TK * (TM + 1));   // [TK][TN + 1]
    const int tiles_m = (g.M + TM - 1) / TM, tiles_n = (g.N + TN - 1) / TN;
    const int64_t per = (int64_t)tiles_m * tiles_n, total = per * g.batch_c * g.batch_n;
    const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;  // rows 2 ty and 2 ty + 1, columns 4 tx to 4 tx + 3
    for (int64_t u = p; u < total; u += P) {
        const int batch = (int)(u / per), r = (int)(u % per);
        const int bc = batch % g.batch_c, bn = batch / g.batch_c;
        const int m0 = r / tiles_n * TM, n0 = r % tiles_n * TN;
        const T *A = reinterpret_cast<const T *>(g.A) + bn * g.a_stride_n + bc * g.a_stride_c;
        const T *B = reinterpret_cast<const T *>(g.B) + bn * g.b_stride_n + bc * g.b_stride_c;
        T *C = reinterpret_cast<T *>(g.C) + bn * g.c_stride_n + bc * g.c_stride_c;
        float acc[2][4] = {};
        for (int k0 = 0; k0 < g.K; k0 += TK) {
            for (int i = tid; i < TK * TM; i += kThreads) {
                const int kk = g.trans_a ? i / TM : i % TK, mm = g.trans_a ? i % TM : i / TK;
                const int m = m0 + mm, k = k0 + kk;
                float v = 0.0f;
                if (m < g.M && k < g.K) v = to_f32(g.trans_a ? A[(int64_t)k * g.lda + m] : A[(int64_t)m * g.lda + k]);
                sA[kk][mm] = v;
            }
            for (int i = tid; i < TK * TN; i += kThreads) {
                const int kk = g.trans_b ? i % TK : i / TN, nn = g.trans_b ? i / TK : i % TN;
                const int n = n0 + nn, k = k0 + kk;
                float v = 0.0f;
                if (n < g.N && k < g.K) v = to_f32(g.trans_b ? B[(int64_t)n * g.ldb + k] : B[(int64_t)k * g.ldb + n]);
                sB[kk][nn] = v;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < TK; ++kk) {
                const float a0 = sA[kk][ty * 2], a1 = sA[kk][ty * 2 + 1];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float bv = sB[kk][tx * 4 + j];
                    acc[0][j] += a0 * bv;
                    acc[1][j] += a1 * bv;
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int m = m0 + ty * 2 + i, n = n0 + tx * 4 + j;
                if (m < g.M && n < g.N) C[(int64_t)m * g.ldc + n] = from_f32<T>(apply_act(g.act, acc[i][j]));
            }
    }
}

template <typename T>
__device__ void simt_typed(const GemmSimtArgs &g, int p, int P, float *smem) {
    if (g.phase == 1) {
        switch (g.wm) {
            case 1: simt_sums<T, 1>(g, p, P); break;
            case 2: simt_sums<T, 2>(g, p, P); break;
            default: simt_sums<T, 4>(g, p, P); break;
        }
        return;
    }
    if (g.wm == 0) {
        simt_small<T>(g, p, P, smem);
        return;
    }
    if (p >= g.runs) return;
    switch (g.wm) {
        case 1: simt_products<T, 1>(g, p, smem); break;
        case 2: simt_products<T, 2>(g, p, smem); break;
        default: simt_products<T, 4>(g, p, smem); break;
    }
}

}  // namespace

__device__ __noinline__ void run_gemm_simt(const GemmSimtArgs &g, int p, int P, char *smem) {
    float *s = reinterpret_cast<float *>(smem);
    switch (g.dtype) {
        case DT_F32: simt_typed<float>(g, p, P, s); break;
        case DT_F16: simt_typed<__half>(g, p, P, s); break;
        case DT_BF16: simt_typed<__nv_bfloat16>(g, p, P, s); break;
        default: break;
    }
}

}  // namespace arkb
